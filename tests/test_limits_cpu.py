"""Limits that the library's index types have to hold, taken from its own
headers: compiled and run on the host."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "minirender_gb300", "csrc")


def _run(tmp_path, body):
    from minirender_gb300 import build
    cuda = os.path.join(os.path.dirname(os.path.realpath(build.nvcc())), "..", "include")
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text('#include <stdio.h>\n#include <limits>\n#include "internal.h"\nint main() {\n' + body + "\n}\n")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-isystem", cuda, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()


def test_pair_numbers_hold_a_warp_of_frame_sized_records(tmp_path):
    """32 records over every tile of the largest scene, for every tile shape
    that is accepted: the kernel numbers these pairs with PairNo."""
    most, held = _run(tmp_path, """
      unsigned long long most = 0;
      for (int tw = 1; tw <= 4096; tw *= 2)
        for (int th = 1; th <= 4096; th *= 2)
          if (mrg::batch_tile_ok(tw, th)) {
            const unsigned long long tiles = (unsigned long long)(mrg::kMaxSide / tw) * (mrg::kMaxSide / th);
            if (32 * tiles > most) most = 32 * tiles;
          }
      printf("%llu %llu", most, (unsigned long long)std::numeric_limits<mrg::PairNo>::max());""")
    assert int(most) == 1 << 31
    assert int(held) >= int(most)
