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


def test_warps_are_spread_over_the_record_shares(tmp_path):
    """Of each sixteen warps in a row one goes to each share (what the stores'
    sizes count on), and warps that recur at any regular distance meet in no
    share more than twice as often as in the mean."""
    bad_rows, worst = _run(tmp_path, """
      int bad = 0;
      double worst = 0;
      for (uint32_t g = 0; g < 70000; g++) {
        unsigned seen = 0;
        for (uint32_t k = 0; k < 16; k++) seen |= 1u << mrg::share_of_warp(16 * g + k);
        bad += seen != 0xffffu;
      }
      for (uint32_t step = 1; step <= 1024; step++)
        for (uint32_t first = 0; first < 16; first++) {
          int n[mrg::kShares] = {};
          for (uint32_t k = 0; k < 1024; k++) n[mrg::share_of_warp(first + k * step)]++;
          for (int c : n) worst = c > worst ? c : worst;
        }
      printf("%d %g", bad, worst / (1024 / mrg::kShares));""")
    assert int(bad_rows) == 0
    assert float(worst) <= 2
