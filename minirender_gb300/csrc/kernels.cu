// GB300 (sm_103a) kernels of the rasterisation path.
//
// One frame per call (launch_frame):
//   k_begin        vis[] = VIS_EMPTY                 (Renderer::clear, src/Renderer.cpp:113-119)
//                  and, for a frame of one renderable, the vertex pass
//   k_vertex       (frames of several renderables, batches) per-vertex view
//                  transform + projection to pixel space and
//                  per-normal transform, once per frame (the PREMULT loops,
//                  src/Renderer.cpp:344-348, plus htransform :13-20 and the
//                  pixel mapping :193-197, which depend on the vertex only)
//   k_setup        triangle assembly + near clip + triangle setup + cull;
//                  small triangles rasterised by the warp that set them up,
//                  one (triangle, row) per lane; large ones appended to a
//                  warp-compacted record list with their blocks
//                                                   (src/Renderer.cpp:121-269, 351-379)
//   k_raster_large one warp per block (32 rows by a column segment) of a large
//                  sub-triangle, one row per lane, 64-bit atomicMin
//                                                   (src/Renderer.cpp:238-269)
//   k_resolve      deferred pass: re-derives the winning sub-triangle's
//                  barycentrics exactly, shades once per visible pixel and
//                  writes RGB8/depth/ids            (src/Renderer.cpp:271-305, src/io.cpp:358-362)
// Many frames per call (launch_batch):
//   k_vertex (when vertices are shared), then k_setup_batch (sub-triangles
//   with a bounding box of at most small_max pixels rasterised into their
//   scene's visibility words, which the batch before left empty, larger ones
//   become records counted into the scene's tiles), then k_batch: one
//   cooperative, persistent launch -- list ranges, scatter, and a dynamically
//   scheduled loop over strips of all tiles of all scenes, one warp each, that
//   rasterises the tile's records into shared memory (seeded with the small
//   triangles' words, which it empties) and resolves + shades the strip's
//   pixels in place.  The PRE template flag is false for triangle soups: no
//   vertex pass, kernels transform corners themselves.
// Also: k_validate (index checks at upload), k_range (getRangeImage,
// src/Renderer.cpp:388-415).
//
// Exactness: every float operation follows the reference's order; the edge
// functions are advanced column by column from the bounding-box edge exactly
// as the reference loop does (the running sums have no closed form), so every
// rasteriser and the resolve replay that chain.  Values the vertex pass stores
// are the same expressions the reference evaluates per triangle corner.
// Kernels templated on PRE read the vertex-pass buffers; without them
// (triangle soups, allocation-free entry point) vertices are transformed per
// triangle.  ONE: the frame's only renderable is read from the parameters.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "raster.cuh"

namespace cg = cooperative_groups;

namespace mrg {

// ------------------------------------------------------------------ helpers
// Programmatic dependent launch (sm_90+): a kernel launched with programmatic
// stream serialisation may be scheduled while its predecessor is finishing;
// pdl_wait() blocks until the predecessor grid has completed and its writes
// are visible (a no-op for a kernel launched the ordinary way); pdl_trigger()
// lets the successor's blocks start launching.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ int find_base(const uint32_t* base, int lo, int hi, uint32_t g) {
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (base[mid] <= g) lo = mid; else hi = mid;
  }
  return lo;
}

// find_base for the warp's consecutive g (lane 0 holds the smallest; every
// lane calls): 32 candidates a round find lane 0's entry -- three dependent
// loads for 16384 renderables instead of fourteen -- and the other lanes step
// on from there: over 31 renderables with triangles at most, but over any
// number of empty ones, so a longer way is searched again.  n entries; base[n]
// is the end.
__device__ __forceinline__ int find_base_warp(const uint32_t* base, int n, uint32_t g) {
  const int lane = (int)(threadIdx.x & 31);
  const uint32_t g0 = __shfl_sync(0xffffffffu, g, 0);
  int lo = 0;
  for (int m = n; m > 1;) {
    const int step = (m + 31) >> 5, j = lane * step;
    const unsigned hit = __ballot_sync(0xffffffffu, j < m && base[lo + j] <= g0);
    const int at = (31 - __clz((int)(hit | 1u))) * step;
    lo += at;
    m = min(step, m - at);
  }
  for (int last = lo + 32; lo + 1 < n && base[lo + 1] <= g; lo++)
    if (lo == last) return find_base(base, lo, n, g);
  return lo;
}

__device__ __forceinline__ V3 ld3(const float* p, int i) {
  return v3(__ldg(p + 3 * i), __ldg(p + 3 * i + 1), __ldg(p + 3 * i + 2));
}
__device__ __forceinline__ V2 ld2(const float* p, int i) {
  return v2(__ldg(p + 2 * i), __ldg(p + 2 * i + 1));
}

// Two IEEE binary32 additions in one instruction (each half is rounded as the
// scalar addition rounds); the setup and resolve kernels are bound by
// instruction issue.  Products stay scalar: a packed multiply feeding a packed
// add came out one unit in the last place off, as a fused one does.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// htransform, src/Renderer.cpp:13-20
__device__ __forceinline__ V3 htransform(const float* m, V3 p) {
  float iw = rcp(m[12] * p.x + m[13] * p.y + m[14] * p.z + m[15]);
  return v3((m[0] * p.x + m[1] * p.y + m[2] * p.z + m[3]) * iw,
            (m[4] * p.x + m[5] * p.y + m[6] * p.z + m[7]) * iw,
            (m[8] * p.x + m[9] * p.y + m[10] * p.z + m[11]) * iw);
}

// Pixel coordinates and depth term of one corner, src/Renderer.cpp:186-197, 223-224.
__device__ __forceinline__ void project(const View& V, V3 v, float& px, float& py, float& zt) {
  V3 ndc = htransform(V.P, v);
  px = (1 + ndc.x) * (V.w / 2);
  py = (1 - ndc.y) * (V.h / 2);
  zt = V.persp ? -rcp(v.z) : ndc.z;
}

// project() of a triangle's three corners.  For V.simple matrices and finite
// corners off the z = 0 plane the products with zero entries are +-0, which
// change no sum that reaches a pixel coordinate, w is exactly -z, and the
// perspective z term -1/z is the 1/w already taken: 10 operations and a
// reciprocal a corner instead of 35 and two.
__device__ __forceinline__ void project3(const View& V, const Vtx (&v)[3], V2 (&p)[3], float (&zt)[3]) {
  const float size = ((fabsf(v[0].pos.x) + fabsf(v[0].pos.y)) + (fabsf(v[1].pos.x) + fabsf(v[1].pos.y))) +
                     ((fabsf(v[2].pos.x) + fabsf(v[2].pos.y)) +
                      (fabsf(v[0].pos.z) + (fabsf(v[1].pos.z) + fabsf(v[2].pos.z))));  // NaN or inf: not finite
  const float zmin = fminf(fminf(fabsf(v[0].pos.z), fabsf(v[1].pos.z)), fabsf(v[2].pos.z));
  if (V.simple && size < __int_as_float(0x7f800000) && zmin > 0) {
    const float hw = V.w / 2, hh = V.h / 2;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const V3 q = v[c].pos;
      const float iw = rcp(-q.z);
      p[c].x = (1 + (V.P[0] * q.x + V.P[2] * q.z) * iw) * hw;
      p[c].y = (1 - (V.P[5] * q.y + V.P[6] * q.z) * iw) * hh;
      zt[c] = iw;
    }
  } else {
#pragma unroll
    for (int c = 0; c < 3; c++) project(V, v[c].pos, p[c].x, p[c].y, zt[c]);
  }
}

// clip(), src/Renderer.cpp:121-129
template <bool ATTR>
__device__ __forceinline__ Vtx clip_vtx(float z, const Vtx& a, const Vtx& b) {
  float k = (fabsf(b.pos.z - a.pos.z) < 1e-6f) ? 0.5f : (z - a.pos.z) / (b.pos.z - a.pos.z);
  float k1 = 1 - k;
  Vtx v;
  v.pos = add3(ks3(k, b.pos), ks3(k1, a.pos));
  if (ATTR) {
    v.nrm = add3(ks3(k, b.nrm), ks3(k1, a.nrm));
    v.uv = add2(ks2(k, b.uv), ks2(k1, a.uv));
  }
  return v;
}

// clipTriangle, src/Renderer.cpp:131-161, for a triangle with a corner behind
// the near plane: the number of its sub-triangles (0, 1 or 2), and sub-triangle
// `sub` (when there is one of that number) in place of v.
template <bool ATTR>
__device__ __forceinline__ int clip_pick(float zn, Vtx (&v)[3], int sub) {
  if (v[0].pos.z > zn && v[1].pos.z > zn && v[2].pos.z > zn) return 0;
  // rotate until v[0] has the largest z (at most two turns for any input)
  for (int it = 0; it < 3 && (v[0].pos.z < v[1].pos.z || v[0].pos.z < v[2].pos.z); it++) {
    Vtx t0 = v[0]; v[0] = v[2]; v[2] = v[1]; v[1] = t0;
  }
  if (v[1].pos.z > zn) {
    const Vtx a = clip_vtx<ATTR>(zn, v[0], v[2]);
    v[1] = clip_vtx<ATTR>(zn, v[1], v[2]);
    v[0] = a;
    return 1;
  }
  if (v[2].pos.z > zn) {
    const Vtx a = clip_vtx<ATTR>(zn, v[0], v[1]);
    v[2] = clip_vtx<ATTR>(zn, v[1], v[2]);
    v[0] = a;
    return 1;
  }
  const Vtx v01 = clip_vtx<ATTR>(zn, v[0], v[1]);
  if (sub) {  // (v01, v2, v02)
    const Vtx v02 = clip_vtx<ATTR>(zn, v[0], v[2]);
    v[1] = v[2];
    v[2] = v02;
  }
  v[0] = v01;
  return 2;
}

// Attributes of a corner that the fragments of a renderable read
// (DevRenderable::need; a corner cut by the near plane takes all).
__device__ __forceinline__ bool needs(const DevRenderable& R, int what, bool cut) { return cut || (R.need & what); }

// View-space corners of triangle t without the vertex pass (paintMesh,
// src/Renderer.cpp:344-379).
template <bool ATTR>
__device__ __forceinline__ void corners(const DevRenderable& R, int t, const int (&ip)[3], Vtx (&v)[3]) {
  const DevMesh& M = R.mesh;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    v[c].pos = affine(R.mv, ld3(M.pos, ip[c]));
    if (ATTR) {
      v[c].nrm = affine(R.nm, ld3(M.nrm, __ldg(M.nidx + 3 * t + c)));
      v[c].uv = M.has_uv ? ld2(M.uv, __ldg(M.tidx + 3 * t + c)) : v2(0, 0);
    }
  }
}

// The attributes of vertices gv (in the frame's vertex buffers; the corners
// of triangle t) that R's fragments read.  A unified mesh has them all in
// vc: normal and view x, view y and texcoord -- two sectors at most a corner
// where positions, normals and texcoords were three scattered ones.
__device__ __forceinline__ void vertex_attributes(const Geo& G, const DevRenderable& R, int t, const uint32_t (&gv)[3],
                                                  bool cut, Vtx (&v)[3]) {
  const bool nrm = needs(R, kNeedNormal, cut), uv = needs(R, kNeedTexcoord, cut), pos = needs(R, kNeedPosition, cut);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    if (nrm || pos) {
      const float4 a = G.vc[2 * (size_t)gv[c]];
      v[c].nrm = v3(a.x, a.y, a.z);
      v[c].pos.x = a.w;
    }
    if (uv || pos) {
      const float4 b = G.vc[2 * (size_t)gv[c] + 1];
      v[c].pos.y = b.x;
      v[c].uv = v2(b.y, b.z);
    }
  }
  if (!R.unified) {
    const DevMesh& M = R.mesh;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (nrm) {
        const float4 n = G.vn[R.nrm_base + __ldg(M.nidx + 3 * t + c)];
        v[c].nrm = v3(n.x, n.y, n.z);
      }
      if (uv) v[c].uv = M.has_uv ? ld2(M.uv, __ldg(M.tidx + 3 * t + c)) : v2(0, 0);
    }
  }
}

// Corner record of a triangle (32 words, 128 bytes; DevMesh::rec):
//   words 0-8   corner positions p0, p1, p2
//   word 15     layout flag: kRecPerFace or 0
// per-face layout (one normal index and one texcoord index for all three
// corners, as in a soup with face normals: everything in the first 64 bytes)
//   words 9-11  the normal, 12-13 the texcoord, 14 zero
// per-corner layout
//   words 9-11  n0, 12-14 n1, 16-18 n2, 19-24 uv0, uv1, uv2
// Texcoords are zero for meshes without them.
constexpr uint32_t kRecPerFace = 1u;

// The view-space corners with attributes of triangle t from its corner
// record: the same values corners<true> gathers (src/Renderer.cpp:
// 344-348, 356-373).  A per-face record needs its first 64 bytes only.
__device__ __forceinline__ void corners_rec(const DevRenderable& R, int t, Vtx (&v)[3]) {
  const float4* r = R.mesh.rec + (size_t)8 * t;
  float4 q0, q1, q2, q3;  // two 32-byte loads
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=f"(q0.x), "=f"(q0.y), "=f"(q0.z), "=f"(q0.w), "=f"(q1.x), "=f"(q1.y), "=f"(q1.z), "=f"(q1.w) : "l"(r));
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=f"(q2.x), "=f"(q2.y), "=f"(q2.z), "=f"(q2.w), "=f"(q3.x), "=f"(q3.y), "=f"(q3.z), "=f"(q3.w) : "l"(r + 2));
  v[0].pos = affine(R.mv, v3(q0.x, q0.y, q0.z));
  v[1].pos = affine(R.mv, v3(q0.w, q1.x, q1.y));
  v[2].pos = affine(R.mv, v3(q1.z, q1.w, q2.x));
  const V3 n0 = v3(q2.y, q2.z, q2.w);
  if (__float_as_uint(q3.w) == kRecPerFace) {
    const V3 n = affine(R.nm, n0);
    const V2 uv = R.mesh.has_uv ? v2(q3.x, q3.y) : v2(0, 0);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      v[c].nrm = n;
      v[c].uv = uv;
    }
  } else {
    const float4 q4 = __ldg(r + 4), q5 = __ldg(r + 5), q6 = __ldg(r + 6);
    v[0].nrm = affine(R.nm, n0);
    v[1].nrm = affine(R.nm, v3(q3.x, q3.y, q3.z));
    v[2].nrm = affine(R.nm, v3(q4.x, q4.y, q4.z));
    if (R.mesh.has_uv) {
      v[0].uv = v2(q4.w, q5.x);
      v[1].uv = v2(q5.y, q5.z);
      v[2].uv = v2(q5.w, q6.x);
    } else {
      v[0].uv = v[1].uv = v[2].uv = v2(0, 0);
    }
  }
}

struct Setup {
  V2 p0, p2, n1, n2;
  float z[3];
  int x0, y0, x1, y1;
};

// The edge functions of paintTriangle's setup, src/Renderer.cpp:204-224, of a
// triangle with signed area a > 0 (or NaN).
__device__ __forceinline__ void setup_edges(const V2 (&p)[3], const float (&zt)[3], float a, Setup& S) {
  const float i2a = -rcp(a);
  float ex = p[0].x - p[2].x, ey = p[0].y - p[2].y;
  S.n1 = v2(-ey * i2a, ex * i2a);
  ex = p[1].x - p[0].x;
  ey = p[1].y - p[0].y;
  S.n2 = v2(-ey * i2a, ex * i2a);
  S.p0 = p[0];
  S.p2 = p[2];
  S.z[0] = zt[0];
  S.z[1] = zt[1];
  S.z[2] = zt[2];
}
__device__ __forceinline__ float area2(const V2 (&p)[3]) {
  const float d0x = p[0].x - p[1].x, d0y = p[0].y - p[1].y;
  const float d2x = p[2].x - p[1].x, d2y = p[2].y - p[1].y;
  return d0x * d2y - d0y * d2x;
}
// Least and greatest of three coordinates, a NaN among them ignored as the
// reference's running comparisons from +-1e30 ignore it (src/Renderer.cpp:
// 198-203; the sign of a zero, which min and max may choose differently, is
// lost in the clamp and floor that follow).
__device__ __forceinline__ float least(float a, float b, float c) { return fminf(fminf(fminf(a, b), c), 1e30f); }
__device__ __forceinline__ float greatest(float a, float b, float c) { return fmaxf(fmaxf(fmaxf(a, b), c), -1e30f); }
// Pixel of a coordinate clamped to 0..n-1.
__device__ __forceinline__ int pixel_of(float x, float n) { return __float2int_rd(fminf(fmaxf(x, 0.f), n - 1)); }

// paintTriangle setup from projected corners, src/Renderer.cpp:198-224.
// False = nothing to draw (off screen or culled).
__device__ __forceinline__ bool setup_from(const View& V, const V2 (&p)[3], const float (&zt)[3], Setup& S) {
  const float xmin = least(p[0].x, p[1].x, p[2].x), ymin = least(p[0].y, p[1].y, p[2].y);
  const float xmax = greatest(p[0].x, p[1].x, p[2].x), ymax = greatest(p[0].y, p[1].y, p[2].y);
  if (xmax < 0 || ymax < 0 || xmin > V.w || ymin > V.h) return false;
  const float a = area2(p);
  if (a <= 0) return false;  // back-face cull, :207-210
  setup_edges(p, zt, a, S);
  S.x0 = pixel_of(xmin, V.w);
  S.y0 = pixel_of(ymin, V.h);
  S.x1 = pixel_of(xmax, V.w);
  S.y1 = pixel_of(ymax, V.h);
  return true;
}

// Edge functions at the start of row y (pixel centre x0+0.5), :240-242.
__device__ __forceinline__ unsigned long long row_start2(const Setup& S, int y) {
  const float yf = (float)y + 0.5f, ptx = (float)S.x0 + 0.5f;
  return pack2(S.n1.x * (ptx - S.p2.x) + S.n1.y * (yf - S.p2.y), S.n2.x * (ptx - S.p0.x) + S.n2.y * (yf - S.p0.y));
}

// Depth of a covered fragment and its perspective-corrected weights, :247-261.
__device__ __forceinline__ float frag_depth(const Setup& S, bool persp, float e1, float e2,
                                            float& k0, float& k1, float& k2) {
  k0 = 1.f - e1 - e2;
  k1 = e1;
  k2 = e2;
  if (persp) {
    float z = rcp(k0 * S.z[0] + k1 * S.z[1] + k2 * S.z[2]);
    k0 *= S.z[0] * z;
    k1 *= S.z[1] * z;
    k2 *= S.z[2] * z;
    return z;
  }
  return k0 * S.z[0] + k1 * S.z[1] + k2 * S.z[2] + 0.0f * 1.0f;
}

// !(e1 < 0 || e2 < 0 || 1 - e1 - e2 < 0): a NaN is not below zero, and min
// ignores it.
__device__ __forceinline__ bool covered(float e1, float e2) { return !(fminf(fminf(e1, e2), 1 - e1 - e2) < 0); }

// The edge values n columns on: n running sums, column by column.
__device__ __forceinline__ unsigned long long advance2(unsigned long long e, unsigned long long d, int n) {
#pragma unroll 1
  for (; n >= 8; n -= 8) {
#pragma unroll
    for (int k = 0; k < 8; k++) e = add2(e, d);
  }
  if (n & 4) e = add2(add2(add2(add2(e, d), d), d), d);
  if (n & 2) e = add2(add2(e, d), d);
  if (n & 1) e = add2(e, d);
  return e;
}

// Walks row y from the bounding-box edge S.x0 to column xe and calls
// emit(x, packed) for every fragment that would pass z < 1e11f.
template <typename Emit>
__device__ __forceinline__ void walk_row(const Setup& S, bool persp, uint32_t id, int y, int xe, Emit emit) {
  const unsigned long long d = pack2(S.n1.x, S.n2.x);
  unsigned long long e = row_start2(S, y);
  for (int x = S.x0; x <= xe; x++) {
    float e1, e2;
    unpack2(e, e1, e2);
    if (covered(e1, e2)) {
      float k0, k1, k2;
      const float z = frag_depth(S, persp, e1, e2, k0, k1, k2);
      if (z < 1e11f) emit(x, ((unsigned long long)depth_key(z) << 32) | id);
    }
    e = add2(e, d);
  }
}

// Columns S.x0 + lo .. S.x0 + hi outside of which the row that starts with
// edge values (e1, e2) covers nothing: each edge function is a line whose
// crossing of zero bounds the covered run, give or take the rounding of the
// running sums.  err bounds that rounding (a column's sum is off by at most
// half a unit in the last place of the largest edge value per column, taken
// four times over), so the walk may start and stop there and still visits
// every pixel the reference covers.  Values that are not finite bound nothing.
__device__ __forceinline__ void edge_bound(float e, float g, float err, float& lo, float& hi) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(g));
  const float q = -e * r, m = err * fabsf(r) + (fabsf(q) * 2e-6f + 1e-3f);
  if (g > 0) lo = fmaxf(lo, q - m);
  if (g < 0) hi = fminf(hi, q + m);
}
__device__ __forceinline__ void covered_run(const Setup& S, unsigned long long e, int cols, int& lo, int& hi) {
  float e1, e2;
  unpack2(e, e1, e2);
  const float d1 = S.n1.x, d2 = S.n2.x, w = (float)cols;
  const float size = (fabsf(e1) + fabsf(e2) + 1.f) + w * (fabsf(d1) + fabsf(d2));
  const float err = (w + 8.f) * size * 2.4e-7f;
  float a = 0.f, b = w;
  edge_bound(e1, d1, err, a, b);
  edge_bound(e2, d2, err, a, b);
  edge_bound(1.f - e1 - e2, -(d1 + d2), err, a, b);
  lo = (int)ceilf(fminf(a, w));
  hi = (int)floorf(fmaxf(b, -1.f));
}

// The first column of xs..xe of row y that the row may cover, with its running
// edge values e (which step column by column from S.x0), and the length of the
// run up to the last such column (0: none).
__device__ __forceinline__ int row_run(const Setup& S, int y, int& xs, int xe, unsigned long long& e) {
  e = row_start2(S, y);
  int lo, hi;
  covered_run(S, e, xe - S.x0 + 1, lo, hi);
  xs = max(xs, S.x0 + lo);
  const int len = max(0, min(xe, S.x0 + hi) - xs + 1);
  if (len) e = advance2(e, pack2(S.n1.x, S.n2.x), xs - S.x0);
  return len;
}

// The runs of a warp's rows (one row per lane: len columns from the edge
// values e0, its first pixel at `at`), cut into pieces of kPiece columns and
// dealt one per lane: depth and put(pixel, word) of every fragment that passes
// z < 1e11f (src/Renderer.cpp:243-269).  A lane that walked its own row to the
// end would wait for the warp's longest.  256 scenes' fused stage 1826 us with
// pieces of 2, 1879 with 1, 1855 with 4, 2104 with 8.  Called by all lanes of
// the warp.
constexpr int kPiece = 2;
template <typename Cell, typename Put>
__device__ __forceinline__ void raster_runs(const Setup& S, bool persp, uint32_t id, unsigned long long e0, int len,
                                            Cell at, Put put) {
  const int lane = (int)(threadIdx.x & 31);
  const int pieces = (len + kPiece - 1) / kPiece;
  int inc = pieces;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  const int total = __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll 1
  for (int q = 0; q < total; q += 32) {
    const int j = q + lane;
    int own = 0;  // the lane whose row piece j belongs to
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (__shfl_sync(0xffffffffu, inc, own + step - 1) <= j) own += step;
    const int first = kPiece * (j - __shfl_sync(0xffffffffu, inc - pieces, own));
    Setup T;
    T.n1.x = __shfl_sync(0xffffffffu, S.n1.x, own);
    T.n2.x = __shfl_sync(0xffffffffu, S.n2.x, own);
#pragma unroll
    for (int c = 0; c < 3; c++) T.z[c] = __shfl_sync(0xffffffffu, S.z[c], own);
    const uint32_t tid = __shfl_sync(0xffffffffu, id, own);
    unsigned long long e = __shfl_sync(0xffffffffu, e0, own);
    const Cell cell = __shfl_sync(0xffffffffu, at, own) + (Cell)first;
    const int n = __shfl_sync(0xffffffffu, len, own) - first;
    if (j >= total) continue;
    const unsigned long long d = pack2(T.n1.x, T.n2.x);
    e = advance2(e, d, first);
#pragma unroll
    for (int x = 0; x < kPiece; x++) {
      float e1, e2;
      unpack2(e, e1, e2);
      if (x < n && covered(e1, e2)) {
        float k0, k1, k2;
        const float z = frag_depth(T, persp, e1, e2, k0, k1, k2);
        if (z < 1e11f) put(cell + (Cell)x, ((unsigned long long)depth_key(z) << 32) | tid);
      }
      if (x + 1 < kPiece) e = add2(e, d);
    }
  }
}

// Column segments of a large sub-triangle's bounding box (see kLargeCols).
__device__ __forceinline__ int large_seg_cols(int x0, int x1) {
  return kLargeCols * ((x1 - x0) / (kLargeCols * kLargeSegs) + 1);
}
__device__ __forceinline__ int large_segs(int x0, int x1) { return (x1 - x0) / large_seg_cols(x0, x1) + 1; }
__device__ __forceinline__ int large_blocks(int x0, int y0, int x1, int y1) {
  return ((y1 - y0) / kLargeRows + 1) * large_segs(x0, x1);
}

// The counters' slots of a warp: its statistics, and its share of the record
// store and block list.
__device__ __forceinline__ uint32_t warp_slot() { return ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) % kStatSlots; }
__device__ __forceinline__ uint32_t warp_share() { return share_of_warp((blockIdx.x * blockDim.x + threadIdx.x) >> 5); }

// Adds a warp's sub-triangles (small: rasterised by the setup kernel) and
// cut triangles to its statistics slot.  Called by all lanes of the warp.
__device__ __forceinline__ void count_triangles(Counters* c, bool small, bool big, bool cut) {
  const unsigned s = __ballot_sync(0xffffffffu, small), l = __ballot_sync(0xffffffffu, big);
  const unsigned k = __ballot_sync(0xffffffffu, cut);
  if ((threadIdx.x & 31) == 0 && (s | l | k)) {
    StatSlot& slot = c->stat[warp_slot()];
    if (s | l) atomicAdd(&slot.drawn, ((unsigned long long)(__popc(s) + __popc(l)) << 32) | (unsigned)__popc(s));
    if (k) atomicAdd(&slot.clipped, (unsigned long long)__popc(k));
  }
}

__device__ __forceinline__ BigRec to_rec(const Setup& S, uint32_t id) {
  BigRec B;
  B.p0x = S.p0.x; B.p0y = S.p0.y; B.p2x = S.p2.x; B.p2y = S.p2.y;
  B.n1x = S.n1.x; B.n1y = S.n1.y; B.n2x = S.n2.x; B.n2y = S.n2.y;
  B.z0 = S.z[0]; B.z1 = S.z[1]; B.z2 = S.z[2];
  B.id = id;
  B.x0 = S.x0; B.y0 = S.y0; B.x1 = S.x1; B.y1 = S.y1;
  return B;
}

__device__ __forceinline__ Setup rec_setup(const BigRec& B) {
  Setup S;
  S.p0 = v2(B.p0x, B.p0y); S.p2 = v2(B.p2x, B.p2y);
  S.n1 = v2(B.n1x, B.n1y); S.n2 = v2(B.n2x, B.n2y);
  S.z[0] = B.z0; S.z[1] = B.z1; S.z[2] = B.z2;
  S.x0 = B.x0; S.y0 = B.y0; S.x1 = B.x1; S.y1 = B.y1;
  return S;
}

// Leaves a drawn triangle's vertices and renderable k for the resolve.
__device__ __forceinline__ void note_triangle(const Geo& G, const DevRenderable& R, uint32_t k, int t) {
  if (!G.tri) return;
  const int* i = R.mesh.idx + 3 * (size_t)t;
  G.tri[R.tri_base + (uint32_t)t] = make_uint4(R.vert_base + (uint32_t)__ldg(i), R.vert_base + (uint32_t)__ldg(i + 1),
                                               R.vert_base + (uint32_t)__ldg(i + 2), k);
}

// Whether triangle t's indices failed the upload check.
__device__ __forceinline__ bool bad_triangle(const DevMesh& M, int t) { return (M.bad[t >> 5] >> (t & 31)) & 1u; }

// Assembly, near clip and setup of sub-triangle `sub` of triangle t (paintMesh
// + the first half of paintTriangle).  True: it has pixels to test.  n_sub:
// the triangle's sub-triangles (1 when the near plane does not cut it), -1
// when its indices failed the upload check.  The setup kernels take a
// triangle's second half in a round of its own, so only one Setup is live
// (two cost the vertex-pass instance a third of its registers; the round runs
// for warps with such a triangle only).
template <bool PRE>
__device__ __forceinline__ bool sub_setup(const View& V, const Geo& G, const DevRenderable& R, int t, int sub,
                                          Setup& S, int& n_sub, bool& cut) {
  // no_clip (paintTriangle(..., world=false)): never clipped, so the near
  // test compares against +inf
  const float zn = R.no_clip ? __int_as_float(0x7f800000) : V.znear;
  V2 p[3];
  float zt[3];
  Vtx v[3];
  int ip[3];
  if (PRE) {
    float4 a[3];
#pragma unroll
    for (int c = 0; c < 3; c++) ip[c] = (int)R.vert_base + __ldg(R.mesh.idx + 3 * t + c);
    if (bad_triangle(R.mesh, t)) {
      n_sub = -1;
      return false;
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      a[c] = G.va[(uint32_t)ip[c]];
      p[c] = v2(a[c].x, a[c].y);
      zt[c] = a[c].z;
    }
    cut = a[0].w > zn || a[1].w > zn || a[2].w > zn;
  } else {
    // (indices and index check in flight together; with the vertex pass the
    // three registers cost more than the latency)
#pragma unroll
    for (int c = 0; c < 3; c++) ip[c] = __ldg(R.mesh.idx + 3 * t + c);
    if (bad_triangle(R.mesh, t)) {
      n_sub = -1;
      return false;
    }
    corners<false>(R, t, ip, v);
    cut = v[0].pos.z > zn || v[1].pos.z > zn || v[2].pos.z > zn;
  }
  n_sub = 1;
  if (cut) {
    if (PRE) {
#pragma unroll
      for (int c = 0; c < 3; c++)
        v[c].pos = v3(G.vc[2 * (size_t)(uint32_t)ip[c]].w, G.vc[2 * (size_t)(uint32_t)ip[c] + 1].x,
                      G.va[(uint32_t)ip[c]].w);
    }
    n_sub = clip_pick<false>(zn, v, sub);
    if (n_sub <= sub) return false;
  }
  if (!PRE || cut) project3(V, v, p, zt);
  return setup_from(V, p, zt, S);
}

__device__ __forceinline__ long long box_pixels(const Setup& S) {
  return (long long)(S.x1 - S.x0 + 1) * (S.y1 - S.y0 + 1);
}

// The renderable (of lo..hi-1) of global triangle g; with the vertex pass also
// its vertices in the frame's buffers, both from the record the setup kernel
// left: one load where the search, the mesh's index pointer and the indices
// were a chain of eight.
template <bool PRE>
__device__ __forceinline__ uint32_t find_triangle(const Geo& G, int lo, int hi, uint32_t g, uint32_t (&gv)[3]) {
  if (PRE) {
    const uint4 q = G.tri[g];
    gv[0] = q.x;
    gv[1] = q.y;
    gv[2] = q.z;
    return q.w;
  }
  return (uint32_t)find_base(G.tri_base, lo, hi, g);
}

// A pixel's winning sub-triangle: its corners with the attributes its
// fragments read (the sub-triangle's own when the near plane cuts the
// triangle), their pixel coordinates and depth terms.
struct Winner {
  Vtx v[3];
  V2 p[3];
  float zt[3];
};

// The winner of a triangle that the near plane cuts: the sub-triangle's
// corners, projected.  Out of line: few pixels take it, and the batch kernel's
// warps, each in a phase of its own, wait for instructions as it is.
__device__ __noinline__ void cut_winner(const View& V, float zn, int sub, Winner& N) {
  clip_pick<true>(zn, N.v, sub);
#pragma unroll 1
  for (int c = 0; c < 3; c++) project(V, N.v[c].pos, N.p[c].x, N.p[c].y, N.zt[c]);
}
// Sub-triangle `id` of R (src/Renderer.cpp:334-379, 131-161); with the vertex
// pass, gv are the triangle's vertices in the frame's buffers.
template <bool PRE, bool CALL = false>
__device__ __forceinline__ void winner(const View& V, const Geo& G, const DevRenderable& R, uint32_t id,
                                       const uint32_t (&gv)[3], Winner& N) {
  const int t = (int)((id >> 1) - R.tri_base);
  const float zn = R.no_clip ? __int_as_float(0x7f800000) : V.znear;
  bool cut;
  if (PRE) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float4 a = G.va[gv[c]];
      N.p[c] = v2(a.x, a.y);
      N.zt[c] = a.z;
      N.v[c].pos = v3(0, 0, a.w);
      N.v[c].nrm = v3(0, 0, 0);
      N.v[c].uv = v2(0, 0);
    }
  } else if (R.mesh.rec) {
    corners_rec(R, t, N.v);
  } else {
    int ip[3];
#pragma unroll
    for (int c = 0; c < 3; c++) ip[c] = __ldg(R.mesh.idx + 3 * t + c);
    corners<true>(R, t, ip, N.v);
  }
  cut = N.v[0].pos.z > zn || N.v[1].pos.z > zn || N.v[2].pos.z > zn;
  if (PRE) vertex_attributes(G, R, t, gv, cut, N.v);
  if (CALL) {
    if (cut) {
      Winner T = N;
      cut_winner(V, zn, (int)(id & 1u), T);
      N = T;
    } else if (!PRE) {
      project3(V, N.v, N.p, N.zt);
    }
    return;
  }
  if (cut) clip_pick<true>(zn, N.v, (int)(id & 1u));  // that sub-triangle exists: it won this pixel
  if (!PRE || cut) project3(V, N.v, N.p, N.zt);
}

// loadPPM's texel decode b/255.0f (src/io.cpp:410), one division per byte
// value.  In global memory, where the L1 holds it: as a table in shared memory
// every block of the resolve paid for a division per thread and a barrier.
struct DecodeTable {
  float v[256];
  constexpr DecodeTable() : v() {
    for (int i = 0; i < 256; i++) v[i] = (float)i / 255.0f;
  }
};
static __device__ const DecodeTable kDecode;

// Texture and Blinn-Phong lighting of a fragment with perspective-corrected
// weights k0..k2 over the corners vc, src/Renderer.cpp:262-305 (FAST_LIGHT).
__device__ __forceinline__ void shade(const View& V, const DevRenderable& R, const Vtx (&vc)[3], float k0,
                                      float k1, float k2, V3& value, V3& normal_out) {
  V3 color = v3(R.diffuse[0], R.diffuse[1], R.diffuse[2]);
  if (R.has_tex) {
    V2 uv = add2(add2(ks2(k0, vc[0].uv), ks2(k1, vc[1].uv)), ks2(k2, vc[2].uv));
    int ti = (int)((uv.y - floorf(uv.y)) * (float)R.tex_rows);
    int tj = (int)((uv.x - floorf(uv.x)) * (float)R.tex_cols);
    ti = min(max(ti, 0), R.tex_rows - 1);
    tj = min(max(tj, 0), R.tex_cols - 1);
    size_t o = 3 * ((size_t)ti * R.tex_cols + tj);
    if (R.tex8)
      color = v3(__ldg(&kDecode.v[R.tex8[o]]), __ldg(&kDecode.v[R.tex8[o + 1]]), __ldg(&kDecode.v[R.tex8[o + 2]]));
    else
      color = v3(R.texf[o], R.texf[o + 1], R.texf[o + 2]);
  }
  value = v3(R.emissive[0], R.emissive[1], R.emissive[2]);
  if (R.lit) {
    V3 position = add3(add3(ks3(k0, vc[0].pos), ks3(k1, vc[1].pos)), ks3(k2, vc[2].pos));
    V3 LD = v3(V.lightdir[0], V.lightdir[1], V.lightdir[2]);
    V3 lightdir = R.point ? normalized3(sub3(LD, position)) : LD;
    V3 normal = add3(add3(ks3(k0, vc[0].nrm), ks3(k1, vc[1].nrm)), ks3(k2, vc[2].nrm));
    float sdiff = maxr(0.0f, dot3(normal, lightdir)) / len3(normal) + V.ambient;
    value = add3(value, ks3(sdiff, color));
    if (R.shininess != 0) {
      V3 viewDir = normalized3(position);
      V3 lv = sub3(lightdir, viewDir);
      float spec = powf(maxr(dot3(lv, normal), 0.0f) / (len3(lv) * len3(normal)), R.shininess);
      value = add3(value, ks3(spec, v3(R.specular[0], R.specular[1], R.specular[2])));
    }
    normal_out = normal;
  }
}

// The setup (src/Renderer.cpp:198-224) of the winning sub-triangle, the same
// values its raster used; of the bounding box only the column x0 that a
// replay starts from.
__device__ __forceinline__ void winner_setup(const View& V, const Winner& N, Setup& S) {
  setup_edges(N.p, N.zt, area2(N.p), S);
  S.x0 = pixel_of(least(N.p[0].x, N.p[1].x, N.p[2].x), V.w);
}

// The running edge values at pixel (x, y): row start, then column by column
// from the bounding-box edge (src/Renderer.cpp:240-243).
// Long replays, of triangles as wide as the frame, are bound by issue: LONG
// takes 16 sums a turn of the loop, advance2 takes 8 (20 such triangles at
// 16384x16384 resolve in 122.7 ms, 134.8 with 8, 116.8 with 32; but with 32 a
// warp whose pixels lie on either side of a multiple takes both ways: 20,000
// of 38x22 pixels at 1920x1080 57.2 us, 55.2 with 16 and with 8).  The batch
// kernel, whose warps wait for instructions as it is, does without (256 scenes
// 2208 us, 2218 with 32).
template <bool LONG>
__device__ __forceinline__ void replay(const Setup& S, int x, int y, float& e1, float& e2) {
  const unsigned long long d = pack2(S.n1.x, S.n2.x);
  unsigned long long e = row_start2(S, y);
  int n = x - S.x0;
  if (LONG) {
#pragma unroll 1
    for (; n >= 16; n -= 16) {
#pragma unroll
      for (int k = 0; k < 16; k++) e = add2(e, d);
    }
    if (n & 8) {
#pragma unroll
      for (int k = 0; k < 8; k++) e = add2(e, d);
    }
    n &= 7;
  }
  unpack2(advance2(e, d, n), e1, e2);
}

// savePPM conversion, src/io.cpp:358-362.
// (a NaN gives 0 here as there)
__device__ __forceinline__ uint32_t to_byte(float v) {
  return (uint32_t)__float2int_rz(fminf(fmaxf(v * 255.0f, 0.0f), 255.0f));
}

// ------------------------------------------------------------------ kernels
// Vertex i of R, at g in the frame's vertex buffers.
__device__ __forceinline__ void vertex(const Geo& G, const View& V, const DevRenderable& R, uint32_t g, int i) {
  const V3 v = affine(R.mv, ld3(R.mesh.pos, i));
  float px, py, zt;
  project(V, v, px, py, zt);
  G.va[g] = make_float4(px, py, zt, v.z);
  // a mesh of one index per corner for every attribute carries them all here
  V3 n = v3(0, 0, 0);
  V2 uv = v2(0, 0);
  if (R.unified) {
    if (i < R.mesh.n_nrm) n = affine(R.nm, ld3(R.mesh.nrm, i));
    if (i < R.mesh.n_uv) uv = ld2(R.mesh.uv, i);
  }
  G.vc[2 * (size_t)g] = make_float4(n.x, n.y, n.z, v.x);
  G.vc[2 * (size_t)g + 1] = make_float4(v.y, uv.x, uv.y, 0.f);
}
// Normal i of R, at g in the frame's normal buffer.
__device__ __forceinline__ void normal(const Geo& G, const DevRenderable& R, uint32_t g, int i) {
  const V3 n = affine(R.nm, ld3(R.mesh.nrm, i));
  G.vn[g] = make_float4(n.x, n.y, n.z, 0.f);
}

__device__ __forceinline__ void clear_words(unsigned long long* vis, size_t n, size_t i, size_t stride) {
  // two words per store (vis is 16-byte aligned)
  ulonglong2* v2 = reinterpret_cast<ulonglong2*>(vis);
  for (size_t k = i; k < n / 2; k += stride) v2[k] = make_ulonglong2(VIS_EMPTY, VIS_EMPTY);
  if (i == 0 && (n & 1)) vis[n - 1] = VIS_EMPTY;
}
// The first kernel of a frame: vis[0..n) = VIS_EMPTY (Renderer::clear), the
// counters zeroed, and one of
//   - the staging block of a frame of several renderables copied from mapped
//     pinned host memory, so a frame never queues behind other streams'
//     transfers on the copy engine;
//   - VERT: the vertex pass of a frame of one renderable, which comes in the
//     kernel's parameters (one launch less, and the stores of the clear fill
//     the vertex pass's load latency).
// Bound by the vertex pass's dependent loads and, in small frames, by the
// launch: 655,362 vertices and 1920x1080 words 17.6 us between events.
template <bool VERT>
__global__ void __launch_bounds__(256) k_begin(FrameParams F) {
  pdl_trigger();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  if (!VERT)
    for (size_t k = i; k < F.stage_n16; k += stride) F.stage_dst[k] = F.stage_src[k];
  uint32_t* cnt = reinterpret_cast<uint32_t*>(F.counters);
  for (size_t k = i; k < sizeof(Counters) / 4; k += stride) cnt[k] = 0;
  clear_words(F.vis, (size_t)F.v.W * F.v.H, i, stride);
  if (VERT) {
    for (size_t g = i; g < (size_t)F.g.n_verts + F.g.n_nrms; g += stride) {
      if (g < F.g.n_verts) vertex(F.g, F.v, F.one, (uint32_t)g, (int)g);
      else normal(F.g, F.one, (uint32_t)(g - F.g.n_verts), (int)(g - F.g.n_verts));
    }
  }
}

// Index check of a mesh upload (one bit per triangle), and for meshes with
// corner records the gather of each valid triangle's corner attributes.
__global__ void k_validate(DevMesh M, uint32_t* bad, float4* rec) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  bool b = false;
  int ip[3] = {0, 0, 0}, in[3] = {0, 0, 0}, it[3] = {0, 0, 0};
  if (t < M.n_tri) {
    for (int c = 0; c < 3; c++) {
      ip[c] = M.idx[3 * t + c];
      in[c] = M.nidx[3 * t + c];
      b |= ip[c] < 0 || ip[c] >= M.n_pos || in[c] < 0 || in[c] >= M.n_nrm;
      if (M.has_uv) {
        it[c] = M.tidx[3 * t + c];
        b |= it[c] < 0 || it[c] >= M.n_uv;
      }
    }
  }
  unsigned m = __ballot_sync(0xffffffffu, b);
  if ((threadIdx.x & 31) == 0 && (t >> 5) < ((M.n_tri + 31) >> 5)) bad[t >> 5] = m;
  if (rec && t < M.n_tri && !b) {
    // the layout of corners_rec
    float f[28];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      f[3 * c + 0] = M.pos[3 * ip[c] + 0];
      f[3 * c + 1] = M.pos[3 * ip[c] + 1];
      f[3 * c + 2] = M.pos[3 * ip[c] + 2];
    }
    const bool per_face = in[0] == in[1] && in[1] == in[2] && it[0] == it[1] && it[1] == it[2];
    float4* r = rec + (size_t)8 * t;
    if (per_face) {
      f[9] = M.nrm[3 * in[0] + 0];
      f[10] = M.nrm[3 * in[0] + 1];
      f[11] = M.nrm[3 * in[0] + 2];
      f[12] = M.has_uv ? M.uv[2 * it[0] + 0] : 0.f;
      f[13] = M.has_uv ? M.uv[2 * it[0] + 1] : 0.f;
      f[14] = 0.f;
      f[15] = __uint_as_float(kRecPerFace);
#pragma unroll
      for (int k = 0; k < 4; k++) r[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
    } else {
      const int nw[3] = {9, 12, 16}, uw[3] = {19, 21, 23};
#pragma unroll
      for (int c = 0; c < 3; c++) {
        f[nw[c] + 0] = M.nrm[3 * in[c] + 0];
        f[nw[c] + 1] = M.nrm[3 * in[c] + 1];
        f[nw[c] + 2] = M.nrm[3 * in[c] + 2];
        f[uw[c] + 0] = M.has_uv ? M.uv[2 * it[c] + 0] : 0.f;
        f[uw[c] + 1] = M.has_uv ? M.uv[2 * it[c] + 1] : 0.f;
      }
      f[15] = 0.f;
      f[25] = f[26] = f[27] = 0.f;
#pragma unroll
      for (int k = 0; k < 7; k++) r[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
    }
  }
}

// Vertex pass of several renderables: threads [0, n_verts) transform and
// project positions, threads [n_verts, n_verts + n_nrms) transform normals.
// BATCH: the view of a vertex is scenes[R.scene].v, else V.  Bound by the
// search for its renderable and by bytes; normals of meshes whose attributes
// share one index array go beside the positions (Geo::vc), so most threads of
// the second range have gone: 256 scenes of 64 primitives 254 -> 88 us.
template <bool BATCH>
__global__ void __launch_bounds__(256) k_vertex(Geo G, View V, const SceneRec* scenes) {
  pdl_wait();
  pdl_trigger();
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if ((g & ~31u) + 32 <= G.n_verts) {  // (a whole warp)
    const DevRenderable& R = G.rs[find_base_warp(G.vert_base, G.n_renderables, g)];
    if constexpr (BATCH) vertex(G, scenes[R.scene].v, R, g, (int)(g - R.vert_base));
    else vertex(G, V, R, g, (int)(g - R.vert_base));
  } else if (g < G.n_verts) {
    const DevRenderable& R = G.rs[find_base(G.vert_base, 0, G.n_renderables, g)];
    if constexpr (BATCH) vertex(G, scenes[R.scene].v, R, g, (int)(g - R.vert_base));
    else vertex(G, V, R, g, (int)(g - R.vert_base));
  } else if (g - G.n_verts < G.n_nrms) {
    const uint32_t gn = g - G.n_verts;
    const DevRenderable& R = G.rs[find_base(G.nrm_base, 0, G.n_renderables, gn)];
    normal(G, R, gn, (int)(gn - R.nrm_base));
  }
}

// Threads per block of the setup kernels.  Their warps share nothing
// (statistics go to slots, records are reserved by a warp at a time), and a
// block keeps its place until its slowest warp is done: 1080p mesh setup 38.6
// us with 64 threads, 40.6 with 128, 42.6 with 256; 10M-triangle soup 323, 325
// and 338; 256 scenes 334, 340 and 371.
constexpr int kSetupThreads = 64;

// Where small triangles' fragments go: the frame's visibility buffer...
struct FrameTarget {
  static constexpr bool one = true;  // (every tag is 0)
  unsigned long long* vis;
  int W;
  bool persp;
  // (a frame has at most 2^28 pixels)
  __device__ unsigned long long* row(uint32_t, int y) const { return vis + (uint32_t)y * (uint32_t)W; }
  __device__ bool perspective(uint32_t) const { return persp; }
};
// ...or, in a batch, the visibility buffer of the triangle's scene (tag).
struct BatchTarget {
  static constexpr bool one = false;
  const SceneRec* scenes;
  __device__ unsigned long long* row(uint32_t sc, int y) const {
    return scenes[sc].vis + (size_t)y * scenes[sc].v.W;
  }
  __device__ bool perspective(uint32_t sc) const { return scenes[sc].v.persp != 0; }
};

// Raster of a sub-triangle whose bounding box spans at most 4x4 pixels by
// one thread (src/Renderer.cpp:238-269); each row starts from its
// bounding-box edge and steps column by column.  row(y) gives the visibility
// words of row y.
// LIST: the covered cells first (bit 4 * row + column), then one covered pixel
// per turn of a loop, whose depth and atomic a warp issues as often as its
// fullest lane has pixels (5-6 for triangles of 1-4 square pixels) instead of
// once for each of the 16 cells that any lane covers: 5 % less of a
// 10M-triangle soup's setup, 8 % of 16 soups'.  The vertex-pass kernels take
// the plain walk: the list's registers are spilled there (1080p mesh 9 % more).
template <bool LIST, typename RowFn>
__device__ __forceinline__ void raster_tiny(const Setup& Q, bool persp, uint32_t id, RowFn row_of) {
  const unsigned long long d = pack2(Q.n1.x, Q.n2.x);
  unsigned cov = 0;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int y = Q.y0 + r;
    if (!LIST && y > Q.y1) break;
    unsigned long long e = row_start2(Q, y);
#pragma unroll
    for (int c = 0; c < 4; c++) {
      float e1, e2;
      unpack2(e, e1, e2);
      if (LIST) {
        if (covered(e1, e2)) cov |= 1u << (4 * r + c);
      } else if (Q.x0 + c <= Q.x1 && covered(e1, e2)) {
        float k0, k1, k2;
        const float z = frag_depth(Q, persp, e1, e2, k0, k1, k2);
        if (z < 1e11f) atomicMin(row_of(y) + Q.x0 + c, ((unsigned long long)depth_key(z) << 32) | id);
      }
      if (c < 3) e = add2(e, d);
    }
  }
  if (!LIST) return;
  cov &= (0x1111u * ((2u << (Q.x1 - Q.x0)) - 1u)) & ((1u << (4 * (Q.y1 - Q.y0 + 1))) - 1u);
  while (cov) {
    const int b = __ffs((int)cov) - 1, r = b >> 2, c = b & 3;
    cov &= cov - 1;
    const int y = Q.y0 + r;
    float e1, e2, k0, k1, k2;
    unsigned long long e = row_start2(Q, y);
    if (c > 0) e = add2(e, d);
    if (c > 1) e = add2(e, d);
    if (c > 2) e = add2(e, d);
    unpack2(e, e1, e2);
    const float z = frag_depth(Q, persp, e1, e2, k0, k1, k2);
    if (z < 1e11f) atomicMin(row_of(y) + Q.x0 + c, ((unsigned long long)depth_key(z) << 32) | id);
  }
}

// Raster of the warp's small sub-triangles (one per lane where `on`; ids step
// by two from lane to lane), whose frame is `tag`, with 64-bit atomicMin into
// the target (src/Renderer.cpp:238-269).  When every one in the warp spans at
// most 4x4 pixels the lanes rasterise their own (LIST: see raster_tiny);
// otherwise their rows are numbered by a prefix sum and taken one per lane,
// each lane fetching its row's setup from the lane that holds it.  (Staged in
// shared memory, the setups cost the vertex gathers 4 KB of L1 a block: 6 %
// more of the 1080p mesh's setup.)  Called by all lanes.
template <bool LIST, class Target>
__device__ __forceinline__ void raster_small(const Setup& S, bool on, uint32_t id, uint32_t tag, const Target& T) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, on);
  if (m == 0) return;
  const int span = on ? max(S.x1 - S.x0, S.y1 - S.y0) + 1 : 0;
  if (__reduce_max_sync(0xffffffffu, (unsigned)span) <= 4u) {
    if (on) raster_tiny<LIST>(S, T.perspective(tag), id, [&](int y) { return T.row(tag, y); });
    return;
  }
  const int rows = on ? S.y1 - S.y0 + 1 : 0;
  int inc = rows;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if ((int)lane >= o) inc += u;
  }
  const int total = __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll 1
  for (int b = 0; b < total; b += 32) {
    const int i = b + (int)lane;
    int own = 0;  // the lane whose record row i belongs to
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (__shfl_sync(0xffffffffu, inc, own + step - 1) <= i) own += step;
    const int k = i - __shfl_sync(0xffffffffu, inc - rows, own);
    Setup U;
    U.p0 = v2(__shfl_sync(0xffffffffu, S.p0.x, own), __shfl_sync(0xffffffffu, S.p0.y, own));
    U.p2 = v2(__shfl_sync(0xffffffffu, S.p2.x, own), __shfl_sync(0xffffffffu, S.p2.y, own));
    U.n1 = v2(__shfl_sync(0xffffffffu, S.n1.x, own), __shfl_sync(0xffffffffu, S.n1.y, own));
    U.n2 = v2(__shfl_sync(0xffffffffu, S.n2.x, own), __shfl_sync(0xffffffffu, S.n2.y, own));
#pragma unroll
    for (int c = 0; c < 3; c++) U.z[c] = __shfl_sync(0xffffffffu, S.z[c], own);
    // (frame coordinates fit 16 bits: sides <= 65536)
    const uint32_t at = __shfl_sync(0xffffffffu, (uint32_t)S.x0 | ((uint32_t)S.y0 << 16), own);
    U.x0 = (int)(at & 0xffffu);
    U.x1 = __shfl_sync(0xffffffffu, S.x1, own);
    const uint32_t tg = T.one ? 0u : __shfl_sync(0xffffffffu, tag, own);
    if (i < total) {
      const int y = (int)(at >> 16) + k;
      unsigned long long* row = T.row(tg, y);
      walk_row(U, T.perspective(tg), id + 2u * (uint32_t)(own - (int)lane), y, U.x1,
               [&](int x, unsigned long long v) { atomicMin(row + x, v); });
    }
  }
}

// Appends the warp's large sub-triangles (one per lane where `big`) to its
// share of the record store, and their blocks to its share of the block list.
// False in a lane whose record found no place (a fixed record store).
__device__ __forceinline__ bool append_large(const FrameParams& F, const Setup& S, bool big, uint32_t id) {
  const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  const unsigned m = __ballot_sync(0xffffffffu, big);
  if (m == 0) return true;
  unsigned base = 0;
  if (lane == 0) base = atomicAdd(&F.counters->share[warp_share()].rec_count, (unsigned)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  unsigned n_items = 0;
  const bool placed = base + __popc(m & lt) < F.rec_share;
  base += warp_share() * F.rec_share;
  if (big && placed) {
    F.recs[base + __popc(m & lt)] = to_rec(S, id);
    n_items = (unsigned)large_blocks(S.x0, S.y0, S.x1, S.y1);
  }
  // the blocks: one range per warp, each lane's at its exclusive prefix,
  // written by all lanes (a screen-sized triangle has hundreds)
  unsigned inc = n_items;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (unsigned)o) inc += u;
  }
  const unsigned total = __shfl_sync(0xffffffffu, inc, 31);
  if (total == 0) return placed || !big;
  unsigned long long ibase = 0;
  if (lane == 0) ibase = atomicAdd(&F.counters->share[warp_share()].item_count, (unsigned long long)total);
  ibase = __shfl_sync(0xffffffffu, ibase, 0);
  LargeItem* items = F.items + (size_t)warp_share() * F.item_share;
  for (unsigned b = 0; b < total; b += 32) {
    const unsigned i = b + lane;
    unsigned own = 0;  // the lane whose record block i belongs to
#pragma unroll
    for (unsigned step = 16; step; step >>= 1)
      if (__shfl_sync(0xffffffffu, inc, own + step - 1) <= i) own += step;
    const unsigned k = i - __shfl_sync(0xffffffffu, inc - n_items, own);
    if (i >= total) continue;
    const LargeItem item{base + __popc(m & ((1u << own) - 1u)), k};
    // blocks past the end of the list: the record's remaining ones go to the
    // spill list (one entry per record, so it cannot overflow)
    if (ibase + i < F.item_share) items[ibase + i] = item;
    else if (k == 0 || ibase + i == F.item_share) F.spill[atomicAdd(&F.counters->spill_count, 1u)] = item;
  }
  return placed || !big;
}

// Renderable k.  ONE: the frame's only renderable, which the kernels read
// from their parameters (constant bank) instead of through the staged table:
// no search, and no pointer to fetch before the first index can be read.
template <bool ONE>
__device__ __forceinline__ const DevRenderable& renderable(const FrameParams& F, uint32_t k) {
  if constexpr (ONE) return F.one;
  else return F.g.rs[k];
}

// Blocks of 256 threads per SM the register budget of the setup kernels must
// allow.  With the vertex pass the kernel waits on index -> vertex gathers
// and more resident warps hide that, until they spill: 5 (1080p mesh: 42.5
// us, 44.6 with 6).  Without it (triangle soups) it is bound by its strided
// position loads and by instruction issue, and spilling and a smaller share of
// the L1 cost more than the extra warps hide: 4 (64 registers).
template <bool PRE>
constexpr int kSetupMinBlocks = PRE ? 5 : 4;
template <bool PRE, bool ONE>
__global__ void __launch_bounds__(kSetupThreads, kSetupMinBlocks<PRE> * 256 / kSetupThreads) k_setup(FrameParams F) {
  pdl_wait();
  const unsigned lane = threadIdx.x & 31;
  const uint32_t g = (((blockIdx.x * blockDim.x + threadIdx.x) >> 5) << F.tri_shift) + lane;
  const bool in = lane < (1u << F.tri_shift) && g < F.g.n_tris;
  const uint32_t k = ONE ? 0u : (uint32_t)find_base_warp(F.g.tri_base, F.g.n_renderables, min(g, F.g.n_tris - 1));
  const DevRenderable& R = renderable<ONE>(F, k);
  const int t = (int)(g - R.tri_base);
  int n_sub = in ? 1 : 0;
#pragma unroll 1
  for (int sub = 0; sub < 2; sub++) {
    if (sub && !__any_sync(0xffffffffu, n_sub == 2)) break;
    Setup S;
    bool small = false, big = false, cut = false;
    if (n_sub > sub && sub_setup<PRE>(F.v, F.g, R, t, sub, S, n_sub, cut)) {
      small = box_pixels(S) <= (long long)F.small_max;
      big = !small;
    }
    if (PRE && !ONE && (small || big)) note_triangle(F.g, R, k, t);
    if (sub == 0 && n_sub < 0) atomicOr(&F.counters->error_flags, 1u);
    count_triangles(F.counters, small, big, sub == 0 && cut && n_sub > 0);
    const uint32_t id = 2u * g + (uint32_t)sub;
    if (!append_large(F, S, big, id)) small = true;  // rasterised here, as small ones are
    raster_small<!PRE>(S, small, id, 0u, FrameTarget{F.vis, F.v.W, F.v.persp != 0});
  }
}

// Large sub-triangles, one warp per block of kLargeRows rows by one column
// segment of a record's bounding box (src/Renderer.cpp:238-269): each lane
// finds its row's covered run in the segment, then the runs are walked a row
// per lane, or dealt in pieces where a few rows or ragged runs would leave
// lanes waiting.  Then the spill list: records with the blocks that
// did not fit the list.  An ordinary launch: with no large record every warp leaves at once.
// Bound by the serial walk of a row, which is why rows are cut into segments
// (large_segs): 64 primitives at 1280x720, 30.4 us with whole rows, 12 so.
__device__ __forceinline__ void raster_block(const FrameParams& F, bool persp, uint32_t rec, uint32_t k) {
  const BigRec& R = F.recs[rec];
  const Setup S = rec_setup(R);
  const uint32_t id = R.id;
  const int segs = large_segs(S.x0, S.x1), w = large_seg_cols(S.x0, S.x1);
  const int b = (int)k / segs, c = (int)k - b * segs;
  const int y = S.y0 + b * kLargeRows + (int)(threadIdx.x & 31);
  int xs = S.x0 + c * w, len = 0;
  unsigned long long e = 0;
  if (y <= S.y1) len = row_run(S, y, xs, min(xs + w - 1, S.x1), e);
  const uint32_t at = (uint32_t)y * (uint32_t)F.v.W + (uint32_t)xs;
  const auto put = [&](uint32_t p, unsigned long long v) { atomicMin(F.vis + p, v); };
  // A row per lane walks as many columns as the longest run has; 32 pieces take
  // about three columns' time and that of the sums from the run's start, some
  // 40 to a column's.  (Without these: 200 triangles as wide as a 65536x32
  // frame, whose segments are of 4096 columns, 20.7 ms, 6.2 so.)
  const unsigned longest = __reduce_max_sync(0xffffffffu, (unsigned)len);
  const unsigned pieces = __reduce_add_sync(0xffffffffu, (unsigned)(len + kPiece - 1) / kPiece);
  if ((pieces + 31) / 32 * (104 + max(longest, 16u)) < 40 * longest) {
    raster_runs(S, persp, id, e, len, at, put);
  } else {
    const unsigned long long d = pack2(S.n1.x, S.n2.x);
    for (int x = 0; x < len; x++) {
      float e1, e2;
      unpack2(e, e1, e2);
      if (covered(e1, e2)) {
        float k0, k1, k2;
        const float z = frag_depth(S, persp, e1, e2, k0, k1, k2);
        if (z < 1e11f) put(at + (uint32_t)x, ((unsigned long long)depth_key(z) << 32) | id);
      }
      e = add2(e, d);
    }
  }
}

__global__ void __launch_bounds__(256) k_raster_large(FrameParams F) {
  pdl_wait();
  pdl_trigger();
  // the shares' blocks in one numbering: lane l holds the end of share l's, and
  // a warp takes every nw-th block of all of them
  const int lane = (int)(threadIdx.x & 31);
  const uint32_t mine =
      lane < kShares ? (uint32_t)min(F.counters->share[lane].item_count, (unsigned long long)F.item_share) : 0u;
  uint32_t end = mine;
#pragma unroll
  for (int o = 1; o < kShares; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, end, o, kShares);
    if (lane % kShares >= o) end += u;
  }
  const uint32_t n = __shfl_sync(0xffffffffu, end, kShares - 1);
  const uint32_t n_spill = F.counters->spill_count;
  const bool persp = F.v.persp != 0;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  for (uint32_t it = w0; it < n; it += nw) {
    const int own = __popc(__ballot_sync(0xffffffffu, lane < kShares && end <= it));
    const uint32_t at = it - __shfl_sync(0xffffffffu, end - mine, own);
    const LargeItem item = F.items[(size_t)own * F.item_share + at];
    raster_block(F, persp, item.rec, item.k);
  }
  // The spill list: `per` warps on a record, so that two thirds of them have
  // work where there are few records (all of them at once have more atomics in
  // flight than L2 takes), each starting at a block of its own, so that many
  // records do not meet at their first pixels.  With one warp a record, all
  // from the first block on: 1000 frame-sized triangles' first frame 31.9 ms
  // at 3840x2160 (23.3 so), 7.9 ms at 1920x1080 in the fixed store (5.2).
  if (n_spill == 0) return;
  const uint32_t per = n_spill < nw ? max(1u, 2 * nw / (3 * n_spill)) : 1u, groups = nw / per;
  if (w0 >= groups * per) return;
  for (uint32_t it = w0 / per; it < n_spill; it += groups) {
    const LargeItem item = F.spill[it];
    const BigRec& R = F.recs[item.rec];
    const uint32_t left = (uint32_t)large_blocks(R.x0, R.y0, R.x1, R.y1) - item.k;
    const uint32_t first = __umulhi(it * 0x9E3779B1u, left);
    for (uint32_t j = w0 % per; j < left; j += per) {
      const uint32_t k = first + j;
      raster_block(F, persp, item.rec, item.k + (k < left ? k : k - left));
    }
  }
}

// Deferred resolve + shade: one thread per pixel, 128-thread blocks over
// 32x4-pixel tiles (a block keeps its registers until its slowest warp is
// done: 1080p mesh 36.8 us, 38.9 with 64 threads and with 256; 4K soup 219, 221
// and 227).  Bound by its chain of gathers -- word, triangle, corners, texel --
// where neighbouring pixels' triangles lie apart (1080p mesh of 1.31M
// triangles: 53 % of issue slots used, 36.8 us; 52 with attributes in six
// arrays and a search for the renderable), by instruction issue where corner
// records shorten it (10M-triangle soup: 72 %, 219 us; 282).  More blocks per
// SM spill.
constexpr int kResolveTileW = 32, kResolveTileH = 4, kResolveThreads = kResolveTileW * kResolveTileH;
template <bool PRE, bool ONE>
__global__ void __launch_bounds__(kResolveThreads, 1024 / kResolveThreads) k_resolve(FrameParams F) {
  pdl_wait();
  // 32x4-pixel block tiles, 16x2 per warp: neighbouring rows of a small
  // triangle are shaded by the same warp, so its corner data is fetched once
  const int tiles_x = (F.v.W + kResolveTileW - 1) / kResolveTileW;
  const int bx = blockIdx.x % tiles_x, by = blockIdx.x / tiles_x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int x = bx * kResolveTileW + (lane & 15) + 16 * (w & 1), y = by * kResolveTileH + (lane >> 4) + 2 * (w >> 1);
  if (x >= F.v.W || y >= F.v.H) return;
  const size_t px = (size_t)y * F.v.W + x;
  // the winner's setup is re-derived and its edge functions replayed to
  // column x, then texture and lighting (src/Renderer.cpp:247-305, FAST_LIGHT)
  const unsigned long long vw = F.vis[px];
  V3 value = v3(F.v.bg[0], F.v.bg[1], F.v.bg[2]), normal = v3(0, 0, 1);
  float depth = 1e11f;
  uint32_t id = MR_NO_TRIANGLE;
  if (vw != VIS_EMPTY) {
    id = (uint32_t)vw;
    uint32_t k = 0, gv[3] = {0, 0, 0};
    if constexpr (!ONE) k = find_triangle<PRE>(F.g, 0, F.g.n_renderables, id >> 1, gv);
    const DevRenderable& R = renderable<ONE>(F, k);
    if constexpr (ONE && PRE) {
#pragma unroll
      for (int c = 0; c < 3; c++) gv[c] = (uint32_t)__ldg(R.mesh.idx + 3 * (size_t)(id >> 1) + c);
    }
    Winner N;
    winner<PRE>(F.v, F.g, R, id, gv, N);
    Setup S;
    winner_setup(F.v, N, S);
    float e1, e2, k0, k1, k2;
    replay<true>(S, x, y, e1, e2);
    depth = frag_depth(S, F.v.persp != 0, e1, e2, k0, k1, k2);
    shade(F.v, R, N.v, k0, k1, k2, value, normal);
  }
  if (F.rgb8) {
    F.rgb8[3 * px + 0] = to_byte(value.x);
    F.rgb8[3 * px + 1] = to_byte(value.y);
    F.rgb8[3 * px + 2] = to_byte(value.z);
  }
  if (F.depth) F.depth[px] = depth;
  if (F.ids) F.ids[px] = id;
  if (F.rgbf) {
    F.rgbf[3 * px + 0] = value.x;
    F.rgbf[3 * px + 1] = value.y;
    F.rgbf[3 * px + 2] = value.z;
  }
  if (F.normals) {
    F.normals[3 * px + 0] = normal.x;
    F.normals[3 * px + 1] = normal.y;
    F.normals[3 * px + 2] = normal.z;
  }
}

// ---------------------------------------------------------------- batches
// put(tile, lane) for the tiles of the warp's records, one pair a lane: lane's
// record covers n tiles, nx to a row, from `first` (pitch: tiles per row of its
// scene).  With a record per lane, a triangle as large as its frame was one
// lane's chain of hundreds of atomics that the whole grid waited for: 24 scenes
// of 256x256 98 us of k_batch, 53 so where such triangles occur, 68 and 59 where
// hardly; 256 scenes 1811-2006 us, 1777-1820 so.  (In the setup's counts, whose
// atomics return nothing: 256 scenes 360 us, 340.)  Called by all lanes.
template <typename Put>
__device__ __forceinline__ void each_tile(uint32_t first, uint32_t pitch, uint32_t nx, PairNo n, Put put) {
  const int lane = (int)(threadIdx.x & 31);
  PairNo inc = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const PairNo u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  const PairNo total = __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll 1
  for (PairNo q = 0; q < total; q += 32) {
    const PairNo j = q + (PairNo)lane;
    int own = 0;  // the lane whose record pair j belongs to
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (__shfl_sync(0xffffffffu, inc, own + step - 1) <= j) own += step;
    const PairNo k = j - __shfl_sync(0xffffffffu, inc - n, own);
    const uint32_t cols = __shfl_sync(0xffffffffu, nx, own);
    const uint32_t row = k / cols;
    const uint32_t t = __shfl_sync(0xffffffffu, first, own) + row * __shfl_sync(0xffffffffu, pitch, own) + (k - row * cols);
    if (j < total) put(t, own);
  }
}

// Setup of every triangle of every scene: sub-triangles of at most small_max
// pixels of bounding box are rasterised into their scene's words, the others
// become records (warp-compacted), counted into their scene's tiles.  Bound by
// dependent loads (renderable, indices, vertices, view): 49 % of issue slots
// used; 256 scenes 334 us.
template <bool PRE>
__global__ void __launch_bounds__(kSetupThreads, kSetupMinBlocks<PRE> * 256 / kSetupThreads) k_setup_batch(BatchParams B) {
  const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  const uint32_t g = (((blockIdx.x * blockDim.x + threadIdx.x) >> 5) << B.tri_shift) + lane;
  uint32_t scene = 0;
  const bool in = lane < (1u << B.tri_shift) && g < B.g.n_tris;
  const uint32_t rk = (uint32_t)find_base_warp(B.g.tri_base, B.g.n_renderables, min(g, B.g.n_tris - 1));
  const DevRenderable* R = nullptr;
  if (in) {
    R = &B.g.rs[rk];
    scene = R->scene;
  }
  int n_sub = R ? 1 : 0;
#pragma unroll 1
  for (int sub = 0; sub < 2; sub++) {
    // (the second round, of triangles cut in two, is rare and a warp's own)
    if (sub && !__any_sync(0xffffffffu, n_sub == 2)) break;
    Setup S;
    bool small = false, big = false, cut = false;
    if (n_sub > sub && sub_setup<PRE>(B.scenes[scene].v, B.g, *R, (int)(g - R->tri_base), sub, S, n_sub, cut)) {
      small = box_pixels(S) <= (long long)B.small_max;
      big = !small;
    }
    if (PRE && (small || big)) note_triangle(B.g, *R, rk, (int)(g - R->tri_base));
    if (sub == 0 && n_sub < 0) atomicOr(&B.counters->error_flags, 1u);
    count_triangles(B.counters, small, big, sub == 0 && cut && n_sub > 0);
    // record slots, one reservation per warp in its share of the store
    const unsigned m = __ballot_sync(0xffffffffu, big);
    unsigned base = 0;
    if (lane == 0 && m) base = atomicAdd(&B.counters->share[warp_share()].rec_count, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    const uint32_t id = 2u * g + (uint32_t)sub;
    uint32_t first = 0, pitch = 0, nx = 1;
    PairNo n = 0;
    if (big) {
      const unsigned at = base + __popc(m & lt), slot = warp_share() * B.rec_share + at;
      if (at < B.rec_share) {
        B.recs[slot] = to_rec(S, id);
        B.rec_scene[slot] = scene;
        const SceneRec& SR = B.scenes[scene];
        const int tx0 = S.x0 / B.tile_w, ty0 = S.y0 / B.tile_h;
        nx = (uint32_t)(S.x1 / B.tile_w - tx0 + 1);
        n = nx * (PairNo)(S.y1 / B.tile_h - ty0 + 1);
        pitch = (uint32_t)SR.tiles_x;
        first = SR.tile_base + (uint32_t)ty0 * pitch + (uint32_t)tx0;
      }
    }
    if (m) each_tile(first, pitch, nx, n, [&](uint32_t t, int) { atomicAdd(B.tile_count + t, 1u); });
    if (B.small_max > 0) raster_small<!PRE>(S, small, id, scene, BatchTarget{B.scenes});
  }
}

constexpr int kStripMax = 256;
// Rows of a tile that one warp of k_batch takes at a time: the strip holds at
// most strip_px pixels (or one row).
__host__ __device__ inline int strip_rows(int tw, int th, int strip_px) {
  const int r = tw < strip_px ? strip_px / tw : 1;
  return th < r ? th : r;
}
// Words of shared memory between a strip's rows: rows of 16 pixels and more
// are skewed so the same column of several rows falls in different banks.
__host__ __device__ inline int strip_pitch(int tw) { return tw >= 16 ? tw + 4 : tw; }

// The records bins[s..e) of a tile, rasterised by one warp into its strip
// (px0..px1, py0..py1): 32 records at a time, the (record, row) pairs inside
// the strip enumerated by a prefix sum and taken one per lane.
// The fragments are merged into the strip's visibility words.
__device__ __forceinline__ void raster_strip(const BatchParams& B, uint32_t s, uint32_t e, int px0, int py0, int px1,
                                             int py1, bool persp, int pitch, unsigned long long* svis) {
  const int lane = (int)(threadIdx.x & 31);
#pragma unroll 1
  for (uint32_t c0 = s; c0 < e; c0 += 32) {
    uint32_t rec = 0;
    int rows = 0;
    if (c0 + lane < e) {
      rec = B.bins[c0 + lane];
      const int4 box = *reinterpret_cast<const int4*>(&B.recs[rec].x0);  // x0, y0, x1, y1
      if (max(box.x, px0) <= min(box.z, px1)) rows = max(0, min(box.w, py1) - max(box.y, py0) + 1);
    }
    int inc = rows;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    const int total = __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll 1
    for (int b = 0; b < total; b += 32) {
      const int i = b + lane;
      int own = 0;  // the lane whose record row i belongs to
#pragma unroll
      for (int step = 16; step; step >>= 1)
        if (__shfl_sync(0xffffffffu, inc, own + step - 1) <= i) own += step;
      const int k = i - __shfl_sync(0xffffffffu, inc - rows, own);
      const uint32_t r = __shfl_sync(0xffffffffu, rec, own);
      Setup S;
      uint32_t id = 0, at = 0;
      int len = 0;
      unsigned long long e = 0;
      S.n1 = S.n2 = v2(0, 0);
      S.z[0] = S.z[1] = S.z[2] = 0;
      if (i < total) {
        const BigRec& R = B.recs[r];
        S = rec_setup(R);
        id = R.id;
        const int y = max(S.y0, py0) + k;
        int xs = max(S.x0, px0);
        len = row_run(S, y, xs, min(S.x1, px1), e);
        at = (uint32_t)((y - py0) * pitch + xs - px0);
      }
      raster_runs(S, persp, id, e, len, at, [&](uint32_t c, unsigned long long v) { atomicMin(svis + c, v); });
    }
    __syncwarp();
  }
}

// The batch's persistent kernel (cooperative launch, grid-wide barriers):
//   1. a range of the list for each tile's records, 2. record indices
//   scattered into the ranges, 3. the tiles of all scenes, in strips of at
//   most 256 pixels, one warp each: the strip's visibility words start from
//   the scene's small-triangle words; its records are rasterised into shared
//   memory, then every pixel is resolved, shaded and written to its scene's
//   outputs.
// A strip is one warp's alone and each warp takes its own from a work counter,
// so no warp waits for another once the lists stand (with a block per tile the
// barriers between the phases were 38 % of the warps' time, with strips handed
// to a block in groups a fifth).  256 scenes 1826 us at 71 % of issue slots, 16
// soups 197, 24 scenes of 256x256 54.
// 64 registers: with 80, three blocks of 256 threads an SM, the 256 scenes take
// 2068 us and the soups 199.
template <bool PRE>
__global__ void __launch_bounds__(256, 4) k_batch(BatchParams B) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SceneRec s_scene[8];
  __shared__ unsigned long long s_at[8];
  cg::grid_group grid = cg::this_grid();
  const uint32_t nb = gridDim.x, nt = blockDim.x;
  const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
  const int TW = B.tile_w, TH = B.tile_h, SH = strip_rows(TW, TH, B.strip_px), pitch = strip_pitch(TW), lw = __ffs(TW) - 1;
  unsigned long long* svis = reinterpret_cast<unsigned long long*>(smem) + (size_t)w * SH * pitch;
  // 1. the tiles' ranges, in any order: one atomic per warp of tiles
  for (uint32_t t0 = (blockIdx.x * nt + threadIdx.x) & ~31u; t0 < B.n_tiles; t0 += nb * nt) {
    const uint32_t t = t0 + lane, v = t < B.n_tiles ? B.tile_count[t] : 0u;
    unsigned long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    unsigned long long base = 0;
    if (lane == 31 && inc) base = atomicAdd(&B.counters->bin_needed, inc);
    base = __shfl_sync(0xffffffffu, base, 31);
    // (a batch of 2^32 pairs and more is refused once it is read: its ranges
    // may overlap, but every entry below bin_cap is a record's index)
    if (t < B.n_tiles) B.tile_start[t] = (uint32_t)(base + inc - v);
  }
  grid.sync();
  // 2. scatter
  const uint32_t gw = (blockIdx.x * nt + threadIdx.x) >> 5, share = gw % kShares;
  const uint32_t nrec = min(B.counters->share[share].rec_count, B.rec_share);
  const uint32_t per = (nb * (nt >> 5) + kShares - 1 - share) / kShares;  // warps on this share
  for (uint32_t r0 = (gw / kShares) * 32; r0 < nrec; r0 += per * 32) {
    const uint32_t i = share * B.rec_share + r0 + lane;
    uint32_t first = 0, pitch_t = 0, nx = 1;  // the record's first tile, tiles per row of its scene, columns
    PairNo n = 0;                             // and number of its tiles
    if (r0 + lane < nrec) {
      const BigRec& R = B.recs[i];
      const SceneRec& SR = B.scenes[B.rec_scene[i]];
      const int tx0 = R.x0 / TW, ty0 = R.y0 / TH;
      nx = (uint32_t)(R.x1 / TW - tx0 + 1);
      n = nx * (PairNo)(R.y1 / TH - ty0 + 1);
      pitch_t = (uint32_t)SR.tiles_x;
      first = SR.tile_base + (uint32_t)ty0 * pitch_t + (uint32_t)tx0;
    }
    each_tile(first, pitch_t, nx, n, [&](uint32_t t, int own) {
      const uint32_t pos = B.tile_start[t] + atomicAdd(B.tile_fill + t, 1u);
      if (pos < B.bin_cap) B.bins[pos] = i - lane + own;
      else B.counters->bin_overflow = 1;
    });
  }
  grid.sync();
  // 3. strips.  A fetch is one strip, or as many as make half of strip_px where
  // tiles are smaller (the counter takes one atomic at a time: 64 scenes of
  // 512x512 in 4x16 tiles 2.5 % more with all of strip_px).  A warp's place is
  // kept in shared memory: in registers it spills what the shading needs (256
  // scenes 1.4 % more).
  const int ls2 = __ffs(TH / SH) - 1;  // strips per tile, a power of two
  const uint32_t run = max(1u, (uint32_t)B.strip_px / (uint32_t)(2 * TW * SH));  // strips per fetch, likewise
  if (lane == 0) s_at[w] = ~0ull;
  for (;;) {
    __syncwarp();  // the last strip's words and scene may be overwritten
    unsigned long long u = s_at[w] + 1;
    if (!(u & (run - 1))) {
      uint32_t f = 0;
      if (lane == 0) f = atomicAdd(&B.counters->work_next, 1u);
      u = (unsigned long long)__shfl_sync(0xffffffffu, f, 0) * run;
    }
    __syncwarp();
    if (lane == 0) s_at[w] = u;
    const uint32_t t = (uint32_t)(u >> ls2), strip = (uint32_t)u & ((1u << ls2) - 1u);
    if (t >= B.n_tiles) break;
    // the scene: the last j with scene_tile_base[j] <= t (bases ascending,
    // the first 0), 32 candidates at a time
    int sc = 0;
    for (int n = B.n_scenes; n > 1;) {
      const int step = (n + 31) >> 5, j = sc + lane * step;
      const unsigned m = __ballot_sync(0xffffffffu, lane * step < n && B.scene_tile_base[j] <= t);
      const int at = (31 - __clz((int)m)) * step;
      sc += at;
      n = min(step, n - at);
    }
    __syncwarp();
    {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(&B.scenes[sc]);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&s_scene[w]);
      for (int i = lane; i < (int)(sizeof(SceneRec) / 4); i += 32) dst[i] = src[i];
    }
    __syncwarp();
    const SceneRec& C = s_scene[w];
    const int lt = (int)(t - C.tile_base), ty = lt / C.tiles_x, tx = lt - ty * C.tiles_x;
    const int px0 = tx * TW, py0 = ty * TH + (int)strip * SH;
    const int px1 = min(px0 + TW, C.v.W) - 1, py1 = min(py0 + SH, C.v.H) - 1;
    if (py0 > py1) continue;
    const bool persp = C.v.persp != 0;
    // the tile's list (truncated at capacity on overflow)
    const uint32_t ls = min(B.tile_start[t], B.bin_cap), le = min(B.tile_start[t] + B.tile_count[t], B.bin_cap);
    // the strip starts from the small triangles' words (or empty): two
    // words a load, all of a lane's in flight at once; what is not empty is
    // left empty for the next batch
    bool drawn = false;
    {
      const bool pairs = ((C.v.W & 1) | (int)((uintptr_t)C.vis >> 3 & 1)) == 0 && px1 - px0 + 1 == TW;
      ulonglong2 v[kStripMax / 64];
#pragma unroll
      for (int j = 0; j < kStripMax / 64; j++) {
        const int i = 64 * j + 2 * lane, cy = i >> lw, x = px0 + (i & (TW - 1)), y = py0 + cy;
        v[j] = make_ulonglong2(VIS_EMPTY, VIS_EMPTY);
        if (C.vis && i < SH * TW && y <= py1) {
          unsigned long long* q = C.vis + ((uint32_t)y * (uint32_t)C.v.W + (uint32_t)x);
          if (pairs) {
            v[j] = *reinterpret_cast<const ulonglong2*>(q);
          } else {
            if (x <= px1) v[j].x = q[0];
            if (x + 1 <= px1) v[j].y = q[1];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kStripMax / 64; j++) {
        const int i = 64 * j + 2 * lane, cy = i >> lw, cx = i & (TW - 1);
        if (i >= SH * TW) break;
        if ((v[j].x & v[j].y) != VIS_EMPTY) {
          drawn = true;
          unsigned long long* q = C.vis + ((uint32_t)(py0 + cy) * (uint32_t)C.v.W + (uint32_t)(px0 + cx));
          if (v[j].x != VIS_EMPTY) q[0] = VIS_EMPTY;
          if (v[j].y != VIS_EMPTY) q[1] = VIS_EMPTY;
        }
        *reinterpret_cast<ulonglong2*>(svis + cy * pitch + cx) = v[j];
      }
    }
    __syncwarp();
    if (ls < le) raster_strip(B, ls, le, px0, py0, px1, py1, persp, pitch, svis);
    // nothing drawn: the background, four pixels a lane where whole groups
    // of four lie aligned in every output
    if (ls >= le && !__any_sync(0xffffffffu, drawn) && px1 - px0 + 1 == TW && (C.v.W & 3) == 0 &&
        (((uintptr_t)C.depth | (uintptr_t)C.ids) & 15) == 0 && ((uintptr_t)C.rgb8 & 3) == 0) {
      const uint32_t c = to_byte(C.v.bg[0]) | ((uint32_t)to_byte(C.v.bg[1]) << 8) | ((uint32_t)to_byte(C.v.bg[2]) << 16);
      for (int i = 4 * lane; i < SH * TW; i += 128) {
        const int y = py0 + (i >> lw);
        if (y > py1) break;
        const uint32_t px = (uint32_t)y * (uint32_t)C.v.W + (uint32_t)(px0 + (i & (TW - 1)));
        if (C.rgb8) {
          uint32_t* o = reinterpret_cast<uint32_t*>(C.rgb8 + 3 * (size_t)px);
          o[0] = c | (c << 24);
          o[1] = (c >> 8) | (c << 16);
          o[2] = (c >> 16) | (c << 8);
        }
        if (C.depth) *reinterpret_cast<float4*>(C.depth + px) = make_float4(1e11f, 1e11f, 1e11f, 1e11f);
        if (C.ids) *reinterpret_cast<uint4*>(C.ids + px) = make_uint4(MR_NO_TRIANGLE, MR_NO_TRIANGLE, MR_NO_TRIANGLE, MR_NO_TRIANGLE);
      }
      continue;
    }
    const uint32_t id0 = 2u * B.g.tri_base[C.rs_begin];  // ids are reported per scene
#pragma unroll 1
    for (int i = lane; i < SH * TW; i += 32) {
      const int cy = i >> lw, cx = i & (TW - 1), x = px0 + cx, y = py0 + cy;
      if (x > px1 || y > py1) continue;
      const uint32_t px = (uint32_t)y * (uint32_t)C.v.W + (uint32_t)x;
      const unsigned long long vw = svis[cy * pitch + cx];
      V3 value, normal;
      float depth;
      const uint32_t id = (uint32_t)vw;
      if (vw == VIS_EMPTY) {
        value = v3(C.v.bg[0], C.v.bg[1], C.v.bg[2]);
        depth = 1e11f;
      } else {
        uint32_t gv[3];
        const DevRenderable& R = B.g.rs[find_triangle<PRE>(B.g, (int)C.rs_begin, (int)C.rs_end, id >> 1, gv)];
        Winner N;
        winner<PRE, PRE>(C.v, B.g, R, id, gv, N);
        Setup S;
        winner_setup(C.v, N, S);
        float e1, e2;
        replay<false>(S, x, y, e1, e2);
        float k0, k1, k2;
        depth = frag_depth(S, persp, e1, e2, k0, k1, k2);
        shade(C.v, R, N.v, k0, k1, k2, value, normal);
      }
      if (C.rgb8) {
        uint8_t* o8 = C.rgb8 + 3 * (size_t)px;
        o8[0] = to_byte(value.x);
        o8[1] = to_byte(value.y);
        o8[2] = to_byte(value.z);
      }
      if (C.depth) C.depth[px] = depth;
      if (C.ids) C.ids[px] = vw == VIS_EMPTY ? MR_NO_TRIANGLE : id - id0;
    }
  }
}

__global__ void k_range(int W, int H, Mat4 M, const float* depth, float* xyz) {
  const float* P = M.m;
  size_t px = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (px >= (size_t)W * H) return;
  int i = (int)(px / W), j = (int)(px - (size_t)i * W);
  bool persp = P[15] == 0;
  float zfar = persp ? P[11] / (P[10] + 1) : (P[11] - 1) / P[10];
  float fardepth = persp ? zfar : 1.0f;
  float w = (float)W, h = (float)H;
  float d = depth[px];
  float* o = xyz + 3 * px;
  if (d > fardepth) {
    o[0] = 0; o[1] = 0; o[2] = 0;
  } else {
    float u = (j + 0.5f) / (w / 2) - 1;
    float v = -(i + 0.5f) / (h / 2) + 1;
    float z = -d;
    o[0] = -(u + P[2]) * z / P[0];
    o[1] = -(v + P[6]) * z / P[5];
    o[2] = z;
  }
}

// ------------------------------------------------------------ host launchers
static int grid_for(size_t n, int block) { return (int)((n + block - 1) / block); }

static int sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
  }
  return sms;
}

cudaError_t launch_validate(const DevMesh& M, uint32_t* bad, cudaStream_t st) {
  if (M.n_tri <= 0) return cudaSuccess;
  k_validate<<<grid_for((size_t)M.n_tri, 256), 256, 0, st>>>(M, bad, const_cast<float4*>(M.rec));
  return cudaGetLastError();
}

// Ordinary launch allowed to overlap its predecessor's tail (the kernel calls
// pdl_wait() before touching anything the predecessor writes).
template <typename... Exp, typename... Act>
static cudaError_t launch_after(void (*k)(Exp...), int grid, int block, cudaStream_t st, Act&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, std::forward<Act>(args)...);
}

static cudaError_t launch_coop(const void* fn, int grid, int block, void** args, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// Triangles a warp of the setup kernels takes, as a power of two: all 32 lanes
// hold one when that gives every SM 16 warps, fewer in small frames, whose
// time is that of one warp's triangles one row batch after another (UV sphere
// of 3968 triangles 16.4 -> 10.3 us, 64 primitives 17.0 -> 13.9; with 32 warps
// per SM a 20000-triangle soup is slower again, 9.3 -> 11.3).
static int triangle_shift(size_t n_tris) {
  int s = 5;
  while (s > 1 && (n_tris >> s) < (size_t)sm_count() * 16) s--;
  return s;
}

// Launch sequence of one frame.  With F.g.va set, the vertex pass runs first
// and the setup/resolve kernels read its buffers.  staged (frames of several
// renderables) is recorded once the staging block has been read.  ev
// (optional, 6 events) brackets the stages: clear+vertex, setup,
// large-triangle raster, -, resolve.
template <bool PRE, bool ONE>
static cudaError_t launch_stages(const FrameParams& F, cudaStream_t st, cudaEvent_t* ev, cudaEvent_t staged) {
  const size_t npx = (size_t)F.v.W * F.v.H;
  const size_t n_verts = PRE ? (size_t)F.g.n_verts + F.g.n_nrms : 0;
  if (ev) cudaEventRecord(ev[0], st);
  // The clear also brings vis[] into L2 (write-allocate), so the setup
  // kernel's atomics hit L2.
  const int cgrid = std::min(grid_for((npx + 1) / 2, 256), sm_count() * 16);
  cudaError_t le = cudaSuccess;
  if (PRE && ONE) {
    k_begin<true><<<std::max(cgrid, grid_for(n_verts, 256)), 256, 0, st>>>(F);
  } else {
    k_begin<false><<<cgrid, 256, 0, st>>>(F);
    if (staged && !ONE) cudaEventRecord(staged, st);
    // vertex pass, setup and resolve may be scheduled while their predecessor
    // finishes (they wait for it before reading its output)
    if (n_verts) le = launch_after(k_vertex<false>, grid_for(n_verts, 256), 256, st, F.g, F.v, (const SceneRec*)nullptr);
    if (le != cudaSuccess) return le;
  }
  if (ev) cudaEventRecord(ev[1], st);
  if (F.g.n_tris) {
    FrameParams Fs = F;
    Fs.tri_shift = triangle_shift(F.g.n_tris);
    le = launch_after(k_setup<PRE, ONE>, grid_for((size_t)F.g.n_tris << (5 - Fs.tri_shift), kSetupThreads),
                      kSetupThreads, st, Fs);
    if (le != cudaSuccess) return le;
  }
  if (ev) cudaEventRecord(ev[2], st);
  le = launch_after(k_raster_large, sm_count() * 8, 256, st, F);
  if (le != cudaSuccess) return le;
  if (ev) cudaEventRecord(ev[3], st);
  if (ev) cudaEventRecord(ev[4], st);
  const int rgrid = ((F.v.W + kResolveTileW - 1) / kResolveTileW) * ((F.v.H + kResolveTileH - 1) / kResolveTileH);
  le = launch_after(k_resolve<PRE, ONE>, rgrid, kResolveThreads, st, F);
  if (le != cudaSuccess) return le;
  if (ev) cudaEventRecord(ev[5], st);
  return cudaGetLastError();
}

cudaError_t launch_frame(const FrameParams& F, cudaStream_t st, cudaEvent_t* ev, cudaEvent_t staged) {
  const bool pre = F.g.va != nullptr;
  if (F.g.n_renderables == 1)
    return pre ? launch_stages<true, true>(F, st, ev, staged) : launch_stages<false, true>(F, st, ev, staged);
  return pre ? launch_stages<true, false>(F, st, ev, staged) : launch_stages<false, false>(F, st, ev, staged);
}

size_t batch_smem(int tile_w, int tile_h, int threads) {
  // visibility words of one strip per warp
  return (size_t)(threads / 32) * strip_rows(tile_w, tile_h, kStripMax) * strip_pitch(tile_w) * sizeof(unsigned long long);
}
static const void* batch_kernel(bool pre) { return pre ? (const void*)k_batch<true> : (const void*)k_batch<false>; }
// Co-resident blocks of k_batch for the given shape (its cooperative grid).
int batch_grid(int tile_w, int tile_h, int threads, bool pre) {
  int per = 0;
  size_t smem = batch_smem(tile_w, tile_h, threads);
  const void* k = batch_kernel(pre);
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, threads, smem);
  if (per <= 0) return 0;
  return sm_count() * per;
}
cudaError_t launch_batch(const BatchParams& B, int threads, int grid, cudaStream_t st, cudaEvent_t* ev) {
  const bool pre = B.g.va != nullptr;  // null: kernels transform corners themselves
  if (ev) cudaEventRecord(ev[0], st);
  if (pre && B.g.n_verts + B.g.n_nrms > 0) {
    View none = {};
    k_vertex<true><<<grid_for((size_t)B.g.n_verts + B.g.n_nrms, 256), 256, 0, st>>>(B.g, none, B.scenes);
  }
  if (ev) cudaEventRecord(ev[1], st);
  if (B.g.n_tris) {
    BatchParams Bs = B;
    Bs.tri_shift = triangle_shift(B.g.n_tris);
    const int sgrid = grid_for((size_t)B.g.n_tris << (5 - Bs.tri_shift), kSetupThreads);
    if (pre) k_setup_batch<true><<<sgrid, kSetupThreads, 0, st>>>(Bs);
    else k_setup_batch<false><<<sgrid, kSetupThreads, 0, st>>>(Bs);
  }
  if (ev) cudaEventRecord(ev[2], st);
  // strips of 256 pixels, cut to 128 or 64 where that would leave a warp fewer
  // than 6 of them and to 32 where 64 leaves fewer than 2 (a dense strip would
  // be the batch's tail: two 137x96 scenes 67 us with 256, 30 with 32; 24
  // scenes of 256x256 92 with 256, 84 with 64, 89 with 32); smaller ones read a
  // tile's records and vertices more often (16 soups 242 us, 262 with half)
  BatchParams Bc = B;
  Bc.strip_px = kStripMax;
  const unsigned long long px = (unsigned long long)B.n_tiles * B.tile_w * B.tile_h, warps = (unsigned long long)grid * threads / 32;
  while (Bc.strip_px > 64 && px < 6 * warps * Bc.strip_px) Bc.strip_px /= 2;
  if (px < 2 * warps * 64) Bc.strip_px = 32;
  void* args[] = {&Bc};
  cudaError_t e = launch_coop(batch_kernel(pre), grid, threads, args,
                              batch_smem(B.tile_w, B.tile_h, threads), st);
  if (ev) cudaEventRecord(ev[3], st);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t launch_range(int W, int H, const Mat4& P, const float* depth, float* xyz, cudaStream_t st) {
  size_t npx = (size_t)W * H;
  k_range<<<grid_for(npx, 256), 256, 0, st>>>(W, H, P, depth, xyz);
  return cudaGetLastError();
}

}  // namespace mrg
