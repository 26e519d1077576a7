// Data layout shared by the host side of the C ABI and the kernels: one
// resident mesh, one renderable, the view of one frame, the setup record of a
// rasterised sub-triangle, per-frame counters and the kernel parameter
// blocks.  Plain C++ (no device code), so host translation units can include it.
#pragma once
#include <stdint.h>
#include <vector_types.h>

#include <limits>

#include "../../include/minirender_gpu.h"

namespace mrg {

// Packed visibility word: (order-preserving depth key << 32) | sub-triangle
// id.  A pixel nobody wrote keeps VIS_EMPTY, which is larger than any real
// fragment because real fragments need z < 1e11f (the clear value of the
// reference z-buffer, src/Renderer.cpp:116) and id < 0xFFFFFFFF.
static constexpr unsigned long long VIS_EMPTY = ~0ull;

// Limits of a frame's sides and of a batch's tiles.
constexpr int kMaxSide = 1 << 16;
constexpr int kMinTilePx = 64;

// Number of a (record, tile) pair among those of a warp's 32 records.  A
// record as large as the largest scene lies in 2^26 of the smallest tiles:
// 2^31 pairs, one more than an int holds.
using PairNo = uint32_t;
static_assert(32ull * ((unsigned long long)kMaxSide * kMaxSide / kMinTilePx) <= std::numeric_limits<PairNo>::max(),
              "a warp's (record, tile) pairs need a wider PairNo");

// One resident mesh (TriMesh arrays, include/minirender/Scene.h:73-87).
struct DevMesh {
  const float* pos;   // n_pos x 3
  const float* nrm;   // n_nrm x 3
  const float* uv;    // n_uv x 2
  const int32_t* idx;   // 3 per triangle
  const int32_t* nidx;
  const int32_t* tidx;
  const uint32_t* bad;   // bit t set: triangle t has an index out of range
  // Soup-like meshes (3 * n_tri < 2 * n_pos): triangle t's corner positions,
  // normals and texcoords gathered at upload into rec[8t .. 8t+7] (128 B per
  // triangle; the first 64 B hold all of a triangle whose three corners share
  // one normal and one texcoord), so a pixel's winner is read from one record
  // instead of six scattered arrays.  Null otherwise.
  const float4* rec;
  int32_t n_pos, n_nrm, n_uv, n_tri;
  int32_t has_uv;       // texcoords and texcoordsI both non-empty
};

// Meshes that get corner records: those whose vertices are not shared
// (the per-vertex pass would not pay for them alone).
inline bool mesh_wants_records(long long n_tri, long long n_pos) { return n_tri > 0 && 3 * n_tri < 2 * n_pos; }
constexpr size_t kRecBytes = 128;

// One renderable: mesh, matrices and material.
struct DevRenderable {
  float mv[12];         // rows 0..2 of view * transform (src/Renderer.cpp:337)
  float nm[12];         // rows 0..2 of inverse(mv)^T (src/Renderer.cpp:338)
  DevMesh mesh;
  uint32_t tri_base;    // global index of the first triangle
  uint32_t vert_base;   // global index of the first vertex in the per-frame vertex buffers
  uint32_t nrm_base;    // global index of the first normal
  uint32_t scene;       // frame (scene) this renderable belongs to (batches)
  int32_t has_tex;      // texturing on and the material has a texture
  int32_t no_clip;      // MR_RS_NO_CLIP: no near-plane clipping
  int32_t lit;          // lighting on for its fragments (the frame's or its paint call's)
  int32_t point;        // point light for its fragments (the frame's or its paint call's)
  int32_t unified;      // one index per corner for every attribute: see Geo::vc
  int32_t need;         // corner attributes its fragments read (kNeed*)
  float diffuse[3], specular[3], emissive[3], shininess;
  const uint8_t* tex8;  // rows x cols x 3 bytes (decoded b/255), or
  const float* texf;    // rows x cols x 3 floats
  int32_t tex_rows, tex_cols;
};

constexpr int kNeedNormal = 1, kNeedTexcoord = 2, kNeedPosition = 4;

// Renderer state of one frame that the kernels read (src/Renderer.cpp:311-326).
struct View {
  int W, H;
  float w, h;
  float P[16];
  int persp;
  int simple;         // P is a perspective matrix with only the entries [0][0], [0][2], [1][1], [1][2]
                      // and the z row, and w = -z: see project3
  float znear;
  float lightdir[3];  // placed as render() places it (src/Renderer.cpp:317-320)
  float ambient;
  float bg[3];
};

struct Mat4 {
  float m[16];
};

// Geometry of a launch: renderable table, base tables and the per-vertex
// buffers of the vertex pass (va null: kernels transform per triangle).
struct Geo {
  const DevRenderable* rs;
  const uint32_t* tri_base;   // n_renderables + 1 prefix of triangle counts
  const uint32_t* vert_base;  // n_renderables + 1 prefix of vertex counts
  const uint32_t* nrm_base;   // n_renderables + 1 prefix of normal counts
  int n_renderables;
  uint32_t n_tris, n_verts, n_nrms;
  float4* va;                 // (pixel x, pixel y, z term, view z) per vertex
  float4* vc;                 // two per vertex: (view-space normal, view x), (view y, texcoord, 0);
                              // normal and texcoord of unified renderables only
  float4* vn;                 // view-space normal per normal (renderables that are not unified)
  uint4* tri;                 // frames of several renderables with the vertex pass: (vertices, renderable)
                              // per triangle, left by the setup kernel for the resolve
};

// Setup record of a rasterised sub-triangle (64 bytes).
struct __align__(16) BigRec {
  float p0x, p0y, p2x, p2y;   // pixel-space corners 0 and 2
  float n1x, n1y, n2x, n2y;   // edge-function gradients
  float z0, z1, z2;           // iz[] (perspective) or zz[] (orthographic)
  uint32_t id;                // 2 * global triangle + clip sub-triangle
  int32_t x0, y0, x1, y1;     // inclusive clamped pixel bounding box
};

// Triangle statistics, one slot per group of warps (a single counter updated
// by every warp would serialise in L2), each on a sector of its own.
constexpr int kStatSlots = 64;
struct alignas(32) StatSlot {
  unsigned long long drawn;    // rasterised sub-triangles << 32 | of these, in the setup kernel
  unsigned long long clipped;  // triangles cut by the near plane
};

constexpr int kShares = 16;
// The share of the record store and of the block list that setup warp w uses:
// one warp of each sixteen in a row to a share, in an order that differs from
// sixteen to sixteen, so that large triangles that recur every so many warps
// do not all meet in one.  (400,000 triangles at 1080p, the 32 of every
// sixteenth warp large, in the fixed store of the allocation-free entry: 388
// us with w % 16, where five of six found their share full, 215 so.)
#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t share_of_warp(uint32_t w) {
  uint32_t h = (w / kShares) * 0x9E3779B1u;  // (two odd multipliers; any that mix would do)
  h = (h ^ (h >> 15)) * 0x2C1B3C6Du;
  return (w ^ (h >> 28)) % kShares;
}

// Counters of one share of the record store and of the block list.  Every warp
// of the setup waits for these, so they are spread, too: on one address an
// update takes some 2 ns, 10 us of the setup of 327,680 triangles of 18
// pixels.  (64 shares cost the large raster 2 us to add up, 16 cost none.)
struct alignas(32) ShareSlot {
  unsigned long long item_count;  // large-triangle blocks requested (single frames; 64 bits: a frame
                                  // of many screen-sized triangles passes 2^32)
  unsigned int rec_count;         // records requested
};

struct Counters {
  StatSlot stat[kStatSlots];
  ShareSlot share[kShares];
  unsigned long long bin_needed;  // total (tile, record) pairs requested
  unsigned int error_flags;
  unsigned int bin_overflow;
  unsigned int work_next;      // persistent-kernel work counter
  unsigned int spill_count;    // records whose remaining blocks did not fit the block list
};

// One-frame launch.
// Block `k` of the bounding box of large sub-triangle `rec`: kLargeRows rows
// by one column segment, blocks numbered along the rows first; in the spill
// list, every block from `k` to the record's last.
struct LargeItem {
  uint32_t rec, k;
};
constexpr int kLargeRows = 32;
// Columns per segment: 16 columns up to a width of 256, then a 16th of the
// width (in whole 16s).  A segment starts with the replay of the columns left
// of it (one add per column); at most 16 segments keep those adds below a
// sixth of the walk's work.  (64 primitives at 1280x720: 20 us with 64
// columns, 14 with 32, 12 with 16.)
constexpr int kLargeCols = 16, kLargeSegs = 16;

// Records per share in which T triangles always find room: a share's warps hold
// at most T / kShares + 64 of them (of each sixteen setup warps, 2 to 32
// triangles each, one), two sub-triangles each.
inline size_t rec_share_for(size_t T) { return T / (kShares / 2) + 128; }

struct FrameParams {
  View v;
  Geo g;
  DevRenderable one;          // the renderable of a frame that has one (no table is staged for it)
  int small_max;
  int tri_shift;              // log2 of the triangles a warp of the setup kernel takes
  unsigned long long* vis;    // W*H
  BigRec* recs;               // large sub-triangles
  uint32_t rec_share;         // of these, records per share
  LargeItem* items;           // their blocks
  uint32_t item_share;        // of these, blocks per share
  LargeItem* spill;           // an entry per record: records whose blocks did not fit items[]
  const uint4* stage_src;     // the frame's staging block in mapped pinned host memory (several
  uint4* stage_dst;           // renderables), fetched by the clear kernel (no copy-engine transfer)
  uint32_t stage_n16;         // its size in 16-byte units
  uint8_t* rgb8;
  float* depth;
  float* rgbf;
  uint32_t* ids;
  float* normals;
  Counters* counters;
};

// One scene of a batch: its view, tiles and output buffers.
struct SceneRec {
  View v;
  int tiles_x, tiles_y;
  uint32_t tile_base;         // first tile in the batch-wide tile index space
  uint32_t rs_begin, rs_end;  // renderables of this scene
  uint8_t* rgb8;
  float* depth;
  uint32_t* ids;
  unsigned long long* vis;    // visibility words of the small triangles (null: all binned)
};

// Batched launch: many scenes, one persistent fused bin-raster-shade kernel.
struct BatchParams {
  Geo g;
  const SceneRec* scenes;
  const uint32_t* scene_tile_base;  // n_scenes + 1 prefix of tile counts
  int n_scenes;
  uint32_t n_tiles;
  int tile_w, tile_h;               // tile width and height (pixels)
  int strip_px;                     // pixels of a tile that a warp takes at a time
  int tri_shift;                    // log2 of the triangles a warp of the setup kernel takes
  int small_max;                    // bbox pixels up to which the setup kernel rasterises (0: none)
  unsigned long long* vis;          // all scenes' visibility words (small_max > 0)
  BigRec* recs;
  uint32_t rec_share;               // of these, records per share
  uint32_t* rec_scene;              // scene of each record
  uint32_t* tile_count;             // n_tiles
  uint32_t* tile_start;             // n_tiles + 1
  uint32_t* tile_fill;              // n_tiles
  uint32_t* bins;
  uint32_t bin_cap;
  Counters* counters;
};

}  // namespace mrg
