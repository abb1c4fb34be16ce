// hsr_internal.h — data layout shared by the host runtime and the sm_103a kernels.
//
// Pipeline of one launch sequence (a batch of views = draws):
//   k_prep    : view descriptors from the host's page-locked staging, counters to zero
//   k_vertex  : (large sequences of shared vertices) SoA positions -> screen vertex per view (world
//               attributes are transformed per corner where a triangle survives)
//   k_setup   : per face: fast accept or the clip queue (graphics.cpp:132-161), divide / cull /
//               viewport / bbox (graphics.cpp:314-347) -> one 64-byte RasterRec
//   k_emit    : shading payloads and per-tile counts (warp-aggregated atomics) of the records; in
//               sequences of up to 2^21 faces the same grid clips (larger ones: k_post after it)
//   k_scan    : sub-records of triangles that touch many tiles, then exclusive prefix sums of the
//               per-tile counts and of the non-empty tiles (decoupled look-back), and the list of
//               non-empty tiles in tile order
//   k_scatter : (record, tile) pairs into per-tile lists; beside it, in the same grid, the
//               fused clear of the tiles no triangle touches, streamed row by row
//   k_raster  : persistent over the non-empty tiles; one warp owns one screen tile (a CTA
//               where tiles are few), resolves visibility per pixel as min over (depth, later-submitted) — the
//               sequential loop's result — then shades the winners and writes colour /
//               depth / prim id once.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/hsr.h"

namespace hsr {

// Vertices of a clipped polygon: 3 + one per clip plane (7) in exact arithmetic, more where rounding
// bends a polygon that lies along a corner line of the frustum (12 seen).  Vertices past the last
// place are dropped.
constexpr int kMaxPoly = 16;
constexpr int kMaxMeshFaces = 1 << 27;    // hsr_mesh_upload refuses more
constexpr int kVaryings = 13;             // floats in shader_struct_v2f (IShader.h:41-47)
constexpr int kMaxRecordTiles = 32;       // records never touch more tiles (big ones are split)
constexpr int kSubTilesX = 8, kSubTilesY = 4;  // tile block of one sub-record
constexpr int kPayloadFloats = 32;        // per-record shading payload (see Payload layout)

// Error bits in Ctl::error.
enum : uint32_t {
  kErrRecOverflow = 1u,
  kErrClipOverflow = 2u,
  kErrBinOverflow = 4u,
  kErrWaitTimeout = 8u,
  kErrScanTimeout = 16u,
  kErrBigOverflow = 32u,
};
constexpr uint32_t kErrCapacity = kErrRecOverflow | kErrClipOverflow | kErrBinOverflow | kErrBigOverflow;
// A sequence with one of these draws nothing: the binning and the raster return before
// writing (an overflow is re-run with larger scratch; a scan that gave up has no tile lists).
constexpr uint32_t kErrNoDraw = kErrCapacity | kErrScanTimeout;
// Default poll limits of the bounded waits (Scratch::poll_limit overrides both).
constexpr int kPollNs = 64;                // sleep between two polls
constexpr long kDepWaitPolls = 1L << 24;   // raster: a shadow map's tiles (1-2 s)
constexpr long kScanWaitPolls = 1L << 22;  // scan: a predecessor block's prefix

// Record flags.
enum : uint32_t {
  kRecExact = 1u,  // coordinates outside the range where the division-free coverage test is
                   // exact: the raster evaluates the reference's divisions instead
  kRecHole = 2u,   // slot of a huge triangle handed to k_scan: binned nowhere
};

// One triangle that reached the raster (64 bytes).  A, B-A, C-A are the per-triangle
// constants of barycentric() (graphics.cpp:222-233); uz is u.z, constant per triangle.  The
// last 16 bytes are the words the emit pass and the scatter read (one 16-byte load each); a
// record's payload is at the record's own index.
struct __align__(16) RasterRec {
  float ax, ay, e1x, e1y;   // A; e1 = B - A
  float e2x, e2y, uz, d0;   // e2 = C - A; u.z; screen depth of A
  float d1, d2;             // screen depths of B, C
  uint32_t face;            // position of the face in the mesh's face arrays (cull pass's records)
  uint32_t pad;             // reserved (zero)
  uint32_t seq;             // (face << kSeqFaceShift) | (fan << 1) | clipped — submission order
  uint32_t view;            // index of the view in the batch | flags << 28 (kRec*)
  uint32_t xr, yr;          // inclusive pixel range: x0 | x1 << 16, y0 | y1 << 16
};
static_assert(offsetof(RasterRec, seq) == 48 && offsetof(RasterRec, yr) == 60, "binning words in the last 16 bytes");
constexpr uint32_t kRecViewMask = 0x0fffffffu;
constexpr int kRecFlagShift = 28;

// Per-record shading payload (kPayloadFloats floats, same index as the record): the
// reciprocal w of each corner (graphics.cpp:333-337) and the corner varyings the shader
// reads, so that shading a pixel needs the record and this payload only.
//   [0..2] 1/w of corners 0..2, [3] unused,
//   corner k at 4 + 9k: world_pos[3], world_normal[3], uv[2], scalar
//   (scalar = clip_pos.z for ShadowShader, intensity for Ground/Toon).
struct __align__(16) Payload {
  float f[kPayloadFloats];
};
constexpr int kSeqFaceShift = 5;
static_assert(kMaxPoly - 2 <= 1 << (kSeqFaceShift - 1), "the fan index must not reach the face's bits");
// (below 2^32 - 1: the raster's keys hold 0xfffffffe - seq, and 0xffffffff stands for the buffer's depth)
static_assert(((uint64_t)kMaxMeshFaces << kSeqFaceShift) - (1u << kSeqFaceShift) + 2 * (kMaxPoly - 3) + 1 <= 0xfffffffeull,
              "submission words must fit 32 bits");
static_assert(sizeof(RasterRec) == 64, "RasterRec must stay 64 bytes");

// Per-draw descriptor on the device.  The fields every raster tile reads come first, in
// one 128-byte line (the struct is 128-byte aligned); the rest is read by the vertex and
// setup stages and by the shading of tiles that hold fragments.
struct __align__(128) DView {
  // target and tiles (read per raster tile)
  // (depth and prim may be null: planes nobody reads; depth only with the fused clear)
  uint32_t* color; float* depth; uint32_t* prim; int32_t W, H;
  int32_t tile_base, tiles_x, tiles_y, ntiles;
  int32_t shader;
  uint32_t flags;       // HSR_DRAW_*
  float clear_depth;
  uint32_t clear_rgba;
  // ordering inside the batch: views this one waits for (-1 = none)
  int32_t dep0, dep1;
  int32_t has_dependents;  // kTargetReaders | kTileReaders: which later views wait for this one's tiles
  uint32_t prim_base;
  // mesh (device)
  const float* px; const float* py; const float* pz;   // positions, SoA, padded to 4
  const float* nx; const float* ny; const float* nz;   // normals, SoA, padded to 4
  const float2* uv;
  // per-face corner indices, in an order of the library's own (near faces near one another, fv into
  // the library's order of the positions); fv.w is the face's number in the caller's array
  const int4* fv; const int4* fvt; const int4* fvn;
  int32_t npos, nnrm, nuv, nfaces;
  int32_t unified;  // every face corner has equal v, vt and vn indices (fvt, fvn unused)
  // the mesh's positions and normals as (x, y, z, 0), gathered per corner for the world
  // attributes, and which of those the view's shader reads (kWorld*)
  const float4* p4; const float4* n4;
  const float4* pk;  // unified meshes: position, normal and uv of a vertex in one sector (else null)
  uint32_t world;
  // vertex outputs (scratch)
  float4* sv;     // [npos] screen vertex: (x/w, y/w, z/w, 1/w) or plane mask (k_vertex)
  // shading
  float mvp[16];        // camera_vp*model (light_vp*model for SHADOW), host-computed
  hsr_shader_data u;
  const uint32_t* diffuse; int32_t dw, dh, dbpp;
  const uint32_t* normal;  int32_t nw, nh, nbpp;
  // shadow map (colour plane of another target), null when ShaderData::shadow_map is null
  const uint32_t* sm_color; int32_t smW, smH;
  // this view's work chunks in the batch's chunk spaces (a kernel finds the view of chunk c
  // as the last view whose base is <= c): vertex chunks of kVertexChunk positions, setup
  // chunks of kSetupChunk faces, clear chunks of kClearChunk pixels (none for a view drawn
  // without the fused clear)
  int32_t vch_base, vch_npos, vch_count;
  int32_t sch_base;
  int32_t cch_base;
};
// DView::has_dependents: a later view reads the whole target (a shadow map; this view is the last to
// write it or one before that), and a later view draws into the same target (each of its tiles
// waits for this view's tile at the same place).
constexpr int32_t kTargetReaders = 1, kTileReaders = 2;
constexpr int kVertexChunk = 2048;  // positions per vertex-stage chunk
constexpr uint32_t kWorldPos = 1u, kWorldNormal = 2u;  // DView::world
// The world attributes a shader's fragment() reads (IShader.cpp): the world position for the
// view vector and the shadow lookup, the world normal for lighting (and the intensity of
// Ground / Toon, which rides in its w).
__host__ __device__ inline uint32_t world_attrs(int shader) {
  const bool pos = shader == HSR_SHADER_BLINN || shader == HSR_SHADER_NORMALMAP;
  const bool nrm = shader == HSR_SHADER_GROUND || shader == HSR_SHADER_TOON || shader == HSR_SHADER_TEXTURE_WITH_LIGHT ||
                   shader == HSR_SHADER_BLINN || shader == HSR_SHADER_NORMALMAP;
  return (pos ? kWorldPos : 0u) | (nrm ? kWorldNormal : 0u);
}
constexpr int kSetupChunk = 128;    // faces per setup chunk (one per thread of a block)
constexpr int kClearChunk = 1024;   // pixels per clear chunk (32 per lane of a warp)
constexpr int64_t kMaxBatchTiles = (int64_t)1 << 26;  // tiles of one launch sequence (scan word)
static_assert(offsetof(DView, prim_base) + sizeof(uint32_t) <= 128, "per-tile fields must share one line");

struct Ctl {
  uint32_t rec_count;      // records of the cull pass
  uint32_t clip_count;
  uint32_t rec_extra;      // records appended behind them (clipped triangles, sub-records)
  uint32_t scan_ticket;
  uint32_t error;
  uint32_t bin_total;
  uint32_t big_count;      // triangles queued for sub-record expansion
  uint32_t post_next;      // work counter of k_post
  unsigned long long shaded_px;  // pixels whose winner was shaded by the raster
  unsigned long long frag_px;    // covered (pixel, triangle) pairs the raster depth-tested
  uint32_t ne_tiles;             // tiles with at least one record (k_scan)
  float box_px;                  // pixels of the cull pass's records' bounding boxes (k_emit)
  unsigned long long pay_bytes;  // shading payload bytes written (k_emit, k_post, k_scan)
};
static_assert(sizeof(Ctl) == 64, "Ctl is read back whole: keep it one 64-byte block");
constexpr size_t kSplitWords = 128;  // Scratch::split, in the zeroed 256 bytes that hold Ctl, on a line of its own

// A triangle whose bounding box touches more than kMaxRecordTiles tiles, queued by
// the emit and clip passes and expanded into sub-records by k_scan.
struct __align__(16) BigItem {
  RasterRec rec;
  Payload pay;
};

// Work chunk for the vertex and setup kernels: items [begin, end) of one view.
struct Chunk {
  int32_t view;
  int32_t begin;
  int32_t end;
};
constexpr int kSharedViews = 256;  // views whose chunk / tile bases kernels copy to shared memory

// Scratch of one launch sequence (device pointers, sized by the host).
struct Scratch {
  Ctl* ctl;
  uint32_t* view_done;      // [nviews] tiles finished per view, then [kRasterGroups] tile counters and the
                            // count of finished raster CTAs
  RasterRec* recs;  uint32_t rec_cap;
  Payload* pay;             // [rec_cap]
  int2* clipq;      uint32_t clip_cap;   // (view, face) of faces that need clipping
  BigItem* bigq;    uint32_t big_cap;
  uint32_t* tile_count;     // [ntiles]
  uint32_t* tile_fill;      // [ntiles]
  uint32_t* tile_off;       // [ntiles]
  uint32_t* ne_off;         // [ntiles + 1] non-empty tiles before each tile
  uint32_t* tile_list;      // [ntiles] the non-empty tiles in tile order (ne_tiles of them)
  unsigned long long* split;        // parts of huge triangles split, their sub-records, the splitters' beats
                                    // (three words, kSplitWords bytes behind ctl)
  unsigned long long* scan_status;  // [scan blocks]
  uint32_t* bins;   uint32_t bin_cap;
  int32_t ntiles;
  int32_t nviews;
  // the raster launch's part of the tiles, [tile_lo, tile_hi), and the counter that hands them out
  int32_t tile_lo, tile_hi;
  uint32_t* claim;
  // where the raster's last CTA (counted by `finished`) stores the control block: mapped host
  // memory, null for a launch that is not the sequence's last or whose host copies it itself
  Ctl* ctl_out;
  uint32_t* finished;
  float* stash;             // [stash_warps][stash_floats(tile)] per raster warp (may be null)
  uint32_t stash_warps;
  uint32_t faults;          // HSR_FAULT_* injected by the host (tests of the failure paths)
  int32_t poll_limit;       // polls before a bounded wait gives up (0: the defaults above)
};
// Per raster warp of a 16x16 or 32x32 tile, per pixel: the winner's weights b0, b1, b2 as one
// 16-byte entry — what shading would otherwise re-derive from the record.  (The winner's record
// index, which is also its payload index, and its submission word are in the tile's shared state.)
__host__ __device__ constexpr int stash_floats(int tile) { return 4 * tile * tile; }
constexpr int kRasterGroups = 4;  // raster launches of one sequence at most
constexpr int kStashWarpsPerSm = 32;  // raster warps resident per SM at most

// Blocks of 256 threads that walk a mesh array of n items.  (The walks count in 64 bits: an array may
// have up to 2^31 - 1 items, and an int would wrap on the last step.)
inline int item_blocks(int n) {
  const size_t want = ((size_t)(n > 0 ? n : 1) + 255) / 256;
  return (int)(want < 4096 ? want : 4096);
}

// First of n records that share k of `parts` takes, the shares as even as they come (no product that a
// long list could carry past 32 bits).
__host__ __device__ constexpr uint32_t share_begin(uint32_t n, uint32_t k, uint32_t parts) {
  return n / parts * k + (k < n % parts ? k : n % parts);
}

// Warps of the scatter that share the same 32 records: up to kMaxSharers where records are few, and no
// more than there are.
constexpr uint32_t kMaxSharers = 16;
__host__ __device__ constexpr uint32_t scatter_sharers(uint32_t nrec, uint32_t warps) {
  uint32_t parts = warps * 32u / (nrec ? nrec : 1u);
  if (parts > kMaxSharers) parts = kMaxSharers;
  if (parts > warps) parts = warps;
  return parts ? parts : 1u;
}

// What of a sequence's empty tiles the scatter's grid clears: `clear_bytes`, the planes of the views that
// clear, of the three planes of all views' pixels (several draws into one target clear it once).
inline float clear_share(size_t clear_bytes, size_t pixels) {
  return (float)clear_bytes / (12.f * (float)(pixels ? pixels : 1));
}
// Of how many blocks of that grid one scatters while the others clear: two, or three where the pixels to
// clear (of three planes) outweigh the (record, tile) pairs (see k_scatter).
constexpr float kClearHeavy = 10.f;
__host__ __device__ constexpr uint32_t scatter_every(uint32_t empty_tiles, int tile, float share, uint32_t pairs) {
  return (float)empty_tiles * (float)(tile * tile) * share >= kClearHeavy * (float)pairs ? 3u : 2u;
}

// Kernel launchers (kernels_*.cu).  All return cudaError_t as int.
//
// A mesh's position and face arrays, which a mesh of kOrderedFaces faces or more keeps in an order of
// the library's own (see k_place_positions).
struct MeshArrays {
  float *px, *py, *pz;
  float4* p4;
  uint32_t* vorder;                  // [npos] the caller's index of each position
  int4 *fv, *fvt, *fvn;
};
constexpr int kMeshCells = 1 << 18;
// Smaller meshes keep the caller's order.  Device time of a 1280x720 draw in the caller's order and in the
// library's: icospheres of 5k faces 59 -> 60 us, 20k 54.5 -> 54.2, 82k 57.6 -> 55.7, 328k 73 -> 66; grids
// and soups of 33k faces equal, soups of 130k 138 -> 136, 500k 164 -> 158 (grids come in order).  Ordering
// adds 0.4 ms to an upload of any size (0.15 -> 0.6 ms at 5k faces, 2.7 -> 3.1 at 328k).
constexpr int kOrderedFaces = 1 << 15;
struct MeshOrder {                   // the caller's arrays on the device, and scratch
  const float* pos; int npos;        // [npos][3]
  const int32_t* faces; int nfaces;  // [nfaces][3 corners][v, vt, vn]
  uint32_t* cells;                   // kMeshCells + 8 words
  uint32_t* codes;                   // max(npos, nfaces) words
  uint32_t* place;                   // npos words
};
int launch_mesh_order(const MeshOrder& o, const MeshArrays& m, cudaStream_t s);
// Pieces of the caller's arrays, in the caller's order: items first, first + 1, ..., n of them.
int launch_place_positions(const float* pos, int first, int n, const MeshArrays& m, cudaStream_t s);
int launch_place_faces(const int32_t* faces, int first, int n, const MeshArrays& m, cudaStream_t s);
int launch_split_normals(const float* nrm, int n, float* nx, float* ny, float* nz, float4* n4, cudaStream_t s);
// `from` is mapped host memory or device memory; sizes are multiples of 16.
int launch_prep(const void* from, void* to, size_t copy, void* counters, size_t zero, int max_grid, cudaStream_t s);
int launch_vertex(const DView* views, int nviews, int nchunks, cudaStream_t s);
bool culls_own_vertices(size_t faces, size_t positions);  // the cull pass needs no launch_vertex
int launch_setup(const DView* views, int nviews, int nchunks, bool own_vertices, Scratch sc, int grid, cudaStream_t s);
bool clips_with_emit(size_t faces);  // the emit pass's grid also clips (no launch_post)
int launch_emit(const DView* views, int tile, Scratch sc, bool clip, int num_sms, cudaStream_t s);
int launch_post(const DView* views, int tile, Scratch sc, int grid, cudaStream_t s);
// One grid for both parts, or (to time them) a grid of `splitters` blocks and a grid that scans.
enum { kSplitAndScan, kSplitAlone, kScanAlone };
int launch_scan(const DView* views, int tile, Scratch sc, int splitters, int part, cudaStream_t s);
int launch_scatter(const DView* views, int tile, Scratch sc, int grid, int clear_chunks, float clear_share, cudaStream_t s);
int launch_raster(const DView* views, int tile, Scratch sc, int grid, int warps, cudaStream_t s);
int scan_blocks(int ntiles);

}  // namespace hsr
