// kernels_geom.cu — vertex transform and triangle setup (sm_103a).
//
// k_vertex replaces the per-corner IShader::vertex calls of graphics.cpp:380-387.  The
// vertex shader is a pure function of its a2v inputs, and each output stream depends on
// one attribute stream only (clip and world position on `v`, world normal and light
// intensity on `vn`, uv passes through), so every corner gets the same bits whether an
// output is computed once per vertex or once per corner.  The clip position and the
// per-corner work of rasterize_triangle that depends on one vertex alone — the visibility
// test of clip_triangle's fast accept (graphics.cpp:132-134, 140-142) and, for a visible
// vertex, the perspective divide and 1/w (:320-337) — is done here once per vertex (the
// screen vertex, see screen_vertex), so setup divides nothing on the fast path.  World
// position and normal are needed only for the corners of the one triangle in five that
// survives setup: k_emit (and the clipper) transform them per corner (world_pos_of,
// world_normal_of) instead of this pass writing and re-reading them for every vertex.
//
// k_setup (the cull pass) follows graphics.cpp:136-161 (clip) and :314-347 (cull, viewport,
// bounding box) for every face that passes the fast accept and stores one RasterRec per
// surviving triangle; faces that need the clipper are queued.  k_emit writes the surviving
// records' shading payloads and tile counts on dense warps; k_post clips the queued faces (two
// per warp: lane k of a half-warp carries varying k of the polygon through Sutherland-Hodgman)
// and emits their fan triangles.  Triangles that touch more than kMaxRecordTiles tiles are queued
// for the scan (kernels_bin.cu), which splits them into sub-records.
#include <float.h>

#include <algorithm>

#include "hsr_device.cuh"
#include "hsr_launch.cuh"

namespace hsr {

constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------------------------------
// clip-space helpers
// ---------------------------------------------------------------------------------------
enum { PW, PX, NX, PY, NY, PZ, NZ };

// is_inside_plane (graphics.cpp:29-49) on clip coordinates c[0..3]
__device__ __forceinline__ bool inside_plane(const float* c, int plane) {
  switch (plane) {
    case PW: return c[3] >= 1e-5f;
    case PX: return c[0] <= c[3];
    case NX: return c[0] >= -c[3];
    case PY: return c[1] <= c[3];
    case NY: return c[1] >= -c[3];
    case PZ: return c[2] <= c[3];
    default: return c[2] >= -c[3];
  }
}
// get_intersect_ratio (graphics.cpp:51-71)
__device__ __forceinline__ float intersect_ratio(const float* p, const float* q, int plane) {
  switch (plane) {
    case PW: return fd(fs(p[3], 1e-5f), fs(p[3], q[3]));
    case PX: return fd(fs(p[3], p[0]), fs(fs(p[3], p[0]), fs(q[3], q[0])));
    case NX: return fd(fa(p[3], p[0]), fs(fa(p[3], p[0]), fa(q[3], q[0])));
    case PY: return fd(fs(p[3], p[1]), fs(fs(p[3], p[1]), fs(q[3], q[1])));
    case NY: return fd(fa(p[3], p[1]), fs(fa(p[3], p[1]), fa(q[3], q[1])));
    case PZ: return fd(fs(p[3], p[2]), fs(fs(p[3], p[2]), fs(q[3], q[2])));
    default: return fd(fa(p[3], p[2]), fs(fa(p[3], p[2]), fa(q[3], q[2])));
  }
}
__device__ __forceinline__ bool vertex_visible(float4 c) {  // is_vertex_visible (:132-134)
  return fabsf(c.x) <= c.w && fabsf(c.y) <= c.w && fabsf(c.z) <= c.w;
}

// Clip position of vertex i of a view: ObjectToClipPos (IShader.h:55-61), the bits k_vertex
// computed for it.
__device__ __forceinline__ float4 clip_of(const DView& v, int i) {
  return mat_vec(v.mvp, __ldg(v.px + i), __ldg(v.py + i), __ldg(v.pz + i), 1.f);
}

// Screen vertex of one clip position.  A vertex that is visible (is_vertex_visible,
// graphics.cpp:132-134) with w >= 1e-5 stores what rasterize_triangle derives from it
// alone: (x/w, y/w, z/w, 1/w) (graphics.cpp:321-323, 335-337); its |x/w| is <= 1 or NaN.
// Any other vertex stores (kSvSpecial, mask, 0, 0), bit p of the mask being
// is_inside_plane for plane p in the clipper's order (W, +X, -X, +Y, -Y, +Z, -Z) and bit 7
// is_vertex_visible.  A normal screen vertex is inside every plane (|x|,|y|,|z| <= w and
// w >= 1e-5), so its mask is 0xff.
constexpr float kSvSpecial = 4.0f;
__device__ __forceinline__ float4 screen_vertex(float4 c) {
  const bool vis = vertex_visible(c);
  if (vis && c.w >= 1e-5f) return make_float4(fd(c.x, c.w), fd(c.y, c.w), fd(c.z, c.w), fd(1.f, c.w));
  const float a[4] = {c.x, c.y, c.z, c.w};
  uint32_t m = vis ? 0x80u : 0u;
#pragma unroll
  for (int p = PW; p <= NZ; p++)
    if (inside_plane(a, p)) m |= 1u << p;
  return make_float4(kSvSpecial, __uint_as_float(m), 0.f, 0.f);
}
__device__ __forceinline__ bool sv_normal(float4 s) { return !(fabsf(s.x) > 1.f); }

// ObjectToWorldPos (IShader.h:63-65) of an object-space position.
__device__ __forceinline__ float4 world_pos(const DView& v, float x, float y, float z) {
  const float4 w = mat_vec(v.u.model_matrix, x, y, z, 1.f);
  return make_float4(w.x, w.y, w.z, 0.f);
}
__device__ __forceinline__ float4 world_pos_of(const DView& v, int i) {
  const float4 p = __ldg(v.p4 + i);
  return world_pos(v, p.x, p.y, p.z);
}
// ObjectToWorldNormal (IShader.h:71-75) = [n, 1] * model_I of an object-space normal, with the
// intensity of Ground / Toon, saturate(worldN . light_dir) (IShader.cpp:8, :26), in w.
__device__ __forceinline__ float4 world_normal(const DView& v, float nx, float ny, float nz) {
  const float* m = v.u.model_matrix_I;
  F3 wn;
  wn.x = dot4(nx, ny, nz, 1.f, m[0], m[4], m[8], m[12]);
  wn.y = dot4(nx, ny, nz, 1.f, m[1], m[5], m[9], m[13]);
  wn.z = dot4(nx, ny, nz, 1.f, m[2], m[6], m[10], m[14]);
  const F3 L = {v.u.light_dir[0], v.u.light_dir[1], v.u.light_dir[2]};
  return make_float4(wn.x, wn.y, wn.z, saturate(dot3(wn, L)));
}
__device__ __forceinline__ float4 world_normal_of(const DView& v, int i) {
  const float4 n = __ldg(v.n4 + i);
  return world_normal(v, n.x, n.y, n.z);
}
__device__ __forceinline__ uint32_t sv_mask(float4 s) { return sv_normal(s) ? 0xffu : __float_as_uint(s.y); }

// ---------------------------------------------------------------------------------------
// work chunks
// ---------------------------------------------------------------------------------------
// The chunk bases of all views in shared memory (nviews <= kSharedViews), read with
// `base_of` (field selector); every thread of the block calls this (ends with a barrier).
template <class F>
__device__ __forceinline__ const int32_t* share_bases(const DView* views, int nviews, int32_t* s_base, F base_of) {
  if (nviews > kSharedViews) return nullptr;
  for (int i = threadIdx.x; i < nviews; i += blockDim.x) s_base[i] = base_of(views[i]);
  __syncthreads();
  return s_base;
}
// View of chunk c: the last view whose base is <= c (views with no chunks share the next
// view's base and are never returned for a chunk they do not hold).  A block visits its
// chunks in increasing order, so the search walks forward from the view of its previous
// chunk (`hint`), usually zero or one step.
template <class F>
__device__ __forceinline__ int chunk_view(const DView* views, const int32_t* s_base, int nviews, int c, F base_of,
                                          int hint) {
  int k = hint;
  while (k + 1 < nviews && (s_base ? s_base[k + 1] : base_of(views[k + 1])) <= c) k++;
  return k;
}
// The same by binary search, for a block that starts cold.
template <class F>
__device__ __forceinline__ int chunk_view_search(const DView* views, const int32_t* s_base, int nviews, int c,
                                                 F base_of) {
  int lo = 0, hi = nviews - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((s_base ? s_base[mid] : base_of(views[mid])) <= c) lo = mid; else hi = mid - 1;
  }
  return lo;
}
struct VchBase { __device__ int32_t operator()(const DView& v) const { return v.vch_base; } };
struct SchBase { __device__ int32_t operator()(const DView& v) const { return v.sch_base; } };

// Chunk c of the vertex stage: view and position range.
__device__ __forceinline__ Chunk vertex_chunk(const DView* views, const int32_t* s_base, int nviews, int c) {
  const int k = chunk_view_search(views, s_base, nviews, c, VchBase());
  const DView& v = views[k];
  Chunk ch;
  ch.view = k;
  ch.begin = (c - v.vch_base) * kVertexChunk;
  ch.end = min(v.npos, ch.begin + kVertexChunk);
  return ch;
}
// Chunk c of the setup stage: view and face range.
__device__ __forceinline__ Chunk setup_chunk(const DView* views, const int32_t* s_base, int nviews, int c, int hint) {
  const int k = chunk_view(views, s_base, nviews, c, SchBase(), hint);
  const DView& v = views[k];
  Chunk ch;
  ch.view = k;
  ch.begin = (c - v.sch_base) * kSetupChunk;
  ch.end = min(v.nfaces, ch.begin + kSetupChunk);
  return ch;
}

// ---------------------------------------------------------------------------------------
// mesh order (once per mesh)
// ---------------------------------------------------------------------------------------
// A large mesh keeps its positions and its faces grouped by place, in the Morton order of a 64^3
// grid's cells: faces near one another are then culled by the same warp, gather the same vertices
// from neighbouring sectors, reserve neighbouring records and fall into the same tiles.  The
// caller's order of an icosphere (all first children of a subdivision, then all second ones, ...)
// or of a triangle soup is spread over the whole mesh.  The caller's face number travels in fv.w,
// and submission order and primitive ids come from it; a position's normal and uv are found
// through vorder.  So no result depends on this order, and the order inside a cell is left to
// the atomics.  64 requests over eight meshes of 41k-1.3M faces: emit 403 -> 340 us, scatter 322 ->
// 300; 4M-triangle soup: scatter 102 -> 63, raster 817 -> 793.
__device__ __forceinline__ int ordered_int(float f) {  // int order equals float order
  const int b = __float_as_int(f);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ordered_int(int o) { return __int_as_float(o >= 0 ? o : o ^ 0x7fffffff); }

__global__ void k_bounds_init(int* bounds) {
  if (threadIdx.x < 6) bounds[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : (int)0x80000000;
}
// bounds[0..2] minima, [3..5] maxima of the finite coordinates, as ordered ints.
__global__ void __launch_bounds__(256) k_bounds(const float* __restrict__ pos, int n, int* __restrict__ bounds) {
  float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += (size_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float c = pos[3 * i + k];
      if (fabsf(c) <= FLT_MAX) {
        lo[k] = fminf(lo[k], c);
        hi[k] = fmaxf(hi[k], c);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int l = __reduce_min_sync(kFull, ordered_int(lo[k])), h = __reduce_max_sync(kFull, ordered_int(hi[k]));
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&bounds[k], l);
      atomicMax(&bounds[3 + k], h);
    }
  }
}

__device__ __forceinline__ uint32_t spread_bits(uint32_t x) {  // 6 bits, two zeros between
  x = (x | (x << 8)) & 0x0000f00fu;
  x = (x | (x << 4)) & 0x000c30c3u;
  return (x | (x << 2)) & 0x00249249u;
}
// Cell of a point; a coordinate that is not finite lands in an outer cell.
__device__ __forceinline__ uint32_t cell_of(const int* __restrict__ bounds, const float* m) {
  uint32_t code = 0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float lo = from_ordered_int(bounds[k]), span = from_ordered_int(bounds[3 + k]) - lo;
    const float at = span > 0.f ? (m[k] - lo) / span * 64.f : 0.f;
    code |= spread_bits((uint32_t)fminf(fmaxf(at, 0.f), 63.f)) << k;
  }
  return code;
}

// Counts the cells of the items' points: positions (faces null) or face centroids.
__global__ void __launch_bounds__(256) k_cells(const float* __restrict__ pos, const int32_t* __restrict__ faces, int n,
                                               const int* __restrict__ bounds, uint32_t* __restrict__ cells,
                                               uint32_t* __restrict__ codes) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += (size_t)gridDim.x * blockDim.x) {
    float m[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      if (faces) {
        const int32_t* f = faces + 9 * i;
        m[k] = (pos[3 * (size_t)f[0] + k] + pos[3 * (size_t)f[3] + k] + pos[3 * (size_t)f[6] + k]) / 3.f;
      } else {
        m[k] = pos[3 * i + k];
      }
    }
    codes[i] = cell_of(bounds, m);
    atomicAdd(&cells[codes[i]], 1u);
  }
}

// Exclusive prefix sums of the kMeshCells counts, in place, by one block.
__global__ void __launch_bounds__(1024) k_cell_scan(uint32_t* __restrict__ cells) {
  __shared__ uint32_t sums[32];
  constexpr int kEach = kMeshCells / 1024;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* mine = reinterpret_cast<uint4*>(cells + (size_t)threadIdx.x * kEach);
  uint32_t sum = 0;
  for (int k = 0; k < kEach / 4; k++) {
    const uint4 q = mine[k];
    sum += q.x + q.y + q.z + q.w;
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t own = sums[lane];
    uint32_t w = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, w, o);
      if (lane >= o) w += y;
    }
    sums[lane] = w - own;
  }
  __syncthreads();
  uint32_t run = sums[warp] + incl - sum;
  for (int k = 0; k < kEach / 4; k++) {
    const uint4 q = mine[k];
    uint4 o;
    o.x = run; run += q.x;
    o.y = run; run += q.y;
    o.z = run; run += q.z;
    o.w = run; run += q.w;
    mine[k] = o;
  }
}

// Positions first, first + 1, ... (raw) to their places (their own with cells null): SoA, float4, the
// caller's index of each place and, where asked for, the place of each index.
__global__ void __launch_bounds__(256) k_place_positions(const float* __restrict__ pos, int first, int n,
                                                         uint32_t* __restrict__ cells, const uint32_t* __restrict__ codes,
                                                         float* __restrict__ px, float* __restrict__ py,
                                                         float* __restrict__ pz, float4* __restrict__ p4,
                                                         uint32_t* __restrict__ vorder, uint32_t* __restrict__ place) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t own = (uint32_t)first + (uint32_t)i, at = cells ? atomicAdd(&cells[codes[i]], 1u) : own;
    const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    px[at] = x;
    py[at] = y;
    pz[at] = z;
    p4[at] = make_float4(x, y, z, 0.f);
    vorder[at] = own;
    if (place) place[own] = at;
  }
}

// Faces first, first + 1, ... (raw), likewise; their corners' positions have moved to `place` (null: not).
__global__ void __launch_bounds__(256) k_place_faces(const int32_t* __restrict__ faces, int first, int n,
                                                     uint32_t* __restrict__ cells, const uint32_t* __restrict__ codes,
                                                     const uint32_t* __restrict__ place, int4* __restrict__ fv,
                                                     int4* __restrict__ fvt, int4* __restrict__ fvn) {
  auto at_place = [&](int32_t v) { return place ? (int)place[v] : v; };
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t own = (uint32_t)first + (uint32_t)i, at = cells ? atomicAdd(&cells[codes[i]], 1u) : own;
    const int32_t* r = faces + 9 * i;
    fv[at] = make_int4(at_place(r[0]), at_place(r[3]), at_place(r[6]), (int)own);
    fvt[at] = make_int4(r[1], r[4], r[7], 0);
    fvn[at] = make_int4(r[2], r[5], r[8], 0);
  }
}

int launch_place_positions(const float* pos, int first, int n, const MeshArrays& m, cudaStream_t s) {
  if (n <= 0) return 0;
  k_place_positions<<<item_blocks(n), 256, 0, s>>>(pos, first, n, nullptr, nullptr, m.px, m.py, m.pz, m.p4, m.vorder, nullptr);
  return (int)cudaGetLastError();
}
int launch_place_faces(const int32_t* faces, int first, int n, const MeshArrays& m, cudaStream_t s) {
  if (n <= 0) return 0;
  k_place_faces<<<item_blocks(n), 256, 0, s>>>(faces, first, n, nullptr, nullptr, nullptr, m.fv, m.fvt, m.fvn);
  return (int)cudaGetLastError();
}

int launch_mesh_order(const MeshOrder& o, const MeshArrays& m, cudaStream_t s) {
  const int pg = item_blocks(o.npos), fg = item_blocks(o.nfaces);
  int* bounds = reinterpret_cast<int*>(o.cells + kMeshCells);
  auto group = [&](const int32_t* faces, int n, int grid) {
    cudaError_t e = cudaMemsetAsync(o.cells, 0, sizeof(uint32_t) * kMeshCells, s);
    if (e != cudaSuccess) return e;
    k_cells<<<grid, 256, 0, s>>>(o.pos, faces, n, bounds, o.cells, o.codes);
    k_cell_scan<<<1, 1024, 0, s>>>(o.cells);
    return cudaGetLastError();
  };
  k_bounds_init<<<1, 32, 0, s>>>(bounds);
  k_bounds<<<std::min(pg, 1024), 256, 0, s>>>(o.pos, o.npos, bounds);
  cudaError_t e = group(nullptr, o.npos, pg);
  if (e != cudaSuccess) return (int)e;
  k_place_positions<<<pg, 256, 0, s>>>(o.pos, 0, o.npos, o.cells, o.codes, m.px, m.py, m.pz, m.p4, m.vorder, o.place);
  e = group(o.faces, o.nfaces, fg);
  if (e != cudaSuccess) return (int)e;
  k_place_faces<<<fg, 256, 0, s>>>(o.faces, 0, o.nfaces, o.cells, o.codes, o.place, m.fv, m.fvt, m.fvn);
  return (int)cudaGetLastError();
}

// Normals (raw xyz) as SoA and float4.
__global__ void __launch_bounds__(256) k_split_normals(const float* __restrict__ nrm, int n, float* __restrict__ nx,
                                                       float* __restrict__ ny, float* __restrict__ nz,
                                                       float4* __restrict__ n4) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n; i += (size_t)gridDim.x * blockDim.x) {
    const float x = nrm[3 * i], y = nrm[3 * i + 1], z = nrm[3 * i + 2];
    nx[i] = x;
    ny[i] = y;
    nz[i] = z;
    n4[i] = make_float4(x, y, z, 0.f);
  }
}
int launch_split_normals(const float* nrm, int n, float* nx, float* ny, float* nz, float4* n4, cudaStream_t s) {
  if (n <= 0) return 0;
  k_split_normals<<<item_blocks(n), 256, 0, s>>>(nrm, n, nx, ny, nz, n4);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// vertex stage
// ---------------------------------------------------------------------------------------
// One vertex chunk (kVertexChunk positions, 8 per thread, 256 threads): ObjectToClipPos /
// ObjectToViewPos (IShader.h:55-61) -> screen vertex.
__device__ __forceinline__ void vertex_chunk_work(const DView& v, const Chunk& ch) {
  // item i = begin + threadIdx.x + 256 k: consecutive threads read consecutive floats and
  // write consecutive float4s, so every load and store instruction of a warp is one
  // contiguous span; the loads of a thread are issued before any is used
  constexpr int kPer = kVertexChunk / 256;
  const int i0 = ch.begin + (int)threadIdx.x;
  float mvp[16];  // loaded once (read again after each store: 64 requests 83 -> 103 us)
#pragma unroll
  for (int k = 0; k < 16; k++) mvp[k] = v.mvp[k];
  float4* const sv = v.sv;
  float xs[kPer], ys[kPer], zs[kPer];
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int i = i0 + 256 * k;
    const bool in = i < ch.end;
    xs[k] = in ? __ldg(v.px + i) : 0.f;
    ys[k] = in ? __ldg(v.py + i) : 0.f;
    zs[k] = in ? __ldg(v.pz + i) : 0.f;
  }
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int i = i0 + 256 * k;
    if (i >= ch.end) break;
    sv[i] = screen_vertex(mat_vec(mvp, xs[k], ys[k], zs[k], 1.f));
  }
}

// One block per chunk (the blocks are short and many: their prologues overlap others' work).
__global__ void __launch_bounds__(256) k_vertex(const DView* views, int nviews) {
  __shared__ int32_t s_base[kSharedViews];
  chain_wait();
  const int32_t* base = share_bases(views, nviews, s_base, VchBase());
  const Chunk ch = vertex_chunk(views, base, nviews, (int)blockIdx.x);
  vertex_chunk_work(views[ch.view], ch);
}

int launch_vertex(const DView* views, int nviews, int nchunks, cudaStream_t s) {
  if (nchunks <= 0) return 0;
  return launch_chained(k_vertex, nchunks, 256, 0, s, views, nviews);
}

// ---------------------------------------------------------------------------------------
// setup stage
// ---------------------------------------------------------------------------------------
constexpr int kSetupCoverPixels = 12;  // pixel ranges up to this size are tested in setup

__device__ __forceinline__ bool coord_ok(float c) {
  // |c| == 0 or 2^-8 <= |c| <= 2^20, on the bits of |c| (NaN and inf are above the range)
  const uint32_t b = __float_as_uint(c) & 0x7fffffffu;
  return b == 0u || b - 0x3b800000u <= 0x49800000u - 0x3b800000u;
}

// Perspective divide of rasterize_triangle (graphics.cpp:321-323): clip / w per component.
__device__ __forceinline__ F3 ndc_of(float4 c) { return {fd(c.x, c.w), fd(c.y, c.w), fd(c.z, c.w)}; }

// Cull, viewport, bounding box of one fan triangle from its corners' NDC coordinates
// (graphics.cpp:324-347).
__device__ __forceinline__ bool build_rec(const DView& v, F3 n0, F3 n1, F3 n2, uint32_t seq, uint32_t view,
                                          RasterRec& r) {
  // is_back_facing (:172-180), evaluated left to right
  float sa = fs(fm(n0.x, n1.y), fm(n0.y, n1.x));
  sa = fa(sa, fm(n1.x, n2.y));
  sa = fs(sa, fm(n1.y, n2.x));
  sa = fa(sa, fm(n2.x, n0.y));
  sa = fs(sa, fm(n2.y, n0.x));
  if (sa <= 0.f) return false;
  const F3 s0 = viewport(v.W, v.H, n0), s1 = viewport(v.W, v.H, n1), s2 = viewport(v.W, v.H, n2);
  // bounding box with std::min / std::max (:339-347)
  float bminx, bminy, bmaxx, bmaxy;
  const float clampx = (float)(v.W - 1), clampy = (float)(v.H - 1);
  const float sx[3] = {s0.x, s1.x, s2.x}, sy[3] = {s0.y, s1.y, s2.y};
  if (!(sx[0] != sx[0] || sx[1] != sx[1] || sx[2] != sx[2] || sy[0] != sy[0] || sy[1] != sy[1] || sy[2] != sy[2])) {
    // no NaN: the chains below reduce to min / max (a signed zero only reaches the (int)
    // conversions and the < 0 tests, which treat -0 and +0 alike)
    bminx = fmaxf(0.f, fminf(fminf(sx[0], sx[1]), sx[2]));
    bmaxx = fminf(clampx, fmaxf(fmaxf(sx[0], sx[1]), sx[2]));
    bminy = fmaxf(0.f, fminf(fminf(sy[0], sy[1]), sy[2]));
    bmaxy = fminf(clampy, fmaxf(fmaxf(sy[0], sy[1]), sy[2]));
  } else {
    bminx = FLT_MAX; bminy = FLT_MAX; bmaxx = -FLT_MAX; bmaxy = -FLT_MAX;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      bminx = std_max(0.f, std_min(bminx, sx[i]));
      bmaxx = std_min(clampx, std_max(bmaxx, sx[i]));
      bminy = std_max(0.f, std_min(bminy, sy[i]));
      bmaxy = std_min(clampy, std_max(bmaxy, sy[i]));
    }
  }
  // pixels visited: x from (int)bboxmin.x while x <= bboxmax.x (:350-351)
  const int32_t x0 = cvt_i32(bminx), y0 = cvt_i32(bminy);
  if (x0 < 0 || y0 < 0 || bmaxx < 0.f || bmaxy < 0.f) return false;
  const int32_t x1 = (int32_t)floorf(bmaxx), y1 = (int32_t)floorf(bmaxy);
  if (x0 > x1 || y0 > y1) return false;
  // barycentric() constants (:222-233): u.z = (C.x-A.x)(B.y-A.y) - (B.x-A.x)(C.y-A.y)
  const float e1x = fs(s1.x, s0.x), e1y = fs(s1.y, s0.y);
  const float e2x = fs(s2.x, s0.x), e2y = fs(s2.y, s0.y);
  const float uz = fs(fm(e2x, e1y), fm(e1x, e2y));
  if (!(fabsf(uz) > 0.01f)) return false;  // degenerate: every pixel gets (-1,1,1)
  const bool ok = coord_ok(s0.x) && coord_ok(s0.y) && coord_ok(s1.x) && coord_ok(s1.y) &&
                  coord_ok(s2.x) && coord_ok(s2.y) && fabsf(uz) <= 0x1p30f;
  // a small pixel range is tested here with the raster's own coverage test: a triangle
  // that covers none of its pixels would only be visited and rejected pixel by pixel
  if ((x1 - x0 + 1) * (y1 - y0 + 1) <= kSetupCoverPixels) {
    bool any = false;
    for (int32_t y = y0; y <= y1 && !any; y++)
      for (int32_t x = x0; x <= x1 && !any; x++) {
        float b0, b1, b2;
        any = cover_test(s0.x, s0.y, e1x, e1y, e2x, e2y, uz, !ok, (float)x, (float)y, b0, b1, b2);
      }
    if (!any) return false;
  }
  r.ax = s0.x; r.ay = s0.y; r.e1x = e1x; r.e1y = e1y;
  r.e2x = e2x; r.e2y = e2y; r.uz = uz; r.d0 = s0.z;
  r.d1 = s1.z; r.d2 = s2.z;
  r.seq = seq;
  r.xr = (uint32_t)x0 | ((uint32_t)x1 << 16);
  r.yr = (uint32_t)y0 | ((uint32_t)y1 << 16);
  r.view = view | ((ok ? 0u : kRecExact) << kRecFlagShift);
  r.face = 0u;
  r.pad = 0u;
  return true;
}

// Corner varyings c[k] in shader_struct_v2f order (13 floats) -> payload.
__device__ __forceinline__ void make_payload(int shader, const float* c0, const float* c1, const float* c2,
                                             Payload& p) {
  const float* c[3] = {c0, c1, c2};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    p.f[k] = fd(1.f, c[k][3]);                                   // recip_w (graphics.cpp:333-337)
    p.f[3 + k] = shader == HSR_SHADER_SHADOW ? c[k][2] : c[k][12];
    p.f[6 + 2 * k] = c[k][10];
    p.f[7 + 2 * k] = c[k][11];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      p.f[12 + 3 * k + q] = c[k][7 + q];
      p.f[21 + 3 * k + q] = c[k][4 + q];
    }
  }
  p.f[30] = 0.f;
  p.f[31] = 0.f;
}

__device__ __forceinline__ void store_payload(Payload* dst, const Payload& p, int nf4) {
  float4* d = reinterpret_cast<float4*>(dst);
  const float4* s = reinterpret_cast<const float4*>(&p);
#pragma unroll
  for (int q = 0; q < 8; q += 2) {
    if (q + 1 < nf4) st_v8(d + q, s[q], s[q + 1]);
    else if (q < nf4) d[q] = s[q];
  }
}

// Slot of this lane's item when `want`, one atomicAdd per warp (~0u otherwise).
__device__ __forceinline__ uint32_t warp_reserve(bool want, uint32_t* counter) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(kFull, want);
  if (!m) return ~0u;
  const int leader = __ffs(m) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
  base = __shfl_sync(kFull, base, leader);
  return want ? base + (uint32_t)__popc(m & ((1u << lane) - 1u)) : ~0u;
}

// Slot of this thread's item when `want`, one atomicAdd per block (~0u otherwise).  Every
// thread of the block calls this.  All warps of the grid append to one counter, and a
// returning atomic on a single address is served one at a time: reserving per block
// instead of per warp divides those atomics by the warps of a block.
template <int THREADS>
__device__ __forceinline__ uint32_t block_reserve(bool want, uint32_t* counter) {
  __shared__ uint32_t s_count[THREADS / 32];
  __shared__ uint32_t s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(kFull, want);
  if (lane == 0) s_count[warp] = (uint32_t)__popc(m);
  __syncthreads();
  if (warp == 0) {
    const uint32_t c = lane < THREADS / 32 ? s_count[lane] : 0u;
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < THREADS / 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(kFull, incl, THREADS / 32 - 1);
    if (lane < THREADS / 32) s_count[lane] = incl - c;
    if (lane == 0) s_base = total ? atomicAdd(counter, total) : 0u;
  }
  __syncthreads();
  return want ? s_base + s_count[warp] + (uint32_t)__popc(m & ((1u << lane) - 1u)) : ~0u;
}

// Store the records of a warp at their slots (at most one per lane, each touching
// <= kMaxRecordTiles tiles) with their payloads, and count the tiles they touch,
// aggregating equal tiles across lanes.  All 32 lanes call this.
// With `in_place`, the record is already stored (the emit pass): only its payload (at the
// record's own index) and its tile counts are written.
__device__ void append_counts(bool valid, uint32_t slot, const RasterRec& r, const Payload& pl, int nf4, const DView& v,
                              int T, const Scratch& sc, bool in_place = false) {
  const int lane = threadIdx.x & 31;
  int tx0 = 0, ty0 = 0, ntw = 1, nt = 0;
  if (valid) {
    if (!in_place) store_rec(&sc.recs[slot], r);
    store_payload(&sc.pay[slot], pl, nf4);
    rec_tiles(r, T, tx0, ty0, ntw, nt);
  }
  auto count = [&](bool in, int tile, int) {
    const unsigned grp = __match_any_sync(kFull, in ? tile : -1);
    if (in && lane == __ffs(grp) - 1) atomicAdd(&sc.tile_count[tile], (uint32_t)__popc(grp));
  };
  const int tile0 = v.tile_base + ty0 * v.tiles_x + tx0;
  for_each_pair(nt, ntw, tile0, v.tiles_x, count, [&](int most) {
    int kx = 0, row = tile0;
    for (int k = 0; k < most; k++) {
      count(k < nt, row + kx, lane);
      if (++kx == ntw) { kx = 0; row += v.tiles_x; }
    }
  });
}

// append_counts at slots reserved by the caller, checked against the record capacity.
__device__ void append_small(bool valid, uint32_t slot, RasterRec r, const Payload& pl, int nf4, const DView& v,
                             int T, const Scratch& sc) {
  const bool ok = valid && slot < sc.rec_cap;
  if (valid && !ok) atomicOr(&sc.ctl->error, kErrRecOverflow);
  append_counts(ok, slot, r, pl, nf4, v, T, sc);
}

// Hand over a triangle that touches more than kMaxRecordTiles tiles at the queue slot `bslot`:
// the places of its sub-records among all (behind the clipper's records) are reserved here, in
// RasterRec::pad of the queued record, so that several CTAs can split one triangle without talking to
// each other.
__device__ __forceinline__ void queue_big(uint32_t bslot, RasterRec& r, const Payload& pl, int nf4, int T,
                                          const Scratch& sc) {
  const int ts = __ffs(T) - 1;
  auto tiles = [ts](uint32_t range) { return (int)((range >> 16 >> ts) - ((range & 0xffffu) >> ts)) + 1; };
  r.pad = (uint32_t)atomicAdd(sc.split + 1, (unsigned long long)sub_records(tiles(r.xr), tiles(r.yr)));
  if (bslot < sc.big_cap) {
    store_rec(&sc.bigq[bslot].rec, r);
    store_payload(&sc.bigq[bslot].pay, pl, nf4);
  } else {
    atomicOr(&sc.ctl->error, kErrBigOverflow);
  }
}

// True when the reference's clipper returns 0 vertices for this face without creating any
// new vertex: Sutherland-Hodgman copies a polygon whose vertices are all inside a plane
// unchanged, so if the three corners pass every plane before some plane (in the order
// W, +X, -X, +Y, -Y, +Z, -Z of graphics.cpp:152-158) and all fail that plane, that stage
// emits nothing and the face is dropped (CLIP_IN2OUT / CLIP_OUT2IN return 0).  Faces whose
// corners straddle a plane first go to the full clipper.  m0..m2 are the corners' plane
// masks (see screen_vertex).
__device__ __forceinline__ bool clip_trivially_empty(uint32_t m0, uint32_t m1, uint32_t m2) {
#pragma unroll
  for (int plane = PW; plane <= NZ; plane++) {
    const uint32_t all = (m0 & m1 & m2) >> plane & 1u, any = (m0 | m1 | m2) >> plane & 1u;
    if (!any) return true;
    if (!all) return false;
  }
  return false;
}

constexpr int kSetupThreads = kSetupChunk;  // one face per thread; a block's barriers span 4 warps
constexpr int kEmitThreads = 256;
constexpr int kPolyStride = kVaryings;  // floats per polygon vertex in shared memory


// Cull pass, one thread per face: fast accept, cull, viewport, bounding box and the
// coverage check of small ranges; a surviving triangle's 64-byte record is stored at a
// block-reserved slot (its payload and tile counts are still to come: k_emit), and
// faces that need the clipper are queued.  Four in five faces of the serving batches die
// here, so the per-record work runs in k_emit on dense warps instead of on the few lanes
// that survive in each warp of this pass.
//
// Persistent: block b takes chunks b, b + grid, ... (kSetupChunk faces each) and loads the face
// indices of its next chunk while it culls the current one, so the index stream from HBM
// overlaps the gathers and arithmetic instead of waiting at the head of every chunk.
// OWN: the screen vertices are computed here (no vertex stage), else gathered.
template <bool OWN>
__device__ __forceinline__ void cull_face(const DView& v, int f, uint32_t view, int4 iv, bool& valid,
                                          bool& needs_clip, RasterRec& r) {
  const int pi[3] = {iv.x, iv.y, iv.z};
  float4 sv[3];
#pragma unroll
  for (int k = 0; k < 3; k++) sv[k] = OWN ? screen_vertex(clip_of(v, pi[k])) : v.sv[pi[k]];
  bool accept = sv_normal(sv[0]) && sv_normal(sv[1]) && sv_normal(sv[2]);
  if (!accept) {
    const uint32_t m0 = sv_mask(sv[0]), m1 = sv_mask(sv[1]), m2 = sv_mask(sv[2]);
    if (m0 & m1 & m2 & 0x80u) {
      // all three visible, one with w < 1e-5: fast accept (graphics.cpp:140-148), divide here
      accept = true;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const F3 n = ndc_of(clip_of(v, pi[k]));
        sv[k] = make_float4(n.x, n.y, n.z, 0.f);
      }
    } else {
      needs_clip = !clip_trivially_empty(m0, m1, m2);
    }
  }
  if (accept)
    valid = build_rec(v, {sv[0].x, sv[0].y, sv[0].z}, {sv[1].x, sv[1].y, sv[1].z}, {sv[2].x, sv[2].y, sv[2].z},
                      (uint32_t)iv.w << kSeqFaceShift, view, r);
  r.face = (uint32_t)f;
}

template <bool OWN>
__global__ void __launch_bounds__(kSetupThreads, 8) k_setup(const DView* views, int nviews,
                                                         int nchunks, Scratch sc) {
  __shared__ int32_t s_base[kSharedViews];
  chain_wait();
  const int32_t* base = share_bases(views, nviews, s_base, SchBase());
  int c = (int)blockIdx.x;
  const int c_end = nchunks;
  if (c >= c_end) return;
  Chunk ch = setup_chunk(views, base, nviews, c, 0);
  int4 iv = make_int4(0, 0, 0, 0);
  if (ch.begin + (int)threadIdx.x < ch.end) iv = __ldg(&views[ch.view].fv[ch.begin + (int)threadIdx.x]);
  for (;;) {
    // the next chunk's face indices: issued now, consumed next iteration
    const bool more = c + (int)gridDim.x < c_end;
    Chunk chn = ch;
    int4 ivn = make_int4(0, 0, 0, 0);
    if (more) {
      chn = setup_chunk(views, base, nviews, c + (int)gridDim.x, ch.view);
      if (chn.begin + (int)threadIdx.x < chn.end) ivn = __ldg(&views[chn.view].fv[chn.begin + (int)threadIdx.x]);
    }
    const DView& v = views[ch.view];
    const int f = ch.begin + (int)threadIdx.x;
    bool needs_clip = false, valid = false;
    RasterRec r;
    if (f < ch.end) cull_face<OWN>(v, f, (uint32_t)ch.view, iv, valid, needs_clip, r);
    const uint32_t slot = block_reserve<kSetupThreads>(valid, &sc.ctl->rec_count);
    if (valid) {
      if (slot < sc.rec_cap) {
        store_rec(&sc.recs[slot], r);
      } else {
        atomicOr(&sc.ctl->error, kErrRecOverflow);
      }
    }
    const uint32_t cslot = warp_reserve(needs_clip, &sc.ctl->clip_count);
    if (needs_clip) {
      if (cslot < sc.clip_cap) sc.clipq[cslot] = make_int2(ch.view, f);
      else atomicOr(&sc.ctl->error, kErrClipOverflow);
    }
    if (!more) break;
    c += (int)gridDim.x;
    ch = chn;
    iv = ivn;
  }
}

// Payload of an unclipped face (Payload layout): the corner varyings of its three vertex()
// calls and their 1/w.  A mesh whose corners index positions, normals and uvs alike gives each
// corner's attributes in one 32-byte sector (DView::pk), and the corner's 1/w is computed from
// its position with the operations k_vertex used for the screen vertex (clip = mvp * [p, 1],
// 1 / clip.w; graphics.cpp:333-337), so no screen vertex is gathered again.
__device__ __forceinline__ void face_payload(const DView& v, int f, int nf4, int4 iv, Payload& pl) {
  int4 it = iv, in = iv;  // meshes whose v, vt and vn indices agree skip two loads
  if (!v.unified) {
    if (v.uv && nf4 >= 3) it = __ldg(&v.fvt[f]);
    if (v.world & kWorldNormal) in = __ldg(&v.fvn[f]);
  }
  const int pi[3] = {iv.x, iv.y, iv.z}, ti[3] = {it.x, it.y, it.z}, ni[3] = {in.x, in.y, in.z};
  const bool shadow = v.shader == HSR_SHADER_SHADOW;
  const bool need_nrm = (v.world & kWorldNormal) != 0u;
  const bool need_uv = v.uv && nf4 >= 3;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float px, py, pz, nx = 0.f, ny = 0.f, nz = 0.f;
    float2 t = make_float2(0.f, 0.f);
    if (v.pk) {
      const float4 a = __ldg(&v.pk[2 * (size_t)pi[k]]);
      px = a.x; py = a.y; pz = a.z; nx = a.w;
      if (need_nrm || need_uv) {
        const float4 b = __ldg(&v.pk[2 * (size_t)pi[k] + 1]);
        ny = b.x; nz = b.y; t = make_float2(b.z, b.w);
      }
    } else {
      const float4 p = __ldg(v.p4 + pi[k]);
      px = p.x; py = p.y; pz = p.z;
      if (need_nrm) {
        const float4 n = __ldg(v.n4 + ni[k]);
        nx = n.x; ny = n.y; nz = n.z;
      }
      if (need_uv) t = __ldg(&v.uv[ti[k]]);
    }
    const float4 c = mat_vec(v.mvp, px, py, pz, 1.f);  // ObjectToClipPos (IShader.h:55-61)
    const float4 wp = (v.world & kWorldPos) ? world_pos(v, px, py, pz) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 wn = need_nrm ? world_normal(v, nx, ny, nz) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (!need_uv) t = make_float2(0.f, 0.f);
    pl.f[k] = fd(1.f, c.w);  // recip_w
    // ShadowShader's interpolated clip z (ObjectToViewPos, IShader.cpp:170-174), else intensity
    pl.f[3 + k] = shadow ? c.z : wn.w;
    pl.f[6 + 2 * k] = t.x;
    pl.f[7 + 2 * k] = t.y;
    pl.f[12 + 3 * k] = wn.x; pl.f[13 + 3 * k] = wn.y; pl.f[14 + 3 * k] = wn.z;
    pl.f[21 + 3 * k] = wp.x; pl.f[22 + 3 * k] = wp.y; pl.f[23 + 3 * k] = wp.z;
  }
  pl.f[30] = 0.f;
  pl.f[31] = 0.f;
}

// Homogeneous clipping (graphics.cpp:73-161), two faces per warp: each half-warp clips its own
// face (`active`), lane k of the half carrying varying k of the polygon through
// Sutherland-Hodgman while every lane evaluates the plane tests on the clip coordinates; lanes
// j < n-2 of the half then build the fan triangles (:394-405).  The halves run the same
// instructions, each masked to its own polygon; every __syncwarp is reached by all 32 lanes.
__device__ void clip_face(bool active, const DView& v, int view, int face, int T, const Scratch& sc, float* A,
                          float* B, uint32_t rec_base, uint32_t& pay_bytes) {
  const int lane = threadIdx.x & 31, hl = lane & 15;
  if (active && hl < 3) {
    const int4 iv = __ldg(&v.fv[face]), it = __ldg(&v.fvt[face]), in = __ldg(&v.fvn[face]);
    const int pi = hl == 0 ? iv.x : (hl == 1 ? iv.y : iv.z);
    const int ti = hl == 0 ? it.x : (hl == 1 ? it.y : it.z);
    const int ni = hl == 0 ? in.x : (hl == 1 ? in.y : in.z);
    float* o = A + hl * kPolyStride;
    const float4 c = clip_of(v, pi);
    o[0] = c.x; o[1] = c.y; o[2] = c.z; o[3] = c.w;
    const float4 wp = (v.world & kWorldPos) ? world_pos_of(v, pi) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 wn = (v.world & kWorldNormal) ? world_normal_of(v, ni) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 t = v.uv ? __ldg(&v.uv[ti]) : make_float2(0.f, 0.f);
    o[4] = wp.x; o[5] = wp.y; o[6] = wp.z;
    o[7] = wn.x; o[8] = wn.y; o[9] = wn.z;
    o[10] = t.x; o[11] = t.y; o[12] = wn.w;
  }
  __syncwarp();
  int n = active ? 3 : 0;
  float* src = A;
  float* dst = B;
#pragma unroll
  for (int plane = PW; plane <= NZ; plane++) {
    // a polygon with fewer than 3 vertices is dropped (its later planes are skipped)
    int m = 0;
    if (n >= 3) {
      for (int i = 0; i < n; i++) {
        const float* prev = src + (i == 0 ? n - 1 : i - 1) * kPolyStride;
        const float* curr = src + i * kPolyStride;
        const bool pin = inside_plane(prev, plane), cin = inside_plane(curr, plane);
        if (pin != cin && m < kMaxPoly) {
          const float t = intersect_ratio(prev, curr, plane);
          if (hl < kVaryings) dst[m * kPolyStride + hl] = fa(prev[hl], fm(fs(curr[hl], prev[hl]), t));
          m++;
        }
        if (cin && m < kMaxPoly) {
          if (hl < kVaryings) dst[m * kPolyStride + hl] = curr[hl];
          m++;
        }
      }
      n = m;
    }
    __syncwarp();
    float* tmp = src; src = dst; dst = tmp;
  }
  bool valid = false;
  RasterRec r;
  Payload pl;
  if (n >= 3 && hl < n - 2) {
    const float* p0 = src;
    const float* p1 = src + (hl + 1) * kPolyStride;
    const float* p2 = src + (hl + 2) * kPolyStride;
    const uint32_t seq = ((uint32_t)__ldg(&v.fv[face].w) << kSeqFaceShift) | ((uint32_t)hl << 1) | 1u;
    valid = build_rec(v, ndc_of(make_float4(p0[0], p0[1], p0[2], p0[3])), ndc_of(make_float4(p1[0], p1[1], p1[2], p1[3])),
                      ndc_of(make_float4(p2[0], p2[1], p2[2], p2[3])), seq, (uint32_t)view, r);
    if (valid) make_payload(v.shader, p0, p1, p2, pl);
  }
  int tx0, ty0, ntw, nt = 0;
  if (valid) rec_tiles(r, T, tx0, ty0, ntw, nt);
  const bool big = valid && nt > kMaxRecordTiles;
  const int nf4 = payload_f4(v.shader);
  const uint32_t slot = rec_base + warp_reserve(valid && !big, &sc.ctl->rec_extra);
  append_small(valid && !big, slot, r, pl, nf4, v, T, sc);
  if (valid && !big && slot < sc.rec_cap) pay_bytes += 16u * (uint32_t)nf4;
  const uint32_t bslot = warp_reserve(big, &sc.ctl->big_count);
  if (big) queue_big(bslot, r, pl, nf4, T, sc);
  __syncwarp();
}

// Emit pass over the records of k_setup (dense: one thread per surviving triangle): the
// shading payload, the tile counts, and the hand-over of huge triangles to k_scan (their
// slot becomes a hole the binning skips).  Grid-stride with warp-uniform trip counts, so
// the warp collectives of append_counts see every lane.
__device__ __forceinline__ void emit_records(const DView* views, int T, const Scratch& sc, uint32_t block,
                                             uint32_t nblocks) {
  const int lane = threadIdx.x & 31;
  const uint32_t nrec = min(sc.ctl->rec_count, sc.rec_cap);
  const uint32_t stride = nblocks * blockDim.x;
  uint32_t pay_bytes = 0;  // payload bytes this lane wrote for the raster (split ones: k_scan)
  float box_px = 0.f;      // pixels of its records' bounding boxes
  for (uint32_t i0 = block * blockDim.x + (threadIdx.x & ~31u); i0 < nrec; i0 += stride) {
    const uint32_t i = i0 + (uint32_t)lane;
    bool valid = false;
    RasterRec r;
    Payload pl;
    int nf4 = 0;
    const DView* v = views;
    if (i < nrec) {
      // the words this pass needs (the face, and seq, view, pixel range in the last 16 bytes); the
      // whole record only for a huge triangle.  Every record below rec_count is the
      // cull pass's: the clipper's and the sub-records come behind it.
      const uint4 a = *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(&sc.recs[i]) + 48);
      const int f = (int)sc.recs[i].face;
      r.seq = a.x; r.view = a.y; r.xr = a.z; r.yr = a.w;
      valid = true;
      v = views + (r.view & kRecViewMask);
      nf4 = payload_f4(v->shader);
      if (nf4 > 0) {
        face_payload(*v, f, nf4, __ldg(&v->fv[f]), pl);
      }
    }
    int tx0, ty0, ntw, nt = 0;
    if (valid) {
      rec_tiles(r, T, tx0, ty0, ntw, nt);
      box_px += (float)(((r.xr >> 16) - (r.xr & 0xffffu) + 1u) * ((r.yr >> 16) - (r.yr & 0xffffu) + 1u));
    }
    const bool big = valid && nt > kMaxRecordTiles;
    const bool small = valid && !big;
    if (small) {
      pay_bytes += 16u * (uint32_t)nf4;
    }
    append_counts(small, i, r, pl, nf4, *v, T, sc, true);
    const uint32_t bslot = warp_reserve(big, &sc.ctl->big_count);
    if (big) {
      r = sc.recs[i];
      sc.recs[i].view = r.view | (kRecHole << kRecFlagShift);
      queue_big(bslot, r, pl, nf4, T, sc);
    }
  }
  // one atomic of each a block on the control block's line, which serves them one by one (a warp
  // each: 26 -> 32 us in a 1920x1080 frame of 120k faces; now 24.6)
  __shared__ uint32_t s_pay[kEmitThreads / 32];
  __shared__ float s_box[kEmitThreads / 32];
  pay_bytes = __reduce_add_sync(kFull, pay_bytes);
#pragma unroll
  for (int o = 16; o; o >>= 1) box_px += __shfl_down_sync(kFull, box_px, o);
  if (lane == 0) {
    s_pay[threadIdx.x >> 5] = pay_bytes;
    s_box[threadIdx.x >> 5] = box_px;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long pay = 0;
    float box = 0.f;
    for (int w = 0; w < kEmitThreads / 32; w++) {
      pay += s_pay[w];
      box += s_box[w];
    }
    if (pay) atomicAdd(&sc.ctl->pay_bytes, pay);
    if (box > 0.f) atomicAdd(&sc.ctl->box_px, box);
  }
}

// The clip queue of k_setup, two faces per warp: warp w of the grid begins with pair w, and where
// there are more pairs than warps claims the next one while it works on one (a fixed order
// leaves some warps with the faces that make many triangles: 65k faces 100 us, claimed 88 us;
// without claims and their round trip a short queue saves 2-8 us).  Each face is a chain of
// dependent loads, so resident warps set the throughput.
__device__ __forceinline__ void clip_queue(const DView* views, int T, const Scratch& sc, uint32_t block,
                                           uint32_t nblocks) {
  __shared__ float poly[kEmitThreads / 32][2][2][kMaxPoly * kPolyStride];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4;
  const uint32_t nclip = min(sc.ctl->clip_count, sc.clip_cap);
  const uint32_t rec_base = sc.ctl->rec_count;  // the cull pass's records come first
  uint32_t pay_bytes = 0;  // payload bytes this lane wrote, added to the control block once (its line
                           // serves one atomic at a time, the record slots' among them)
  const uint32_t claimed = 2u * nblocks * (kEmitThreads / 32);  // pairs from here on are claimed
  uint32_t item = 2u * (block * (kEmitThreads / 32) + (uint32_t)warp);
  while (item < nclip) {
    uint32_t next = nclip;
    if (lane == 0 && claimed < nclip) next = claimed + atomicAdd(&sc.ctl->post_next, 2u);
    const uint32_t mine = item + (uint32_t)half;
    const bool active = mine < nclip;
    const int2 vf = active ? sc.clipq[mine] : make_int2(0, 0);
    clip_face(active, views[vf.x], vf.x, vf.y, T, sc, poly[warp][half][0], poly[warp][half][1], rec_base, pay_bytes);
    item = __shfl_sync(kFull, next, 0);
  }
  pay_bytes = __reduce_add_sync(kFull, pay_bytes);
  if (lane == 0 && pay_bytes) atomicAdd(&sc.ctl->pay_bytes, (unsigned long long)pay_bytes);
}

// Emit and clip both read what k_setup left and append independently (the clipper's records go
// behind the cull pass's, counted apart).  CLIP: one grid, whose first `clip_blocks` blocks clip
// while the others emit; otherwise the grid emits, and k_post clips after it.
template <bool CLIP>
__global__ void __launch_bounds__(kEmitThreads, 4) k_emit(const DView* views, int T, Scratch sc,
                                                          int clip_blocks) {
  chain_wait();
  // as one block: another block of this grid may set the word meanwhile, and the blocks that emit meet
  // at a barrier
  if (__syncthreads_or((sc.ctl->error & kErrCapacity) != 0u)) return;
  if (CLIP && (int)blockIdx.x < clip_blocks) {
    clip_queue(views, T, sc, blockIdx.x, (uint32_t)clip_blocks);
    return;
  }
  const uint32_t first = CLIP ? (uint32_t)clip_blocks : 0u;
  emit_records(views, T, sc, blockIdx.x - first, gridDim.x - first);
}

__global__ void __launch_bounds__(kEmitThreads, 3) k_post(const DView* views, int T, Scratch sc) {
  chain_wait();
  if (sc.ctl->error & kErrCapacity) return;
  clip_queue(views, T, sc, blockIdx.x, gridDim.x);
}

// For a small sequence the shorter chain counts: one grid saves a launch and the clipper's latency
// (whole calls: 1000x600 with shadow, 10k faces, 158 -> 150 us; 1080p frame, 655k faces, 360 -> 352
// us).  For a large one the clipper's registers and shared memory cost the emit pass more than the
// overlap gains (16 views, 2.4M faces: equal; 4M-triangle soup 68 + 22 -> 90 us; 64 requests, 40M
// faces, 401 + 84 -> 565 us).
constexpr size_t kOneGridFaces = (size_t)1 << 21;
bool clips_with_emit(size_t faces) { return faces <= kOneGridFaces; }

int launch_emit(const DView* views, int tile, Scratch sc, bool clip, int num_sms, cudaStream_t s) {
  const int clip_blocks = clip ? num_sms * 2 : 0, grid = clip_blocks + num_sms * 8;
  return clip ? launch_chained(k_emit<true>, grid, kEmitThreads, 0, s, views, tile, sc, clip_blocks)
              : launch_chained(k_emit<false>, grid, kEmitThreads, 0, s, views, tile, sc, clip_blocks);
}

int launch_post(const DView* views, int tile, Scratch sc, int grid, cudaStream_t s) {
  return launch_chained(k_post, grid, kEmitThreads, 0, s, views, tile, sc);
}

// A small sequence's cull pass transforms the corners itself: each vertex about six times, but the
// vertex stage's launch and its write and read of the screen vertices are saved (whole calls: 2,048
// faces 68.6 -> 65.9 us, 5,120 faces 81 -> 77.5, 262,144 faces 181 -> 179.5; 655,364 faces equal).
// So does a large one with a position a face or more, where a vertex serves three corners or
// fewer (vertex + cull of 4M faces with 3 positions each 176 -> 133 us, with 1.5 144 -> 127, with
// 1.06 134 -> 123; closed meshes have half a position a face: 64 requests 793 -> 1,000 us).
constexpr size_t kOwnVertexFaces = (size_t)1 << 18;
bool culls_own_vertices(size_t faces, size_t positions) { return faces <= kOwnVertexFaces || positions >= faces; }

int launch_setup(const DView* views, int nviews, int nchunks, bool own_vertices, Scratch sc, int grid, cudaStream_t s) {
  if (nchunks <= 0) return 0;
  const int g = std::max(1, std::min(grid, nchunks));
  return own_vertices ? launch_chained(k_setup<true>, g, kSetupThreads, 0, s, views, nviews, nchunks, sc)
                      : launch_chained(k_setup<false>, g, kSetupThreads, 0, s, views, nviews, nchunks, sc);
}

}  // namespace hsr
