// kernels_raster.cu — persistent per-tile raster + resolve + shade (sm_103a).
//
// Reference: rasterize_triangle (graphics.cpp:314-376).  The reference walks triangles in
// submission order and, per pixel of the bounding box, keeps a fragment when
// `!(frag_depth > depth)`.  With finite depths that sequential loop leaves, per pixel, the
// fragment of minimum depth, and among equal minima the LAST submitted one; a previous
// buffer depth equal to that minimum loses.  Fragment depths are never -0 or NaN
// (interpolate_depth starts from +0), so the order-independent rule
//     min over (depth, later-submitted)
// with the buffer's depth as the weakest entry reproduces the loop exactly, whatever
// order the tile lists hold.  All shaders return `discard = false` and have no side
// effects (IShader.cpp:14,38,56,76,108,161,179), so shading only the winner equals
// shading every passing fragment in order.
//
// Coverage.  barycentric() (graphics.cpp:222-233) divides by u.z three times per pixel.
// With u = (ux, uy, uz) and s = ux + uy (all rounded exactly as there),
//     1 - s/uz < 0  <=>  s/uz rounds above 1  <=>  s > uz (uz > 0) or s < uz (uz < 0),
//     uy/uz < 0     <=>  uy != 0 with the opposite sign of uz (no underflow to -0),
// so the test needs no division.  The equivalence holds when nonzero |ux|, |uy| cannot
// underflow after the division; setup marks records outside that range (kRecExact) and
// those evaluate the reference's divisions literally.  Covered pixels then compute the
// three IEEE quotients for the depth.
#include <float.h>

#include "hsr_device.cuh"
#include "hsr_launch.cuh"

namespace hsr {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kNone = 0xffffffffu;

// View owning tile t: the last view whose first tile is <= t (views hold consecutive tile
// ranges in batch order).  `tbase` is the shared copy when the batch has at most
// kSharedViews views, else null and the descriptors are searched in global memory.
__device__ __forceinline__ int find_view(const DView* views, const int32_t* tbase, int nviews, int t) {
  int lo = 0, hi = nviews - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((tbase ? tbase[mid] : views[mid].tile_base) <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Poll until *p reaches `need`.  Bounded: after the poll limit the wait sets kErrWaitTimeout and
// gives up, and once any wait of the sequence has given up the others stop waiting (so a
// dependency that never completes costs one limit, not one per tile).
__device__ __forceinline__ void wait_at_least(const Scratch& sc, const uint32_t* p, uint32_t need) {
  const long limit = sc.poll_limit > 0 ? (long)sc.poll_limit : kDepWaitPolls;
  long spins = 0;
  while (*reinterpret_cast<const volatile uint32_t*>(p) < need) {
    if (++spins > limit || (*reinterpret_cast<volatile uint32_t*>(&sc.ctl->error) & kErrWaitTimeout)) {
      atomicOr(&sc.ctl->error, kErrWaitTimeout);
      return;
    }
    __nanosleep(kPollNs);
  }
}

// Wait until the target that view `dep` is the last to write (a shadow map) is complete: every
// non-empty tile of that view and of the earlier views into the same target (its dep1 chain) is
// done; their empty tiles were cleared in the scatter grid, which runs before the raster.
// HSR_FAULT_DEPENDENCY_STALL makes the wait ask for one tile more than the view has.
__device__ __forceinline__ void wait_target(const Scratch& sc, const DView* views, int dep) {
  for (int d = dep; d >= 0; d = views[d].dep1) {
    const int tb = views[d].tile_base;
    const uint32_t need = sc.ne_off[tb + views[d].ntiles] - sc.ne_off[tb] +
                          ((sc.faults & HSR_FAULT_DEPENDENCY_STALL) ? 1u : 0u);
    wait_at_least(sc, &sc.view_done[d], need);
  }
  __threadfence();
}

// Wait for tile `lt` of the earlier views into this view's target.  Views of one target share their
// tile grid and a tile reads no pixel but its own, so the last of them that has records there is
// the only one to wait for (it waited for those before it).  A finished tile's fill cursor, spent
// after the binning, holds kTileDone (HSR_FAULT_DEPENDENCY_STALL withholds it).
constexpr uint32_t kTileDone = 0xffffffffu;
__device__ __forceinline__ void wait_tile(const Scratch& sc, const DView* views, int dep, int lt) {
  for (int d = dep; d >= 0; d = views[d].dep1) {
    const int t = views[d].tile_base + lt;
    if (sc.tile_count[t] == 0u) continue;
    wait_at_least(sc, &sc.tile_fill[t], kTileDone);
    break;
  }
  __threadfence();
}

// Ordered bits of a float: unsigned order equals float order (-inf < ... < -0 < +0 < ... < +inf).
__device__ __forceinline__ uint32_t ord_bits(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ord(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
// Key of the depth already in the buffer: it loses every tie (low word above any fragment's),
// -0 compares equal to +0 as `frag_depth > depth` does, NaN admits every fragment.
__device__ __forceinline__ unsigned long long buffer_key(float d) {
  if (d == 0.f) d = 0.f;
  if (d != d) d = __int_as_float(0x7f800000);
  return ((unsigned long long)ord_bits(d) << 32) | 0xffffffffull;
}

// The non-empty records of one batch of a tile list, compacted.  A candidate reads three 16-byte
// entries (consecutive records are consecutive entries, so a quarter-warp's loads of different
// records fall in different banks).
struct __align__(16) BatchRecs {
  float4 a4[32];       // ax, ay, e1x, e1y (edges signed so that u.z > 0)
  float4 b4[32];       // e2x, e2y, u.z of the sign test (NaN with kRecExact: never passes), u.z
  int4 m4[32];         // candidate -> pixel: see pixel_of
  float4 d4[32];       // screen depths d0, d1, d2 of the corners, submission order (bits)
  uint32_t ri[32];     // record index (also the index of its payload)
  uint32_t first[32];  // a bit per remainder candidate: set where a record's candidates begin
};

// Ordered bits of a depth no fragment of the record lies below (0: unknown).  interpolate_depth
// (graphics.cpp:186-194) sums d_k b_k with weights that a covered pixel has >= 0 and that add up to
// 1 within 4 units of 2^-24 (b0 = 1 - s / uz, b1 + b2 = s / uz, each operation rounded once), itself
// with five roundings; so for depths >= 2^-100, where what the products lose by underflow does not
// count, no sum is below (1 - 2^-20) times the smallest.  The literal divisions (kRecExact) may
// underflow, and NaN compares false: no bound.
__device__ __forceinline__ uint32_t lowest_depth(const RasterRec& r) {
  const bool known = r.d0 >= 0x1p-100f && r.d1 >= 0x1p-100f && r.d2 >= 0x1p-100f &&
                     !((r.view >> kRecFlagShift) & kRecExact);
  return known ? ord_bits(fm(fminf(fminf(r.d0, r.d1), r.d2), 0x1.ffffep-1f)) : 0u;
}
// Candidates per pixel of the visited tiles (the records' bounding boxes, added up by the emit pass)
// from which covered candidates are tested against lowest_depth before they are queued (HIDE): a
// shared load and a compare a candidate, which save the divisions and the atomic of the hidden
// ones.  Raster without and with the test, soups in 1920x1080 by candidates a pixel, tile 8 | 16:
//    5.6   86 -> 89 us  |  88 ->  88          20.7  197 -> 168 us | 240 -> 199
//    7.3  102 -> 102    | 113 -> 110          61    447 -> 332    | 559 -> 408
//   14.2  154 -> 143    | 180 -> 160         205  1,417 -> 963    | 1,700 -> 1,153
// So the two are equal at 7 or a little below, and 10 leaves meshes out (about 3 a pixel), where nearly
// every covered candidate wins when it is tested (64 requests 1,730 -> 1,786 us).  The 4M-triangle
// soup has 26: 784 -> 666 us.
constexpr float kHideCandidates = 10.f;

// Pixel of candidate i: q = i - m.x counts a record's range in row-major order, width w;
// m.y = ceil(65536 / w) divides by w (q < 1024, w <= 32), m.z = (first pixel) - m.x, m.w = T - w.
__device__ __forceinline__ int pixel_of(int4 m, int i) {
  const int row = (int)(((uint32_t)(i - m.x) * (uint32_t)m.y) >> 16);
  return i + m.z + row * m.w;
}

// Covered candidates waiting for their weights, depth and visibility update (a ring of 64 per
// warp): the cross products (u.x, u.y) of barycentric() and the record | pixel << 5.  The
// coverage pass fills it at the rate candidates are tested; the weights' three divisions and
// the depth test then run on full warps of covered candidates.
struct CandQueue {
  float2 u[64];
  uint16_t jp[64];
};

// Per-warp tile state in shared memory: per pixel the key (ordered depth | submission) and
// the index of the record that holds it, which is also the index of its payload.  8x8 tiles
// also keep the winner's barycentric weights (24 bytes a pixel in all), so shading reads no
// record; 16x16 and 32x32 tiles keep 12 bytes a pixel and the weights in the warp's stash.
template <int NPIX>
struct TileState {
  static constexpr bool kKeep = NPIX <= 64;
  uint32_t z[NPIX];  // the key's upper half
  uint2 win[NPIX];   // its lower half, the record (one store a winner)
  __device__ __forceinline__ unsigned long long key(int p) const { return ((unsigned long long)z[p] << 32) | win[p].x; }
  float b0[kKeep ? NPIX : 1], b1[kKeep ? NPIX : 1], b2[kKeep ? NPIX : 1];
};

// Everything one raster CTA keeps in shared memory, in one dynamically sized block (a 32x32
// tile needs more than the 48 KB of static shared memory; the launch opts in above that).
template <int T, int WARPS>
struct RasterSmem {
  TileState<T * T> st[WARPS];
  BatchRecs br[WARPS];
  CandQueue cq[WARPS];
  float u8f[256];
  int32_t tbase[kSharedViews];
  // pixels shaded and candidates covered in each warp's tiles, added to the control block once a CTA:
  // its counters share a line with the claim, and atomics on one line are served one by one (two a
  // tile besides the claim made the claim a quarter of the time with 8x8 tiles: 2560x1440
  // close-up 127 -> 108 us, 1280x720 grid 106 -> 86 us)
  unsigned long long shaded[WARPS], frags[WARPS];
  uint32_t done[WARPS];  // finished tiles of the warp's view not yet counted in view_done
  uint32_t claim;  // list position of the tile the CTA shares
};

// Shade the winners of one tile and write colour, depth and prim id (fused clear writes the
// clear values where nothing won).  S is the shader, known at compile time.  Without kept
// weights (16x16 and 32x32 tiles) the winner's weights come from the warp's stash in global
// memory (written by the visibility pass, read back from L2), or, with no stash, are evaluated
// again from its record: the same operations on the same values as in the visibility pass
// either way, so the same bits.
//
// The warp shades the rows of 32 pixels q0, q0 + qstep, ...; `by_warp` (a tile shared by a CTA) gives
// the warp whose stash holds each winner's weights, relative to the one `stash` belongs to.

// The first and the last sector of the payload floats a shader reads, into L1.
template <int NF4>
__device__ __forceinline__ void prefetch_payload(const Payload* p) {
  if constexpr (NF4 > 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
  if constexpr (NF4 > 2) asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(p) + 16 * (NF4 - 1)));
}
template <int T, int S>
__device__ __forceinline__ uint32_t shade_tile(const DView& v, const Scratch& sc, const TileState<T * T>& st, int ox,
                                               int oy, bool clear, const ByteTables& bt, const float* stash, int q0,
                                               int qstep, const uint32_t* by_warp) {
  constexpr int PPL = T * T / 32;
  constexpr int NF4 = payload_f4_of<S>();
  const int lane = threadIdx.x & 31;
  uint32_t shaded = 0;
  // (the compiler reads a descriptor's field again after a store: 64 requests 1,554 -> 1,567 us)
  const int W = v.W, H = v.H;
  uint32_t* const color = v.color;
  float* const depth = v.depth;
  uint32_t* const prims = v.prim;
#pragma unroll 1
  for (int q = q0; q < PPL; q += qstep) {
    // the next row's payloads start on their way to L1 while this row is shaded (a whole tile's at
    // once push each other out: 64 requests at tile 16 raster 1,745 -> 1,716 us, and 1,760 then)
    if (NF4 > 0 && q + qstep < PPL) {
      const uint32_t rn = st.win[lane + 32 * (q + qstep)].y;
      if (rn != kNone) prefetch_payload<NF4>(&sc.pay[rn]);
    }
    const int p = lane + 32 * q;
    const int x = ox + p % T, y = oy + p / T;
    if (x >= W || y >= H) continue;
    const size_t idx = (size_t)y * W + x;
    uint32_t ri = st.win[p].y;
    // without the fused clear the buffer's depth enters here, after the fragments' minimum
    if (!clear && ri != kNone && st.key(p) >= buffer_key(__ldcg(&depth[idx]))) ri = kNone;
    if (ri != kNone) {
      shaded++;
      float b0, b1, b2;
      uint32_t pay, seq;
      // a record's payload index is its own index, and the winner's submission is the low word of
      // its key: the payload's loads wait for nothing but the record index
      if constexpr (TileState<T * T>::kKeep) {
        b0 = st.b0[p]; b1 = st.b1[p]; b2 = st.b2[p];
        pay = ri;
        seq = 0xfffffffeu - st.win[p].x;
      } else if (stash) {
        pay = ri;
        seq = 0xfffffffeu - st.win[p].x;
        const float* from = by_warp ? stash + (size_t)by_warp[p] * (size_t)stash_floats(T) : stash;
        const float4 w = __ldcg(reinterpret_cast<const float4*>(from) + p);
        b0 = w.x; b1 = w.y; b2 = w.z;
      } else {
        const RasterRec r = sc.recs[ri];
        cover_test(r.ax, r.ay, r.e1x, r.e1y, r.e2x, r.e2y, r.uz, ((r.view >> kRecFlagShift) & kRecExact) != 0u,
                   (float)x, (float)y, b0, b1, b2);
        pay = ri;
        seq = r.seq;
      }
      float P[NF4 > 0 ? NF4 * 4 : 4];
      if constexpr (NF4 > 0) {
        const float4* src = reinterpret_cast<const float4*>(&sc.pay[pay]);
#pragma unroll
        for (int k = 0; k < NF4; k++) reinterpret_cast<float4*>(P)[k] = src[k];
      }
      const uint32_t prim = v.prim_base + (seq >> kSeqFaceShift) + 1u;
      const uint32_t alpha = clear ? v.clear_rgba : __ldcg(&color[idx]);
      color[idx] = pack_rgb(fragment_s<S>(v, P, b0, b1, b2, prim, bt), alpha);
      if (depth) depth[idx] = from_ord(st.z[p]);
      if (prims) prims[idx] = prim;
    } else if (clear) {
      color[idx] = v.clear_rgba;
      if (depth) depth[idx] = v.clear_depth;
      if (prims) prims[idx] = 0u;
    }
  }
  return shaded;
}

// One warp per non-empty screen tile (k_scan lists them in tile order; the scatter grid has
// cleared the others).  For each batch of 32 records of the tile list, every record's
// bounding-box pixels inside the tile form a run of candidates; the non-empty runs are
// compacted, and the lanes walk the candidates 32 at a time, so the work is proportional to the
// pixels the triangles can touch rather than to records x 32 lanes: first the whole windows of
// 32 of each record, then the remainders laid end to end (warp prefix sum), where the record
// owning a candidate is found from a bit set at each record's first one.  A covered candidate
// resolves visibility by the smallest key
//     (ordered depth << 32) | (0xfffffffe - seq)
// in shared memory: smallest depth first, and among equal depths the later submission.
// The halves are separate words: a 32-bit atomicMin on the depth decides nearly all, and only
// where a depth is met again does a second one decide on the submission (64-bit shared atomics
// took 14 of the load/store unit's cycles a warp; raster of the 4M-triangle soup 669 -> 654 us,
// 16 recorded views 306 -> 301 us, 64 requests 1,718 -> 1,708 us).
// The lane whose key is then the minimum records the winner's record (two lanes of one step
// never hold the same key: one triangle covers a pixel once).  Shading then runs once per pixel
// with a winner.
//
// A view's tiles start their coverage at once; only shading waits for what it reads of other
// views (the shadow map; in a draw without the fused clear the depth and alpha that earlier
// draws left at this tile).
//
// SHARED: a whole CTA takes one tile.  Each warp rasterises an equal share of the tile's list
// into a tile state of its own, the states are merged by the smaller key (the order of the list
// never matters), and the pixel rows are shaded by the warps in turn.
// HIDE: see kHideCandidates.
template <int T, int WARPS, bool SHARED, bool HIDE>
__device__ __forceinline__ void raster_tiles(const DView* views, const Scratch& sc,
                                             RasterSmem<T, WARPS>& sm, const int32_t* tbase, uint32_t nlist,
                                             const uint32_t* tile_list) {
  constexpr int NPIX = T * T;
  constexpr int PPL = NPIX / 32;
  constexpr bool kKeep = TileState<NPIX>::kKeep;
  const ByteTables bt{sm.u8f};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  TileState<NPIX>& st = sm.st[warp];
  BatchRecs& br = sm.br[warp];
  CandQueue& cq = sm.cq[warp];
  float* stash = nullptr;
  if constexpr (!kKeep) {
    const uint32_t gw = blockIdx.x * (uint32_t)WARPS + (uint32_t)warp;
    if (sc.stash && gw < sc.stash_warps) stash = sc.stash + (size_t)gw * (size_t)stash_floats(T);
  }
  const uint32_t nrec = min(sc.ctl->rec_count + sc.ctl->rec_extra, sc.rec_cap);

  // The non-empty tiles are handed out by one counter over their list, each when its warp is ready
  // for it: the list is in tile order and dependencies only point to lower tile indices, so
  // nobody waits for a tile that is not yet being drawn.  (Claimed two tiles ahead, to hide the
  // counter and the lists, tiles lay with warps that were busy or waiting while others were done
  // or waited for them: 64 requests 1,705 -> 1,523 us, six objects 135 -> 92, 16 views 301 -> 272,
  // 1080p frame 184 -> 166, the 4M-triangle soup 653 -> 600.  To claim one before the shading
  // waits gave half of that.)
  const uint32_t ntiles = (uint32_t)sc.ntiles;
  const uint32_t lane_magic = (65536u + (uint32_t)lane) / ((uint32_t)lane + 1u);  // ceil(65536 / (lane + 1))
  const uint32_t upto = (2u << lane) - 1u;  // this lane and those below
  uint32_t li = 0;  // position in the list
  if (SHARED) {
    if (threadIdx.x == 0) sm.claim = atomicAdd(sc.claim, 1u);
    __syncthreads();
    li = sm.claim;
  } else {
    if (lane == 0) li = atomicAdd(sc.claim, 1u);
    li = __shfl_sync(kFull, li, 0);
  }
  uint32_t t = li < nlist ? tile_list[li] : ntiles;
  uint32_t n = 0, off = 0;
  if (t < ntiles) {
    n = sc.tile_count[t];
    off = sc.tile_off[t];
  }
  // views of a warp's tiles only move forward: after the first, search on from the last one
  int vi = t < ntiles ? find_view(views, tbase, sc.nviews, (int)t) : 0;
  if (lane == 0) sm.done[warp] = 0u;
  uint32_t ri_ahead = !SHARED && (uint32_t)lane < n ? sc.bins[off + (uint32_t)lane] : kNone;
  int ready = -1;  // the shadow map's view last seen complete
  for (;;) {
    if (t >= ntiles) break;
    uint32_t t_next = ntiles, n_next = 0, off_next = 0;
    const DView& v = views[vi];
    const int lt = (int)t - v.tile_base;
    const int tx = lt % v.tiles_x, ty = lt / v.tiles_x;
    const int ox = tx * T, oy = ty * T;
    const bool clear = (v.flags & HSR_DRAW_CLEAR) != 0u;

    // this warp's records: all of the tile's list, or its share of it
    uint32_t b = 0, end = n;
    if (SHARED) {
      b = share_begin(n, (uint32_t)warp, WARPS);
      end = share_begin(n, (uint32_t)warp + 1u, WARPS);
    }
    {  // every pixel starts from the clear depth, or from nothing where the buffer's is read later
      const unsigned long long k0 = clear ? buffer_key(v.clear_depth) : ~0ull;
#pragma unroll 8
      for (int q = 0; q < PPL; q++) {
        st.z[lane + 32 * q] = (uint32_t)(k0 >> 32);
        st.win[lane + 32 * q] = make_uint2((uint32_t)k0, kNone);
      }
    }
    const uint32_t share = b;
    uint32_t frags = 0;  // covered candidates (warp-uniform)
    for (; b < end; b += 32) {
      const uint32_t cnt = min(32u, end - b);
      uint32_t c = 0, w = 1, ri = ri_ahead;
      int p0 = 0;  // the first pixel of the record's range in the tile
      RasterRec rr;
      if ((uint32_t)lane < cnt) {
        // the tile's first indices came with the tile before, later ones of a 16x16 or 32x32 tile (many
        // batches) during the batch before
        if (SHARED ? (kKeep || b == share) : (kKeep && b > 0u)) ri = sc.bins[off + b + (uint32_t)lane];
        if (ri < nrec) {  // an index past the records never comes from a consistent bin pass
          rr = sc.recs[ri];
          const int lx0 = max((int)(rr.xr & 0xffffu) - ox, 0), lx1 = min((int)(rr.xr >> 16) - ox, T - 1);
          const int ly0 = max((int)(rr.yr & 0xffffu) - oy, 0), ly1 = min((int)(rr.yr >> 16) - oy, T - 1);
          if (lx0 <= lx1 && ly0 <= ly1) {
            w = (uint32_t)(lx1 - lx0 + 1);
            c = w * (uint32_t)(ly1 - ly0 + 1);
            p0 = ly0 * T + lx0;
          }
        }
      }
      // whole windows of 32 candidates of one record are walked record by record; the
      // remainders (at most 31 a record) are laid end to end and share windows.  The pass is
      // issue-bound (73 % issue active, 87 of about 130 warp instructions a window went into
      // finding each candidate's owner, its pixel and the sign tests), so this counts slots:
      // raster of the 4M-triangle soup at tile 16 1,024 -> 817 us, the 1080p frame at tile 8
      // 253 -> 219 us, 64 served requests 1,835 -> 1,744 us.
      const uint32_t whole = c & ~31u, rest = c & 31u;
      uint32_t incl = rest;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
      }
      const int W = (int)__shfl_sync(kFull, incl, 31);
      const uint32_t start = incl - rest;
      const unsigned ne = __ballot_sync(kFull, rest > 0u);
      unsigned big = __ballot_sync(kFull, whole > 0u);
      const unsigned exact = __ballot_sync(kFull, c > 0u && ((rr.view >> kRecFlagShift) & kRecExact) != 0u);
      const int magic = (int)__shfl_sync(kFull, lane_magic, (int)w - 1);
      // records with a remainder come first, in order; those without fill the entries behind them
      const int k = rest > 0u ? __popc(ne & (upto >> 1)) : __popc(ne) + __popc((big & ~ne) & (upto >> 1));
      br.first[lane] = 0u;
      __syncwarp();
      if (c > 0u) {
        // u.z made positive: the edges negated turn every cross product and u.z into their exact
        // negatives, so the decisions and the quotients stay the same (a zero weight may change
        // its sign, which no depth, colour or comparison shows: each is a sum with a nonzero
        // term or one that starts from +0)
        const uint32_t sg = __float_as_uint(rr.uz) & 0x80000000u;
        auto flip = [sg](float f) { return __uint_as_float(__float_as_uint(f) ^ sg); };
        const float uz = fabsf(rr.uz);
        br.a4[k] = make_float4(rr.ax, rr.ay, flip(rr.e1x), flip(rr.e1y));
        br.b4[k] = make_float4(flip(rr.e2x), flip(rr.e2y),
                               ((rr.view >> kRecFlagShift) & kRecExact) ? __int_as_float(0x7fffffff) : uz, uz);
        const int base = (int)start - (int)whole;  // candidate number of the record's first pixel
        br.m4[k] = HIDE ? make_int4(base, magic | ((T - (int)w) << 20), p0 - base, (int)lowest_depth(rr))
                        : make_int4(base, magic, p0 - base, T - (int)w);
        br.d4[k] = make_float4(rr.d0, rr.d1, rr.d2, __uint_as_float(rr.seq));
        br.ri[k] = ri;
        if (rest > 0u) atomicOr(&br.first[start >> 5], 1u << (start & 31u));
      }
      __syncwarp();
      if (!kKeep && b + 32u + (uint32_t)lane < end) ri_ahead = sc.bins[off + b + 32u + (uint32_t)lane];
      // Visibility of `cnt` queued candidates from the ring head, one per lane: weights
      // (the divisions of barycentric()), depth, and the smaller key.
      uint32_t qh = 0, qn = 0;  // ring head and queued count (warp-uniform)
      auto resolve = [&](uint32_t cnt) {
        __syncwarp();
        const bool act = (uint32_t)lane < cnt;
        uint32_t z = 0u, order = 0u, old = 0u;
        int p = 0, j = 0;
        float b0 = 0.f, b1 = 0.f, b2 = 0.f;
        if (act) {
          const uint32_t e = (qh + (uint32_t)lane) & 63u;
          const uint32_t jp = cq.jp[e];
          j = (int)(jp & 31u);
          p = (int)(jp >> 5);
          const float2 u = cq.u[e];
          const float4 d4 = br.d4[j];
          cover_weights(u.x, u.y, br.b4[j].w, b0, b1, b2);
          // interpolate_depth (graphics.cpp:186-194)
          z = ord_bits(fa(fa(fa(0.f, fm(d4.z, b2)), fm(d4.y, b1)), fm(d4.x, b0)));
          order = 0xfffffffeu - __float_as_uint(d4.w);
          old = atomicMin(&st.z[p], z);
        }
        __syncwarp();
        bool wins = act && old >= z && st.z[p] == z;
        if (__any_sync(kFull, wins && old == z)) {  // an equal depth, here or in the buffer
          if (wins && old > z) st.win[p].x = 0xffffffffu;
          __syncwarp();
          if (wins) wins = atomicMin(&st.win[p].x, order) > order;
          __syncwarp();
          wins = wins && st.win[p].x == order;
        }
        if (wins) {
          st.win[p] = make_uint2(order, br.ri[j]);
          if constexpr (kKeep) {
            st.b0[p] = b0;
            st.b1[p] = b1;
            st.b2[p] = b2;
          } else if (stash) {
            __stcg(reinterpret_cast<float4*>(stash) + p, make_float4(b0, b1, b2, 0.f));
          }
        }
        qh = (qh + cnt) & 63u;
        qn -= cnt;
        __syncwarp();
      };
      // One window: candidate i of record j, counted when `in`.
      auto window = [&](int i, int j, bool in) {
        const float4 a4 = br.a4[j], b4 = br.b4[j];
        int4 m4 = br.m4[j];
        const uint32_t lowest = (uint32_t)m4.w;
        if (HIDE) {  // as laid out above
          m4.w = m4.y >> 20;
          m4.y &= 0xfffff;
        }
        const int p = pixel_of(m4, i);
        const float x = (float)(ox | (p & (T - 1))), y = (float)(oy + p / T);
        float ux, uy;
        bool covered = cover_terms_pos(a4.x, a4.y, a4.z, a4.w, b4.x, b4.y, b4.z, x, y, ux, uy) && in;
        if (exact && in && b4.z != b4.z) covered = cover_exact(ux, uy, b4.w);
        unsigned cm = __ballot_sync(kFull, covered);
        frags += (uint32_t)__popc(cm);
        if (HIDE) {  // leave out what cannot win any more
          covered = covered && lowest <= st.z[p];
          cm = __ballot_sync(kFull, covered);
        }
        if (covered) {  // queue behind the pending ones (at most 31 are pending here)
          const uint32_t e = (qh + qn + (uint32_t)__popc(cm & (upto >> 1))) & 63u;
          cq.u[e] = make_float2(ux, uy);
          cq.jp[e] = (uint16_t)(j | (p << 5));
        }
        qn += (uint32_t)__popc(cm);
        if (qn >= 32u) resolve(32u);
      };
      // whole windows: every lane works on the same record
      while (big) {
        const int src = __ffs(big) - 1;
        big &= big - 1u;
        const int j = __shfl_sync(kFull, k, src);
        const int first = __shfl_sync(kFull, (int)start - (int)whole, src);
        const int n32 = __shfl_sync(kFull, (int)whole, src);
        for (int q = 0; q < n32; q += 32) window(first + q + lane, j, true);
      }
      // remainders: the owner of a candidate is the last record beginning at or before it
      int before = -1;
      for (int base = 0; base < W; base += 32) {
        const uint32_t here = br.first[base >> 5];
        window(base + lane, before + __popc(here & upto), base + lane < W);
        before += __popc(here);
      }
      if (qn) resolve(qn);  // before the next batch replaces the runs the queue points to
    }
    if (lane == 0) {
      if (v.dep0 >= 0 && v.dep0 != ready) wait_target(sc, views, v.dep0);
      if (v.dep1 >= 0) wait_tile(sc, views, v.dep1, lt);
    }
    ready = v.dep0;
    __syncwarp();
    const TileState<NPIX>* win = &st;
    const float* wstash = stash;
    const uint32_t* by_warp = nullptr;
    int q0 = 0, qstep = 1;
    if (SHARED) {
      // merge into the first warp's state: the smaller key per pixel (equal keys are the same
      // buffer depth or the same triangle); the second state's depth words then hold the
      // winner's warp
      __syncthreads();
      for (int p = threadIdx.x; p < NPIX; p += WARPS * 32) {
        unsigned long long k = sm.st[0].key(p);
        int w = 0;
#pragma unroll
        for (int o = 1; o < WARPS; o++) {
          const unsigned long long ko = sm.st[o].key(p);
          if (ko < k) { k = ko; w = o; }
        }
        if (w) {
          sm.st[0].z[p] = sm.st[w].z[p];
          sm.st[0].win[p] = sm.st[w].win[p];
          if constexpr (kKeep) {
            sm.st[0].b0[p] = sm.st[w].b0[p];
            sm.st[0].b1[p] = sm.st[w].b1[p];
            sm.st[0].b2[p] = sm.st[w].b2[p];
          }
        }
        if constexpr (!kKeep) sm.st[1].z[p] = (uint32_t)w;
      }
      __syncthreads();
      win = &sm.st[0];
      q0 = warp;
      qstep = WARPS;
      if constexpr (!kKeep) {
        by_warp = sm.st[1].z;
        if (stash) wstash = stash - (size_t)warp * (size_t)stash_floats(T);
      }
    }
    uint32_t shaded = 0;
#define HSR_SHADE(S) shaded = shade_tile<T, S>(v, sc, *win, ox, oy, clear, bt, wstash, q0, qstep, by_warp); break
    switch (v.shader) {
      case HSR_SHADER_GROUND: HSR_SHADE(HSR_SHADER_GROUND);
      case HSR_SHADER_TOON: HSR_SHADE(HSR_SHADER_TOON);
      case HSR_SHADER_TEXTURE: HSR_SHADE(HSR_SHADER_TEXTURE);
      case HSR_SHADER_TEXTURE_WITH_LIGHT: HSR_SHADE(HSR_SHADER_TEXTURE_WITH_LIGHT);
      case HSR_SHADER_BLINN: HSR_SHADE(HSR_SHADER_BLINN);
      case HSR_SHADER_NORMALMAP: HSR_SHADE(HSR_SHADER_NORMALMAP);
      case HSR_SHADER_SHADOW: HSR_SHADE(HSR_SHADER_SHADOW);
      default: HSR_SHADE(HSR_SHADER_FLAT);
    }
#undef HSR_SHADE
    shaded = __reduce_add_sync(kFull, shaded);
    if (lane == 0) {
      sm.shaded[warp] += shaded;
      sm.frags[warp] += frags;
    }
    if (!SHARED) {
      if (lane == 0) li = atomicAdd(sc.claim, 1u);
      li = __shfl_sync(kFull, li, 0);
      if (li < nlist) {
        t_next = tile_list[li];
        n_next = sc.tile_count[t_next];
        off_next = sc.tile_off[t_next];
      }
    }
    // the next tile's view: at or behind this one
    auto view_of = [&](uint32_t tile) {
      if (tile >= ntiles) return -1;
      if (!tbase) return find_view(views, tbase, sc.nviews, (int)tile);
      int k = vi;
      while (k + 1 < sc.nviews && tbase[k + 1] <= (int)tile) k++;
      return k;
    };
    int vi_next = SHARED ? vi : view_of(t_next);
    if (v.has_dependents) {
      // publish this tile's writes before counting it done (a later view reads them); a warp counts
      // its tiles of a view at once when it leaves the view, which is when its last one is done
      if (lane == 0) sm.done[warp]++;
      if (SHARED || vi_next != vi || (v.has_dependents & kTileReaders)) {
        __threadfence();
        if (SHARED) __syncthreads(); else __syncwarp();
        if (SHARED ? threadIdx.x == 0 : lane == 0) {
          if (v.has_dependents & kTargetReaders) atomicAdd(&sc.view_done[vi], sm.done[warp]);
          if ((v.has_dependents & kTileReaders) && !(sc.faults & HSR_FAULT_DEPENDENCY_STALL))
            atomicExch(&sc.tile_fill[t], kTileDone);
          sm.done[warp] = 0u;
        }
      }
    }
    if (SHARED) {
      __syncthreads();  // the merged state and the claim word are free again
      if (threadIdx.x == 0) sm.claim = atomicAdd(sc.claim, 1u);
      __syncthreads();
      li = sm.claim;
      if (li < nlist) t_next = tile_list[li];
      if (t_next < ntiles) {
        n_next = sc.tile_count[t_next];
        off_next = sc.tile_off[t_next];
      }
      vi_next = view_of(t_next);
    }
    if (!SHARED) ri_ahead = (uint32_t)lane < n_next ? sc.bins[off_next + (uint32_t)lane] : kNone;
    t = t_next;
    n = n_next;
    off = off_next;
    vi = vi_next;
  }
}

// The list's tiles by warps, or (`shared`) by CTAs.  (The barrier between the two keeps the compiler from
// laying the loops out together, with 168 bytes of spills more for 8x8 tiles.)
template <int T, int WARPS, bool HIDE>
__device__ __forceinline__ void raster_list(const DView* views, const Scratch& sc, RasterSmem<T, WARPS>& sm,
                                            const int32_t* tbase, uint32_t nlist, bool shared, const uint32_t* list) {
  if (!shared) raster_tiles<T, WARPS, false, HIDE>(views, sc, sm, tbase, nlist, list);
  __syncthreads();
  if (shared) raster_tiles<T, WARPS, true, HIDE>(views, sc, sm, tbase, nlist, list);
}

// With few non-empty tiles most warps have none and the sequence lasts as long as its longest tile:
// up to kSharedTilesPerCta tiles per CTA of the grid, each CTA takes a tile (tile 8, one draw each:
// 91 tiles 24.6 -> 10.2 us, 1,026 tiles 32.8 -> 16.4 us, 1,369 tiles 34.8 -> 18.4 us; tile 16, 687
// tiles of a served request 98 -> 31 us).  Far more tiles keep every warp busy by themselves, and
// the barriers cost: the two are equal at about 10 tiles per CTA (86 us each at 10.6) and one
// warp per tile wins by 1.55x at 20 (113 against 176 us) and 1.7x at 47.
constexpr uint32_t kSharedTilesPerCta = 4;

// Four-warp CTAs are compiled for 7 per SM (72 registers a thread, fewer spills than at 8 per
// SM's 64: measured faster on the serving batches, 1.72 -> 1.65 ms).
template <int T, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 4 ? 7 : 32 / WARPS) k_raster(const DView* views, Scratch sc) {
  extern __shared__ __align__(16) unsigned char raster_smem[];
  RasterSmem<T, WARPS>& sm = *reinterpret_cast<RasterSmem<T, WARPS>*>(raster_smem);
  build_byte_tables(sm.u8f);
  if (threadIdx.x < WARPS) sm.shaded[threadIdx.x] = sm.frags[threadIdx.x] = 0ull;
  chain_wait();
  const int32_t* tbase = sc.nviews <= kSharedViews ? sm.tbase : nullptr;
  if (tbase)
    for (int i = threadIdx.x; i < sc.nviews; i += blockDim.x) sm.tbase[i] = views[i].tile_base;
  __syncthreads();
  if (!(sc.ctl->error & kErrNoDraw)) {
    // this launch's part of the list (all of it unless the sequence is drawn in groups)
    const uint32_t lo = sc.tile_lo > 0 ? sc.ne_off[sc.tile_lo] : 0u;
    const uint32_t nlist = sc.ne_off[sc.tile_hi] - lo;
    const uint32_t* list = sc.tile_list + lo;
    // uniform over the grid: every warp of every CTA has a stash, or none does
    const bool stashes = TileState<T * T>::kKeep || !sc.stash || gridDim.x * (uint32_t)WARPS <= sc.stash_warps;
    const bool shared = stashes && nlist <= kSharedTilesPerCta * gridDim.x;
    if (sc.ctl->box_px < kHideCandidates * (float)(T * T) * (float)sc.ctl->ne_tiles)
      raster_list<T, WARPS, false>(views, sc, sm, tbase, nlist, shared, list);
    else
      raster_list<T, WARPS, true>(views, sc, sm, tbase, nlist, shared, list);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long shaded = 0, frags = 0;
#pragma unroll
    for (int w = 0; w < WARPS; w++) {
      shaded += sm.shaded[w];
      frags += sm.frags[w];
    }
    if (shaded) atomicAdd(&sc.ctl->shaded_px, shaded);
    if (frags) atomicAdd(&sc.ctl->frag_px, frags);
    if (sc.ctl_out) {  // the sequence's last CTA hands the control block to the host
      __threadfence();
      if (atomicAdd(sc.finished, 1u) == gridDim.x - 1u) {
        __threadfence();
        const uint4* from = reinterpret_cast<const uint4*>(sc.ctl);
#pragma unroll
        for (int k = 0; k < (int)(sizeof(Ctl) / 16); k++) reinterpret_cast<uint4*>(sc.ctl_out)[k] = __ldcg(from + k);
        __threadfence_system();
      }
    }
  }
}

template <int T, int WARPS>
static int launch_t(const DView* views, Scratch sc, int grid, cudaStream_t s) {
  constexpr size_t smem = sizeof(RasterSmem<T, WARPS>);
  if (smem > 48 * 1024) {  // opt in to more than the default 48 KB of dynamic shared memory
    const cudaError_t e =
        cudaFuncSetAttribute(k_raster<T, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  return launch_chained(k_raster<T, WARPS>, grid, WARPS * 32, smem, s, views, sc);
}

int launch_raster(const DView* views, int tile, Scratch sc, int grid, int warps, cudaStream_t s) {
  if (warps != 4 && warps != 8) return (int)cudaErrorInvalidValue;
  switch (tile) {
    case 8: return warps == 4 ? launch_t<8, 4>(views, sc, grid, s) : launch_t<8, 8>(views, sc, grid, s);
    case 16: return warps == 4 ? launch_t<16, 4>(views, sc, grid, s) : (int)cudaErrorInvalidValue;
    case 32: return warps == 4 ? launch_t<32, 4>(views, sc, grid, s) : (int)cudaErrorInvalidValue;
    default: return (int)cudaErrorInvalidValue;
  }
}

}  // namespace hsr
