// kernels_bin.cu — tile binning (sm_103a).  The reference has no binning: it loops over
// each triangle's bounding box (graphics.cpp:349-375).  Here the (record, tile) pairs are
// laid out per tile so that one warp can own a tile in the raster.
//
// k_prep    the launch sequence's first kernel: view descriptors from the host's page-locked
//           staging, counters to zero.
// k_scan    sub-records of triangles that touch more than kMaxRecordTiles tiles, then exclusive
//           prefix sums of the per-tile counts and of the non-empty tiles, single pass with
//           decoupled look-back, and the list of non-empty tiles in tile order;
//           block order comes from a ticket so a block only waits on blocks that already
//           run, and every wait is bounded (error bit + give up, never a hang).
// k_scatter writes record indices into the per-tile lists with warp-aggregated atomics;
//           a record touches at most kMaxRecordTiles tiles (k_scan splits larger ones).
//           The same grid clears the tiles no record touches, streamed in row order.
#include <algorithm>

#include "hsr_device.cuh"
#include "hsr_launch.cuh"

namespace hsr {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;  // tiles per scan block
constexpr unsigned long long kFlagAgg = 1ull << 62;
constexpr unsigned long long kFlagPre = 2ull << 62;
constexpr unsigned long long kValMask = (1ull << 62) - 1;

__host__ __device__ __forceinline__ int scan_blocks_hd(int ntiles) { return (ntiles + kScanTile - 1) / kScanTile; }
int scan_blocks(int ntiles) { return scan_blocks_hd(ntiles); }

__device__ __forceinline__ unsigned long long ld_volatile64(const unsigned long long* p) {
  return *reinterpret_cast<const volatile unsigned long long*>(p);
}

// Scan word: bits 0-35 the count prefix, bits 36-61 the non-empty tile prefix, 62-63 the
// look-back flags.  Neither field can carry into the next: a batch has fewer than 2^26
// tiles (kMaxBatchTiles), and 2^36 (record, tile) pairs would need more records than the
// device memory holds (each record touches at most kMaxRecordTiles tiles).
constexpr int kCntBits = 36;
constexpr unsigned long long kCntMask = (1ull << kCntBits) - 1;
constexpr unsigned long long kOneTile = 1ull << kCntBits;

__device__ __forceinline__ unsigned long long scan_item(uint32_t count) {
  return (unsigned long long)count + (count ? kOneTile : 0ull);
}

// First kernel of a sequence: copies `copy` bytes of view descriptors from mapped host memory and
// clears `zero` bytes of counters (both multiples of 16).  One launch in place of a copy
// and a memset, which the kernels behind it could not overlap.
__global__ void __launch_bounds__(256) k_prep(const uint4* __restrict__ from, uint4* __restrict__ to, size_t copy,
                                              uint4* __restrict__ counters, size_t zero) {
  const size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  for (size_t i = i0; i < copy / 16; i += step) to[i] = __ldcv(from + i);
  for (size_t i = i0; i < zero / 16; i += step) counters[i] = make_uint4(0u, 0u, 0u, 0u);
}

int launch_prep(const void* from, void* to, size_t copy, void* counters, size_t zero, int max_grid, cudaStream_t s) {
  const size_t want = (std::max(copy, zero) / 16 + 255) / 256;
  const int grid = (int)std::min<size_t>(std::max<size_t>(want, 1), (size_t)max_grid);
  k_prep<<<grid, 256, 0, s>>>(static_cast<const uint4*>(from), static_cast<uint4*>(to), copy, static_cast<uint4*>(counters), zero);
  return (int)cudaGetLastError();
}

// A huge triangle's tile rectangle splits into sub-records over blocks of kSubTilesX x kSubTilesY
// tiles (same triangle constants and seq, pixel range clipped to the block, each with its own copy
// of the payload, since a record's payload index is its own index), and every tile of the
// rectangle is counted once.  The sub-ranges partition the triangle's pixel range, so each pixel is
// still tested exactly once.  `parts` warps share the triangle.  Every kStepsToBeat steps the warp counts up
// a word that the waiting blocks watch.
// (A warp and not a CTA each: most queued triangles have some tens of tiles, and what takes the time
// is the chain of loads from the queue to the view.)
constexpr uint32_t kStepsToBeat = 1024;  // a millisecond or so, whatever the triangle's size
__device__ __forceinline__ void split_triangle(const DView* views, int T, const Scratch& sc, const BigItem& bi,
                                               uint32_t first, int part, int parts) {
  const RasterRec b = bi.rec;
  const DView& v = views[b.view & kRecViewMask];
  int tx0, ty0, ntw, nt;
  rec_tiles(b, T, tx0, ty0, ntw, nt);
  const int nth = nt / ntw;
  const int nbx = (ntw + kSubTilesX - 1) / kSubTilesX;
  const int nsub = (int)sub_records(ntw, nth);
  const uint32_t base = first + b.pad;
  const int i0 = part * 32 + (int)(threadIdx.x & 31u), step = parts * 32;
  if ((uint64_t)base + (uint64_t)nsub > (uint64_t)sc.rec_cap) {
    if (i0 == 0) atomicOr(&sc.ctl->error, kErrRecOverflow);
    return;
  }
  uint32_t steps = 0;
  auto beat = [&] {  // (the first lane has the most steps)
    if ((++steps & (kStepsToBeat - 1u)) == 0u && (threadIdx.x & 31u) == 0u) atomicAdd(sc.split + 2, 1ull);
  };
  const int nf4 = payload_f4(v.shader);
  for (int k = i0; k < nsub * nf4; k += step, beat())
    reinterpret_cast<float4*>(&sc.pay[base + (uint32_t)(k / nf4)])[k % nf4] =
        reinterpret_cast<const float4*>(&bi.pay)[k % nf4];
  if (i0 == 0 && nf4) atomicAdd(&sc.ctl->pay_bytes, 16ull * (unsigned long long)(nf4 * nsub));
  const int x0 = (int)(b.xr & 0xffffu), x1 = (int)(b.xr >> 16);
  const int y0 = (int)(b.yr & 0xffffu), y1 = (int)(b.yr >> 16);
  for (int sidx = i0; sidx < nsub; sidx += step, beat()) {
    const int bx = sidx % nbx, by = sidx / nbx;
    const int stx0 = tx0 + bx * kSubTilesX, stx1 = min(tx0 + ntw - 1, stx0 + kSubTilesX - 1);
    const int sty0 = ty0 + by * kSubTilesY, sty1 = min(ty0 + nth - 1, sty0 + kSubTilesY - 1);
    RasterRec w = b;
    w.xr = (uint32_t)max(x0, stx0 * T) | ((uint32_t)min(x1, stx1 * T + T - 1) << 16);
    w.yr = (uint32_t)max(y0, sty0 * T) | ((uint32_t)min(y1, sty1 * T + T - 1) << 16);
    w.pad = 0u;
    store_rec(&sc.recs[base + (uint32_t)sidx], w);
  }
  for (int k = i0; k < nt; k += step, beat())
    atomicAdd(&sc.tile_count[v.tile_base + (ty0 + k / ntw) * v.tiles_x + tx0 + k % ntw], 1u);
}

// Sub-records of the queued huge triangles, then the scan, in one grid: blocks take tickets; where
// triangles are queued the first ones split them (up to kMaxParts warps each), and a scan block waits,
// bounded, until all are split, which only blocks with lower tickets do.  Most draws queue none and
// scan at once.
//
// A launch less and no wait where nothing is split, the look-back over 32 predecessors at a time (one
// per lane; it was one after the other) and a triangle split by up to 256 warps (it was a CTA): split
// and scan 12.1 -> 6.0 us for 91 tiles, 22 -> 14 for a 1920x1080 frame over a ground plane (four
// triangles of 8,000 to 32,000 tiles), 24.5 -> 12 for 64 requests; whole calls of a 128x128 draw
// 65.8 -> 64.2 us, of six objects in 1280x720 224 -> 219, of a recorded 1280x720 frame 178.7 -> 175.9.
constexpr uint32_t kMaxParts = 256;
constexpr uint32_t kScanWarps = kScanThreads / 32;
__global__ void __launch_bounds__(kScanThreads) k_scan(const DView* views, int T, Scratch sc, uint32_t splitters,
                                                           int part) {
  __shared__ unsigned long long warp_sums[kScanThreads / 32];
  __shared__ unsigned long long s_prefix;
  __shared__ uint32_t s_block;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nblocks = scan_blocks_hd(sc.ntiles);
  unsigned long long* split_done = sc.split;  // parts of triangles split
  const long limit = sc.poll_limit > 0 ? (long)sc.poll_limit : kScanWaitPolls;
  chain_wait();
  if (threadIdx.x == 0) s_block = atomicAdd(&sc.ctl->scan_ticket, 1u);
  __syncthreads();
  // (kScanAlone: the splitters' grid before this one took the first tickets)
  uint32_t blk = s_block - (part == kScanAlone ? splitters : 0u);
  const uint32_t nbig = min(sc.ctl->big_count, sc.big_cap);
  if (nbig > 0u) {
    const uint32_t parts = min(max(splitters * kScanWarps / nbig, 1u), kMaxParts), units = nbig * parts;
    const uint32_t first = min(splitters, (units + kScanWarps - 1) / kScanWarps);
    if (part != kScanAlone && blk < first) {
      const bool skip = (sc.ctl->error & kErrCapacity) != 0u;  // nothing will be drawn
      // (the clipper's count is final, and grows by the sub-records' only when all parts are done)
      const uint32_t base = sc.ctl->rec_count + sc.ctl->rec_extra;
      uint32_t mine = 0;  // the CTA's parts
      for (uint32_t u0 = blk * kScanWarps; u0 < units; u0 += first * kScanWarps) {
        const uint32_t u = u0 + (uint32_t)warp;
        if (!skip && u < units) split_triangle(views, T, sc, sc.bigq[u / parts], base, (int)(u % parts), (int)parts);
        mine += min((uint32_t)kScanWarps, units - u0);
      }
      __syncthreads();
      if (threadIdx.x == 0 && !(sc.faults & HSR_FAULT_SCAN_STALL)) {  // injected stall: no report
        __threadfence();
        atomicAdd(split_done, (unsigned long long)mine);
      }
      return;
    }
    if (part == kSplitAlone) return;
    if (part == kSplitAndScan) blk -= first;
    if (blk >= (uint32_t)nblocks) return;
    if (threadIdx.x == 0) {
      unsigned long long seen = 0;
      for (long spins = 0;;) {  // the limit counts from the last sign of a splitter
        const unsigned long long s = ld_volatile64(split_done), beats = ld_volatile64(sc.split + 2);
        if (s >= units) break;
        if (s + beats != seen) { seen = s + beats; spins = 0; }
        if (++spins > limit) {
          atomicOr(&sc.ctl->error, kErrScanTimeout);
          break;
        }
        __nanosleep(kPollNs);
      }
      __threadfence();
      if ((int)blk == nblocks - 1) sc.ctl->rec_extra += (uint32_t)ld_volatile64(sc.split + 1);
    }
    __syncthreads();
  }
  if (part == kSplitAlone || blk >= (uint32_t)nblocks) return;
  const int base = (int)blk * kScanTile + (int)threadIdx.x * kScanItems;
  uint32_t vals[kScanItems];
  static_assert(kScanItems == 4, "one 16-byte load");
  if (base + kScanItems <= sc.ntiles) {
    const uint4 c = __ldcg(reinterpret_cast<const uint4*>(sc.tile_count + base));
    vals[0] = c.x; vals[1] = c.y; vals[2] = c.z; vals[3] = c.w;
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; k++) vals[k] = base + k < sc.ntiles ? __ldcg(sc.tile_count + base + k) : 0u;
  }
  unsigned long long local = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) local += scan_item(vals[k]);
  // block-wide exclusive scan of the thread sums
  unsigned long long incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long w = lane < kScanThreads / 32 ? warp_sums[lane] : 0ull;
    unsigned long long wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(kFull, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < kScanThreads / 32) warp_sums[lane] = wi - w;  // exclusive per warp
    const unsigned long long agg = __shfl_sync(kFull, wi, kScanThreads / 32 - 1);  // the block's; publish, look back
    unsigned long long* st = sc.scan_status;
    unsigned long long prefix = 0;
    if (blk == 0 && nbig == 0u && (sc.faults & HSR_FAULT_SCAN_STALL)) {
      // injected stall (the splitters' where there are any): withhold the prefix and wait on a word nothing sets (its own)
      if (lane == 0) {
        long spins = 0;
        while ((ld_volatile64(&st[0]) >> 62) == 0) {
          if (++spins > limit) {
            atomicOr(&sc.ctl->error, kErrScanTimeout);
            break;
          }
          __nanosleep(kPollNs);
        }
      }
    } else if (blk == 0) {
      if (lane == 0) atomicExch(&st[0], kFlagPre | agg);
    } else {
      if (lane == 0) atomicExch(&st[blk], kFlagAgg | agg);
      long spins = 0;
      for (int p = (int)blk - 1; p >= 0;) {
        // lane l looks at the l-th predecessor; before block 0 there is a prefix of nothing
        const unsigned long long s = p >= lane ? ld_volatile64(&st[p - lane]) : kFlagPre;
        const unsigned pre = __ballot_sync(kFull, (s >> 62) == 2), none = __ballot_sync(kFull, (s >> 62) == 0);
        const unsigned use = pre ? (pre & -pre) | ((pre & -pre) - 1u) : kFull;  // up to the nearest prefix
        if (none & use) {
          if (++spins > limit) {
            if (lane == 0) atomicOr(&sc.ctl->error, kErrScanTimeout);
            break;
          }
          __nanosleep(kPollNs);
          continue;
        }
        unsigned long long sum = (use >> lane & 1u) ? s & kValMask : 0ull;
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
        prefix += sum;
        if (pre) break;
        p -= 32;
      }
      if (lane == 0) atomicExch(&st[blk], kFlagPre | (prefix + agg));
    }
    if (lane == 0) {
      s_prefix = prefix;
      if ((int)blk == nblocks - 1) {
        const unsigned long long total = prefix + agg;
        const unsigned long long pairs = total & kCntMask;
        const uint32_t ne = (uint32_t)(total >> kCntBits);
        sc.ctl->bin_total = (uint32_t)min(pairs, 0xffffffffull);
        if (pairs > sc.bin_cap) atomicOr(&sc.ctl->error, kErrBinOverflow);
        sc.ctl->ne_tiles = ne;
        sc.ne_off[sc.ntiles] = ne;
      }
    }
  }
  __syncthreads();
  unsigned long long run = s_prefix + warp_sums[warp] + (incl - local);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const int t = base + k;
    if (t < sc.ntiles) {
      const uint32_t ne = (uint32_t)(run >> kCntBits);
      sc.tile_off[t] = (uint32_t)(run & kCntMask);  // below bin_cap unless the batch overflows
      sc.ne_off[t] = ne;
      if (vals[k]) sc.tile_list[ne] = (uint32_t)t;
    }
    run += scan_item(vals[k]);
  }
}

int launch_scan(const DView* views, int tile, Scratch sc, int splitters, int part, cudaStream_t s) {
  const int grid = (part == kScanAlone ? 0 : splitters) + (part == kSplitAlone ? 0 : scan_blocks_hd(sc.ntiles));
  return launch_chained(k_scan, grid, kScanThreads, 0, s, views, tile, sc, (uint32_t)splitters, part);
}

// ---------------------------------------------------------------------------------------
// (record, tile) pairs into the per-tile lists, 32 records a warp at a time.  Where records are few
// (large triangles), up to kMaxSharers warps take the same 32 and share their pairs' steps, each
// with an atomic's round trip (1000x600 with shadow, 3,779 records of 15 tiles each: 22.5 -> 12.3 us, 2560x1440
// close-up 16.4 -> 10.2 us; a quarter million records and more keep their warps to themselves).
__device__ __forceinline__ void scatter_records(const DView* views, int T, const Scratch& sc, uint32_t block,
                                                uint32_t nblocks) {
  const int lane = threadIdx.x & 31;
  const uint32_t nrec = min(sc.ctl->rec_count + sc.ctl->rec_extra, sc.rec_cap);
  if (sc.ctl->error & kErrNoDraw) return;
  const uint32_t warps = nblocks * (blockDim.x >> 5);
  const int parts = (int)scatter_sharers(nrec, warps);
  const uint32_t me = block * (blockDim.x >> 5) + (threadIdx.x >> 5), stride = warps / (uint32_t)parts * 32u;
  if (me / (uint32_t)parts * 32u >= stride) return;
  const int part = (int)(me % (uint32_t)parts);
  const int ts = __ffs(T) - 1;  // T is a power of two
  // warp-uniform trip count so every lane takes part in the warp-level collectives
  for (uint32_t i0 = me / (uint32_t)parts * 32u; i0 < nrec; i0 += stride) {
    const uint32_t i = i0 + (uint32_t)lane;
    const bool ok = i < nrec;
    int ntw = 1, nt = 0, tile0 = 0, tiles_x = 0;
    // the record's view and pixel range: its last 16 bytes (seq, view, xr, yr) in one load
    const uint4 w = ok ? *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(&sc.recs[i]) + 48)
                       : make_uint4(0u, kRecHole << kRecFlagShift, 0u, 0u);
    if (ok && !((w.y >> kRecFlagShift) & kRecHole)) {  // holes: huge triangles split by k_scan
      const uint32_t xr = w.z, yr = w.w;
      const DView& v = views[w.y & kRecViewMask];
      tiles_x = v.tiles_x;
      const int tx0 = (int)(xr & 0xffffu) >> ts, ty0 = (int)(yr & 0xffffu) >> ts;
      tile0 = v.tile_base + ty0 * tiles_x + tx0;
      ntw = ((int)(xr >> 16) >> ts) - tx0 + 1;
      nt = min(ntw * (((int)(yr >> 16) >> ts) - ty0 + 1), kMaxRecordTiles);
    }
    auto put = [&](uint32_t tile, uint32_t at, uint32_t rec) {
      const uint32_t pos = sc.tile_off[tile] + at;
      if (pos < sc.bin_cap) sc.bins[pos] = rec;
    };
    auto pairs = [&](bool in, int tile, int own) {
      const unsigned grp = __match_any_sync(kFull, in ? tile : -1);
      const int leader = __ffs(grp) - 1;
      uint32_t b = 0;
      if (in && lane == leader) b = atomicAdd(&sc.tile_fill[tile], (uint32_t)__popc(grp));
      b = __shfl_sync(kFull, b, leader);
      if (in) put((uint32_t)tile, b + (uint32_t)__popc(grp & ((1u << lane) - 1u)), i0 + (uint32_t)own);
    };
    for_each_pair(nt, ntw, tile0, tiles_x, pairs, [&](int most) {
      const int magic = (65535 + ntw) / ntw;  // k / ntw = (k * magic) >> 16 for k < 32, ntw <= 32
      if (most < 8) {
        for (int k = part; k < most; k += parts) {
          const int ky = (k * magic) >> 16;
          pairs(k < nt, tile0 + ky * tiles_x + (k - ky * ntw), lane);
        }
        return;
      }
      // many tiles a lane (the sub-records of split triangles, which end the record list and fill
      // whole warps): four cursors asked for before the first is used, as the round trips
      // are the time (scatter of the 2560x1440 close-up 31 -> 16 us, of the 1080p frame over a
      // ground plane 43 -> 29 us).  With few tiles lanes share them and one atomic for all is better
      // (64 requests 350 against 338 us).
      for (int k = 4 * part; k < most; k += 4 * parts) {
        int tile[4];
        uint32_t b[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int ky = ((k + u) * magic) >> 16;
          tile[u] = tile0 + ky * tiles_x + (k + u - ky * ntw);
          b[u] = k + u < nt ? atomicAdd(&sc.tile_fill[tile[u]], 1u) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (k + u < nt) put((uint32_t)tile[u], b[u], i);
      }
    }, part, parts);
  }
}

// The fused clear (renderbuffer_clear_color / renderbuffer_clear_depth, renderbuffer.cpp:59-75,
// prim ids -> 0) of the pixels whose tile holds no record: the raster visits only the
// non-empty tiles and writes every pixel of those.  A chunk is kClearChunk consecutive pixels
// of one view in row-major order, so a warp's stores form one contiguous run per plane (16 bytes
// a lane where four neighbours are all cleared); the pixel's tile count (the same word for up
// to T neighbours) decides whether it is written.
// Block `block` of the `nblocks` clearing blocks takes chunks warp by warp; `cbase` holds the
// views' chunk bases when the batch has at most kSharedViews views (else null).
__device__ __forceinline__ void clear_empty_tiles(const DView* views, int T, int nchunks, const Scratch& sc,
                                                  int block, int nblocks, const int32_t* cbase) {
  if (sc.ctl->error & kErrNoDraw) return;  // an overflowing or stalled sequence draws nothing
  const int ts = __ffs(T) - 1;
  const int nv = sc.nviews;
  const int lane = (int)threadIdx.x & 31, wpb = (int)blockDim.x >> 5;
  // one chunk per warp at a time: each warp's view lookup and tile counts are an independent
  // chain of loads, so a block keeps several chunks in flight
  for (int c = block * wpb + ((int)threadIdx.x >> 5); c < nchunks; c += nblocks * wpb) {
    // the view of chunk c: the last view whose base is <= c (views without chunks share
    // their successor's base and are never the last such view)
    int lo = 0, hi = nv - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((cbase ? cbase[mid] : views[mid].cch_base) <= c) lo = mid; else hi = mid - 1;
    }
    const DView& v = views[lo];
    const int W = v.W, npx = v.W * v.H;  // below 2^30 (targets are at most 32768 x 32768)
    const int cbeg = (c - v.cch_base) * kClearChunk, cend = min(cbeg + kClearChunk, npx);
    const int32_t tb = v.tile_base, tx = v.tiles_x;
    // groups of 4 consecutive pixels (a group may run on into the next row): lane l takes the
    // groups starting at cbeg + 4l + 128k, k < kGroups; all of a lane's tile counts are in
    // flight before its stores
    constexpr int kGroups = kClearChunk / 128;
    const int g0 = cbeg + 4 * lane;
    int y = g0 / W, x = g0 - y * W;
    const int qy = 128 / W, qx = 128 - qy * W;  // the step of 128 pixels in rows and columns
    uint32_t empty = 0;  // bit 4k + d: pixel g0 + 128k + d is in the chunk and its tile has no record
#pragma unroll
    for (int k = 0; k < kGroups; k++) {
#pragma unroll
      for (int d = 0; d < 4; d++) {
        int xx = x + d, yy = y;
        if (xx >= W) {  // the group runs on into the next row(s)
          yy += xx / W;
          xx -= (xx / W) * W;
        }
        if (g0 + 128 * k + d < cend && sc.tile_count[tb + (yy >> ts) * tx + (xx >> ts)] == 0u)
          empty |= 1u << (4 * k + d);
      }
      x += qx;
      y += qy;
      if (x >= W) { x -= W; y++; }
    }
    if (!__any_sync(0xffffffffu, empty != 0u)) continue;
    const uint32_t rgba = v.clear_rgba;
    const float depth = v.clear_depth;
    uint32_t* const prim = v.prim;
    // a group starts at a multiple of 4 pixels, so with 16-byte aligned planes (the library
    // allocates them 256-byte aligned) a full group is one 16-byte store per plane
    const bool vec = ((reinterpret_cast<uintptr_t>(v.color) | reinterpret_cast<uintptr_t>(v.depth) |
                       reinterpret_cast<uintptr_t>(prim)) & 15u) == 0u;
#pragma unroll
    for (int k = 0; k < kGroups; k++) {
      const uint32_t m = (empty >> (4 * k)) & 15u;
      if (!m) continue;
      const int i = g0 + 128 * k;
      if (m == 15u && vec) {
        *reinterpret_cast<uint4*>(v.color + i) = make_uint4(rgba, rgba, rgba, rgba);
        if (v.depth) *reinterpret_cast<float4*>(v.depth + i) = make_float4(depth, depth, depth, depth);
        if (prim) *reinterpret_cast<uint4*>(prim + i) = make_uint4(0u, 0u, 0u, 0u);
      } else {
#pragma unroll
        for (int d = 0; d < 4; d++) {
          if (m >> d & 1u) {
            v.color[i + d] = rgba;
            if (v.depth) v.depth[i + d] = depth;
            if (prim) prim[i + d] = 0u;
          }
        }
      }
    }
  }
}

// Scatter and clear in one grid (when the batch has clear chunks): some blocks clear, the others
// scatter, so the store-bound clear runs beside the atomic-bound scatter instead of after it.  Of
// every two blocks one clears; where the pixels to clear outweigh the
// (record, tile) pairs, two of three do (16 views, 15 pixels a pair: 92 -> 76 us; at 6 a pair, 64
// requests, that is 299 -> 354).
constexpr int kClearMinBlocks = 3;

__global__ void __launch_bounds__(256) k_scatter(const DView* views, int T, Scratch sc, int nchunks,
                                                 float clear_share) {
  __shared__ int32_t s_cbase[kSharedViews];
  const uint32_t b = blockIdx.x, g = gridDim.x;
  chain_wait();
  const uint32_t ne = sc.ctl->ne_tiles, nt = (uint32_t)sc.ntiles;
  if (ne >= nt) nchunks = 0;  // every tile is the raster's: all blocks scatter
  const uint32_t every = scatter_every(nt - min(ne, nt), T, clear_share, sc.ctl->bin_total);
  const uint32_t first = b / every * (every - 1u);  // clearing blocks before this group
  if (nchunks > 0 && b % every != 0u) {  // block-uniform
    const bool in_shared = sc.nviews <= kSharedViews;
    if (in_shared)
      for (int i = threadIdx.x; i < sc.nviews; i += blockDim.x) s_cbase[i] = views[i].cch_base;
    __syncthreads();
    clear_empty_tiles(views, T, nchunks, sc, (int)(first + b % every - 1u), (int)(g - (g + every - 1u) / every),
                      in_shared ? s_cbase : nullptr);
  } else if (nchunks > 0) {
    scatter_records(views, T, sc, b / every, (g + every - 1u) / every);
  } else {
    scatter_records(views, T, sc, b, g);
  }
}

// `grid` blocks of 256 threads (at least kClearMinBlocks when the batch clears, so both parts have
// blocks).
int launch_scatter(const DView* views, int tile, Scratch sc, int grid, int nchunks, float clear_share, cudaStream_t s) {
  if (nchunks > 0 && grid < kClearMinBlocks) grid = kClearMinBlocks;
  return launch_chained(k_scatter, grid > 0 ? grid : 1, 256, 0, s, views, tile, sc, nchunks, clear_share);
}

}  // namespace hsr
