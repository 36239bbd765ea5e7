// Tensor-core X-step (tcgen05, sm_103a): per channel, the Hermitian product of
// the input spectra accumulated over time (Correlation_core::integration_step,
// sfxc/src/correlation_core.cc:241-273) as a real Gram matrix on the 5th-
// generation tensor cores.
//
// Each spectrum value x is stored as two FP16 numbers, hi = fp16(s*x) and
// lo = fp16(s*x - hi) (s a power of two), so hi + lo carries ~22 bits.
// Spectra layout (written by the windowed FFT, tc_index): per row, 32 stream
// slots x [hi.re, hi.im, lo.re, lo.im] FP16 per channel, stored as one
// 128-byte line per (group of four channels, slot quad), so a channel's
// slots are eight 32-byte pieces 128 B apart.  One TMA box per channel and
// K-tile gathers them, with the 32-byte swizzle, into the canonical MN-major
// layout: atoms of 8 rows x 32 B (16 components), the nq M atoms 256 B
// apart, 8-row groups 256 nq bytes apart.  The M index of a component is
// 4 * stream + {hi.re, hi.im, lo.re, lo.im}.  Only the slot quads that hold
// streams are loaded (24 streams, 16384 channels, 0.5 s: 1.74 -> 1.45 ms).  The MMA computes
// D = A A^T (128 x 16 nq, FP32 accumulation in TMEM); summing the four hi/lo
// combinations of a stream pair gives the compensated product, and the
// epilogue forms
//   Re V(a,b) = sum over re-re and im-im pairs,  Im V(a,b) = im-re minus re-im
// with lane shuffles over the 4 TMEM lanes (D rows) of one stream.
//
// Persistent CTA per SM, 10 warps, warp-specialised, over groups of 2
// channels: warp 0 streams K-tiles with TMA (cp.async.bulk.tensor, 32-byte
// swizzle, 2 boxes of 2 KB x nq per stage, 4 to 8 stages) without stopping at
// group boundaries; warp 1 issues 2 channels x 4 MMAs (K = 16) per stage into
// one of two TMEM buffers (2 x 256 columns) and commits each stage to its
// "empty" barrier and each finished group to the buffer's "full" barrier;
// warps 2-9 (one per channel and TMEM lane quarter) read the finished buffer,
// add the visibilities to the accumulator (8 loads in flight per lane) and
// release the buffer, while the next group accumulates in the other one.  Every wait is bounded: on timeout the
// CTA records an error and stops, waits (bounded) for its loads and MMAs in
// flight, frees its TMEM and returns.
#include <algorithm>
#include <cstdint>
#include <cuda.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include "device.cuh"
#include "kernels.hpp"
#include "tc_ptx.cuh"

namespace sfxc {
namespace {
using namespace tc;

constexpr int kChan = 2;        // channels per group (one TMEM buffer)
constexpr int kRowsK = 64;      // FFT rows per K-tile
constexpr int kMaxStages = 8;
constexpr int kStagesBytes = 131072;  // the stage ring (4 stages of 32 streams; 3 measured 17 % slower, 6 stages 3 %)
constexpr int kThreads = 320;   // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr uint32_t kBufCols = kChan * 128;      // TMEM columns per buffer
// One channel's K-tile: TMA box {16 components, 8 rows, nq slot quads, 8 row
// groups, 1 channel group} = 2 KB x nq at row group rg and channel group cg.
__device__ __forceinline__ void tma_load_tile(void *dst, const CUtensorMap *map, int rg, int cg, uint64_t *bar) {
  tma_load_5d(dst, map, 0, 0, 0, rg, cg, bar);
}

// Tensor maps of the four channels of a channel group (base offsets 32 B apart).
struct TcMaps {
  CUtensorMap m[4];
};

__global__ void __launch_bounds__(kThreads, 1)
    xcorr_tc_kernel(const __grid_constant__ TcMaps tmaps, int nrows, int K, int kpad, int nq, int nst,
                    const int *__restrict__ blmap, int npad, float inv_scale2, float2 *__restrict__ acc, int *__restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);  // stages 1 KB aligned
  __shared__ uint64_t full[kMaxStages], empty[kMaxStages], tfull[2], tempty[2], done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ngroups = (K + kChan - 1) / kChan;
  const int nkt = (nrows + kRowsK - 1) / kRowsK;
  // one channel's K-tile (64 rows x 16 nq components x 2 B) and a stage of two
  const int ctile = kRowsK * 32 * nq, sbytes = kChan * ctile;
  // this CTA's groups: blockIdx.x, blockIdx.x + gridDim.x, ...
  const int my_groups = blockIdx.x < ngroups ? (ngroups - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

  if (warp == 0) {
    tmem_alloc(&tmem_base, 512);
  }
  if (tid == 0) {
    for (int s = 0; s < kMaxStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 8);  // one arrival per epilogue warp
    }
    mbar_init(&done, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  volatile int *vfailed = &failed;

  if (tid == 0) {
    // ---- TMA producer: every K-tile of every group, one stage ring
    int it = 0;
    for (int i = 0; i < my_groups && !*vfailed; i++) {
      const int g = blockIdx.x + i * gridDim.x;
      for (int kt = 0; kt < nkt; kt++, it++) {
        const int s = it % nst, n = it / nst;
        if ((n > 0 && !mbar_wait(&empty[s], (n - 1) & 1)) || *vfailed) {
          *vfailed = 1;
          break;
        }
        mbar_expect_tx(&full[s], sbytes);
        uint8_t *st = base + s * sbytes;
#pragma unroll
        for (int c = 0; c < kChan; c++) {
          const int ch = g * kChan + c;
          tma_load_tile(st + c * ctile, &tmaps.m[ch & 3], kt * (kRowsK / 8), ch >> 2, &full[s]);
        }
      }
    }
    // loads still in flight (the last nst tiles) land before the CTA may exit
    for (int i = it > nst ? it - nst : 0; i < it; i++)
      if (!mbar_wait(&full[i % nst], (i / nst) & 1)) *vfailed = 1;
  } else if (tid == 32) {
    // ---- MMA issuer
    const uint32_t idesc = idesc_f16(128, 16 * nq);
    int it = 0;
    for (int i = 0; i < my_groups && !*vfailed; i++) {
      const int b = i & 1, u = i >> 1;
      if (u > 0 && !mbar_wait(&tempty[b], (u - 1) & 1)) {  // the epilogue has read buffer b
        *vfailed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      bool ok = true;
      for (int kt = 0; kt < nkt; kt++, it++) {
        const int s = it % nst, n = it / nst;
        if (!mbar_wait(&full[s], n & 1)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t st = smem_u32(base) + s * sbytes;
#pragma unroll
        for (int c = 0; c < kChan; c++) {
#pragma unroll
          for (int ks = 0; ks < kRowsK / 16; ks++) {
            // 16 K-rows = two 8-row groups of nq atoms; M atoms 256 B apart
            const uint64_t d = smem_desc32(st + c * ctile + ks * 512 * nq, 256, 256 * nq);
            mma_f16(tmem + b * kBufCols + c * 128, d, d, idesc, (kt > 0 || ks > 0) ? 1u : 0u);
          }
        }
        mma_commit(&empty[s]);
      }
      if (!ok) {
        *vfailed = 1;
        break;
      }
      mma_commit(&tfull[b]);  // the group's sums are complete when its MMAs are
    }
    mma_commit(&done);  // arrives once every MMA issued above has completed
  } else if (warp >= 2) {
    // ---- epilogue: warp w reads channel (w - 2) / 4 of the group, TMEM lanes
    // 32 (w % 4) .. + 31 (D rows)
    const int q = warp & 3, c = (warp - 2) >> 2, m = q * 32 + lane, a = m >> 2, p = m & 3;
    for (int i = 0; i < my_groups; i++) {
      const int b = i & 1, u = i >> 1;
      if (!mbar_wait(&tfull[b], u & 1)) {
        *vfailed = 1;
        break;
      }
      if (*vfailed) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int k = (blockIdx.x + i * gridDim.x) * kChan + c;
#pragma unroll 1
      for (int j = 0; 2 * j < nq && 8 * q < npad; j++) {
        float v[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + b * kBufCols + c * 128 + j * 32, v);
        float re8[8], im8[8];
#pragma unroll
        for (int bb = 0; bb < 8; bb++) {
          const float A = v[4 * bb] + v[4 * bb + 2], B = v[4 * bb + 1] + v[4 * bb + 3];
          // row component p: 0 hi.re, 1 hi.im, 2 lo.re, 3 lo.im; columns likewise
          float re = (p & 1) ? B : A, im = (p & 1) ? A : -B;
          re += __shfl_xor_sync(0xffffffffu, re, 1);
          im += __shfl_xor_sync(0xffffffffu, im, 1);
          re += __shfl_xor_sync(0xffffffffu, re, 2);
          im += __shfl_xor_sync(0xffffffffu, im, 2);
          re8[bb] = re;
          im8[bb] = im;
        }
        if (p == 0 && k < K && a < npad) {
          // the 8 baselines' accumulator loads in flight together
          int mv[8];
          float2 o[8];
#pragma unroll
          for (int bb = 0; bb < 8; bb++) mv[bb] = j * 8 + bb < npad ? __ldg(blmap + a * npad + j * 8 + bb) : -1;
#pragma unroll
          for (int bb = 0; bb < 8; bb++)
            if (mv[bb] >= 0) o[bb] = acc[(int64_t)(mv[bb] >> 1) * kpad + k];
#pragma unroll
          for (int bb = 0; bb < 8; bb++)
            if (mv[bb] >= 0) {
              o[bb].x += re8[bb] * inv_scale2;
              o[bb].y += ((mv[bb] & 1) ? -im8[bb] : im8[bb]) * inv_scale2;
              acc[(int64_t)(mv[bb] >> 1) * kpad + k] = o[bb];
            }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[b]);  // buffer b may be overwritten
    }
  }
  __syncthreads();
  if (!mbar_wait(&done, 0)) *vfailed = 1;  // no MMA in flight past this point
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  __syncthreads();
  if (*vfailed && tid == 0) atomicExch(err, 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------
// Row-gathered tensor-core X-step: the same compensated Gram products, with
// each channel's FFT rows taken in the order of a per-channel row list, cut
// into segments that go to separate accumulators:
//   * pulsar binning (Correlation_core_pulsar::integration_step,
//     sfxc/src/correlation_core_pulsar.cc:101-146 with the bins of 210-238):
//     each channel's rows sorted by bin (pulsar_sort_kernel), one segment per
//     bin, the segment's Gram stored as acc[bin];
//   * jobs of 33 to 64 streams (S = 64 slots): rows in order, one segment.
// A tile is up to kRows listed rows of one segment.  Warps 0-3 take the tiles
// in turn: each copies its tile's rows with 16-byte cp.async, only the slot
// quads that hold streams, straight into 128-byte-swizzled MN-major atoms of
// 64 components (list entries of -1 read as zero rows),
// and publishes it after a proxy fence when its next tile is on the way, so
// eight tiles are in flight.  Warp 4 issues the MMAs -- per 16 rows, block I = 0
// (and 1 for S = 64): M = 128 rows of components from 128 I, N = the
// components from 128 I to the last stream (FP32 accumulation in the
// segment's TMEM buffer; the rows of M past the last stream are whatever lies
// behind the tile and are not read back).  The remaining warps bring each
// finished buffer to its accumulator while the next segments accumulate in
// the other buffers: for S = 32 four warps per TMEM lane quarter, each taking
// every fourth segment; for S = 64 two, each taking every other 16 columns.
// Only the producers follow the row list: the tile's place goes through
// shared memory to the MMA warp and the segment's from there to the epilogue.
// Every wait is bounded: on timeout the CTA records an error and stops,
// waits (bounded) for its copies and MMAs in flight, frees its TMEM and
// returns.
//
// Bound: with binning, the chains of small steps a segment of few rows takes
// in each role (copies about 700 cycles a segment and warp, MMA issue and its
// commits 700, epilogue 1300 over four sets): 526,000 (channel, bin) segments
// of 30 rows of 20 streams 6.36 -> 2.87 ms.  Copying chunk by chunk instead of
// four at a time, to overlap their shuffles and addresses, takes 3.8 ms, eight
// at a time 3.1; 32-byte-swizzled atoms 3.85 against 3.79 then.  For 33 to 64
// streams, L2 and DRAM reads of 32-byte pieces: 40 streams, 4096 channels,
// 1953 rows 2.57 -> 0.82 ms (3.1 TB/s of spectra) -- slot quads without streams
// were read too, and a CTA took the four channels of a group one after the
// other, by when their common 128-byte lines had left L2 (6.4 TB/s from DRAM
// for 1.6 of spectra); now four CTAs take them at the same time.
template <int S>
struct GatherShape {
  static constexpr int kRows = S == kTcSlots ? 64 : 32;  // rows per tile (at most 16 KB)
  static constexpr int kStagesBytes = 131072;            // the stage ring: one CTA per SM
  static constexpr int kMaxStages = 16;
  static constexpr int kProducers = 4;                   // warps 0-3
  static constexpr int kSets = S == kTcSlots ? 4 : 2;    // epilogue warps per TMEM lane quarter
  static constexpr bool kBySegment = S == kTcSlots;      // the sets take whole segments in turn
  static constexpr int kSlots = S == kTcSlots ? 8 : 12;  // 16-column chunks per epilogue warp and segment
  static constexpr int kThreads = 32 * (kProducers + 1 + 4 * kSets);
  // + alignment + what M = 128 reads behind the last stage (one atom column)
  static constexpr size_t kSmem = kStagesBytes + 1024 + kRows * 128;
};

struct GatherArgs {
  const uint8_t *spec;  // TC layout with S slots
  int nrows;            // rows in the buffer; list entries outside [0, nrows) read as zeros
  int kpad, K, nstreams, npad, nbl, nbins;
  const int *rowlist;   // per channel list_len entries (row or -1); NULL: the rows in order
  int list_len;
  const int2 *segs;     // per (channel, bin): first list entry, entries (a multiple of 16); NULL: one segment
  const int *blmap;
  float inv_scale2;
  float2 *acc;          // [bin][baseline][kpad]
  int *err;
  int nq, nst;          // slot quads with streams; stages of the ring
  int parts, part_bins; // units of work: channel groups of four x parts of the bins (a multiple of 8 bins each)
  int n0, n1, col1;     // MMA N of blocks 0 and 1 (n1 = 0: one block), TMEM column of block 1
  int buf_stride, nbuf; // TMEM columns per buffer, number of buffers
  int accumulate;       // 0: every (bin, channel) segment is the only one of its launch and is stored as it is
};

constexpr int kMaxBufs = 8;

// The tiles of this CTA in processing order: its units (unit blockIdx.x, then
// + gridDim.x) of a group of four channels and a part of the bins; within a
// unit bin by bin; within a bin the group's four channels; within a segment R
// rows at a time.  The four channels of a group read the four 32-byte pieces
// of the same 128-byte spectra lines and write the same 32-byte accumulator
// sectors close together in time.  Warp-wide: lane l holds the segment of
// (bin, channel) number kb + l of the unit, and that of kb + 32 + l is on its way.
struct GWalk {
  int u, nunits, grp, kb, kend, cur, e0, len, t0, lane;
  int2 seg, next_seg;
  unsigned mask;
  __device__ int2 load(const GatherArgs &g, int k) const {
    const int ch = 4 * grp + (k & 3);
    if (k >= kend || ch >= g.K) return make_int2(0, 0);
    return g.segs ? __ldg(g.segs + (size_t)ch * g.nbins + (k >> 2)) : make_int2(0, (g.nrows + 15) & ~15);
  }
  __device__ void unit(const GatherArgs &g) {
    grp = u / g.parts;
    const int part = u - grp * g.parts;
    kb = g.segs ? 4 * part * g.part_bins : part;
    kend = g.segs ? min(4 * g.nbins, kb + 4 * g.part_bins) : part + 1;
    next_seg = load(g, kb + lane);
  }
  __device__ void batch(const GatherArgs &g) {
    seg = next_seg;
    next_seg = load(g, kb + 32 + lane);
    mask = __ballot_sync(0xffffffffu, seg.y > 0);
    cur = -1;
  }
  __device__ void init(const GatherArgs &g) {
    lane = threadIdx.x & 31;
    nunits = (g.K + 3) / 4 * g.parts;
    u = blockIdx.x;
    cur = -1;
    len = t0 = 0;
    mask = 0;
    kb = kend = 0;
    if (u < nunits) {
      unit(g);
      batch(g);
    }
  }
  // the next tile: e0 + t0 its first list entry
  __device__ bool next(const GatherArgs &g, int R) {
    t0 += R;
    if (t0 < len) return true;
    for (;;) {
      const unsigned rest = mask & (cur < 0 ? ~0u : ~1u << cur);
      if (rest) {
        cur = __ffs(rest) - 1;
        break;
      }
      if (u >= nunits) return false;
      kb += 32;
      if (kb >= kend) {
        u += gridDim.x;
        mask = 0;
        if (u >= nunits) return false;
        unit(g);
      }
      batch(g);
    }
    e0 = __shfl_sync(0xffffffffu, seg.x, cur);
    len = __shfl_sync(0xffffffffu, seg.y, cur);
    t0 = 0;
    return true;
  }
};

// A tile in the ring: rows (a multiple of 16; -1: no more tiles), channel,
// bin, bit 0 / 1: first / last of its segment.
struct GTile {
  int rows, ch, bin, flags;
};

template <int S>
__global__ void __launch_bounds__(GatherShape<S>::kThreads, 1) xcorr_tc_gather_kernel(const __grid_constant__ GatherArgs g) {
  using G = GatherShape<S>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);  // stages 1 KB aligned
  __shared__ uint64_t full[G::kMaxStages], empty[G::kMaxStages], tfull[kMaxBufs], tempty[kMaxBufs], done;
  __shared__ GTile tiles[G::kMaxStages];
  __shared__ int2 segs[kMaxBufs];  // channel (-1: no more segments) and bin of each TMEM buffer
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 4) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    for (int s = 0; s < G::kMaxStages; s++) {
      mbar_init(&full[s], 32);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kMaxBufs; b++) {
      mbar_init(&tfull[b], 2);  // the MMAs' commit and the issuer
      mbar_init(&tempty[b], G::kBySegment ? 4 : 4 * G::kSets);  // one arrival per epilogue warp of the segment
    }
    mbar_init(&done, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = tmem_base;
  volatile int *vfailed = &failed;
  constexpr int kAtoms = G::kRows * 128;         // a column of atoms: kRows rows x 64 components
  const int sbytes = (g.nq + 3) / 4 * kAtoms;    // one stage

  if (warp < G::kProducers) {
    // ---- producers: tile it is warp it % 4's; its rows' 16-byte chunks (2 nq
    // a row) lane by lane; the list entries of the warp's next tile load while
    // the current one is issued
    constexpr int E = G::kRows / 32, U = 4;
    const int cpr = 2 * g.nq, dj = 32 / cpr, dc = 32 % cpr, j0 = lane / cpr, c0 = lane % cpr;
    const int64_t rstride = (int64_t)g.kpad * S * 8;  // bytes per row
    GWalk walk;
    walk.init(g);
    int it = -1;  // the tile the walk stands at
    struct Mine {
      GTile t;
      int row[E];
    } cur, nxt;
    auto advance = [&](int steps, Mine &m) -> bool {  // to the warp's next tile; false: `it` is the number of tiles
      for (int i = 0; i < steps; i++) {
        it++;
        if (!walk.next(g, G::kRows)) return false;
      }
      m.t.rows = min(G::kRows, walk.len - walk.t0);
      m.t.ch = 4 * walk.grp + ((walk.kb + walk.cur) & 3);
      m.t.bin = (walk.kb + walk.cur) >> 2;
      m.t.flags = (walk.t0 == 0 ? 1 : 0) | (walk.t0 + G::kRows >= walk.len ? 2 : 0);
      const int e = walk.e0 + walk.t0 + lane;
#pragma unroll
      for (int i = 0; i < E; i++)
        m.row[i] = !g.rowlist ? e + 32 * i
                   : lane + 32 * i < m.t.rows ? __ldg(g.rowlist + (size_t)m.t.ch * g.list_len + e + 32 * i) : -1;
      return true;
    };
    auto publish = [&](int tile) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(&full[tile % g.nst]);
    };
    bool have = advance(warp + 1, cur);
    int mine = it, last = -1;
    bool ok = true;
    while (have) {
      const bool have_next = advance(4, nxt);
      const int s = mine % g.nst, n = mine / g.nst;
      ok = __all_sync(0xffffffffu, (n == 0 || mbar_wait(&empty[s], (n - 1) & 1)) && !*vfailed);
      if (!ok) break;
      if (lane == 0) tiles[s] = cur.t;
      const uint32_t st = smem_u32(base) + s * sbytes;
      const uint8_t *chbase = g.spec + tc_index(0, g.kpad, cur.t.ch, 0, S) * 8;
      const int total = cur.t.rows * cpr;
      int j = j0, c = c0;
      for (int x = lane; x < total + lane; x += 32 * U) {  // U chunks a lane at a time, to overlap their latencies
        int jj[U], cc[U], row[U];
#pragma unroll
        for (int i = 0; i < U; i++) {
          jj[i] = j;
          cc[i] = c;
          j += dj;
          c += dc;
          if (c >= cpr) {
            c -= cpr;
            j++;
          }
        }
#pragma unroll
        for (int i = 0; i < U; i++) {
          row[i] = __shfl_sync(0xffffffffu, cur.row[0], jj[i] & 31);
          if (E > 1) {
            const int r1 = __shfl_sync(0xffffffffu, cur.row[E - 1], jj[i] & 31);
            if (jj[i] >= 32) row[i] = r1;
          }
        }
#pragma unroll
        for (int i = 0; i < U; i++) {
          const bool in = (unsigned)row[i] < (unsigned)g.nrows;
          const uint8_t *src = chbase + (in ? row[i] : 0) * rstride + (cc[i] >> 1) * 128 + (cc[i] & 1) * 16;
          if (x + 32 * i < total) cp_async16(st + (cc[i] >> 3) * kAtoms + sw128_offset(jj[i], cc[i]), src, in ? 16u : 0u);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (last >= 0) {  // the warp's previous tile has landed: publish it to the tensor cores
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        publish(last);
      }
      last = mine;
      mine += 4;
      cur = nxt;
      have = have_next;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (last >= 0) publish(last);
    if (ok && it % 4 == warp) {  // after the last tile, in its warp's turn: the end
      const int s = it % g.nst, n = it / g.nst;
      if (n > 0 && !mbar_wait(&empty[s], (n - 1) & 1)) ok = false;
      if (lane == 0) tiles[s].rows = -1;
      mbar_arrive(&full[s]);
    }
    if (!ok) *vfailed = 1;
  } else if (tid == 4 * 32) {
    // ---- MMA issuer
    const uint32_t id0 = idesc_f16(128, g.n0), id1 = idesc_f16(128, g.n1 > 0 ? g.n1 : 16);
    int s = 0, b = 0, sphase = 0, u = 0;  // stage and its parity, TMEM buffer and its uses
    uint32_t d0 = tmem;
    const uint64_t ring = smem_desc(smem_u32(base), kAtoms, 1024);
    bool ok = true;
    // buffer b is free: the epilogue has read its previous segment
    auto claim = [&]() { return (u == 0 || mbar_wait(&tempty[b], (u - 1) & 1)) && !*vfailed; };
    auto advance = [&]() {
      if (++b == g.nbuf) {
        b = 0;
        u++;
      }
    };
    for (;;) {
      if (!mbar_wait(&full[s], sphase) || *vfailed) {
        ok = false;
        break;
      }
      const GTile t = tiles[s];
      if (t.rows < 0) break;
      if (t.flags & 1) {
        if (!claim()) {
          ok = false;
          break;
        }
        segs[b] = make_int2(t.ch, t.bin);
        d0 = tmem + (uint32_t)(b * g.buf_stride);
      }
      fence_after_sync();
      uint32_t acc_flag = t.flags & 1 ? 0u : 1u;
      uint64_t a0 = ring + (uint32_t)((s * sbytes) >> 4);
#pragma unroll
      for (int ks = 0; ks < G::kRows / 16; ks++, a0 += 2048 >> 4) {
        if (ks * 16 >= t.rows) break;
        // 16 K rows = two 8-row groups of 1 KB; block 1 starts two atoms in
        mma_f16(d0, a0, a0, id0, acc_flag);
        if (S > kTcSlots) {
          const uint64_t a1 = a0 + (2 * kAtoms >> 4);
          mma_f16(d0 + (uint32_t)g.col1, a1, a1, id1, acc_flag);
        }
        acc_flag = 1u;
      }
      mma_commit(&empty[s]);
      if (++s == g.nst) {
        s = 0;
        sphase ^= 1;
      }
      if (t.flags & 2) {
        mma_commit(&tfull[b]);  // the segment's sums are complete when its MMAs are
        mbar_arrive(&tfull[b]);
        advance();
      }
    }
    for (int e = 0; ok && e < (G::kBySegment ? G::kSets : 1); e++) {  // the end, to every set
      if (!claim()) ok = false;
      segs[b] = make_int2(-1, 0);
      mbar_arrive(&tfull[b]);
      mbar_arrive(&tfull[b]);
      advance();
    }
    if (!ok) *vfailed = 1;
    mma_commit(&done);  // arrives once every MMA issued above has completed
  } else if (warp > G::kProducers) {
    // ---- epilogue: a warp reads TMEM lane quarter q = warp % 4 (D rows 32 q ..
    // 32 q + 31 of each block), in chunks of 16 columns (4 streams).  Lane
    // 4 i + p of a chunk has component p of row stream 8 q + i (0 hi.re, 1
    // hi.im, 2 lo.re, 3 lo.im; columns likewise) for the 4 column streams;
    // the exchange that sums the four components leaves column stream p's sum
    // in lane p, which stores it.
    const int q = warp & 3, set = (warp - G::kProducers - 1) >> 2;
    const int p = lane & 3;
    int off[G::kSlots];   // accumulator index * 2 + conjugate, per chunk; -1: no such baseline
    unsigned active = 0;  // chunks with a baseline
#pragma unroll
    for (int i = 0; i < G::kSlots; i++) {
      const int I = i >> 3, chunk = G::kBySegment ? i : 2 * (i & 7) + set;
      const int a = 32 * I + 8 * q + (lane >> 2), bs = 32 * I + 4 * chunk + p;
      const int v = a < g.nstreams && bs < g.nstreams && chunk < (I ? g.n1 : g.n0) / 16 ? __ldg(g.blmap + a * g.npad + bs) : -1;
      off[i] = v < 0 ? -1 : (v >> 1) * g.kpad * 2 + (v & 1);
      if (__any_sync(0xffffffffu, v >= 0)) active |= 1u << i;
    }
    int b = 0, u = 0;
    auto skip = [&](int n) {
      for (int i = 0; i < n; i++)
        if (++b == g.nbuf) {
          b = 0;
          u ^= 1;
        }
    };
    if (G::kBySegment) skip(set);
    for (;;) {
      if (!__all_sync(0xffffffffu, mbar_wait(&tfull[b], u) && !*vfailed)) {
        *vfailed = 1;
        break;
      }
      fence_after_sync();
      const int2 sg = segs[b];
      if (sg.x < 0) break;
      float2 *accb = g.acc + (size_t)sg.y * g.nbl * g.kpad + sg.x;
#pragma unroll
      for (int i = 0; i < G::kSlots; i++) {
        if (!(active >> i & 1)) continue;
        const int I = i >> 3, chunk = G::kBySegment ? i : 2 * (i & 7) + set;
        float2 o = make_float2(0.f, 0.f);
        float2 *dst = accb + (off[i] >> 1);
        if (g.accumulate && off[i] >= 0) o = *dst;
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * g.buf_stride + (I ? g.col1 : 0) + 16 * chunk), v);
        float re[4], im[4];
#pragma unroll
        for (int bb = 0; bb < 4; bb++) {
          const float A = v[4 * bb] + v[4 * bb + 2], B = v[4 * bb + 1] + v[4 * bb + 3];
          re[bb] = (p & 1) ? B : A;
          im[bb] = (p & 1) ? A : -B;
        }
        // (component p + p ^ 1) + (the other two): lanes keep the column
        // streams of their own low bit, then of their own high bit
        float r2[2], i2[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const float kr = (p & 1) ? re[2 * h + 1] : re[2 * h], sr = (p & 1) ? re[2 * h] : re[2 * h + 1];
          const float ki = (p & 1) ? im[2 * h + 1] : im[2 * h], si = (p & 1) ? im[2 * h] : im[2 * h + 1];
          r2[h] = kr + __shfl_xor_sync(0xffffffffu, sr, 1);
          i2[h] = ki + __shfl_xor_sync(0xffffffffu, si, 1);
        }
        const float kr = (p & 2) ? r2[1] : r2[0], sr = (p & 2) ? r2[0] : r2[1];
        const float ki = (p & 2) ? i2[1] : i2[0], si = (p & 2) ? i2[0] : i2[1];
        const float vr = kr + __shfl_xor_sync(0xffffffffu, sr, 2);
        const float vi = ki + __shfl_xor_sync(0xffffffffu, si, 2);
        if (off[i] >= 0) {
          o.x += vr * g.inv_scale2;
          o.y += ((off[i] & 1) ? -vi : vi) * g.inv_scale2;
          *dst = o;
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[b]);  // buffer b may be overwritten
      skip(G::kBySegment ? G::kSets : 1);
    }
  }
  __syncthreads();
  if (!mbar_wait(&done, 0)) *vfailed = 1;  // no MMA in flight past this point
  fence_after_sync();
  __syncthreads();
  if (*vfailed && tid == 0) atomicExch(g.err, 1);
  fence_before_sync();
  __syncthreads();
  if (warp == 4) {
    fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// Rows of each channel sorted stably by pulsar bin, each bin's run padded
// with -1 entries to a multiple of 16 rows: rowlist[ch][list_len] and
// segs[ch][bin] = (first entry, entries).  bins: [channel][row].  One warp
// per channel; shared counters per warp.
__global__ void __launch_bounds__(128) pulsar_sort_kernel(const int16_t *__restrict__ bins, int nrows, int K,
                                                          int nbins, int list_len, int *__restrict__ rowlist,
                                                          int2 *__restrict__ segs) {
  extern __shared__ int cnt[];  // per warp: count[nbins], cursor[nbins]
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ch = blockIdx.x * 4 + w;
  if (ch >= K) return;  // whole warps
  int *count = cnt + w * 2 * nbins, *cursor = count + nbins;
  for (int b = lane; b < nbins; b += 32) count[b] = 0;
  __syncwarp();
  const int16_t *br = bins + (size_t)ch * nrows;
  for (int r = lane; r < nrows; r += 32) atomicAdd(&count[br[r]], 1);
  __syncwarp();
  if (lane == 0) {
    int pos = 0;
    for (int b = 0; b < nbins; b++) {
      const int len = (count[b] + 15) & ~15;
      segs[(size_t)ch * nbins + b] = make_int2(pos, len);
      cursor[b] = pos;
      pos += len;
    }
  }
  __syncwarp();
  int *list = rowlist + (size_t)ch * list_len;
  for (int b = lane; b < nbins; b += 32)  // padding entries of each run
    for (int e = cursor[b] + count[b]; e < cursor[b] + ((count[b] + 15) & ~15); e++) list[e] = -1;
  __syncwarp();
  for (int r0 = 0; r0 < nrows; r0 += 32) {
    const int r = r0 + lane;
    const int b = r < nrows ? br[r] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, b);
    const int rank = __popc(same & ((1u << lane) - 1u));
    const int pos = b >= 0 ? cursor[b] + rank : 0;
    __syncwarp();
    if (b >= 0) {
      list[pos] = r;
      if (rank == 0) cursor[b] = pos + __popc(same);
    }
    __syncwarp();
  }
}

}  // namespace

// + alignment + what the M = 128 operand reads behind the last stage's last row group
size_t xcorr_tc_smem_bytes() { return kStagesBytes + 1024 + 2048; }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda).
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

cudaError_t launch_xcorr_tc(const void *spec, int nrows, int kpad, int K, const int *blmap, int npad,
                            float inv_scale2, float2 *acc, int *err, cudaStream_t st) {
  if (nrows <= 0) return cudaSuccess;
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  // per channel of a group (base + 32 B each): 16 components of a slot quad,
  // rows within an 8-row group (kpad * 256 B apart), the 8 slot quads (128 B
  // apart), 8-row groups, channel groups (1 KB apart).  Rows from nrows up to
  // the next multiple of 8 must be zero in the buffer (the caller clears
  // them); row groups past the end read as zeros.
  if (kpad % 4 != 0 || npad % 4 != 0 || npad <= 0 || npad > kTcSlots) return cudaErrorInvalidValue;
  TcMaps maps;
  const cuuint64_t R = (cuuint64_t)kpad * 256;
  const cuuint64_t dims[5] = {16, 8, 8, (cuuint64_t)(nrows + 7) / 8, (cuuint64_t)kpad / 4};
  const cuuint64_t strides[4] = {R, 128, 8 * R, 1024};
  const int nq = npad / 4;  // slot quads with streams: only these are read
  const cuuint32_t box[5] = {16, 8, (cuuint32_t)nq, (cuuint32_t)kRowsK / 8, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  for (int cc = 0; cc < 4; cc++)
    if (enc(&maps.m[cc], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, static_cast<char *>(const_cast<void *>(spec)) + 32 * cc,
            dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B,
            CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
  const size_t smem = xcorr_tc_smem_bytes();
  cudaError_t e = cudaFuncSetAttribute(xcorr_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0) nsm = 1;
  const int ngroups = (K + kChan - 1) / kChan;
  const int nst = std::min(kMaxStages, kStagesBytes / (kChan * kRowsK * 32 * nq));
  xcorr_tc_kernel<<<std::min(ngroups, nsm), kThreads, smem, st>>>(maps, nrows, K, kpad, nq, nst, blmap, npad,
                                                                   inv_scale2, acc, err);
  return cudaGetLastError();
}

template <int S>
static cudaError_t launch_gather(const GatherArgs &g, cudaStream_t st) {
  using G = GatherShape<S>;
  cudaError_t e = cudaFuncSetAttribute(xcorr_tc_gather_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)G::kSmem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0) nsm = 1;
  const int ngroups = (g.K + 3) / 4;
  GatherArgs a = g;
  // a multiple of the producer warps (8 or more), so that a stage is always
  // the same warp's and that warp sees every phase of its barriers; the same
  // for the buffers and the epilogue sets that take whole segments (4 or 8)
  a.nst = std::min(G::kMaxStages, G::kStagesBytes / (G::kRows * 128 * ((a.nq + 3) / 4))) / G::kProducers * G::kProducers;
  if (G::kBySegment) a.nbuf = a.nbuf / G::kSets * G::kSets;
  if (a.rowlist) {
    // parts of the bins (at least 16) so that every CTA has 12 units or more:
    // the last, partly filled round is then at most a twelfth
    a.parts = std::max(1, std::min((12 * nsm + ngroups - 1) / ngroups, a.nbins / 16));
    a.part_bins = a.parts > 1 ? ((a.nbins + a.parts - 1) / a.parts + 7) / 8 * 8 : a.nbins;
    a.parts = (a.nbins + a.part_bins - 1) / a.part_bins;
  } else {
    a.parts = 4;  // one channel a unit
    a.part_bins = 1;
  }
  xcorr_tc_gather_kernel<S><<<std::min(ngroups * a.parts, nsm), G::kThreads, G::kSmem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_xcorr_tc_gather(const void *spec, int slots, int nrows, int kpad, int K, int nstreams,
                                   const int *blmap, int npad, int nbl, int nbins, const int *rowlist, int list_len,
                                   const int2 *segs, float inv_scale2, float2 *acc, int *err, cudaStream_t st) {
  if (nrows <= 0 || K <= 0) return cudaSuccess;
  // 64 slots only for what 32 do not hold: their second row block is always issued
  if (nstreams <= 0 || slots != (nstreams <= kTcSlots ? kTcSlots : kTcSlotsWide) || nstreams > kTcSlotsWide)
    return cudaErrorInvalidValue;
  GatherArgs g;
  g.spec = static_cast<const uint8_t *>(spec);
  g.nrows = nrows;
  g.kpad = kpad;
  g.K = K;
  g.nstreams = nstreams;
  g.npad = npad;
  g.nbl = nbl;
  g.nbins = rowlist ? nbins : 1;
  g.rowlist = rowlist;
  g.list_len = list_len;
  g.segs = rowlist ? segs : nullptr;
  g.blmap = blmap;
  g.inv_scale2 = inv_scale2;
  g.acc = acc;
  g.err = err;
  g.nq = (nstreams + 3) / 4;
  auto up16 = [](int x) { return (x + 15) & ~15; };
  auto up32 = [](int x) { return (x + 31) & ~31; };
  const int comps = 4 * nstreams;
  g.n0 = up16(std::min(comps, 256));
  g.n1 = comps > 128 ? up16(comps - 128) : 0;
  g.col1 = up32(g.n0);
  g.buf_stride = g.col1 + up32(g.n1);
  g.nbuf = std::min(kMaxBufs, 512 / g.buf_stride);
  // with a row list (pulsar binning: the whole integration in one launch) each
  // (bin, channel) segment is the only one of its accumulator entries
  g.accumulate = rowlist ? 0 : 1;
  if (slots == kTcSlots) return launch_gather<kTcSlots>(g, st);
  return launch_gather<kTcSlotsWide>(g, st);
}

void launch_pulsar_sort(const int16_t *bins, int nrows, int K, int nbins, int list_len, int *rowlist, int2 *segs,
                        cudaStream_t st) {
  const size_t smem = (size_t)4 * 2 * nbins * sizeof(int);
  if (smem > 48 * 1024) cudaFuncSetAttribute(pulsar_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  pulsar_sort_kernel<<<(K + 3) / 4, 128, smem, st>>>(bins, nrows, K, nbins, list_len, rowlist, segs);
}

}  // namespace sfxc
