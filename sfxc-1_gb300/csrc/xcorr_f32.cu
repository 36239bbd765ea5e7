// X-step on CUDA cores without binning (Correlation_core::integration_step,
// sfxc/src/correlation_core.cc:241-273), in FP32.
#include <algorithm>

#include "device.cuh"
#include "kernels.hpp"
#include "tc_ptx.cuh"

namespace sfxc {
namespace {

// spec: [stream][row][kpad] complex64.  A column is a 32-channel tile and a
// part of the stream-pair tiles; the columns' rows, laid end to end in steps
// of R rows, are dealt to the CTAs in equal consecutive shares, so that every
// SM works to the end whatever the number of columns.  A CTA stages R rows x
// np8 streams x 32 channels per step through a 4-deep cp.async ring; each
// thread owns one channel and one 8x8 tile of stream pairs in registers (16
// shared-memory loads for 256 multiply-adds; 4x4 tiles load as many cycles as
// they multiply).  A diagonal unit takes two diagonal tiles a and b, the upper
// triangle of a above its diagonal, that of b below, and both tiles'
// autocorrelations, which are real, on it.  Where the units are few, groups of
// warps each take a stretch of consecutive rows and add their tiles up in shared
// memory (every G-th row instead lost the cancellation of products that turn by
// 1/G from row to row, as a tone's do at some fringe rates: errors of 5e-8 of the
// terms' sum where consecutive rows lose 1e-9).  A share's sums of a column go to
// a slot of the partial sums, added later in order, so results do not depend on
// timing.
//
// Bounds: FP32 multiply-adds with three register operands, which run at 26 of
// 38 T lane operations/s here; three quarters of the instructions are such,
// the pipe is 55 % busy.  32 streams, 4096 channels, 62.5 ms of 64 MS/s:
// 0.43 ms where 4x4 tiles in registers took 0.76 (22 % against 45 % of the
// shared-memory bandwidth); whole jobs beside their F-step: 32 streams, 1 s,
// 22.6 -> 18.6 ms, 16 streams, 0.5 s, 5.5 -> 4.25 ms.  Two to five small CTAs
// per SM instead of row groups took 5.4 ms on the latter (single-row steps).
constexpr int kRing = 4;
// Rows a thread sums in registers at most; longer sums lose more to rounding, and
// shorter ones cost more flushes.  33 streams, 1952 rows, autocorrelations against
// FP64: 9.4e-8 (1.37e-7 with 256 rows; 1.19e-7 for blocks of about 200 rows of the
// 4x4 tiles), in the mean over 62 shapes 2.5 % of the X-step and 1.2 % of a job.
constexpr int kRun = 128;

// first step of CTA i's share
__device__ __host__ __forceinline__ long long share_begin(long long total, int ctas, int i) { return total * i / ctas; }
// CTA whose share holds step w
__device__ __host__ __forceinline__ int share_of(long long total, int ctas, long long w) {
  int i = (int)(w * ctas / total);
  while (i + 1 < ctas && share_begin(total, ctas, i + 1) <= w) i++;
  while (i > 0 && share_begin(total, ctas, i) > w) i--;
  return i;
}

template <bool DIAG>
__device__ __forceinline__ void tile_row(float2 (&v)[8][8], const float2 *xa, const float2 *xb) {
  float2 a[8], b[8];
#pragma unroll
  for (int p = 0; p < 8; p++) {
    a[p] = xa[p * 32];
    b[p] = xb[p * 32];
  }
#pragma unroll
  for (int p = 0; p < 8; p++)
#pragma unroll
    for (int q = 0; q < 8; q++) {
      float2 &s = v[p][q];
      if (DIAG && p == q) {
        s.x = fmaf(a[p].x, a[p].x, fmaf(a[p].y, a[p].y, s.x));
        s.y = fmaf(b[p].x, b[p].x, fmaf(b[p].y, b[p].y, s.y));
      } else {
        const float2 x = DIAG && p > q ? b[q] : a[p];                        // the lower stream
        const float2 y = !DIAG ? b[q] : p > q ? b[p] : a[q];                 // conjugated
        s.x = fmaf(x.x, y.x, fmaf(x.y, y.y, s.x));
        s.y = fmaf(x.y, y.x, fmaf(-x.x, y.y, s.y));
      }
    }
}

// GROUPS: row groups, 0 for one (with the count a constant 1 the compiler's code
// for that case was 3 to 6 % slower)
template <int THREADS, int GROUPS>
__global__ void __launch_bounds__(THREADS, 1) xcorr_tile8_kernel(const __grid_constant__ TileArgs a) {
  extern __shared__ __align__(16) float2 xs[];  // kRing x [R rows][np8 streams][32 channels]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = GROUPS > 0 ? GROUPS : a.groups;
  const int wu = warp % a.units_per_part, wg = warp / a.units_per_part;  // unit of the part, row group
  const int stage = a.R * a.np8 * 32, rstride = a.np8 * 32;
  const int gstep = a.R / G;
  const int run = max(1, kRun * G / a.R);
  const long long total = (long long)a.nct * a.nparts * a.nsteps;
  const long long w0 = share_begin(total, gridDim.x, blockIdx.x), w1 = share_begin(total, gridDim.x, blockIdx.x + 1);
  // staging: thread's 16-byte piece (two channels) of streams st0, st0 + dst, ...
  const int st0 = threadIdx.x >> 4, dst_st = blockDim.x >> 4, cc = (threadIdx.x & 15) * 2;
  const uint32_t ring0 = tc::smem_u32(xs + st0 * 32 + cc);
  const int64_t sstride = (int64_t)a.nrows_total * a.kpad;
  for (long long w = w0; w < w1;) {
    const int col = (int)(w / a.nsteps), s0 = (int)(w % a.nsteps);
    const int ns = (int)min(min((long long)(a.nsteps - s0), w1 - w), (long long)run);
    const int ct = col / a.nparts, part = col % a.nparts;
    const int unit = part * a.units_per_part + wu;
    const int2 u = unit < a.nunits ? a.units[unit] : make_int2(-1, -1);
    const bool diag = u.y < 0;  // tiles u.x and -u.y - 2 (-1: none)
    const int ta = u.x, tb = diag ? (u.y < -1 ? -u.y - 2 : u.x) : u.y;
    const int k = ct * 32 + lane;
    // channel kk + 1 may be K, which lies inside the padded row (kpad >= K + 3)
    const bool kok = ct * 32 + cc < a.K;
    const float2 *const src0 = a.spec + (int64_t)st0 * sstride + ct * 32 + cc;
    // a step stages R / G rows of each row group, from the group's stretch of ns R / G;
    // row rr of group g in slot rr G + g
    const int gspan = ns * gstep;
    const int64_t gstride = gspan * (int64_t)a.kpad;
    auto issue = [&](int step) {
      if (step < ns) {
        const int row0 = s0 * a.R + step * gstep;
        uint32_t d0 = ring0 + (uint32_t)((step % kRing) * stage) * 8u;
        const float2 *p0 = src0 + (int64_t)row0 * a.kpad;
        for (int st = st0; st < a.np8; st += dst_st) {
          const bool ok = kok && st < a.nstreams;
          const float2 *p = p0;
          uint32_t d = d0;
          if constexpr (GROUPS > 0) {
            for (int rr = 0; rr < gstep; rr++) {
              const float2 *q = p;
#pragma unroll
              for (int g = 0; g < GROUPS; g++) {
                const bool in = ok && row0 + rr + g * gspan < a.nrows;
                tc::cp_async16(d, in ? q : a.spec, in ? 16 : 0);
                q += gstride;
                d += rstride * 8;
              }
              p += a.kpad;
            }
          } else {
            for (int rr = 0; rr < a.R; rr++) {
              const bool in = ok && row0 + rr < a.nrows;
              tc::cp_async16(d, in ? p : a.spec, in ? 16 : 0);
              p += a.kpad;
              d += rstride * 8;
            }
          }
          p0 += dst_st * sstride;
          d0 += dst_st * 256;
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");  // possibly empty: keeps the group count per step
    };
#pragma unroll 1
    for (int s = 0; s < kRing - 1; s++) issue(s);
    float2 v[8][8];
#pragma unroll
    for (int p = 0; p < 8; p++)
#pragma unroll
      for (int q = 0; q < 8; q++) v[p][q] = make_float2(0.f, 0.f);
    // the ring's rows as this warp reads them (rows past the end are zeros).
    // The warps of a CTA take different ones of the three loops below, so they
    // meet at a named barrier, which counts the warps that arrive wherever they
    // are in the code; __syncthreads() in a branch has to be reached by the whole
    // block.  (One loop for all, the branch behind its barrier, was 4 % slower at
    // 96 streams, 3 % at 56, the same up to 48.)
    const GroupSync meet{1, (int)blockDim.x};
    auto rows = [&](auto tile) {
#pragma unroll 1
      for (int step = 0; step < ns; step++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
        meet();  // step's rows are in; every thread is done with the slot refilled next
        issue(step + kRing - 1);
        const float2 *x = xs + (step % kRing) * stage + wg * rstride + lane;
#pragma unroll 1
        for (int rr = wg; rr < a.R; rr += G, x += G * rstride) tile(x + ta * 256, x + tb * 256);
      }
    };
    if (ta < 0)
      rows([&](const float2 *, const float2 *) {});
    else if (diag)
      rows([&](const float2 *xa, const float2 *xb) { tile_row<true>(v, xa, xb); });
    else
      rows([&](const float2 *xa, const float2 *xb) { tile_row<false>(v, xa, xb); });
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the ring is free
    // the row groups' tiles added up pairwise, in a fixed order, into group 0's
    for (int h = 1; h < G; h *= 2) {
      float2 *area = xs + ((wg / (2 * h)) * a.units_per_part + wu) * 2048 + lane;
      if (wg % (2 * h) == h) {
#pragma unroll
        for (int p = 0; p < 64; p++) area[p * 32] = v[p / 8][p % 8];
      }
      __syncthreads();
      if (wg % (2 * h) == 0 && wg + h < G) {
#pragma unroll
        for (int p = 0; p < 64; p++) {
          const float2 y = area[p * 32];
          float2 &x = v[p / 8][p % 8];
          x = make_float2(x.x + y.x, x.y + y.y);
        }
      }
      __syncthreads();
    }
    if (ta >= 0 && wg == 0 && k < a.K) {
      // the column's first CTA writes slot 0, the next slot 1, ...; a column in
      // one share goes straight to the accumulators (their only writer)
      const int slot = blockIdx.x - share_of(total, gridDim.x, (long long)col * a.nsteps);
      float2 *const dst = a.part ? a.part + (int64_t)slot * a.nbl * a.kpad : a.acc;
      // the destination holds an earlier sum: the accumulators, or this share's earlier run of the column
      const bool add = !a.part || (s0 > 0 && w > w0);
      auto put = [&](int i, int j, float2 x) {
        if (i >= a.npad || j >= a.npad) return;
        const int m = __ldg(a.blmap + i * a.npad + j);
        if (m < 0) return;
        float2 *o = dst + (int64_t)(m >> 1) * a.kpad + k;
        if (m & 1) x.y = -x.y;
        // (the entry's only writer: the adds land in program order, and the
        // thread does not wait for them)
        if (add)
          atomicAdd(o, x);
        else
          *o = x;
      };
#pragma unroll
      for (int p = 0; p < 8; p++)
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const float2 x = v[p][q];
          if (!diag) {
            put(8 * ta + p, 8 * tb + q, x);
          } else if (p == q) {
            put(8 * ta + p, 8 * ta + p, make_float2(x.x, 0.f));
            if (tb != ta) put(8 * tb + p, 8 * tb + p, make_float2(x.y, 0.f));
          } else if (p < q) {
            put(8 * ta + p, 8 * ta + q, x);
          } else if (tb != ta) {
            put(8 * tb + q, 8 * tb + p, x);
          }
        }
    }
    w += ns;
  }
}

// Partial sums of the columns' shares into the accumulators, in share order.
__global__ void tile8_reduce_kernel(const float2 *__restrict__ part, const int *__restrict__ blpart, int nparts,
                                    int nsteps, long long total, int ctas, int nbl, int kpad, int K,
                                    float2 *__restrict__ acc) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (k >= K) return;
  const long long col = (long long)(k / 32) * nparts + __ldg(blpart + b);
  const int n = share_of(total, ctas, (col + 1) * nsteps - 1) - share_of(total, ctas, col * nsteps) + 1;
  float2 s = acc[(int64_t)b * kpad + k];
  for (int r = 0; r < n; r++) {
    const float2 x = part[((int64_t)r * nbl + b) * kpad + k];
    s = make_float2(s.x + x.x, s.y + x.y);
  }
  acc[(int64_t)b * kpad + k] = s;
}

struct TilePlan {
  int warps, groups, nparts, upp, R, ctas, nct, nsteps, slots;
  size_t smem;
  long long total;
};
TilePlan tile_plan(int nunits, int nstreams, int K, int nrows) {
  TilePlan p{};
  const int np8 = (nstreams + 7) / 8 * 8, row = np8 * 256;
  // up to eight units (one warp each, 220 registers a thread) per CTA and one CTA
  // per SM; with one or two units, eight or four groups of rows.  Five or six
  // units (17 to 24, 41 to 48 streams) leave the four schedulers one warp here
  // and two there, so these take two groups too, in 10 or 12 warps of 168
  // registers (21 words spilled): 20 streams, 4096 channels, 0.2 s of 32 MS/s 0.764
  // -> 0.727 ms, 16384 channels 0.817 -> 0.795 (4x4 register tiles 0.764); 48 streams,
  // 1024 channels, 83 ms 1.18 -> 1.07 (1.78).  Past 64 streams a step of two rows is
  // more than its 32 KB.
  p.nparts = (nunits + 7) / 8;
  p.upp = (nunits + p.nparts - 1) / p.nparts;
  p.groups = p.upp == 1 ? 8 : p.upp == 2 ? 4 : p.upp <= 4 || (p.upp <= 6 && 2 * row <= 32768) ? 2 : 1;
  p.warps = p.upp * p.groups;
  p.R = std::max(p.groups, 32768 / row / p.groups * p.groups);
  p.smem = std::max((size_t)kRing * p.R * row, p.groups > 1 ? (size_t)p.groups / 2 * p.upp * 16384 : 0);
  p.nct = (K + 31) / 32;
  p.nsteps = (nrows + p.R - 1) / p.R;
  p.total = (long long)p.nct * p.nparts * p.nsteps;
  // a share of at least eight steps, or the partial sums outweigh the work
  p.ctas = (int)std::max<long long>(1, std::min<long long>(sm_count(), p.total / 8));
  p.slots = 1;
  for (long long c = 0; c < (long long)p.nct * p.nparts; c++)
    p.slots = std::max(p.slots, share_of(p.total, p.ctas, (c + 1) * p.nsteps - 1) - share_of(p.total, p.ctas, c * p.nsteps) + 1);
  return p;
}

}  // namespace

std::vector<int2> tile8_units(const std::vector<int> &blmap, int npad, int nstreams, std::vector<int> &blpart, int nbl) {
  const int T = (nstreams + 7) / 8;
  auto used = [&](int I, int J) {
    for (int i = 8 * I; i < std::min(8 * I + 8, npad); i++)
      for (int j = std::max(i, 8 * J); j < std::min(8 * J + 8, npad); j++)
        if (blmap[(size_t)i * npad + j] >= 0) return true;
    return false;
  };
  std::vector<int2> units;
  for (int I = 0; I < T; I++)
    for (int J = I + 1; J < T; J++)
      if (used(I, J)) units.push_back(make_int2(I, J));
  for (int I = 0; I < T; I += 2) units.push_back(make_int2(I, I + 1 < T ? -(I + 1) - 2 : -1));
  // the part (of at most eight units) each baseline's sums come from
  const int nparts = ((int)units.size() + 7) / 8, upp = ((int)units.size() + nparts - 1) / nparts;
  blpart.assign(nbl, 0);
  for (size_t u = 0; u < units.size(); u++) {
    auto mark = [&](int I, int J) {
      for (int i = 8 * I; i < std::min(8 * I + 8, npad); i++)
        for (int j = std::max(i, 8 * J); j < std::min(8 * J + 8, npad); j++) {
          const int m = blmap[(size_t)i * npad + j];
          if (m >= 0) blpart[m >> 1] = (int)u / upp;
        }
    };
    if (units[u].y >= 0) {
      mark(units[u].x, units[u].y);
    } else {
      mark(units[u].x, units[u].x);
      if (units[u].y < -1) mark(-units[u].y - 2, -units[u].y - 2);
    }
  }
  return units;
}

size_t xcorr_f32_scratch_bytes(int nunits, int nstreams, int K, int nrows, int nbl, int kpad) {
  if (nrows <= 0 || nunits <= 0) return 0;
  const TilePlan p = tile_plan(nunits, nstreams, K, nrows);
  return p.slots > 1 ? (size_t)p.slots * nbl * kpad * sizeof(float2) : 0;
}

cudaError_t launch_xcorr_f32(const float2 *spec, int nrows_total, int kpad, int nstreams, int npad, int nrows, int K,
                             const int2 *units, int nunits, const int *blmap, const int *blpart, int nbl, float2 *acc,
                             float2 *scratch, size_t scratch_bytes, cudaStream_t st) {
  if (nrows <= 0 || K <= 0 || nunits <= 0) return cudaSuccess;
  const TilePlan p = tile_plan(nunits, nstreams, K, nrows);
  if (p.slots > 1 && scratch_bytes < (size_t)p.slots * nbl * kpad * sizeof(float2)) return cudaErrorInvalidValue;
  TileArgs a;
  a.spec = spec;
  a.nrows_total = nrows_total;
  a.kpad = kpad;
  a.nstreams = nstreams;
  a.np8 = (nstreams + 7) / 8 * 8;
  a.npad = npad;
  a.nrows = nrows;
  a.K = K;
  a.units = units;
  a.nunits = nunits;
  a.units_per_part = p.upp;
  a.nparts = p.nparts;
  a.groups = p.groups;
  a.nct = p.nct;
  a.nsteps = p.nsteps;
  a.R = p.R;
  a.blmap = blmap;
  a.nbl = nbl;
  a.acc = acc;
  a.part = p.slots > 1 ? scratch : nullptr;
  auto kern = p.warps > 8     ? xcorr_tile8_kernel<384, 2>
              : p.groups == 1 ? xcorr_tile8_kernel<256, 0>
              : p.groups == 2 ? xcorr_tile8_kernel<256, 2>
              : p.groups == 4 ? xcorr_tile8_kernel<256, 4>
                              : xcorr_tile8_kernel<256, 8>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
  kern<<<p.ctas, p.warps * 32, p.smem, st>>>(a);
  if (a.part)
    tile8_reduce_kernel<<<dim3((K + 255) / 256, nbl), 256, 0, st>>>(scratch, blpart, p.nparts, p.nsteps, p.total, p.ctas,
                                                                    nbl, kpad, K, acc);
  return cudaGetLastError();
}

}  // namespace sfxc
