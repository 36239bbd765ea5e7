// F-step, stage 2 (Delay_correction::do_task, sfxc/src/delay_correction.cc:57-75):
// window, sideband flip, real FFT of rot = 2N samples per output row as an
// N-point complex FFT of (x[2e], x[2e+1]), the real-FFT split and the channel
// selection, written in the FP32 or the tensor-core spectra layout.
#include <algorithm>
#include <cstdio>

#include "device.cuh"
#include "fft_pack.cuh"
#include "kernels.hpp"
#include "tc_ptx.cuh"

namespace sfxc {
namespace {

// A group of T = N/NV threads transforms one row of NS = 2 S streams at a
// time, two streams per packed transform; groups synchronise only themselves
// and each runs over its own rows.  The real-FFT split pairs bins k and
// N - k: after the last pass thread t holds the bins t + T m, and the threads
// are dealt so that t and T - t sit in one warp sixteen lanes apart, so the
// split is a register shuffle and each thread makes both bins of its pairs
// (no trip through shared memory) for all its streams: with S = 2 the
// 32-byte piece of the tensor-core layout.
//
// NV = 16 (from 2048 points): a row's samples come by bulk copy into the
// transform buffers while the previous row is split and written.  NV = 8
// (up to 1024 points): many small groups, which hide each other's loads.
// 8192 points (LONG): one packed pair fills the shared memory, so a CTA takes
// two streams (16-byte pieces) and reads the window through the cache: the
// streams of 8192 points of a 40-stream job, 976 rows of 4096 channels, 1.07 ->
// 0.78 ms against one group of threads per stream.  16384 points:
// window_long_kernel.
//
// What bounds it: 42 instructions per point (73.5 with scalar FP32 and the
// split through shared memory) and 59 bytes of shared-memory and L1 traffic
// per point, by warps few enough (8 to 16 per SM, the transforms fill the
// registers and 213 KB of shared memory) that latency counts.  Measured at 32
// streams, against the one-stream-per-thread form with three trips through
// shared memory: 4096 channels, tensor-core layout, 0.5 s of 64 MS/s 3.78 ->
// 3.25 ms (3.8 TB/s of algorithmic traffic; 2.7 ms without its copies and
// stores), FP32 layout, 1 s, 6.43 -> 5.27 ms (two groups per CTA, out of step
// with each other; four streams in one group 6.60); 256 channels (16 uneven
// streams, 0.25 s) 0.55 -> 0.31 ms, where NV = 16 with bulk copies took 0.85
// (many small copies) and with register loads 0.37.  The tensor-core layout
// with NV = 8 took 4.2 ms at 4096 channels, with the next row's samples in
// registers 4.1 (the loads queue behind the row's stores).
template <int LOGN, int OUT_TC>
struct PackWin {
  static constexpr int NV = LOGN <= 10 ? 8 : 16;
  static constexpr bool BULK = NV == 16;
  using F = PackShape<LOGN, NV>;
  static constexpr int N = F::N, T = F::T;
  static constexpr bool LONG = LOGN == 13;
  static constexpr int S = (OUT_TC && !LONG) || !BULK ? 2 : 1, NS = 2 * S;
  static constexpr int THREADS = BULK && S == 2 ? 256 : 512;
  static_assert(T >= 32 && T <= THREADS, "whole warps");
  static constexpr int GROUPS = THREADS / T;
  static constexpr int BUF = S * F::ELEMS;  // one group's buffer, float4
  static constexpr size_t SMEM = (size_t)GROUPS * BUF * 16 + ((size_t)F::tw_len() + (LONG ? 0 : N) + N / 2 + 1) * 8;
};

// FP16 hi and lo parts of both lanes of a complex pair (packed conversions)
__device__ __forceinline__ void tc_split(cpair x, uint2 &a, uint2 &b) {
  const __half2 ha = __floats2half2_rn(x.re.x, x.im.x), hb = __floats2half2_rn(x.re.y, x.im.y);
  const float2 fa = __half22float2(ha), fb = __half22float2(hb);
  const float2 lr = sub2(x.re, make_float2(fa.x, fb.x)), li = sub2(x.im, make_float2(fa.y, fb.y));
  const __half2 la = __floats2half2_rn(lr.x, li.x), lb = __floats2half2_rn(lr.y, li.y);
  a = make_uint2(*reinterpret_cast<const unsigned *>(&ha), *reinterpret_cast<const unsigned *>(&la));
  b = make_uint2(*reinterpret_cast<const unsigned *>(&hb), *reinterpret_cast<const unsigned *>(&lb));
}

__device__ __forceinline__ float2 shfl2(float2 v, int src) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// OUT_TC: 0 writes the FP32 layout, 32 or 64 the tensor-core layout with that many slots
template <int LOGN, int OUT_TC>
__global__ void __launch_bounds__(PackWin<LOGN, OUT_TC>::THREADS, 1)
    window_pack_kernel(const StreamDev *__restrict__ streams, int nstreams, int row0, int nrows, int nrows_total,
                       int rows_per_group, const float *__restrict__ window, const float2 *__restrict__ tw_rot,
                       int nper, int M, int kpad, void *__restrict__ spec_out, float tc_scale, int *__restrict__ err) {
  using W = PackWin<LOGN, OUT_TC>;
  using F = typename W::F;
  constexpr int N = W::N, T = W::T, S = W::S, NS = W::NS, NV = W::NV, GROUPS = W::GROUPS;
  extern __shared__ __align__(16) float4 psm[];
  const int g = threadIdx.x / T, t = threadIdx.x % T, lane = threadIdx.x & 31;
  const int nsg = (nstreams + NS - 1) / NS;
  const int s0 = (blockIdx.x % nsg) * NS;  // first stream; stream group fastest
  const int nv = min(NS, nstreams - s0);
  // the group's rows k0, k0 + KS, ...: a run of its own, or, for the short
  // rows of NV = 8, every GROUPS-th row of the CTA's run (neighbouring groups
  // then share their half rows in the cache)
  constexpr int KS = W::BULK ? 1 : GROUPS;
  const int c0 = (blockIdx.x / nsg) * GROUPS * rows_per_group;
  const int k0 = W::BULK ? c0 + g * rows_per_group : c0 + g;
  const int k1 = min(nrows, W::BULK ? k0 + rows_per_group : c0 + GROUPS * rows_per_group);
  // every window but NONE covers the whole transform input
  const bool full = nper == 2 * N;

  float4 *buf = psm + g * W::BUF;
  float2 *tab = reinterpret_cast<float2 *>(psm + GROUPS * W::BUF);
  float2 *wsm = tab + F::tw_len();           // window, N float2
  float2 *twr = wsm + (W::LONG ? 0 : N);     // exp(-2 pi i q / 2N), q <= N/2
  fill_pack_table<LOGN, NV>(tab, tw_rot + 2 * N, threadIdx.x, W::THREADS);
  // the window carries the tensor-core layout's power-of-two scale and the split's 1/2 (both exact)
  const float ws = (OUT_TC ? tc_scale : 1.0f) * 0.5f;
  if (!W::LONG) {
    for (int i = threadIdx.x; i < N; i += W::THREADS) {
      const float2 w = __ldg(reinterpret_cast<const float2 *>(window) + i);
      wsm[i] = make_float2(w.x * ws, w.y * ws);
    }
  }
  for (int i = threadIdx.x; i <= N / 2; i += W::THREADS) twr[i] = __ldg(tw_rot + i);
  // the CTA's streams: source, channel shift, slot and sign of the odd samples
  // (a stream in the other sideband has them negated)
  __shared__ const float *ssrc[NS];
  __shared__ int2 sinfo[NS];
  __shared__ float ssgn[NS];
  __shared__ uint64_t bar[W::BULK ? GROUPS : 1][S];
  if (threadIdx.x < NS) {
    const StreamDev &s = streams[s0 + min((int)threadIdx.x, nv - 1)];
    ssrc[threadIdx.x] = s.ts + (int64_t)row0 * N;
    sinfo[threadIdx.x] = make_int2(s.output_offset - s.temp_fft_offset, s.slot);
    ssgn[threadIdx.x] = s.flip != 0 ? -1.f : 1.f;
  }
  if (W::BULK && t == 0) {
#pragma unroll
    for (int s = 0; s < S; s++) tc::mbar_init(&bar[g][s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int shift0 = sinfo[0].x, slot0 = sinfo[0].y;
  const int64_t fstride = (int64_t)nrows_total * kpad;  // FP32 layout: from one slot to the next
  bool flip = false, fast = nv == NS && (OUT_TC == 0 || (slot0 & (NS - 1)) == 0);
#pragma unroll
  for (int j = 0; j < NS; j++) {
    flip = flip || ssgn[j] < 0.f;
    // consecutive slots (whole 32-byte pieces), all shifted alike
    fast = fast && sinfo[j].y == slot0 + j && sinfo[j].x == shift0;
  }

  // thread of the last pass: t and T - t sixteen lanes apart in one warp
  // (0 and T/2 pair with themselves)
  const int wl = t & 15, ww = t >> 5;
  const int tl = (t & 16) == 0 ? 16 * ww + wl : (ww == 0 && wl == 0 ? T / 2 : T - 16 * ww - wl);
  const int partner = tl == 0 || tl == T / 2 ? lane : lane ^ 16;
  auto sync = [&] {
    if constexpr (T == W::THREADS)
      __syncthreads();
    else if constexpr (T > 32)
      GroupSync{1 + g, T}();
    else
      __syncwarp();
  };

  // The samples of row k of the run by bulk copies into the transform buffer
  // of their own pair (the pair's first stream at float2 0, the second at N),
  // issued once the previous row's last pass has read that buffer; the half
  // row after them is fetched into L2 on the way.
  const float2 *rawb = reinterpret_cast<const float2 *>(buf);
  const uint32_t row_bytes = (uint32_t)nper * 4;
  int lost = -1;  // the row whose copies did not arrive in time: reported, no further copies
  auto issue = [&](int k, int s) {
    const int n = min(2, nv - 2 * s);
    if (!W::BULK || t != 0 || k >= k1 || lost >= 0 || n <= 0) return;
    tc::mbar_expect_tx(&bar[g][s], n * row_bytes);
    for (int j = 0; j < n; j++) {
      const float *src = ssrc[2 * s + j] + k * (int64_t)N;
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       tc::smem_u32(rawb + s * 2 * F::ELEMS + j * N)),
                   "l"(src), "r"(row_bytes), "r"(tc::smem_u32(&bar[g][s]))
                   : "memory");
      if (k + 1 < k1)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src + nper), "r"(4 * N) : "memory");
    }
  };
  auto landed = [&](int k, int s) {
    if (lost >= 0 || 2 * s >= nv) return;
    if (!tc::mbar_wait(&bar[g][s], (uint32_t)(k - k0) & 1)) {
      atomicExch(err, 1);
      lost = k;
    }
  };
  // NV = 8: the samples straight into registers
  auto load_pair = [&](float2(&x)[2][NV], int k, int s) {
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const bool ok = k < k1 && 2 * s + j < nv;
      const float2 *src = reinterpret_cast<const float2 *>(ssrc[2 * s + j] + k * (int64_t)N) + t;
#pragma unroll
      for (int q = 0; q < NV; q++) x[j][q] = ok && (q < NV / 2 || full) ? src[q * T] : make_float2(0.f, 0.f);
    }
  };
  // pair s of row k, windowed and transformed over the first digit
  auto windowed = [&](cpair(&v)[NV], const float2(&x)[2][NV], int s) {
#pragma unroll
    for (int q = 0; q < NV; q++) {
      float2 w;
      if constexpr (W::LONG) {
        w = __ldg(reinterpret_cast<const float2 *>(window) + t + q * T);
        w = make_float2(w.x * ws, w.y * ws);
      } else {
        w = wsm[t + q * T];
      }
      v[q].re = make_float2(x[0][q].x * w.x, x[1][q].x * w.x);
      v[q].im = make_float2(x[0][q].y * w.y, x[1][q].y * w.y);
    }
    if (flip) {
#pragma unroll
      for (int q = 0; q < NV; q++) v[q].im = mul2(v[q].im, make_float2(ssgn[2 * s], ssgn[2 * s + 1]));
    }
    dftn(v);
  };

  // the thread's lowest and highest channel of a row (both then in steps of T)
  const int chl = tl - shift0, chh = N - tl - shift0;
  const int offl = OUT_TC ? (int)tc_index(0, kpad, chl, slot0, OUT_TC) : chl;
  const int offh = OUT_TC ? (int)tc_index(0, kpad, chh, slot0, OUT_TC) : chh;
  constexpr int STEP = OUT_TC ? T * OUT_TC : T;  // T: a multiple of the four channels of a line

  float2 x0[2][NV];  // NV = 8: the next row's first pair
  if constexpr (W::BULK) {
#pragma unroll
    for (int s = 0; s < S; s++) issue(k0, s);
  } else {
    load_pair(x0, k0, 0);
  }
#pragma unroll 1
  for (int k = k0; k < k1; k += KS) {
    {
      cpair v[S][NV];
      if constexpr (W::BULK) {
#pragma unroll
        for (int s = 0; s < S; s++) {
          landed(k, s);
          const float2 *src = rawb + s * 2 * F::ELEMS + t;
          float2 x[2][NV];
#pragma unroll
          for (int q = 0; q < NV; q++)
#pragma unroll
            for (int j = 0; j < 2; j++)
              x[j][q] = (q < NV / 2 || full) && 2 * s + j < nv ? src[j * N + q * T] : make_float2(0.f, 0.f);
          windowed(v[s], x, s);
        }
      } else {
        float2 x1[2][NV];
        load_pair(x1, k, 1);
        windowed(v[0], x0, 0);
        windowed(v[S - 1], x1, 1);
      }
      pack_first<LOGN>(v, buf, tab, t, sync);
    }
    sync();
    if constexpr (F::NMID >= 1) {
      pack_middle<LOGN, S, NV, 1>(buf, tab, t);
      sync();
    }
    if constexpr (F::NMID >= 2) {
      pack_middle<LOGN, S, NV, 2>(buf, tab, t);
      sync();
    }
    cpair z[S][NV];
#pragma unroll
    for (int s = 0; s < S; s++) {
      pack_last<LOGN>(z[s], buf + s * F::ELEMS, tl);
      if constexpr (W::BULK) {  // once every thread has read a pair's buffer, the next row's samples may come
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        sync();
        issue(k + 1, s);
      }
    }
    // the upper bins go to the partner; thread 0 pairs T m with T (NV - m)
    // and has the middle bin N/2 = (NV/2) T to itself
    cpair zmid[S];
#pragma unroll
    for (int s = 0; s < S; s++) zmid[s] = z[s][NV / 2];
    if (t < 32) {
#pragma unroll
      for (int s = 0; s < S; s++) {
        const cpair z0 = z[s][0];
        if (tl == 0) {
#pragma unroll
          for (int m = NV / 2; m < NV - 1; m++) z[s][m] = z[s][m + 1];
          z[s][NV - 1] = z0;
        }
      }
    }
    uint2 *trow = reinterpret_cast<uint2 *>(spec_out) + (int64_t)(row0 + k) * kpad * (OUT_TC ? OUT_TC : 1) +
                  (OUT_TC ? 0 : slot0 * fstride);
    // bin q of every stream of the row to channel q - shift; ch, off: channel
    // and offset within the row where all streams go together
    auto store = [&](int q, int ch, int off, const cpair(&x)[S]) {
      uint2 o[NS];
#pragma unroll
      for (int s = 0; s < S; s++) {
        if constexpr (OUT_TC != 0) {
          tc_split(x[s], o[2 * s], o[2 * s + 1]);
        } else {
          o[2 * s] = make_uint2(__float_as_uint(x[s].re.x), __float_as_uint(x[s].im.x));
          o[2 * s + 1] = make_uint2(__float_as_uint(x[s].re.y), __float_as_uint(x[s].im.y));
        }
      }
      if (fast) {
        if ((unsigned)ch > (unsigned)M) return;
        if constexpr (OUT_TC == 0) {
#pragma unroll
          for (int j = 0; j < NS; j++) trow[off + j * fstride] = o[j];
        } else if constexpr (NS == 2) {
          *reinterpret_cast<uint4 *>(trow + off) = make_uint4(o[0].x, o[0].y, o[1].x, o[1].y);
        } else {
          asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(trow + off), "r"(o[0].x), "r"(o[0].y),
                       "r"(o[1].x), "r"(o[1].y), "r"(o[NS - 2].x), "r"(o[NS - 2].y), "r"(o[NS - 1].x),
                       "r"(o[NS - 1].y)
                       : "memory");
        }
        return;
      }
#pragma unroll
      for (int j = 0; j < NS; j++) {
        const int2 si = sinfo[j];
        const int c = q - si.x;
        if (j >= nv || (unsigned)c > (unsigned)M) continue;
        if constexpr (OUT_TC == 0) {
          trow[(si.y - slot0) * fstride + c] = o[j];
        } else {
          // 16-byte pieces of two streams where their slots allow it
          if (j % 2 == 0 && j + 1 < nv && (si.y & 1) == 0 && sinfo[j + 1].x == si.x && sinfo[j + 1].y == si.y + 1)
            *reinterpret_cast<uint4 *>(trow + tc_index(0, kpad, c, si.y, OUT_TC)) =
                make_uint4(o[j].x, o[j].y, o[j + 1].x, o[j + 1].y);
          else if (j % 2 == 0 || (si.y & 1) == 0 || sinfo[j - 1].x != si.x || sinfo[j - 1].y != si.y - 1)
            trow[tc_index(0, kpad, c, si.y, OUT_TC)] = o[j];
        }
      }
    };
    // X[q] = E + O w, X[N - q] = conj(E - O w), E and O from Z[q] and conj Z[N - q]
    auto split = [&](float2 w, const cpair(&zk)[S], const cpair(&zc)[S], cpair(&xq)[S], cpair(&xn)[S]) {
#pragma unroll
      for (int s = 0; s < S; s++) {
        const float2 er = add2(zk[s].re, zc[s].re), ei = sub2(zk[s].im, zc[s].im);
        const cpair o = {add2(zk[s].im, zc[s].im), sub2(zc[s].re, zk[s].re)};
        const cpair ow = mulw(o, w);
        xq[s] = {add2(er, ow.re), add2(ei, ow.im)};
        xn[s] = {sub2(er, ow.re), sub2(ow.im, ei)};
      }
    };
    float2 w = twr[tl];
#pragma unroll
    for (int m = 0; m < NV / 2; m++) {
      const int q = tl + T * m;
      const float2 wm = w;
      if (m + 1 < NV / 2) w = twr[q + T];  // ahead of this bin's stores
      cpair zk[S], zc[S], xq[S], xn[S];
#pragma unroll
      for (int s = 0; s < S; s++) {
        zk[s] = z[s][m];
        zc[s] = {shfl2(z[s][NV - 1 - m].re, partner), shfl2(z[s][NV - 1 - m].im, partner)};
      }
      split(wm, zk, zc, xq, xn);
      store(q, chl + T * m, offl + STEP * m, xq);
      store(N - q, chh - T * m, offh - STEP * m, xn);
      if constexpr (!W::BULK)
        if (m == 0) load_pair(x0, k + KS, 0);
    }
    if (t < 32 && tl == 0) {
      cpair xq[S], xn[S];
      split(twr[N / 2], zmid, zmid, xq, xn);
      store(N / 2, chl + NV / 2 * T, offl + NV / 2 * STEP, xq);
    }
  }
  if (W::BULK && lost >= 0) {  // bounded; nothing lands after the CTA has gone
#pragma unroll
    for (int s = 0; s < S; s++)
      if (2 * s < nv) tc::mbar_wait(&bar[g][s], (uint32_t)(lost - k0) & 1);
  }
  // channels outside a stream's bins (a stream that covers part of the band)
#pragma unroll 1
  for (int j = 0; j < nv; j++) {
    const StreamDev &s = streams[s0 + j];
    const int sh = s.output_offset - s.temp_fft_offset, sl = s.slot;
    if (sh >= 0 && sh + M <= N) continue;
#pragma unroll 1
    for (int r = k0; r < k1; r += KS)
      for (int ch = t; ch <= M; ch += T) {
        if ((unsigned)(ch + sh) <= (unsigned)N) continue;
        if constexpr (OUT_TC != 0)
          reinterpret_cast<uint2 *>(spec_out)[tc_index(row0 + r, kpad, ch, sl, OUT_TC)] = make_uint2(0u, 0u);
        else
          reinterpret_cast<float2 *>(spec_out)[((int64_t)sl * nrows_total + row0 + r) * kpad + ch] =
              make_float2(0.f, 0.f);
      }
  }
}

// Rows a group of threads takes in one run, with one CTA per SM, `groups` groups a
// CTA and nsg groups of streams: the CTAs fill `waves` waves (the autotuner's
// count), or by default two, or one where that takes less than `percent` of the
// time, counted in rows with the CTA's start (its tables, the first row's samples)
// as one.  Short runs of few streams gain by one wave (4 streams, 4096 channels,
// 976 rows, one wave of 7 rows a run against two of 4: 0.84 of the time in the
// tensor-core layout, 0.86 in FP32); where the counts are close, two waves even
// out the SMs (32 streams, 8192 points, FP32, 1952 rows: one wave 1.07).
int run_rows(int nsg, int nrows, int groups, int waves, int percent) {
  auto rows = [&](int w) {
    const int ctas = std::max(1, w * sm_count() / nsg);
    return std::max(1, (nrows + ctas * groups - 1) / (ctas * groups));
  };
  auto time = [&](int r) {
    const int grid = nsg * ((nrows + r * groups - 1) / (r * groups));
    return (long long)((grid + sm_count() - 1) / sm_count()) * (r + 1);
  };
  if (waves > 0) return rows(waves);
  return time(rows(1)) * 100 < time(rows(2)) * percent ? rows(1) : rows(2);
}
// From 2048 points on: over 456 shapes (1 to 32 streams, 16 to 125 ms of 32 and 64
// MS/s) 0.932 of two waves' time in the mean, at most 1.04.  The one-stream
// kernel's 8-byte pieces in the tensor-core layout lose up to 5 % in one wave where
// the counts are within a twentieth (24 streams, 488 rows).
constexpr int kOneWave = 97, kOneWaveLongTc = 94;

template <int LOGN, int OUT_TC>
void pack_launch(const StreamDev *d_streams, int nstreams, int row0, int nrows, int nrows_total, const float *window,
                 const float2 *tw_rot, int nper, int M, int kpad, void *spec, float tc_scale, int *err, cudaStream_t st,
                 int waves) {
  using W = PackWin<LOGN, OUT_TC>;
  const int nsg = (nstreams + W::NS - 1) / W::NS;
  const int rows_per_group = run_rows(nsg, nrows, W::GROUPS, waves, W::BULK ? kOneWave : 0);
  const unsigned grid = (unsigned)(nsg * ((nrows + rows_per_group * W::GROUPS - 1) / (rows_per_group * W::GROUPS)));
  auto kern = window_pack_kernel<LOGN, OUT_TC>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W::SMEM);
  kern<<<grid, W::THREADS, W::SMEM, st>>>(d_streams, nstreams, row0, nrows, nrows_total, rows_per_group, window, tw_rot,
                                          nper, M, kpad, spec, tc_scale, err);
}

// 16384 points: one stream of a row fills the shared memory, so the two packed
// lanes are its transform's even and odd points, z[2n] and z[2n+1], in the
// 8192-point passes; with P[k] = (A, B) their transforms, Z[k] = A + W^k B and
// Z[k + 8192] = A - W^k B (W = exp(-2 pi i / 16384)).  The thread that holds
// P[k] gets P[8192 - k] from its partner, and the four bins of Z that come of
// them, k, 16384 - k, 8192 - k and 8192 + k, are two pairs of the real split,
// which again fill the two lanes.
//
// Bound: in the tensor-core layout the 8-byte pieces of one stream (a partial
// sector costs the L2 as much as a whole one); without them the chain of five
// passes of 16 warps in step.  24 streams, 0.5 s of 64 MS/s: tensor-core layout
// 5.53 -> 5.18 ms (5.49 with the whole window loaded after the samples have
// landed), FP32 layout 3.55 -> 3.60 ms, against one scalar transform of 1024
// threads.
constexpr int kLongN = 16384;
struct LongWin {
  using F = PackShape<13, 16>;
  static constexpr int N = F::N, T = F::T, THREADS = T;
  static constexpr size_t SMEM = (size_t)F::ELEMS * 16 + ((size_t)F::tw_len() + N / 2 + 1) * 8;
};

template <int OUT_TC>
__global__ void __launch_bounds__(LongWin::THREADS, 1)
    window_long_kernel(const StreamDev *__restrict__ streams, int nstreams, int row0, int nrows, int nrows_total,
                       int rows_per_group, const float *__restrict__ window, const float2 *__restrict__ tw_rot,
                       int nper, int M, int kpad, void *__restrict__ spec_out, float tc_scale, int *__restrict__ err) {
  using F = LongWin::F;
  constexpr int N = LongWin::N, T = LongWin::T, NV = 16;
  extern __shared__ __align__(16) float4 psm[];
  const int t = threadIdx.x, lane = t & 31;
  const StreamDev &sd = streams[blockIdx.x % nstreams];  // stream fastest
  const int k0 = (blockIdx.x / nstreams) * rows_per_group, k1 = min(nrows, k0 + rows_per_group);
  const bool full = nper == 2 * kLongN;

  float4 *buf = psm;
  float2 *tab = reinterpret_cast<float2 *>(psm + F::ELEMS);
  float2 *twr = tab + F::tw_len();  // exp(-2 pi i q / 32768), q <= 4096
  fill_pack_table<13, NV>(tab, tw_rot + 2 * kLongN, t, T, 2);
  for (int i = t; i <= N / 2; i += T) twr[i] = __ldg(tw_rot + i);
  const float ws = (OUT_TC ? tc_scale : 1.0f) * 0.5f;
  __shared__ uint64_t bar;
  if (t == 0) {
    tc::mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const float *src = sd.ts + (int64_t)row0 * kLongN;
  const int shift = sd.output_offset - sd.temp_fft_offset, slot = sd.slot;
  // window scale of the even and of the odd samples (a stream in the other sideband has these negated)
  const float wse = ws, wso = sd.flip != 0 ? -ws : ws;

  const int wl = t & 15, ww = t >> 5;
  const int tl = (t & 16) == 0 ? 16 * ww + wl : (ww == 0 && wl == 0 ? T / 2 : T - 16 * ww - wl);
  const int partner = tl == 0 || tl == T / 2 ? lane : lane ^ 16;

  const uint32_t row_bytes = (uint32_t)nper * 4;
  int lost = -1;  // the row whose copy did not arrive in time: reported, no further copies
  auto issue = [&](int k) {
    if (t != 0 || k >= k1 || lost >= 0) return;
    const float *p = src + k * (int64_t)kLongN;
    tc::mbar_expect_tx(&bar, row_bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     tc::smem_u32(buf)),
                 "l"(p), "r"(row_bytes), "r"(tc::smem_u32(&bar))
                 : "memory");
    if (k + 1 < k1)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p + nper), "r"(4 * kLongN) : "memory");
  };
  // offsets of the thread's channels tl + T m, N - tl - T m, N + tl + T m and
  // 2 N - tl - T m of a row at m = 0
  int ch[4], off[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    ch[i] = (i & 1 ? -tl : tl) + (i == 0 ? 0 : i == 3 ? 2 * N : N) - shift;
    off[i] = OUT_TC ? (int)tc_index(0, kpad, ch[i], slot, OUT_TC) : ch[i];
  }
  constexpr int STEP = OUT_TC ? T * OUT_TC : T;

  issue(k0);
#pragma unroll 1
  for (int k = k0; k < k1; k++) {
    {
      cpair v[1][NV];
      float4 w0[NV / 2];  // the window of the first half, on its way while the samples land
#pragma unroll
      for (int q = 0; q < NV / 2; q++) w0[q] = __ldg(reinterpret_cast<const float4 *>(window) + t + q * T);
      if (lost < 0 && !tc::mbar_wait(&bar, (uint32_t)(k - k0) & 1)) {
        atomicExch(err, 1);
        lost = k;
      }
#pragma unroll
      for (int q = 0; q < NV; q++) {
        if (q < NV / 2 || full) {
          const float4 w = q < NV / 2 ? w0[q % (NV / 2)] : __ldg(reinterpret_cast<const float4 *>(window) + t + q * T);
          const float4 x = buf[t + q * T];
          v[0][q].re = make_float2(x.x * (w.x * wse), x.z * (w.z * wse));
          v[0][q].im = make_float2(x.y * (w.y * wso), x.w * (w.w * wso));
        } else {
          v[0][q] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        }
      }
      dftn(v[0]);
      pack_first<13>(v, buf, tab, t, [] { __syncthreads(); });
    }
    __syncthreads();
    pack_middle<13, 1, NV, 1>(buf, tab, t);
    __syncthreads();
    pack_middle<13, 1, NV, 2>(buf, tab, t);
    __syncthreads();
    cpair z[NV];
    pack_last<13>(z, buf, tl);
    // once every thread has read the buffer, the next row's samples may come
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    issue(k + 1);
    // the upper half goes to the partner; thread 0 pairs T m with T (16 - m)
    // and has the middle, N/2 = 8 T, to itself
    const cpair zmid = z[NV / 2];
    if (t < 32) {
      const cpair z0 = z[0];
      if (tl == 0) {
#pragma unroll
        for (int m = NV / 2; m < NV - 1; m++) z[m] = z[m + 1];
        z[NV - 1] = z0;
      }
    }
    uint2 *trow = reinterpret_cast<uint2 *>(spec_out) +
                  (OUT_TC ? (int64_t)(row0 + k) * kpad * OUT_TC : ((int64_t)slot * nrows_total + row0 + k) * kpad);
    auto store = [&](int c, int o, float re, float im) {
      if ((unsigned)c > (unsigned)M) return;
      if constexpr (OUT_TC != 0) {
        const __half2 h = __floats2half2_rn(re, im);
        const float2 f = __half22float2(h);
        const __half2 l = __floats2half2_rn(re - f.x, im - f.y);
        trow[o] = make_uint2(*reinterpret_cast<const unsigned *>(&h), *reinterpret_cast<const unsigned *>(&l));
      } else {
        trow[o] = make_uint2(__float_as_uint(re), __float_as_uint(im));
      }
    };
    // P[b] and P[8192 - b], w = exp(-2 pi i b / 32768), u = w^2 = W^b -> bins
    // b, 16384 - b (first lane), 8192 - b, 8192 + b (second); the first of a
    // lane is E + O w, the second conj(E - O w), the second lane's w -i conj(w)
    auto bins = [&](cpair a, cpair c, float2 w, float2 u, cpair &xq, cpair &xn) {
      const cpair A = {make_float2(a.re.x, c.re.x), make_float2(a.im.x, c.im.x)};
      const cpair B = {make_float2(a.re.y, c.re.y), make_float2(a.im.y, c.im.y)};
      // W^b B of the first lane, W^(8192 - b) B = -conj(W^b) B of the second
      const float2 ux = make_float2(u.x, -u.x);
      const cpair tw = {fma2(B.re, ux, mul2(B.im, dup2(-u.y))), fma2(B.re, dup2(u.y), mul2(B.im, ux))};
      const cpair zk = A + tw, d = A - tw;
      const cpair zc = {make_float2(d.re.y, d.re.x), make_float2(d.im.y, d.im.x)};
      const float2 er = add2(zk.re, zc.re), ei = sub2(zk.im, zc.im);
      const cpair o = {add2(zk.im, zc.im), sub2(zc.re, zk.re)};
      const float2 wx = make_float2(w.x, -w.y), wy = make_float2(w.y, -w.x), ny = make_float2(-w.y, w.x);
      const cpair ow = {fma2(o.re, wx, mul2(o.im, ny)), fma2(o.re, wy, mul2(o.im, wx))};
      xq = {add2(er, ow.re), add2(ei, ow.im)};
      xn = {sub2(er, ow.re), sub2(ow.im, ei)};
    };
    const float2 *w14 = tw_rot + 2 * kLongN;
    float2 u = __ldg(w14 + tl);
#pragma unroll
    for (int m = 0; m < NV / 2; m++) {
      const float2 um = u;
      if (m + 1 < NV / 2) u = __ldg(w14 + tl + T * (m + 1));
      const cpair zc = {shfl2(z[NV - 1 - m].re, partner), shfl2(z[NV - 1 - m].im, partner)};
      cpair xq, xn;
      bins(z[m], zc, twr[tl + T * m], um, xq, xn);
      store(ch[0] + T * m, off[0] + STEP * m, xq.re.x, xq.im.x);
      store(ch[3] - T * m, off[3] - STEP * m, xn.re.x, xn.im.x);
      store(ch[1] - T * m, off[1] - STEP * m, xq.re.y, xq.im.y);
      store(ch[2] + T * m, off[2] + STEP * m, xn.re.y, xn.im.y);
    }
    if (t < 32 && tl == 0) {  // b = 8192 - b
      cpair xq, xn;
      bins(zmid, zmid, twr[N / 2], __ldg(w14 + N / 2), xq, xn);
      store(ch[0] + T * NV / 2, off[0] + STEP * NV / 2, xq.re.x, xq.im.x);
      store(ch[3] - T * NV / 2, off[3] - STEP * NV / 2, xn.re.x, xn.im.x);
    }
  }
  if (lost >= 0) tc::mbar_wait(&bar, (uint32_t)(lost - k0) & 1);  // bounded; nothing lands after the CTA has gone
  // channels outside the stream's bins (a stream that covers part of the band)
  if (shift >= 0 && shift + M <= kLongN) return;
#pragma unroll 1
  for (int r = k0; r < k1; r++)
    for (int c = t; c <= M; c += T) {
      if ((unsigned)(c + shift) <= (unsigned)kLongN) continue;
      if constexpr (OUT_TC != 0)
        reinterpret_cast<uint2 *>(spec_out)[tc_index(row0 + r, kpad, c, slot, OUT_TC)] = make_uint2(0u, 0u);
      else
        reinterpret_cast<float2 *>(spec_out)[((int64_t)slot * nrows_total + row0 + r) * kpad + c] =
            make_float2(0.f, 0.f);
    }
}

template <int OUT_TC>
void long_launch(const StreamDev *d_streams, int nstreams, int row0, int nrows, int nrows_total, const float *window,
                 const float2 *tw_rot, int nper, int M, int kpad, void *spec, float tc_scale, int *err, cudaStream_t st,
                 int waves) {
  const int rows_per_group = run_rows(nstreams, nrows, 1, waves, OUT_TC ? kOneWaveLongTc : kOneWave);
  const unsigned grid = (unsigned)(nstreams * ((nrows + rows_per_group - 1) / rows_per_group));
  auto kern = window_long_kernel<OUT_TC>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LongWin::SMEM);
  kern<<<grid, LongWin::THREADS, LongWin::SMEM, st>>>(d_streams, nstreams, row0, nrows, nrows_total, rows_per_group,
                                                      window, tw_rot, nper, M, kpad, spec, tc_scale, err);
}

}  // namespace

void launch_window_fft(const StreamDev *d_streams, int nstreams, int row0, int nrows, int nrows_total,
                       const float *window, const float2 *tw_rot, int rot, int nper, int M, int kpad, void *spec,
                       int tc_slots, float tc_scale, int *err, cudaStream_t st, int waves) {
#define SFXC_WINDOW(points, launch, ...)                                                                         \
  case 2 * points:                                                                                             \
    if (tc_slots == kTcSlots)                                                                                  \
      launch<__VA_ARGS__ kTcSlots>(d_streams, nstreams, row0, nrows, nrows_total, window, tw_rot, nper, M, kpad,   \
                                   spec, tc_scale, err, st, waves);                                               \
    else if (tc_slots == kTcSlotsWide)                                                                         \
      launch<__VA_ARGS__ kTcSlotsWide>(d_streams, nstreams, row0, nrows, nrows_total, window, tw_rot, nper, M,     \
                                       kpad, spec, tc_scale, err, st, waves);                                     \
    else                                                                                                       \
      launch<__VA_ARGS__ 0>(d_streams, nstreams, row0, nrows, nrows_total, window, tw_rot, nper, M, kpad, spec,    \
                            tc_scale, err, st, waves);                                                            \
    break;
#define SFXC_COMMA ,
  switch (rot) {
    SFXC_WINDOW(256, pack_launch, 8 SFXC_COMMA)
    SFXC_WINDOW(512, pack_launch, 9 SFXC_COMMA)
    SFXC_WINDOW(1024, pack_launch, 10 SFXC_COMMA)
    SFXC_WINDOW(2048, pack_launch, 11 SFXC_COMMA)
    SFXC_WINDOW(4096, pack_launch, 12 SFXC_COMMA)
    SFXC_WINDOW(8192, pack_launch, 13 SFXC_COMMA)
    SFXC_WINDOW(16384, long_launch, )
    default: break;  // sizes outside 2^9..2^15 samples are rejected by set_parameters
  }
#undef SFXC_COMMA
#undef SFXC_WINDOW
}

}  // namespace sfxc
