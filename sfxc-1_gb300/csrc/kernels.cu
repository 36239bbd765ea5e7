// CUDA kernels of the correlator-node path (sm_103a).
//
//   block_params_kernel  per-block FP64 delay and fringe parameters of the F-step's
//                        block stage (fstep.cu).
//   bitstat_kernel       per-code sample counts with cal-diode on/off split, from
//                        popcounts (bit_statistics.cc:36-47, bit2float_worker.cc:341-346).
//   pulsar_bins_kernel / xcorr_f32_kernel  bin per (FFT, channel) in FP64 and binned
//                        accumulation on CUDA cores (correlation_core_pulsar.cc:210-238).
//   norm_* kernels       Correlation_core::integration_normalize (275-314).
#include <algorithm>
#include <cstdio>

#include "device.cuh"
#include "kernels.hpp"

namespace sfxc {

// ------------------------------------------------------------------------
// Per-block FP64 parameters of the F-step, one thread per 256-sample block
// (all lanes busy on the reduced-rate FP64 pipe).  Follows
// Delay_correction::do_task / fractional_bit_shift / fringe_stopping
// (sfxc/src/delay_correction.cc:40-47, 97-103, 139-160): the integer and
// fractional delay at the block centre, the fringe phase at the block start
// and its linear step over the block, the amplitude at the centre.  The
// phases leave FP64 only after reduction to one turn.
__device__ __forceinline__ void block_params_one(const StreamDev &s, int bl, int lane);

// CTAs of 128 blocks, strided over the stream's blocks when the grid is
// smaller than the stream (a capped grid leaves room on the SMs to a
// kernel running beside it).
__global__ void __launch_bounds__(128) block_params_kernel(const StreamDev *__restrict__ streams) {
  const StreamDev &s = streams[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (int base = blockIdx.x * blockDim.x; base < s.n_blocks; base += gridDim.x * blockDim.x) {
    // whole warps stay (neighbour exchange below); lanes past the end compute
    // their block's times (the spline extrapolates) and store nothing
    if (base + (int)(threadIdx.x & ~31) >= s.n_blocks) break;
    block_params_one(s, base + threadIdx.x, lane);
  }
}

__device__ __forceinline__ void block_params_one(const StreamDev &s, int bl, int lane) {
  constexpr double kInvTick = 1.0 / 512000000.0, kInv2Pi = 0.15915494309189533577;
  const int64_t ct = s.start_ticks + (int64_t)(s.block0 + bl) * kNd * s.tps;
  // node intervals: the times grow with the block, so each is walked forward
  // from the launch's first interval (or from the previous time's)
  auto tsec = [&s](int64_t t) { return (double)(t - s.scan_begin) * kInvTick; };
  auto delay = [&s](int64_t t, double v, int i) {
    const double r = spline_eval_at(s.spline, s.spline_n, 0, v, i);
    return s.no_clock ? r : r + (s.clock_offset + (double)(t - s.clock_epoch) * kInvTick * s.clock_rate);
  };
  auto phase = [&s](double v, int i) { return s.phase_zero ? 0.0 : spline_eval_at(s.spline, s.spline_n, 1, v, i); };
  const double v0 = tsec(ct), vc = tsec(ct + s.half_len_ticks);
  const int i0 = spline_walk(s.spline, s.spline_n, v0, s.spline_lo);
  const int ic = spline_walk(s.spline, s.spline_n, vc, i0);
  const double delay_c = delay(ct + s.half_len_ticks, vc, ic);
  const double delay_0 = delay(ct, v0, i0);
  const double phase_0 = phase(v0, i0);
  // the end of a block is the start of the next when a block is a whole
  // number of ticks: take it from the next lane
  const bool chained = s.fft_len_ticks == (int64_t)kNd * s.tps;
  double delay_1 = __shfl_down_sync(0xffffffffu, delay_0, 1);
  double phase_1 = __shfl_down_sync(0xffffffffu, phase_0, 1);
  if (!chained || lane == 31) {
    const double v1 = tsec(ct + s.fft_len_ticks);
    const int i1 = spline_walk(s.spline, s.spline_n, v1, ic);
    delay_1 = delay(ct + s.fft_len_ticks, v1, i1);
    phase_1 = phase(v1, i1);
  }
  if (bl >= s.n_blocks) return;
  const double ampl = s.amp_one ? 1.0 : spline_eval_at(s.spline, s.spline_n, 2, vc, ic);
  const double dis = __dmul_rn(delay_c, (double)s.sample_rate);
  const int integer_delay = (int)floor(__dadd_rn(dis, 0.5));
  // the fractional-delay ramp (phase at bin 0 and step per bin) is stored in
  // FP32 and needs no more: |frac| <= 1/2, the terms stay within a few turns
  const float frac = (float)(dis - integer_delay);
  const float tmp1 = frac * s.frac_scale_f;
  const float tmp2 = (float)(integer_delay & (4 * s.oversamp - 1)) * s.int_phase_q_f;
  const float cterm = tmp2 - tmp1 * s.half_bw_f;  // half turns, as all phases of the record
  const float lterm = tmp1 * s.rate_per_bin_f;
  // the fringe phase in FP64 (tens of millions of turns); a zero LO offset or
  // phase model adds exact zeros, skipped
  double phi = s.center_freq * delay_0, phi_end = s.center_freq * delay_1;
  if (s.lo_offset != 0.0) {
    const double lo_phase = s.start_phase + s.lo_offset * ((double)(ct - s.start_ticks) * kInvTick);
    phi = phi + lo_phase;
    phi_end = phi_end + lo_phase + s.fft_len_sec * s.lo_offset;
  } else {
    phi = phi + s.start_phase;
    phi_end = phi_end + s.start_phase;
  }
  if (!s.phase_zero) {
    phi = phi + phase_0 * kInv2Pi;
    phi_end = phi_end + phase_1 * kInv2Pi;
  }
  const double turns = rint(phi);
  phi = s.fringe_mult * (phi - turns);
  phi_end = s.fringe_mult * (phi_end - turns);
  BlockPar bp;
  bp.ph = make_float4(cterm - 2.0f * rintf(0.5f * cterm), lterm, (float)phi,
                      (float)((phi_end - phi) * (1.0 / kNd)));
  sincospif(16.0f * bp.ph.y, &bp.steps.y, &bp.steps.x);
  sincospif(16.0f * bp.ph.w, &bp.steps.w, &bp.steps.z);
  bp.amp = (float)ampl;
  // unpack source of the pair (bl, bl + 1) when both lie in one recorded segment
  const int o0 = (s.block0 + bl) * kNd;
  bp.seg = find_segment(s, o0);
  const DevSegment sg = s.segs[bp.seg];
  bp.src_bit = (bl + 1 < s.n_blocks && sg.src_bit >= 0 && o0 >= sg.out0 && o0 + 2 * kNd <= sg.out0 + sg.n)
                   ? sg.src_bit + (long long)(o0 - sg.out0) * s.bits
                   : -1;
  s.bpar[bl] = bp;
}

// Channel extraction: output byte `ob` of subband s packs spb = 8/fan_out
// samples (extract_byte); sample j reads word ob*spb+j.
__global__ void extract_kernel(const uint8_t *__restrict__ in, int64_t nout, int N, int bits, int fan_out,
                               const int *__restrict__ tracks, uint8_t *__restrict__ out) {
  const int64_t ob = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int sb = blockIdx.y;
  if (ob >= nout) return;
  out[(int64_t)sb * nout + ob] = extract_byte(in + ob * (8 / fan_out) * N, N, bits, fan_out, tracks + sb * fan_out);
}

// ------------------------------------------------------------------------
// Bit statistics.
// Code counts of 8 bits (mask 0x55) or 32 bits (mask 0x55555555): 2-bit
// codes -> c[code] with code = 2 * high bit + low bit; 1-bit -> c[bit value].
__device__ __forceinline__ void count_codes(uint32_t x, int nbits, int bits, uint32_t (&c)[4]) {
  if (bits == 2) {
    const uint32_t m = nbits == 32 ? 0x55555555u : 0x55u;
    const uint32_t lo = x & m, hi = (x >> 1) & m;
    c[3] = __popc(hi & lo);
    c[2] = __popc(hi & ~lo & m);
    c[1] = __popc(~hi & lo & m);
    c[0] = nbits / 2 - c[1] - c[2] - c[3];
  } else {
    c[1] = __popc(nbits == 32 ? x : x & 0xFFu);
    c[0] = nbits - c[1];
    c[2] = c[3] = 0;
  }
}

// Cal-diode state over increasing counted-byte indices: toggles at t0,
// t0 + period, ... (once when period <= 0, never when t0 <= 0).  at() places
// the walker with one division, advance() steps it forward without any.
struct CalWalk {
  int on;
  int64_t next, period;
  __device__ __forceinline__ void at(const StreamDev &s, int64_t c) {
    on = 1;
    next = INT64_MAX;
    period = s.tsys_period;
    if (s.tsys_two_bit) {
      on = s.tsys_on0;
      if (s.tsys_t0 > 0) {
        if (c >= s.tsys_t0) {
          const int64_t flips = period > 0 ? 1 + (c - s.tsys_t0) / period : 1;
          on ^= (int)(flips & 1);
          next = period > 0 ? s.tsys_t0 + flips * period : INT64_MAX;
        } else {
          next = s.tsys_t0;
        }
      }
    }
  }
  __device__ __forceinline__ void advance(int64_t c) {
    while (c >= next) {
      on ^= 1;
      next = period > 0 ? next + period : INT64_MAX;
    }
  }
};

struct CodeCounts {
  uint32_t on[4], off[4];
  __device__ __forceinline__ void add(uint32_t x, int nbits, int bits, int cal_on) {
    uint32_t c[4];
    count_codes(x, nbits, bits, c);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      on[k] += cal_on ? c[k] : 0u;
      off[k] += cal_on ? 0u : c[k];
    }
  }
};

// Code counts of the counted bytes src[0, n) (counted index cfirst + j for
// src[j]) by a group of NL threads: bytes before the first 16-byte boundary
// and after the last one singly, the middle as 16-byte loads (four in flight
// per thread) counted a word at a time unless a cal-diode toggle falls
// inside the word.
template <int NL>
__device__ __forceinline__ void count_span(const StreamDev &s, const uint8_t *src, int n, int64_t cfirst, int lane,
                                           CodeCounts &cc) {
  const int bits = s.bits;
  const int head = min(n, (int)((16 - ((uintptr_t)src & 15)) & 15));
  const int nvec = (n - head) / 16;
  const int tail0 = head + 16 * nvec;
  for (int j = lane; j < head + (n - tail0); j += NL) {
    const int pos = j < head ? j : tail0 + (j - head);
    CalWalk w;
    w.at(s, cfirst + pos);
    cc.add(__ldg(src + pos), 8, bits, w.on);
  }
  if (lane >= nvec) return;
  const uint4 *vsrc = reinterpret_cast<const uint4 *>(src + head);
  const int64_t cvec = cfirst + head;
  CalWalk w;
  w.at(s, cvec + 16 * (int64_t)lane);
  for (int q0 = lane; q0 < nvec; q0 += 4 * NL) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int q = q0 + u * NL;
      v[u] = q < nvec ? __ldg(vsrc + q) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int q = q0 + u * NL;
      if (q >= nvec) break;
      const int64_t c0 = cvec + 16 * (int64_t)q;
      w.advance(c0);
      const uint32_t ww[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
      if (c0 + 16 <= w.next) {
#pragma unroll
        for (int k = 0; k < 4; k++) cc.add(ww[k], 32, bits, w.on);
      } else {
        for (int b = 0; b < 16; b++) {
          w.advance(c0 + b);
          cc.add((ww[b >> 2] >> (8 * (b & 3))) & 0xFFu, 8, bits, w.on);
        }
      }
    }
  }
}

// Bit statistics over the counted-byte ranges, as per-code counts split by
// the cal-diode state: s.hist[0..3] on, [4..7] off (the byte histogram of
// bit_statistics.cc:36-47 enters the levels and tsys values only through
// these counts).  Work items (stream, first range, range count, offset):
// range count > 0 packs that many short ranges, one warp per range; range
// count 0 is the 64 KB piece at `offset` of one long range, all warps.
__global__ void __launch_bounds__(256) bitstat_kernel(const StreamDev *__restrict__ streams,
                                                     const int4 *__restrict__ items, int nitems) {
  const int4 it = items[blockIdx.x];
  const StreamDev &s = streams[it.x];
  CodeCounts cc = {{0, 0, 0, 0}, {0, 0, 0, 0}};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (it.z > 0) {
    for (int r = it.y + warp; r < it.y + it.z; r += blockDim.x >> 5) {
      const DevStatRange rg = s.stats[r];
      count_span<32>(s, s.src + rg.src_byte, rg.n, rg.cidx, lane, cc);
    }
  } else {
    const DevStatRange rg = s.stats[it.y];
    const int n = min(65536, rg.n - it.w);
    count_span<256>(s, s.src + rg.src_byte + it.w, n, (int64_t)rg.cidx + it.w, threadIdx.x, cc);
  }
  // warp sums, one global update per counter and warp
#pragma unroll
  for (int k = 0; k < 4; k++) {
    uint32_t a = cc.on[k], b = cc.off[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      if (a) atomicAdd(&s.hist[k], (unsigned long long)a);
      if (b) atomicAdd(&s.hist[4 + k], (unsigned long long)b);
    }
  }
}

// ------------------------------------------------------------------------
// X-step on CUDA cores with pulsar binning (Correlation_core_pulsar::
// integration_step, sfxc/src/correlation_core_pulsar.cc:101-146; without
// bins: xcorr_f32.cu).
// spec: [stream][row][kpad] complex64.  Work items -- (32-channel tile, part
// of the stream-pair tiles) -- are dealt to persistent CTAs.  A
// CTA stages R rows x npad streams x 32 channels per step through a 4-deep
// cp.async ring (one barrier per R rows), so the loads of three steps are in
// flight while one is multiplied; each thread owns one channel and up to TPW
// tiles of 4x4 stream pairs (i in tile row I, j in tile column J, I <= J) in
// registers, and adds them to acc[bin] with float2 atomics when its channel's
// pulsar bin changes and when its item ends.
// blmap[i*npad+j] gives (baseline << 1 | conj) or -1.
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

template <int TPW>
__global__ void __launch_bounds__(384, 1) xcorr_f32_kernel(const __grid_constant__ F32Args a) {
  extern __shared__ __align__(16) float2 xs[];  // kF32Stages x [R rows][npad streams][32 channels]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int nct = (a.K + 31) / 32;
  const int nitems = nct * a.nparts;
  const int stage_f2 = a.R * a.npad * 32;  // float2 per stage
  const int chunks = a.R * a.npad * 16;    // 16-byte copies per stage
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int part = item % a.nparts, ct = item / a.nparts;
    const int k = ct * 32 + lane;
    const int rz = a.nrows;
    const int t_end = min(a.ntiles, (part + 1) * a.tiles_per_part);
    int ti[TPW], tj[TPW];
    float2 v[TPW][4][4];
#pragma unroll
    for (int t = 0; t < TPW; t++) {
      const int tile = part * a.tiles_per_part + warp + t * nwarps;
      ti[t] = tile < t_end ? a.tiles[2 * tile] : -1;
      tj[t] = tile < t_end ? a.tiles[2 * tile + 1] : -1;
#pragma unroll
      for (int p = 0; p < 4; p++)
#pragma unroll
        for (int q = 0; q < 4; q++) v[t][p][q] = make_float2(0.f, 0.f);
    }
    // add the register tiles to acc[bin] and clear them.  Each (bin, baseline,
    // channel) entry has one writer thread per launch, so the results do not
    // depend on timing.
    auto flush = [&](int bin) {
      if (k >= a.K || bin < 0) return;
#pragma unroll
      for (int t = 0; t < TPW; t++) {
        if (ti[t] < 0) continue;
#pragma unroll
        for (int p = 0; p < 4; p++)
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int m = __ldg(a.blmap + (ti[t] * 4 + p) * a.npad + tj[t] * 4 + q);
            if (m >= 0) {
              const float2 x = v[t][p][q];
              const float2 y = make_float2(x.x, (m & 1) ? -x.y : x.y);
              // the entry's only writer in this launch: its adds land in
              // program order, so the sum does not depend on timing; the
              // atomic lets the thread go on without waiting for the load
              atomicAdd(a.acc + ((int64_t)bin * a.nbl + (m >> 1)) * a.kpad + k, y);
            }
            v[t][p][q] = make_float2(0.f, 0.f);
          }
      }
    };
    const int nsteps = (rz + a.R - 1) / a.R;
    auto issue = [&](int step) {
      if (step < nsteps) {
        float2 *dst = xs + (step % kF32Stages) * stage_f2;
        const int rs = step * a.R;
        for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
          const int rr = c / (a.npad * 16), rem = c - rr * (a.npad * 16), st = rem >> 4, cc = (rem & 15) * 2;
          const int row = rs + rr, kk = ct * 32 + cc;
          // channel kk + 1 may be K, which lies inside the padded row (kpad >= K + 3)
          const bool ok = row < rz && st < a.nstreams && kk < a.K;
          const float2 *src = ok ? a.spec + ((int64_t)st * a.nrows_total + row) * a.kpad + kk : a.spec;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst + (rr * a.npad + st) * 32 + cc)),
                       "l"(src), "r"(ok ? 16 : 0)
                       : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");  // possibly empty: keeps the group count per step
    };
#pragma unroll 1
    for (int s = 0; s < kF32Stages - 1; s++) issue(s);
    int cur = -1;
#pragma unroll 1
    for (int step = 0; step < nsteps; step++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kF32Stages - 2) : "memory");
      __syncthreads();  // step's rows are in; every thread is done with the slot refilled next
      issue(step + kF32Stages - 1);
      const float2 *xst = xs + (step % kF32Stages) * stage_f2;
#pragma unroll 1
      for (int rr = 0; rr < a.R; rr++) {
        const int row = step * a.R + rr;
        if (row >= rz) break;
        const int bin = k < a.K ? __ldg(a.bins + (int64_t)k * a.nrows + row) : -1;
        if (bin != cur) {
          flush(cur);
          cur = bin;
        }
        const float2 *xr = xst + rr * a.npad * 32 + lane;
#pragma unroll
        for (int t = 0; t < TPW; t++) {
          if (ti[t] < 0) continue;
          float2 xi[4], xj[4];
#pragma unroll
          for (int p = 0; p < 4; p++) {
            xi[p] = xr[(ti[t] * 4 + p) * 32];
            xj[p] = xr[(tj[t] * 4 + p) * 32];
          }
#pragma unroll
          for (int p = 0; p < 4; p++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
              // x_i * conj(x_j)
              v[t][p][q].x = fmaf(xi[p].x, xj[q].x, fmaf(xi[p].y, xj[q].y, v[t][p][q].x));
              v[t][p][q].y = fmaf(xi[p].y, xj[q].x, fmaf(-xi[p].x, xj[q].y, v[t][p][q].y));
            }
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    flush(cur);
    __syncthreads();  // the ring is refilled by the next item
  }
}

// ------------------------------------------------------------------------
// Pulsar bins (Correlation_core_pulsar::dedisperse_buffer) in FP64, evaluated
// with the reference's operation order so that every bin matches; written
// [channel][row] (row fastest) for the per-channel sort and the binned X-steps.
// A thread per row takes kBinChans channels: the row's own phase (a division)
// is computed once for all of them, and the division by the gate's length is
// left out when that is 1, where it changes nothing.  Bound by the FP64 pipe:
// 16 M bins 1.83 -> 1.19 ms, and it runs
// beside the F-step.
constexpr int kBinChans = 16;
__global__ void __launch_bounds__(128) pulsar_bins_kernel(int nrows, int K, double start_phase, double rate_term,
                                                          double fft_duration, const double *__restrict__ offsets,
                                                          double g0, double g1, int nbins, int16_t *__restrict__ bins) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrows) return;
  const double us_per_day = 86400000000.0;
  // start_phase + (coef[1] + 60 F0) * fft_duration * current_fft * 1440 / us_per_day
  double ph = __dmul_rn(rate_term, fft_duration);
  ph = __dmul_rn(ph, (double)r);
  ph = __dmul_rn(ph, 1440.0);
  ph = __ddiv_rn(ph, us_per_day);
  ph = __dadd_rn(start_phase, ph);
  const double len = __dsub_rn(g1, g0), scale = (double)(nbins - 1);
  const bool whole = len == 1.0;
  const int k1 = min(K, (int)(blockIdx.y + 1) * kBinChans);
  for (int k = blockIdx.y * kBinChans; k < k1; k++) {
    double p = __dsub_rn(ph, __ldg(offsets + k));
    p = __dsub_rn(p, floor(p));
    const double p1 = __dadd_rn(p, 1.0);
    int bin = 0;
    if (p >= g0 ? p < g1 : p1 < g1) {
      double x = __dmul_rn(__dsub_rn(p >= g0 ? p : p1, g0), scale);
      if (!whole) x = __ddiv_rn(x, len);
      bin = (int)x + 1;
    }
    bins[(int64_t)k * nrows + r] = (int16_t)bin;
  }
}

// ------------------------------------------------------------------------
// Normalisation.  norms[i] = max(1, sum_k Re acc[auto_i][k] / M) in FP64.
__global__ void norm_autos_kernel(const float2 *__restrict__ acc, int kpad, int M, int nstreams, int nbl,
                                  double *norms) {
  __shared__ double red[256];
  const int i = blockIdx.x;
  acc += ((int64_t)blockIdx.y * nbl + i) * kpad;
  double s = 0.0;
  for (int k = threadIdx.x; k <= M; k += blockDim.x) s += (double)acc[k].x;
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double n = red[0] / M;
    norms[blockIdx.y * nstreams + i] = n < 1 ? 1 : n;
  }
}

// Output z (a pulsar bin or phase centre; accumulators and norms one after
// another): M + 1 normalised channels of baseline b at out + z out_stride + b
// bl_stride bytes, which may lie on 4-byte boundaries only (the output's
// file layout), so the parts are stored singly; flagfac[b] = N1*N2 (crosses).
// A cross baseline's FP64 norm is the same for all its channels: one thread
// of the CTA (all of whose threads share the baseline) computes it.
__global__ void normalize_kernel(const float2 *__restrict__ acc, int kpad, int M, int nstreams, int nbl,
                                 const int *__restrict__ bl, const double *__restrict__ norms,
                                 const double *__restrict__ flagfac, uint8_t *__restrict__ out, size_t out_stride,
                                 size_t bl_stride) {
  const int b = blockIdx.y;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  acc += (int64_t)blockIdx.z * nbl * kpad;
  norms += (int64_t)blockIdx.z * nstreams;
  __shared__ float cross_norm;
  if (b >= nstreams && threadIdx.x == 0)
    cross_norm = (float)sqrt(flagfac[b] * norms[bl[2 * b]] * norms[bl[2 * b + 1]]);
  __syncthreads();
  if (k > M) return;
  const float2 v = acc[(int64_t)b * kpad + k];
  float2 o;
  if (b < nstreams) {
    o = make_float2((float)((double)v.x / norms[b]), 0.f);
  } else {
    const float norm = cross_norm;
    o = make_float2(v.x / norm, v.y / norm);
  }
  float *d = reinterpret_cast<float *>(out + blockIdx.z * out_stride + b * bl_stride) + 2 * k;
  d[0] = o.x;
  d[1] = o.y;
}

// ------------------------------------------------------------------------
// Phased array: Correlation_core_phased::integration_step (sfxc/src/
// correlation_core_phased.cc:113-126) -- each FFT's spectra of all streams
// added, in stream order, to the buffer of its sub-integration; one thread
// per channel keeps the running sum of the current buffer in registers.
__global__ void phased_kernel(const float2 *__restrict__ spec, int nrows_total, int kpad, int nstreams, int r0,
                              int nrows, int K, int nsub, float2 *__restrict__ acc) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K || nrows <= 0) return;
  int s = r0 / nsub;
  float2 sum = acc[(size_t)s * kpad + k];
  for (int r = 0; r < nrows; r++) {
    const int sr = (r0 + r) / nsub;
    if (sr != s) {
      acc[(size_t)s * kpad + k] = sum;
      s = sr;
      sum = acc[(size_t)s * kpad + k];
    }
    for (int i = 0; i < nstreams; i++) {
      const float2 x = spec[((size_t)i * nrows_total + r) * kpad + k];
      sum = make_float2(sum.x + x.x, sum.y + x.y);
    }
  }
  acc[(size_t)s * kpad + k] = sum;
}

// ------------------------------------------------------------------------
// Extra phase centres: Correlation_core::sub_integration (sfxc/src/
// correlation_core.cc:516-559) with uvshift (561-593).  Every channel of
// every baseline of the sub-integration goes to each centre's accumulator;
// a cross baseline of centre c >= 1 first gets the amplitude and the phase
// phi + k delta of its residual delay (FP64 angle, FP32 product, as the
// reference's FP64 recurrence and complex<float> arithmetic).
//
// A thread takes kPcChans channels, kPcThreads apart.  Its first channel's
// factor is the FP64 product of two table entries (16 runs of 8 channels, 8
// channels of a run), the next ones follow by an FP64 rotation of kPcThreads
// steps; the CTA computes the tables' sines and cosines, 25 a centre, five
// centres at once.  At most 16 products of rounding 1e-16 each, far below the
// FP32 product.  Bound by the FP64 pipe: 16 centres, 120 cross baselines, 2048
// channels 217 -> 120 us a sub-integration (a sine and cosine per channel
// before; one per thread and centre 150).
constexpr int kPcThreads = 128, kPcChans = 16, kPcTab = 25, kPcBatch = kPcThreads / kPcTab;
__global__ void __launch_bounds__(kPcThreads) pc_dump_kernel(float2 *__restrict__ acc, float2 *__restrict__ pcacc,
                                                             const UvShift *__restrict__ uvp, int nstreams, int nbl,
                                                             int kpad, int K, int npc) {
  // of the next centres: exp(i (phi + (first channel + 8 e) delta)), e < 16;
  // exp(i e delta), e < 8; exp(i kPcThreads delta)
  __shared__ double2 tab[kPcBatch][kPcTab];
  const int t = threadIdx.x, k0 = blockIdx.x * kPcThreads * kPcChans + t, b = blockIdx.y;
  const size_t i0 = (size_t)b * kpad + k0, cstride = (size_t)nbl * kpad;
  const int n = k0 < K ? min(kPcChans, (K - 1 - k0) / kPcThreads + 1) : 0;
  float2 x[kPcChans];
#pragma unroll
  for (int j = 0; j < kPcChans; j++) {
    if (j >= n) break;
    x[j] = acc[i0 + j * kPcThreads];
  }
#pragma unroll
  for (int j = 0; j < kPcChans; j++) {
    if (j >= n) break;
    const float2 y = pcacc[i0 + j * kPcThreads];
    pcacc[i0 + j * kPcThreads] = make_float2(y.x + x[j].x, y.y + x[j].y);
    acc[i0 + j * kPcThreads] = make_float2(0.f, 0.f);
  }
  for (int c0 = 1; c0 < npc; c0 += kPcBatch) {
    const int c1 = min(npc, c0 + kPcBatch);
    if (b >= nstreams) {
      __syncthreads();
      const int tc = t / kPcTab, e = t % kPcTab;
      if (c0 + tc < c1) {
        const UvShift u = uvp[(size_t)(c0 + tc - 1) * nbl + b];
        const double angle = e < 16   ? fma((double)(k0 - t + 8 * e), u.delta, u.phi)
                             : e < 24 ? (e - 16) * u.delta
                                      : kPcThreads * u.delta;
        double sn, cs;
        sincos(angle, &sn, &cs);
        tab[tc][e] = make_double2(cs, sn);
      }
      __syncthreads();
    }
    if (n == 0) continue;
    for (int c = c0; c < c1; c++) {
      float2 *p = pcacc + c * cstride + i0;
      float2 y[kPcChans];  // all on their way together
#pragma unroll
      for (int j = 0; j < kPcChans; j++) y[j] = j < n ? p[j * kPcThreads] : make_float2(0.f, 0.f);
      if (b < nstreams) {
#pragma unroll
        for (int j = 0; j < kPcChans; j++)
          if (j < n) p[j * kPcThreads] = make_float2(y[j].x + x[j].x, y[j].y + x[j].y);
        continue;
      }
      const float amp = (float)uvp[(size_t)(c - 1) * nbl + b].amp;
      const double2 r0 = tab[c - c0][t >> 3], r1 = tab[c - c0][16 + (t & 7)], st = tab[c - c0][24];
      double cs = fma(r0.x, r1.x, -(r0.y * r1.y)), sn = fma(r0.x, r1.y, r0.y * r1.x);
#pragma unroll
      for (int j = 0; j < kPcChans; j++) {
        const float cf = (float)cs, sf = (float)sn, xr = amp * x[j].x, xi = amp * x[j].y;
        if (j < n) p[j * kPcThreads] = make_float2(y[j].x + (xr * cf - xi * sf), y[j].y + (xr * sf + xi * cf));
        const double nc = fma(cs, st.x, -(sn * st.y));
        sn = fma(cs, st.y, sn * st.x);
        cs = nc;
      }
    }
  }
}

// ------------------------------------------------------------------------
// Spectral reduction (number_channels < fft_size_correlation):
// Correlation_core::integration_write, sfxc/src/correlation_core.cc:413-439.
// One CTA per normalised spectrum X[0..M]: optional normalisation to unit
// amplitude, the mask, an unnormalised complex-to-real FFT of 2M points (the
// imaginary parts of DC and Nyquist ignored) as one M-point complex FFT of
// the even and odd lags, the lags folded to 2 nch (lag nch the mean of +-nch),
// the lag window, a real FFT of 2 nch points as one nch-point complex FFT and
// the real split, a division by 2M.  Both transforms are in-place radix-2 in
// shared memory: the work is one spectrum per baseline per integration.

// in-place radix-2 transform of the 2^logn values a[] in bit-reversed order:
// sign -1 forward, +1 backward; twiddles exp(-2 pi i j / len) = tw2M[j 2M / len]
__device__ void smem_fft_radix2(float2 *a, int logn, int sign, const float2 *__restrict__ tw2M, int M) {
  const int n = 1 << logn;
  for (int s = 1; s <= logn; s++) {
    const int len = 1 << s, half = len >> 1, stride = (2 * M) >> s;
    for (int b = threadIdx.x; b < n / 2; b += blockDim.x) {
      const int j = b & (half - 1), i = (b - j) * 2 + j;
      float2 w = __ldg(tw2M + j * stride);
      if (sign > 0) w.y = -w.y;
      const float2 u = a[i], x = a[i + half];
      const float2 v = make_float2(x.x * w.x - x.y * w.y, x.x * w.y + x.y * w.x);
      a[i] = make_float2(u.x + v.x, u.y + v.y);
      a[i + half] = make_float2(u.x - v.x, u.y - v.y);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) reduce_kernel(const float2 *__restrict__ in, int M, int logM, int nch,
                                                     int lognch, const float *__restrict__ mask,
                                                     const float *__restrict__ lagwin, int normalize,
                                                     const float2 *__restrict__ tw2M, int nbl,
                                                     uint8_t *__restrict__ out, size_t out_stride, size_t bl_stride) {
  extern __shared__ __align__(16) float2 rsm[];
  float2 *a = rsm;                                   // M complex
  float *lag = reinterpret_cast<float *>(rsm + M);   // 2 nch lags
  const float2 *X = in + (size_t)blockIdx.x * (M + 1);
  auto load = [&](int k) {
    float2 x = X[k];
    if (normalize) {
      const float m = hypotf(x.x, x.y);
      if (m != 0.0f) x = make_float2(x.x / m, x.y / m);
    }
    const float mk = mask[k];
    return make_float2(x.x * mk, x.y * mk);
  };
  // c2r of 2M points: even lags e = IDFT(X[k] + conj X[M-k]), odd lags
  // o = IDFT((X[k] - conj X[M-k]) e^{i pi k / M}); z = e + i o
  for (int k = threadIdx.x; k < M; k += blockDim.x) {
    float2 xk = load(k), xm = load(M - k);
    if (k == 0) xk.y = xm.y = 0.0f;
    const float2 e = make_float2(xk.x + xm.x, xk.y - xm.y);
    const float2 d = make_float2(xk.x - xm.x, xk.y + xm.y);
    const float2 w = __ldg(tw2M + k);  // exp(-i pi k / M); d * conj(w)
    const float2 o = make_float2(d.x * w.x + d.y * w.y, d.y * w.x - d.x * w.y);
    a[__brev((unsigned)k) >> (32 - logM)] = make_float2(e.x - o.y, e.y + o.x);
  }
  __syncthreads();
  smem_fft_radix2(a, logM, +1, tw2M, M);
  auto lag_at = [&](int q) { return (q & 1) ? a[q >> 1].y : a[q >> 1].x; };  // r[q], q < 2M
  for (int q = threadIdx.x; q < 2 * nch; q += blockDim.x) {
    float v;
    if (q < nch)
      v = lag_at(q);
    else if (q == nch)
      v = (lag_at(nch) + lag_at(2 * M - nch)) / 2;
    else
      v = lag_at(2 * M - nch + (q - nch));
    lag[q] = v * lagwin[q];
  }
  __syncthreads();
  for (int n = threadIdx.x; n < nch; n += blockDim.x)
    a[__brev((unsigned)n) >> (32 - lognch)] = make_float2(lag[2 * n], lag[2 * n + 1]);
  __syncthreads();
  smem_fft_radix2(a, lognch, -1, tw2M, M);
  // r2c split: A[k] = E + W^k O, W = exp(-2 pi i / 2nch) = tw2M[M / nch]
  // spectrum blockIdx.x: baseline of an output, 4-byte aligned as normalize_kernel's
  float *Y = reinterpret_cast<float *>(out + blockIdx.x / nbl * out_stride + blockIdx.x % nbl * bl_stride);
  const float scale = (float)(2 * M);
  for (int k = threadIdx.x; k <= nch; k += blockDim.x) {
    const float2 zk = a[k & (nch - 1)], zc = a[(nch - k) & (nch - 1)];
    const float er = 0.5f * (zk.x + zc.x), ei = 0.5f * (zk.y - zc.y);
    const float orr = 0.5f * (zk.y + zc.y), oi = -0.5f * (zk.x - zc.x);
    const float2 w = __ldg(tw2M + (size_t)k * (M / nch));
    Y[2 * k] = (er + (orr * w.x - oi * w.y)) / scale;
    Y[2 * k + 1] = (ei + (orr * w.y + oi * w.x)) / scale;
  }
}

// ------------------------------------------------------------------------
// launchers
int sm_count() {
  static const int n = [] {  // initialised once, also when contexts are planned from several threads
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    return cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0 ? v : 1;
  }();
  return n;
}

void launch_block_params(const StreamDev *d_streams, int nstreams, int max_blocks, cudaStream_t st,
                         int ctas_per_sm) {
  int x = (max_blocks + 127) / 128;
  if (ctas_per_sm > 0) x = std::max(1, std::min(x, ctas_per_sm * sm_count() / nstreams));
  block_params_kernel<<<dim3(x, nstreams), 128, 0, st>>>(d_streams);
}

void launch_fstep_block(const StreamDev *d_streams, int nstreams, int max_blocks, const float2 *tw256,
                        cudaStream_t st) {
  launch_block_params(d_streams, nstreams, max_blocks, st);
  launch_fstep(d_streams, nstreams, max_blocks, tw256, st, 0);
}

void launch_extract(const uint8_t *in, int64_t nout, int N, int bits, int nsub, int fan_out, const int *tracks,
                    uint8_t *out, cudaStream_t st) {
  extract_kernel<<<dim3((unsigned)((nout + 255) / 256), nsub), 256, 0, st>>>(in, nout, N, bits, fan_out, tracks, out);
}

// ------------------------------------------------------------- phase cal ---
// Phase-cal folding (Input_node_data_writer::do_phasecal,
// sfxc/src/input_node_data_writer.cc:230-312): byte j of run r, data[off + j],
// holds the samples of bins ((bin0 + j) mod pb) * spb + q, q < spb = 8 / bits,
// LSB first, and they go to accumulator row r.row (pb * spb int32 bins).
// Thread t takes every pb-th byte of the run, those of byte-bin t, so that a
// warp reads consecutive bytes, and adds its spb sums once: integer sums, so
// neither the order nor the atomics change the result.
template <int BITS>
__global__ void __launch_bounds__(256) phasecal_kernel(const uint8_t *data, const PcalRun *runs, int pb,
                                                       int32_t *acc) {
  constexpr int SPB = 8 / BITS;
  const PcalRun r = runs[blockIdx.y];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= pb) return;
  int j = t - r.bin0;
  if (j < 0) j += pb;
  int sum[SPB] = {};
  for (; j < r.n; j += pb) {
    const uint32_t v = __ldg(data + r.off + j);
#pragma unroll
    for (int q = 0; q < SPB; q++) {
      // Bit2float / do_phasecal sample values: 2-bit {-7, -2, 2, 7}, 1-bit {-5, 5}
      if (BITS == 2)
        sum[q] += (int)(int8_t)(uint8_t)(0x0702FEF9u >> (8 * ((v >> (2 * q)) & 3)));
      else
        sum[q] += ((v >> q) & 1) ? 5 : -5;
    }
  }
  int32_t *a = acc + (int64_t)r.row * pb * SPB + (int64_t)t * SPB;
#pragma unroll
  for (int q = 0; q < SPB; q++)
    if (sum[q]) atomicAdd(a + q, sum[q]);
}

void launch_phasecal(const uint8_t *data, const PcalRun *runs, int nruns, int pb, int bits, int32_t *acc,
                     cudaStream_t st) {
  for (int r0 = 0; r0 < nruns; r0 += 65535) {
    const dim3 grid((unsigned)((pb + 255) / 256), (unsigned)std::min(65535, nruns - r0));
    if (bits == 2)
      phasecal_kernel<2><<<grid, 256, 0, st>>>(data, runs + r0, pb, acc);
    else
      phasecal_kernel<1><<<grid, 256, 0, st>>>(data, runs + r0, pb, acc);
  }
}

void launch_bitstat(const StreamDev *d_streams, const int4 *d_items, int nitems, cudaStream_t st) {
  if (nitems > 0) bitstat_kernel<<<nitems, 256, 0, st>>>(d_streams, d_items, nitems);
}

void launch_phased(const float2 *spec, int nrows_total, int kpad, int nstreams, int r0, int nrows, int K, int nsub,
                   float2 *acc, cudaStream_t st) {
  phased_kernel<<<(K + 127) / 128, 128, 0, st>>>(spec, nrows_total, kpad, nstreams, r0, nrows, K, nsub, acc);
}

void launch_pc_dump(float2 *acc, float2 *pcacc, const UvShift *uvp, int nstreams, int nbl, int kpad, int K, int npc,
                    cudaStream_t st) {
  const int chans = kPcThreads * kPcChans;
  if (nbl > 0)
    pc_dump_kernel<<<dim3((K + chans - 1) / chans, nbl), kPcThreads, 0, st>>>(acc, pcacc, uvp, nstreams, nbl, kpad, K,
                                                                              npc);
}

cudaError_t launch_reduce(const float2 *in, int nbl, int nout, int M, int nch, const float *mask,
                          const float *lag_window, int normalize, const float2 *tw2M, uint8_t *out, size_t out_stride,
                          size_t bl_stride, cudaStream_t st) {
  const int nspec = nbl * nout;
  if (nspec <= 0) return cudaSuccess;
  const int logM = 31 - __builtin_clz((unsigned)M), lognch = 31 - __builtin_clz((unsigned)nch);
  const size_t smem = (size_t)M * sizeof(float2) + (size_t)2 * nch * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(reduce_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  reduce_kernel<<<nspec, 256, smem, st>>>(in, M, logM, nch, lognch, mask, lag_window, normalize, tw2M, nbl, out,
                                          out_stride, bl_stride);
  return cudaGetLastError();
}

// Work split of the binned FP32 X-step for ntiles stream-pair tiles: parts of at
// most 36 tiles (12 warps x 3), the smallest tiles-per-warp that fits a part
// into 12 warps, rows per step so that a step stages at most 32 KB.
F32Plan xcorr_f32_plan(int ntiles, int npad) {
  F32Plan p;
  if (ntiles <= 0 || npad <= 0 || npad * 256 > kF32StageBytes * 4) return p;
  p.nparts = (ntiles + 35) / 36;
  p.tiles_per_part = (ntiles + p.nparts - 1) / p.nparts;
  for (p.tpw = 1; p.tpw < 3 && (p.tiles_per_part + p.tpw - 1) / p.tpw > 12; p.tpw++) {
  }
  p.warps = (p.tiles_per_part + p.tpw - 1) / p.tpw;
  p.R = std::max(1, kF32StageBytes / (npad * 256));
  p.smem = (size_t)kF32Stages * p.R * npad * 256;
  return p;
}

template <int TPW>
static void f32_launch(const F32Args &a, const F32Plan &p, cudaStream_t st) {
  auto kern = xcorr_f32_kernel<TPW>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
  kern<<<std::min((a.K + 31) / 32 * a.nparts, sm_count()), p.warps * 32, p.smem, st>>>(a);
}

void launch_xcorr_f32_binned(const float2 *spec, int nrows_total, int kpad, int nstreams, int npad, int nrows, int K,
                             const int *tiles, int ntiles, const int *blmap, int nbl, const int16_t *bins, float2 *acc,
                             cudaStream_t st) {
  if (nrows <= 0 || K <= 0) return;
  F32Plan p = xcorr_f32_plan(ntiles, npad);
  if (p.tpw <= 0) return;
  // every row of a channel in one work item (each accumulator entry has one
  // writer); finer parts of the tile set give the SMs enough items (each part
  // stages the rows again, mostly from L2)
  const int nct = (K + 31) / 32;
  const int np = std::min(ntiles, std::max(p.nparts, (2 * sm_count() + nct - 1) / nct));
  if (np > p.nparts) {
    p.nparts = np;
    p.tiles_per_part = (ntiles + np - 1) / np;
    for (p.tpw = 1; p.tpw < 3 && (p.tiles_per_part + p.tpw - 1) / p.tpw > 12; p.tpw++) {
    }
    p.warps = (p.tiles_per_part + p.tpw - 1) / p.tpw;
  }
  const F32Args a{spec, nrows_total, kpad, nstreams, npad, nrows, K, tiles, ntiles, p.tiles_per_part, p.nparts, p.R,
                  blmap, nbl, bins, acc};
  switch (p.tpw) {
    case 1: f32_launch<1>(a, p, st); break;
    case 2: f32_launch<2>(a, p, st); break;
    default: f32_launch<3>(a, p, st); break;
  }
}

void launch_pulsar_bins(int nrows, int K, double start_phase, double rate_term, double fft_duration,
                        const double *offsets, double g0, double g1, int nbins, int16_t *bins, cudaStream_t st) {
  pulsar_bins_kernel<<<dim3((nrows + 127) / 128, (K + kBinChans - 1) / kBinChans), 128, 0, st>>>(
      nrows, K, start_phase, rate_term, fft_duration, offsets, g0, g1, nbins, bins);
}

void launch_normalize(const float2 *acc, int kpad, int M, int nstreams, int nbl, int nout, const int *bl, double *norms,
                      const double *flagfac, uint8_t *out, size_t out_stride, size_t bl_stride, cudaStream_t st) {
  norm_autos_kernel<<<dim3(nstreams, nout), 256, 0, st>>>(acc, kpad, M, nstreams, nbl, norms);
  normalize_kernel<<<dim3((M + 1 + 255) / 256, nbl, nout), 256, 0, st>>>(acc, kpad, M, nstreams, nbl, bl, norms,
                                                                          flagfac, out, out_stride, bl_stride);
}

}  // namespace sfxc
