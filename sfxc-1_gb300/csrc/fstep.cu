// F-step, stage 1: Delay_correction::fractional_bit_shift / fringe_stopping
// (sfxc/src/delay_correction.cc:82-184) on the unpacked samples of
// Bit2float_worker (sfxc/src/bit2float_worker.cc:327-425), from the per-block
// records of block_params_kernel.
#include <algorithm>

#include "device.cuh"
#include "fft_pack.cuh"
#include "kernels.hpp"
#include "phasor.cuh"
#include "tc_ptx.cuh"

namespace sfxc {
namespace {

// Sixteen threads take four consecutive 256-sample blocks b0..b3 as packed
// pairs: lane 0 of the forward transform holds x_b0 + i x_b1, lane 1 x_b2 + i
// x_b3 (X_b0[k] and X_b1[k] from Z[k] +/- conj Z[256-k], the partner's value
// by shuffle); then the inverse transforms of (b0, b2) and of (b1, b3).  Per
// block: DC and Nyquist halved, phase ramp exp(-i (c + k l)) on k <= 128,
// upper half zero, inverse 256-point transform (as conj(FFT(conj Y))), fringe
// rotation of the real part.
//
// Bounds: 49 instructions per sample at 0.47 issued per cycle and scheduler
// (16 warps per SM: a packed transform takes 64 registers), fetched as mostly
// straight code by warps out of step with each other (a fifth of the stalls;
// both inverses unrolled 3.46 ms, CTA-wide barriers 3.0 to 3.4), and 54 % of
// the shared-memory bandwidth.  Measured, 32 streams, 0.5 s of 64 MS/s 2-bit:
// 3.23 -> 2.96 ms (346 Gsamples/s), against pairs of blocks in scalar
// transforms at 85 instructions per sample; 16 streams with 1-bit and 2-bit
// samples 0.50 -> 0.40 ms.  A sixteenth of the pairs straddles two protocol
// records: walking those sample by sample (each step two dependent loads)
// made the packed form 4.0 ms; their words are put together by plan_bits.
constexpr int kBuf = 16 * 17;          // float4: one packed 256-point transform
constexpr int kExt = 8 * 16 + 1;       // float4: the half spectra of (b1, b3), bins 0..128
constexpr int kRec = 12;               // float4: four blocks' records
constexpr int kScratch = kBuf + kExt + 2 * kRec;  // per 16 threads; two sets of records
constexpr int kThreads = 256;

// 256-point forward transform by 16 threads: v[r] = x[t + 16 r] -> X[t + 16 r].
// tab[(k - 1) 16 + t] = exp(-2 pi i k t / 256) as (x, x, y, y); half: v[9..15] == 0.
template <bool HALF>
__device__ __forceinline__ void fft256(cpair (&v)[16], float4 *sm, const float4 *tab, int t) {
  dft16(v, HALF);
#pragma unroll
  for (int k = 1; k < 16; k++) v[k] = mulw(v[k], tab[(k - 1) * 16 + t]);
  __syncwarp();  // the buffer's earlier contents have been read
#pragma unroll
  for (int k = 0; k < 16; k++) put_pair(sm, t + 17 * k, v[k]);
  __syncwarp();
#pragma unroll
  for (int n = 0; n < 16; n++) v[n] = get_pair(sm, 17 * t + n);
  dft16(v);
}

// A thread's share of the samples of a pair of blocks, fetched ahead of their
// use: words t and 16 + t of the pair (2-bit samples, 16 a word) or word t
// (1-bit, 32 a word), and which of their bits are recorded samples.
struct PairWords {
  uint32_t w0, w1, m0, m1;
};
// 32 stream bits from `bit` on (the input has spare bytes after the last sample)
__device__ __forceinline__ uint32_t stream_bits(const StreamDev &s, long long bit) {
  const uint32_t *w = reinterpret_cast<const uint32_t *>(s.src) + (bit >> 5);
  return __funnelshift_r(__ldg(w), __ldg(w + 1), (uint32_t)bit & 31);
}
// 32 bits of samples from sample o on through the plan, from segment si on: zero
// bits and a zero mask where there is no recorded sample.
__device__ __noinline__ uint2 plan_bits(const StreamDev &s, int o, int si) {
  const int lb = s.bits - 1, limit = (s.block0 + s.n_blocks) * kNd;  // lb: log2 of the bits per sample
  uint32_t word = 0, mask = 0;
  for (int f = 0; f < 32 && o < limit;) {  // f bits filled
    int4 g = __ldg(reinterpret_cast<const int4 *>(s.segs) + si);  // out0, n, src_bit
    while (si + 1 < s.nsegs && g.x + g.y <= o) g = __ldg(reinterpret_cast<const int4 *>(s.segs) + ++si);
    const long long src = (long long)((unsigned long long)(uint32_t)g.z | (unsigned long long)(uint32_t)g.w << 32);
    const bool inside = o >= g.x && o < g.x + g.y;
    int n = min((32 - f) >> lb, limit - o);  // samples taken here
    if (inside)
      n = min(n, g.x + g.y - o);
    else if (o < g.x)
      n = min(n, g.x - o);
    if (inside && src >= 0) {
      const uint32_t ones = 0xFFFFFFFFu >> (32 - (n << lb));
      word |= (stream_bits(s, src + ((long long)(o - g.x) << lb)) & ones) << f;
      mask |= ones << f;
    }
    o += n;
    f += n << lb;
  }
  return make_uint2(word, mask);
}
// pair of blocks bl, bl + 1, whose first block's record is p
__device__ __forceinline__ PairWords fetch_pair(const StreamDev &s, const BlockPar *p, int bl, int t) {
  PairWords w{0, 0, 0, 0};
  if (bl >= s.n_blocks) return w;
  const bool two = s.bits == 2;
  const long long bit = p->src_bit;
  if (bit >= 0) {  // both blocks inside one segment of recorded samples
    w.w0 = stream_bits(s, bit + 32 * t);
    if (two) w.w1 = stream_bits(s, bit + 512 + 32 * t);
    w.m0 = w.m1 = 0xFFFFFFFFu;
  } else {
    const int o0 = (s.block0 + bl) * kNd;
    const uint2 a = plan_bits(s, o0 + (two ? 16 : 32) * t, p->seg);
    w.w0 = a.x;
    w.m0 = a.y;
    w.m1 = 0xFFFFFFFFu;
    if (two) {
      const uint2 b = plan_bits(s, o0 + kNd + 16 * t, p->seg);
      w.w1 = b.x;
      w.m1 = b.y;
    }
  }
  return w;
}

// Samples of blocks bl and bl + 1 -> x0[r], x1[r] = sample t + 16 r of each:
// the half warp shares its words through 64 words of scratch.
__device__ __forceinline__ void unpack_pair(bool two, const PairWords &p, int t, uint32_t *ws, float (&x0)[16],
                                            float (&x1)[16]) {
  __syncwarp();
  ws[t] = p.w0;
  ws[16 + t] = p.w1;
  ws[32 + t] = p.m0;
  ws[48 + t] = p.m1;
  const bool holes = __any_sync(0xffffffffu, (p.m0 & p.m1) != 0xFFFFFFFFu);
  __syncwarp();
  const uint4 *wq = reinterpret_cast<const uint4 *>(ws);
  if (two) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const uint4 u = wq[q];
      const uint32_t uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float x = code_value2((uu[i] >> (2 * t)) & 3);
        if (q < 4)
          x0[4 * q + i] = x;
        else
          x1[4 * (q - 4) + i] = x;
      }
    }
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint4 u = wq[q];
      const uint32_t uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        // samples t and 16 + t of the word: bit set +5, clear -5 (0xC0A00000)
        const float a = __uint_as_float(((uu[i] << (31 - t)) & 0x80000000u) ^ 0xC0A00000u);
        const float b = __uint_as_float(((uu[i] << (15 - t)) & 0x80000000u) ^ 0xC0A00000u);
        const int r = 2 * (4 * q + i);
        if (q < 2) {
          x0[r] = a;
          x0[r + 1] = b;
        } else {
          x1[r - 16] = a;
          x1[r - 15] = b;
        }
      }
    }
  }
  if (holes) {  // invalid or inserted samples, blocks past the stream's end: zeros
#pragma unroll
    for (int r = 0; r < 16; r++) {
      const uint32_t a = two ? ws[32 + r] >> (2 * t) : ws[32 + r / 2] >> (t + 16 * (r & 1));
      const uint32_t b = two ? ws[48 + r] >> (2 * t) : ws[40 + r / 2] >> (t + 16 * (r & 1));
      x0[r] = a & 1 ? x0[r] : 0.f;
      x1[r] = b & 1 ? x1[r] : 0.f;
    }
  }
}

__device__ __forceinline__ float4 ld4(const float4 *p) { return *p; }
// a rotating phasor: multiply by the lane's own step
struct Rotor {
  cpair e, st;
  float2 nim;  // -st.im
  __device__ __forceinline__ void set(float c0, float s0, float c1, float s1) {
    st = {make_float2(c0, c1), make_float2(s0, s1)};
    nim = make_float2(-s0, -s1);
  }
  __device__ __forceinline__ void next() {
    const float2 c = fma2(e.re, st.re, mul2(e.im, nim));
    e.im = fma2(e.im, st.re, mul2(e.re, st.im));
    e.re = c;
  }
};

// Unpacked samples of one stream's blocks (inspection of the Bit2float_worker
// output), by the block stage's own unpacking: a half warp per pair of blocks.
__global__ void __launch_bounds__(kThreads) unpack_kernel(const StreamDev *__restrict__ stream, float *__restrict__ out) {
  __shared__ __align__(16) uint32_t words[kThreads / 16][64];
  const StreamDev &s = *stream;
  const int t = threadIdx.x & 15, grp = threadIdx.x >> 4, bl = (blockIdx.x * (kThreads / 16) + grp) * 2;
  if ((bl & ~3) >= s.n_blocks) return;  // whole warps (four blocks each)
  float x0[16], x1[16];
  unpack_pair(s.bits == 2, fetch_pair(s, s.bpar + bl, bl, t), t, words[grp], x0, x1);
#pragma unroll
  for (int r = 0; r < 16; r++) {
    float *const o = out + (int64_t)bl * kNd + t + 16 * r;
    if (bl < s.n_blocks) o[0] = x0[r];
    if (bl + 1 < s.n_blocks) o[kNd] = x1[r];
  }
}

// CTAs of 64 blocks a round, rounds strided over the stream's blocks.
__global__ void __launch_bounds__(kThreads, 2) fstep_block_kernel(const StreamDev *__restrict__ streams,
                                                                 const float2 *__restrict__ tw) {
  extern __shared__ __align__(16) float4 fsm[];  // 16 x kScratch
  __shared__ float4 tab[15 * 16];
  const int t = threadIdx.x & 15, grp = threadIdx.x >> 4, lane = threadIdx.x & 31;
  const StreamDev &s = streams[blockIdx.y];
  if (threadIdx.x < 240) {
    const float2 w = __ldg(tw + (threadIdx.x / 16 + 1) * (threadIdx.x & 15));
    tab[threadIdx.x] = make_float4(w.x, w.x, w.y, w.y);
  }
  __syncthreads();
  float4 *sm = fsm + grp * kScratch, *ext = sm + kBuf;
  const int partner = (lane & 16) | ((16 - t) & 15);
  const int n_blocks = s.n_blocks, stride = gridDim.x * 64;
  float *const ts = s.ts;
  const BlockPar *const bpar = s.bpar;
  int bl0 = blockIdx.x * 64 + grp * 4;
  const bool two = s.bits == 2;
  // the records of the round's four blocks come to shared memory a round
  // ahead (192 contiguous bytes; those past the stream's end are left out)
  BlockPar *rec0 = reinterpret_cast<BlockPar *>(ext + kExt), *rec1 = rec0 + 4;
  auto fetch_records = [&](BlockPar *dst, int bl) {
    if (t < kRec && bl + t / 3 < n_blocks)
      tc::cp_async16(tc::smem_u32(reinterpret_cast<float4 *>(dst) + t), reinterpret_cast<const float4 *>(bpar + bl) + t, 16);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto records_here = [&] {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
  };
  fetch_records(rec0, bl0);
  records_here();
  PairWords wa = fetch_pair(s, rec0, bl0, t), wb = fetch_pair(s, rec0 + 2, bl0 + 2, t);
  for (; (bl0 & ~7) < n_blocks; bl0 += stride) {  // whole warps (8 blocks each)
    cpair v[16];
    {
      float x0[16], x1[16];
      unpack_pair(two, wa, t, reinterpret_cast<uint32_t *>(sm), x0, x1);
#pragma unroll
      for (int r = 0; r < 16; r++) {
        v[r].re.x = x0[r];
        v[r].im.x = x1[r];
      }
      unpack_pair(two, wb, t, reinterpret_cast<uint32_t *>(sm), x0, x1);
#pragma unroll
      for (int r = 0; r < 16; r++) {
        v[r].re.y = x0[r];
        v[r].im.y = x1[r];
      }
    }
    const bool all = bl0 + 4 <= n_blocks;
    fetch_records(rec1, bl0 + stride);
    auto rec = [&](int i) { return rec0 + (all || bl0 + i < n_blocks ? i : 0); };
    fft256<false>(v, sm, tab, t);
    __syncwarp();  // ahead of the half spectra in the buffer
    {
        // the upper half to the partner; thread 0 pairs 16 r with 16 (16 - r)
        // and has bin 128 to itself
        const cpair zmid = v[8];
        if (t == 0) {
          const cpair z0 = v[0];
#pragma unroll
          for (int r = 8; r < 15; r++) v[r] = v[r + 1];
          v[15] = z0;
        }
        // ramp phasors of (b0, b2) and (b1, b3): exp(i pi (c + k l)), in steps of 16 bins
        Rotor ra, rb;
        {
          const float4 p0 = ld4(&rec(0)->ph), p2 = ld4(&rec(2)->ph), p1 = ld4(&rec(1)->ph), p3 = ld4(&rec(3)->ph);
          ra.e = phasor(fmaf((float)t, p0.y, p0.x), fmaf((float)t, p2.y, p2.x));
          rb.e = phasor(fmaf((float)t, p1.y, p1.x), fmaf((float)t, p3.y, p3.x));
        }
        {
          const float4 s0 = ld4(&rec(0)->steps), s2 = ld4(&rec(2)->steps);
          const float4 s1 = ld4(&rec(1)->steps), s3 = ld4(&rec(3)->steps);
          ra.set(s0.x, s0.y, s2.x, s2.y);
          rb.set(s1.x, s1.y, s3.x, s3.y);
        }
        const float2 hf = dup2(t == 0 ? 0.5f : 1.0f);  // bin 0 of thread 0 (the split's 1/2 is in the amplitude)
#pragma unroll
        for (int r = 0; r < 9; r++) {
          cpair f0 = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, f1 = f0;
          if (r < 8 || t == 0) {
            const cpair zk = r < 8 ? v[r] : zmid;
            cpair zc = zmid;
            if (r < 8) {
              const cpair u = v[15 - r];
              zc = {make_float2(__shfl_sync(0xffffffffu, u.re.x, partner), __shfl_sync(0xffffffffu, u.re.y, partner)),
                    make_float2(__shfl_sync(0xffffffffu, u.im.x, partner), __shfl_sync(0xffffffffu, u.im.y, partner))};
            }
            float2 er = add2(zk.re, zc.re), ei = sub2(zk.im, zc.im);  // 2 X_b0, 2 X_b2
            float2 qr = add2(zk.im, zc.im), qi = sub2(zc.re, zk.re);  // 2 X_b1, 2 X_b3
            if (r == 0 || r == 8) {
              const float2 f = r == 0 ? hf : dup2(0.5f);
              er = mul2(er, f);
              ei = mul2(ei, f);
              qr = mul2(qr, f);
              qi = mul2(qi, f);
            }
            // conj(F e^{-i phi})
            f0 = {fma2(er, ra.e.re, mul2(ei, ra.e.im)), sub2(mul2(er, ra.e.im), mul2(ei, ra.e.re))};
            f1 = {fma2(qr, rb.e.re, mul2(qi, rb.e.im)), sub2(mul2(qr, rb.e.im), mul2(qi, rb.e.re))};
          }
          if (r < 8 || t == 0) {
            put_pair(sm, 16 * r + t, f0);
            put_pair(ext, 16 * r + t, f1);
          }
          if (r < 8) {
            ra.next();
            rb.next();
          }
        }
    }
    // the inverses of blocks (b0, b2) and (b1, b3)
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      {
        const float4 *half = h ? ext : sm;
#pragma unroll
        for (int r = 0; r < 8; r++) v[r] = get_pair(half, 16 * r + t);
        v[8] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        if (t == 0) v[8] = get_pair(half, 128);
        fft256<true>(v, sm, tab, t);
        // v = conj(z), z the inverse transforms of blocks b_h and b_{h+2}:
        // fringe rotation Re(z e^{-i phi}) x amplitude
        Rotor f;
        {
          const BlockPar *qa = rec(h), *qb = rec(h + 2);
          const float4 p0 = ld4(&qa->ph), p1 = ld4(&qb->ph), s0 = ld4(&qa->steps), s1 = ld4(&qb->steps);
          f.e = phasor(fmaf((float)t, p0.w, p0.z), fmaf((float)t, p1.w, p1.z));
          f.set(s0.z, s0.w, s1.z, s1.w);
          const float2 amp = make_float2(0.5f * qa->amp, 0.5f * qb->amp);
          f.e.re = mul2(f.e.re, amp);
          f.e.im = mul2(f.e.im, amp);
        }
        float *oa = ts + (int64_t)(bl0 + h) * kNd + t;
        if (all) {
#pragma unroll
          for (int r = 0; r < 16; r++) {
            const float2 y = sub2(mul2(v[r].re, f.e.re), mul2(v[r].im, f.e.im));
            __stcg(oa + 16 * r, y.x);
            __stcg(oa + 2 * kNd + 16 * r, y.y);
            f.next();
          }
        } else {  // the stream's last blocks, rolled
          __syncwarp();
          const bool oka = bl0 + h < n_blocks, okb = bl0 + h + 2 < n_blocks;
#pragma unroll
          for (int r = 0; r < 16; r++) put_pair(sm, 16 * r + t, v[r]);
#pragma unroll 1
          for (int r = 0; r < 16; r++) {
            const cpair z = get_pair(sm, 16 * r + t);
            const float2 y = sub2(mul2(z.re, f.e.re), mul2(z.im, f.e.im));
            if (oka) __stcg(oa + 16 * r, y.x);
            if (okb) __stcg(oa + 2 * kNd + 16 * r, y.y);
            f.next();
          }
        }
      }
    }
    records_here();
    {
      BlockPar *r = rec0;
      rec0 = rec1;
      rec1 = r;
    }
    const int nb = bl0 + stride;
    wa = fetch_pair(s, rec0, nb, t);
    wb = fetch_pair(s, rec0 + 2, nb + 2, t);
  }
}

}  // namespace

void launch_unpack(const StreamDev *d_stream, int n_blocks, float *out, cudaStream_t st) {
  constexpr int per_cta = kThreads / 8;
  unpack_kernel<<<(n_blocks + per_cta - 1) / per_cta, kThreads, 0, st>>>(d_stream, out);
}

void launch_fstep(const StreamDev *d_streams, int nstreams, int max_blocks, const float2 *tw256, cudaStream_t st,
                  int ctas_per_sm) {
  // by default about five waves of 2 resident CTAs per SM, each CTA looping
  // over rounds (32 streams, 0.5 s: one wave 3.13 ms, two 3.07, three 3.02,
  // five 2.99); the autotuner may pick another count per shape
  const int per_stream = std::max(1, (ctas_per_sm > 0 ? ctas_per_sm : 10) * sm_count() / nstreams);
  dim3 grid(std::min((max_blocks + 63) / 64, per_stream), nstreams);
  constexpr int smem = 16 * kScratch * sizeof(float4);
  cudaFuncSetAttribute(fstep_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  fstep_block_kernel<<<grid, kThreads, smem, st>>>(d_streams, tw256);
}

}  // namespace sfxc
