// FFT building blocks on packed pairs: every value is a float2 whose two
// lanes belong to two independent transforms (two streams, two blocks), so
// one packed FP32 instruction (add/mul/fma .f32x2) does both.  The packed
// forms run at the lane rate of the scalar ones (36.5-39.8 against 38.3 T
// lane operations/s measured on 152 SMs at 2.07 GHz) with half the issue
// slots, which is what the radix-16 kernels were short of.
//
// A transform of N = NV T points is done by T threads that each hold NV = 16
// or 8 values of S packed transforms.  The passes work in place: a pass reads
// and writes one thread's own NV places, so one barrier lies between two
// passes and none inside a pass.  Digits: input n = t + T q; pass 1
// transforms over q (k0 in place of q, then the twiddle W_N^(t k0)); what is
// left is a T-point transform over t for each k0.  Element (p, k0), p < T,
// lives at p + k0 (T + 1): unit stride over p and odd stride over k0, so
// 16-byte accesses whose lanes run over t (pass 1) or over k0 (later passes)
// touch every bank once per eight lanes.
#pragma once
#include <cuda_runtime.h>

namespace sfxc {

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long *>(&a)), "l"(*reinterpret_cast<unsigned long long *>(&b)));
  return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }

// a complex value of each lane
struct cpair {
  float2 re, im;
};
__device__ __forceinline__ cpair operator+(cpair a, cpair b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ cpair operator-(cpair a, cpair b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a * (x + i y), the same factor in both lanes
__device__ __forceinline__ cpair mulw(cpair a, float x, float y) {
  const float2 wx = dup2(x), wy = dup2(y), ny = dup2(-y);
  return {fma2(a.re, wx, mul2(a.im, ny)), fma2(a.re, wy, mul2(a.im, wx))};
}
__device__ __forceinline__ cpair mulw(cpair a, float2 w) { return mulw(a, w.x, w.y); }
// the same with the factor as (x, x, y, y): no register copies, one more product
__device__ __forceinline__ cpair mulw(cpair a, float4 w) {
  const float2 wx = make_float2(w.x, w.y), wy = make_float2(w.z, w.w);
  const float2 n = mul2(a.im, dup2(-1.0f));
  return {fma2(a.re, wx, mul2(n, wy)), fma2(a.re, wy, mul2(a.im, wx))};
}

// 4-point forward transform, outputs in natural order
__device__ __forceinline__ void dft4(cpair &a0, cpair &a1, cpair &a2, cpair &a3) {
  const cpair t0 = a0 + a2, t1 = a0 - a2, t2 = a1 + a3, d = a1 - a3;  // t3 = -i d
  a0 = t0 + t2;
  a2 = t0 - t2;
  a1 = {add2(t1.re, d.im), sub2(t1.im, d.re)};
  a3 = {sub2(t1.re, d.im), add2(t1.im, d.re)};
}
__device__ __forceinline__ void dft2(cpair &a, cpair &b) {
  const cpair t = a;
  a = t + b;
  b = t - b;
}
// a * exp(-2 pi i m / 16)
template <int m>
__device__ __forceinline__ cpair w16p(cpair a) {
  constexpr float C1 = 0.92387953251128674f, S1 = 0.38268343236508978f, R2 = 0.70710678118654752f;
  if constexpr (m == 1) return mulw(a, C1, -S1);
  if constexpr (m == 2) return {mul2(add2(a.re, a.im), dup2(R2)), mul2(sub2(a.im, a.re), dup2(R2))};
  if constexpr (m == 3) return mulw(a, S1, -C1);
  if constexpr (m == 6) return {mul2(sub2(a.im, a.re), dup2(R2)), mul2(add2(a.re, a.im), dup2(-R2))};
  if constexpr (m == 9) return mulw(a, -C1, S1);
  static_assert(m == 1 || m == 2 || m == 3 || m == 6 || m == 9, "twiddle not needed");
  return a;
}
// 8-point forward transform in place, outputs in natural order
__device__ __forceinline__ void dft8(cpair *v) {
  cpair e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4(e0, e1, e2, e3);
  dft4(o0, o1, o2, o3);
  o1 = w16p<2>(o1);
  o3 = w16p<6>(o3);
  v[0] = e0 + o0;
  v[4] = e0 - o0;
  v[1] = e1 + o1;
  v[5] = e1 - o1;
  v[2] = {add2(e2.re, o2.im), sub2(e2.im, o2.re)};  // o2 * -i
  v[6] = {sub2(e2.re, o2.im), add2(e2.im, o2.re)};
  v[3] = e3 + o3;
  v[7] = e3 - o3;
}
// 16-point forward transform as 4 x 4, natural order in and out.
// half: the caller guarantees v[9..15] == 0 (the first stage drops the
// additions of zeros).
__device__ __forceinline__ void dft16(cpair (&v)[16], bool half = false) {
  if (half) {
    {  // (v0, v4, v8, 0)
      const cpair a0 = v[0], a1 = v[4], a2 = v[8];
      const cpair t0 = a0 + a2, t1 = a0 - a2;
      v[0] = t0 + a1;
      v[8] = t0 - a1;
      v[4] = {add2(t1.re, a1.im), sub2(t1.im, a1.re)};
      v[12] = {sub2(t1.re, a1.im), add2(t1.im, a1.re)};
    }
#pragma unroll
    for (int n = 1; n < 4; n++) {  // (v[n], v[n + 4], 0, 0)
      const cpair a = v[n], b = v[n + 4];
      v[n] = a + b;
      v[n + 8] = a - b;
      v[n + 4] = {add2(a.re, b.im), sub2(a.im, b.re)};
      v[n + 12] = {sub2(a.re, b.im), add2(a.im, b.re)};
    }
  } else {
#pragma unroll
    for (int n = 0; n < 4; n++) dft4(v[n], v[n + 4], v[n + 8], v[n + 12]);
  }
  v[5] = w16p<1>(v[5]);
  v[9] = w16p<2>(v[9]);
  v[13] = w16p<3>(v[13]);
  v[6] = w16p<2>(v[6]);
  v[14] = w16p<6>(v[14]);
  v[7] = w16p<3>(v[7]);
  v[11] = w16p<6>(v[11]);
  v[15] = w16p<9>(v[15]);
  dft4(v[0], v[1], v[2], v[3]);
  dft4(v[4], v[5], v[6], v[7]);
  {  // v[10] enters as -i v[10]
    const cpair a = v[8], b = v[10];
    const cpair t0 = {add2(a.re, b.im), sub2(a.im, b.re)}, t1 = {sub2(a.re, b.im), add2(a.im, b.re)};
    const cpair t2 = v[9] + v[11], d = v[9] - v[11];
    v[8] = t0 + t2;
    v[10] = t0 - t2;
    v[9] = {add2(t1.re, d.im), sub2(t1.im, d.re)};
    v[11] = {sub2(t1.re, d.im), add2(t1.im, d.re)};
  }
  dft4(v[12], v[13], v[14], v[15]);
  cpair o[16];
#pragma unroll
  for (int k1 = 0; k1 < 4; k1++)
#pragma unroll
    for (int k2 = 0; k2 < 4; k2++) o[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = o[i];
}

template <int NV>
__device__ __forceinline__ void dftn(cpair (&v)[NV]) {
  if constexpr (NV == 2) dft2(v[0], v[1]);
  if constexpr (NV == 4) dft4(v[0], v[1], v[2], v[3]);
  if constexpr (NV == 8) dft8(v);
  if constexpr (NV == 16) dft16(v);
}

// Shape of an N-point transform by T = N / NV threads: radix NV over the
// first digit, NMID radix-NV passes, radix RL last.
template <int LOGN, int NV>
struct PackShape {
  static constexpr int N = 1 << LOGN, T = N / NV, LV = NV == 16 ? 4 : 3;
  static constexpr int P = T + 1;        // stride of k0
  static constexpr int ELEMS = NV * P;   // float4 elements of one packed transform's buffer
  static constexpr int NMID = (LOGN - LV - 1) / LV;
  static constexpr int RL = 1 << (LOGN - LV - LV * NMID);  // 2 .. NV
  // twiddles W_L^(p k), k = 1..NV-1, p < L / NV, after the radix-NV pass of
  // each sub-length L = N, T, T / NV (while a further pass follows)
  static constexpr int tw_len() {
    int n = 0, L = N;
    for (int i = 0; i <= NMID; i++) {
      n += (NV - 1) * (L / NV);
      L /= NV;
    }
    return n;
  }
};

// The twiddle tables of PackShape<LOGN, NV> from tw[j step] = exp(-2 pi i j / N):
// for each pass, tab[off + (k - 1) (L / NV) + p] = W_L^(p k).
template <int LOGN, int NV>
__device__ __forceinline__ void fill_pack_table(float2 *tab, const float2 *__restrict__ tw, int tid, int nthr,
                                                int step = 1) {
  using F = PackShape<LOGN, NV>;
  int off = 0, L = F::N;
#pragma unroll
  for (int i = 0; i <= F::NMID; i++) {
    const int H = L / NV;
    for (int e = tid; e < (NV - 1) * H; e += nthr) tab[off + e] = __ldg(tw + (1 + e / H) * (e % H) * (F::N / L) * step);
    off += (NV - 1) * H;
    L = H;
  }
}

__device__ __forceinline__ void put_pair(float4 *sm, int i, cpair v) {
  sm[i] = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
__device__ __forceinline__ cpair get_pair(const float4 *sm, int i) {
  const float4 q = sm[i];
  return {make_float2(q.x, q.y), make_float2(q.z, q.w)};
}

// v[s][k] *= tab[(k - 1) H + p], k = 1..NV-1
template <int H, int S, int NV>
__device__ __forceinline__ void twiddle_pass(cpair (&v)[S][NV], const float2 *tab, int p) {
#pragma unroll
  for (int k = 1; k < NV; k++) {
    const float2 w = tab[(k - 1) * H + p];
#pragma unroll
    for (int s = 0; s < S; s++) v[s][k] = mulw(v[s][k], w);
  }
}

// End of pass 1 of thread t on S packed transforms (buffers ELEMS apart):
// v[s][k0], the transform over q of x[t + T q], twiddled and written to the
// thread's places (t, k0), once `sync` has every thread past reading the
// buffer's earlier contents.
template <int LOGN, int S, int NV, class Sync>
__device__ __forceinline__ void pack_first(cpair (&v)[S][NV], float4 *sm, const float2 *tab, int t, Sync sync) {
  using F = PackShape<LOGN, NV>;
  twiddle_pass<F::T>(v, tab, t);
  sync();
#pragma unroll
  for (int k = 0; k < NV; k++)
#pragma unroll
    for (int s = 0; s < S; s++) put_pair(sm, s * F::ELEMS + t + k * F::P, v[s][k]);
}

// Middle pass I (1..NMID) of thread t, in place: the sub-length is L = N /
// NV^I; the thread's lane digit k0 = t % NV picks the buffer row, the rest of
// t the digit already transformed (hi) and the position p < L / NV.
template <int LOGN, int S, int NV, int I>
__device__ __forceinline__ void pack_middle(float4 *sm, const float2 *tab, int t) {
  using F = PackShape<LOGN, NV>;
  constexpr int L = F::N >> (F::LV * I), H = L / NV;
  constexpr int OFF = (NV - 1) * (I == 1 ? F::T : F::T + F::T / NV);
  static_assert(I <= 2 && H >= 1, "at most two middle passes");
  const int u = t / NV;             // u < T / NV
  const int p = u % H, hi = u / H;  // hi: digit k1 when I == 2 (L = T / NV)
  float4 *base = sm + (t % NV) * F::P + hi * L + p;
  cpair v[S][NV];
#pragma unroll
  for (int q = 0; q < NV; q++)
#pragma unroll
    for (int s = 0; s < S; s++) v[s][q] = get_pair(base, s * F::ELEMS + q * H);
#pragma unroll
  for (int s = 0; s < S; s++) dftn(v[s]);
  twiddle_pass<H>(v, tab + OFF, p);
#pragma unroll
  for (int k = 0; k < NV; k++)
#pragma unroll
    for (int s = 0; s < S; s++) put_pair(base, s * F::ELEMS + k * H, v[s][k]);
}

// Last pass of thread t: z[m] = X[t + T m].
template <int LOGN, int NV>
__device__ __forceinline__ void pack_last(cpair (&z)[NV], const float4 *sm, int t) {
  using F = PackShape<LOGN, NV>;
  constexpr int R = F::RL, G = NV / R;
  // the R positions of a sub-transform are adjacent; the digits before the
  // last, k0 + NV k1 (+ NV^2 k2), number the N / R sub-transforms t + T g
  const float4 *row = sm + (t % NV) * F::P;
#pragma unroll
  for (int g = 0; g < G; g++) {
    const int j = t / NV + (F::T / NV) * g;
    const int pos = F::NMID == 0 ? 0 : F::NMID == 1 ? j * R : (j % NV) * (F::T / NV) + (j / NV) * R;
    cpair u[R];
#pragma unroll
    for (int n = 0; n < R; n++) u[n] = get_pair(row, pos + n);
    dftn(u);
#pragma unroll
    for (int n = 0; n < R; n++) z[g + G * n] = u[n];
  }
}

}  // namespace sfxc
