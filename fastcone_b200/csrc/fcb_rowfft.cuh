// fcb_rowfft.cuh -- convolution of detector rows with a fixed real kernel, one pass over HBM.
//
// out[i] = sum_j kern(i - j) in[j] for rows of W values, i, j in [0, W): the ramp filters of
// the FDK pre-processing (even kernels) and the Hilbert transform of the Katsevich filter (an
// odd one).  A linear convolution of W values is a cyclic one of any length L >= 2 W - 1, so
// L = 2 N with N >= W from a short list of sizes (2^a and 3 * 2^a), whatever W is.
//
// A row stays on the chip from its load to its store: the row's values in pairs are the
// complex sequence z[n] = x[2n] + i x[2n+1] (upper half zero), whose N-point transform is
// computed in shared memory, multiplied by the kernel's spectrum and transformed back.
//   stage 1  radix A over n1      n = n1 BC + n2 C + n3,  k = k1 + A k2 + AB k3
//   stage 2  radix B over n2
//   stage 3  radix C over n3 of the columns j = k1 + A k2 and AB - j together: they hold k and
//            N - k, which the real-sequence step needs side by side, so the spectrum product
//            and the first inverse stage follow in registers
//   stages 2 and 1 back.  Stage 1 reads only n1 < A / 2 (the rest is padding) and, going back,
//   computes only those outputs.
// Each row has its own transform (two rows are not packed into one complex row): a NaN, an
// infinity or a much larger neighbour stays in its row.  Twiddles and spectra come from tables
// made in FP64.
//
// What bounds it: about 6700 warp instructions per row of 1536 values (two thirds of them FP32
// arithmetic) against 12 KB of HBM traffic, so issue (55 % busy) and shared memory (49 %), not
// HBM.  A row's buffer limits how many rows an SM holds (13 of 1536 values), so latency is
// hidden inside the warp: the next rows' values are loaded into registers while the current ones
// are transformed, and the tables sit in shared memory (one persistent CTA per SM loads them
// once).  1440 x 1024 rows of 1536 values, cosine weight and Shepp-Logan, on one B200: 14.2 ms
// (21.4 ms with short-lived CTAs, tables through L1 and no prefetch); cuFFT R2C, a spectrum pass
// and C2R between padding and cropping passes took 89.6 ms.  Error against 64 bits 4.2e-6 of the
// result's norm there (cuFFT's 6.7e-6: the result is small against the smooth input); over 70
// widths from 32 to 2048, smooth rows, Ram-Lak with and without the weight and Shepp-Logan, 0.38
// to 0.91 of cuFFT's.
//
// The stages are functions of (thread, row buffer), so that the host can run them too (a CPU test does).
#pragma once

#include <math.h>
#include <stdint.h>

#if defined(__CUDACC__)
#include "fcb_internal.h"
#define FCB_HD __host__ __device__ __forceinline__
#else
#define FCB_HD inline
#endif

namespace fcb {
namespace rf {

struct cf {
  float x, y;
};
FCB_HD cf operator+(cf a, cf b) { return {a.x + b.x, a.y + b.y}; }
FCB_HD cf operator-(cf a, cf b) { return {a.x - b.x, a.y - b.y}; }
// a * w, and a * conj(w)
FCB_HD cf cmul(cf a, cf w) { return {fmaf(a.x, w.x, -a.y * w.y), fmaf(a.x, w.y, a.y * w.x)}; }
FCB_HD cf cmulc(cf a, cf w) { return {fmaf(a.x, w.x, a.y * w.y), fmaf(a.y, w.x, -a.x * w.y)}; }
// a * w forward, a * conj(w) backward
template <bool INV>
FCB_HD cf tw(cf a, cf w) { return INV ? cmulc(a, w) : cmul(a, w); }
// a * (-i) forward, a * i backward
template <bool INV>
FCB_HD cf rot(cf a) { return INV ? cf{-a.y, a.x} : cf{a.y, -a.x}; }

// ---- transforms of R values in registers, natural order in and out
template <bool INV>
FCB_HD void dft4(cf& a0, cf& a1, cf& a2, cf& a3)
{
  const cf t0 = a0 + a2, t1 = a0 - a2, t2 = a1 + a3, t3 = rot<INV>(a1 - a3);
  a0 = t0 + t2; a1 = t1 + t3; a2 = t0 - t2; a3 = t1 - t3;
}
template <bool INV>
FCB_HD void dft3(cf& a0, cf& a1, cf& a2)
{
  const cf t = a1 + a2, u = a1 - a2;
  const cf m = {fmaf(-0.5f, t.x, a0.x), fmaf(-0.5f, t.y, a0.y)};
  const cf d = rot<INV>(cf{0.86602540378443865f * u.x, 0.86602540378443865f * u.y});
  a0 = a0 + t; a1 = m + d; a2 = m - d;
}
template <bool INV>
FCB_HD void dft8(cf (&a)[8])
{
  constexpr float R = 0.70710678118654752f;
  cf b[4], c[4];
  for (int r = 0; r < 4; r++) {
    b[r] = a[r] + a[r + 4];
    c[r] = a[r] - a[r + 4];
  }
  // c[r] *= W8^r: (1 -+ i) / sqrt 2, -+ i, (-1 -+ i) / sqrt 2
  const cf r1 = rot<INV>(c[1]), r3 = rot<INV>(c[3]);
  c[1] = {R * (c[1].x + r1.x), R * (c[1].y + r1.y)};
  c[2] = rot<INV>(c[2]);
  c[3] = {R * (r3.x - c[3].x), R * (r3.y - c[3].y)};
  dft4<INV>(b[0], b[1], b[2], b[3]);
  dft4<INV>(c[0], c[1], c[2], c[3]);
  for (int q = 0; q < 4; q++) {
    a[2 * q] = b[q];
    a[2 * q + 1] = c[q];
  }
}
// exp(-2 pi i j / 16), j = 0 .. 9
FCB_HD cf w16(int j)
{
  constexpr float C1 = 0.92387953251128674f, S1 = 0.38268343236508977f, R = 0.70710678118654752f;
  switch (j) {
    case 0: return {1.0f, 0.0f};
    case 1: return {C1, -S1};
    case 2: return {R, -R};
    case 3: return {S1, -C1};
    case 4: return {0.0f, -1.0f};
    case 5: return {-S1, -C1};
    case 6: return {-R, -R};
    case 7: return {-C1, -S1};
    case 8: return {-1.0f, 0.0f};
    default: return {-C1, S1};
  }
}
// exp(-2 pi i j / 12), j = 0 .. 5
FCB_HD cf w12(int j)
{
  constexpr float C = 0.86602540378443865f;
  switch (j) {
    case 0: return {1.0f, 0.0f};
    case 1: return {C, -0.5f};
    case 2: return {0.5f, -C};
    case 3: return {0.0f, -1.0f};
    case 4: return {-0.5f, -C};
    default: return {-C, -0.5f};
  }
}
// a * exp(-+ 2 pi i j / M) for the multiples of an eighth that need no full product
template <int M, bool INV>
FCB_HD cf wconst(cf a, int j)
{
  if (j == 0) return a;
  if (4 * j == M) return rot<INV>(a);
  if (8 * j == M) {
    constexpr float R = 0.70710678118654752f;
    const cf b = rot<INV>(a);
    return {R * (a.x + b.x), R * (a.y + b.y)};
  }
  if (8 * j == 3 * M) {
    constexpr float R = 0.70710678118654752f;
    const cf b = rot<INV>(a);
    return {R * (b.x - a.x), R * (b.y - a.y)};
  }
  return tw<INV>(a, M == 16 ? w16(j) : w12(j));
}

template <int R, bool INV>
struct Dft;
template <bool INV>
struct Dft<4, INV> {
  static FCB_HD void run(cf (&a)[4]) { dft4<INV>(a[0], a[1], a[2], a[3]); }
};
template <bool INV>
struct Dft<6, INV> {  // 2 x 3, prime factors: n = 3 n1 + 2 n2, k = 3 k1 + 4 k2 (mod 6)
  static FCB_HD void run(cf (&a)[6])
  {
    cf s0 = a[0] + a[3], s1 = a[2] + a[5], s2 = a[4] + a[1];
    cf d0 = a[0] - a[3], d1 = a[2] - a[5], d2 = a[4] - a[1];
    dft3<INV>(s0, s1, s2);
    dft3<INV>(d0, d1, d2);
    a[0] = s0; a[4] = s1; a[2] = s2;
    a[3] = d0; a[1] = d1; a[5] = d2;
  }
};
template <bool INV>
struct Dft<8, INV> {
  static FCB_HD void run(cf (&a)[8]) { dft8<INV>(a); }
};
template <bool INV>
struct Dft<16, INV> {  // 4 x 4
  static FCB_HD void run(cf (&a)[16])
  {
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) dft4<INV>(a[n2], a[4 + n2], a[8 + n2], a[12 + n2]);
#pragma unroll
    for (int k1 = 1; k1 < 4; k1++)
#pragma unroll
      for (int n2 = 1; n2 < 4; n2++) a[4 * k1 + n2] = wconst<16, INV>(a[4 * k1 + n2], k1 * n2);
    cf b[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
      dft4<INV>(a[4 * k1], a[4 * k1 + 1], a[4 * k1 + 2], a[4 * k1 + 3]);
#pragma unroll
      for (int k2 = 0; k2 < 4; k2++) b[k1 + 4 * k2] = a[4 * k1 + k2];
    }
#pragma unroll
    for (int k = 0; k < 16; k++) a[k] = b[k];
  }
};

// ---- a row transform of N = A B C complex values (B = 1: two stages)
template <int A_, int B_, int C_>
struct Shape {
  static constexpr int A = A_, B = B_, C = C_, N = A * B * C, BC = B * C, AB = A * B, HA = A / 2;
  // Row buffer: [k1 or n1][k2 or n2][n3 or k3] with strides S1, S2, 1.  S2 odd: the columns of
  // stage 3 start in different (64-bit) banks; S1 = 8 mod 16 spreads stage 2's, whose lanes run
  // over C values of a few n1.
  static constexpr int S2 = C + 1;
  static constexpr int S1 = B == 1 ? S2 : (B * S2 + 7) / 16 * 16 + 8;
  static constexpr int BUF = A * S1;          // complex values per row buffer
  static constexpr int NB1 = BC, NB2 = B == 1 ? 0 : A * C, NB3 = AB / 2;  // butterflies (pairs in stage 3)
  static constexpr int T1 = A * BC, T2 = B == 1 ? 0 : B * C;               // twiddle tables (complex)
  static constexpr int G = NB3 * C;           // spectrum table (float4)
  static_assert(A % 2 == 0 && (B == 1 || B % 2 == 0) && S1 >= B * S2, "row transform shape");
};

// columns (k1, k2) and (p1, p2) of stage 3's pair q; false for the two columns that are
// their own partners (0 and AB / 2)
template <class S>
FCB_HD bool pair_of(int q, int& k1, int& k2, int& p1, int& p2)
{
  if constexpr (S::B == 1) {
    k1 = q; k2 = 0; p1 = q == 0 ? S::A / 2 : S::A - q; p2 = 0;
    return q != 0;
  } else {
    constexpr int M = (S::HA - 1) * S::B;
    if (q < M) {
      k1 = 1 + q / S::B; k2 = q % S::B;
      p1 = S::A - k1; p2 = S::B - 1 - k2;
      return true;
    }
    const int r = q - M;
    if (r < S::B / 2) {
      k1 = p1 = S::HA; k2 = r; p2 = S::B - 1 - r;
      return true;
    }
    k1 = p1 = 0; k2 = r - S::B / 2;
    p2 = k2 == 0 ? S::B / 2 : S::B - k2;
    return k2 != 0;
  }
}

// Stage 1: x[n1] = z[n1 BC + m], n1 < A / 2 -> buf[k1][m], twiddled
template <class S>
FCB_HD void stage1(const cf (&x)[S::HA], int m, cf* buf, const cf* t1)
{
  cf e[S::HA], o[S::HA];
#pragma unroll
  for (int r = 0; r < S::HA; r++) {
    e[r] = x[r];
    o[r] = S::A == 8 ? wconst<8, false>(x[r], r) : S::A == 12 ? wconst<12, false>(x[r], r) : wconst<16, false>(x[r], r);
  }
  Dft<S::HA, false>::run(e);
  Dft<S::HA, false>::run(o);
  cf* p = buf + (m / S::C) * S::S2 + m % S::C;
#pragma unroll
  for (int q = 0; q < S::HA; q++) {
    p[(2 * q) * S::S1] = q == 0 ? e[0] : cmul(e[q], t1[(2 * q) * S::BC + m]);
    p[(2 * q + 1) * S::S1] = cmul(o[q], t1[(2 * q + 1) * S::BC + m]);
  }
}
// Stage 1 back: x[n1] for n1 < A / 2
template <class S>
FCB_HD void stage1_back(cf (&x)[S::HA], int m, const cf* buf, const cf* t1)
{
  cf e[S::HA], o[S::HA];
  const cf* p = buf + (m / S::C) * S::S2 + m % S::C;
#pragma unroll
  for (int q = 0; q < S::HA; q++) {
    e[q] = q == 0 ? p[0] : cmulc(p[(2 * q) * S::S1], t1[(2 * q) * S::BC + m]);
    o[q] = cmulc(p[(2 * q + 1) * S::S1], t1[(2 * q + 1) * S::BC + m]);
  }
  Dft<S::HA, true>::run(e);
  Dft<S::HA, true>::run(o);
#pragma unroll
  for (int r = 0; r < S::HA; r++)
    x[r] = e[r] + (S::A == 8 ? wconst<8, true>(o[r], r) : S::A == 12 ? wconst<12, true>(o[r], r) : wconst<16, true>(o[r], r));
}
// Stage 2 forward (twiddle after) and backward (before), butterfly b = (k1, n3), in place
template <class S, bool INV>
FCB_HD void stage2(int b, cf* buf, const cf* t2)
{
  const int n3 = b % S::C, k1 = b / S::C;
  cf* p = buf + k1 * S::S1 + n3;
  cf a[S::B];
#pragma unroll
  for (int r = 0; r < S::B; r++) {
    a[r] = p[r * S::S2];
    if (INV && r > 0) a[r] = cmulc(a[r], t2[r * S::C + n3]);
  }
  Dft<S::B, INV>::run(a);
#pragma unroll
  for (int r = 0; r < S::B; r++) {
    if (!INV && r > 0) a[r] = cmul(a[r], t2[r * S::C + n3]);
    p[r * S::S2] = a[r];
  }
}
// The spectrum product for k and N - k (a = Z[k], b = Z[N - k]; see spectrum_entry)
template <bool ODD>
FCB_HD void product(cf& a, cf& b, float s, float tr, float ti)
{
  const cf e = {a.x + b.x, a.y - b.y};       // a + conj b
  const cf o = {a.y + b.y, b.x - a.x};       // -i (a - conj b)
  // E = s e + t o, O = s o + conj(t) e
  const cf E = {fmaf(s, e.x, fmaf(tr, o.x, -ti * o.y)), fmaf(s, e.y, fmaf(tr, o.y, ti * o.x))};
  const cf O = {fmaf(s, o.x, fmaf(tr, e.x, ti * e.y)), fmaf(s, o.y, fmaf(tr, e.y, -ti * e.x))};
  const cf u = {E.x - O.y, E.y + O.x};       // E + i O
  const cf v = {E.x + O.y, O.x - E.y};       // conj(E - i O)
  a = ODD ? cf{-u.y, u.x} : u;               // times i
  b = ODD ? cf{v.y, -v.x} : v;               // times -i
}
struct f4 {
  float s, tr, ti, pad;
};
// Stage 3 and back, pair q, in place
template <class S, bool ODD>
FCB_HD void stage3(int q, cf* buf, const f4* g)
{
  int k1, k2, p1, p2;
  const bool two = pair_of<S>(q, k1, k2, p1, p2);
  cf* pu = buf + k1 * S::S1 + k2 * S::S2;
  cf* pv = buf + p1 * S::S1 + p2 * S::S2;
  cf u[S::C], v[S::C];
#pragma unroll
  for (int r = 0; r < S::C; r++) {
    u[r] = pu[r];
    v[r] = pv[r];
  }
  Dft<S::C, false>::run(u);
  Dft<S::C, false>::run(v);
  if (two) {
    // u[k3] = Z[j + AB k3], its partner v[C - 1 - k3]
#pragma unroll
    for (int r = 0; r < S::C; r++) {
      const f4 w = g[r * S::NB3 + q];
      product<ODD>(u[r], v[S::C - 1 - r], w.s, w.tr, w.ti);
    }
  } else {
    // column 0 pairs k3 with C - k3 (0 and C / 2 with themselves), column AB / 2 with C - 1 - k3;
    // the table's entries r <= C / 2 are column 0's, the others column AB / 2's first ones, whose
    // last one stands in the partner's slot (see spectrum_entry)
#pragma unroll
    for (int r = 0; r <= S::C / 2; r++) {
      const f4 w = g[r * S::NB3 + q];
      if (r == 0 || 2 * r == S::C) {
        cf c = u[r];
        product<ODD>(u[r], c, w.s, w.tr, w.ti);
      } else {
        product<ODD>(u[r], u[S::C - r], w.s, w.tr, w.ti);
      }
    }
#pragma unroll
    for (int r = 0; r < S::C / 2; r++) {
      const f4 w = r + S::C / 2 + 1 < S::C ? g[(r + S::C / 2 + 1) * S::NB3 + q] : g[S::G];
      product<ODD>(v[r], v[S::C - 1 - r], w.s, w.tr, w.ti);
    }
  }
  Dft<S::C, true>::run(u);
  Dft<S::C, true>::run(v);
#pragma unroll
  for (int r = 0; r < S::C; r++) {
    pu[r] = u[r];
    pv[r] = v[r];
  }
}

// Frequency k of spectrum-table entry e < G + 1 (entry e = k3 * NB3 + q).
template <class S>
FCB_HD int entry_k(int e)
{
  if (e == S::G) return S::AB / 2 + S::AB * (S::C / 2 - 1);
  const int q = e % S::NB3, r = e / S::NB3;
  int k1, k2, p1, p2;
  if (pair_of<S>(q, k1, k2, p1, p2)) return k1 + S::A * k2 + S::AB * r;
  if (r <= S::C / 2) return S::AB * r;
  return S::AB / 2 + S::AB * (r - S::C / 2 - 1);
}
// With X the length-2N transform of the real row and H the kernel's, E = (Z[k] + conj Z[N-k]) / 2
// and O = (Z[k] - conj Z[N-k]) / 2i give X[k] = E + w O, conj X[N-k] = E - w O, w = exp(-pi i k / N).
// H X in the same form is E' = s E + d w O, O' = s O + d conj(w) E with s = (H[k] + conj H[N-k]) / 2,
// d = (H[k] - conj H[N-k]) / 2.  An even kernel's H is real (h1 = H[k], h2 = H[N-k]); an odd one's
// is i h, the factor i leaves the sums and (h1, -h2) take the places of (h1, h2).  The halves of E
// and O and the inverse transform's 1 / N go into s and t = d w.
FCB_HD f4 spectrum_entry(double h1, double h2, bool odd, double wr, double wi, int N)
{
  if (odd) h2 = -h2;
  const double c = 0.25 / N;
  const double s = c * (h1 + h2), d = c * (h1 - h2);
  return {(float)s, (float)(d * wr), (float)(d * wi), 0.0f};
}

// =====================================================================================
// Device side
// =====================================================================================
#if defined(__CUDACC__)

// Tables in FP64, one thread per entry.
// time-domain kernel of a real even frequency response f of a cyclic length Lf: h[m], m < W
static __global__ void rc_time_kernel(const double* __restrict__ f, int nb, int Lf, int W, double* __restrict__ h)
{
  __shared__ double part[128];
  const int m = blockIdx.x;
  double a = 0.0;
  for (int k = threadIdx.x; k < nb; k += 128) {
    const double c = (k == 0 || 2 * k == Lf) ? 1.0 : 2.0;
    a += c * f[k] * cospi(2.0 * (double)(int)(((long long)k * m) % Lf) / (double)Lf);
  }
  part[threadIdx.x] = a;
  __syncthreads();
  for (int o = 64; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) h[m] = part[0] / Lf;
}
// spectrum over L = 2 N of the kernel h[0 .. W) (even), or, h null, of the band-limited Hilbert
// kernel 2 / (pi m), m odd (odd: H = i times the value)
static __global__ void rc_spec_kernel(const double* __restrict__ h, int W, int N, double* __restrict__ H)
{
  __shared__ double part[128];
  const int k = blockIdx.x;
  double a = 0.0;
  for (int m = threadIdx.x; m < W; m += 128) {
    const double ph = (double)(int)(((long long)k * m) % (2 * N)) / (double)N;
    if (h) a += (m ? 2.0 : 1.0) * h[m] * cospi(ph);
    else if (m & 1) a -= 2.0 * (2.0 / (M_PI * m)) * sinpi(ph);
  }
  part[threadIdx.x] = a;
  __syncthreads();
  for (int o = 64; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) H[k] = part[0];
}
template <class S>
__global__ void rc_table_kernel(const double* __restrict__ H, bool odd, cf* t1, cf* t2, f4* g)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < S::T1) {
    const int k1 = i / S::BC, m = i % S::BC;
    const double ph = -2.0 * (double)((k1 * m) % S::N) / (double)S::N;
    t1[i] = {(float)cospi(ph), (float)sinpi(ph)};
  }
  if (i < S::T2) {
    const int k2 = i / S::C, n3 = i % S::C;
    const double ph = -2.0 * (double)((k2 * n3) % S::BC) / (double)S::BC;
    t2[i] = {(float)cospi(ph), (float)sinpi(ph)};
  }
  if (i <= S::G) {
    const int k = entry_k<S>(i);
    const double ph = -(double)k / (double)S::N;
    g[i] = spectrum_entry(H[k], H[S::N - k], odd, cospi(ph), sinpi(ph), S::N);
  }
}

// One persistent CTA per SM: the tables, GPC groups of T threads, and R row buffers per group.
template <class S_, int T_, int R_, int GPC_>
struct Config {
  using S = S_;
  static constexpr int T = T_, R = R_, GPC = GPC_;
  static constexpr int TABLE = (S::G + 1) * (int)sizeof(f4) + (S::T1 + S::T2) * (int)sizeof(cf);
  static constexpr int SMEM = TABLE + GPC * R * S::BUF * (int)sizeof(cf);
  static constexpr int ROUNDS = (R * S::NB1 + T - 1) / T;  // stage-1 butterflies per thread
  static_assert(SMEM <= 227 * 1024 && T % 32 == 0 && T * GPC <= 1024 && (T == 32 || GPC <= 15), "row transform CTA");
};

template <class K, bool ODD, class IO>
__global__ void __launch_bounds__(K::T * K::GPC, 1) rowconv_kernel(const IO io, const uint4* __restrict__ tables,
                                                                   long long row0, int nrows)
{
  using S = typename K::S;
  extern __shared__ __align__(16) unsigned char rc_smem[];
  for (int i = threadIdx.x; i < K::TABLE / 16; i += K::T * K::GPC) reinterpret_cast<uint4*>(rc_smem)[i] = tables[i];
  const f4* g = reinterpret_cast<const f4*>(rc_smem);
  const cf* t1 = reinterpret_cast<const cf*>(g + S::G + 1);
  const cf* t2 = t1 + S::T1;
  const int grp = threadIdx.x / K::T, tid = threadIdx.x % K::T;
  cf* buf = reinterpret_cast<cf*>(rc_smem + K::TABLE) + grp * K::R * S::BUF;
  auto sync = [grp] {
    if constexpr (K::T == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(K::T) : "memory");
  };
  // groups take R rows at a time, consecutive ones on different SMs
  const int stride = K::GPC * gridDim.x * K::R;
  int r0 = (grp * gridDim.x + blockIdx.x) * K::R;
  cf x[K::ROUNDS][S::HA];  // the next rows' values, loaded while the current ones are transformed
  auto fetch = [&](int rn) {
#pragma unroll
    for (int i = 0; i < K::ROUNDS; i++) {
      const int b = tid + i * K::T, r = b / S::NB1, m = b % S::NB1;
      const bool in = r < K::R && rn + r < nrows;
#pragma unroll
      for (int a = 0; a < S::HA; a++) x[i][a] = in ? io.load(row0 + rn + r, a * S::BC + m) : cf{0.0f, 0.0f};
    }
  };
  fetch(r0);
  __syncthreads();
  for (; r0 < nrows; r0 += stride) {
    const int nr = min(K::R, nrows - r0);
#pragma unroll
    for (int i = 0; i < K::ROUNDS; i++) {
      const int b = tid + i * K::T, r = b / S::NB1, m = b % S::NB1;
      if (r < nr) {
        const auto row = io.row(row0 + r0 + r);
#pragma unroll
        for (int a = 0; a < S::HA; a++) x[i][a] = io.weigh(row, a * S::BC + m, x[i][a]);
        stage1<S>(x[i], m, buf + r * S::BUF, t1);
      }
    }
    if (r0 + stride < nrows) fetch(r0 + stride);
    sync();
    if constexpr (S::B > 1) {
      for (int b = tid; b < nr * S::NB2; b += K::T) stage2<S, false>(b % S::NB2, buf + b / S::NB2 * S::BUF, t2);
      sync();
    }
    for (int b = tid; b < nr * S::NB3; b += K::T) stage3<S, ODD>(b % S::NB3, buf + b / S::NB3 * S::BUF, g);
    sync();
    if constexpr (S::B > 1) {
      for (int b = tid; b < nr * S::NB2; b += K::T) stage2<S, true>(b % S::NB2, buf + b / S::NB2 * S::BUF, t2);
      sync();
    }
    for (int b = tid; b < nr * S::NB1; b += K::T) {
      const int r = b / S::NB1, m = b % S::NB1;
      cf y[S::HA];
      stage1_back<S>(y, m, buf + r * S::BUF, t1);
#pragma unroll
      for (int a = 0; a < S::HA; a++) io.store(row0 + r0 + r, a * S::BC + m, y[a]);
    }
    sync();  // the next rows overwrite the buffers
  }
}

// f(Config) for the smallest size N >= W (work grows with N: a width just above a size pays for the next
// one and its fewer rows per SM, 64 x 256 rows of 512 and 513 values 63 and 89 us, 1024 and 1025 106 and
// 182, 2048 and 2049 217 and 323, where cuFFT between its passes took 182 and 269, 345 and 1298, 682 and
// 2731; at every width measured from 48 to 4096 less than half of its time); false when there is none
// (W > RC_MAX_W).
constexpr int RC_MAX_W = 4096;
template <class F>
bool rc_dispatch(int W, F&& f)
{
  if (W <= 32) f(Config<Shape<8, 1, 4>, 32, 8, 16>{});
  else if (W <= 48) f(Config<Shape<12, 1, 4>, 32, 16, 16>{});
  else if (W <= 64) f(Config<Shape<8, 1, 8>, 32, 8, 16>{});
  else if (W <= 96) f(Config<Shape<12, 1, 8>, 32, 16, 15>{});
  else if (W <= 128) f(Config<Shape<16, 1, 8>, 32, 4, 16>{});
  else if (W <= 192) f(Config<Shape<12, 4, 4>, 32, 4, 16>{});
  else if (W <= 256) f(Config<Shape<16, 1, 16>, 32, 4, 12>{});
  else if (W <= 384) f(Config<Shape<12, 8, 4>, 32, 2, 16>{});
  else if (W <= 512) f(Config<Shape<8, 8, 8>, 32, 1, 16>{});
  else if (W <= 768) f(Config<Shape<12, 8, 8>, 32, 2, 15>{});
  else if (W <= 1024) f(Config<Shape<16, 8, 8>, 32, 1, 16>{});
  else if (W <= 1536) f(Config<Shape<12, 16, 8>, 32, 1, 13>{});
  else if (W <= 2048) f(Config<Shape<16, 16, 8>, 64, 1, 9>{});
  else if (W <= 3072) f(Config<Shape<12, 16, 16>, 96, 1, 5>{});
  else if (W <= RC_MAX_W) f(Config<Shape<16, 16, 16>, 128, 1, 4>{});
  else return false;
  return true;
}

// The tables of one kernel and row length: one device block, made once, read-only afterwards.
struct RowConv {
  int W = 0;
  unsigned char* block = nullptr;
  RowConv() = default;
  RowConv(const RowConv&) = delete;
  RowConv& operator=(const RowConv&) = delete;
  ~RowConv() { cudaFree(block); }

  // response (nb = Lf / 2 + 1 values of a cyclic length Lf): the even kernel it describes;
  // NULL: the odd Hilbert kernel.  Synchronous (legacy default stream).
  int create(int width, const double* response, int nb, int Lf)
  {
    W = width;
    int rc = FCB_OK;
    if (!rc_dispatch(W, [&](auto k) { rc = build<typename decltype(k)::S>(response, nb, Lf); }))
      return set_error(FCB_ERR_INVALID, "row too long for the row transform");
    return rc;
  }
  template <class S>
  int build(const double* response, int nb, int Lf)
  {
    const size_t nf = response ? nb : 0, nh = response ? W : 0;
    const size_t bytes = (S::G + 1) * sizeof(f4) + (S::T1 + S::T2) * sizeof(cf) + (nf + nh + S::N + 1) * sizeof(double);
    FCB_CUDA_TRY(cudaMalloc((void**)&block, bytes));
    f4* g = reinterpret_cast<f4*>(block);
    cf* t1 = reinterpret_cast<cf*>(g + S::G + 1);
    cf* t2 = t1 + S::T1;
    double* H = reinterpret_cast<double*>(t2 + S::T2);  // FP64 working values behind the tables
    double *f = H + S::N + 1, *h = f + nf;
    if (response) {
      FCB_CUDA_TRY(cudaMemcpy(f, response, nb * sizeof(double), cudaMemcpyHostToDevice));
      rc_time_kernel<<<W, 128>>>(f, nb, Lf, W, h);
    }
    rc_spec_kernel<<<S::N + 1, 128>>>(response ? h : nullptr, W, S::N, H);
    const int n = S::T1 > S::G + 1 ? S::T1 : S::G + 1;
    rc_table_kernel<S><<<(n + 127) / 128, 128>>>(H, response == nullptr, t1, t2, g);
    FCB_CUDA_TRY(cudaGetLastError());
    FCB_CUDA_TRY(cudaStreamSynchronize(0));  // the tables are read on any stream from here on
    return FCB_OK;
  }
  // rows that the device's row groups hold at one time
  long long wave_rows() const
  {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long n = 0;
    rc_dispatch(W, [&](auto k) { n = (long long)decltype(k)::GPC * decltype(k)::R * sms; });
    return n;
  }
  // Convolves `nrows` rows from row `first` on through `io`, stream-ordered.
  template <bool ODD, class IO>
  int run(const IO& io, long long nrows, cudaStream_t st, long long first = 0) const
  {
    int rc = FCB_OK;
    rc_dispatch(W, [&](auto k) {
      using K = decltype(k);
      rc = launch<K, ODD>(io, nrows, st, first);
    });
    return rc;
  }
  template <class K, bool ODD, class IO>
  int launch(const IO& io, long long nrows, cudaStream_t st, long long first) const
  {
    auto kern = rowconv_kernel<K, ODD, IO>;
    FCB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, K::SMEM));
    int dev = 0, sms = 148;
    FCB_CUDA_TRY(cudaGetDevice(&dev));
    FCB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (long long r0 = 0; r0 < nrows; r0 += 1 << 30) {
      const int n = (int)(nrows - r0 < (1 << 30) ? nrows - r0 : (1 << 30));
      const int units = (n + K::R - 1) / K::R;
      kern<<<(unsigned)(units < sms ? units : sms), K::T * K::GPC, K::SMEM, st>>>(
          io, reinterpret_cast<const uint4*>(block), first + r0, n);
      FCB_CUDA_TRY(cudaGetLastError());
    }
    return FCB_OK;
  }
};
#endif  // __CUDACC__

}  // namespace rf
}  // namespace fcb
