// fcb_katsevich.cu -- Katsevich filtering for helical cone-beam data (sm_100a).
//
// The reference has only the Katsevich backprojection weight (coneBeamGPU.cu:258-338) and
// expects pre-filtered, windowed data.  This file supplies the filtering of Katsevich's
// exact helical inversion in the flat-detector form of Noo, Pack & Heuscher (Phys. Med.
// Biol. 48 (2003) 3787-3818), on the virtual detector through the rotation axis
// (source-detector distance = source-axis distance D).  Detector pixel (i, j) sits at
// w = (i - W/2) pw, v = (j - H/2) pw; the published coordinate u runs along the source's
// direction of travel, u = s_u * w with s_u = -1 for a right-handed helix (angles and
// height increasing together).  Stages:
//   1. derivative at fixed ray direction  g1 = dg/dlam + (u^2+D^2)/D dg/du + u v/D dg/dv
//      and length correction g2 = D / sqrt(u^2+D^2+v^2) g1
//   2. forward height rebinning onto kappa-lines v_k(u, psi) = P/(2 pi)(psi + psi/tan(psi) u/D)
//      (per-(kappa, column) interpolation table built on the host in FP64); both stages are
//      kats_kappa_kernel, which keeps g2 in shared memory, above 768 rows (and for less than 16
//      above rf::RC_MAX_W columns) kats_deriv_kernel and kats_rebin_fwd_kernel
//   3. Hilbert transform along u, band-limited kernel (1 - cos(pi n))/(pi n): a linear
//      convolution, in place by the one-pass row transform (fcb_rowfft.cuh), for rows above
//      rf::RC_MAX_W by cuFFT on zero-padded rows; kats_hilbert_kernel is the direct O(W^2) form,
//      kept for comparison
//   4. backward rebinning through the kappa-line of smallest |psi| (kats_rebin_bwd_kernel,
//      per-(row, column) table).
// The views go through in batches.  On the 736 x 64 helix of 4640 views (one B200) the filter
// takes 3.5 ms: 2.1 ms row transforms of 594,000 kappa rows (issue-bound, see there), 1.0 ms
// kappa rows (issue 60 %, the L2 latency of tables and views), 0.4 ms backward rebinning; with
// whole-array passes and cuFFT it took 9.0 ms, with the forward rebinning inside the row
// transform's loads 6.1 ms (each warp's dependent table-then-tap loads stalled the transform).
// Backprojection with weight U over each voxel's PI interval and norm dlam/(2 pi D) then
// reconstructs (fdk_tma_kernel with the Tam-Danielsson window).
#include <cufft.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "fcb_internal.h"
#include "fcb_rowfft.cuh"

namespace fcb {

// Element-wise stages: each thread handles CPT consecutive columns (4 with 16-byte vector
// loads and stores when W is a multiple of 4, else 1); grid.x runs over the column groups of
// one view, grid.y over the views.
template <int CPT>
__device__ __forceinline__ void ldv(const float* __restrict__ p, float (&v)[CPT])
{
  if constexpr (CPT == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else {
    v[0] = *p;
  }
}
template <int CPT>
__device__ __forceinline__ void ldv(const int* __restrict__ p, int (&v)[CPT])
{
  if constexpr (CPT == 4) {
    const int4 x = *reinterpret_cast<const int4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else {
    v[0] = *p;
  }
}
template <int CPT>
__device__ __forceinline__ void stv(float* __restrict__ p, const float (&v)[CPT])
{
  if constexpr (CPT == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else *p = v[0];
}

// Reciprocals of the step sizes, computed once on the host: the kernel multiplies instead
// of dividing (no per-element IEEE division).
struct KatsDerivConst {
  float idl, hidl;   // 1 / dlam, 1 / (2 dlam)
  float idu, hidu;   // 1 / du, 1 / (2 du), du = su pw
  float ipw, hipw;   // 1 / pw, 1 / (2 pw)
  float pw, D, iD, su;
};

// One column of one view: where the differences read (central inside, one-sided at the ends:
// numpy.gradient, edge order 1) and their step sizes.
struct KatsColumn {
  const float *m, *c, *p;  // views t - 1, t, t + 1; the view itself beyond the ends
  int i, dl, dr;           // the column, the offsets of the columns to the left and right
  float sl, su;            // 1 / step between views and between columns
  float q2, q2d, u;        // u^2 + D^2, the same / D, u
};
__device__ __forceinline__ KatsColumn kats_column(const float* m, const float* c, const float* p, int i, int W,
                                                  const KatsDerivConst& K)
{
  KatsColumn X;
  X.c = c;
  X.m = m ? m : c;
  X.p = p ? p : c;
  X.i = i;
  X.sl = m && p ? K.hidl : K.idl;
  X.dl = i > 0 ? -1 : 0;
  X.dr = i < W - 1 ? 1 : 0;
  X.su = X.dr - X.dl == 2 ? K.hidu : K.idu;
  X.u = K.su * (float)(i - W / 2) * K.pw;
  X.q2 = X.u * X.u + K.D * K.D;
  X.q2d = X.q2 * K.iD;
  return X;
}
// The derivative at fixed ray direction and the length correction at row j.  I indexes a view from
// its uniform base address: 32 bits where they hold its H W values.
template <typename I>
__device__ __forceinline__ float kats_deriv(const KatsColumn& X, int j, int H, int W, const KatsDerivConst& K)
{
  const I o = (I)j * (I)W + (I)X.i;
  const I up = j > 0 ? o - (I)W : o, dn = j < H - 1 ? o + (I)W : o;
  const float dl = (X.p[o] - X.m[o]) * X.sl;
  const float dgu = (X.c[o + X.dr] - X.c[o + X.dl]) * X.su;
  const float dgv = (X.c[dn] - X.c[up]) * (j > 0 && j < H - 1 ? K.hipw : K.ipw);
  const float v = (float)(j - H / 2) * K.pw;
  const float g1 = dl + X.q2d * dgu + (X.u * v * K.iD) * dgv;
  return g1 * (K.D * rsqrtf(X.q2 + v * v));
}

// What a column of view `tl` of the batch from view t0 on differentiates; `before` is view
// t0 - 1 (null at the first view).
__device__ __forceinline__ KatsColumn kats_view(const float* g, const float* before, int t0, int tl, int n, size_t plane,
                                                int i, int W, const KatsDerivConst& C)
{
  const int t = t0 + tl;
  const float* c = g + (size_t)t * plane;
  return kats_column(t == 0 ? nullptr : tl == 0 ? before : c - plane, c, t + 1 < n ? c + plane : nullptr, i, W, C);
}

// Derivative and forward rebinning: the kappa rows of views t0 + blockIdx.y * kv ... (nv of
// them in all), columns blockIdx.x * 32 + lane, at a row pitch of L:
//   out[tl][k][i] = g2[j0] * (1 - a) + g2[j0 + 1] * a from the (kappa, column) table (j0, a).
// The strip's derivatives of one view sit in shared memory between the two, since each is read about
// 2 K / H times (the strip takes 128 bytes a row: up to 768 rows leave two CTAs per SM).  A CTA takes
// KK_VIEWS views where that leaves 20 CTAs' views per SM (736 x 64, 4640 views: 3.50 ms for the whole
// filter, 3.58 with one), else one (64 x 700, 80 views: 80 us, 178 with four).
// I: as in kats_deriv, for the K L values too.
constexpr int KK_VIEWS = 4;
template <typename I>
__global__ void __launch_bounds__(256, 5) kats_kappa_kernel(const float* __restrict__ g,
                                                            const float* __restrict__ before,
                                                            float* __restrict__ out, const float2* __restrict__ tab,
                                                            int n, int H, int W, int K, int L, int t0, int nv, int kv,
                                                            const KatsDerivConst C)
{
  extern __shared__ float kk_g2[];  // [H][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  const int l0 = blockIdx.y * kv, l1 = min(nv, l0 + kv);
  for (int tl = l0; tl < l1; tl++) {
    if (i < W) {
      const KatsColumn X = kats_view(g, before, t0, tl, n, (size_t)H * W, i, W, C);
#pragma unroll 2
      for (int j = warp; j < H; j += 8) kk_g2[j * 32 + lane] = kats_deriv<I>(X, j, H, W, C);
    }
    __syncthreads();
    if (i < W) {
      float* row = out + (size_t)tl * K * L;
#pragma unroll 4
      for (int k = warp; k < K; k += 8) {
        const float2 ja = __ldg(tab + ((I)k * (I)W + (I)i));
        const int j0 = __float_as_int(ja.x);
        float val = 0.0f;
        if (j0 >= 0) {  // (and at most H - 2)
          const float v0 = kk_g2[j0 * 32 + lane], v1 = kk_g2[j0 * 32 + lane + 32];
          val = fmaf(ja.y, v1 - v0, v0);
        }
        row[(I)k * (I)L + (I)i] = val;
      }
    }
    __syncthreads();
  }
}

// The same in two passes over global memory, columns across the CTA and KK_ROWS rows or lines per CTA
// (blockIdx.z), for detectors too tall to stage a strip (128 x 1000, 80 views: 176 us for the whole
// filter, 511 where every tap was derived where it is read), and for a few rows beyond the row transform's
// length, whose strips are too little work per CTA (8192 x 8, 600 views: 1.41 ms, 1.51 staged).
constexpr int KK_ROWS = 16;
template <typename I>
__global__ void __launch_bounds__(256) kats_deriv_kernel(const float* __restrict__ g, const float* __restrict__ before,
                                                         float* __restrict__ g2, int n, int H, int W, int t0,
                                                         const KatsDerivConst C)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x, tl = blockIdx.y;
  if (i >= W) return;
  const KatsColumn X = kats_view(g, before, t0, tl, n, (size_t)H * W, i, W, C);
  float* out = g2 + (size_t)tl * H * W;
  const int j0 = blockIdx.z * KK_ROWS, j1 = min(H, j0 + KK_ROWS);
#pragma unroll 4
  for (int j = j0; j < j1; j++) out[(I)j * (I)W + (I)i] = kats_deriv<I>(X, j, H, W, C);
}
template <typename I>
__global__ void __launch_bounds__(256) kats_rebin_fwd_kernel(const float* __restrict__ g2, float* __restrict__ out,
                                                             const float2* __restrict__ tab, int H, int W, int K, int L)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x, tl = blockIdx.y;
  if (i >= W) return;
  const float* col = g2 + (size_t)tl * H * W + i;
  float* row = out + (size_t)tl * K * L;
  const int k0 = blockIdx.z * KK_ROWS, k1 = min(K, k0 + KK_ROWS);
#pragma unroll 4
  for (int k = k0; k < k1; k++) {
    const float2 ja = __ldg(tab + ((I)k * (I)W + (I)i));
    const int j0 = __float_as_int(ja.x);
    float val = 0.0f;
    if (j0 >= 0) {  // (and at most H - 2)
      const float* c = col + (I)j0 * (I)W;
      const float v0 = c[0], v1 = c[W];
      val = fmaf(ja.y, v1 - v0, v0);
    }
    row[(I)k * (I)L + (I)i] = val;
  }
}

// kappa rows for rf::rowconv_kernel, in place at an even pitch of L
struct KatsRows {
  float* g;
  int W, L;
  struct Row {};
  __device__ __forceinline__ Row row(long long) const { return Row{}; }
  __device__ __forceinline__ rf::cf load(long long gr, int n) const
  {
    if (2 * n >= W) return rf::cf{0.0f, 0.0f};
    const float2 v = *reinterpret_cast<const float2*>(g + (size_t)gr * L + 2 * n);
    return rf::cf{v.x, 2 * n + 1 < W ? v.y : 0.0f};
  }
  __device__ __forceinline__ rf::cf weigh(const Row&, int, rf::cf v) const { return v; }
  __device__ __forceinline__ void store(long long gr, int n, rf::cf v) const
  {
    if (2 * n < W) *reinterpret_cast<float2*>(g + (size_t)gr * L + 2 * n) = make_float2(v.x, v.y);
  }
};

// Hilbert transform of each row along u: out[i] = sgn * sum_j h(i - j) in[j],
// h(m) = 2 / (pi m) for odd m, 0 otherwise; one block per row (stride L), the row staged in
// shared memory (so the transform may run in place).
__global__ void kats_hilbert_kernel(float* __restrict__ rows, int W, int L, float sgn)
{
  extern __shared__ float row[];
  const size_t r = blockIdx.x;
  for (int j = threadIdx.x; j < W; j += blockDim.x) row[j] = rows[r * L + j];
  __syncthreads();
  const float c = sgn * 0.63661977236758134f;  // 2 / pi
  for (int i = threadIdx.x; i < W; i += blockDim.x) {
    float acc = 0.0f;
    // j = i - m with m odd: j runs over the columns of opposite parity to i
    for (int j = (i & 1) ^ 1; j < W; j += 2) acc = fmaf(row[j], __frcp_rn((float)(i - j)), acc);
    rows[r * L + i] = c * acc;
  }
}

// spec[r][k] *= i * himag[k] (the kernel is odd, so its spectrum is purely imaginary)
// One block per row.
__global__ void kats_spec_kernel(cufftComplex* __restrict__ spec, const float* __restrict__ himag,
                                 int nb)
{
  cufftComplex* row = spec + (size_t)blockIdx.x * nb;
  for (int k = threadIdx.x; k < nb; k += blockDim.x) {
    const float h = himag[k];
    const cufftComplex z = row[k];
    row[k] = make_cuFloatComplex(-z.y * h, z.x * h);
  }
}

// gF[t0 + tl][j][i] = scale * (g4[tl][k0][i] * (1-a) + g4[tl][k0+1][i] * a) from the
// (row, column) table; g4 holds the transformed kappa rows (length L) of views t0, t0 + 1, ...
template <int CPT>
__global__ void kats_rebin_bwd_kernel(const float* __restrict__ g4, float* __restrict__ gF,
                                      const int* __restrict__ k0tab, const float* __restrict__ atab,
                                      int H, int W, int K, int L, float scale, int t0)
{
  const int Wq = W / CPT;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= H * Wq) return;
  const int tl = blockIdx.y;
  const int j = q / Wq, i0 = (q - j * Wq) * CPT;
  int k0[CPT];
  float a[CPT], r[CPT];
  ldv<CPT>(k0tab + (size_t)j * W + i0, k0);
  ldv<CPT>(atab + (size_t)j * W + i0, a);
  const float* base = g4 + (size_t)tl * K * L + i0;
#pragma unroll
  for (int m = 0; m < CPT; m++) {
    const float* col = base + m;
    const float v0 = col[(size_t)k0[m] * L], v1 = col[(size_t)(k0[m] + 1) * L];
    r[m] = scale * fmaf(a[m], v1 - v0, v0);
  }
  stv<CPT>(gF + ((size_t)(t0 + tl) * H + j) * W + i0, r);
}

}  // namespace fcb

using namespace fcb;

// np.interp-style lookup on an increasing abscissa: fractional index of x in xs.
static double frac_index(const std::vector<double>& xs, double x)
{
  const int n = (int)xs.size();
  if (x <= xs[0]) return 0.0;
  if (x >= xs[n - 1]) return (double)(n - 1);
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (xs[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo + (x - xs[lo]) / (xs[hi] - xs[lo]);
}

// A strip of 32 columns of a view's derivatives, and whether it is staged (see kats_kappa_kernel).
static size_t kats_strip(int H) { return (size_t)H * 32 * sizeof(float); }
static bool kats_staged(int H, int W) { return kats_strip(H) <= 96 * 1024 && (W <= rf::RC_MAX_W || H >= 16); }

static float int_bits(int v)
{
  float f;
  memcpy(&f, &v, sizeof f);
  return f;
}

// Reusable Katsevich filter for one helix and detector: the kappa-line tables, the Hilbert
// kernel's spectrum and the buffers of one batch of views are made once; execute() is
// stream-ordered, allocates nothing and does not synchronise.
struct fcb_katsevich_plan {
  int nviews = 0, H = 0, W = 0, K = 0;
  int vb = 0;  // views per batch
  int L = 0;   // row pitch of g4 (and g3): W rounded up to 4 in the row transform, 2 W for cuFFT
  float dlam = 0.0f, pw = 0.0f, D = 0.0f, su = 0.0f;
  float2* dfja = nullptr;  // forward table
  int* dbk = nullptr;      // backward table
  float* dba = nullptr;
  float* g4 = nullptr;     // kappa rows of one batch [vb][K][L], transformed in place
  float* edge = nullptr;   // the view before a batch, when out is in
  float* g2 = nullptr;     // two passes: derivatives of one batch [vb][H][W]
  int sms = 148;
  rf::RowConv conv;  // rows up to rf::RC_MAX_W
  // longer rows: cuFFT
  int nb = 0;
  float* g3 = nullptr;  // kappa rows of one batch, [W, L) zero
  float* dhim = nullptr;
  cufftComplex* hspec = nullptr;
  cufftHandle pf = 0, pi = 0;
  ~fcb_katsevich_plan()
  {
    if (pf) cufftDestroy(pf);
    if (pi) cufftDestroy(pi);
    cudaFree(g3); cudaFree(g4); cudaFree(g2); cudaFree(edge); cudaFree(dfja); cudaFree(dba); cudaFree(dbk);
    cudaFree(hspec); cudaFree(dhim);
  }
};

extern "C" int fcb_katsevich_plan_create(int nviews, int H, int W, const float* angles, float D,
                                         float pw, float pitch, int nkappa,
                                         fcb_katsevich_plan** out)
try {
  if (!out) return set_error(FCB_ERR_INVALID, "plan output pointer is NULL");
  *out = nullptr;
  if (!angles || nviews < 2 || H < 2 || W < 2 || !(D > 0) || !(pw > 0) || pitch == 0.0f)
    return set_error(FCB_ERR_INVALID, "bad Katsevich filter arguments");
  if (nviews > 65535 || H > 32768 || (nkappa > 1 && nkappa > 65535))
    return set_error(FCB_ERR_INVALID, "Katsevich filter sizes above the grid limits (65535 views)");
  // mean angular step; float32 angles of several turns carry ~1e-6 rad of rounding each
  const double dlam = ((double)angles[nviews - 1] - (double)angles[0]) / (nviews - 1);
  for (int t = 1; t < nviews; t++) {
    const double d = (double)angles[t] - (double)angles[t - 1];
    if (fabs(d - dlam) > 1e-3 * fabs(dlam) + 1e-5)
      return set_error(FCB_ERR_INVALID, "Katsevich filtering needs uniformly spaced views");
  }
  const double turn = (double)angles[nviews - 1] - (double)angles[0];
  const double su = ((turn >= 0.0) == (pitch >= 0.0)) ? -1.0 : 1.0;
  const int K = nkappa > 1 ? nkappa : 2 * H;
  // kappa-line tables (FP64): v_k(u_i, psi_k), forward (kappa, column) and backward (row, column)
  std::vector<double> u(W), v(H);
  for (int i = 0; i < W; i++) u[i] = su * (double)(i - W / 2) * pw;
  for (int j = 0; j < H; j++) v[j] = (double)(j - H / 2) * pw;
  double umax = 0.0;
  for (int i = 0; i < W; i++) umax = std::max(umax, fabs(u[i]));
  const double am = atan(umax / D);
  const double P = pitch;
  std::vector<float2> fja((size_t)K * W);  // (j0 as bits, a)
  std::vector<int> bk0((size_t)H * W);
  std::vector<float> ba((size_t)H * W);
  std::vector<double> vk(K);
  for (int i = 0; i < W; i++) {
    for (int k = 0; k < K; k++) {
      const double psi = -M_PI / 2 - am + (M_PI + 2 * am) * k / (double)(K - 1);
      const double cot = fabs(psi) < 1e-12 ? 1.0 : psi / tan(psi);
      vk[k] = (P / (2 * M_PI)) * (psi + cot * u[i] / D);
      // forward: linear interpolation in v, zero outside the detector rows
      const double x = vk[k];
      if (x < v[0] || x > v[H - 1]) {
        fja[(size_t)k * W + i] = make_float2(int_bits(-1), 0.0f);
      } else {
        const double f = frac_index(v, x);
        const int j0 = std::min((int)floor(f), H - 2);
        fja[(size_t)k * W + i] = make_float2(int_bits(j0), (float)(f - j0));
      }
    }
    for (int j = 0; j < H; j++) {
      const double f = frac_index(vk, v[j]);
      const int k0 = std::min((int)floor(f), K - 2);
      bk0[(size_t)j * W + i] = k0;
      ba[(size_t)j * W + i] = (float)(f - k0);
    }
  }
  auto* pl = new fcb_katsevich_plan();
  pl->nviews = nviews; pl->H = H; pl->W = W; pl->K = K;
  pl->dlam = (float)dlam; pl->pw = pw; pl->D = D; pl->su = (float)su;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&pl->sms, cudaDevAttrMultiProcessorCount, dev);
  const bool fused = W <= rf::RC_MAX_W;
  int rc = FCB_OK;
  do {
    if (cudaMalloc(&pl->dfja, fja.size() * sizeof(float2)) || cudaMalloc(&pl->dba, ba.size() * 4) ||
        cudaMalloc(&pl->dbk, bk0.size() * 4)) {
      cudaGetLastError();
      rc = set_error(FCB_ERR_NOMEM, "Katsevich filter tables");
      break;
    }
    if (cudaMemcpy(pl->dfja, fja.data(), fja.size() * sizeof(float2), cudaMemcpyHostToDevice) ||
        cudaMemcpy(pl->dba, ba.data(), ba.size() * 4, cudaMemcpyHostToDevice) ||
        cudaMemcpy(pl->dbk, bk0.data(), bk0.size() * 4, cudaMemcpyHostToDevice)) {
      rc = set_error(FCB_ERR_CUDA, "Katsevich table upload failed");
      break;
    }
    if (fused) {
      rc = pl->conv.create(W, nullptr, 0, 0);
      if (rc) break;
      pl->L = (W + 3) & ~3;
      // Kappa rows of a batch: up to 512 MB, whole waves of the row transform where they fill
      // one.  Batches that stay in L2 do not pay: the three kernels are not bound by HBM, and
      // each of their launches ends in a partly filled wave (the helix above: 64 MB of rows
      // 4.10 ms, 128 MB 3.92, 256 MB 3.68, 512 MB 3.54, 1 GB 3.44).
      long long budget = 512ll << 20;
      if (const char* e = getenv("FCB_KATS_BATCH_MB")) budget = (long long)std::max(1, atoi(e)) << 20;
      long long vb = std::max<long long>(1, budget / (4ll * pl->L * (kats_staged(H, W) ? K : std::max(K, H))));
      const long long wave = pl->conv.wave_rows();
      if (vb * K >= wave) vb = vb * K / wave * wave / K;
      pl->vb = (int)std::min<long long>(nviews, std::max<long long>(1, vb));
    } else {
      // transform batches of whole views, up to 256 MiB of spectra each
      pl->L = 2 * W;
      pl->nb = W + 1;
      pl->vb = (int)std::min<long long>(nviews, std::max<long long>(1, (256ll << 20) / (8ll * pl->nb * K)));
    }
    const long long rows = (long long)pl->vb * K;
    if (cudaMalloc(&pl->edge, (size_t)H * W * 4) || cudaMalloc(&pl->g4, (size_t)rows * pl->L * 4) ||
        (!kats_staged(H, W) && cudaMalloc(&pl->g2, (size_t)pl->vb * H * W * 4))) {
      cudaGetLastError();
      rc = set_error(FCB_ERR_NOMEM, "Katsevich filter scratch");
      break;
    }
    if (fused) break;
    // spectrum of the Hilbert kernel embedded in L = 2W: h(m) = 2/(pi m) for odd m,
    // h(L-m) = -h(m); H[k] = -2 i sum_{m odd < W} h(m) sin(2 pi k m / L)
    const int L = pl->L, nb = pl->nb;
    std::vector<float> himag(nb);
    for (int k = 0; k < nb; k++) {
      double acc = 0.0;
      for (int m = 1; m < W; m += 2) acc += (2.0 / (M_PI * m)) * sin(2.0 * M_PI * (double)k * m / L);
      himag[k] = (float)(-2.0 * acc);
    }
    if (cudaMalloc(&pl->g3, (size_t)rows * L * 4) || cudaMalloc(&pl->dhim, nb * 4) ||
        cudaMalloc(&pl->hspec, (size_t)rows * nb * sizeof(cufftComplex))) {
      cudaGetLastError();
      rc = set_error(FCB_ERR_NOMEM, "Katsevich filter scratch");
      break;
    }
    if (cudaMemset(pl->g3, 0, (size_t)rows * L * 4) != cudaSuccess ||
        cudaMemcpy(pl->dhim, himag.data(), nb * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
      rc = set_error(FCB_ERR_CUDA, "Katsevich scratch initialisation failed");
      break;
    }
    int n1[1] = {L};
    if (cufftPlanMany(&pl->pf, 1, n1, nullptr, 1, L, nullptr, 1, nb, CUFFT_R2C, (int)rows) != CUFFT_SUCCESS ||
        cufftPlanMany(&pl->pi, 1, n1, nullptr, 1, nb, nullptr, 1, L, CUFFT_C2R, (int)rows) != CUFFT_SUCCESS) {
      rc = set_error(FCB_ERR_CUDA, "cufftPlanMany failed");
      break;
    }
  } while (0);
  if (rc) {
    delete pl;
    return rc;
  }
  *out = pl;
  return ok();
}
FCB_CATCH_STATUS

extern "C" int fcb_katsevich_plan_execute(fcb_katsevich_plan* pl, const float* in, float* out,
                                          void* stream)
try {
  if (!pl || !in || !out) return set_error(FCB_ERR_INVALID, "NULL plan or buffer");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int nviews = pl->nviews, H = pl->H, W = pl->W, K = pl->K, L = pl->L, nb = pl->nb, vb = pl->vb;
  // 16-byte vector accesses need 4 | W and 16-byte aligned caller buffers (the plan's own are)
  const bool v4 = (W % 4) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  const int cpt = v4 ? 4 : 1;
  const unsigned bx_hw = (unsigned)(((long long)H * (W / cpt) + 255) / 256);
  KatsDerivConst KC;
  {
    const double dl = pl->dlam, du = (double)pl->su * pl->pw, pw = pl->pw, D = pl->D;
    KC.idl = (float)(1.0 / dl);
    KC.hidl = (float)(0.5 / dl);
    KC.idu = (float)(1.0 / du);
    KC.hidu = (float)(0.5 / du);
    KC.ipw = (float)(1.0 / pw);
    KC.hipw = (float)(0.5 / pw);
    KC.pw = pl->pw;
    KC.D = pl->D;
    KC.iD = (float)(1.0 / D);
    KC.su = pl->su;
  }
  // the published Hilbert transform runs along increasing u; along w it changes sign when u = -w
  const char* de = getenv("FCB_KATS_DIRECT_HILBERT");
  const bool direct = de && de[0] == '1';  // the direct sum, for comparison
  const bool fused = W <= rf::RC_MAX_W;
  if (!fused && (cufftSetStream(pl->pf, st) != CUFFT_SUCCESS || cufftSetStream(pl->pi, st) != CUFFT_SUCCESS))
    return set_error(FCB_ERR_CUDA, "cufftSetStream failed");
  // out may be in: a batch's derivatives also read the last view of the batch before, which is
  // kept aside before that batch is written.  Buffers that overlap in some other way go through
  // a copy.
  const size_t plane = (size_t)H * W, nhw = (size_t)nviews * plane;
  const float* src = in;
  float* copy = nullptr;
  if (in != out && in < out + nhw && out < in + nhw) {
    FCB_TRY(scratch_alloc((void**)&copy, nhw * sizeof(float), st));
    src = copy;
    const cudaError_t e = cudaMemcpyAsync(copy, in, nhw * sizeof(float), cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) {
      scratch_free(copy, st);
      return set_error(FCB_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  const bool stage = kats_staged(H, W);
  const bool wide = std::max((long long)H * W, (long long)K * L) > 0x7fffffffll;  // 64-bit indices
  auto kappa = wide ? kats_kappa_kernel<size_t> : kats_kappa_kernel<unsigned>;
  auto deriv = wide ? kats_deriv_kernel<size_t> : kats_deriv_kernel<unsigned>;
  auto rebin = wide ? kats_rebin_fwd_kernel<size_t> : kats_rebin_fwd_kernel<unsigned>;
  if (stage) FCB_CUDA_TRY(cudaFuncSetAttribute(kappa, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
  const unsigned strips = (unsigned)((W + 31) / 32), bx = std::min(256u, strips * 32), gx = (W + bx - 1) / bx;
  // one batch: kappa rows of views [t0, t0 + nv), their Hilbert transform, backward rebinning
  auto batch = [&](int t0, int nv) -> int {
    const long long rows = (long long)nv * K;
    float* g3 = fused || direct ? pl->g4 : pl->g3;
    const float* before = t0 == 0 ? nullptr : in == out ? pl->edge : src + (size_t)(t0 - 1) * plane;
    if (stage) {
      const int kv = (long long)strips * nv >= 20ll * pl->sms ? KK_VIEWS : 1;
      kappa<<<dim3(strips, (nv + kv - 1) / kv), 256, kats_strip(H), st>>>(src, before, g3, pl->dfja, nviews, H, W, K, L, t0,
                                                                          nv, kv, KC);
    } else {
      deriv<<<dim3(gx, nv, (H + KK_ROWS - 1) / KK_ROWS), bx, 0, st>>>(src, before, pl->g2, nviews, H, W, t0, KC);
      rebin<<<dim3(gx, nv, (K + KK_ROWS - 1) / KK_ROWS), bx, 0, st>>>(pl->g2, g3, pl->dfja, H, W, K, L);
    }
    FCB_CUDA_TRY(cudaGetLastError());
    if (in == out && t0 + nv < nviews)
      FCB_CUDA_TRY(cudaMemcpyAsync(pl->edge, in + (size_t)(t0 + nv - 1) * plane, plane * sizeof(float),
                                   cudaMemcpyDeviceToDevice, st));
    float scale = pl->su;
    if (direct) {
      kats_hilbert_kernel<<<(unsigned)rows, 256, W * sizeof(float), st>>>(g3, W, L, pl->su);
      scale = 1.0f;
    } else if (fused) {
      FCB_TRY(pl->conv.run<true>(KatsRows{pl->g4, W, L}, rows, st));
    } else {
      // R2C of the zero-padded kappa rows (the padding in g3 stays zero), multiplication by the
      // kernel's spectrum, C2R into g4; the backward rebinning applies 1/L and the sign
      if (cufftExecR2C(pl->pf, g3, pl->hspec) != CUFFT_SUCCESS) return set_error(FCB_ERR_CUDA, "cufftExecR2C failed");
      kats_spec_kernel<<<(unsigned)rows, 256, 0, st>>>(pl->hspec, pl->dhim, nb);
      if (cufftExecC2R(pl->pi, pl->hspec, pl->g4) != CUFFT_SUCCESS) return set_error(FCB_ERR_CUDA, "cufftExecC2R failed");
      scale = pl->su / (float)L;
    }
    if (v4) kats_rebin_bwd_kernel<4><<<dim3(bx_hw, nv), 256, 0, st>>>(pl->g4, out, pl->dbk, pl->dba, H, W, K, L, scale, t0);
    else kats_rebin_bwd_kernel<1><<<dim3(bx_hw, nv), 256, 0, st>>>(pl->g4, out, pl->dbk, pl->dba, H, W, K, L, scale, t0);
    FCB_CUDA_TRY(cudaGetLastError());
    return FCB_OK;
  };
  int rc = FCB_OK;
  for (int t0 = 0; t0 < nviews && rc == FCB_OK; t0 += vb) rc = batch(t0, std::min(vb, nviews - t0));
  scratch_free(copy, st);
  if (rc) return rc;
  FCB_CUDA_TRY(cudaGetLastError());
  return ok();
}
FCB_CATCH_STATUS

extern "C" int fcb_katsevich_plan_destroy(fcb_katsevich_plan* pl)
try {
  delete pl;
  return ok();
}
FCB_CATCH_STATUS

extern "C" int fcb_katsevich_filter_device(const float* in, float* out, int nviews, int H, int W,
                                           const float* angles, float D, float pw, float pitch,
                                           int nkappa, void* stream)
try {
  if (!in || !out) return set_error(FCB_ERR_INVALID, "bad Katsevich filter arguments");
  fcb_katsevich_plan* pl = nullptr;
  FCB_TRY(fcb_katsevich_plan_create(nviews, H, W, angles, D, pw, pitch, nkappa, &pl));
  const int rc = fcb_katsevich_plan_execute(pl, in, out, stream);
  // the plan's buffers are freed below; wait for the queued work that uses them
  const cudaError_t e = cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream));
  fcb_katsevich_plan_destroy(pl);
  if (rc) return rc;
  if (e != cudaSuccess) return set_error(FCB_ERR_CUDA, cudaGetErrorString(e));
  return ok();
}
FCB_CATCH_STATUS
