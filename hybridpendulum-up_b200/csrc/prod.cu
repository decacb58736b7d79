// Clebsch-Gordan product rule of fftSO3_prod.m:209-265 (complex branch):
//   FG^l_{mn} = sum_{l1,l2} (2l1+1)(2l2+1)/(2l+1)
//               sum_{m1,n1} F^{l1}_{m1 n1} G^{l2}_{m-m1, n-n1} <l1 m1; l2 m-m1|l m><l1 n1; l2 n-n1|l n>
// These are the degrees l <= lmax of the transform of the pointwise product of
// the two functions.  The product has degrees up to 2 lmax, and against a
// degree l <= lmax its integrand is a polynomial of degree 3 lmax, which the
// quadrature of bandlimit Bg integrates exactly for 3 lmax < 2 Bg.  So, with
// the 2 Bg nodes beta_j, Bg = ceil((3B - 2) / 2):
//   S_j[m][n] = sum_l (2l+1) d^l_mn(beta_j) F^l_mn, and the same of G    (k_prod_conv)
//   H_j[m][n] = sum_{m1,n1} SF_j[m1][n1] SG_j[m-m1][n-n1]                (k_prod_conv)
//   FG^l_mn   = sum_j w_j d^l_mn(beta_j) H_j[m][n]                       (k_prod_out)
// (the sum over alpha and gamma of a product is the convolution over m and n).
// The triple sum over (l1, l2, l) with a dense Clebsch-Gordan table that this
// replaces is O(B^7) per product, this is O(B^5): B = 12, 16 products: 2.71 ms
// before.  The convolution is the bound, FP64 multiply-adds fed from shared
// memory: a thread forms R consecutive n of one m, so that a step (m1, n1)
// costs it one broadcast of SF and one new value of SG for R complex products.
#include <algorithm>
#include "common.cuh"
#include "plan.hpp"

using namespace hp;

constexpr int kProdR = 6;                     // outputs per thread of the convolution
// bytes of H per launch, less where the memory does not hold them (64 MB, which
// would stay in L2, leaves short launches: B = 20, 190 products 8.93 ms against
// 8.26; B = 32, 16 products 11.36 against 11.14)
constexpr long long kProdH = 256LL << 20;

__device__ __forceinline__ bool finite2(double2 a) { return isfinite(a.x) && isfinite(a.y); }

// What the infinite and NaN entries of SF add to H, each where it meets SG and
// nowhere else.  Called by blocks that have any, after their other sums.
__device__ __noinline__ void prod_conv_nonfinite(int B, const double* __restrict__ dj, const double2* __restrict__ Fb,
                                                 double2* sf, const double2* sg, double2* Hj) {
  const int lmax = B - 1, D = 2 * lmax + 1, SW = D + 2 * kProdR;
  for (int e = threadIdx.x; e < D * D; e += blockDim.x) {
    const int mi = e % D, ni = e / D, l0 = max(abs(mi - lmax), abs(ni - lmax));
    double2 a = make_double2(0.0, 0.0);
    for (int l = l0; l < B; ++l) {
      const long long q = e + (long long)D * D * l;
      const double w = (2 * l + 1) * dj[q];
      a.x = fma(w, Fb[q].x, a.x); a.y = fma(w, Fb[q].y, a.y);
    }
    sf[mi * D + ni] = finite2(a) ? make_double2(0.0, 0.0) : a;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < D * D; e += blockDim.x) {
    const int mi = e % D, ni = e / D;
    double2 h = Hj[e];
    for (int m1i = max(0, mi - lmax); m1i <= min(D - 1, mi + lmax); ++m1i)
      for (int n1i = max(0, ni - lmax); n1i <= min(D - 1, ni + lmax); ++n1i) {
        const double2 f = sf[m1i * D + n1i];
        if (f.x == 0.0 && f.y == 0.0) continue;
        const double2 g = sg[(mi - m1i + lmax) * SW + kProdR + ni - n1i + lmax];
        h.x = fma(f.x, g.x, fma(-f.y, g.y, h.x));
        h.y = fma(f.x, g.y, fma(f.y, g.x, h.y));
      }
    Hj[e] = h;
  }
}

// Block = (node j, product b).  SG rows have R zeros on both sides, so that the
// shifted reads need no bounds checks.  An infinite or NaN entry of SF would make
// NaN of the zeros, in entries of H that it has no part in, so those entries wait
// until the others are summed (checks in the loop itself cost 8 to 57 % of the pass, this under 1 %).
__global__ void __launch_bounds__(128) k_prod_conv(int B, int NJ, const double* __restrict__ d,
                                                   const double2* __restrict__ F, const double2* __restrict__ G,
                                                   double2* __restrict__ H) {
  const int lmax = B - 1, D = 2 * lmax + 1, SW = D + 2 * kProdR;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sf = reinterpret_cast<double2*>(smraw);     // [m][n]
  double2* sg = sf + D * D;                            // [m][R + n + R]
  const int j = blockIdx.x;
  const long long b = blockIdx.y, per = (long long)D * D * B;
  const double* dj = d + (size_t)j * D * D * B;
  const double2* Fb = F + b * per;
  const double2* Gb = G + b * per;
  for (int e = threadIdx.x; e < D * SW; e += blockDim.x) sg[e] = make_double2(0.0, 0.0);
  __syncthreads();
  bool bad = false;
  for (int e = threadIdx.x; e < D * D; e += blockDim.x) {   // e = m + D n, the order of d and F
    const int mi = e % D, ni = e / D, l0 = max(abs(mi - lmax), abs(ni - lmax));
    double2 a = make_double2(0.0, 0.0), c = a;
    for (int l = l0; l < B; ++l) {
      const long long q = e + (long long)D * D * l;
      const double w = (2 * l + 1) * dj[q];
      const double2 u = Fb[q], v = Gb[q];
      a.x = fma(w, u.x, a.x); a.y = fma(w, u.y, a.y);
      c.x = fma(w, v.x, c.x); c.y = fma(w, v.y, c.y);
    }
    bad |= !finite2(a);
    sf[mi * D + ni] = finite2(a) ? a : make_double2(0.0, 0.0);
    sg[mi * SW + kProdR + ni] = c;
  }
  bad = __syncthreads_or(bad);
  const int NR = (D + kProdR - 1) / kProdR;            // groups of R outputs per row
  double2* Hj = H + (b * NJ + j) * (long long)D * D;
  for (int it = threadIdx.x; it < D * NR; it += blockDim.x) {
    // lanes run along m: the loops over m1 differ by lane, the shifted rows do not collide
    const int mi = it % D, n0 = (it / D) * kProdR;      // m = mi - lmax, outputs n0 .. n0 + R-1 (index n + lmax)
    double2 acc[kProdR];
#pragma unroll
    for (int r = 0; r < kProdR; ++r) acc[r] = make_double2(0.0, 0.0);
    // m2 = m - m1 in [-lmax, lmax]: index mi - m1i + lmax in [0, D)
    for (int m1i = max(0, mi - lmax); m1i <= min(D - 1, mi + lmax); ++m1i) {
      const double2* fr = sf + m1i * D;
      const double2* gr = sg + (mi - m1i + lmax) * SW + kProdR;
      // n2 index = n - n1i + lmax for output n; inside [0, D) for some output of
      // the group when n1i in [n0 - lmax, n0 + R-1 + lmax]
      const int lo = max(0, n0 - lmax), hi = min(D - 1, n0 + kProdR - 1 + lmax);
      // win[r] = SG at n0 + r - n1i + lmax: one step of n1 shifts it by one
      double2 win[kProdR];
#pragma unroll
      for (int r = 0; r + 1 < kProdR; ++r) win[r] = gr[n0 + r - lo + 1 + lmax];
#pragma unroll 2
      for (int n1i = lo; n1i <= hi; ++n1i) {
#pragma unroll
        for (int r = kProdR - 1; r > 0; --r) win[r] = win[r - 1];
        win[0] = gr[n0 - n1i + lmax];
        const double2 f = fr[n1i];
#pragma unroll
        for (int r = 0; r < kProdR; ++r) {
          acc[r].x = fma(f.x, win[r].x, fma(-f.y, win[r].y, acc[r].x));
          acc[r].y = fma(f.x, win[r].y, fma(f.y, win[r].x, acc[r].y));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kProdR; ++r)
      if (n0 + r < D) Hj[mi + (long long)D * (n0 + r)] = acc[r];
  }
  if (bad) {
    __syncthreads();
    prod_conv_nonfinite(B, dj, Fb, sf, sg, Hj);
  }
}

// One thread per (m, n, l), batch element: the quadrature over the nodes.
__global__ void k_prod_out(int B, int NJ, const double* __restrict__ d, const double* __restrict__ w,
                           const double2* __restrict__ H, double2* __restrict__ FG) {
  const int lmax = B - 1, D = 2 * lmax + 1, DD = D * D;
  const int fi = blockIdx.x * blockDim.x + threadIdx.x;
  if (fi >= DD * B) return;
  const int l = fi / DD, e = fi - l * DD, m = e % D - lmax, n = e / D - lmax;
  const long long b = blockIdx.y;
  double2 acc = make_double2(0.0, 0.0);
  if (abs(m) <= l && abs(n) <= l) {
    const double2* h = H + b * NJ * DD + e;
    for (int j = 0; j < NJ; ++j) {
      const double q = w[j] * d[(size_t)j * DD * B + fi];
      const double2 v = h[(long long)j * DD];
      acc.x = fma(q, v.x, acc.x);
      acc.y = fma(q, v.y, acc.y);
    }
    // the quadrature sums over the 2Bg alpha and gamma samples; the convolution
    // is their mean
    acc.x *= (double)NJ * NJ;
    acc.y *= (double)NJ * NJ;
  }
  FG[b * DD * B + fi] = acc;
}

int hp_prod_launch(hp_plan* p, const double2* F, const double2* G, double2* FG, int batch, cudaStream_t s) {
  const int B = p->B, D = p->D, Bg = (3 * B - 1) / 2, NJ = 2 * Bg;
  if (B > 32) { hp_set_error("fftSO3_prod supports B <= 32"); return HP_ERR_UNSUPPORTED; }
  int st = HP_OK;
  bool fresh = true;
  for (auto& kv : p->ws) if (kv.first == "prod.d" && kv.second.p) fresh = false;
  const size_t nd = (size_t)D * D * B * NJ;
  // the table, the weights and the factorials of its recursion
  double* d = (double*)p->ws_get("prod.d", sizeof(double) * (nd + NJ + 2 * B), &st);
  if (st) return st;
  double* w = d + nd;
  if (fresh) {
    st = hp_tables_on_grid(p, Bg, w + NJ, d, w, s);
    if (st) { p->ws_release("prod.d"); return st; }
  }
  const long long hb = sizeof(double2) * (long long)NJ * D * D;
  long long nb = std::max(1LL, std::min<long long>(std::min(batch, 65535), kProdH / hb));
  double2* H = (double2*)p->ws_get_units("prod.H", (size_t)hb, nb, 1, &nb, &st);
  if (st) return st;
  const size_t smem = sizeof(double2) * ((size_t)D * D + (size_t)D * (D + 2 * kProdR));
  HP_CUDA_TRY(cudaFuncSetAttribute(k_prod_conv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long long per = (long long)D * D * B;
  for (long long b0 = 0; b0 < batch; b0 += nb) {
    const int k = (int)std::min(nb, batch - b0);
    ProfScope _ps(p, "prod", s);
    k_prod_conv<<<dim3(NJ, k), 128, smem, s>>>(B, NJ, d, F + b0 * per, G + b0 * per, H);
    k_prod_out<<<dim3((unsigned)((per + 127) / 128), k), 128, 0, s>>>(B, NJ, d, w, H, FG + b0 * per);
    HP_CUDA_TRY(cudaGetLastError());
  }
  return HP_OK;
}
