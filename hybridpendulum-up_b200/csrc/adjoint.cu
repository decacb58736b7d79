// Adjoint of the propagation step and the parameter gradients of a
// trajectory (reverse mode through forward-Euler steps with checkpoints).
//
// With the plain coefficient inner product <X, Y> = Re sum conj(X) Y and
// W = diag(2l+1), the derivative A = Lie + Damp + Gyro + Grav + Noise of
// pendulum.m:388-527 has the exact discrete adjoint
//   A^H = -W (Lie + Gyro + Grav - Noise) W^-1 - sum_i b_i M_i D_i
// because
//   * u^l_i is anti-Hermitian and M_i (multiply by x_i on the omega grid) is
//     self-adjoint, so the Lie term and the gyroscopic term D_i M_j M_k are
//     anti-self-adjoint and commute with W;
//   * the gravity term -D_i Grav_i is a Galerkin product with a real
//     function of R, self-adjoint in the (2l+1)-weighted inner product, so
//     Grav_i^H = W Grav_i W^-1;
//   * the noise multiplier is real and diagonal;
//   * (b_i D_i M_i)^H = -b_i M_i D_i (D_i = 2 pi i kappa / L is imaginary);
//     M_i and D_i do not commute on the grid, so this term is applied as its
//     own pass (multiply by D_i, inverse FFT, times x_i, FFT).
// The first bracket is the forward derivative kernel with b = 0, G -> -G and
// the gravity taps of W Grav W^-1 (the other terms keep l and commute with W).
// B = 12, 24^3, FP64: a reverse step's terms beyond its derivative evaluation
// took 4.3 ms as 37 passes over whole arrays; now 7 passes.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "plan.hpp"

using namespace hp;

#define ADJ_CHECK(expr)         \
  do {                          \
    int _s = (expr);            \
    if (_s != HP_OK) return _s; \
  } while (0)

namespace {

constexpr int kDotBlocks = 592;  // 4 per SM

// Lines of N points along `axis` (stride N^axis inside a row), one thread per
// line: what the axis contributes to the adjoint and to the gradients.  With
// ifft the unnormalised inverse, u = ifft(i d lam), v = ifft(F), x the grid
// coordinate and d = 2 pi kappa / L of this axis:
//   dot   += scale * weight * Re<lam, D M F> = -scale * weight / N sum_j x_j Re conj(u_j) v_j
//   out   += coef * M D lam = coef * fft(x u) / N            (out may be null)
//   Y1, Y2 = ifft(lam), ifft(F)                              (may be null)
// Lanes run along the contiguous omega index, so the strided axes read and
// write whole lines; the contiguous axis (AXIS0) goes through tiles in shared
// memory (one thread per contiguous line, straight from global memory, read
// 16 bytes of every 16 N).  v waits in shared memory while u is formed.  One
// pass of this kernel replaces a pass M D lam, a pass D M F and a dot.
template <int N> __host__ __device__ constexpr int line_threads(bool axis0) {
  return axis0 ? 64 : (N <= 32 ? 128 : 64);
}
template <int N> __host__ __device__ constexpr size_t line_smem(bool axis0) {
  return sizeof(double2) * (axis0 ? 2 * (size_t)line_threads<N>(true) * (N + 1) : (size_t)line_threads<N>(false) * N);
}

struct LineArgs {
  const double2* lam;
  const double2* F;
  double2* out;
  double2* Y1;
  double2* Y2;
  int axis;
  double coef, scale, Llen;
  int half, slot;
  double* acc;
};

__device__ __forceinline__ double row_weight(const RowLayout& L, long long row, int half) {
  return (half && L.rows[row].y > 0) ? 2.0 : 1.0;
}

// acc[slot][block] += the block's sum of v
__device__ __forceinline__ void block_add(double v, double* acc, int slot) {
  __shared__ double red[4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)blockDim.x / 32; ++k) t += red[k];
    acc[(long long)slot * gridDim.x + blockIdx.x] += t;
  }
}

template <int N, bool AXIS0>
__global__ void __launch_bounds__(line_threads<N>(AXIS0)) k_adj_line(RowLayout L, LineArgs A) {
  constexpr int NT = line_threads<N>(AXIS0);
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sv = reinterpret_cast<double2*>(smraw);   // v: AXIS0 [line][N+1], else [j][thread]
  double2* st = sv + NT * (N + 1);                   // AXIS0: the lam tile, later fft(x u)
  const int tid = threadIdx.x;
  const long long nlines = L.nrows * (L.nx / N), groups = (nlines + NT - 1) / NT;
  long long stride = 1;
  for (int a = 0; a < A.axis; ++a) stride *= N;
  const double tp = 2.0 * M_PI / A.Llen;
  double dot = 0.0;
  for (long long g = blockIdx.x; g < groups; g += gridDim.x) {
    const long long t = g * NT + tid;
    const bool ok = t < nlines;
    const int cnt = (int)min((long long)NT, nlines - g * NT);      // lines of this group
    const long long g0 = g * NT * N;                               // AXIS0: the group's first value
    long long base = 0, row = 0;
    if (AXIS0) {
      __syncthreads();   // the previous group's tiles are done with
      for (int e = tid; e < cnt * N; e += NT) {
        cp_async<16>(st + (e / N) * (N + 1) + e % N, A.lam + g0 + e, true);
        if (A.F) cp_async<16>(sv + (e / N) * (N + 1) + e % N, A.F + g0 + e, true);
      }
      cp_async_wait_all();
      __syncthreads();
      if (ok) row = t / (L.nx / N);
    } else if (ok) {
      const long long per = L.nx / N, q = t % per;
      row = t / per;
      base = row * L.nx + q / stride * stride * N + q % stride;
    }
    double2* v = AXIS0 ? sv + tid * (N + 1) : sv + tid;
    constexpr int VS = AXIS0 ? 1 : NT;                             // distance of the values of v
    double2 x[N];
    if (ok) {
      if (A.F) {
#pragma unroll
        for (int j = 0; j < N; ++j) x[j] = AXIS0 ? v[j] : A.F[base + j * stride];
        fft<N, true>(x);
#pragma unroll
        for (int j = 0; j < N; ++j) v[j * VS] = x[j];
        if (!AXIS0 && A.Y2) {
#pragma unroll
          for (int j = 0; j < N; ++j) A.Y2[base + j * stride] = x[j];
        }
      }
      if (!AXIS0 && A.Y1) {
#pragma unroll
        for (int j = 0; j < N; ++j) x[j] = A.lam[base + j * stride];
        fft<N, true>(x);
#pragma unroll
        for (int j = 0; j < N; ++j) A.Y1[base + j * stride] = x[j];
      }
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const double2 u = AXIS0 ? st[tid * (N + 1) + j] : A.lam[base + j * stride];
        const double dk = tp * kappa_first(j, N);
        x[j] = make_double2(-dk * u.y, dk * u.x);   // i dk lam
      }
      fft<N, true>(x);
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const double xc = (-A.Llen / 2 + A.Llen * j / N) / N;
        x[j] = xc * x[j];
        if (A.F) s += x[j].x * v[j * VS].x + x[j].y * v[j * VS].y;
      }
      if (A.F) dot -= A.scale * row_weight(L, row, A.half) * s;
      if (A.out) {
        fft<N, false>(x);
        if (AXIS0) {
#pragma unroll
          for (int j = 0; j < N; ++j) st[tid * (N + 1) + j] = x[j];
        } else {
#pragma unroll
          for (int j = 0; j < N; ++j) {
            double2 o = A.out[base + j * stride];
            o.x += A.coef * x[j].x;
            o.y += A.coef * x[j].y;
            A.out[base + j * stride] = o;
          }
        }
      }
    }
    if (AXIS0 && A.out) {
      __syncthreads();
      for (int e = tid; e < cnt * N; e += NT) {
        const double2 w = st[(e / N) * (N + 1) + e % N];
        double2 o = A.out[g0 + e];
        o.x += A.coef * w.x;
        o.y += A.coef * w.y;
        A.out[g0 + e] = o;
      }
    }
  }
  if (A.F) block_add(dot, A.acc, A.slot);
}

// The gradient of gyro_i: Re<lam, -D_i M_j M_k F> from a = ifft_j ifft_k lam and
// b = ifft_j ifft_k F, per point d_i x_j x_k Im(conj(a) b) / N^2.  Y1, Y2 hold
// the inverse transforms along one of the two axes (oaxis), the lines run
// along the other (axis); daxis = i.
template <int N, bool AXIS0>
__global__ void __launch_bounds__(line_threads<N>(AXIS0)) k_gyro_dot(RowLayout L, const double2* __restrict__ Y1,
                                                                     const double2* __restrict__ Y2, int axis, int oaxis,
                                                                     int daxis, double scale, double Llen, int half,
                                                                     double* __restrict__ acc, int slot) {
  constexpr int NT = line_threads<N>(AXIS0);
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sa = reinterpret_cast<double2*>(smraw);
  double2* sb = sa + NT * (N + 1);                    // AXIS0 only
  const int tid = threadIdx.x;
  const long long per = L.nx / N, nlines = L.nrows * per, groups = (nlines + NT - 1) / NT;
  long long stride = 1, os = 1, ds = 1;
  for (int a = 0; a < axis; ++a) stride *= N;
  for (int a = 0; a < oaxis; ++a) os *= N;
  for (int a = 0; a < daxis; ++a) ds *= N;
  double dot = 0.0;
  for (long long g = blockIdx.x; g < groups; g += gridDim.x) {
    const long long t = g * NT + tid;
    const int cnt = (int)min((long long)NT, nlines - g * NT);
    const long long g0 = g * NT * N;
    if (AXIS0) {
      __syncthreads();
      for (int e = tid; e < cnt * N; e += NT) {
        cp_async<16>(sa + (e / N) * (N + 1) + e % N, Y1 + g0 + e, true);
        cp_async<16>(sb + (e / N) * (N + 1) + e % N, Y2 + g0 + e, true);
      }
      cp_async_wait_all();
      __syncthreads();
    }
    if (t >= nlines) continue;
    const long long row = t / per, q = t % per;
    const long long w = q / stride * stride * N + q % stride, base = row * L.nx + w;   // the line's first point
    double2* a = AXIS0 ? sa + tid * (N + 1) : sa + tid;
    constexpr int VS = AXIS0 ? 1 : NT;
    double2 x[N];
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = AXIS0 ? a[j] : Y1[base + j * stride];
    fft<N, true>(x);
#pragma unroll
    for (int j = 0; j < N; ++j) a[j * VS] = x[j];
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = AXIS0 ? sb[tid * (N + 1) + j] : Y2[base + j * stride];
    fft<N, true>(x);
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const double xc = -Llen / 2 + Llen * j / N;
      const double2 u = a[j * VS];
      s += xc * (u.x * x[j].y - u.y * x[j].x);
    }
    const double dk = 2.0 * M_PI / Llen * kappa_first((int)(w / ds % N), N);
    const double xo = -Llen / 2 + Llen * (double)(w / os % N) / N;
    dot += scale * row_weight(L, row, half) * dk * xo / ((double)N * N) * s;
  }
  block_add(dot, acc, slot);
}

template <int N>
int adj_line_launch(hp_plan* p, const LineArgs& A, cudaStream_t s) {
  ProfScope _ps(p, "adj.axis", s);
  auto go = [&](auto kern, bool a0) -> int {
    HP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)line_smem<N>(a0)));
    kern<<<kDotBlocks, line_threads<N>(a0), line_smem<N>(a0), s>>>(p->layout(), A);
    HP_CUDA_TRY(cudaGetLastError());
    return HP_OK;
  };
  return A.axis == 0 ? go(k_adj_line<N, true>, true) : go(k_adj_line<N, false>, false);
}

template <int N>
int gyro_dot_launch(hp_plan* p, const double2* Y1, const double2* Y2, int axis, int oaxis, int daxis, double scale,
                    double* acc, int slot, cudaStream_t s) {
  ProfScope _ps(p, "adj.axis", s);
  const int half = p->symmetry == HP_REAL;
  auto go = [&](auto kern, bool a0) -> int {
    HP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)line_smem<N>(a0)));
    kern<<<kDotBlocks, line_threads<N>(a0), line_smem<N>(a0), s>>>(p->layout(), Y1, Y2, axis, oaxis, daxis, scale,
                                                                   p->model.L, half, acc, slot);
    HP_CUDA_TRY(cudaGetLastError());
    return HP_OK;
  };
  return axis == 0 ? go(k_gyro_dot<N, true>, true) : go(k_gyro_dot<N, false>, false);
}

// every omega grid size
int adj_line(hp_plan* p, const LineArgs& A, cudaStream_t s) {
  switch (p->N) {
#define X(n) case n: return adj_line_launch<n>(p, A, s);
    HP_FOR_EACH_N(X)
#undef X
    default:
      hp_set_error("omega grid size 2Bx not supported (even, 4..64)");
      return HP_ERR_UNSUPPORTED;
  }
}

int gyro_dot(hp_plan* p, const double2* Y1, const double2* Y2, int axis, int oaxis, int daxis, double scale, double* acc,
             int slot, cudaStream_t s) {
  switch (p->N) {
#define X(n) case n: return gyro_dot_launch<n>(p, Y1, Y2, axis, oaxis, daxis, scale, acc, slot, s);
    HP_FOR_EACH_N(X)
#undef X
    default:
      hp_set_error("omega grid size 2Bx not supported (even, 4..64)");
      return HP_ERR_UNSUPPORTED;
  }
}

// Gradient slots: b[0..2], gyro[3..5], gscale[6..8], G pairs [9..14]
// ((0,0),(0,1),(0,2),(1,1),(1,2),(2,2)).
constexpr int kSlots = 15;

// out = (add ? lam : 0) + a * A^H lam   (internal layout, FP64 buffers), and
// with F also acc += dt * Re<lam, dA/dtheta F> for every parameter theta.  The
// terms of the derivative are linear in their parameters, so dA/dtheta F is
// the term itself with unit coefficient:
//   damping   dA/db_i F    =  D_i M_i F,  gyroscope dA/dgyro_i F = -D_i M_j M_k F,
//   gravity   dA/dgs_i F   = -D_i Grav_i F,  noise dA/dG_ij F = c_ij F.
// The bracket of A^H is one derivative evaluation that adds itself to lam (its
// gravity taps are those of W Grav W^-1); each axis then takes one pass
// (k_adj_line) for its damping adjoint and damping gradient.  Dots of fields
// kept on the grid along one axis (Y1, Y2) give the gyroscopic gradients.
int adjoint_apply(hp_plan* p, const double2* lam, const double2* F, double2* out, double a, int add, double dt,
                  double* acc, cudaStream_t s) {
  const DerivParams base = hp_model_params(p);
  DerivParams q = base;
  for (int i = 0; i < 3; ++i) q.b[i] = 0.0;
  for (int i = 0; i < 9; ++i) q.G[i] = -base.G[i];
  int st = HP_OK;
  bool have = false;
  for (auto& kv : p->ws) if (kv.first == "adj.taps" && kv.second.p) have = true;
  const size_t per = p->precision == HP_FP64 ? sizeof(double) * tap_stride<double>() : sizeof(float) * tap_stride<float>();
  void* taps = p->ws_get("adj.taps", per * p->nrows, &st);
  if (st) return st;
  if (!have) ADJ_CHECK(hp_adjoint_gravity_taps(p, taps, s));
  q.taps = taps;
  const size_t ib = 16 * (size_t)p->nrows * p->nx;
  double2 *y1 = nullptr, *y2 = nullptr;
  if (F && p->ndim == 3) {
    y1 = (double2*)p->ws_get("adj.t", ib, &st);
    if (st) return st;
    y2 = (double2*)p->ws_get("adj.y", ib, &st);
    if (st) return st;
  }
  ADJ_CHECK(hp_derivative_eval_prm(p, q, lam, add ? lam : nullptr, -a, out, nullptr, 0.0, s));
  if (F) ADJ_CHECK(hp_gravity_noise_dots64(p, F, lam, acc, kDotBlocks, 6, dt, s));
  for (int i = p->ndim - 1; i >= 0; --i) {
    LineArgs A{};
    A.lam = lam;
    A.F = F;
    A.out = base.b[i] != 0.0 ? out : nullptr;
    A.Y1 = i > 0 ? y1 : nullptr;
    A.Y2 = i > 0 ? y2 : nullptr;
    A.axis = i;
    A.coef = -a * base.b[i];
    A.scale = dt;
    A.Llen = base.L;
    A.half = p->symmetry == HP_REAL;
    A.slot = i;
    A.acc = acc;
    if (F || A.out) ADJ_CHECK(adj_line(p, A, s));
    if (!y1) continue;
    if (i == 2) {   // on the grid along axis 2: gyro_0 along axis 1, gyro_1 along axis 0
      ADJ_CHECK(gyro_dot(p, y1, y2, 1, 2, 0, dt, acc, 3, s));
      ADJ_CHECK(gyro_dot(p, y1, y2, 0, 2, 1, dt, acc, 4, s));
    } else if (i == 1) {
      ADJ_CHECK(gyro_dot(p, y1, y2, 0, 1, 2, dt, acc, 5, s));
    }
  }
  return HP_OK;
}

int check_mem(int mem) {
  if (mem != HP_DEVICE && mem != HP_HOST) { hp_set_error("mem must be HP_DEVICE or HP_HOST"); return HP_ERR_INVALID; }
  return HP_OK;
}

// full-layout (mem) -> internal FP64, symmetrised for HP_REAL plans
int load_full(hp_plan* p, const double* src, int mem, double2* dst, cudaStream_t s) {
  const double2* in = (const double2*)src;
  if (mem == HP_HOST) {
    int st = HP_OK;
    const size_t fb = 16 * (size_t)p->n_full();
    double2* a = (double2*)p->ws_get("adj.full_a", fb, &st);
    if (st) return st;
    HP_CUDA_TRY(cudaMemcpyAsync(a, src, fb, cudaMemcpyHostToDevice, s));
    in = a;
  }
  return p->symmetry == HP_REAL ? hp_full_to_internal_sym(p, in, dst, s) : hp_full_to_internal(p, in, dst, s);
}

int store_full(hp_plan* p, const double2* src, double* dst, int mem, cudaStream_t s) {
  int st = HP_OK;
  const size_t fb = 16 * (size_t)p->n_full();
  double2* out = (double2*)dst;
  if (mem == HP_HOST) {
    out = (double2*)p->ws_get("adj.full_a", fb, &st);
    if (st) return st;
  }
  ADJ_CHECK(hp_internal_to_full(p, src, out, s));
  if (mem == HP_HOST) HP_CUDA_TRY(cudaMemcpyAsync(dst, out, fb, cudaMemcpyDeviceToHost, s));
  return HP_OK;
}

}  // namespace

extern "C" int hp_pendulum_derivative_adjoint(hp_plan* p, const double* lam, double* out, int mem) {
  if (!p || !lam || !out) { hp_set_error("null argument"); return HP_ERR_INVALID; }
  ADJ_CHECK(check_mem(mem));
  if (!p->has_model) { hp_set_error("no model: call hp_plan_set_model first"); return HP_ERR_NO_MODEL; }
  if (p->den_mR) { hp_set_error("the adjoint covers coefficient-gravity models (hp_plan_set_model)"); return HP_ERR_UNSUPPORTED; }
  if (p->so3d64) { hp_set_error("the adjoint covers the pendulum models (no attitude diffusion)"); return HP_ERR_UNSUPPORTED; }
  if (tw_init() != 0) { hp_set_error("twiddle table upload failed"); return HP_ERR_CUDA; }
  cudaStream_t s = p->stream;
  int st = HP_OK;
  const size_t ib = 16 * (size_t)p->nrows * p->nx;
  double2* li = (double2*)p->ws_get("adj.lam", ib, &st);
  if (st) return st;
  double2* lo = (double2*)p->ws_get("adj.lam2", ib, &st);
  if (st) return st;
  // no symmetrisation here: the operator is applied to the given rows
  {
    const size_t fb = 16 * (size_t)p->n_full();
    const double2* in = (const double2*)lam;
    if (mem == HP_HOST) {
      double2* a = (double2*)p->ws_get("adj.full_a", fb, &st);
      if (st) return st;
      HP_CUDA_TRY(cudaMemcpyAsync(a, lam, fb, cudaMemcpyHostToDevice, s));
      in = a;
    }
    ADJ_CHECK(hp_full_to_internal(p, in, li, s));
  }
  ADJ_CHECK(adjoint_apply(p, li, nullptr, lo, 1.0, 0, 0.0, nullptr, s));
  ADJ_CHECK(store_full(p, lo, out, mem, s));
  HP_CUDA_TRY(cudaStreamSynchronize(s));
  return HP_OK;
}

extern "C" int hp_pendulum_adjoint(hp_plan* p, const double* F0, const double* lamT, int nsteps, double dt,
                                   int method, int checkpoint_every, double* lam0, hp_model_grad* grad, int mem) {
  if (!p || !F0 || !lamT || nsteps < 0 || checkpoint_every < 1) { hp_set_error("bad argument"); return HP_ERR_INVALID; }
  ADJ_CHECK(check_mem(mem));
  if (!p->has_model) { hp_set_error("no model: call hp_plan_set_model first"); return HP_ERR_NO_MODEL; }
  if (p->den_mR) { hp_set_error("the adjoint covers coefficient-gravity models (hp_plan_set_model)"); return HP_ERR_UNSUPPORTED; }
  if (p->so3d64) { hp_set_error("the adjoint covers the pendulum models (no attitude diffusion)"); return HP_ERR_UNSUPPORTED; }
  if (method != HP_EULER) { hp_set_error("the adjoint covers forward-Euler trajectories"); return HP_ERR_UNSUPPORTED; }
  if (!std::isfinite(dt)) { hp_set_error("dt must be finite"); return HP_ERR_INVALID; }
  if (tw_init() != 0) { hp_set_error("twiddle table upload failed"); return HP_ERR_CUDA; }
  cudaStream_t s = p->stream;
  int st = HP_OK;
  const size_t ib = 16 * (size_t)p->nrows * p->nx;
  const int ck = std::min(checkpoint_every, std::max(nsteps, 1));
  const int nseg = nsteps > 0 ? (nsteps + ck - 1) / ck : 0;
  // checkpoints [nseg] + one segment of states [ck] + the adjoint pair
  char* ckpt = (char*)p->ws_get("adj.ckpt", ib * (size_t)std::max(nseg, 1), &st);
  if (st) return st;
  char* seg = (char*)p->ws_get("adj.seg", ib * (size_t)ck, &st);
  if (st) return st;
  double2* la = (double2*)p->ws_get("adj.lam", ib, &st);
  if (st) return st;
  double2* lb = (double2*)p->ws_get("adj.lam2", ib, &st);
  if (st) return st;
  double* acc = (double*)p->ws_get("adj.acc", sizeof(double) * kSlots * kDotBlocks, &st);
  if (st) return st;
  HP_CUDA_TRY(cudaMemsetAsync(acc, 0, sizeof(double) * kSlots * kDotBlocks, s));
  auto state = [&](char* b, int i) { return reinterpret_cast<double2*>(b + ib * (size_t)i); };

  // forward sweep, keeping the state at the start of every segment
  {
    const size_t fb = 16 * (size_t)p->n_full();
    const double2* in = (const double2*)F0;
    if (mem == HP_HOST) {
      double2* a = (double2*)p->ws_get("adj.full_a", fb, &st);
      if (st) return st;
      HP_CUDA_TRY(cudaMemcpyAsync(a, F0, fb, cudaMemcpyHostToDevice, s));
      in = a;
    }
    ADJ_CHECK(hp_full_to_internal(p, in, state(ckpt, 0), s));
  }
  for (int g = 0; g + 1 < nseg; ++g) {
    double2* x = state(seg, 0);
    HP_CUDA_TRY(cudaMemcpyAsync(x, state(ckpt, g), ib, cudaMemcpyDeviceToDevice, s));
    for (int j = 0; j < ck; ++j) {
      double2* dst = (j + 1 < ck) ? state(seg, (j + 1) % ck) : state(ckpt, g + 1);
      ADJ_CHECK(hp_derivative_eval(p, state(seg, j), state(seg, j), dt, dst, nullptr, 0.0, s));
    }
  }
  // reverse sweep
  ADJ_CHECK(load_full(p, lamT, mem, la, s));
  for (int g = nseg - 1; g >= 0; --g) {
    const int len = std::min(ck, nsteps - g * ck);
    HP_CUDA_TRY(cudaMemcpyAsync(state(seg, 0), state(ckpt, g), ib, cudaMemcpyDeviceToDevice, s));
    for (int j = 1; j < len; ++j)
      ADJ_CHECK(hp_derivative_eval(p, state(seg, j - 1), state(seg, j - 1), dt, state(seg, j), nullptr, 0.0, s));
    for (int j = len - 1; j >= 0; --j) {
      ADJ_CHECK(adjoint_apply(p, la, state(seg, j), lb, dt, 1, dt, acc, s));
      std::swap(la, lb);
    }
  }
  if (lam0) ADJ_CHECK(store_full(p, la, lam0, mem, s));
  std::vector<double> h((size_t)kSlots * kDotBlocks);
  HP_CUDA_TRY(cudaMemcpyAsync(h.data(), acc, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s));
  HP_CUDA_TRY(cudaStreamSynchronize(s));
  double tot[kSlots];
  for (int k = 0; k < kSlots; ++k) {
    double v = 0.0;
    for (int b = 0; b < kDotBlocks; ++b) v += h[(size_t)k * kDotBlocks + b];
    tot[k] = v;
  }
  if (grad) {
    for (int i = 0; i < 3; ++i) {
      grad->b[i] = tot[i];
      grad->gyro[i] = tot[3 + i];
      grad->gscale[i] = tot[6 + i];
    }
    const int pi[6] = {0, 0, 0, 1, 1, 2}, pj[6] = {0, 1, 2, 1, 2, 2};
    for (int q = 0; q < 6; ++q) {
      grad->G[pi[q] * 3 + pj[q]] = tot[9 + q];
      grad->G[pj[q] * 3 + pi[q]] = tot[9 + q];
    }
  }
  return HP_OK;
}
