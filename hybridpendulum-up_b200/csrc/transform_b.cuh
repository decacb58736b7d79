// Per-bandlimit kernels of the SO(3) transforms and their launchers: the
// synthesis (beta contraction, gamma and alpha FFTs; ifftSO3R.m:16-37) and the
// two-stage analysis (alpha/gamma FFTs, beta contraction; fftSO3R.m:89-106).
// Included by transform.cu (configurations and declarations only) and by
// transform_b0.cu .. transform_b3.cu, each of which instantiates the launchers
// for the bandlimits B with B mod 4 equal to its part number, so that the
// kernels compile in parallel.  Each translation unit holds its own twiddle
// table, which the launchers fill before their first launch (tw_init).
#pragma once
#include <algorithm>
#include "common.cuh"
#include "plan.hpp"

using namespace hp;

static inline int smem_limit() {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return v;
}

// ------------------------------------------------------------ synthesis ----
// Bulk (TMA engine) copy of a contiguous shared-memory run to global memory:
// both addresses 16-byte aligned, size a multiple of 16 bytes.  The issuing
// thread later waits for the source to have been read (wait_group.read) before
// the buffer is rewritten, and for completion (wait_group) before exit.
__device__ __forceinline__ void bulk_s2g(void* gdst, const void* ssrc, unsigned bytes, uint64_t pol) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(ssrc);
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;" ::"l"(gdst), "r"(s),
               "r"(bytes), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// orders this thread's shared-memory writes before later bulk-copy reads of them
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Two staging runs of N floats (the real and the imaginary parts of x), both
// starting LEAD floats (0 or 2) before a 16-byte boundary: an 8-byte store
// for the lead, 16-byte stores, an 8-byte store for an even remainder.
template <int N, int LEAD>
__device__ __forceinline__ void stage_run(float* st, float* st2, const float2 (&x)[N]) {
  static_assert(N % 2 == 0 && (LEAD == 0 || LEAD == 2), "even runs, 8-byte aligned");
  if constexpr (LEAD == 2) {
    *reinterpret_cast<float2*>(st) = make_float2(x[0].x, x[1].x);
    *reinterpret_cast<float2*>(st2) = make_float2(x[0].y, x[1].y);
  }
  constexpr int n4 = (N - LEAD) / 4;
#pragma unroll
  for (int i = 0; i < n4; ++i) {
    const int a = LEAD + 4 * i;
    *reinterpret_cast<float4*>(st + a) = make_float4(x[a].x, x[a + 1].x, x[a + 2].x, x[a + 3].x);
    *reinterpret_cast<float4*>(st2 + a) = make_float4(x[a].y, x[a + 1].y, x[a + 2].y, x[a + 3].y);
  }
  constexpr int a = LEAD + 4 * n4;
  if constexpr (a < N) {
    *reinterpret_cast<float2*>(st + a) = make_float2(x[a].x, x[a + 1].x);
    *reinterpret_cast<float2*>(st2 + a) = make_float2(x[a].y, x[a + 1].y);
  }
}

// (m, n) pairs with their row start, l-run length, m slot and n bin, longest
// runs first (the order keeps the lanes of a warp on loops of similar length),
// pairs of equal length by m, then n.  k = max(|m|, |n|) sets the length, so an
// entry gives its pair in closed form: 4k + 1 pairs with m >= 0 have that k (two
// for each m < k, 2k + 1 for m = k), 8k of all pairs (2k + 1 for m = -k, two for
// each m between, 2k + 1 for m = k).  The device writes the table: a plan's first
// transform waits for no copy from the host.
template <int B, bool CPLX>
__global__ void k_pairs(RowLayout L, int2* __restrict__ out) {
  constexpr int lmax = B - 1, D = 2 * lmax + 1, NPAIR = (CPLX ? D : B) * D;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= NPAIR) return;
  auto first = [](int k) { return CPLX ? (k ? (2 * k - 1) * (2 * k - 1) : 0) : k * (2 * k - 1); };
  int k = 0;
  while (first(k + 1) <= q) ++k;
  int r = q - first(k), m = k, n;
  const int head = CPLX && k ? 2 * k + 1 : 0;          // the pairs with m = -k
  const int mid = CPLX ? 2 * (2 * k - 1) : 2 * k;      // those between
  if (k == 0) {
    n = 0;
  } else if (r < head) {
    m = -k;
    n = r - k;
  } else if ((r -= head) < mid) {
    m = (CPLX ? 1 - k : 0) + r / 2;
    n = r & 1 ? k : -k;
  } else {
    n = r - mid - k;
  }
  const int mi = CPLX ? m + lmax : m, bin = n >= 0 ? n : n + 2 * B;
  out[q] = make_int2(L.seg[(m - L.m_lo) * D + n + lmax], (B - k) | (mi << 8) | (bin << 16) | ((n == 0 ? 1 : 0) << 24));
}

// the plan's pair table
template <int B, bool CPLX> static const int2* pair_table(hp_plan* p, int* st, cudaStream_t s) {
  constexpr int NPAIR = (CPLX ? 2 * B - 1 : B) * (2 * B - 1);
  const char* key = CPLX ? "tf.pairs_c" : "tf.pairs_r";
  bool have = false;
  for (auto& kv : p->ws) if (kv.first == key) have = true;
  int2* t = (int2*)p->ws_get(key, sizeof(int2) * NPAIR, st);
  if (*st) return nullptr;
  if (!have) {
    k_pairs<B, CPLX><<<(NPAIR + 127) / 128, 128, 0, s>>>(p->layout(), t);
    if (cudaGetLastError() != cudaSuccess) { hp_set_error("pair table launch failed"); *st = HP_ERR_CUDA; }
  }
  return t;
}

// (2l+1) d^l_mn at the first B nodes as [group][row][NN], group g holding the
// nodes g NN .. g NN + NN-1 (zero past the last beta); groups are gs values apart,
// a multiple of 16 bytes
template <typename T>
__global__ void k_sd_table(RowLayout L, const T* __restrict__ wig, T* __restrict__ out, int NN, int gs, int ngroups) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ngroups * gs) return;
  const int g = t / gs, e = t - g * gs, r = e / NN, b = g * NN + e % NN;
  out[t] = r < L.nrows && b < 2 * L.B ? (T)(2 * L.rows[r].x + 1) * wig[(size_t)b * L.nrows + r] : (T)0;
}

#include "synth.cuh"
#include "synth2.cuh"

template <int B, typename T, bool CPLX>
int synth_launch(hp_plan* p, const c2<T>* Fp, void* f, cudaStream_t s) {
  if (tw_init() != 0) { hp_set_error("twiddle table upload failed"); return HP_ERR_CUDA; }
  if constexpr (!CPLX && RealSynthCfg<B, T>::ok) return synth_real_launch<B, T>(p, Fp, reinterpret_cast<T*>(f), s);
  else return synth2_launch<B, T, CPLX>(p, Fp, f, p->nx, "tf.G", s);
}

// ----------------------------------------- analysis without atomics ----
// Stage 1 (k_anal_ag): block = (beta, chunk of PA omega points).  For each
// omega point the alpha FFT over a and the gamma FFT over c of f(., b, ., w)
// (times an optional grid multiplier) give Q_b[m][n]; it is written to
// Qg[(m, n bin)][b][w] with the chunk's omega points consecutive.  Bound by the
// shared-memory pipe: unpadded tiles put the lanes of a warp on one to four
// banks in the reads of both FFTs and of the store, with one or two blocks of
// 256 threads per SM.  16 x 16 omega points, before / now (us): B = 16 FP32 125 /
// 38, FP64 240 / 67; B = 32 FP32 792 / 304, FP64 1778 / 891; 16^3, B = 10 FP64 318
// / 109.
// nx: the number of omega points (the plan's, or a batch of functions on SO(3)).
// Stage 2 (k_anal_beta): thread = ((m, n) pair, omega point), all l of the
// pair: F^l_mn[w] = sum_b w_b d^l_mn(beta_b) Q_b[m][n][w], written straight
// into the [row][omega] layout.  Every output has one owner: no atomics.
// Shapes of stage 1.  Rows in shared memory are padded so that lanes on
// consecutive rows hit distinct banks: input lines (2B values of one (omega,
// gamma) column) start an odd number of 16-byte units apart and are read 16
// bytes at a time; rows of the output tile [omega][m][2B] are 2B + 1 values, an
// omega point's rows an odd number of values apart.
template <int B, typename T, bool CPLX> struct AnalCfg {
  using C = c2<T>;
  static constexpr int NB2 = 2 * B, NM = CPLX ? 2 * B - 1 : B;
  static constexpr int items = CPLX ? 2 * B : B;    // alpha items per omega point
  static constexpr int NT = 128;
  static constexpr int VAL = (int)sizeof(T) * (CPLX ? 2 : 1);       // bytes of a density value
  static constexpr int LS = ((NB2 * VAL + 15) / 16) | 1;            // 16-byte units per input line
  static constexpr int GQ = NB2 + 1, TSQ = (NM * GQ) | 1;           // output row, output omega point (values)
  static constexpr long long bytes(int pa) {
    const long long in = (long long)pa * NB2 * LS * 16, q = (long long)pa * TSQ * (long long)sizeof(C);
    const long long tile = ((in > q ? in : q) + 15) / 16 * 16;
    return tile + (CPLX ? 0 : (long long)NB2 * LS * 16);            // + this beta's grid multiplier (real densities)
  }
  // the largest omega batch with one alpha item per thread and three blocks per
  // SM; at least 4 (32-byte stores in FP32) where two blocks allow it
  static constexpr int pick() {
    int pa = 16;
    while (pa > 1 && (pa * items > NT || bytes(pa) > (pa > 4 ? 72 : 110) * 1024)) pa /= 2;
    return pa;
  }
  static constexpr int PA = pick();
  // blocks per SM that the registers are held to
  static constexpr int MINB = sizeof(T) == 4 ? (NB2 <= 24 ? 6 : NB2 <= 32 ? 4 : NB2 <= 48 ? 3 : 2)
                                             : (NB2 <= 12 ? 6 : NB2 <= 20 ? 4 : NB2 <= 32 ? 3 : 2);
};

// 16-byte reads of N consecutive values (16-byte aligned)
template <int N> __device__ __forceinline__ void load_line(const float* s, float (&v)[N]) {
#pragma unroll
  for (int i = 0; i + 4 <= N; i += 4) {
    const float4 q = *reinterpret_cast<const float4*>(s + i);
    v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
  }
  if constexpr (N % 4) {
    const float2 q = *reinterpret_cast<const float2*>(s + N - 2);
    v[N - 2] = q.x; v[N - 1] = q.y;
  }
}
template <int N> __device__ __forceinline__ void load_line(const double* s, double (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const double2 q = *reinterpret_cast<const double2*>(s + i);
    v[i] = q.x; v[i + 1] = q.y;
  }
}

template <int B, typename T, int PA, bool CPLX>
__global__ void __launch_bounds__(AnalCfg<B, T, CPLX>::NT, (AnalCfg<B, T, CPLX>::MINB))
    k_anal_ag(const void* __restrict__ fin, const double* __restrict__ mult, c2<T>* __restrict__ Qg, long long w0,
              long long nwc) {
  using C = c2<T>;
  using Cfg = AnalCfg<B, T, CPLX>;
  constexpr int NB2 = 2 * B, NM = Cfg::NM, MLO = CPLX ? -(B - 1) : 0;
  constexpr int NT = Cfg::NT, VAL = Cfg::VAL, LB = Cfg::LS * 16, GQ = Cfg::GQ, TSQ = Cfg::TSQ;
  extern __shared__ __align__(16) unsigned char smraw[];
  // input lines [PA][c] of LB bytes; the alpha stage reads its lines into
  // registers before a barrier, so its output [PA][m][c or q] reuses the space
  C* sQ = reinterpret_cast<C*>(smraw);
  unsigned char* smult = smraw + Cfg::bytes(PA) - (CPLX ? 0 : (size_t)NB2 * LB);   // [c] lines of the multiplier
  const int b = blockIdx.y;
  const long long wl0 = (long long)blockIdx.x * PA;                       // chunk-local omega
  const int pc = (int)min((long long)PA, nwc - wl0);
  const int tid = threadIdx.x;
  // load f(., b, c, w): 2B consecutive a per (c, w), by asynchronous copies, all
  // in flight at once (pieces of 16 bytes, 8 where 2B values are not a multiple
  // of 16 bytes); a density buffer off a 16-byte boundary is copied by values
  constexpr int PB = (NB2 * VAL) % 16 == 0 ? 16 : 8, PPR = NB2 * VAL / PB;
  const unsigned char* src = reinterpret_cast<const unsigned char*>(fin) + ((w0 + wl0) * NB2 * NB2 + b) * (size_t)(NB2 * VAL);
  if ((reinterpret_cast<unsigned long long>(fin) & 15ull) == 0) {
    for (int e = tid; e < pc * NB2 * PPR; e += NT) {
      const int run = e / PPR, piece = e - run * PPR;
      cp_async<PB>(smraw + (size_t)run * LB + piece * PB, src + (size_t)run * (NB2 * NB2 * VAL) + piece * PB, true);
    }
  } else {
    for (int e = tid; e < pc * NB2 * (NB2 * VAL / (int)sizeof(T)); e += NT) {
      constexpr int TPR = NB2 * VAL / (int)sizeof(T);
      const int run = e / TPR, i = e - run * TPR;
      reinterpret_cast<T*>(smraw + (size_t)run * LB)[i] = reinterpret_cast<const T*>(src + (size_t)run * (NB2 * NB2 * VAL))[i];
    }
  }
  if (!CPLX && mult)   // the grid multiplier of this beta (density-gravity terms)
    for (int e = tid; e < NB2 * NB2; e += NT) {
      const int c = e / NB2, a = e % NB2;
      reinterpret_cast<T*>(smult + (size_t)c * LB)[a] = (T)mult[a + NB2 * (b + NB2 * c)];
    }
  cp_async_wait_all();
  __syncthreads();
  // alpha, one item per thread.  Real densities: item (p, c), columns c and c + B
  // share one complex FFT, z = f_c + i f_{c+B}: X_c[m] = (Z[m] + conj Z[-m]) / 2,
  // X_{c+B}[m] = (Z[m] - conj Z[-m]) / 2i.  Complex densities: item (p, c).
  {
    const bool act = tid < pc * Cfg::items;
    const int pp = tid / Cfg::items, c = tid % Cfg::items;
    C x[NB2];
    if (act) {
      const unsigned char* line = smraw + (size_t)(pp * NB2 + c) * LB;
      if constexpr (CPLX) {
        const C* r = reinterpret_cast<const C*>(line);
#pragma unroll
        for (int a = 0; a < NB2; ++a) x[a] = r[a];
      } else {
        T u[NB2], v[NB2];
        load_line<NB2>(reinterpret_cast<const T*>(line), u);
        load_line<NB2>(reinterpret_cast<const T*>(line + (size_t)B * LB), v);
#pragma unroll
        for (int a = 0; a < NB2; ++a) x[a] = mk(u[a], v[a]);
        if (mult) {
          load_line<NB2>(reinterpret_cast<const T*>(smult + (size_t)c * LB), u);
          load_line<NB2>(reinterpret_cast<const T*>(smult + (size_t)(c + B) * LB), v);
#pragma unroll
          for (int a = 0; a < NB2; ++a) { x[a].x *= u[a]; x[a].y *= v[a]; }
        }
      }
    }
    __syncthreads();
    if (act) {
      fft<NB2, true>(x);
      C* dst = sQ + (size_t)pp * TSQ + c;
      if constexpr (CPLX) {
#pragma unroll
        for (int mi = 0; mi < NM; ++mi) {
          const int m = mi + MLO;
          dst[mi * GQ] = x[m >= 0 ? m : m + NB2];
        }
      } else {
#pragma unroll
        for (int m = 0; m < NM; ++m) {
          const C zp = x[m], zm = x[(NB2 - m) % NB2];
          dst[m * GQ] = mk((T)0.5 * (zp.x + zm.x), (T)0.5 * (zp.y - zm.y));
          dst[m * GQ + B] = mk((T)0.5 * (zp.y + zm.y), (T)0.5 * (zm.x - zp.x));
        }
      }
    }
  }
  __syncthreads();
  // gamma: item (p, m): FFT(+) over c, in place (bins n mod 2B)
  for (int it = tid; it < pc * NM; it += NT) {
    C* row = sQ + (size_t)(it / NM) * TSQ + (it % NM) * GQ;
    C x[NB2];
#pragma unroll
    for (int j = 0; j < NB2; ++j) x[j] = row[j];
    fft<NB2, true>(x);
#pragma unroll
    for (int j = 0; j < NB2; ++j) row[j] = x[j];
  }
  __syncthreads();
  // store: Qg[((m * 2B + q) * 2B + b) * nwc + w], consecutive omega points
  C* out = Qg + (long long)b * nwc + wl0;
  if (pc == PA) {
#pragma unroll 4
    for (int e = tid; e < NM * NB2 * PA; e += NT) {
      const int pp = e % PA, mq = e / PA;
      out[(long long)mq * NB2 * nwc + pp] = sQ[pp * TSQ + mq + mq / NB2];
    }
  } else {
    for (int e = tid; e < NM * NB2 * pc; e += NT) {
      const int pp = e % pc, mq = e / pc;
      out[(long long)mq * NB2 * nwc + pp] = sQ[pp * TSQ + mq + mq / NB2];
    }
  }
}

// The warp's table rows go to shared memory in one go, and the next four betas'
// Q values load while the current four are summed: the table values, read from
// L2 as the betas advanced, and the four loads in flight had been the stalls
// (FP64, before / now: B = 10, 16^3 97 / 69 us; B = 24, 24 x 24 356 / 197 us).
template <int B, typename T, bool CPLX>
__global__ void __launch_bounds__(128) k_anal_beta(RowLayout L, const c2<T>* __restrict__ Qg,
                                                   const T* __restrict__ dw, const int2* __restrict__ pairs,
                                                   int npairs, c2<T>* __restrict__ out, long long w0, long long nwc) {
  using C = c2<T>;
  constexpr int NB2 = 2 * B;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pi = blockIdx.y * 4 + warp;
  if (pi >= npairs) return;
  const int2 pe = pairs[pi];
  const int s = pe.x, len = pe.y & 0xff, mi = (pe.y >> 8) & 0xff, q = (pe.y >> 16) & 0xff;
  T* d = reinterpret_cast<T*>(smraw) + warp * (B * NB2);
  {
    // rows are 2B values, a multiple of 16 bytes in FP64 and of 8 in FP32
    constexpr int PB = (NB2 * sizeof(T)) % 16 == 0 ? 16 : 8, EPP = PB / (int)sizeof(T);
    const T* src = dw + (size_t)s * NB2;
    for (int e = lane; e < len * NB2 / EPP; e += 32) cp_async<PB>(d + e * EPP, src + e * EPP, true);
  }
  const long long wl = (long long)blockIdx.x * 32 + lane;
  const bool ok = wl < nwc;
  const C* qsrc = Qg + ((long long)(mi * NB2 + q) * NB2) * nwc + wl;
  C v[4], nv[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) nv[u] = ok ? qsrc[(long long)u * nwc] : czero<C>();   // 2B >= 4
  C acc[B];
#pragma unroll
  for (int j = 0; j < B; ++j) acc[j] = czero<C>();
  cp_async_wait_all();
  __syncwarp();
  if (!ok) return;
#pragma unroll 1
  for (int b0 = 0; b0 < NB2; b0 += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      v[u] = nv[u];
      nv[u] = b0 + 4 + u < NB2 ? qsrc[(long long)(b0 + 4 + u) * nwc] : czero<C>();
    }
#pragma unroll
    for (int j = 0; j < B; ++j) {
      if (j < len) {
        const T* dj = d + j * NB2 + b0;
#pragma unroll
        for (int u = 0; u < 4; u += 2) {   // pairs of betas (2B is even), 8 or 16 bytes
          if (NB2 % 4 == 0 || b0 + u < NB2) {
            struct alignas(2 * sizeof(T)) Two { T x, y; };
            const Two w = *reinterpret_cast<const Two*>(dj + u);
            acc[j].x = fma(w.x, v[u].x, acc[j].x);
            acc[j].y = fma(w.x, v[u].y, acc[j].y);
            acc[j].x = fma(w.y, v[u + 1].x, acc[j].x);
            acc[j].y = fma(w.y, v[u + 1].y, acc[j].y);
          }
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < B; ++j)
    if (j < len) out[(long long)(s + j) * L.nx + w0 + wl] = acc[j];
}

// dw[row][b] = w_b d^l_mn(beta_b)
template <typename T>
__global__ void k_dw_table(RowLayout L, const T* __restrict__ wig, const double* __restrict__ qw,
                           T* __restrict__ dw) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int NB2 = 2 * L.B;
  if (t >= L.nrows * NB2) return;
  const long long r = t / NB2;
  const int b = (int)(t % NB2);
  dw[t] = (T)(qw[b] * (double)wig[(size_t)b * L.nrows + r]);
}

// qkey: the workspace buffer of Q
template <int B, typename T, bool CPLX>
int anal2_launch(hp_plan* p, const void* f, const double* mult, c2<T>* out, long long nx, const char* qkey,
                 cudaStream_t s) {
  if (tw_init() != 0) { hp_set_error("twiddle table upload failed"); return HP_ERR_CUDA; }
  using C = c2<T>;
  using Cfg = AnalCfg<B, T, CPLX>;
  constexpr int PA = Cfg::PA, NB2 = 2 * B, NM = Cfg::NM;
  const size_t smem = (size_t)Cfg::bytes(PA);
  if (smem > (size_t)smem_limit()) { hp_set_error("analysis tiles exceed shared memory"); return HP_ERR_UNSUPPORTED; }
  int st = HP_OK;
  // pair table (shared with the synthesis) and the w_b d table
  constexpr int NPAIR = NM * (2 * B - 1);
  const int2* dpairs = pair_table<B, CPLX>(p, &st, s);
  if (st) return st;
  const char* dkey = sizeof(T) == 8 ? "tf.dw64" : "tf.dw32";
  bool have = false;
  for (auto& kv : p->ws) if (kv.first == dkey) have = true;
  T* dw = (T*)p->ws_get(dkey, sizeof(T) * p->nrows * NB2, &st);
  if (st) return st;
  if (!have) {
    const long long n = p->nrows * NB2;
    k_dw_table<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        p->layout(), sizeof(T) == 8 ? (const T*)(const void*)p->wig64 : (const T*)(const void*)p->wig32, p->qw, dw);
    HP_CUDA_TRY(cudaGetLastError());
  }
  // omega chunks keep the staged tiles within 2 GB
  const long long per_w = (long long)NM * NB2 * NB2 * (long long)sizeof(C);
  long long nwc = std::max(32LL, (2LL << 30) / per_w / 32 * 32);
  nwc = std::min(nwc, (nx + 31) / 32 * 32);
  RowLayout L = p->layout();
  L.nx = nx;
  C* Qg = (C*)p->ws_get(qkey, (size_t)per_w * nwc, &st);
  if (st) return st;
  HP_CUDA_TRY(cudaFuncSetAttribute(k_anal_ag<B, T, PA, CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (long long w0 = 0; w0 < nx; w0 += nwc) {
    const long long nw = std::min(nwc, nx - w0);
    {
      ProfScope _ps(p, "tf.anal.ag", s);
      dim3 ga((unsigned)((nw + PA - 1) / PA), (unsigned)NB2);
      k_anal_ag<B, T, PA, CPLX><<<ga, Cfg::NT, smem, s>>>(f, mult, Qg, w0, nw);
      HP_CUDA_TRY(cudaGetLastError());
    }
    if constexpr (sizeof(T) == 4) {
      // AUTO: tensor cores from B = 15 (B=15, 32x32: 0.046 vs 0.052 ms; B=30: 0.24 vs
      // 0.50 ms), CUDA cores below (B=8: 0.015 vs 0.009 ms, set-up dominates)
      const bool tc = p->beta_engine == HP_BETA_TENSOR || p->beta_engine == HP_BETA_TENSOR_BF16 ||
                      (p->beta_engine == HP_BETA_AUTO && p->B >= 15);
      if (tc && tc_beta_supported(p)) {
        st = tc_beta_forward(p, reinterpret_cast<const float2*>(Qg), dpairs, NPAIR, reinterpret_cast<float2*>(out),
                             w0, nw, s);
        if (st) return st;
        continue;
      }
    }
    ProfScope _ps(p, "tf.anal.beta", s);
    dim3 gb((unsigned)((nw + 31) / 32), (unsigned)((NPAIR + 3) / 4));
    constexpr size_t bsm = 4 * sizeof(T) * (size_t)B * NB2;
    HP_CUDA_TRY(cudaFuncSetAttribute(k_anal_beta<B, T, CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsm));
    k_anal_beta<B, T, CPLX><<<gb, 128, bsm, s>>>(L, Qg, dw, dpairs, NPAIR, out, w0, nw);
    HP_CUDA_TRY(cudaGetLastError());
  }
  return HP_OK;
}


// explicit instantiations of the launchers for one bandlimit (used by the
// part files)
#ifdef HP_TRANSFORM_PART
#define HP_INST_B(b)                                                                                   \
  template int synth_launch<b, float, false>(hp_plan*, const float2*, void*, cudaStream_t);        \
  template int synth_launch<b, float, true>(hp_plan*, const float2*, void*, cudaStream_t);         \
  template int synth_launch<b, double, false>(hp_plan*, const double2*, void*, cudaStream_t);      \
  template int synth_launch<b, double, true>(hp_plan*, const double2*, void*, cudaStream_t);       \
  template int anal2_launch<b, float, false>(hp_plan*, const void*, const double*, float2*, long long, const char*, cudaStream_t);\
  template int anal2_launch<b, float, true>(hp_plan*, const void*, const double*, float2*, long long, const char*, cudaStream_t);\
  template int anal2_launch<b, double, false>(hp_plan*, const void*, const double*, double2*, long long, const char*, cudaStream_t);\
  template int anal2_launch<b, double, true>(hp_plan*, const void*, const double*, double2*, long long, const char*, cudaStream_t);\
  template int synth2_launch<b, double, false>(hp_plan*, const double2*, void*, long long, const char*, cudaStream_t);
#endif
