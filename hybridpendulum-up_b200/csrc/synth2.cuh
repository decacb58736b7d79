// Synthesis in two passes (ifftSO3R.m:16-37), for complex plans and for the
// real ones that the rule of RealSynthCfg leaves out: bandlimits whose tables
// and buffers do not fit the one-pass kernel, and the smallest.  Included by
// transform_b.cuh.
//   k_synth_beta  warp = one (m, n) pair x 32 omega points: the pair's l-run of
//                 coefficients stays in registers, every beta's sum
//                 G_b[m][n] = sum_l (2l+1) d^l_mn(beta_b) F^l_mn goes to G;
//   k_synth_ga    block = NB betas x PA omega points: gamma FFT over n, alpha
//                 FFT over m, the 2B-runs of the density leave by bulk copies;
//                 on small grids it forms the sums itself (synth_fused).
// What bounds it: G is written and read once (NM * 2B values per omega point
// and beta).  The omega points are taken in chunks whose G stays in L2, so that
// HBM sees little more than F and the density.  The one-kernel form before read
// the coefficients of a pair again for every one or two betas and its d rows
// from L2 for every batch; 88 % of its time at B = 32 was the latency of those
// reads.  24 x 24 omega points, before / now (both passes): B = 32 complex FP32
// 5.85 / 1.24 ms, FP64 14.0 / 2.40; B = 24 complex FP32 1.35 / 0.56; B = 20 real
// FP32 0.49 / 0.16.  Where both forms exist the one-pass kernel is faster (24^3,
// B = 12 FP32: 0.48 against 0.66 ms, B = 15 FP64: 1.93 against 2.58).
#pragma once
#include "row_groups.hpp"

// G of one chunk of omega points: half of the 126 MB L2.  A chunk has at least 32
// points (the lanes of k_synth_beta) where the memory allows it: more than this
// for complex FP64 from B = 26 on, and all of the L2 at B = 32 (132 MB).
constexpr long long kSynthG = 64LL << 20;

template <int B, typename T, bool CPLX> struct Synth2Cfg {
  using C = c2<T>;
  static constexpr int NB2 = 2 * B, NM = CPLX ? 2 * B - 1 : B, NCOL = CPLX ? 2 * B : B;
  // omega points per tile: whole 32-byte sectors of G (16-byte pieces cost
  // k_synth_beta a tenth of its time at B = 32, FP32, complex)
  static constexpr int PA = sizeof(T) == 4 ? 4 : 2;
  static constexpr int NT = NCOL * PA > 128 ? 256 : 128;
  static constexpr int VAL = (int)sizeof(T) * (CPLX ? 2 : 1);     // bytes of a density value
  // staging run of one (omega point, gamma column): NB lines, an odd number of
  // 16-byte units apart
  static constexpr int rs_bytes(int nb) { return (((nb * NB2 * VAL + 15) / 16) | 1) * 16; }
  static constexpr long long bytes(int nb, int pa) {
    const long long g = (long long)nb * NM * NB2 * pa * (long long)sizeof(C);
    const long long st = (long long)pa * NB2 * rs_bytes(nb);
    return g > st ? g : st;
  }
  // three blocks per SM where a tile allows it; the alpha stage is one round
  static constexpr bool fits(int nb, int pa) { return bytes(nb, pa) <= 72 * 1024 && nb * NCOL * pa <= NT; }
  static constexpr int pick_nb() {
    int nb = 1;
    while (nb < 8 && nb < NB2 && fits(nb + 1, PA)) ++nb;
    return nb;
  }
  static constexpr int NB = pick_nb();
  static constexpr bool fusable = B <= 6;   // see synth_fused
  // blocks per SM the registers allow
  static constexpr int MINB = NT == 256 ? 1 : sizeof(T) == 8 ? 2 : (NB2 <= 24 ? 5 : NB2 <= 40 ? 4 : 2);
};

// Small grids of small bandlimits take one kernel, k_synth_ga forming its own sums:
// there the second launch costs more than reading the coefficients once per
// group of betas.  Density call, us, one kernel before there were two / two / this:
// real FP32 B = 3, 8 x 8 10.4 / 12.4 / 8.4, B = 5, 24 x 24 15.9 / 16.5 / 14.5; complex
// FP32 B = 5, 24 x 24 16.5 / 18.6 / 16.5; real FP64 B = 4, 4^3 13.4 / 15.4 / 13.4.  The
// lines: FP64 B = 5, 24 x 24 (72000) 16.6 either way, B = 4, 16^3 (262144) 23.7 two,
// 27.8 one; FP32 real B = 4, 16^3 22.3 two, 18.6 one, complex B = 5, 12^3 (216000) 24.7
// either way, B = 5, 16^3 (512000) 35.0 two, 37.1 one.  B = 7 FP32 complex, 8 x 8: 12.5
// two, 14.5 one.
template <typename T> bool synth_fused(int B, long long nx) {
  return B <= 6 && (long long)B * B * B * nx <= (sizeof(T) == 8 ? 64LL << 10 : 256LL << 10);
}

// dtab: [row][DS] (2l+1) d^l_mn(beta_b), DS = 2B rounded up to 4; Fp: [row][nx];
// G: [w / PA][b][m][n bin ^ x(m)][w % PA] of the chunk's omega points.
template <int B, typename T, bool CPLX>
__global__ void __launch_bounds__(128) k_synth_beta(long long nx, const c2<T>* __restrict__ Fp,
                                                    const T* __restrict__ dtab, const int2* __restrict__ pairs,
                                                    int npairs, c2<T>* __restrict__ G, long long w0, long long nwc) {
  using C = c2<T>;
  using Cfg = Synth2Cfg<B, T, CPLX>;
  constexpr int NB2 = 2 * B, NM = Cfg::NM, PA = Cfg::PA, DS = (NB2 + 3) / 4 * 4;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, pi = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (pi >= npairs) return;
  const int2 pe = pairs[pi];
  const int s = pe.x, len = pe.y & 0xff, mi = (pe.y >> 8) & 0xff, q = (pe.y >> 16) & 0xff;
  // the warp's table rows (whole groups of four: the rows past the run multiply
  // zero coefficients) go to shared memory in one go; read from L2 a sector at
  // a time as the betas advance, they were the stall of three issues in four
  T* d = reinterpret_cast<T*>(smraw) + (threadIdx.x >> 5) * (rows_copied(B) * DS);
  {
    constexpr int EPP = 16 / (int)sizeof(T);
    const T* dsrc = dtab + (size_t)s * DS;
    for (int e = lane; e < rows_copied(len) * DS / EPP; e += 32) cp_async<16>(d + e * EPP, dsrc + e * EPP, true);
  }
  const long long wl = (long long)blockIdx.x * 32 + lane;
  const C* src = Fp + (size_t)s * nx + w0 + wl;
  C v[B];
#pragma unroll
  for (int j = 0; j < B; ++j) v[j] = j < len && wl < nwc ? src[(size_t)j * nx] : czero<C>();
  cp_async_wait_all();
  __syncwarp();
  if (wl >= nwc) return;
  C* g = G + (((wl / PA) * NB2 * NM + mi) * NB2 + (q ^ GSwz<B, C, PA>::x(mi))) * PA + wl % PA;
#pragma unroll 1
  for (int b0 = 0; b0 < NB2; b0 += 4) {
    C acc[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = czero<C>();
    // four rows at a time, their table loads (one address per warp) together
#pragma unroll
    for (int j0 = 0; j0 < B; j0 += 4) {
      if (j0 < len) {
        struct alignas(16) Vec { T x[4]; };
        Vec w[4];
#pragma unroll
        for (int j = 0; j < 4 && j0 + j < B; ++j) w[j] = *reinterpret_cast<const Vec*>(d + (j0 + j) * DS + b0);
#pragma unroll
        for (int j = 0; j < 4 && j0 + j < B; ++j)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            acc[u].x = fma(w[j].x[u], v[j0 + j].x, acc[u].x);
            acc[u].y = fma(w[j].x[u], v[j0 + j].y, acc[u].y);
          }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (b0 + u < NB2) g[(size_t)(b0 + u) * NM * NB2 * PA] = acc[u];
  }
}

// FUSED: the tile of G is summed here, from Fp and the table (w0 = 0, G unused).
template <int B, typename T, bool CPLX, bool FUSED>
__global__ void __launch_bounds__(Synth2Cfg<B, T, CPLX>::NT, Synth2Cfg<B, T, CPLX>::MINB)
    k_synth_ga(const c2<T>* __restrict__ G, void* __restrict__ fout, long long w0, long long nx,
               const c2<T>* __restrict__ Fp, const T* __restrict__ dtab, const int2* __restrict__ pairs) {
  using C = c2<T>;
  using Cfg = Synth2Cfg<B, T, CPLX>;
  constexpr int NB2 = 2 * B, NM = Cfg::NM, NCOL = Cfg::NCOL, PA = Cfg::PA, NB = Cfg::NB, NT = Cfg::NT;
  using Swz = GSwz<B, C, PA>;
  constexpr int K = Swz::K, RS = Cfg::rs_bytes(NB);
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sG = reinterpret_cast<C*>(smraw);
  constexpr int NGRP = (NB2 + NB - 1) / NB;
  const int b0 = (blockIdx.x % NGRP) * NB, nbv = min(NB, NB2 - b0);
  const long long wb = blockIdx.x / NGRP;
  const int tid = threadIdx.x;
  if constexpr (FUSED) {
    constexpr int NPAIR = NM * (2 * B - 1), DS = (NB2 + 3) / 4 * 4;
    for (int it = tid; it < NPAIR * PA; it += NT) {
      const int2 pe = pairs[it / PA];
      const int s = pe.x, len = pe.y & 0xff, mi = (pe.y >> 8) & 0xff, q = (pe.y >> 16) & 0xff, pt = it % PA;
      const bool ok = wb * PA + pt < nx;
      const C* src = Fp + (size_t)s * nx + (ok ? wb * PA + pt : 0);
      const T* d = dtab + (size_t)s * DS + b0;       // a last group's unused betas read on, into the rows behind
      C acc[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) acc[u] = czero<C>();
#pragma unroll 4
      for (int j = 0; j < len; ++j) {
        const C v = src[(size_t)j * nx];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          acc[u].x = fma(d[j * DS + u], v.x, acc[u].x);
          acc[u].y = fma(d[j * DS + u], v.y, acc[u].y);
        }
      }
      C* g = sG + (mi * NB2 + (q ^ Swz::x(mi))) * PA + pt;
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (u < nbv) g[u * NM * NB2 * PA] = acc[u];
    }
  } else {
    const C* src = G + (wb * NB2 + b0) * NM * NB2 * PA;
    constexpr int EPP = 16 / (int)sizeof(C);
    const int n = nbv * NM * NB2 * PA / EPP;
    for (int e = tid; e < n; e += NT) cp_async<16>(sG + e * EPP, src + (size_t)e * EPP, true);
    cp_async_wait_all();
  }
  __syncthreads();
  // gamma stage: item (bb, m, p), in place; bin B is empty
  for (int it = tid; it < nbv * NM * PA; it += NT) {
    const int rowi = it / PA, s = Swz::x(rowi % NM);
    C* base = sG + (size_t)rowi * NB2 * PA + it % PA;
    C* cls[K];
#pragma unroll
    for (int k = 0; k < K; ++k) cls[k] = base + (k ^ s) * PA;
    C x[NB2];
#pragma unroll
    for (int j = 0; j < NB2; ++j) x[j] = j == B ? czero<C>() : cls[j % K][(j / K * K) * PA];
    fft<NB2, false>(x);
#pragma unroll
    for (int j = 0; j < NB2; ++j) cls[j % K][(j / K * K) * PA] = x[j];
  }
  __syncthreads();
  // alpha stage, one round.  Real plans: two columns c, c + B per complex FFT
  // (the Hermitian extensions of H[.][c]); complex plans: one column.
  const int p = tid % PA, c = (tid / PA) % NCOL, bb = tid / (PA * NCOL);
  const bool act = bb < nbv;
  C x[NB2];
  if (act) {
    const C* h = sG + (size_t)bb * NM * NB2 * PA + p;
    x[B] = czero<C>();
    if constexpr (CPLX) {
#pragma unroll
      for (int mi = 0; mi < NM; ++mi) {
        const int m = mi - (B - 1);
        x[m >= 0 ? m : m + NB2] = h[(mi * NB2 + (c ^ Swz::x(mi))) * PA];
      }
    } else {
#pragma unroll
      for (int m = 0; m < B; ++m) {
        const C u = h[(m * NB2 + (c ^ Swz::x(m))) * PA], v = h[(m * NB2 + ((c + B) ^ Swz::x(m))) * PA];
        if (m == 0) {
          x[0] = mk(u.x, v.x);
        } else {
          x[m] = cadd_i<false>(u, v);
          x[NB2 - m] = mk(u.x + v.y, v.x - u.y);
        }
      }
    }
    fft<NB2, false>(x);
  }
  __syncthreads();
  if (act) {   // staging runs [c][p] of nbv lines, aliasing sG
    unsigned char* st = smraw + (size_t)(c * PA + p) * RS;
    if constexpr (CPLX) {
      C* o = reinterpret_cast<C*>(st) + bb * NB2;
#pragma unroll
      for (int a = 0; a < NB2; ++a) o[a] = x[a];
    } else {
      T* o = reinterpret_cast<T*>(st) + bb * NB2;
      T* o2 = reinterpret_cast<T*>(st + (size_t)B * PA * RS) + bb * NB2;
      if constexpr (sizeof(T) == 4) {
        if (((bb * NB2) & 3) == 0) stage_run<NB2, 0>(o, o2, x);
        else stage_run<NB2, 2>(o, o2, x);
      } else {
#pragma unroll
        for (int i = 0; i < NB2; i += 2) {
          *reinterpret_cast<double2*>(o + i) = make_double2(x[i].x, x[i + 1].x);
          *reinterpret_cast<double2*>(o2 + i) = make_double2(x[i].y, x[i + 1].y);
        }
      }
    }
  }
  // bulk copies where every run starts and ends on a 16-byte boundary
  constexpr int VAL = Cfg::VAL;
  const bool bulk = (reinterpret_cast<unsigned long long>(fout) & 15ull) == 0 && (b0 * NB2 * VAL) % 16 == 0 &&
                    (nbv * NB2 * VAL) % 16 == 0 && (NB2 * NB2 * VAL) % 16 == 0;
  if (bulk) fence_proxy_async_smem();
  __syncthreads();
  // f[a + 2B (b + 2B (c + 2B w))]; runs go [c][p], the points past the end of a
  // batch that PA does not divide are left out
  const int pc = (int)min((long long)PA, nx - w0 - wb * PA);
  auto dst = [&](int run) -> unsigned char* {
    const long long w = w0 + wb * PA + run % PA;
    return reinterpret_cast<unsigned char*>(fout) + (((size_t)w * NB2 + run / PA) * NB2 + b0) * NB2 * VAL;
  };
  if (bulk) {
    const uint64_t pol = l2_policy_evict_first();
    if ((tid & 31) == 0)
      for (int run = tid >> 5; run < PA * NB2; run += NT / 32)
        if (run % PA < pc) bulk_s2g(dst(run), smraw + (size_t)run * RS, (unsigned)(nbv * NB2 * VAL), pol);
    bulk_commit();
    bulk_wait_all();   // shared memory must outlive the copies reading it
  } else {
    for (int run = tid >> 5; run < PA * NB2; run += NT / 32) {
      if (run % PA >= pc) continue;
      T* o = reinterpret_cast<T*>(dst(run));
      const T* src = reinterpret_cast<const T*>(smraw + (size_t)run * RS);
      for (int e = tid & 31; e < nbv * NB2 * (VAL / (int)sizeof(T)); e += 32) o[e] = src[e];
    }
  }
}

// (2l+1) d^l_mn(beta_b) as [row][DS], zero beyond b = 2B and in the kRowPad rows
// behind the last one (k_synth_beta reads whole groups of rows)
template <typename T>
__global__ void k_dsyn_table(RowLayout L, const T* __restrict__ wig, int DS, T* __restrict__ out) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (L.nrows + kRowPad) * DS) return;
  const long long r = t / DS;
  const int b = (int)(t % DS);
  out[t] = r < L.nrows && b < 2 * L.B ? (T)(2 * L.rows[r].x + 1) * wig[(size_t)b * L.nrows + r] : (T)0;
}

// gkey: the workspace buffer of G
template <int B, typename T, bool CPLX>
int synth2_launch(hp_plan* p, const c2<T>* Fp, void* f, long long nx, const char* gkey, cudaStream_t s) {
  using C = c2<T>;
  using Cfg = Synth2Cfg<B, T, CPLX>;
  if (tw_init() != 0) { hp_set_error("twiddle table upload failed"); return HP_ERR_CUDA; }
  constexpr int NB2 = 2 * B, NM = Cfg::NM, PA = Cfg::PA, NB = Cfg::NB, NPAIR = NM * (2 * B - 1), DS = (NB2 + 3) / 4 * 4;
  int st = HP_OK;
  const int2* dpairs = pair_table<B, CPLX>(p, &st, s);
  if (st) return st;
  const char* dkey = sizeof(T) == 8 ? "tf.dsyn64" : "tf.dsyn32";
  bool have = false;
  for (auto& kv : p->ws) if (kv.first == dkey) have = true;
  T* dtab = (T*)p->ws_get(dkey, sizeof(T) * (p->nrows + kRowPad) * DS, &st);
  if (st) return st;
  if (!have) {
    const long long n = (p->nrows + kRowPad) * DS;
    k_dsyn_table<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        p->layout(), sizeof(T) == 8 ? (const T*)(const void*)p->wig64 : (const T*)(const void*)p->wig32, DS, dtab);
    HP_CUDA_TRY(cudaGetLastError());
  }
  constexpr size_t smem = (size_t)Cfg::bytes(NB, PA);
  constexpr int NGRP = (NB2 + NB - 1) / NB;
  if constexpr (Cfg::fusable) {
    if (synth_fused<T>(B, nx)) {
      HP_CUDA_TRY(cudaFuncSetAttribute(k_synth_ga<B, T, CPLX, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      ProfScope _ps(p, "tf.synth", s);
      k_synth_ga<B, T, CPLX, true><<<(unsigned)((nx + PA - 1) / PA * NGRP), Cfg::NT, smem, s>>>(nullptr, f, 0, nx, Fp, dtab,
                                                                                               dpairs);
      HP_CUDA_TRY(cudaGetLastError());
      return HP_OK;
    }
  }
  const long long per_w = (long long)NM * NB2 * NB2 * (long long)sizeof(C);
  long long nwc = std::max(32LL, kSynthG / per_w / 32 * 32);
  nwc = std::min(nwc, (nx + 31) / 32 * 32);
  long long units = 0;   // whole tiles of PA points
  C* G = (C*)p->ws_get_units(gkey, (size_t)per_w * PA, nwc / PA, 1, &units, &st);
  if (st) return st;
  nwc = units * PA;
  HP_CUDA_TRY(cudaFuncSetAttribute(k_synth_ga<B, T, CPLX, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (long long w0 = 0; w0 < nx; w0 += nwc) {
    const long long nw = std::min(nwc, nx - w0);
    {
      ProfScope _ps(p, "tf.synth.beta", s);
      constexpr size_t dsm = 4 * sizeof(T) * (size_t)(rows_copied(B) * DS);
      HP_CUDA_TRY(cudaFuncSetAttribute(k_synth_beta<B, T, CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dsm));
      k_synth_beta<B, T, CPLX><<<dim3((unsigned)((nw + 31) / 32), (unsigned)((NPAIR + 3) / 4)), 128, dsm, s>>>(
          nx, Fp, dtab, dpairs, NPAIR, G, w0, nw);
      HP_CUDA_TRY(cudaGetLastError());
    }
    ProfScope _ps(p, "tf.synth", s);
    k_synth_ga<B, T, CPLX, false><<<(unsigned)((nw + PA - 1) / PA * NGRP), Cfg::NT, smem, s>>>(G, f, w0, nx, Fp, dtab, dpairs);
    HP_CUDA_TRY(cudaGetLastError());
  }
  return HP_OK;
}
