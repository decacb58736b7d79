// Synthesis of real densities (ifftSO3R.m:16-37, pendulum.m:284-304) with the
// coefficients of the next omega batch copied to shared memory while the
// current one is transformed.  Included by transform_b.cuh.
//
// Block = (NN nodes beta_b and their mirrors beta_{2B-1-b} = pi - beta_b, a
// range of omega points walked in batches of P).  Per batch:
//   beta   G[slot][m][n] = sum_l (2l+1) d^l_mn(beta) F^l_mn for the 2 NN betas,
//          one item per (m, n >= 0, omega point) forming the rows (m, n) and
//          (m, -n) together: by d^l_mn(pi - beta) = (-1)^(l+m) d^l_{m,-n}(beta)
//          the table values d_{m,n} and d_{m,-n} of the nodes serve all four
//          (row, node or mirror) sums, so the table holds half of the betas;
//   gamma  2B-point FFT over n, in place;
//   alpha  2B-point FFT over m, two real columns per complex FFT;
//   store  the 2B-runs of the density leave by bulk copies.
// What bounds it: before this form the beta stage read its coefficients from
// L2 as it needed them, and two thirds of a block's time (B = 15, FP32) was the
// latency of those loads.  Here the loads of batch k+1 are issued as
// asynchronous copies right after the beta stage of batch k has read the
// buffer, and land during the FFT stages; the rows are also read once per
// 2 NN betas instead of once per 4.  At 24^3, before / now (us): B = 15 FP32
// 1243 / 886, FP64 3762 / 1930; B = 12 FP32 633 / 479, FP64 2026 / 943; B = 8
// FP32 191 / 119, FP64 395 / 252.  Now the shared-memory pipe is busy 40 % of
// the time and the rest is barriers and latency at 16 warps per SM (8 in FP64);
// two independent teams of threads per block, the store by vector stores, or
// the copies spread over more lanes measured no better.
#pragma once

template <int B, typename T> struct RealSynthCfg {
  static constexpr long long nrows = (long long)B * (B + 1) * (4 * B - 1) / 6;
  static constexpr int NT = sizeof(T) == 4 ? 512 : 256;   // 128 / 255 registers for the register FFTs
  static constexpr int NB2 = 2 * B;
  // staging run: 2 NN lines of 2B values, padded so that consecutive runs
  // start an odd number of 16-byte units apart (conflict-free 16-byte stores)
  static constexpr int rs(int nn) {
    constexpr int u = 16 / (int)sizeof(T);
    int units = (2 * nn * NB2 + u - 1) / u;
    return (units | 1) * u;
  }
  static constexpr long long d_bytes(int nn) { return (nn * nrows * (long long)sizeof(T) + 15) / 16 * 16; }
  static constexpr long long c_bytes(int p) { return nrows * p * 2 * (long long)sizeof(T); }
  static constexpr long long p_bytes() { return ((long long)B * B * 8 + 15) / 16 * 16; }
  static constexpr long long g_bytes(int nn, int p) {
    const long long g = 2LL * nn * B * NB2 * p * 2 * (long long)sizeof(T);
    const long long st = (long long)p * NB2 * rs(nn) * (long long)sizeof(T);
    return g > st ? g : st;
  }
  static constexpr long long bytes(int nn, int p) { return d_bytes(nn) + p_bytes() + c_bytes(p) + g_bytes(nn, p); }
  static constexpr bool fits(int nn, int p) {
    // FP32 runs start and end on 16-byte boundaries when nn or B is even
    return bytes(nn, p) <= 227 * 1024 && 2 * nn * B * p <= NT && (sizeof(T) == 8 || nn % 2 == 0 || B % 2 == 0);
  }
  // nodes per block and omega points per batch: the pair with the most FFTs
  // per round (threads in use x share of the last group's nodes), the more
  // nodes at equal use (fewer reads of the coefficients)
  static constexpr long long score(int nn, int p) {
    return fits(nn, p) ? (1000LL * B / ((B + nn - 1) / nn * nn)) * (2 * nn * B * p) * 16 + nn : 0;
  }
  static constexpr int pick(bool want_nn) {
    long long best = 0;
    int bn = 0, bp = 0;
    for (int p = sizeof(T) == 4 ? 4 : 2; p <= 4; p += 2)
      for (int nn = 1; nn <= B; ++nn)
        if (score(nn, p) > best) { best = score(nn, p); bn = nn; bp = p; }
    return want_nn ? bn : bp;
  }
  static constexpr int NN = pick(true), P = pick(false);
  // The rule of the dispatch: tables and buffers of two nodes or more fit, and the
  // bandlimit is not one of the smallest; elsewhere the two passes of synth2.cuh
  // are faster.  24^3, us, this / two passes: B = 8 FP32 119 / 171, B = 16 FP32
  // 1209 / 1518, B = 12 FP64 943 / 1251; the other way at B = 5 FP32, 90 / 50, and
  // B = 6 FP64, 145 / 100.  The upper edge, at 16^3: FP32 B = 16 359 / 418, B = 17
  // 610 / 818; FP64 B = 16 662 / 802.  With one node per block every coefficient is
  // read B times and a quarter of the threads have an FFT: FP32 B = 18 968 / 784,
  // FP64 B = 17 1761 / 1244, B = 18 1892 / 1283 (24 x 24 points: FP32 B = 18 152 /
  // 116, FP64 B = 17 265 / 174).  On 16 x 16 points they are level at B = 16 (FP32 33 / 32).
  static constexpr bool ok = NN > 1 && B >= (sizeof(T) == 4 ? 6 : 7) && nrows < 65536;
};

// Row m of the G planes keeps its gamma index j at j ^ x(m), so that the rows
// that one 128-byte wavefront touches (U units of one complex value, P per
// row) fall on distinct banks: rows are 2B P units apart, which alone
// separates D0 of them.
template <int B, typename C, int P> struct GSwz {
  static constexpr int U = 128 / (int)sizeof(C), ROWS = U / P;
  static constexpr int gcd(int a, int b) { return b ? gcd(b, a % b) : a; }
  static constexpr int D0 = U / gcd(2 * B * P, U) < ROWS ? U / gcd(2 * B * P, U) : ROWS;
  static constexpr int K = ROWS / D0;               // classes, a power of two dividing 2B
  static_assert((2 * B) % K == 0, "classes permute the gamma index");
  __device__ static int x(int m) { return (m / D0) % K; }
};

template <int B, typename T, int NN, int P>
__global__ void __launch_bounds__(RealSynthCfg<B, T>::NT, 1)
    k_synth_real(long long nx, const c2<T>* __restrict__ Fp, const T* __restrict__ dtab,
                 const int2* __restrict__ pairs, T* __restrict__ fout, int nbatch) {
  using C = c2<T>;
  using Cfg = RealSynthCfg<B, T>;
  using Swz = GSwz<B, C, P>;
  constexpr int NT = Cfg::NT, NB2 = 2 * B, NG = (B + NN - 1) / NN, RS = Cfg::rs(NN);
  constexpr int nrows = (int)Cfg::nrows, NITEM = B * B * P;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x;
  T* sD = reinterpret_cast<T*>(smraw);                                       // [row][NN]
  int2* sPairs = reinterpret_cast<int2*>(smraw + Cfg::d_bytes(NN));
  C* sC = reinterpret_cast<C*>(smraw + Cfg::d_bytes(NN) + Cfg::p_bytes());   // [row][P]
  C* sG = reinterpret_cast<C*>(smraw + Cfg::d_bytes(NN) + Cfg::p_bytes() + Cfg::c_bytes(P));
  T* sOut = reinterpret_cast<T*>(sG);
  // omega blocks of one chunk of every beta group are consecutive blocks (L2 reuse of the rows)
  const int grp = blockIdx.x % NG;
  const long long chunk = blockIdx.x / NG;
  const int b0 = grp * NN, cnt = min(NN, B - b0);
  // tables by asynchronous copies, which land with those of the first batch.  By
  // loads, round after round, they were a good part of a block's life on small
  // grids (us, before / now: B = 9, 8 x 8 points, whole call 15.5 / 13.5; synthesis
  // at B = 16, 16 x 16 41.4 / 33.3, 8^3 72 / 56, 16^3 379 / 359; FP64 16^3 681 / 663)
  {
    constexpr int EP = 16 / (int)sizeof(T), GS = (int)(Cfg::d_bytes(NN) / (int)sizeof(T));
    const T* src = dtab + (size_t)grp * GS;
    for (int e = tid; e < GS / EP; e += NT) cp_async<16>(sD + e * EP, src + e * EP, true);
    for (int e = tid; e < B * B; e += NT) cp_async<8>(sPairs + e, pairs + e, true);
  }
  // one batch of coefficients: the rows arrive omega-blocked, [w / P][row][w % P],
  // one contiguous run per batch (from [row][omega], 32 bytes per row, the B = 15
  // FP32 synthesis at 24^3 took 1025 us instead of 882)
  auto fill = [&](long long w0) {
    const C* src = Fp + w0 * nrows;
    constexpr int EPP = 16 / (int)sizeof(C);           // elements per 16-byte piece
    for (int e = tid; e < nrows * P / EPP; e += NT) cp_async<16>(sC + e * EPP, src + (size_t)e * EPP, true);
  };
  const bool al16 = (reinterpret_cast<unsigned long long>(fout) & 15ull) == 0;
  long long w0 = chunk * nbatch * P;
  const long long w1 = min(nx, w0 + (long long)nbatch * P);
  if (w0 < w1) fill(w0);
  for (; w0 < w1; w0 += P) {
    cp_async_wait_all();
    if (al16) bulk_wait_read_all();
    __syncthreads();
    // beta stage; every other round runs backwards through the length-sorted
    // items, so that a thread with long sums gets short ones next
#pragma unroll 1
    for (int r = 0; r * NT < NITEM; ++r) {
      const int it = (r & 1) ? (r + 1) * NT - 1 - tid : r * NT + tid;
      const bool item = it < NITEM;
      const int p = it % P;
      const int2 pe = item ? sPairs[it / P] : make_int2(0, 0);   // length 0: nothing summed
      const int sp = pe.x & 0xffff, sn = (int)((unsigned)pe.x >> 16);
      const int len = pe.y & 0xff, mi = (pe.y >> 8) & 0xff, n = (pe.y >> 16) & 0xff;
      C a[NN], am[NN], b[NN], bm[NN];   // (node, n), (mirror, n), (node, -n), (mirror, -n)
#pragma unroll
      for (int k = 0; k < NN; ++k) a[k] = am[k] = b[k] = bm[k] = czero<C>();
      const C *cp = sC + sp * P + p, *cn = sC + sn * P + p;
      const T *dp = sD + sp * NN, *dn = sD + sn * NN;
      auto row = [&](int l, bool odd) {
        const C vp = cp[l * P], vn = cn[l * P];
        T x[NN], y[NN];
        if constexpr (NN * sizeof(T) % 16 == 0) {
          constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
          for (int k = 0; k < NN; k += V) {
            struct alignas(16) Vec { T v[V]; };
            *reinterpret_cast<Vec*>(x + k) = *reinterpret_cast<const Vec*>(dp + l * NN + k);
            *reinterpret_cast<Vec*>(y + k) = *reinterpret_cast<const Vec*>(dn + l * NN + k);
          }
        } else {
#pragma unroll
          for (int k = 0; k < NN; ++k) { x[k] = dp[l * NN + k]; y[k] = dn[l * NN + k]; }
        }
#pragma unroll
        for (int k = 0; k < NN; ++k) {
          a[k].x = fma(x[k], vp.x, a[k].x);  a[k].y = fma(x[k], vp.y, a[k].y);
          b[k].x = fma(y[k], vn.x, b[k].x);  b[k].y = fma(y[k], vn.y, b[k].y);
          const T xs = odd ? -x[k] : x[k], ys = odd ? -y[k] : y[k];
          am[k].x = fma(ys, vp.x, am[k].x);  am[k].y = fma(ys, vp.y, am[k].y);
          bm[k].x = fma(xs, vn.x, bm[k].x);  bm[k].y = fma(xs, vn.y, bm[k].y);
        }
      };
      int l = 0;
#pragma unroll 1
      for (; l + 1 < len; l += 2) { row(l, false); row(l + 1, true); }
      if (l < len) row(l, false);
      if (!item) continue;
      // the mirror sign of the first row, l = B - len
      const T sg = ((B - len + mi) & 1) ? (T)-1 : (T)1;
      const int q1 = n, q2 = n ? NB2 - n : B, s = Swz::x(mi);
#pragma unroll
      for (int k = 0; k < NN; ++k) {
        if (k >= cnt) break;
        C* g = sG + ((size_t)(k * B + mi) * NB2) * P + p;                       // slot of node k
        C* gm = sG + ((size_t)((2 * cnt - 1 - k) * B + mi) * NB2) * P + p;      // and of its mirror
        g[(q1 ^ s) * P] = a[k];
        gm[(q1 ^ s) * P] = sg * am[k];
        g[(q2 ^ s) * P] = n ? b[k] : czero<C>();                                // bin B is empty
        gm[(q2 ^ s) * P] = n ? sg * bm[k] : czero<C>();
      }
    }
    __syncthreads();
    if (w0 + P < w1) fill(w0 + P);
    const bool act = tid < 2 * cnt * B * P;
    // gamma stage: item (slot, m, p)
    if (act) {
      const int rowi = tid / P, s = Swz::x(rowi % B);
      C* base = sG + (size_t)rowi * NB2 * P + tid % P;
      constexpr int K = Swz::K;
      C* cls[K];                                       // j ^ s by the low bits of j
#pragma unroll
      for (int k = 0; k < K; ++k) cls[k] = base + (k ^ s) * P;
      C x[NB2];
#pragma unroll
      for (int j = 0; j < NB2; ++j) x[j] = cls[j % K][(j / K * K) * P];
      fft<NB2, false>(x);
#pragma unroll
      for (int j = 0; j < NB2; ++j) cls[j % K][(j / K * K) * P] = x[j];
    }
    __syncthreads();
    // alpha stage: f_c = Re FFT(w_m H[m][c]) = FFT(h_c), h_c the Hermitian
    // extension of H[.][c]; columns c and c + B share one complex FFT
    const int p = tid % P, c = (tid / P) % B, slot = tid / (P * B);
    C x[NB2];
    if (act) {
      const C* h = sG + (size_t)slot * B * NB2 * P + p;
      x[B] = czero<C>();
#pragma unroll
      for (int m = 0; m < B; ++m) {
        const C u = h[(m * NB2 + (c ^ Swz::x(m))) * P], v = h[(m * NB2 + ((c + B) ^ Swz::x(m))) * P];
        if (m == 0) {
          x[0] = mk(u.x, v.x);
        } else {
          x[m] = cadd_i<false>(u, v);                       // u + i v
          x[NB2 - m] = mk(u.x + v.y, v.x - u.y);            // conj(u) + i conj(v)
        }
      }
      fft<NB2, false>(x);
    }
    __syncthreads();
    if (act) {   // staging runs [c][p] of 2 cnt lines, aliasing sG
      T* st = sOut + (size_t)(c * P + p) * RS + slot * NB2;
      T* st2 = sOut + (size_t)((c + B) * P + p) * RS + slot * NB2;
      if constexpr (sizeof(T) == 4) {
        if (((slot * NB2) & 3) == 0) stage_run<NB2, 0>(st, st2, x);
        else stage_run<NB2, 2>(st, st2, x);
      } else {
#pragma unroll
        for (int i = 0; i < NB2; i += 2) {
          *reinterpret_cast<double2*>(st + i) = make_double2(x[i].x, x[i + 1].x);
          *reinterpret_cast<double2*>(st2 + i) = make_double2(x[i].y, x[i + 1].y);
        }
      }
    }
    if (al16) fence_proxy_async_smem();
    __syncthreads();
    // f[a + 2B (beta + 2B (c + 2B w))]: the node lines b0 .. b0+cnt-1 and the
    // mirror lines 2B-b0-cnt .. 2B-1-b0 of one (w, c), each contiguous in f and
    // in the staging buffer; one run where they meet (the last group)
    const bool one = b0 + cnt == B;
    const int len1 = (one ? 2 * cnt : cnt) * NB2, len2 = one ? 0 : cnt * NB2;
    if (al16) {
      const uint64_t pol = l2_policy_evict_first();
      // one lane per warp walks its share of the runs: a copy issued by every
      // lane of a warp costs a turn of about 140 cycles per lane
      if ((tid & 31) == 0)
        for (int run = tid >> 5; run < P * NB2; run += NT / 32) {
          const int cc = run / P, pp = run % P;
          T* dst = fout + ((size_t)(w0 + pp) * NB2 + cc) * NB2 * NB2;
          const T* src = sOut + (size_t)run * RS;
          bulk_s2g(dst + b0 * NB2, src, (unsigned)(len1 * sizeof(T)), pol);
          if (!one) bulk_s2g(dst + (NB2 - b0 - cnt) * NB2, src + len1, (unsigned)(len2 * sizeof(T)), pol);
        }
      bulk_commit();
    } else {
      const int lane = tid & 31, warp = tid >> 5;
      for (int run = warp; run < P * NB2; run += NT / 32) {
        const int cc = run / P, pp = run % P;
        const size_t line = ((size_t)(w0 + pp) * NB2 + cc) * NB2;
        const T* src = sOut + (size_t)run * RS;
        for (int o = lane; o < len1 + len2; o += 32)
          fout[(line + b0) * NB2 + o + (o < len1 ? 0 : (size_t)(NB2 - 2 * b0 - 2 * cnt) * NB2)] = src[o];
      }
    }
  }
  if (al16) bulk_wait_all();   // shared memory must outlive the bulk copies reading it
}

// Entry q < B^2: the pair (m, n >= 0) with row starts of (m, n) and (m, -n),
// length of their l-run, m and n; longest runs first.  The (max(m, n) + 1)^2
// pairs up to max(m, n) come before all others, so q gives its pair in closed
// form, and the table is built on the device in the buffer of the d table:
// a new plan's first synthesis needs no allocation, copy and wait for it.
template <int B>
__global__ void k_node_pairs(RowLayout L, int2* __restrict__ out) {
  constexpr int lmax = B - 1, D = 2 * lmax + 1;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= B * B) return;
  int lmin = 0;
  while ((lmin + 1) * (lmin + 1) <= q) ++lmin;
  const int r = q - lmin * lmin, m = min(r, lmin), n = r < lmin ? lmin : r - lmin;
  const int* seg = L.seg + (m - L.m_lo) * D + lmax;
  out[q] = make_int2((int)((unsigned)seg[n] | ((unsigned)seg[-n] << 16)), (B - lmin) | (m << 8) | (n << 16));
}

template <int B, typename T>
int synth_real_launch(hp_plan* p, const c2<T>* Fp, T* f, cudaStream_t s) {
  using Cfg = RealSynthCfg<B, T>;
  constexpr int NN = Cfg::NN, P = Cfg::P, NG = (B + NN - 1) / NN;
  int st = HP_OK;
  // (2l+1) d at the nodes as [group][row][NN], then the pairs (8-byte aligned)
  const char* key = sizeof(T) == 8 ? "tf.sdn64" : "tf.sdn32";
  bool have = false;
  for (auto& kv : p->ws) if (kv.first == key) have = true;
  constexpr int gs = (int)(Cfg::d_bytes(NN) / (int)sizeof(T)), n = NG * gs;
  constexpr size_t nd = sizeof(T) * (size_t)n;
  char* tab = (char*)p->ws_get(key, nd + sizeof(int2) * B * B, &st);
  if (st) return st;
  T* dtab = (T*)tab;
  int2* dpairs = (int2*)(tab + nd);
  if (!have) {
    k_sd_table<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        p->layout(), sizeof(T) == 8 ? (const T*)(const void*)p->wig64 : (const T*)(const void*)p->wig32, dtab, NN, gs, NG);
    HP_CUDA_TRY(cudaGetLastError());
    k_node_pairs<B><<<(B * B + 127) / 128, 128, 0, s>>>(p->layout(), dpairs);
    HP_CUDA_TRY(cudaGetLastError());
  }
  constexpr size_t smem = (size_t)Cfg::bytes(NN, P);
  const long long nbatches = p->nx / P;   // N is even: nx is a multiple of 4
  long long gx = std::max(1LL, 148LL * p->tune.synth_waves / NG);
  const int nbatch = (int)std::max(1LL, (nbatches + gx - 1) / gx);
  gx = (nbatches + nbatch - 1) / nbatch;
  HP_CUDA_TRY(cudaFuncSetAttribute(k_synth_real<B, T, NN, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ProfScope _ps(p, "tf.synth", s);
  k_synth_real<B, T, NN, P><<<(unsigned)(gx * NG), Cfg::NT, smem, s>>>(p->nx, Fp, dtab, dpairs, f, nbatch);
  HP_CUDA_TRY(cudaGetLastError());
  return HP_OK;
}
