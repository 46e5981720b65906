// linalg.cu -- FP64 complex dense kernels for the stabilisation path:
// GEMM, Householder QR with Q formation (zgeqrf/zungqr conventions), LU with
// partial pivoting (zgetf2's pivots) with the right-hand sides solved in the
// same pass, and log-det.
//
// GB300 runs FP64 at a small fraction of its FP32 rate, so every routine
// spreads its work over all SMs: the factorisations are cooperative kernels
// that pipeline over columns, the products give every warp its share of the
// outputs and of the sums.
#include <algorithm>
#include <type_traits>
#include "linalg.cuh"
#include "warp_sum.cuh"

namespace pqmc {

// ---------------------------------------------------------------------------
// C = alpha * op(A) * op(B) + beta * C, op in {N, C (conjugate transpose)}.
//
// FP64 issue bounds it: a multiply-add holds an SM quarter for 64 cycles, so
// one warp per quarter is enough and operands come straight from L1 (two
// 16-byte loads per four multiply-adds).  What is left is to give every
// quarter the same work: a warp makes 32, 16, 8 or 4 outputs with the sum over
// k in 1, 2, 4 or 8 shares, whichever leaves the fullest quarter the least.
// Measured for 196 x 196 x 392, 392 x 392 x 196 and 32 x 32 x 8: 111, 207 and
// 2.6 us (FP64 issue alone 103 and 206); as 32 x 32 tiles through shared
// memory, 49 and 169 CTAs, 432, 428 and 19.
constexpr int ZG_AHEAD = 4;   // elements of the sum in flight
template <bool TA, bool TB>
__global__ void __launch_bounds__(128) k_zgemm(int m, int n, int k, int ls, cplx alpha, const cplx* __restrict__ A,
                                               int lda, const cplx* __restrict__ B, int ldb, cplx beta,
                                               cplx* __restrict__ C, int ldc) {
  // a warp's outputs: 2^lr x 2^lc of them, 2^ls shares of the sum
  const int lr = (6 - ls) >> 1, lc = (5 - ls) >> 1;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int o = lane & ((32 >> ls) - 1), h = lane >> (5 - ls);
  const int r = ((2 * blockIdx.x + (w & 1)) << lr) + (o & ((1 << lr) - 1));
  const int c = ((2 * blockIdx.y + (w >> 1)) << lc) + (o >> lr);
  if (((2 * blockIdx.x + (w & 1)) << lr) >= m || ((2 * blockIdx.y + (w >> 1)) << lc) >= n) return;   // the whole warp
  const int kl = (k + (1 << ls) - 1) >> ls, k0 = min(k, h * kl), k1 = min(k, k0 + kl);
  const int ra = min(r, m - 1), cb = min(c, n - 1);
  const size_t da = TA ? 1 : lda, db = TB ? ldb : 1;
  const double2* a = reinterpret_cast<const double2*>(A) + (TA ? (size_t)lda * ra : (size_t)ra) + da * k0;
  const double2* b = reinterpret_cast<const double2*>(B) + (TB ? (size_t)cb : (size_t)ldb * cb) + db * k0;
  const double2 zero = make_double2(0.0, 0.0);
  double2 va[ZG_AHEAD], vb[ZG_AHEAD];
  cplx acc = mk(0.0);
#pragma unroll
  for (int e = 0; e < ZG_AHEAD; ++e) {
    va[e] = k0 + e < k1 ? __ldg(a + da * e) : zero;
    vb[e] = k0 + e < k1 ? __ldg(b + db * e) : zero;
  }
  for (int q = 0; q < kl; q += ZG_AHEAD) {   // the same number of steps in every lane
    a += da * ZG_AHEAD;
    b += db * ZG_AHEAD;
#pragma unroll
    for (int e = 0; e < ZG_AHEAD; ++e) {
      if (q + e >= kl) break;
      cplx x = mk(va[e].x, va[e].y), y = mk(vb[e].x, vb[e].y);
      const bool more = k0 + q + e + ZG_AHEAD < k1;
      va[e] = more ? __ldg(a + da * e) : zero;
      vb[e] = more ? __ldg(b + db * e) : zero;
      if (TA) x = cconj(x);
      if (TB) y = cconj(y);
      acc = cfma(x, y, acc);
    }
  }
  for (int d = 16; d >= (32 >> ls); d >>= 1) {
    acc.x += __shfl_xor_sync(~0u, acc.x, d);
    acc.y += __shfl_xor_sync(~0u, acc.y, d);
  }
  if (h == 0 && r < m && c < n) {
    cplx* p = C + r + (size_t)ldc * c;
    cplx v = cmul(alpha, acc);
    if (beta.x != 0.0 || beta.y != 0.0) v = cfma(beta, *p, v);
    *p = v;
  }
}

int zgemm(cudaStream_t s, char ta, char tb, int m, int n, int k, cplx alpha, const cplx* A, int lda,
          const cplx* B, int ldb, cplx beta, cplx* C, int ldc) {
  int dev = 0, nsm = 0;
  PQMC_CUDA(cudaGetDevice(&dev));
  PQMC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // shares of the sum: FP64 instructions of the fullest SM quarter, a CTA
  // being a warp on each; the largest share that is no worse
  int ls = 0;
  long best = 0;
  dim3 grid;
  for (int l = 0; l <= 3; ++l) {
    const int th = 2 << ((6 - l) >> 1), tw = 2 << ((5 - l) >> 1);
    const dim3 g((m + th - 1) / th, (n + tw - 1) / tw);
    const long rounds = ((long)g.x * g.y + nsm - 1) / nsm, cost = rounds * (4L * ((k + (1 << l) - 1) >> l) + 2 * l + 8);
    if (l == 0 || cost < best) {
      best = cost;
      ls = l;
      grid = g;
    }
  }
  bool TA = (ta == 'C'), TB = (tb == 'C');
  if (!TA && !TB) k_zgemm<false, false><<<grid, 128, 0, s>>>(m, n, k, ls, alpha, A, lda, B, ldb, beta, C, ldc);
  else if (TA && !TB) k_zgemm<true, false><<<grid, 128, 0, s>>>(m, n, k, ls, alpha, A, lda, B, ldb, beta, C, ldc);
  else if (!TA && TB) k_zgemm<false, true><<<grid, 128, 0, s>>>(m, n, k, ls, alpha, A, lda, B, ldb, beta, C, ldc);
  else k_zgemm<true, true><<<grid, 128, 0, s>>>(m, n, k, ls, alpha, A, lda, B, ldb, beta, C, ldc);
  PQMC_LAUNCHED();
  return PQMC_OK;
}

// ---------------------------------------------------------------------------
// Column pipeline shared by the two factorisations.  Columns are dealt out to
// CTAs of 128 threads (a warp on each SM quarter) and stay in shared memory;
// the CTA that finishes a column publishes it once in the work matrix `pub`,
// which starts out filled with a bit pattern no published value has, and the
// others poll the very words they need: a published value is its own flag,
// so a step costs one L2 round trip and no grid barrier.  The launch is
// cooperative (every CTA resident); every poll is bounded.
constexpr int LT = 128;
constexpr unsigned long long LA_EMPTY = ~0ull;   // memset 0xff; a NaN pattern publish() never writes

__device__ __forceinline__ void publish(cplx* p, cplx v) {
  unsigned long long x = (unsigned long long)__double_as_longlong(v.x), y = (unsigned long long)__double_as_longlong(v.y);
  if (x == LA_EMPTY) x = 0x7ff8000000000000ull;
  if (y == LA_EMPTY) y = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}

// rows k >= k0 with k % LT == threadIdx.x of a published column into dst, as
// they arrive.  False when a word did not come in ~2 s.
__device__ __forceinline__ bool poll_col(const cplx* src, cplx* dst, int k0, int m) {
  const long long t0 = clock64();
  for (int k = k0 + (((int)threadIdx.x - k0) & (LT - 1)); k < m; k += 4 * LT) {
    unsigned need = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (k + e * LT < m) need |= 1u << e;
    while (need) {
      unsigned long long x[4], y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (need >> e & 1u)
          asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                       : "=l"(x[e]), "=l"(y[e])
                       : "l"(src + k + e * LT)
                       : "memory");
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if ((need >> e & 1u) && x[e] != LA_EMPTY && y[e] != LA_EMPTY) {
          dst[k + e * LT] = mk(__longlong_as_double((long long)x[e]), __longlong_as_double((long long)y[e]));
          need &= ~(1u << e);
        }
      if (need && clock64() - t0 > PQMC_WAIT_CYCLES) return false;
    }
  }
  return true;
}

// two published words to dst, by a whole warp
__device__ __forceinline__ bool poll_pair(const cplx* src, cplx* dst) {
  const long long t0 = clock64();
  const int w = threadIdx.x & 1;
  for (;;) {
    unsigned long long x, y;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(src + w) : "memory");
    if (__all_sync(0xffffffffu, x != LA_EMPTY && y != LA_EMPTY)) {
      if ((threadIdx.x & 31) < 2) dst[w] = mk(__longlong_as_double((long long)x), __longlong_as_double((long long)y));
      return true;
    }
    if (__any_sync(0xffffffffu, clock64() - t0 > PQMC_WAIT_CYCLES)) return false;
  }
}

// own rows k >= k0 (k % LT == threadIdx.x) of a column whose words this thread
// has seen published (or published itself), asynchronously
__device__ __forceinline__ void fetch_col(const cplx* src, cplx* dst, int k0, int m) {
  for (int k = k0 + (((int)threadIdx.x - k0) & (LT - 1)); k < m; k += LT)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + k)),
                 "l"(src + k)
                 : "memory");
}
__device__ __forceinline__ void fetch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// sums of four doubles over the CTA, to every thread, with one barrier and 8
// FP64 additions in a row (lanes take over one of the four values as the
// tree narrows; 20 + 12 for four plain trees).  red: [2][4][4], the half
// alternates from call to call.  The order is the same in every CTA.
__device__ __forceinline__ void cta_sum4(double& a, double& b, double& c, double& d, double (*red)[4][4], int& half) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool up = lane & 16, u8 = lane & 8;
  double k0 = up ? c : a, k1 = up ? d : b;
  k0 += __shfl_xor_sync(full, up ? a : c, 16);
  k1 += __shfl_xor_sync(full, up ? b : d, 16);
  double k = u8 ? k1 : k0;
  k += __shfl_xor_sync(full, u8 ? k0 : k1, 8);
  k += __shfl_xor_sync(full, k, 4);
  k += __shfl_xor_sync(full, k, 2);
  k += __shfl_xor_sync(full, k, 1);
  if ((lane & 7) == 0) red[half][lane >> 3][warp] = k;
  __syncthreads();
  double r = red[half][(lane >> 2) & 3][lane & 3];
  r += __shfl_xor_sync(full, r, 1);
  r += __shfl_xor_sync(full, r, 2);
  a = __shfl_sync(full, r, 0);
  b = __shfl_sync(full, r, 4);
  c = __shfl_sync(full, r, 8);
  d = __shfl_sync(full, r, 12);
  half ^= 1;
}

// Sums over the CTA in two halves: the warps' shares to `red`, and after a
// barrier c (sum - beta a) with one real component per lane.
__device__ __forceinline__ void cta_part2(double a, double b, double (*red)[4]) {
  a = warp_sum(a);
  b = warp_sum(b);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = a;
    red[1][threadIdx.x >> 5] = b;
  }
}
__device__ __forceinline__ double cta_total(const double* r) { return (r[0] + r[1]) + (r[2] + r[3]); }
// component (lane >> 2) & 1 of value (lane >> 3) & (NV - 1): c (sum - beta a)
template <int NV, bool BETA>
__device__ __forceinline__ double cta_coef(const double (*red)[4], cplx c, double beta, cplx a) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, im = (lane >> 2) & 1;
  double r = cta_total(red[(lane >> 2) & (2 * NV - 1)]);
  if (BETA) r = fma(-beta, im ? a.y : a.x, r);
  const double o = __shfl_xor_sync(full, r, 4);
  return fma(flip_sign(c.y, !im), o, c.x * r);
}
__device__ __forceinline__ cplx cta_value(double f, int v) {
  return mk(__shfl_sync(0xffffffffu, f, 8 * v), __shfl_sync(0xffffffffu, f, 8 * v + 4));
}
// a sum over the CTA to every thread, one barrier
__device__ __forceinline__ double cta_sum1(double a, double (*red)[4]) {
  a = warp_sum(a);
  if ((threadIdx.x & 31) == 0) red[0][threadIdx.x >> 5] = a;
  __syncthreads();
  return cta_total(red[0]);
}

// the CTA's largest v >= 0 to every thread (two barriers)
__device__ __forceinline__ int cta_max(int v, int* red) {
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = max(max(red[0], red[1]), max(red[2], red[3]));
  __syncthreads();
  return v;
}

// zlarfg for the column [alpha; x], ss = sum |x|^2, kept as the vector
// u = [z; x], z = alpha - beta, that is z times zlarfg's v: then
// H^H = I + c u u^H with c = 1/(beta z), and tau = -z/beta.  One square root
// and one reciprocal, and two products fewer in a step's chain than with v.
// n2 = |alpha|^2 + ss in 2^-664 .. 2^530, or ss = 0.
struct Reflector {
  cplx z, c;
  double beta;
};
__device__ __forceinline__ Reflector reflector(cplx alpha, double ss, double n2) {
  Reflector h;
  // signs and zeros are looked at as bits: an FP64 comparison costs what a multiplication costs
  const int sign = ~__double2hiint(alpha.x) & (int)0x80000000;
  const double root = sqrt(n2);   // |beta|
  h.beta = __hiloint2double(__double2hiint(root) | sign, __double2loint(root));
  h.z = mk(alpha.x - h.beta, alpha.y);
  // 1 / (|beta| |z|^2); c = conj(z) / (beta |z|^2)
  const double r = 1.0 / (root * fma(h.z.x, h.z.x, h.z.y * h.z.y));
  const bool im = threadIdx.x & 1;   // a component per lane
  const double q = flip_sign((im ? h.z.y : h.z.x) * r, im != (sign != 0));
  h.c = mk(__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1));
  if (__double_as_longlong(ss) == 0 && (__double_as_longlong(alpha.y) << 1) == 0) {   // nothing below the diagonal: H = I
    h.z = h.c = mk(0.0);
    h.beta = alpha.x;
  }
  return h;
}

// ---------------------------------------------------------------------------
// Columns j = b, b + G, ... of Q = H_0 ... H_(n-1), H_i = I + c_i u_i u_i^H, by
// the triangular factor of their product: H_0 ... H_(n-1) = I + U T U^H with
// T^-1 = diag(1/c_i) - (strictly upper part of U^H U) (T. Joffrain, T. M. Low,
// E. S. Quintana-Orti, R. van de Geijn, F. G. Van Zee, Accumulating Householder
// transformations, revisited, ACM TOMS 32, 2006).  So column j is
// e_j + U y, T^-1 y = U^H e_j, in three steps: the products c_i u_i^H u_j,
// published for the others; the triangular system, one unknown a step; and U y.
//
// Applying the reflectors to the column one after the other is the same number
// of multiply-adds, but each waits for a sum over the CTA: 4.4k cycles a
// reflector at 288 rows.  Here only the triangular system is a chain, of 1.1k
// cycles a step, and FP64 issue and the loops' own instructions bound the rest
// (76k, 153k and 159k cycles for the products, the system and U y of the last
// column at 288 x 144; the whole factorisation took 617 us with this and 733
// without, 1054 and 1158 at 392 x 196; 628 and 1072 with sqrt(), a division and
// the sums of UT_SUM).  One or two columns per CTA.  `gs` (n x n, column k holds
// the products of column k) starts out LA_EMPTY like `pub`.
constexpr int UT_SUM = 16;   // terms of U y in a sum of their own: one after another they gave 1.06 times the error
__device__ __forceinline__ void form_q_ut(int m, int n, int b, int G, int nl, cplx* cols, cplx* pub, cplx* xs,
                                          const cplx* s_z, const cplx* s_c, const double* s_up, cplx* s_y, bool apart,
                                          int* s_fail) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  cplx* gs = pub + (size_t)m * n;
  auto one = [](double up) { return __double2hiint(up) == 0x3ff00000; };
  for (int l = 0; l < nl; ++l)
    if (const int j = b + l * G; tid == (j & (LT - 1))) cols[(size_t)l * m + j] = s_z[j];   // u_j
  __syncthreads();
  // c_i u_i^H u_j: a lane per i, a quarter of the rows per warp
  for (int l = 0; l < nl; ++l) {
    const int j = b + l * G, len = (m - j + 3) / 4, k0 = j + warp * len, k1 = min(m, k0 + len);
    const cplx* u = cols + (size_t)l * m;
    for (int i0 = 0; i0 < j; i0 += 32) {
      const int i = i0 + lane;
      const double2* p = reinterpret_cast<const double2*>(pub) + (size_t)m * min(i, j - 1);
      constexpr int AHEAD = 8;
      double2 v[AHEAD];
#pragma unroll
      for (int q = 0; q < AHEAD; ++q) v[q] = k0 + q < k1 ? p[k0 + q] : make_double2(0.0, 0.0);
      cplx acc = mk(0.0);
      for (int k = k0; k < k1; k += AHEAD)
#pragma unroll
        for (int q = 0; q < AHEAD; ++q)
          if (k + q < k1) {
            const cplx x = mk(v[q].x, -v[q].y);
            v[q] = k + q + AHEAD < k1 ? p[k + q + AHEAD] : make_double2(0.0, 0.0);
            acc = cfma(x, u[k + q], acc);
          }
      if (i < j) xs[(size_t)warp * n + i] = acc;
    }
    __syncthreads();
    for (int i = tid; i < j; i += LT) {
      cplx g = cadd(cadd(xs[i], xs[(size_t)n + i]), cadd(xs[2 * (size_t)n + i], xs[3 * (size_t)n + i]));
      if (!one(s_up[i])) g = cscale(g, s_up[i]);
      publish(gs + (size_t)n * j + i, cmul(cconj(s_c[i]), g));
    }
    __syncthreads();   // the shares are read
  }
  // c_i (U^H e_j)_i, then from the last unknown to the first
  const int jlast = b + (nl - 1) * G;
  for (int l = 0; l < nl; ++l) {
    const int j = b + l * G;
    for (int i = tid; i <= j; i += LT) {
      cplx v = i < j ? pub[(size_t)m * i + j] : s_z[j];
      if (i < j && !one(s_up[i])) v = cscale(v, s_up[i]);
      s_y[(size_t)l * n + i] = cmul(cconj(s_c[i]), cconj(v));
    }
  }
  auto fetch_g = [&](int k) {
    if (k > 0)
      for (int i = tid; i < k; i += LT)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(xs + (size_t)(k & 3) * m + i)),
                     "l"(gs + (size_t)n * k + i)
                     : "memory");
    fetch_commit();
  };
  for (int q = 0; q < 4; ++q) fetch_g(jlast - q);
  bool ok = true;
  const long long t0 = clock64();
  auto product = [&](int k, int i) {   // c_i u_i^H u_k
    cplx v = xs[(size_t)(k & 3) * m + i];
    while ((unsigned long long)__double_as_longlong(v.x) == LA_EMPTY || (unsigned long long)__double_as_longlong(v.y) == LA_EMPTY) {
      if (!ok || clock64() - t0 > PQMC_WAIT_CYCLES) {
        ok = false;
        break;
      }
      unsigned long long x, y;
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(gs + (size_t)n * k + i) : "memory");
      v = mk(__longlong_as_double((long long)x), __longlong_as_double((long long)y));
    }
    return v;
  };
  // Two unknowns a step, k and k - 1, every thread forming the second for
  // itself; the thread that holds it stores it when nobody reads it any more.
  // The number of columns is a constant of the loop bodies: a multiply-add
  // that a predicate switches off takes its 64 cycles all the same.
  cplx late_y[2];
  int late_k = -1, late_l = 0;
  auto store_late = [&]() {
    if (late_k >= 0)
      for (int l = late_l; l < nl; ++l) s_y[(size_t)l * n + late_k] = late_y[l - late_l];
    late_k = -1;
  };
  auto step = [&](auto cols_on, int k, int la) {
    constexpr int NL = decltype(cols_on)::value;
    const cplx d = product(k, k - 1);
    cplx* yb = s_y + (size_t)la * n;
    cplx y0[NL], y1[NL];
#pragma unroll
    for (int q = 0; q < NL; ++q) {
      y0[q] = b + (la + q) * G >= k ? yb[q * n + k] : mk(0.0);
      y1[q] = cfma(d, y0[q], yb[q * n + k - 1]);
    }
    for (int i = tid; i < k - 1; i += LT) {
      const cplx v0 = product(k, i), v1 = product(k - 1, i);
#pragma unroll
      for (int q = 0; q < NL; ++q) yb[q * n + i] = cfma(v1, y1[q], cfma(v0, y0[q], yb[q * n + i]));
    }
    if (tid == ((k - 1) & (LT - 1))) {
      late_k = k - 1;
      late_l = la;
#pragma unroll
      for (int q = 0; q < NL; ++q) late_y[q] = y1[q];
    }
  };
  for (int k = jlast; k > 0; k -= 2) {
    fetch_wait<2>();
    __syncthreads();   // unknowns k and k - 1 but for the product of the two
    store_late();
    const int la = nl > 1 && b < k - 1 ? 1 : 0;   // columns that have unknown k - 1
    if (nl - la == 2) step(std::integral_constant<int, 2>(), k, la);
    else step(std::integral_constant<int, 1>(), k, la);
    fetch_g(k - 4);
    fetch_g(k - 5);
  }
  __syncthreads();
  store_late();
  fetch_wait<0>();
  if (!ok) *s_fail = 1;
  __syncthreads();
  // e_j + U y, own rows; the terms in sums of UT_SUM where there is room
  cplx* sums = apart ? s_y + (size_t)nl * n : cols;
  auto flush = [&]() {
    for (int l = 0; l < nl; ++l)
      for (int k = tid; k < m; k += LT) {
        const size_t e = (size_t)l * m + k;
        cols[e] = cadd(cols[e], sums[e]);
        sums[e] = mk(0.0);
      }
  };
  for (int l = 0; l < nl; ++l)
    for (int k = tid; k < m; k += LT) {
      sums[(size_t)l * m + k] = mk(0.0);
      cols[(size_t)l * m + k] = mk(k == b + l * G ? 1.0 : 0.0);
    }
  for (int q = 0; q < 3; ++q) {
    if (q <= jlast) fetch_col(pub + (size_t)m * q, xs + (size_t)q * m, q, m);
    fetch_commit();
  }
  for (int i = 0; i <= jlast; ++i) {
    fetch_wait<2>();
    cplx* x = xs + (size_t)(i & 3) * m;
    const int k0 = i + ((tid - i) & (LT - 1));
    if (!one(s_up[i]))
      for (int k = k0; k < m; k += LT) x[k] = cscale(x[k], s_up[i]);
    if (tid == (i & (LT - 1))) x[i] = s_z[i];
    if (nl == 2 && i <= b) {
      const cplx ya = s_y[i], yb = s_y[(size_t)n + i];
      for (int k = k0; k < m; k += LT) {
        const cplx v = x[k];
        sums[k] = cfma(v, ya, sums[k]);
        sums[(size_t)m + k] = cfma(v, yb, sums[(size_t)m + k]);
      }
    } else {
      const cplx y = s_y[(size_t)(nl - 1) * n + i];
      cplx* c = sums + (size_t)(nl - 1) * m;
      for (int k = k0; k < m; k += LT) c[k] = cfma(x[k], y, c[k]);
    }
    if (apart && i % UT_SUM == UT_SUM - 1) flush();
    if (i + 3 <= jlast) fetch_col(pub + (size_t)m * (i + 3), xs + (size_t)((i + 3) & 3) * m, i + 3, m);
    fetch_commit();
  }
  if (apart) flush();
  fetch_wait<0>();
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Householder QR in place with Q formed (zgeqr2 + zung2r).  A is m x n
// (lda = m), m >= n; d receives diag(R) (real in the LAPACK convention).
// Matches zqdr (src/mod_matrixlib.f90:323-334) with the unit-diagonal R
// discarded as the reference does for the hot path.  With Rout the upper
// triangle of R (n x n, diagonal = d) is written too, and with lndet
// ln det Q = sum over the reflectors of ln det(I - tau v v^H)
// = ln(-z / conj(z)) (a phase; 0 for z = 0).
//
// What is published is the raw column x (rows >= i after the reflectors
// before it), and by its CTA alone, as soon as it has the norm, beta and c.
// The others form x^H a of their next column meanwhile: with u = x - beta e_i,
// u^H a = x^H a - beta a_i, so the reflector is not needed before the last
// three instructions of the coefficient, and the chain of a step is two
// overlapping halves of one column's passage.  The next column comes first
// and is published row by row.  (Every CTA with the norm and reflector of its
// own, 2 of 6 multiply-adds a row and 2.1k cycles of root and division in the
// chain: 875 us at 288 x 144 and 1.35 ms at 392 x 196; 733 us and 1.16 ms so,
// with Q by reflectors.)  Q's columns need only reflectors
// that their CTA has already seen, so their formation starts without waiting
// for the rest.  Bound by that chain (n steps) and, in a step, by the FP64
// pipe.  A column whose entries pass 2^+-256 is held times a power of two
// (exact), and a remainder whose squares could vanish is scaled up before its
// norm is taken, as LAPACK's dznrm2 avoids overflow (the graded
// finite-temperature strings pass 1e154).
//
// Rows 0 .. QR_SELF - 1 of a later column are not published; they take
// QR_COPIES copies of {c, (beta, up)}, so that not every CTA polls one sector.
//
// dynamic shared memory: nst columns of the ring, z and c of n reflectors, the local columns' exponents, the local columns if `in_smem`
// (else they stay in A).  Four CTAs an SM: the compiler takes 80 registers and
// spills without the bound (12x12: 16.29 ms a start, 15.96 with it).
constexpr int QR_COPIES = 4, QR_SELF = 2 * QR_COPIES;
__global__ void __launch_bounds__(LT, 4) k_house_qr(int m, int n, cplx* A, cplx* d, cplx* Rout, cplx* lndet, cplx* pub,
                                                 int in_smem, int nst, int ut, int* err) {
  extern __shared__ cplx qr_dyn[];
  __shared__ double red[2][4][4];
  __shared__ int redi[4];
  __shared__ cplx s_al[2], s_aj[2], s_sc[2][2];
  __shared__ int s_fail;
  const int tid = threadIdx.x, b = blockIdx.x, G = gridDim.x;
  const int nl = (n - b + G - 1) / G;   // local columns b, b + G, ...
  cplx* xs = qr_dyn;
  cplx* s_z = xs + (size_t)nst * m;
  cplx* s_c = s_z + n;
  double* s_up = reinterpret_cast<double*>(s_c + n);   // power of two on x (1 but for vanishing remainders)
  int* s_exp = reinterpret_cast<int*>(s_up + 2 * ((n + 1) / 2));
  cplx* s_y = s_c + n + (n + 1) / 2 + (nl + 3) / 4;   // ut: [nl][n], and with 2 the sums of U y, [nl][m]
  cplx* cols = s_y + (ut ? (size_t)nl * n : 0) + (ut == 2 ? (size_t)nl * m : 0);
  auto col = [&](int l) { return in_smem ? cols + (size_t)l * m : A + (size_t)m * (b + (size_t)l * G); };
  int half = 0;
  if (tid == 0) s_fail = 0;
  for (int l = 0; l < nl; ++l) {
    const cplx* src = A + (size_t)m * (b + (size_t)l * G);
    cplx* c = col(l);
    int e = 0;
    for (int k = tid; k < m; k += LT) {
      const cplx v = src[k];
      e = max(e, top_exp(v));
      if (in_smem) c[k] = v;
    }
    e = cta_max(e, redi) - 1023;
    e = (e < -256 || e > 256) ? min(max(e, -1000), 1000) : 0;
    if (e)
      for (int k = tid; k < m; k += LT) c[k] = cscale(c[k], pow2i(-e));
    if (tid == 0) s_exp[l] = e;
  }
  __syncthreads();
  if (b == 0)
    for (int k = tid; k < m; k += LT) publish(pub + k, col(0)[k]);
  int li = 0, jown = b;   // the next local column, local and global
  for (int i = 0; i < n; ++i) {
    const bool own = i == jown;
    const int l0 = own ? li + 1 : li;   // first local column right of i
    cplx* x = own ? col(li) : xs;
    if (!own && !poll_col(pub + (size_t)m * i, x, i, m)) s_fail = 1;
    const bool row_i = tid == (i & (LT - 1));
    cplx* c0 = l0 < nl ? col(l0) : nullptr;
    // its CTA forms the reflector, and every CTA where the published column has no free rows for it
    const bool self = own || i < QR_SELF;
    cplx alpha = mk(0.0), c = mk(0.0);
    double beta = 0.0, up_x = 1.0, beta_x = 0.0;
    if (self) {
      double ss = 0.0;
      for (int k = i + 1 + ((tid - i - 1) & (LT - 1)); k < m; k += LT) {
        const cplx v = x[k];
        ss = fma(v.x, v.x, fma(v.y, v.y, ss));
      }
      const int h0 = half;
      half ^= 1;
      if (row_i) s_al[h0] = x[i];
      ss = cta_sum1(ss, red[h0]);
      if (s_fail) {
        if (tid == 0) atomicExch(err, PQMC_ERR_TIMEOUT);
        return;
      }
      alpha = s_al[h0];
      double n2 = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, ss));
      int up = 0;
      if (__double2hiint(n2) < (1023 - 664) << 20) {   // below 2^-664 squares may have vanished: scale up
        int e = 0;
        for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) e = max(e, top_exp(x[k]));
        e = cta_max(e, redi);
        up = e ? min(1023 - e, 1000) : 1000;
        up_x = pow2i(up);
        ss = 0.0;
        for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) {
          const cplx v = cscale(x[k], up_x);
          x[k] = v;
          if (k > i) ss += cabs2(v);
        }
        ss = cta_sum1(ss, red[half]);
        half ^= 1;
        alpha = cscale(alpha, up_x);
        n2 = ss + cabs2(alpha);
      }
      const Reflector h = reflector(alpha, ss, n2);
      c = h.c;
      beta = h.beta;
      beta_x = beta * pow2i(-up);
      if (own && i >= QR_SELF && tid < 2 * QR_COPIES) publish(pub + (size_t)m * i + tid, tid & 1 ? mk(beta, up_x) : c);
    }
    cplx f = mk(0.0);
    if (c0) {
      cplx w = mk(0.0);
      for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) w = cfma(cconj(x[k]), c0[k], w);
      int h0 = half;
      half ^= 1;
      if (row_i) {
        if (!self) s_al[h0] = x[i];
        s_aj[h0] = c0[i];
      }
      cta_part2(w.x, w.y, red[h0]);
      if (!self && tid < 32 && !poll_pair(pub + (size_t)m * i + 2 * (b & (QR_COPIES - 1)), s_sc[h0])) s_fail = 1;
      __syncthreads();
      if (s_fail) {
        if (tid == 0) atomicExch(err, PQMC_ERR_TIMEOUT);
        return;
      }
      const cplx aj = s_aj[h0];
      if (!self) {
        alpha = s_al[h0];
        c = s_sc[h0][0];
        beta = s_sc[h0][1].x;
        up_x = s_sc[h0][1].y;
        if (__double2hiint(up_x) != 0x3ff00000) {   // not 1: the dot product of the scaled column
          w = mk(0.0);
          for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) {
            const cplx v = cscale(x[k], up_x);
            x[k] = v;
            w = cfma(cconj(v), c0[k], w);
          }
          alpha = cscale(alpha, up_x);
          h0 = half;
          half ^= 1;
          cta_part2(w.x, w.y, red[h0]);
          __syncthreads();
        }
      }
      f = cta_value(cta_coef<1, true>(red[h0], c, beta, aj), 0);   // c u^H a
    }
    if (row_i) {
      const cplx z = mk(alpha.x - beta, alpha.y);
      x[i] = z;   // u
      s_z[i] = z;
      s_c[i] = c;
      s_up[i] = up_x;
    }
    // H_i^H on the local columns right of i, the next column first
    for (int l = l0; l < nl; ++l) {
      cplx* cl = col(l);
      if (l != l0) {
        cplx w = mk(0.0);
        for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) w = cfma(cconj(x[k]), cl[k], w);
        cta_part2(w.x, w.y, red[half]);
        __syncthreads();
        f = cta_value(cta_coef<1, false>(red[half], c, 0.0, mk(0.0)), 0);
        half ^= 1;
      }
      const bool next = l == l0 && (own ? jown + G : jown) == i + 1;
      for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) {
        const cplx v = cfma(x[k], f, cl[k]);
        cl[k] = v;
        if (next && k > i) publish(pub + (size_t)m * (i + 1) + k, v);
      }
    }
    if (own) {   // diag(R), R
      const int e = s_exp[li];
      const double up = pow2i(e);
      if (tid == 0) d[i] = mk(beta_x * up);
      if (Rout)
        for (int k = tid; k < n; k += LT)
          Rout[k + (size_t)n * i] = k < i ? cscale(col(li)[k], up) : k == i ? mk(beta_x * up) : mk(0.0);
      if (l0 >= nl) break;
      ++li;
      jown += G;
    }
  }
  __threadfence();
  __syncthreads();
  if (lndet && (n - 1) % G == b) {
    double ph = 0.0, z1 = 0.0, z2 = 0.0, z3 = 0.0;
    for (int i = tid; i < n; i += LT) {
      const cplx t = s_z[i];
      if (t.x != 0.0 || t.y != 0.0) {
        const cplx z = cdiv(cneg(t), cconj(t));
        ph += atan2(z.y, z.x);
      }
    }
    cta_sum4(ph, z1, z2, z3, red, half);
    if (tid == 0) lndet[0] = mk(0.0, ph);
  }
  if (ut) {
    form_q_ut(m, n, b, G, nl, cols, pub, xs, s_z, s_c, s_up, s_y, ut == 2, &s_fail);
    if (s_fail) {   // read after the barrier that ends form_q_ut
      if (tid == 0) atomicExch(err, PQMC_ERR_TIMEOUT);
      return;
    }
    for (int l = 0; l < nl; ++l) {
      cplx* dst = A + (size_t)m * (b + (size_t)l * G);
      for (int k = tid; k < m; k += LT) dst[k] = col(l)[k];
    }
    return;
  }
  // zung2r: column j of Q = H_1 ... H_j e_j, the local columns together; the
  // published columns come back through the ring, nst - 1 steps ahead
  const int jlast = b + (nl - 1) * G, ring = nst - 1;   // nst is 2 or 4
  li = nl - 1;
  jown = jlast;
  for (int u = 1; u < nst; ++u) {
    const int i = jlast - u;
    if (i >= 0) fetch_col(pub + (size_t)m * i, xs + (size_t)(i & ring) * m, i, m);
    fetch_commit();
  }
  for (int i = jlast; i >= 0; --i) {
    const cplx z = s_z[i], cc = cconj(s_c[i]);   // H_i = I + conj(c) u u^H
    const double up_x = s_up[i];
    const bool row_i = tid == (i & (LT - 1));
    const int ls = li + 1;
    if (i != jlast) {
      if (nst == 4) fetch_wait<2>();
      else fetch_wait<0>();
      cplx* x = xs + (size_t)(i & ring) * m;
      if (up_x != 1.0)
        for (int k = i + 1 + ((tid - i - 1) & (LT - 1)); k < m; k += LT) x[k] = cscale(x[k], up_x);
      if (row_i) x[i] = z;   // u
      auto apply = [&](auto cols_on, int l) {
        constexpr bool two = decltype(cols_on)::value == 2;
        cplx* c0 = col(l);
        cplx* c1 = two ? col(l + 1) : c0;
        cplx w0 = mk(0.0), w1 = mk(0.0), f0, f1 = mk(0.0);
        for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) {
          const cplx v = cconj(x[k]);
          w0 = cfma(v, c0[k], w0);
          if (two) w1 = cfma(v, c1[k], w1);
        }
        cta_part2(w0.x, w0.y, red[half]);
        if (two) cta_part2(w1.x, w1.y, red[half] + 2);
        __syncthreads();
        const double f = cta_coef<two ? 2 : 1, false>(red[half], cc, 0.0, mk(0.0));
        f0 = cta_value(f, 0);
        if (two) f1 = cta_value(f, 1);
        half ^= 1;
        for (int k = i + ((tid - i) & (LT - 1)); k < m; k += LT) {
          c0[k] = cfma(x[k], f0, c0[k]);
          if (two) c1[k] = cfma(x[k], f1, c1[k]);
        }
      };
      for (int l = ls; l < nl; l += 2) {
        if (l + 1 < nl) apply(std::integral_constant<int, 2>(), l);
        else apply(std::integral_constant<int, 1>(), l);
      }
      const int in = i - (nst - 1);
      if (in >= 0) fetch_col(pub + (size_t)m * in, xs + (size_t)(in & ring) * m, in, m);
      fetch_commit();
    }
    if (i == jown) {   // H_i e_i
      cplx* c = col(li--);
      jown -= G;
      const cplx t = cmul(cc, cconj(z));   // the column has its power of two already
      for (int k = tid; k < m; k += LT) c[k] = k > i ? cmul(t, c[k]) : k == i ? cfma(t, z, mk(1.0)) : mk(0.0);
    }
  }
  if (in_smem)
    for (int l = 0; l < nl; ++l) {
      cplx* dst = A + (size_t)m * (b + (size_t)l * G);
      for (int k = tid; k < m; k += LT) dst[k] = col(l)[k];
    }
}

// ---------------------------------------------------------------------------
// LU with partial pivoting (zgetf2's pivots: largest |re| + |im|, ties to the
// lowest row) of A (n x n, lda = n, destroyed) and A X = B solved in place on
// B (n x nrhs), in one pass: the right-hand sides are further columns of the
// elimination, then each CTA substitutes back on its own ones.  Rows are not
// moved: a row leaves when it becomes a pivot row, so the row every thread
// reads in a step is one nobody writes.  diag: the pivots in order, perm: the
// rows they came from, info[0]: first zero pivot (1-based) or 0.
// Bound like k_house_qr by the chain of a step: poll, the pivot search (on
// the bits, as integers), one reciprocal, the next column's update.
// A step's multipliers -(c[p] / pivot) are formed for 16 columns at a time,
// a real component per lane (two FP64 instructions instead of four a column):
// 196 columns and 392 right-hand sides took 905 us with them in every lane,
// 820 so, and 880 to 950 with a division for the reciprocal and the sums below.
//
// A right-hand side's terms are summed LU_SUM at a time apart from its
// entries (`sums`) and added to them then, in both passes: one term after
// another each rounds at the entry's size, and G came out with twice the error
// of dot products over 32 lanes (1.2e-15 and 6.4e-16 at n = 100; 6.5e-16 so).
// Columns of A keep the plain order, which the pivots and the chain depend on.
// `nsum` columns of sums: where they are one for each of a CTA's right-hand
// sides (`apart`) both passes use them; where shared memory has room for fewer
// the elimination keeps the plain order and the substitution takes nsum
// right-hand sides at a time (at n = 100: 7.4e-16).
constexpr int LU_SUM = 16;
__global__ void __launch_bounds__(LT) k_lu_solve(int n, cplx* A, int nrhs, cplx* B, int ldb, cplx* diag, int* perm,
                                                 int* info, cplx* pub, int in_smem, int nst, int nsum, int apart, int* err) {
  extern __shared__ cplx lu_dyn[];
  __shared__ unsigned long long s_key[2][4];
  __shared__ int s_row[2][4];
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = blockIdx.x, G = gridDim.x, T = n + nrhs;
  const int nl = (T - b + G - 1) / G;
  cplx* xs = lu_dyn;
  cplx* s_rec = xs + (size_t)nst * n;          // reciprocals of the pivots
  int* s_prow = reinterpret_cast<int*>(s_rec + n);
  int* s_ord = s_prow + n;                     // step at which a row became the pivot row
  cplx* sums = s_rec + n + (2 * n + 3) / 4;    // [nsum][n]
  const int lr = b >= n ? 0 : min(nl, (n - b + G - 1) / G);   // first local right-hand side
  cplx* cols = sums + (size_t)nsum * n;
  auto gcol = [&](int l) {
    const size_t j = b + (size_t)l * G;
    return j < (size_t)n ? A + (size_t)n * j : B + (size_t)ldb * (j - n);
  };
  auto col = [&](int l) { return in_smem ? cols + (size_t)l * n : gcol(l); };
  auto sum = [&](int l) { return sums + (size_t)(l - lr) * n; };   // apart
  // own rows' sums of right-hand side l into its entries, but row p, which others read
  auto flush = [&](int l, int p) {
    cplx *c = col(l), *a = sum(l);
    for (int k = tid; k < n; k += LT)
      if (k != p) {
        c[k] = cadd(c[k], a[k]);
        a[k] = mk(0.0);
      }
  };
  if (tid == 0) s_fail = 0;
  for (int k = tid; k < n; k += LT) s_ord[k] = n;
  if (apart)
    for (int k = tid; k < (nl - lr) * n; k += LT) sums[k] = mk(0.0);
  if (in_smem)
    for (int l = 0; l < nl; ++l)
      for (int k = tid; k < n; k += LT) col(l)[k] = gcol(l)[k];
  __syncthreads();
  if (b == 0)
    for (int k = tid; k < n; k += LT) publish(pub + k, col(0)[k]);
  const bool last_owner = (n - 1) % G == b;
  int first_zero = 0;
  int li = 0, jown = b;   // the next local column, local and global
  for (int j = 0; j < n; ++j) {
    const bool own = j == jown;
    const int l0 = own ? li + 1 : li;
    cplx* x = xs + (size_t)(j & 1) * n;   // two in turn: every thread reads the pivot's entry
    if (own) {
      for (int k = tid; k < n; k += LT) x[k] = col(li)[k];
    } else if (!poll_col(pub + (size_t)n * j, x, 0, n)) {
      s_fail = 1;
    }
    // pivot: the largest |re| + |im| of the rows that are left
    unsigned long long key = 0;
    int row = 0x7fffffff;
    for (int k = tid; k < n; k += LT) {
      if (s_ord[k] < n) continue;
      const unsigned long long q = (unsigned long long)__double_as_longlong(fabs(x[k].x) + fabs(x[k].y));
      if (row == 0x7fffffff || q > key) { key = q; row = k; }
    }
    {
      const unsigned full = 0xffffffffu, hi = (unsigned)(key >> 32);
      const unsigned mh = __reduce_max_sync(full, row != 0x7fffffff ? hi : 0u);
      const bool ch = row != 0x7fffffff && hi == mh;
      const unsigned ml = __reduce_max_sync(full, ch ? (unsigned)key : 0u);
      const int mr = __reduce_min_sync(full, ch && (unsigned)key == ml ? row : 0x7fffffff);
      if (lane == 0) {
        s_key[j & 1][warp] = (unsigned long long)mh << 32 | ml;
        s_row[j & 1][warp] = mr;
      }
    }
    __syncthreads();
    if (s_fail) {
      if (tid == 0) atomicExch(err, PQMC_ERR_TIMEOUT);
      return;
    }
    int p = 0x7fffffff;
    unsigned long long pk = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned long long k2 = s_key[j & 1][q];
      const int r2 = s_row[j & 1][q];
      if (r2 != 0x7fffffff && (p == 0x7fffffff || k2 > pk || (k2 == pk && r2 < p))) { p = r2; pk = k2; }
    }
    const cplx piv = x[p];
    // 1/piv, scaled by a power of two where its square could leave the range
    cplx rec = mk(0.0);
    if (((__double_as_longlong(piv.x) | __double_as_longlong(piv.y)) << 1) != 0) {
      const int e = min(max(top_exp(piv) - 1023, -1000), 1000);
      if (e > -400 && e < 400) {
        const double r = 1.0 / fma(piv.x, piv.x, piv.y * piv.y);
        rec = mk(piv.x * r, -piv.y * r);
      } else {
        const double s = pow2i(-e);
        const cplx q = cscale(piv, s);
        const double r = 1.0 / fma(q.x, q.x, q.y * q.y);
        rec = mk(q.x * r * s, -q.y * r * s);   // s last: s r can leave the range where the product does not
      }
    } else if (!first_zero) {
      first_zero = j + 1;
    }
    if (tid == (p & (LT - 1))) s_ord[p] = j;   // only this thread looks at this row's step
    if (tid == 0) {
      s_rec[j] = rec;
      s_prow[j] = p;
      if (last_owner) {
        diag[j] = piv;
        perm[j] = p;
      }
    }
    if (apart && j && j % LU_SUM == 0)
      for (int l = lr; l < nl; ++l) flush(l, p);
    double fl = 0.0;   // -(c[p] / piv) of 16 columns at a time, a real component per lane
    for (int l = l0; l < nl; ++l) {
      cplx* c = apart && l >= lr ? sum(l) : col(l);
      const int lq = (l - l0) & 15;
      if (lq == 0) {
        const bool im = lane & 1;
        const int lv = min(l + (lane >> 1), nl - 1);
        cplx v = col(lv)[p];
        if (apart && lv >= lr) v = cadd(v, sum(lv)[p]);
        fl = fma(flip_sign(rec.y, im), im ? v.x : v.y, -(rec.x * (im ? v.y : v.x)));
      }
      const cplx f = mk(__shfl_sync(0xffffffffu, fl, 2 * lq), __shfl_sync(0xffffffffu, fl, 2 * lq + 1));
      const bool next = l == l0 && (own ? jown + G : jown) == j + 1 && j + 1 < n;
      for (int k = tid; k < n; k += LT) {
        if (s_ord[k] == n) c[k] = cfma(x[k], f, c[k]);
        if (next) publish(pub + (size_t)n * (j + 1) + k, c[k]);
      }
    }
    if (own) {
      if (l0 >= nl) break;
      ++li;
      jown += G;
    }
  }
  if (last_owner && tid == 0) info[0] = first_zero;
  // ---- back substitution: x_j = y(p_j) / u_jj, y(p_k) -= U(p_k, j) x_j -----
  if (lr >= nl) return;
  __threadfence();
  __syncthreads();
  if (apart)
    for (int l = lr; l < nl; ++l) flush(l, -1);
  for (int r0 = lr; r0 < nl; r0 += nsum) {
    const int nb = min(nsum, nl - r0);
    if (!apart)
      for (int l = 0; l < nb; ++l)
        for (int k = tid; k < n; k += LT) sums[(size_t)l * n + k] = mk(0.0);
    for (int u = 0; u < nst - 1; ++u) {
      const int j = n - 1 - u;
      if (j >= 0) fetch_col(pub + (size_t)n * j, xs + (size_t)(j & (nst - 1)) * n, 0, n);
      fetch_commit();
    }
    cplx done = mk(0.0);   // !in_smem: the last unknown, kept in the place of its row's sum
    for (int j = n - 1; j >= 0; --j) {
      if (nst == 4) fetch_wait<2>();
      else fetch_wait<0>();
      const cplx* u = xs + (size_t)(j & (nst - 1)) * n;
      const int p = s_prow[j], pn = j > 0 ? s_prow[j - 1] : -1;
      const cplx rec = s_rec[j];
      __syncthreads();   // the rows of step j + 1 are in
      if (!in_smem && tid == 0 && j < n - 1) sums[s_prow[j + 1]] = done;
      if (j % LU_SUM == LU_SUM - 1)
        for (int l = r0; l < r0 + nb; ++l) {
          cplx *y = col(l), *a = sums + (size_t)(l - r0) * n;
          for (int k = tid; k < n; k += LT)
            if (s_ord[k] < j) {
              y[k] = cadd(y[k], a[k]);
              a[k] = mk(0.0);
            }
        }
      double xl = 0.0;   // y[p] / u_jj of 16 columns at a time, a real component per lane
      for (int l = r0; l < r0 + nb; ++l) {
        cplx *y = col(l), *a = sums + (size_t)(l - r0) * n;
        const int lq = (l - r0) & 15;
        if (lq == 0) {
          const bool im = lane & 1;
          const cplx v = col(min(l + (lane >> 1), r0 + nb - 1))[p];
          xl = fma(flip_sign(rec.y, !im), im ? v.x : v.y, rec.x * (im ? v.y : v.x));
        }
        const cplx xj = mk(__shfl_sync(0xffffffffu, xl, 2 * lq), __shfl_sync(0xffffffffu, xl, 2 * lq + 1));
        const cplx f = cneg(xj);
        for (int k = tid; k < n; k += LT)
          if (s_ord[k] < j) {
            cplx t = a[k];
            if (k == pn) t = cadd(t, y[k]);   // the row that the next step reads, complete
            *(k == pn ? y + k : a + k) = cfma(u[k], f, t);
          }
        if (in_smem && tid == 0) B[j + (size_t)ldb * (b + (size_t)l * G - n)] = xj;
        done = xj;
      }
      const int jn = j - (nst - 1);
      if (jn >= 0) fetch_col(pub + (size_t)n * jn, xs + (size_t)(jn & (nst - 1)) * n, 0, n);
      fetch_commit();
    }
    if (!in_smem) {
      __syncthreads();
      if (tid == 0) sums[s_prow[0]] = done;
      __syncthreads();
      for (int k = tid; k < n; k += LT) gcol(r0)[k] = sums[s_prow[k]];
      __syncthreads();
    }
  }
}

// log det from the pivots: the reference forms the product of the diagonal
// (zdet_lapack, src/mod_matrixlib.f90:624-653) and takes its log; here the
// sum of logs, one pivot per thread (the product alone was a chain of n
// complex multiplications with a log each: 624 us at n = 196), taken back to
// the principal branch of that product where it stays in the double range.
__global__ void __launch_bounds__(LT) k_lu_logdet(int n, const cplx* diag, const int* perm, cplx* out) {
  __shared__ double red[2][4][4];
  int half = 0;
  double re = 0.0, im = 0.0, odd = 0.0, zero = 0.0;
  for (int i = threadIdx.x; i < n; i += LT) {
    const cplx l = clog_(diag[i]);
    re += l.x;
    im += l.y;
    int inv = 0;   // parity of the permutation
    const int pi = perm[i];
    for (int k = 0; k < i; ++k) inv ^= perm[k] > pi;
    odd += inv;
  }
  cta_sum4(re, im, odd, zero, red, half);
  if (threadIdx.x != 0) return;
  const double pi = 3.14159265358979323846;
  if (fmod(odd, 2.0) != 0.0) im += pi;
  if (fabs(re) < 667.0) im = remainder(im, 2.0 * pi);   // |det| in 1e-290 .. 1e290
  out[0] = mk(re, im);
}

int coop_grid(const void* fn, int threads, int want, size_t smem) {
  int dev = 0, nsm = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem);
  int cap = nsm * (per > 0 ? per : 1);
  if (want > cap) want = cap;
  if (want > nsm) want = nsm;
  return want < 1 ? 1 : want;
}

// Grid and shared memory of a column pipeline over `ncol` columns of `len`
// rows.  Two CTAs per SM while their columns fit in half its shared memory
// (at Ns = 392, nelec = 196 a CTA has one column of the QR), one while they
// fit in all of it, and past that the columns stay in global memory: the
// first of the shapes `from` .. `to` - 1 that fits (grid 0: none).
// `fixed`(grid, columns per CTA, in shared memory, room): complex entries
// besides the ring and the columns, of `room` that are left.
struct PipeShape {
  int grid, in_smem, nst;
  size_t smem;
};
enum { PIPE_ONE, PIPE_TWO, PIPE_TWO_SHORT, PIPE_ALL, PIPE_ALL_SHORT, PIPE_GLOBAL, PIPE_GLOBAL_SHORT, PIPE_END };
template <typename FIXED>
static int pipe_shape(const void* fn, int ncol, int len, int from, int to, FIXED fixed, PipeShape* out) {
  int dev = 0, nsm = 0;
  PQMC_CUDA(cudaGetDevice(&dev));
  PQMC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const struct { int per, nst, in; size_t lim; } opt[PIPE_END] = {
      {1, 4, 1, 110 * 1024}, {2, 4, 1, 110 * 1024}, {2, 2, 1, 110 * 1024}, {1, 4, 1, 220 * 1024},
      {1, 2, 1, 220 * 1024}, {1, 4, 0, 220 * 1024}, {1, 2, 0, 220 * 1024}};
  out->grid = 0;
  for (int k = from; k < to; ++k) {
    const auto& o = opt[k];
    PipeShape q;
    q.grid = ncol < o.per * nsm ? ncol : o.per * nsm;
    q.in_smem = o.in;
    q.nst = o.nst;
    const int nl = (ncol + q.grid - 1) / q.grid;
    const size_t used = (size_t)o.nst * len + (o.in ? (size_t)nl * len : 0), most = o.lim / sizeof(cplx);
    if (used > most || (k == PIPE_ONE && nl > 2)) continue;
    q.smem = sizeof(cplx) * (used + fixed(q.grid, nl, o.in, most - used));
    if (q.smem > o.lim) continue;
    PQMC_CUDA(raise_dyn_smem((const char*)fn, (int)q.smem));
    int per = 0;
    PQMC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, LT, q.smem));
    if (per * nsm < q.grid) continue;
    *out = q;
    return PQMC_OK;
  }
  return PQMC_OK;
}
static int pipe_none(int len) {
  set_error("dense factorisation: columns of %d entries do not fit in shared memory", len);
  return PQMC_ERR_ARG;
}

int house_qr(cudaStream_t s, int m, int n, cplx* A, cplx* d, cplx* work, int* err) {
  return house_qr_r(s, m, n, A, d, nullptr, nullptr, work, err);
}

int house_qr_r(cudaStream_t s, int m, int n, cplx* A, cplx* d, cplx* R, cplx* lndet, cplx* work, int* err) {
  PipeShape q;
  // Q by the triangular factor where the work matrix (m x m) has room for its
  // products behind the published columns (a square A has none), with the
  // terms of U y in sums (2) where shared memory has room for those too
  int ut = (size_t)m * (m - n) >= (size_t)n * n ? 2 : 0;
  const auto fixed = [&](int, int nl, int in, size_t) {
    return (size_t)2 * n + (n + 1) / 2 + (nl + 3) / 4 + (ut && in ? (size_t)nl * n : 0) + (ut == 2 && in ? (size_t)nl * m : 0);
  };
  for (;; --ut) {
    PQMC_TRY(pipe_shape((const void*)k_house_qr, n, m, PIPE_ONE, PIPE_TWO_SHORT, fixed, &q));
    if (!q.grid) PQMC_TRY(pipe_shape((const void*)k_house_qr, n, m, PIPE_ALL, PIPE_END, fixed, &q));
    if (!q.grid) return pipe_none(m);
    if (ut == 0 || (q.in_smem && q.nst == 4 && n <= 2 * q.grid)) break;
  }
  PQMC_CUDA(cudaMemsetAsync(work, 0xff, sizeof(cplx) * ((size_t)m * n + (ut ? (size_t)n * n : 0)), s));
  void* args[] = {&m, &n, &A, &d, &R, &lndet, &work, &q.in_smem, &q.nst, &ut, &err};
  PQMC_CUDA(cudaLaunchCooperativeKernel((const void*)k_house_qr, q.grid, LT, args, q.smem, s));
  PQMC_LAUNCHED();
  return PQMC_OK;
}

int lu_solve(cudaStream_t s, int n, cplx* A, int nrhs, cplx* B, int ldb, cplx* diag, int* perm, int* info, cplx* work,
             int* err) {
  PipeShape q;
  // sums for every right-hand side of a CTA while that leaves two CTAs an SM,
  // past that for as many as fit (512 columns and 1024 right-hand sides take
  // 6.7 ms, 8.9 with one CTA an SM; 624 and 1248, of whose 9 sums 4 fit, 15.7,
  // and 21.6 with all of them and the columns in global memory)
  int nsum = 0, apart = 1;
  const auto fixed = [&](int grid, int, int in, size_t room) {
    const size_t base = (size_t)n + (2 * n + 3) / 4;
    const int rhs = (nrhs + grid - 1) / grid;
    nsum = rhs;
    if (!apart) nsum = std::min(rhs, in && room > base ? std::max(1, (int)((room - base) / n)) : 1);
    return base + (size_t)nsum * n;
  };
  PQMC_TRY(pipe_shape((const void*)k_lu_solve, n + nrhs, n, PIPE_ONE, PIPE_ALL, fixed, &q));
  if (!q.grid) {
    apart = 0;
    PQMC_TRY(pipe_shape((const void*)k_lu_solve, n + nrhs, n, PIPE_TWO, PIPE_END, fixed, &q));
    if (!q.grid) return pipe_none(n);
  }
  PQMC_CUDA(cudaMemsetAsync(work, 0xff, sizeof(cplx) * (size_t)n * n, s));
  void* args[] = {&n, &A, &nrhs, &B, &ldb, &diag, &perm, &info, &work, &q.in_smem, &q.nst, &nsum, &apart, &err};
  PQMC_CUDA(cudaLaunchCooperativeKernel((const void*)k_lu_solve, q.grid, LT, args, q.smem, s));
  PQMC_LAUNCHED();
  return PQMC_OK;
}

int lu_logdet(cudaStream_t s, int n, const cplx* diag, const int* perm, cplx* out) {
  k_lu_logdet<<<1, LT, 0, s>>>(n, diag, perm, out);
  PQMC_LAUNCHED();
  return PQMC_OK;
}

// conjugate transpose copy: out(n,m) = a(m,n)^H
__global__ void k_herm_t(int m, int n, const cplx* __restrict__ a, cplx* __restrict__ out) {
  __shared__ cplx t[32][33];
  int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int r = bx + threadIdx.x, c = by + k;
    if (r < m && c < n) t[k][threadIdx.x] = a[r + (size_t)m * c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int r = by + threadIdx.x, c = bx + k;   // out row r (< n), col c (< m)
    if (r < n && c < m) out[r + (size_t)n * c] = cconj(t[threadIdx.x][k]);
  }
}

int herm_t(cudaStream_t s, int m, int n, const cplx* a, cplx* out) {
  dim3 g((m + 31) / 32, (n + 31) / 32), b(32, 8);
  k_herm_t<<<g, b, 0, s>>>(m, n, a, out);
  PQMC_LAUNCHED();
  return PQMC_OK;
}

}  // namespace pqmc
