// meas.cu -- equal-time measurement (ms_take_measurement,
// src/mod_meas.f90:210-544; helpers :64-208; k-space :546-566; window
// averaging :729-763) and the fused sweep driver (src/Main_PQMC.f90:81-156).
//
// One CTA per part of the observables and relative displacement `ind`; its
// threads cover the cells c1, each evaluating its part of the Wick
// contractions of the pair (c1, c2) with rel(c1,c2) = ind, then a fixed-order
// sum per observable.  The per-cell phonon scalars are one more CTA.
#include <algorithm>
#include <string.h>
#include <vector>
#include "chain.cuh"
#include "linalg.cuh"

namespace pqmc {

struct MeasView {
  int ns, nc;
  const cplx* gh;
  const int* sites;   // (2,nc)
  const int* bfi;     // (2,nc)
  const int* xnb;
  const int* ynb;
  const int* cross;   // (2,nc)
  const int* c2_of;   // (nc,nc): c2_of[c1 + nc*ind]
  const double* field;
  int t, n_bf;
  cplx bc[2];
  double hop, ep;
};

__device__ __forceinline__ cplx GH(const MeasView& V, int i, int j) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(V.gh) + i + (size_t)V.ns * j);
  return mk(v.x, v.y);
}
// -g = gh - 1 (its sign goes into the sums)
__device__ __forceinline__ cplx GN(const MeasView& V, int i, int j) {
  cplx v = GH(V, i, j);
  if (i == j) v.x -= 1.0;
  return v;
}

// ---------------------------------------------------------------------------
// The Wick contractions of a pair of cells (cal_wick_contraction, :165-183):
//   mat(i,j) = gh(l2,l1) gh(r2,r1) + gh(r2,l1) g(l2,r1)
// between site pairs (l1,l2) of a bond at c1 and (r1,r2) of one at c2, and
// sums vl(i) mat(i,j) vr(j) over them.  FP64 issue bounds the kernel, so the
// sums are factored.  The first term is a product of one sum over i and one
// over j (the Hartree observables are that product alone).  A bond's four
// spin-flipping pairs carry the coefficients (b, sb, -b', -sb') (s = +1 or
// -1, b the boundary phase, b' its conjugate, :199-208), so the second term
// is four block sums of the 16 products, with signs only; and with the four
// spin-conserving pairs of the physical current it is the trace of P VL Q VR,
// P = gh between the bonds' sites, Q = g, VL and VR with two entries per row.
// That is ~1.3k FP64 operations per pair instead of the ~4.2k of the plain
// contractions.  The division by N_cell is done on the sums.
// ---------------------------------------------------------------------------
struct Bond {     // a cell's two sites and its neighbour's, the phase of the bond
  int s[4];
  cplx b;
};
__device__ __forceinline__ Bond bond(const MeasView& V, int c, int dir) {
  const int n = dir ? V.ynb[c] : V.xnb[c];
  Bond B;
  B.s[0] = V.sites[2 * c];
  B.s[1] = V.sites[2 * c + 1];
  B.s[2] = V.sites[2 * n];
  B.s[3] = V.sites[2 * n + 1];
  B.b = V.cross[2 * c + dir] ? V.bc[dir] : mk(1.0);
  return B;
}
__device__ __forceinline__ double boson(const MeasView& V, int c, int dir) {
  return V.field[V.bfi[2 * c + dir] + (size_t)V.n_bf * V.t];
}

// b1 (b2 t00 + b2' t01) + b1' (b2 t10 + b2' t11)
__device__ __forceinline__ cplx phases(cplx b1, cplx b2, const cplx (&t)[2][2]) {
  const cplx u = cfma(b2, t[0][0], cmul(cconj(b2), t[0][1]));
  const cplx w = cfma(b2, t[1][0], cmul(cconj(b2), t[1][1]));
  return cfma(b1, u, cmul(cconj(b1), w));
}
__device__ __forceinline__ cplx times_i(cplx z, double f) { return mk(-f * z.y, f * z.x); }

// sum of v(i) gh(l2,l1) over a bond's spin-flipping pairs; vx: i hop (b, b,
// -b', -b'), vy: hop (b, -b, -b', b')
__device__ __forceinline__ void spin_sums(const MeasView& V, const Bond& B, cplx* vx, cplx* vy) {
  const cplx a0 = GH(V, B.s[3], B.s[0]), a1 = GH(V, B.s[2], B.s[1]);
  const cplx a2 = GH(V, B.s[1], B.s[2]), a3 = GH(V, B.s[0], B.s[3]);
  *vx = times_i(csub(cmul(B.b, cadd(a0, a1)), cmul(cconj(B.b), cadd(a2, a3))), V.hop);
  const cplx y = csub(cmul(B.b, csub(a0, a1)), cmul(cconj(B.b), csub(a2, a3)));
  *vy = mk(V.hop * y.x, V.hop * y.y);
}

// the second term of the spin currents of two bonds, (vx, vx) and (vy, vy);
// bq: the phase that stands for the right bond's in (vy, vy)
__device__ __forceinline__ void spin_exchange(const MeasView& V, const Bond& L, const Bond& R, cplx bq, cplx* xx,
                                              cplx* yy) {
  cplx pp[2][2], mm[2][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      cplx e[2][2];   // site pairs (l1, l2) = (i, 3 - i), (r1, r2) = (j, 3 - j)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int l = 2 * a + i, r = 2 * b + j;
          e[i][j] = cmul(GH(V, R.s[3 - r], L.s[l]), GN(V, L.s[3 - l], R.s[r]));
        }
      pp[a][b] = cadd(cadd(e[0][0], e[0][1]), cadd(e[1][0], e[1][1]));
      mm[a][b] = cadd(csub(e[0][0], e[0][1]), csub(e[1][1], e[1][0]));
      if (a != b) {
        pp[a][b] = cneg(pp[a][b]);
        mm[a][b] = cneg(mm[a][b]);
      }
    }
  const double h2 = V.hop * V.hop;
  const cplx x = phases(L.b, R.b, pp), y = phases(L.b, bq, mm);
  *xx = mk(h2 * x.x, h2 * x.y);
  *yy = mk(-h2 * y.x, -h2 * y.y);
}

// k z + e w, k the coefficient of a spin-flipping pair in the physical
// current: -i hop (X) or -hop, times sg
template <bool X>
__device__ __forceinline__ cplx flip_keep(double hop, double sg, cplx z, double e, cplx w) {
  const double k = -sg * hop;
  return X ? mk(fma(e, w.x, -k * z.y), fma(e, w.y, k * z.x)) : mk(fma(e, w.x, k * z.x), fma(e, w.y, k * z.y));
}

// sum of v(i) gh(l2,l1) over a bond's eight pairs, e the spin-conserving coefficient
template <bool X>
__device__ __forceinline__ cplx phys_sum(const MeasView& V, const Bond& B, double e) {
  auto g = [&](int l2, int l1) { return GH(V, B.s[l2], B.s[l1]); };
  const cplx f0 = X ? cadd(g(3, 0), g(2, 1)) : csub(g(3, 0), g(2, 1));
  const cplx f1 = X ? cadd(g(1, 2), g(0, 3)) : csub(g(1, 2), g(0, 3));
  const cplx u = flip_keep<X>(V.hop, 1.0, f0, e, cadd(g(2, 0), g(3, 1)));
  const cplx w = flip_keep<X>(V.hop, -1.0, f1, e, cadd(g(0, 2), g(1, 3)));
  return cfma(B.b, u, cmul(cconj(B.b), w));
}

// physical current-current of two bonds along one direction; X: the spin
// part is vx, else vy; e1, e2: ep x of the bonds
template <bool X>
__device__ __forceinline__ cplx phys_pair(const MeasView& V, const Bond& L, const Bond& R, double e1, double e2) {
  cplx t[2][2];
  // columns of P VL and Q VR by the second site, 3 and 2 with the phase, 1
  // and 0 with its conjugate; a column takes two of P's (Q's)
  const double s1 = X ? 1.0 : -1.0;
  cplx y[4][4];   // [l2][r2]
#pragma unroll
  for (int l2 = 0; l2 < 4; ++l2) {
    cplx q[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) q[r] = GN(V, L.s[l2], R.s[r]);
    y[l2][3] = flip_keep<X>(V.hop, 1.0, q[0], e2, q[1]);
    y[l2][2] = flip_keep<X>(V.hop, s1, q[1], e2, q[0]);
    y[l2][1] = flip_keep<X>(V.hop, -1.0, q[2], e2, q[3]);
    y[l2][0] = flip_keep<X>(V.hop, -s1, q[3], e2, q[2]);
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) t[a][b] = mk(0.0);
#pragma unroll
  for (int r2 = 0; r2 < 4; ++r2) {
    cplx q[4], x[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) q[l] = GH(V, R.s[r2], L.s[l]);
    x[3] = flip_keep<X>(V.hop, 1.0, q[0], e1, q[1]);
    x[2] = flip_keep<X>(V.hop, s1, q[1], e1, q[0]);
    x[1] = flip_keep<X>(V.hop, -1.0, q[2], e1, q[3]);
    x[0] = flip_keep<X>(V.hop, -s1, q[3], e1, q[2]);
    const int b = r2 < 2 ? 1 : 0;
#pragma unroll
    for (int l2 = 0; l2 < 4; ++l2) t[l2 < 2 ? 1 : 0][b] = cfma(x[l2], y[l2][r2], t[l2 < 2 ? 1 : 0][b]);
  }
  return csub(cmul(phys_sum<X>(V, L, e1), phys_sum<X>(V, R, e2)), phases(L.b, R.b, t));
}

// The observables of a pair in five parts of about equal work (the current
// correlations along y and x, the spin currents along y, x and crossed) and
// a light one (density, spin, pairing, phonons).  One CTA per part and
// relative displacement: the longest CTA is then 1/5 of a pair, and the
// 6 n_cell CTAs spread evenly.
constexpr int MEAS_PARTS = 6;
constexpr int MEAS_MAX = 9;   // observables of a part, at most
__device__ __constant__ const signed char meas_field[MEAS_PARTS][MEAS_MAX] = {
    {PQMC_F_CJYX_CJYX, -1},
    {PQMC_F_CJXY_CJXY, -1},
    {PQMC_F_JXX_JYX, PQMC_F_JXY_JYY, PQMC_F_JXXH_JYXH, PQMC_F_JXYH_JYYH, PQMC_F_JXXH_JYYH, PQMC_F_JXYH_JYXH, -1},
    {PQMC_F_JYX_JYX, PQMC_F_JYY_JYY, PQMC_F_JYXH_JYXH, PQMC_F_JYYH_JYYH, -1},
    {PQMC_F_JXX_JXX, PQMC_F_JXY_JXY, PQMC_F_JXXH_JXXH, PQMC_F_JXYH_JXYH, -1},
    {PQMC_F_DEN_DEN, PQMC_F_SZ_SZ, PQMC_F_SX_SX, PQMC_F_SY_SY, PQMC_F_SC_SC, PQMC_F_BFX_BFX, PQMC_F_BFX_BFY,
     PQMC_F_BFY_BFY, PQMC_F_BFXY_BFXY}};
__device__ __constant__ const int meas_count[MEAS_PARTS] = {1, 1, 6, 4, 4, 9};

// adds one pair's observables of `part` (uniform over the CTA) to f
__device__ __forceinline__ void pair_obs(const MeasView& V, int part, int c1, int c2, cplx (&f)[MEAS_MAX]) {
  if (part == 0) {
    f[0] = cadd(f[0], phys_pair<true>(V, bond(V, c1, 1), bond(V, c2, 1), V.ep * boson(V, c1, 1),
                                      V.ep * boson(V, c2, 1)));
  } else if (part == 1) {
    f[0] = cadd(f[0], phys_pair<false>(V, bond(V, c1, 0), bond(V, c2, 0), V.ep * boson(V, c1, 0),
                                       V.ep * boson(V, c2, 0)));
  } else if (part < 5) {
    const Bond L = bond(V, c1, part == 3 ? 1 : 0), R = bond(V, c2, part == 4 ? 0 : 1);
    const bool quirk = part == 3;   // (vy, vy) along y takes the left phases twice (:353, :417)
    cplx lx, ly, rx, ry, xx, yy;
    spin_exchange(V, L, R, quirk ? L.b : R.b, &xx, &yy);
    spin_sums(V, L, &lx, &ly);
    spin_sums(V, R, &rx, &ry);
    cplx rq = ry;
    if (quirk) {
      Bond Q = R;
      Q.b = L.b;
      cplx unused;
      spin_sums(V, Q, &unused, &rq);
    }
    const cplx hx = cmul(lx, rx), hy = cmul(ly, rq);
    f[0] = cadd(f[0], cadd(hx, xx));
    f[1] = cadd(f[1], cadd(hy, yy));
    f[2] = cadd(f[2], hx);
    f[3] = cadd(f[3], hy);
    if (part == 2) {
      f[4] = cfma(lx, ry, f[4]);
      f[5] = cfma(ly, rx, f[5]);
    }
  } else {
    const int u1 = V.sites[2 * c1], d1 = V.sites[2 * c1 + 1], u2 = V.sites[2 * c2], d2 = V.sites[2 * c2 + 1];
    const cplx puu = GH(V, u2, u1), pud = GH(V, u2, d1), pdu = GH(V, d2, u1), pdd = GH(V, d2, d1);   // gh(r, l)
    const cplx quu = GN(V, u1, u2), qud = GN(V, u1, d2), qdu = GN(V, d1, u2), qdd = GN(V, d1, d2);   // -g(l, r)
    const cplx a0 = GH(V, u1, u1), a1 = GH(V, d1, u1), a2 = GH(V, u1, d1), a3 = GH(V, d1, d1);       // gh(l2, l1)
    const cplx b0 = GH(V, u2, u2), b1 = GH(V, d2, u2), b2 = GH(V, u2, d2), b3 = GH(V, d2, d2);
    // pairs (u,u), (d,d) on both sides: mat(i,j) for density and s_z
    const cplx s = cadd(cmul(puu, quu), cmul(pdd, qdd)), o = cadd(cmul(pdu, qud), cmul(pud, qdu));
    const cplx den = csub(cmul(cadd(a0, a3), cadd(b0, b3)), cadd(s, o));
    const cplx sz = csub(cmul(csub(a0, a3), csub(b0, b3)), csub(s, o));
    // pairs (u,d), (d,u): s_x = (1 + 2) / 2, s_y = (-i 1 + i 2) / 2
    const cplx e11 = cmul(pdu, qdu), e12 = cmul(puu, qdd), e21 = cmul(pdd, quu), e22 = cmul(pud, qud);
    const cplx d = cadd(e11, e22), x = cadd(e12, e21);
    const cplx sx = csub(cmul(cadd(a1, a2), cadd(b1, b2)), cadd(d, x));
    const cplx sy = csub(csub(d, x), cmul(csub(a1, a2), csub(b1, b2)));
    const cplx sc = csub(cmul(puu, pdd), cmul(pdu, pud));
    f[0] = mk(fma(0.25, den.x, f[0].x), fma(0.25, den.y, f[0].y));
    f[1] = mk(fma(0.25, sz.x, f[1].x), fma(0.25, sz.y, f[1].y));
    f[2] = mk(fma(0.25, sx.x, f[2].x), fma(0.25, sx.y, f[2].y));
    f[3] = mk(fma(0.25, sy.x, f[3].x), fma(0.25, sy.y, f[3].y));
    f[4] = cadd(f[4], sc);
    const double x1x = boson(V, c1, 0), x1y = boson(V, c1, 1), x2x = boson(V, c2, 0), x2y = boson(V, c2, 1);
    f[5].x = fma(x1x, x2x, f[5].x);
    f[6].x = fma(x1x, x2y, f[6].x);
    f[7].x = fma(x1y, x2y, f[7].x);
    f[8].x = fma(x1x * x1y, x2x * x2y, f[8].x);
  }
}

constexpr int MEAS_THREADS = 224;   // at most; a lattice of 14 x 14 cells fills them

// the sums over the CTA of n values per thread, in a fixed order; sum v is
// returned by lane 0 of warp v % warps in `out`
template <class F>
__device__ __forceinline__ void meas_sum(int n, double (*s)[MEAS_THREADS], F out) {
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int v = warp; v < n; v += nw) {
    double a = s[v][lane];
    for (int k = lane + 32; k < blockDim.x; k += 32) a += s[v][k];
    for (int m = 16; m > 0; m >>= 1) a += __shfl_xor_sync(~0u, a, m);
    if (lane == 0) out(v, a);
  }
}

// CTAs 0 .. 6 n_cell - 1: a part of the pair observables at one relative
// displacement `ind`, each thread the pairs (c1, c2) with rel(c1, c2) = ind of
// its cells c1.  The last CTA: BF_KE, BF_PE, BF_X (:249-268).  Measured at
// 196 cells 142 us, of which FP64 issue alone is ~80 (one CTA per
// displacement with all observables as written out: 594 us, and 337 for the
// scalars by one thread); at 16 cells 22 us (196 and 29).
__global__ void __launch_bounds__(MEAS_THREADS) k_meas_pairs(MeasView V, double D, double M, double biased, double delt,
                                                             cplx* acc) {
  __shared__ double s[2 * MEAS_MAX][MEAS_THREADS];
  const int tid = threadIdx.x;
  const double N = (double)V.nc;
  if (blockIdx.x == MEAS_PARTS * V.nc) {
    double ke = 0.0, pe = 0.0, xs = 0.0;
    for (int c = tid; c < V.nc; c += blockDim.x) {
      const double* x = V.field + (size_t)V.n_bf * V.t;
      const int bx = V.bfi[2 * c], by = V.bfi[2 * c + 1];
      const double x1x = x[bx], x1y = x[by], d1 = x1x - x[bx + V.n_bf], d2 = x1y - x[by + V.n_bf];
      ke += (0.5 * D) * (x1x * x1x + x1y * x1y) - biased * (x1x + x1y);
      pe += (1.0 / (2.0 * delt)) * 2.0 - ((0.5 * M) * (d1 * d1 + d2 * d2)) / (delt * delt);
      xs += x1x + x1y;
    }
    s[PQMC_OBS_BF_KE][tid] = ke;
    s[PQMC_OBS_BF_PE][tid] = pe;
    s[PQMC_OBS_BF_X][tid] = xs;
    meas_sum(PQMC_N_SCALAR, s, [&](int v, double a) { acc[v].x += a / N; });
    return;
  }
  const int part = blockIdx.x / V.nc, ind = blockIdx.x % V.nc;
  cplx f[MEAS_MAX];
#pragma unroll
  for (int k = 0; k < MEAS_MAX; ++k) f[k] = mk(0.0);
  for (int c1 = tid; c1 < V.nc; c1 += blockDim.x) pair_obs(V, part, c1, V.c2_of[c1 + (size_t)V.nc * ind], f);
  const int n = meas_count[part];
#pragma unroll
  for (int k = 0; k < MEAS_MAX; ++k)
    if (k < n) {
      s[2 * k][tid] = f[k].x;
      s[2 * k + 1][tid] = f[k].y;
    }
  meas_sum(2 * n, s, [&](int v, double a) {
    cplx* dst = acc + PQMC_N_SCALAR + (size_t)meas_field[part][v >> 1] * V.nc + ind;
    if (v & 1) dst->y += a / N;
    else dst->x += a / N;
  });
}

// ms_k_space_obs of the averaged real-space part: sixteen k per CTA, the sum
// over the cells in MEAS_KSPLIT shares.  FP64 issue bounds it (4 n_cell
// multiply-adds per output); the window's average was divided out of each
// term here before (two divisions per four multiply-adds): 263 us at 196 cells,
// now 13.
constexpr int MEAS_KSPLIT = 8;
__global__ void __launch_bounds__(16 * MEAS_KSPLIT) k_meas_finish(int nc, const cplx* __restrict__ kphase, cplx* acc) {
  __shared__ cplx part[MEAS_KSPLIT][16];
  const int f = blockIdx.x, k = threadIdx.x & 15, h = threadIdx.x >> 4, ik = k + 16 * blockIdx.y;
  const cplx* r = acc + PQMC_N_SCALAR + (size_t)f * nc;
  cplx s = mk(0.0);
  if (ik < nc)
    for (int i = h; i < nc; i += MEAS_KSPLIT) s = cfma(kphase[ik + (size_t)nc * i], r[i], s);
  part[h][k] = s;
  __syncthreads();
  if (h == 0 && ik < nc) {
    for (int j = 1; j < MEAS_KSPLIT; ++j) s = cadd(s, part[j][k]);
    cplx* kd = acc + PQMC_N_SCALAR + (size_t)(PQMC_N_FIELD + f) * nc;
    kd[ik] = cadd(kd[ik], mk(s.x / (double)nc, s.y / (double)nc));
  }
}

// window average
__global__ void k_meas_divide(int n, double div, cplx* acc) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    acc[i] = mk(acc[i].x / div, acc[i].y / div);
}

static MeasView view(pqmc_chain* c, int time) {
  MeasView V;
  V.ns = c->ns;
  V.nc = c->n_cell;
  V.gh = c->g;
  V.sites = c->m_cell_sites;
  V.bfi = c->m_cell_bf;
  V.xnb = c->m_cell_xnb;
  V.ynb = c->m_cell_ynb;
  V.cross = c->m_cell_cross;
  V.c2_of = c->m_c2_of;
  V.field = c->field;
  V.t = time - 1;
  V.n_bf = c->n_bf;
  V.bc[0] = c->h_bc[0];
  V.bc[1] = c->h_bc[1];
  V.hop = c->hop;
  V.ep = c->ep;
  return V;
}

int do_measure(pqmc_chain* c, int time) {
  MeasView V = view(c, time);
  const int threads = std::min(MEAS_THREADS, (c->n_cell + 31) / 32 * 32);
  k_meas_pairs<<<MEAS_PARTS * c->n_cell + 1, threads, 0, c->stream>>>(V, c->M.stiff, c->M.mass, c->M.biased, c->M.delt,
                                                                      c->m_acc);
  PQMC_LAUNCHED();
  return PQMC_OK;
}

int do_finish_record(pqmc_chain* c, int meas_number) {
  const int nc = c->n_cell, n = PQMC_N_SCALAR + PQMC_N_FIELD * nc;
  k_meas_divide<<<(n + 127) / 128, 128, 0, c->stream>>>(n, (double)(2 * meas_number + 1), c->m_acc);
  PQMC_LAUNCHED();
  dim3 g(PQMC_N_FIELD, (nc + 15) / 16);
  k_meas_finish<<<g, 16 * MEAS_KSPLIT, 0, c->stream>>>(nc, c->m_kphase, c->m_acc);
  PQMC_LAUNCHED();
  return PQMC_OK;
}

static int record_width(const pqmc_chain* c) { return PQMC_N_SCALAR + 2 * PQMC_N_FIELD * c->n_cell; }

// the slice loop of Main_PQMC.f90:99-154 for one value of `loop`
static int sweep_one(pqmc_chain* c, int loop, int warmup, int meas_interval, int meas_number, double* records,
                     int cap, int* nrec, int tc_first = 1, int tc_last = 0) {
  const bool forward = (loop % 2) == 0;   // the first loop (loop=1) runs backward (:85)
  const int half = c->ntime / 2;
  const int W = record_width(c);
  if (tc_last <= 0) tc_last = c->ntime;
  for (int tc = tc_first; tc <= tc_last; ++tc) {
    int time;
    if (!forward) {
      time = c->ntime - tc + 1;
      for (int pf = c->n_pf - 1; pf >= 0; --pf) {
        PQMC_TRY(launch_wrap(c, pf, time, false));
        if (c->M.local_update && c->h_pf_v_exist[pf]) PQMC_TRY(launch_update(c, pf, time));
      }
    } else {
      time = tc;
      for (int pf = 0; pf < c->n_pf; ++pf) {
        if (c->M.local_update && c->h_pf_v_exist[pf]) PQMC_TRY(launch_update(c, pf, time));
        PQMC_TRY(launch_wrap(c, pf, time, true));
      }
    }
    if (tc % c->ngroup == 0) PQMC_TRY(do_g_scratch(c, forward ? time + 1 : time, forward, loop));
    if (c->have_meas && loop > warmup && ((loop - warmup) % meas_interval) == 0 && time >= half - meas_number &&
        time <= half + meas_number) {
      PQMC_TRY(do_measure(c, time));
      bool last = (forward && time == half + meas_number) || (!forward && time == half - meas_number);
      if (last) {
        PQMC_TRY(do_finish_record(c, meas_number));
        if (records && *nrec < cap)
          PQMC_CUDA(cudaMemcpyAsync(records + (size_t)2 * W * (*nrec), c->m_acc, sizeof(cplx) * W,
                                    cudaMemcpyDeviceToHost, c->stream));
        PQMC_CUDA(cudaMemsetAsync(c->m_acc, 0, sizeof(cplx) * W, c->stream));
        (*nrec)++;
      }
    }
  }
  return PQMC_OK;
}

}  // namespace pqmc

using namespace pqmc;

extern "C" {

int pqmc_set_meas_layout(pqmc_chain* c, const pqmc_meas_layout* L) {
  if (!c || !L) { set_error("null argument"); return PQMC_ERR_ARG; }
  const int nc = L->n_cell;
  for (int k = 0; k < 2 * nc; ++k)
    if (L->cell_sites[k] < 0 || L->cell_sites[k] >= c->ns || L->cell_bf[k] < 0 || L->cell_bf[k] >= c->n_bf) {
      set_error("meas layout: site/boson index out of range");
      return PQMC_ERR_ARG;
    }
  std::vector<int> c2of((size_t)nc * nc, -1);
  for (int c1 = 0; c1 < nc; ++c1)
    for (int c2 = 0; c2 < nc; ++c2) {
      int ind = L->rel_index[c1 + (size_t)nc * c2];
      if (ind < 0 || ind >= nc || c2of[c1 + (size_t)nc * ind] >= 0) {
        set_error("meas layout: relative index table is not a permutation per cell");
        return PQMC_ERR_ARG;
      }
      c2of[c1 + (size_t)nc * ind] = c2;
    }
  auto up = [&](int** d, const int32_t* h, size_t n) -> int {
    if (*d) cudaFree(*d);
    PQMC_CUDA(cudaMalloc((void**)d, sizeof(int) * n));
    PQMC_CUDA(cudaMemcpy(*d, h, sizeof(int) * n, cudaMemcpyHostToDevice));
    return PQMC_OK;
  };
  PQMC_TRY(up(&c->m_cell_sites, L->cell_sites, 2 * nc));
  PQMC_TRY(up(&c->m_cell_bf, L->cell_bf, 2 * nc));
  PQMC_TRY(up(&c->m_cell_xnb, L->cell_xnb, nc));
  PQMC_TRY(up(&c->m_cell_ynb, L->cell_ynb, nc));
  PQMC_TRY(up(&c->m_cell_cross, L->cell_cross, 2 * nc));
  PQMC_TRY(up(&c->m_c2_of, c2of.data(), (size_t)nc * nc));
  if (c->m_kphase) cudaFree(c->m_kphase);
  PQMC_CUDA(cudaMalloc((void**)&c->m_kphase, sizeof(cplx) * (size_t)nc * nc));
  PQMC_CUDA(cudaMemcpy(c->m_kphase, L->k_phase, sizeof(cplx) * (size_t)nc * nc, cudaMemcpyHostToDevice));
  c->n_cell = nc;
  const int W = record_width(c);
  if (c->m_acc) cudaFree(c->m_acc);
  PQMC_CUDA(cudaMalloc((void**)&c->m_acc, sizeof(cplx) * W));
  PQMC_CUDA(cudaMemset(c->m_acc, 0, sizeof(cplx) * W));
  c->h_bc[0] = mk(L->bc_phase[0], L->bc_phase[1]);
  c->h_bc[1] = mk(L->bc_phase[2], L->bc_phase[3]);
  c->hop = L->hop;
  c->ep = L->ep_parameter;
  c->have_meas = true;
  return PQMC_OK;
}

int pqmc_take_measurement(pqmc_chain* c, int time) {
  if (!c) { set_error("null chain"); return PQMC_ERR_ARG; }
  if (!c->have_meas) { set_error("no measurement layout"); return PQMC_ERR_STATE; }
  if (time < 1 || time >= c->ntime) { set_error("time out of range"); return PQMC_ERR_ARG; }
  PQMC_TRY(do_measure(c, time));
  PQMC_CUDA(cudaStreamSynchronize(c->stream));
  return PQMC_OK;
}

int pqmc_begin_measure(pqmc_chain* c, int forward, int time, int meas_number, double* record_out, int* done) {
  if (!c) { set_error("null chain"); return PQMC_ERR_ARG; }
  if (!c->have_meas) { set_error("no measurement layout"); return PQMC_ERR_STATE; }
  if (time < 1 || time >= c->ntime) { set_error("time out of range"); return PQMC_ERR_ARG; }
  PQMC_TRY(do_measure(c, time));
  const int half = c->ntime / 2;
  bool last = (forward && time == half + meas_number) || (!forward && time == half - meas_number);
  if (done) *done = last ? 1 : 0;
  if (last) {
    PQMC_TRY(do_finish_record(c, meas_number));
    const int W = record_width(c);
    if (record_out)
      PQMC_CUDA(cudaMemcpyAsync(record_out, c->m_acc, sizeof(cplx) * W, cudaMemcpyDeviceToHost, c->stream));
    PQMC_CUDA(cudaMemsetAsync(c->m_acc, 0, sizeof(cplx) * W, c->stream));
  }
  PQMC_CUDA(cudaStreamSynchronize(c->stream));
  return PQMC_OK;
}

int pqmc_sweep(pqmc_chain* c, int first_loop, int n_sweeps, int warmup, int meas_interval, int meas_number,
               double* records, int n_records_cap, int* n_records) {
  if (!c) { set_error("null chain"); return PQMC_ERR_ARG; }
  if (!c->have_g) { set_error("sweep before init_g"); return PQMC_ERR_STATE; }
  if (n_sweeps < 0 || meas_interval < 1 || meas_number < 0) { set_error("bad sweep arguments"); return PQMC_ERR_ARG; }
  if (c->have_meas && (c->ntime / 2 - meas_number < 1 || c->ntime / 2 + meas_number > c->ntime - 1)) {
    set_error("measurement window ntime/2 +- %d leaves 1..ntime-1", meas_number);
    return PQMC_ERR_ARG;
  }
  int nrec = 0;
  for (int loop = first_loop; loop < first_loop + n_sweeps; ++loop) {
    // global step before the sweep (Main_PQMC.f90:87-96), once enabled
    if (c->have_global) PQMC_TRY(pqmc_global_step(c, loop, nullptr));
    PQMC_TRY(sweep_one(c, loop, warmup, meas_interval, meas_number, records, n_records_cap, &nrec));
  }
  PQMC_TRY(check_waits(c, "sweep"));
  if (n_records) *n_records = nrec;
  return PQMC_OK;
}

int pqmc_sweep_slices(pqmc_chain* c, int loop, int first_tc, int n_slices) {
  if (!c) { set_error("null chain"); return PQMC_ERR_ARG; }
  if (!c->have_g) { set_error("sweep before init_g"); return PQMC_ERR_STATE; }
  if (first_tc < 1 || n_slices < 0 || first_tc + n_slices - 1 > c->ntime) {
    set_error("sweep_slices: slices %d..%d outside 1..%d", first_tc, first_tc + n_slices - 1, c->ntime);
    return PQMC_ERR_ARG;
  }
  if (n_slices == 0) return PQMC_OK;
  int nrec = 0;
  PQMC_TRY(sweep_one(c, loop, 1 << 30, 1, 0, nullptr, 0, &nrec, first_tc, first_tc + n_slices - 1));
  return check_waits(c, "sweep_slices");
}

}  // extern "C"
