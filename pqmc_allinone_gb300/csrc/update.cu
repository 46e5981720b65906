// update.cu -- update_phonon_field(ppf, time) (src/mod_update.f90:13-245,
// 475-500) as one cooperative kernel per family step.
//
// Draws:   every CTA walks the family's ran2 stream (each proposal consumes
//          a fixed number of draws, :84 and :117) and keeps its own part.
// Phase 1: every CTA prepares plaquettes blockIdx, blockIdx + CTAs, .., two warps each:
//          the phonon action difference and threshold (:203-228) on one, the
//          new propagators and Delta = expKV_inv(old) expKV(new) - I
//          (:230-245) on the other.
// Phase 2: CTA 0 walks the plaquettes in the reference's Markov order, three
//          proposals at a time (one per warp, each on its own SM quarter;
//          valid up to the first accepted one): R = I + G_SS Delta, det R,
//          Metropolis test (:97-119).  An accepted move is published as
//          (S, T = Delta R^-1); every other CTA applies it out of place,
//          G' = G + G(:,S) T (I - G)(S,:) (:146-187), while CTA 0 scans ahead
//          with G plus that move's correction on the blocks it needs.  One
//          hand-over per accepted move, none per rejection.
//
// What bounds it: FP64 instructions.  A warp's FP64 instruction holds its SM
// quarter for 64 cycles whatever its lanes, dependent or not, so on the one
// chain that matters (CTA 0 from one publication to the next) what counts is how
// many there are: a lane per real component of a 4x4 complex entry (32 lanes,
// half the instructions of 16 complex lanes), the determinant and the inverse
// from the twelve 2x2 minors of the row pairs, and no separate FP32 screen.
// The other CTAs need Ns^2 dim complex multiply-adds per accepted move, 4.3 us
// of the whole chip at Ns = 392 (8.6 us a move with the hand-over).  A family
// step at 4x4 with Gaussian proposals takes 41 us (413 with one worker CTA
// and 16 complex lanes), at 14x14 0.48 ms (0.91).
#include <cooperative_groups.h>
#include "chain.cuh"
#include "linalg.cuh"
#include "rng.cuh"
#include "update_dev.cuh"

namespace cg = cooperative_groups;

namespace pqmc {

// Metropolis / heat-bath threshold on |det R|^2 (cal_prob, src/mod_update.f90:
// 475-500, with the weight ratio of :101-108).  The ratio's modulus is
// |det|^n with n = ncopy (x2 under TR_weight); exp(min(10,w)) >= r with
// w = dE + log|det|^n  <=>  |det|^2 >= (r e^{-dE})^{2/n}.
__device__ __forceinline__ double accept_threshold(const DevModel& M, double dE, double r) {
  const int n = M.ncopy * (M.tr_weight ? 2 : 1);
  double q;
  if (M.metropolis) {
    q = M.greatest_decent ? exp(-dE) : r * exp(-dE);
  } else {
    double rr = r / (1.0 - r);
    if (!(rr <= exp(10.0))) return INFINITY;
    q = rr * exp(-dE);
  }
  if (n == 1) return q * q;
  if (n == 2) return q;
  return pow(q, 2.0 / n);
}

// real component c (0 re, 1 im) of acc + x*y, the two products of cfma in its order
__device__ __forceinline__ double cfma_part(cplx x, cplx y, double acc, int c) {
  const double bx = c ? y.y : y.x, by = flip_sign(c ? y.x : y.y, !c);
  return fma(x.x, bx, fma(x.y, by, acc));
}
__device__ __forceinline__ double ldg_part(const cplx* p, int c) { return __ldcg(reinterpret_cast<const double*>(p) + c); }
__device__ __forceinline__ void st_part(cplx* p, int c, double v) { reinterpret_cast<double*>(p)[c] = v; }
// index of the column pair (a < b) among 01 02 03 12 13 23
__device__ __forceinline__ int pair_index(int a, int b) { return a * (7 - a) / 2 + b - a - 1; }

// closed_norm by a whole warp: the two moduli, each a hypot, side by side
__device__ __forceinline__ double closed_norm_warp(const DevModel& M, int pf, double x, int lane) {
  if (M.expkv_kind != PQMC_EXPKV_EPSOCZ_BLOCK) return closed_norm(M, pf, x);
  const int pd = M.pdim, k = lane & 1;
  const cplx vx = cscale(M.v_coe[pf], x);
  const size_t at = (size_t)pd * pd * pf + k + pd * 2;
  const double c = cabsd(cadd(cmul(M.k_coe[pf], M.kmat[at]), cmul(vx, M.vmat[at])));
  const double a = __shfl_sync(0xffffffffu, c, 0), b = __shfl_sync(0xffffffffu, c, 1);
  return M.delt * sqrt(a * a + b * b);
}

constexpr int UPD_SPEC = 3;   // proposals CTA 0 evaluates at a time (the fourth SM quarter does the bookkeeping)
// 4x4 blocks of one proposal, entry (i, j) at i + 4 j
struct PropBuf {
  cplx g1[16], g2[16], d[16], w[16], r[16], min[12];
};

// ---- hand-over between CTA 0 and the others -------------------------------
// CTA 0 publishes move k by setting UpdSync::seq to k; a CTA that has applied
// move k adds itself to `arrived`, the last one sets `done` to k, and a CTA
// applies move k once seq shows it and `done` the move before (CTA 0 waits
// for the same before it reads what that move left).  What is polled is apart
// from what is added to: 151 CTAs polling `arrived` itself made a hand-over
// 4500 cycles long.  The words run on from launch to launch: a launch reads
// where they stand before its grid barrier.  Every wait is bounded (~2 s).
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ bool wait_count(const unsigned* p, unsigned base, unsigned want) {
  const long long t0 = clock64();
  while (ld_acquire(p) - base < want)
    if (clock64() - t0 > PQMC_WAIT_CYCLES) return false;
  return true;
}

// G' = G + G(:,S) W,  W = T (I - G)(S,:), on the CTA's share of the entries
// (contiguous, at least 128 so that a thread has no more than it must: the
// 4x4 lattice's 1024 entries go to 8 CTAs).  The columns G(:,S) come into
// shared memory (a share of some columns needs all their rows, each for every
// column it has) while W is formed, a real component of each product per
// thread summed over the four sites by shuffles; then UPD_EPT entries per
// thread.  A share of at most UPD_EPT entries per thread (Ns <= 393 on 152
// SMs) stays in the threads' registers from move to move (`keep`).
constexpr int UPD_EPT = 4, UPD_WC = 16;   // entries per thread in flight, columns of W at a time
constexpr size_t UPD_STAGE = 200 * 1024;  // largest stage of the four columns; larger lattices read them from L2
struct Share {
  unsigned e0, e1;
  int c0, c1;
};
template <int DIM>
__device__ __forceinline__ void apply_move(int ns, int rdim, const int* s_S, const cplx* s_T, const cplx* gcur, cplx* gnext,
                                           const Share sh, bool keep, cplx* stage, cplx (&g)[UPD_EPT]) {
  __shared__ cplx s_w[UPD_WC][4];
  const int dim = DIM ? DIM : rdim;
  const unsigned tid = threadIdx.x, nt = blockDim.x, w0 = tid & ~31u;
  int S[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) S[k] = s_S[k];
  // W's entries of G first, the columns' copies behind them
  const int l = tid & 3, part = (tid >> 2) & 1, kw = (tid >> 3) & 3;
  cplx x0 = mk(0.0);
  if (l < dim && sh.c0 + (int)(tid >> 5) <= sh.c1) x0 = ldg_c(gcur + s_S[l] + (size_t)ns * (sh.c0 + (tid >> 5)));
  if (stage) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < dim)
        for (unsigned r = tid; r < (unsigned)ns; r += nt)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                           (uint32_t)__cvta_generic_to_shared(stage + (size_t)k * ns + r)),
                       "l"(gcur + r + (size_t)ns * S[k])
                       : "memory");
  }
  for (int cb = sh.c0; cb <= sh.c1; cb += UPD_WC) {
    const int ncb = min(UPD_WC, sh.c1 - cb + 1);
    // W(k, col) = sum_l T(k, l) (delta - G)(S_l, col): item (col, k, component), four lanes l each
    for (int it = tid; it < ncb * 32; it += nt) {
      const int col = cb + (it >> 5);
      double v = 0.0;
      if (l < dim && kw < dim) {
        const int sl = s_S[l];
        cplx x = (cb == sh.c0 && it == (int)tid) ? x0 : ldg_c(gcur + sl + (size_t)ns * col);
        x = cneg(x);
        if (sl == col) x.x += 1.0;
        v = cfma_part(s_T[kw + 4 * l], x, 0.0, part);
      }
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (l == 0) st_part(&s_w[it >> 5][kw], part, v);
    }
    if (stage && cb == sh.c0) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const unsigned lo = max((unsigned)cb * ns, sh.e0), hi = min((unsigned)(cb + ncb) * ns, sh.e1);
    for (unsigned eb = lo; eb < hi; eb += UPD_EPT * nt) {
      if (!keep) {
#pragma unroll
        for (int q = 0; q < UPD_EPT; ++q)
          if (eb + w0 + q * nt < hi) g[q] = ldg_c(gcur + min(eb + tid + q * nt, hi - 1));
      }
#pragma unroll
      for (int q = 0; q < UPD_EPT; ++q) {
        if (eb + w0 + q * nt >= hi) break;   // the whole warp is past the share
        const unsigned e = min(eb + tid + q * nt, hi - 1);
        const int c = (int)(e / ns), r = (int)(e - (unsigned)c * ns);
        const cplx* w = s_w[c - cb];
        cplx gs[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < dim) gs[k] = stage ? stage[(size_t)k * ns + r] : ldg_c(gcur + r + (size_t)ns * S[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < dim) g[q] = cfma(gs[k], w[k], g[q]);
        if (eb + tid + q * nt < hi) gnext[e] = g[q];
      }
    }
    __syncthreads();   // s_w is rewritten
  }
}

template <int DIM>   // plaquette dimension, 0: at run time
__global__ void __launch_bounds__(256) k_update(DevModel M, DevScalars* sc, UpdCtl* ctl, UpdSync* sync, PlaqPre* pre,
                                                 double* field, cplx* expkv, cplx* expkv_inv, cplx* gA,
                                                 cplx* gB, int pf, int t, int staged) {
  cg::grid_group grid = cg::this_grid();
  extern __shared__ cplx upd_dyn[];   // G(:,S) of the move being applied
  const int ns = M.ns, dim = DIM ? DIM : M.pf_dim[pf], npla = M.pf_npla[pf], pd = M.pdim;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ppb = blockDim.x >> 6;   // plaquettes a CTA prepares at a time, at most
  const unsigned seq0 = ld_acquire(&sync->seq), arr0 = ld_acquire(&sync->arrived), done0 = ld_acquire(&sync->done);

  // ---- the family's ran2 stream: every CTA draws all of it (a chain of
  //      integer steps) and keeps its own plaquettes' numbers ---------------
  Ran2Dev rng;
  if (tid == 0) {
    rng.iran = sc->rng[0]; rng.jran = sc->rng[1]; rng.kran = sc->rng[2];
    rng.mran = sc->rng[3]; rng.nran = sc->rng[4];
    for (int p = 0; p < npla; ++p) {
      const bool mine = p % gridDim.x == blockIdx.x;
      if (M.proposal_kind == PQMC_PROPOSAL_GAUSSIAN) {
        const float u1 = rng.next(), u2 = rng.next();
        if (mine) {
          pre[p].xnew = (double)u1;
          pre[p].dE = (double)u2;
        }
      } else {
        const float u = rng.ran_sysm();              // :84
        if (mine) pre[p].xnew = (double)u;
      }
      const float r = rng.next();                    // :117
      if (mine) pre[p].r = (double)r;
    }
  }
  __syncthreads();

  // ---- phase 1: proposals of all plaquettes in parallel -------------------
  {
    const bool closed = (M.expkv_kind != PQMC_EXPKV_GENERAL);
    __shared__ double s_jump[8];
    // one plaquette per CTA while they last: two warps on SM quarters of their
    // own (four plaquettes in one CTA: 38.6k cycles of a family's 103k at 4x4; one
    // and with nothing formed twice 20.5k, the exponentials of one plaquette)
    for (int p0 = blockIdx.x; p0 < npla; p0 += gridDim.x * ppb) {
      if (p0 != blockIdx.x) __syncthreads();   // s_jump is read
      const int p = p0 + (warp >> 1) * gridDim.x;
      const bool on = p < npla;
      double jump = 0.0, xnew = 0.0;
      int b = 0;
      if (on) {
        b = M.bf[p + M.max_pla * pf];
        // pqmc_bm_gauss_jump's two factors, a warp each (bit-identical with the oracle)
        if (M.proposal_kind == PQMC_PROPOSAL_GAUSSIAN)
          s_jump[warp] = warp & 1 ? pqmc_bm_cos2pi(pre[p].dE) : PQMC_BM_SQRT(PQMC_BM_MUL(-2.0, pqmc_bm_log(pre[p].xnew)));
        else
          jump = M.jump * pre[p].xnew;
      }
      __syncthreads();   // both warps of a plaquette have read its draws
      if (on) {
        if (M.proposal_kind == PQMC_PROPOSAL_GAUSSIAN)
          jump = PQMC_BM_MUL(M.jump, PQMC_BM_MUL(s_jump[warp & ~1], s_jump[warp | 1]));
        xnew = field[b + (size_t)M.n_bf * t] + jump;                // :92
      }
      if (on && (warp & 1)) {
        const double dE = -M.delt * energy_diff(M, field, b, t, jump);  // :87-88
        const double thr = accept_threshold(M, dE, pre[p].r);
        if (lane == 0) {
          pre[p].dE = dE;
          pre[p].thr = thr;
          pre[p].xnew = xnew;
        }
      } else if (on) {
        double norm = 0.0, ch = 0.0, sh = 0.0;
        if (closed) {
          norm = closed_norm_warp(M, pf, xnew, lane);
          ch = cosh(norm);
          sh = sinh(norm);
        } else {
          if (lane < 2) dev_get_expkv(M, pf, p, xnew, lane == 1, lane ? pre[p].einv : pre[p].enew);
          __syncwarp();
        }
        const int i = lane % dim, j = lane / dim;
        const bool act = lane < dim * dim;
        cplx en = mk(0.0);
        if (act) {
          if (closed) {
            en = closed_entry(M, pf, p, xnew, false, i, j, norm, ch, sh);
            pre[p].enew[lane] = en;
            // the inverse: the off-diagonal blocks with the other sign (entries outside them are 0)
            pre[p].einv[lane] = i == j || (en.x == 0.0 && en.y == 0.0) ? en : cneg(en);
          } else {
            en = pre[p].enew[lane];
          }
        }
        __syncwarp();
        // Delta = expKV_inv(old) * expKV(new) - I   :240-243
        const size_t base = M.kv_base(p, pf, t);
        cplx a = mk(0.0);
        for (int k = 0; k < dim; ++k) {
          cplx ekj = shfl_c(en, k + dim * j);
          if (act) a = cfma(expkv_inv[base + i + pd * k], ekj, a);
        }
        if (act) {
          if (i == j) a = csub(a, mk(1.0));
          pre[p].delta[lane] = a;
        }
      }
    }
  }
  grid.sync();

  // ---- phase 2: sequential Metropolis scan + distributed rank-dim updates ---
  __shared__ int s_sites[4 * 512];
  __shared__ PropBuf s_buf[UPD_SPEC];
  __shared__ cplx s_tp[16];   // T of the pending move
  __shared__ int s_dec[UPD_SPEC], s_Sp[4], s_found[2], s_moves;
  __shared__ cplx s_bdet[2];   // determinants of the last two moves
  if (blockIdx.x == 0) {
    for (int e = tid; e < npla * dim && e < 4 * 512; e += blockDim.x)
      s_sites[e] = M.site[(e % dim) + pd * ((e / dim) + M.max_pla * pf)];
    if (tid == 0) {   // every CTA has read the stream's state
      sc->rng[0] = rng.iran; sc->rng[1] = rng.jran; sc->rng[2] = rng.kran;
      sc->rng[3] = rng.mran; sc->rng[4] = rng.nran;
    }
  }
  __syncthreads();
  const unsigned nw = gridDim.x - 1;
  int moves = 0;   // accepted moves: G ends in gA when even
  if (blockIdx.x != 0) {
    // ---- the other CTAs: apply move after move -----------------------------
    __shared__ int s_p, s_S[4];
    __shared__ cplx s_T[16];
    const unsigned total = (unsigned)ns * ns;   // 32-bit: Ns^2 entries fit, and 64-bit divisions cost more than loads
    const unsigned chunk = (total + nw - 1) / nw;
    Share sh;
    sh.e0 = min((blockIdx.x - 1) * chunk, total);
    sh.e1 = min(sh.e0 + chunk, total);
    sh.c0 = (int)(sh.e0 / ns);
    sh.c1 = sh.e1 > sh.e0 ? (int)((sh.e1 - 1) / ns) : sh.c0 - 1;
    const bool keep = chunk <= UPD_EPT * blockDim.x && sh.c1 - sh.c0 < UPD_WC;
    cplx g[UPD_EPT];
#pragma unroll
    for (int q = 0; q < UPD_EPT; ++q) {
      const unsigned e = sh.e0 + tid + q * blockDim.x;
      g[q] = keep && e < sh.e1 ? ldg_c(gA + e) : mk(0.0);
    }
    for (;;) {
      const UpdCtl* cr = ctl + (moves & 1);
      if (warp == 0) {   // the move's record, then everyone's arrival for the one before
        int p = -2;
        if (lane == 0 && wait_count(&sync->seq, seq0, (unsigned)moves + 1)) p = __ldcg(&cr->p);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= 0) {
          if (lane < 16) s_T[lane] = ldg_c(&cr->T[lane]);
          if (lane < 4) s_S[lane] = lane < dim ? __ldcg(&cr->S[lane]) : -1;
          if (lane == 0 && !wait_count(&sync->done, done0, (unsigned)moves)) p = -2;
        }
        if (lane == 0) {
          if (p == -2) atomicExch(&sc->lin_err, PQMC_ERR_TIMEOUT);
          s_p = p;
        }
      }
      __syncthreads();
      if (s_p < 0) break;
      apply_move<DIM>(ns, dim, s_S, s_T, moves & 1 ? gB : gA, moves & 1 ? gA : gB, sh, keep, staged ? upd_dyn : nullptr, g);
      ++moves;
      if (tid == 0) {   // after the barrier that ends apply_move
        fence_gpu();
        if (atomicAdd(&sync->arrived, 1u) - arr0 == (unsigned)moves * nw - 1u) {   // the last of the nw for this move
          fence_gpu();
          asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(&sync->done), "r"(done0 + (unsigned)moves) : "memory");
        }
      }
    }
  } else {
    // ---- CTA 0: the Markov walk ---------------------------------------------
    // ln_cw += log(real(R_elec)) per accept (:142), kept as a product
    // mantissa * 2^expo and logged once at the end
    double lprod = 1.0;
    long long lexp = 0;
    long long na = 0;
    int next = 0, prev = -1;
    const int i4 = lane & 3, j4 = (lane >> 2) & 3, part = lane >> 4;   // a real component of entry (i4, j4)
    const bool act = i4 < dim && j4 < dim;
    const int at = i4 + 4 * j4;
    while (warp <= UPD_SPEC) {
      UpdCtl* cw = ctl + (moves & 1);
      const bool has_prev = moves > 0;
      const cplx* gcur = moves > 0 && !(moves & 1) ? gB : gA;   // G before the pending move
      if (warp < UPD_SPEC) {
        PropBuf& B = s_buf[warp];
        // G before the pending move is what the move before it left
        bool ok = true;
        if (moves > 1) {
          if (lane == 0) ok = wait_count(&sync->done, done0, (unsigned)(moves - 1));
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok && lane == 0) atomicExch(&sc->lin_err, PQMC_ERR_TIMEOUT);   // whichever warp publishes
        }
        int found = -1, win = 0;
        for (int p0 = next; p0 < npla && found < 0; p0 += UPD_SPEC) {
          const int p = p0 + warp;
          int dec = 0;
          cplx det = mk(0.0);
          if (p < npla) {
            const int* Sp = s_sites + p * dim;
            const PlaqPre* pp = pre + p;
            // one round trip: G(S,S), G(S,S') and G(S',S) of the pending move, Delta
            double g0 = 0.0, g1 = 0.0, g2 = 0.0, dl = 0.0;
            if (act) {
              g0 = ldg_part(gcur + Sp[i4] + (size_t)ns * Sp[j4], part);
              if (has_prev) {
                g1 = ldg_part(gcur + Sp[i4] + (size_t)ns * s_Sp[j4], part);
                g2 = ldg_part(gcur + s_Sp[i4] + (size_t)ns * Sp[j4], part);
              }
              dl = ldg_part(&pp->delta[i4 + dim * j4], part);
            }
            const double thr = __ldcg(&pp->thr);
            st_part(&B.g1[at], part, g1);
            st_part(&B.g2[at], part, -g2);   // (I - G)(S',S): the family's plaquettes share no site
            st_part(&B.d[at], part, dl);
            __syncwarp();
            double g = g0;
            if (has_prev) {   // + G(S,S') T (I - G)(S',S)
              double a = 0.0;
              if (act)
#pragma unroll
                for (int k = 0; k < dim; ++k) a = cfma_part(B.g1[i4 + 4 * k], s_tp[k + 4 * j4], a, part);
              st_part(&B.w[at], part, a);
              __syncwarp();
              if (act)
#pragma unroll
                for (int k = 0; k < dim; ++k) g = cfma_part(B.w[i4 + 4 * k], B.g2[k + 4 * j4], g, part);
              __syncwarp();
            }
            st_part(&B.w[at], part, g);
            __syncwarp();
            // R = I + g_h_sub * Delta    :97-100
            double r = (i4 == j4 && !part) ? 1.0 : 0.0;
            if (act)
#pragma unroll
              for (int k = 0; k < dim; ++k) r = cfma_part(B.w[i4 + 4 * k], B.d[k + 4 * j4], r, part);
            if (DIM == 4) {
              st_part(&B.r[at], part, r);
              __syncwarp();
              // the 2x2 minors of rows 0,1 (six) and of rows 2,3 (six), a real component per lane
              const int q = lane % 12, c = lane / 12;
              if (c < 2) {
                const int pr = q % 6, ro = q < 6 ? 0 : 2;
                const int ja = pr < 3 ? 0 : pr < 5 ? 1 : 2, jb = pr < 3 ? pr + 1 : pr < 5 ? pr - 1 : 3;
                const cplx u = B.r[ro + 4 * ja], v = B.r[ro + 1 + 4 * jb], x = B.r[ro + 4 * jb], y = B.r[ro + 1 + 4 * ja];
                st_part(&B.min[q], c, cfma_part(u, v, -cfma_part(x, y, 0.0, c), c));
              }
              __syncwarp();
              // det = sum over the column pairs of the complementary minors' products, with sign
              const int dq = lane & 7, dc = (lane >> 3) & 1;
              double dt = 0.0;
              if (dq < 6) {
                dt = cfma_part(B.min[dq], B.min[11 - dq], 0.0, dc);
                dt = flip_sign(dt, dq == 1 || dq == 4);
              }
#pragma unroll
              for (int o = 4; o > 0; o >>= 1) dt += __shfl_xor_sync(0xffffffffu, dt, o);
              det = mk(__shfl_sync(0xffffffffu, dt, 0), __shfl_sync(0xffffffffu, dt, 8));
            } else {
              if (act) st_part(&B.r[i4 + dim * j4], part, r);
              __syncwarp();
              det = warp_det(dim, B.r, lane);
            }
            dec = (det.x * det.x + det.y * det.y) >= thr;   // :112-117
          }
          if (lane == 0) s_dec[warp] = dec;
          asm volatile("bar.sync 1, %0;" ::"n"(32 * UPD_SPEC) : "memory");
          int wa = 0;
          while (wa < UPD_SPEC && !s_dec[wa]) ++wa;
          na += min(wa, npla - p0);
          if (wa < UPD_SPEC) found = p0 + wa;
          win = wa;
          if (found == p) {   // accepted :122-187: T = Delta R^-1, by the warp that holds R
            if (DIM == 4) {
              // R^-1 = adj / det; the cofactor of (i, j) along the other row of its row pair, with the
              // minors of the pair that (i, j) is not in
              const int io = i4 ^ 1, mo = i4 < 2 ? 6 : 0;
              const int c0 = j4 == 0 ? 1 : 0, c1 = j4 <= 1 ? 2 : 1, c2 = j4 == 3 ? 2 : 3;
              double cof = cfma_part(B.r[io + 4 * c0], B.min[mo + pair_index(c1, c2)], 0.0, part);
              cof = cfma_part(cneg(B.r[io + 4 * c1]), B.min[mo + pair_index(c0, c2)], cof, part);
              cof = cfma_part(B.r[io + 4 * c2], B.min[mo + pair_index(c0, c1)], cof, part);
              cof = flip_sign(cof, (i4 + j4) & 1);
              st_part(&B.g1[at], part, cof);
              // 1 / det = conj(det) / |det|^2, scaled by a power of two where the square could leave the range
              const int de = top_exp(det) - 1023;
              double rd;
              if (de > -400 && de < 400) {
                rd = flip_sign(part ? det.y : det.x, part) / (det.x * det.x + det.y * det.y);
              } else {
                const double sc = pow2i(-min(max(de, -1000), 1000));
                const cplx ds = cscale(det, sc);
                rd = flip_sign(part ? ds.y : ds.x, part) / (ds.x * ds.x + ds.y * ds.y) * sc;
              }
              const cplx rdet = mk(__shfl_sync(0xffffffffu, rd, 0), __shfl_sync(0xffffffffu, rd, 16));
              __syncwarp();
              st_part(&B.w[j4 + 4 * i4], part, cfma_part(B.g1[at], rdet, 0.0, part));
            } else {
              if (lane == 0) dev_inverse_small(dim, B.r);                      // :171
              __syncwarp();
              if (act) st_part(&B.w[at], part, part ? B.r[i4 + dim * j4].y : B.r[i4 + dim * j4].x);
            }
            __syncwarp();
            double a = 0.0;
            if (act) {
#pragma unroll
              for (int k = 0; k < dim; ++k) a = cfma_part(B.d[i4 + 4 * k], B.w[k + 4 * j4], a, part);   // :173
              st_part(&cw->T[at], part, a);
            }
            st_part(&s_tp[at], part, a);   // no proposal is being evaluated with the old one any more
            if (lane < dim) {
              cw->S[lane] = s_sites[p * dim + lane];
              s_Sp[lane] = s_sites[p * dim + lane];
            }
            if (lane == 0) s_bdet[moves & 1] = det;
          }
          if (found < 0) asm volatile("bar.sync 1, %0;" ::"n"(32 * UPD_SPEC) : "memory");   // s_dec is rewritten
        }
        next = found >= 0 ? found + 1 : npla;
        // publish, by the warp that has the move (warp 0 the end)
        if (found >= 0 ? win == warp : warp == 0) {
          __syncwarp();
          if (lane == 0) {
            // the end is published once the last move is in: the CTAs then copy G if need be
            if (found < 0) ok = wait_count(&sync->done, done0, (unsigned)moves) && ok;
            if (!ok) atomicExch(&sc->lin_err, PQMC_ERR_TIMEOUT);
            const int end = ok ? found : -1;
            s_found[moves & 1] = end;
            cw->p = end;
            fence_gpu();
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(&sync->seq), "r"(seq0 + (unsigned)moves + 1u) : "memory");
          }
        }
      } else if (prev >= 0) {
        // bookkeeping of the pending move, beside the scan: field, expKV, weight
        const PlaqPre* pp = pre + prev;
        if (lane == 0) {
          cplx relec = s_bdet[(moves + 1) & 1];
          if (M.tr_weight) relec = cmul(relec, cconj(relec));
          cplx base = relec, ac = mk(1.0);
          for (int k = 0; k < M.ncopy; ++k) ac = cmul(ac, base);
          int ex;
          lprod *= frexp(ac.x, &ex);
          lexp += ex;
          double m2 = frexp(lprod, &ex);
          lprod = m2;
          lexp += ex;
          field[M.bf[prev + M.max_pla * pf] + (size_t)M.n_bf * t] = __ldcg(&pp->xnew);
        }
        const size_t base2 = M.kv_base(prev, pf, t);
        if (lane < pd * pd) {
          const int ii = lane % pd, jj = lane / pd;
          const bool in = ii < dim && jj < dim;
          expkv[base2 + lane] = in ? ldg_c(&pp->enew[ii + dim * jj]) : mk(0.0);
          expkv_inv[base2 + lane] = in ? ldg_c(&pp->einv[ii + dim * jj]) : mk(0.0);
        }
      }
      // the walk's warps and the bookkeeping one go on together
      asm volatile("bar.sync 2, %0;" ::"n"(32 * (UPD_SPEC + 1)) : "memory");
      prev = s_found[moves & 1];
      if (prev < 0) break;
      ++moves;
    }
    if (tid == 0) sc->neg_acc += na;
    if (tid == 32 * UPD_SPEC && moves > 0) {
      double l = (lprod > 0.0) ? log(lprod) + (double)lexp * 0.69314718055994530942 : log(lprod);
      sc->ln_cw = cadd(sc->ln_cw, mk(l));
      sc->pos_acc += moves;
    }
    if (tid == 0) s_moves = moves;
    __syncthreads();
    moves = s_moves;
  }
  if (moves & 1) {
    const long total = (long)ns * ns;
    for (long e = blockIdx.x * (long)blockDim.x + tid; e < total; e += (long)gridDim.x * blockDim.x)
      gA[e] = ldg_c(gB + e);
  }
}

static const void* update_fn(int dim) { return dim == 4 ? (const void*)k_update<4> : (const void*)k_update<0>; }

int update_setup(pqmc_chain* c) {
  const long elems = (long)c->ns * c->ns;
  const long blocks = 1 + (elems + 127) / 128;
  int want = blocks < 4096 ? (int)blocks : 4096;
  int npla_max = 0;
  for (int n : c->h_pf_npla) npla_max = n > npla_max ? n : npla_max;
  if (want < (npla_max + 3) / 4) want = (npla_max + 3) / 4;
  if (want < 2) want = 2;
  for (int f = 0; f < c->n_pf; ++f)
    if (c->h_pf_npla[f] * c->h_pf_dim[f] > 4 * 512) {
      set_error("update kernel stages at most 2048 plaquette sites per family");
      return PQMC_ERR_ARG;
    }
  const size_t stage = sizeof(cplx) * 4 * (size_t)c->ns;
  c->upd_smem = stage <= UPD_STAGE ? (int)stage : 0;
  c->upd_blocks = want;
  for (int f = 0; f < c->n_pf; ++f) {
    const void* fn = update_fn(c->h_pf_dim[f]);
    PQMC_CUDA(raise_dyn_smem((const char*)fn, c->upd_smem));
    const int nb = coop_grid(fn, 256, want, c->upd_smem);
    if (nb < c->upd_blocks) c->upd_blocks = nb;
  }
  if (c->upd_blocks < 2) {
    set_error("update kernel needs two co-resident blocks");
    return PQMC_ERR_CUDA;
  }
  // no more CTAs than have entries (151 shares of Ns = 150 leave the last one
  // empty): a share without entries would pass no barrier between two moves
  const long chunk = (elems + c->upd_blocks - 2) / (c->upd_blocks - 1);
  c->upd_blocks = 1 + (int)((elems + chunk - 1) / chunk);
  return PQMC_OK;
}

int launch_update(pqmc_chain* c, int pf, int time) {
  int t = time - 1, staged = c->upd_smem > 0;
  void* args[] = {&c->M, &c->sc, &c->ctl, &c->upd_sync, &c->pre, &c->field, &c->expkv, &c->expkv_inv, &c->g, &c->g_alt, &pf, &t,
                  &staged};
  PQMC_CUDA(cudaLaunchCooperativeKernel(update_fn(c->h_pf_dim[pf]), c->upd_blocks, 256, args, c->upd_smem, c->stream));
  PQMC_LAUNCHED();
  return PQMC_OK;
}

}  // namespace pqmc
