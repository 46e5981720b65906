// adjoint.cu -- gradient of the projector log-weight
//   W(x) = Re log det(P^H B(Lt..1) P),  B(tau) = E_{n_pf}(tau) ... E_1(tau)
// with respect to every phonon field x_{b,tau}.  The value is
// cal_new_weight_T0 (src/mod_evolution.f90:359-408); the gradient is the
// Green's-function trace formula
//   dW/dx_{b,tau} = c Re Tr[E_p^-1 dE_p/dx  G_before(S_p,S_p)]
// where p is the plaquette carrying boson b in family f, G_before is the
// equal-time Green's function R'(L'R')^-1 L' positioned just before E_f(tau)
// acts (the matrix the local update at (f,tau) sees), and c = ncopy (x2 under
// TR_weight).
//
// Reverse sweep with checkpoints: one right-to-left pass gives the value
// (cal_new_weight_T0 from the trial state) and stores the orthonormal left
// factor every ngroup slices; a left-to-right pass recomputes
// G from the left checkpoint and the current right factor at each block start
// and wraps it family by family through the block (the slices between
// checkpoints are recomputed, not stored).
#include "chain.cuh"
#include "linalg.cuh"
#include "update_dev.cuh"
#include "wrap.cuh"

namespace pqmc {

// dE/dx of the closed-form propagators (get_expKV_epsocz / _epsoc /
// epsocz_block): the scalars every entry of a plaquette shares ...
struct DEscal {
  double dch, f, df;   // d cosh(n)/dx, sinh(n)/n, d(sinh(n)/n)/dx
};
__device__ __forceinline__ DEscal closed_dscal(const DevModel& M, int pf, double x) {
  const int pd = M.pdim;
  const cplx kc = M.k_coe[pf], vc = M.v_coe[pf];
  // norm(x) and dnorm/dx
  double norm, dnorm;
  if (M.expkv_kind == PQMC_EXPKV_EPSOCZ_BLOCK) {
    const cplx* K = M.kmat + (size_t)pd * pd * pf;
    const cplx* V = M.vmat + (size_t)pd * pd * pf;
    const cplx vx = cscale(vc, x);
    cplx h11 = cadd(cmul(kc, K[0 + pd * 2]), cmul(vx, V[0 + pd * 2]));
    cplx h21 = cadd(cmul(kc, K[1 + pd * 2]), cmul(vx, V[1 + pd * 2]));
    cplx d11 = cmul(vc, V[0 + pd * 2]), d21 = cmul(vc, V[1 + pd * 2]);
    double s = cabs2(h11) + cabs2(h21);
    const double rs = sqrt(s);
    norm = M.delt * rs;
    double ds = 2.0 * (h11.x * d11.x + h11.y * d11.y + h21.x * d21.x + h21.y * d21.y);
    dnorm = M.delt * ds / (2.0 * rs);
  } else {
    double a = cabsd(kc), b = cabsd(vc);
    double s = a * a + (b * x) * (b * x);
    const double rs = sqrt(s);
    norm = M.delt * rs;
    dnorm = M.delt * (b * b * x) / rs;
  }
  const double ch = cosh(norm), sh = sinh(norm);
  DEscal q;
  q.dch = sh * dnorm;
  q.f = sh / norm;
  q.df = (ch - q.f) * dnorm / norm;
  return q;
}
// ... and entry (i,j)
__device__ __forceinline__ cplx closed_dentry(const DevModel& M, int pf, int pla, double x, const DEscal& q, int i,
                                              int j) {
  const int pd = M.pdim, dim = M.pf_dim[pf];
  const cplx kc = M.k_coe[pf], vc = M.v_coe[pf];
  const cplx* K = M.kmat + (size_t)pd * pd * pf;
  const cplx* V = M.vmat + (size_t)pd * pd * pf;
  const cplx* BC = M.bcp + (size_t)pd * pd * (pla + (size_t)M.max_pla * pf);
  const bool cross = M.cross[pla + M.max_pla * pf] != 0;
  if (i == j) return mk(q.dch);
  const int h = dim / 2;
  bool upper = (i < h && j >= h), lower = (i >= h && j < h);
  if (!upper && !lower) return mk(0.0);
  int a = upper ? i : j, b = upper ? j : i;
  if (M.expkv_kind == PQMC_EXPKV_EPSOC && !(a == 0 && b == 1)) return mk(0.0);
  cplx hab = cadd(cmul(kc, K[a + pd * b]), cmul(cscale(vc, x), V[a + pd * b]));
  cplx dh = cmul(vc, V[a + pd * b]);
  cplx sub = cscale(hab, -M.delt), dsub = cscale(dh, -M.delt);
  if (cross) {
    sub = cmul(sub, BC[a + pd * b]);
    dsub = cmul(dsub, BC[a + pd * b]);
  }
  // d/dx [sub sinh(n)/n] = dsub sinh/n + sub (cosh n - sinh/n) dn / n
  cplx e = cadd(cscale(dsub, q.f), cscale(sub, q.df));
  return upper ? e : cconj(e);
}

// One family at one slice of the gradient's left-to-right pass: the trace
// terms grad(b, t) of its plaquettes from G, and the wrap of G by it
// (left_evolve).  Both read the same G and neither the other's result, so
// they share a launch: the first n_gb CTAs take the plaquettes, 16 lanes
// each, one entry of E^-1 dE per lane; the rest the wrap's pairs.  The
// plaquette part is one chain of FP64 transcendentals (sqrt, cosh, sinh,
// three divisions), formed once per plaquette on all 16 lanes at the price
// of one: a thread per plaquette that formed them again for each of its 16
// entries took 84 us a family at 10x10 and 69 at 4x4.
__global__ void __launch_bounds__(WRAP_THREADS) k_grad_wrap(
    DevModel M, int pf, int t, int n_gb, const double* __restrict__ field, double* grad, double scale, int n_items,
    const int* __restrict__ ipla, const int* __restrict__ isites, const int* __restrict__ idim,
    const cplx* __restrict__ expkv, const cplx* __restrict__ expkv_inv, const cplx* __restrict__ G,
    cplx* __restrict__ gout) {
  if ((int)blockIdx.x >= n_gb) {
    wrap_pair(M, pf, t, 1, n_items, ipla, isites, idim, expkv, expkv_inv, G, gout, (int)blockIdx.x - n_gb);
    return;
  }
  __shared__ cplx s_pm[WRAP_PAIRS][2][16];   // E at x + h and x - h (general form)
  const int grp = threadIdx.x >> 4, lane = threadIdx.x & 31, sl = lane & 15, base = lane & 16;
  const int p = (int)blockIdx.x * WRAP_PAIRS + grp;
  const bool on = p < M.pf_npla[pf];
  const int dim = M.pf_dim[pf], pd = M.pdim, ns = M.ns;
  const int i = sl % dim, j = sl / dim;
  const bool act = on && sl < dim * dim;
  const int b = on ? M.bf[p + M.max_pla * pf] : 0;
  const double x = on ? field[b + (size_t)M.n_bf * t] : 0.0;
  // G(S_j, S_i) and row i of E^-1, in flight during the scalars
  cplx g = mk(0.0), ei[4];
  if (act) g = G[M.site[j + pd * (p + M.max_pla * pf)] + (size_t)ns * M.site[i + pd * (p + M.max_pla * pf)]];
#pragma unroll
  for (int k = 0; k < 4; ++k) ei[k] = (act && k < dim) ? expkv_inv[M.kv_base(p, pf, t) + i + pd * k] : mk(0.0);
  cplx de = mk(0.0);
  if (M.expkv_kind == PQMC_EXPKV_GENERAL) {   // central difference of the exponential, one side per lane
    const double h = 1e-5 * (1.0 + fabs(x));
    if (on && sl < 2) dev_get_expkv(M, pf, p, sl ? x - h : x + h, false, s_pm[grp][sl]);
    __syncwarp();
    if (act) de = cscale(csub(s_pm[grp][0][sl], s_pm[grp][1][sl]), 0.5 / h);
  } else if (on) {
    const DEscal q = closed_dscal(M, pf, x);
    if (act) de = closed_dentry(M, pf, p, x, q, i, j);
  }
  __syncwarp();
  // Tr[E^-1 dE G(S,S)] = sum_ij (E^-1 dE)_ij G(S_j, S_i)
  cplx a = mk(0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const cplx dk = shfl_c(de, base + k + dim * j);
    if (k < dim) a = cfma(ei[k], dk, a);
  }
  double tr = act ? fma(a.x, g.x, -(a.y * g.y)) : 0.0;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
  if (on && sl == 0) grad[b + (size_t)M.n_bf * t] = scale * tr;
}

static int launch_grad_wrap(pqmc_chain* c, int pf, int tau, double* grad, double scale) {
  const int npla = c->h_pf_npla[pf];
  if (npla == 0 || !c->h_pf_v_exist[pf]) return launch_wrap(c, pf, tau, true);
  const WrapItems& w = c->wrap[pf];
  const int n_gb = (npla + WRAP_PAIRS - 1) / WRAP_PAIRS;
  k_grad_wrap<<<n_gb + wrap_blocks(w.n_items), WRAP_THREADS, 0, c->stream>>>(
      c->M, pf, tau - 1, n_gb, c->field, grad, scale, w.n_items, w.d_pla, w.d_sites, w.d_dim, c->expkv, c->expkv_inv,
      c->g, c->g_alt);
  PQMC_LAUNCHED();
  cplx* t = c->g;
  c->g = c->g_alt;
  c->g_alt = t;
  return PQMC_OK;
}

}  // namespace pqmc

using namespace pqmc;

extern "C" int pqmc_cal_new_weight(pqmc_chain* c, double* ln_cw_out);

extern "C" int pqmc_set_field_device(pqmc_chain* c, const double* dfield) {
  if (!c || !dfield) { set_error("set_field_device: null argument"); return PQMC_ERR_ARG; }
  PQMC_CUDA(cudaMemcpyAsync(c->field, dfield, sizeof(double) * (size_t)c->n_bf * c->ntime, cudaMemcpyDeviceToDevice,
                            c->stream));
  PQMC_CUDA(cudaStreamSynchronize(c->stream));
  return PQMC_OK;
}

// logw_out: host, 2 doubles (complex log-weight as cal_new_weight_T0);
// grad_dev: device, (n_bf, ntime) doubles (gradient of Re logw).
extern "C" int pqmc_logweight_grad(pqmc_chain* c, double* logw_out, double* grad_dev) {
  if (!c || !grad_dev) { set_error("logweight_grad: null argument"); return PQMC_ERR_ARG; }
  if (c->finite_t) { set_error("logweight_grad: the projector log-weight only (the chain is at finite temperature)"); return PQMC_ERR_STATE; }
  const int ns = c->ns, ne = c->nelec, nt = c->ntime, ng = c->ngroup;
  cudaStream_t s = c->stream;
  const size_t qb = sizeof(cplx) * (size_t)ns * ne;
  const int nck = nt / ng + 1;
  cplx* ck = nullptr;
  PQMC_CUDA(cudaMallocAsync((void**)&ck, qb * nck, s));
  // right-to-left pass: cal_new_weight_T0 with the orthonormal left factor
  // checkpointed every ngroup slices (one propagation for value and
  // checkpoints)
  int st = do_new_weight_ck(c, ck);
  int info = 0;
  DevScalars h;
  if (st == PQMC_OK && (cudaMemcpyAsync(&h, c->sc, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                        cudaStreamSynchronize(s) != cudaSuccess)) {
    set_error("logweight_grad: reading the weight failed");
    st = PQMC_ERR_CUDA;
  }
  if (st == PQMC_OK) info = h.lu_info;
  if (st == PQMC_OK && h.lin_err != 0) st = check_factor(c, "logweight_grad");
  if (st == PQMC_OK && info != 0) {
    set_error("logweight_grad: zero pivot %d", info);
    st = PQMC_ERR_SINGULAR;
  }
  if (st != PQMC_OK) {
    cudaFreeAsync(ck, s);
    return st;
  }
  if (logw_out) {
    logw_out[0] = h.ln_cw.x;
    logw_out[1] = h.ln_cw.y;
  }
  // forward pass: R starts as the trial state; at each block start G from the checkpoint
  PQMC_CUDA(cudaMemcpyAsync(c->rmat, c->slater_q, qb, cudaMemcpyDeviceToDevice, s));
  const double scale = (double)c->M.ncopy * (c->M.tr_weight ? 2.0 : 1.0);
  cplx* gsave = c->g;   // keep the chain's G: compute into the pair (g, g_alt) then restore
  cplx* gsave_alt = c->g_alt;
  cplx* gtmp = nullptr;
  PQMC_CUDA(cudaMallocAsync((void**)&gtmp, sizeof(cplx) * (size_t)ns * ns, s));
  PQMC_CUDA(cudaMemcpyAsync(gtmp, c->g, sizeof(cplx) * (size_t)ns * ns, cudaMemcpyDeviceToDevice, s));
  PQMC_CUDA(cudaMemsetAsync(grad_dev, 0, sizeof(double) * (size_t)c->n_bf * nt, s));
  for (int t0 = 0; t0 < nt; t0 += ng) {
    const int t1 = (t0 + ng < nt) ? t0 + ng : nt;
    // G = R (L R)^-1 L with L = ck[slot]^H, slot = t1/ng (left part covers slices > t1)... the
    // left factor that pairs with R at tau = t0 is the checkpoint at t0
    const cplx* Xl = ck + (size_t)ns * ne * (t0 / ng);
    PQMC_TRY(zgemm(s, 'C', 'N', ne, ne, ns, mk(1.0), Xl, ns, c->rmat, ns, mk(0.0), c->pbp, ne));
    PQMC_TRY(herm_t(s, ns, ne, Xl, c->lmat));
    PQMC_TRY(lu_solve(s, ne, c->pbp, ns, c->lmat, ne, c->lcol, c->ipiv, &c->sc->lu_info, c->g_alt, &c->sc->lin_err));
    PQMC_TRY(zgemm(s, 'N', 'N', ns, ns, ne, mk(1.0), c->rmat, ns, c->lmat, ne, mk(0.0), c->g, ns));
    for (int tau = t0 + 1; tau <= t1; ++tau) {
      for (int pf = 0; pf < c->n_pf; ++pf) PQMC_TRY(launch_grad_wrap(c, pf, tau, grad_dev, scale));
    }
    PQMC_TRY(launch_propagate(c, c->rmat, ne, t0 + 1, t1, true));
    if (t1 < nt) PQMC_TRY(house_qr(s, ns, ne, c->rmat, c->dtmp, c->g_alt, &c->sc->lin_err));
  }
  // restore the chain's Green's function
  c->g = gsave;
  c->g_alt = gsave_alt;
  PQMC_CUDA(cudaMemcpyAsync(c->g, gtmp, sizeof(cplx) * (size_t)ns * ns, cudaMemcpyDeviceToDevice, s));
  PQMC_CUDA(cudaFreeAsync(gtmp, s));
  PQMC_CUDA(cudaFreeAsync(ck, s));
  return check_waits(c, "logweight_grad");
}
