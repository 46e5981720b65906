// wrap.cuh -- the FP64 two-way wrap of G by one family, shared by the chain's
// wrap (chain.cu) and the gradient's wrap with its trace terms (adjoint.cu).
#pragma once
#include "chain.cuh"
#include "update_dev.cuh"

namespace pqmc {

constexpr int WRAP_THREADS = 128;               // 8 pairs of cover items per CTA
constexpr int WRAP_PAIRS = WRAP_THREADS / 16;

inline int wrap_blocks(int n_items) {
  return (int)(((long)n_items * n_items + WRAP_PAIRS - 1) / WRAP_PAIRS);
}

// One pair (row item, column item) per 16 lanes, one entry of its block per
// lane: h = A g, then h B, each a sum of up to four products in k order, the
// operands of the other lanes by shuffles.  Bound by the FP64 pipe (8 complex
// multiply-adds an entry; a warp instruction holds an SM quarter for ~32 ns
// whatever its lanes), so what matters is that every quarter has warps: a
// thread per pair (16 entries, 512 FP64 instructions in a row) left half of
// the quarters idle at Ns = 392 and ran a 4x4 lattice on two warps.
__device__ __forceinline__ void wrap_pair(const DevModel& M, int pf, int t, int left, int n_items,
                                          const int* __restrict__ ipla, const int* __restrict__ isites,
                                          const int* __restrict__ idim, const cplx* __restrict__ expkv,
                                          const cplx* __restrict__ expkv_inv, const cplx* __restrict__ gin,
                                          cplx* __restrict__ gout, int block) {
  const int lane = threadIdx.x & 31, sl = lane & 15, base = lane & 16;
  const int a = sl & 3, b = sl >> 2;
  const long pair = (long)block * WRAP_PAIRS + (threadIdx.x >> 4);
  const bool on = pair < (long)n_items * n_items;
  const int ir = on ? (int)(pair % n_items) : 0, ic = on ? (int)(pair / n_items) : 0;
  const int ns = M.ns, pd = M.pdim;
  const int dr = idim[ir], dc = idim[ic];
  const bool act = on && a < dr && b < dc;
  const size_t at = act ? isites[4 * ir + a] + (size_t)ns * isites[4 * ic + b] : 0;
  const int pr = ipla[ir], pc = ipla[ic];
  cplx g = mk(0.0), am[4], bm[4];
  if (act) g = gin[at];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    am[k] = bm[k] = mk(0.0);
    if (act && pr >= 0 && k < dr) am[k] = ((left ? expkv : expkv_inv) + M.kv_base(pr, pf, t))[a + pd * k];
    if (act && pc >= 0 && k < dc) bm[k] = ((left ? expkv_inv : expkv) + M.kv_base(pc, pf, t))[k + pd * b];
  }
  cplx h = mk(0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const cplx gk = shfl_c(g, base + k + 4 * b);
    if (k < dr) h = cfma(am[k], gk, h);
  }
  if (pr < 0) h = g;
  cplx o = mk(0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const cplx hk = shfl_c(h, base + a + 4 * k);
    if (k < dc) o = cfma(hk, bm[k], o);
  }
  if (pc < 0) o = h;
  if (act) gout[at] = o;
}

}  // namespace pqmc
