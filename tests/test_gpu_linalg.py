"""The FP64 factorisations at the edges of their column pipeline: fewer rows
than threads, exactly a block of 128 and one past it, one and two columns
per CTA, and right-hand sides beside the factored columns.

Tolerances: backward-stable factorisations of matrices of condition ~10, so
errors are a small multiple of eps * n; 1e-11 leaves two orders of room at
the largest size.
"""
import ctypes
from dataclasses import replace

import numpy as np
import pytest

from pqmc_allinone_gb300 import model as M
from tests.helpers import SEED_WORDS, epsocz_small, general_bond_model, rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,ne", [(1, 1), (2, 1), (5, 3), (64, 31), (128, 127), (200, 128), (257, 129), (392, 196), (512, 256)])
def test_lu_solve_through_the_allocation_free_entry(ns, ne):
    """G = R (X^H R)^-1 X^H and log det(X^H R) against numpy."""
    torch = pytest.importorskip("torch")
    from pqmc_allinone_gb300.abi import load_library
    rng = np.random.default_rng(1000 * ns + ne)

    def orth():
        return np.linalg.qr(rng.normal(size=(ns, ne)) + 1j * rng.normal(size=(ns, ne)))[0]

    x = orth()
    r = x @ (rng.permutation(np.eye(ne)) * np.exp(1j * rng.uniform(0, 6, ne))) + 0.2 * orth()
    lib = load_library()
    fn = lib.pqmc_cal_g_and_det_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3
    fn.restype = ctypes.c_int
    dev = [torch.from_numpy(np.asfortranarray(a).ravel(order="F").view(np.float64).copy()).cuda() for a in (x, r)]
    g_d = torch.zeros(2 * ns * ns, dtype=torch.float64, device="cuda")
    ld_d = torch.zeros(2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert fn(dev[0].data_ptr(), dev[1].data_ptr(), ns, ne, g_d.data_ptr(), ld_d.data_ptr(), None) == 0, lib.pqmc_last_error()
    g = g_d.cpu().numpy().view(np.complex128).reshape((ns, ns), order="F")
    lr = x.conj().T @ r
    assert rel_fro(g, r @ np.linalg.solve(lr, x.conj().T)) < 1e-11
    sign, logabs = np.linalg.slogdet(lr)
    ld = ld_d.cpu().numpy()
    assert abs(ld[0] - logabs) < 1e-11 * max(1.0, ne)
    assert abs(np.exp(1j * ld[1]) - sign) < 1e-10


def test_singular_matrix_is_reported():
    torch = pytest.importorskip("torch")
    from pqmc_allinone_gb300.abi import load_library
    lib = load_library()
    x = torch.zeros(2 * 6 * 3, dtype=torch.float64, device="cuda")
    out = torch.zeros(2 * 6 * 6 + 2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    fn = lib.pqmc_cal_g_and_det_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3
    fn.restype = ctypes.c_int
    assert fn(x.data_ptr(), x.data_ptr(), 6, 3, out.data_ptr(), out[72:].data_ptr(), None) == 3   # PQMC_ERR_SINGULAR


@pytest.mark.parametrize("L", [(4, 4), (4, 6), (8, 8), (6, 12), (12, 14)])
def test_qr_strings_against_the_oracle(L):
    """Q and D of every block (zgeqrf's signs): Ns = 32 .. 336, nelec = 16 .. 168."""
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    m, f = epsocz_small(L=L, ntime=20, ngroup=10, alpha=0.3)
    o = OracleChain(m, field=f, seed_words=SEED_WORDS, meas=False)
    g = PqmcChain(m, field=f, rng_words=SEED_WORDS)
    for c in (o, g):
        c.init_expkv()
        c.init_g(1)
    for blk in range(1, m.nblock + 1):
        (qo, do), (qg, dg) = o.qd(blk), g.qd(blk)
        assert rel_fro(qg, qo) < 1e-10 and np.allclose(dg, do, rtol=1e-10, atol=1e-12), blk
    assert rel_fro(g.g(), o.g()) < 1e-10


def test_square_qr_with_two_columns_per_cta():
    """Finite temperature at Ns = 320: 320 columns, R and det Q returned."""
    from oracle.finite_t import dense_g_and_weight
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    m, f = epsocz_small(L=(10, 16), ntime=10, ngroup=5, alpha=0.3)
    o = OracleChain(m, field=f, seed_words=SEED_WORDS, meas=False)
    o.init_expkv()
    g = PqmcChain(m, field=f, rng_words=SEED_WORDS)
    g.set_temperature(False)
    g.init_expkv()
    g.init_g(1)
    gd, ld = dense_g_and_weight(o)
    assert rel_fro(g.g(), gd) < 1e-10
    assert abs(g.state()["ln_cw"].real - ld.real) <= 1e-9 * abs(ld.real)


@pytest.mark.parametrize("L", [(4, 6), (6, 6), (10, 10), (12, 18)])
def test_update_shares(L):
    """Rank-dim updates of G by shares of the entries: a few CTAs, all of
    them, entries kept in registers (Ns <= 393) and read again (Ns = 432)."""
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    m, f = epsocz_small(L=L, ntime=10, ngroup=5, alpha=0.3)
    o = OracleChain(m, field=f, seed_words=SEED_WORDS, meas=False)
    g = PqmcChain(m, field=f, rng_words=SEED_WORDS)
    for c in (o, g):
        c.init_expkv()
        c.init_g(1)
    for pf in (4, 3):
        for c in (o, g):
            c.right_evolve_g(m.ntime, pf)
            c.update_phonon_field(pf, m.ntime)
        so, sg = o.state(), g.state()
        assert sg["rng"] == so["rng"] and np.array_equal(g.field(), o.field())
        assert sg["positive_accept"] == so["positive_accept"] > 0
        assert rel_fro(g.g(), o.g()) < 1e-10


@pytest.mark.parametrize("build,L", [(epsocz_small, (12, 12)), (general_bond_model, 12), (epsocz_small, (16, 16))])
def test_propagation_in_passes(build, L):
    """Families of 72 and 128 plaquettes of four and two sites: more items than
    the CTA has lanes, with and without a remainder, in both directions."""
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    m, f = build(L=L, ntime=4, ngroup=2, lam=0.8)
    o = OracleChain(m, field=f, seed_words=SEED_WORDS, meas=False)
    g = PqmcChain(m, field=f, rng_words=SEED_WORDS, meas=False)
    for c in (o, g):
        c.init_expkv()
    for t in (1, 3):   # through every slice from the right, and from both sides
        for c in (o, g):
            c.init_g(t)
        assert rel_fro(g.g(), o.g()) < 1e-11
    g.close()


def _families_cut(keep, L=(4, 6)):
    """epsocz_small with family keep[i][0] cut to its first keep[i][1] plaquettes, in that order."""
    m, f = epsocz_small(L=L, ntime=4, ngroup=2, lam=0.8)
    pfs = [m.spec.pfs[k] for k, _ in keep]
    m = M.build_model(replace(m.spec, pfs=pfs), twist_seed=7, twist=1e-3)
    m.pf = [M.PfTables(t.dim, min(n, t.n_pla), t.site_list[:n], t.crossing[:n], t.bc_phases[:n], t.bf_list[:n])
            for t, (_, n) in zip(m.pf, keep)]
    return m, f


@pytest.mark.parametrize("L,keep", [((4, 6), [(0, 0), (0, 99), (1, 99), (2, 99), (3, 99)]),      # the first family empty
                                    ((4, 6), [(0, 99), (1, 99), (1, 0), (1, 0), (2, 99), (3, 99)]),   # two in the middle
                                    ((4, 6), [(0, 99), (1, 99), (2, 99), (3, 99), (0, 0)]),      # the last
                                    ((4, 6), [(0, 0), (1, 0)]),                                  # all
                                    ((12, 12), [(0, 99), (1, 3), (1, 0), (2, 99), (3, 65), (0, 0)])])   # and uneven ones
def test_families_without_plaquettes(L, keep):
    """Families of no plaquettes, and of different numbers, through every slice
    in both directions; their slices leave the factors as they are."""
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    m, f = _families_cut(keep, L)
    o = OracleChain(m, field=f, seed_words=SEED_WORDS, meas=False)
    g = PqmcChain(m, field=f, rng_words=SEED_WORDS, meas=False)
    for c in (o, g):
        c.init_expkv()
    for t in (1, 3):
        for c in (o, g):
            c.init_g(t)
        assert rel_fro(g.g(), o.g()) < 1e-11
    g.close()


def test_lu_solve_sums_terms_apart(ns=392, ne=196, tol=7.4e-15):
    """The error of G's first columns against extended precision, for a dense
    unitary X^H R.  The multiply-adds of the kernels in numpy, two roundings
    per component, give 8.6e-15 with the terms of the triangular solves added
    one after another and 6.4e-15 with sums of 16 terms; the bound is the
    geometric mean."""
    torch = pytest.importorskip("torch")
    from pqmc_allinone_gb300.abi import load_library
    rng = np.random.default_rng(ns + ne)

    def normal(a, b):
        return rng.normal(size=(a, b)) + 1j * rng.normal(size=(a, b))

    x, u = np.linalg.qr(normal(ns, ne))[0], np.linalg.qr(normal(ne, ne))[0]
    r = np.linalg.qr(x @ u + 0.3 * normal(ns, ne) / np.sqrt(2 * ns))[0]
    lib = load_library()
    fn = lib.pqmc_cal_g_and_det_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3
    fn.restype = ctypes.c_int
    dev = [torch.from_numpy(np.asfortranarray(a).ravel(order="F").view(np.float64).copy()).cuda() for a in (x, r)]
    out = torch.zeros(2 * ns * ns + 2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert fn(dev[0].data_ptr(), dev[1].data_ptr(), ns, ne, out.data_ptr(), out[2 * ns * ns:].data_ptr(), None) == 0
    g = out[:2 * ns * ns].cpu().numpy().view(np.complex128).reshape((ns, ns), order="F")
    # 16 columns of the answer: a 64-bit solve, refined with residuals in extended precision
    a, b = x.conj().T.astype(np.clongdouble) @ r.astype(np.clongdouble), x[:16].conj().T.astype(np.clongdouble)
    inv = np.linalg.inv(a.astype(np.complex128))
    y = (inv @ b.astype(np.complex128)).astype(np.clongdouble)
    for _ in range(3):
        y = y + inv @ (b - a @ y).astype(np.complex128)
    ref = r.astype(np.clongdouble) @ y
    err = float(np.linalg.norm((g[:, :16] - ref).astype(np.complex128)) / np.linalg.norm(ref.astype(np.complex128)))
    assert err < tol, err


@pytest.mark.parametrize("L", [(16, 22), (20, 22)])
def test_lu_solve_past_the_shared_memory(L):
    """Finite temperature at Ns = 704, where the substitution takes one of a
    CTA's right-hand sides at a time, and 880, where the columns stay in
    global memory."""
    from oracle.finite_t import dense_g_and_weight
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    m, f = epsocz_small(L=L, ntime=4, ngroup=2, alpha=0.3)
    o = OracleChain(m, field=f, seed_words=SEED_WORDS, meas=False)
    o.init_expkv()
    g = PqmcChain(m, field=f, rng_words=SEED_WORDS, meas=False)
    g.set_temperature(False)
    g.init_expkv()
    g.init_g(1)
    gd, ld = dense_g_and_weight(o)
    assert rel_fro(g.g(), gd) < 1e-10
    assert abs(g.state()["ln_cw"].real - ld.real) <= 1e-9 * abs(ld.real)


def test_update_without_empty_shares():
    """Ns = 150: 22500 entries in shares of 150 are one share fewer than 152 SMs have CTAs for."""
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    spec = general_bond_model(L=4)[0].spec
    pfs = [replace(spec.pfs[0], tsl=[2, 0, 0, 1], offset=[o, 0], bf_index=1) for o in (0, 1)]
    m = M.build_model(replace(spec, lat_size=[10, 15], pfs=pfs, beta=0.4, ngroup=2), twist_seed=3, twist=1e-3)
    assert m.ns == 150
    f = M.field_gaussian(m, 5)
    o = OracleChain(m, field=f, seed_words=SEED_WORDS, meas=False)
    g = PqmcChain(m, field=f, rng_words=SEED_WORDS, meas=False)
    for c in (o, g):
        c.init_expkv()
        c.init_g(1)
    for pf in (2, 1):
        for c in (o, g):
            c.right_evolve_g(m.ntime, pf)
            c.update_phonon_field(pf, m.ntime)
        so, sg = o.state(), g.state()
        assert sg["rng"] == so["rng"] and np.array_equal(g.field(), o.field())
        assert sg["positive_accept"] == so["positive_accept"] > 0
        assert rel_fro(g.g(), o.g()) < 1e-10
    g.close()


@pytest.mark.parametrize("exponent", [-1016, -500, 500, 1016])
def test_lu_solve_at_the_ends_of_the_range(exponent):
    """Pivots near 2^-1016 .. 2^1016: G = R (X^H R)^-1 X^H does not depend on
    R's scale.  Backward-stable for a unitary X^H R of order 8: a few eps n,
    below 1e-14; a reciprocal with bits lost below 2^-1022 gives 1e-13."""
    torch = pytest.importorskip("torch")
    from pqmc_allinone_gb300.abi import load_library
    n = 8
    rng = np.random.default_rng(5)
    r = np.ldexp(1.0, exponent) * np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))[0]
    lib = load_library()
    fn = lib.pqmc_cal_g_and_det_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3
    fn.restype = ctypes.c_int
    dev = [torch.from_numpy(np.asfortranarray(a).ravel(order="F").view(np.float64).copy()).cuda()
           for a in (np.eye(n, dtype=np.complex128), r)]
    out = torch.zeros(2 * n * n + 2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert fn(dev[0].data_ptr(), dev[1].data_ptr(), n, n, out.data_ptr(), out[2 * n * n:].data_ptr(), None) == 0
    o = out.cpu().numpy()
    assert rel_fro(o[:2 * n * n].view(np.complex128).reshape((n, n), order="F"), np.eye(n)) < 1e-14
    assert abs(o[-2] - n * exponent * np.log(2.0)) < 1e-11


def test_update_with_a_determinant_past_the_square_root_of_the_range():
    """A move whose |det R| is about 1e184: its square is infinite, 1 / det and the new G are not."""
    from oracle.oracle import OracleChain
    from pqmc_allinone_gb300.engine import PqmcChain
    from pqmc_allinone_gb300.rng import seed_words
    spec = general_bond_model(L=4)[0].spec
    hop = np.diag([1, 1, 1], 1) + np.diag([1, 1, 1], -1)
    pf = replace(spec.pfs[0], dim=4, tsl=[4, 0, 0, 1], offset=[0, 0], int_subsites=[0, 0, 1, 1, 0, 1, 2, 0, 1, 3, 0, 1],
                 kmat=[complex(v) for v in hop.ravel()], vmat=[complex(v) for v in np.eye(4).ravel()], bf_index=1)
    m = M.build_model(replace(spec, pfs=[pf], beta=0.4, ngroup=2), twist_seed=3, twist=1e-3)
    m.D, m.M, m.jump_distance = 1e-9, 0.0, 5700.0   # a spring so soft that such a jump is accepted
    f = np.zeros((m.n_bf, m.ntime), order="F")
    o = OracleChain(m, field=f, seed_words=seed_words(4), meas=False)
    g = PqmcChain(m, field=f, rng_words=seed_words(4), meas=False)
    for c in (o, g):
        c.init_expkv()
        c.init_g(1)
    before = g.g()
    for c in (o, g):
        c.update_phonon_field(1, 1)
    assert o.state()["positive_accept"] == g.state()["positive_accept"] == 1 and o.state()["ln_cw"].real > 400
    assert np.array_equal(g.field(), o.field())
    assert rel_fro(o.g(), before) > 0.1 and rel_fro(g.g(), o.g()) < 1e-10
    g.close()


def test_a_family_without_plaquettes_changes_nothing():
    """Sweep, weight and gradient, and a mixed-precision batch, with and without it: the same bits."""
    torch = pytest.importorskip("torch")
    from pqmc_allinone_gb300.autograd import log_weight
    from pqmc_allinone_gb300.engine import PqmcBatch, PqmcChain
    out = []
    for keep in ([(0, 99), (1, 99), (2, 99), (3, 99)], [(2, 0), (0, 99), (1, 99), (3, 0), (2, 99), (3, 99), (1, 0)]):
        m, f = _families_cut(keep)
        c = PqmcChain(m, field=f, rng_words=SEED_WORDS, meas=False)
        x = torch.from_numpy(np.ascontiguousarray(f)[None].copy()).cuda().requires_grad_(True)
        w = log_weight(x, [c])
        (grad,) = torch.autograd.grad(w.sum(), x)
        c.set_field(f)
        c.init_expkv()
        c.init_g(1)
        c.sweep_slices(1, 1, m.ntime)
        c.sweep_slices(2, 1, m.ntime)
        b = PqmcBatch([m], [f], [SEED_WORDS], precision=1)
        b.init()
        b.sweep(1)
        b.sweep(2)
        out.append((w.detach().cpu().numpy(), grad.cpu().numpy(), c.field(), c.g(), b.chains[0].field(), b.chains[0].g()))
        b.close()
        c.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
