"""Performance cases: the work that a user of this library has it do.

Each case goes through the public Python entry points (``PqmcBatch``,
``PqmcChain``, ``autograd.log_weight``) on the spin-orbit lattice of the
configurations (2 sites and 2 bonds per cell, 4 checkerboard families of
4-site plaquettes, dtau = 0.1, half filling, x ~ N(0, 0.5^2), a stabilised
recompute every 10 slices).  Kinds:

``block``     a mixed-precision batch advanced by one stabilisation block,
              the step that a long run repeats; fields and states come back
``uneven``    a whole sweep of chains of different L and Lt in one mixed-precision
              batch; fields and states come back
``sweep``     a whole sweep of a mixed-precision batch with its equal-time
              measurement; records, fields, G and states come back
``plain``     one FP64 chain by one stabilisation block
``measured``  one FP64 chain by a whole sweep with its measurement
``init``      a new field for one FP64 chain: propagators, strings, G and
              weight, on the projector or the finite-temperature path
``global``    the driver's global step of one FP64 chain (k-space, rotate and
              k-space/time moves, G anew after an acceptance)
``measure``   one equal-time record of one FP64 chain
``grad``      the differentiable log-weight, forward and backward, of several
              chains
"""
from __future__ import annotations

import functools

import numpy as np
import torch

from pqmc_allinone_gb300 import model as M
from pqmc_allinone_gb300.abi import global_params
from pqmc_allinone_gb300.autograd import log_weight
from pqmc_allinone_gb300.engine import PqmcBatch, PqmcChain
from pqmc_allinone_gb300.rng import seed_words

NGROUP = 10      # slices between recomputes in every configuration
DIM, NPF = 4, 4  # plaquette dimension, families


def listed():
    return [
        # the production run: 64 chains of 14x14 at Lt = 1000, one block at a time
        {"name": "block 64x 14x14", "kind": "block", "chains": 64, "lx": 14, "ly": 14, "lt": 1000, "alpha": 0.3, "lam": 0.8},
        # a parameter scan: chains of L = 8, 10, 12 and Lt = 20, 40, 60 with their own lambda, side by side
        {"name": "uneven 36x 8-12", "kind": "uneven", "chains": 36, "lmin": 8, "lmax": 12, "lt": 20, "alpha": 0.3},
        # a middle-sized ensemble with an odd number of chains on a rectangular lattice, measured sweep by sweep
        {"name": "sweep 11x 8x10", "kind": "sweep", "chains": 11, "lx": 8, "ly": 10, "lt": 40, "alpha": 0.3, "lam": 0.8},
        # the small workload of the benchmark: launches and latency count
        {"name": "sweep 8x 6x6", "kind": "sweep", "chains": 8, "lx": 6, "ly": 6, "lt": 100, "alpha": 0.3, "lam": 0.8},
        # production size in plain FP64, the form whose decisions follow the reference bit for bit
        {"name": "plain 14x14", "kind": "plain", "lx": 14, "ly": 14, "lt": 1000, "alpha": 0.3, "lam": 0.8},
        # the smallest configuration: 4x4, Lt = 80, Gaussian proposals, measured every sweep
        {"name": "measured 4x4", "kind": "measured", "lx": 4, "ly": 4, "lt": 80, "alpha": 0.0, "lam": 0.8, "gauss": True},
        # a chain that starts from an imported field
        {"name": "init 12x12", "kind": "init", "lx": 12, "ly": 12, "lt": 200, "alpha": 0.3, "lam": 0.8, "proj": True},
        # the same at finite temperature
        {"name": "init T>0 6x8", "kind": "init", "lx": 6, "ly": 8, "lt": 80, "alpha": 0.3, "lam": 0.8, "proj": False},
        # global moves before a backward sweep
        {"name": "global 14x14", "kind": "global", "lx": 14, "ly": 14, "lt": 100, "alpha": 0.3, "lam": 0.8},
        # one measurement at production size
        {"name": "measure 14x14", "kind": "measure", "lx": 14, "ly": 14, "lt": 20, "alpha": 0.3, "lam": 0.8},
        # gradients for a field optimisation: an ensemble, and a pair of small chains
        {"name": "grad 8x 10x10", "kind": "grad", "chains": 8, "lx": 10, "ly": 10, "lt": 100, "alpha": 0.3, "lam": 0.8},
        {"name": "grad 2x 4x4", "kind": "grad", "chains": 2, "lx": 4, "ly": 4, "lt": 40, "alpha": 0.0, "lam": 0.8},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _even(rng, lo, hi):
    return 2 * rng.randint(lo // 2, hi // 2)


def draw(rng):
    kind = rng.choice(["block", "block", "uneven", "sweep", "sweep", "plain", "measured", "init", "init", "global", "measure", "grad"])
    c = {"kind": kind, "alpha": rng.choice([0.0, 0.3]), "lx": _even(rng, 4, 14), "ly": _even(rng, 4, 14),
         "lt": 10 * _log(rng, 2, 100), "lam": round(rng.uniform(0.5, 1.0), 3)}
    if kind == "block":
        c["chains"] = _log(rng, 1, 64)
    elif kind == "uneven":
        lmin = _even(rng, 4, 10)
        c = {"kind": kind, "alpha": c["alpha"], "chains": _log(rng, 3, 36), "lmin": lmin, "lmax": _even(rng, lmin + 2, 12),
             "lt": 10 * _log(rng, 1, 3)}
    elif kind == "sweep":
        c |= {"chains": _log(rng, 1, 12), "lx": _even(rng, 4, 10), "ly": _even(rng, 4, 10), "lt": 10 * _log(rng, 2, 10)}
    elif kind == "measured":
        c |= {"lx": _even(rng, 4, 6), "ly": _even(rng, 4, 8), "lt": 10 * _log(rng, 2, 10), "gauss": rng.random() < 0.5}
    elif kind == "init":
        c |= {"proj": rng.random() < 0.5, "lt": 10 * _log(rng, 2, 20)}
        if not c["proj"]:
            c |= {"lx": _even(rng, 4, 8), "ly": _even(rng, 4, 8), "lt": 10 * _log(rng, 2, 8)}
    elif kind == "global":
        c["lt"] = 10 * _log(rng, 2, 10)
    elif kind == "measure":
        c["lt"] = 20
    elif kind == "grad":
        c |= {"chains": _log(rng, 1, 8), "lx": _even(rng, 4, 10), "ly": _even(rng, 4, 10), "lt": 10 * _log(rng, 2, 10)}
    return c


# ---- inputs -----------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _model(lx, ly, lt, alpha, lam, gauss=False):
    spec = M.epsocz_spec((lx, ly), lam=lam, alpha=alpha, ntime=lt, ngroup=NGROUP, filling=0.5,
                         jump_distance=0.3 if gauss else 0.5,
                         proposal_kind=M.PROPOSAL_GAUSSIAN if gauss else M.PROPOSAL_UNIFORM)
    return M.build_model(spec, twist_seed=11, twist=1e-3)


def _case_model(c):
    return _model(c["lx"], c["ly"], c["lt"], c["alpha"], c["lam"], c.get("gauss", False))


def _seed(seed, i):
    return (int(seed) * 1009 + 3000 + i) % (1 << 30)


def _uneven_models(c):
    """Chain i takes the i-th of the (L, Lt) classes in turn, and a lambda of its own."""
    out = []
    for i in range(c["chains"]):
        sizes = range(c["lmin"], c["lmax"] + 1, 2)
        L = sizes[i % len(sizes)]
        lt = c["lt"] * (1 + (i // len(sizes)) % 3)
        out.append(_model(L, L, lt, c["alpha"], round(0.5 + 0.5 * ((i * 0.618) % 1.0), 3)))
    return out


def _models(c):
    return _uneven_models(c) if c["kind"] == "uneven" else [_case_model(c)] * c.get("chains", 1)


def _fields(c, seed):
    return [M.field_gaussian(m, _seed(seed, i)) for i, m in enumerate(_models(c))]


class _Cursor:
    """(loop, first slice) of the next block in the sweep order."""

    def __init__(self, lt):
        self.lt, self.loop, self.tc = lt, 1, 1

    def next(self):
        at = (self.loop, self.tc)
        self.tc += NGROUP
        if self.tc > self.lt:
            self.loop, self.tc = self.loop + 1, 1
        return at

    @staticmethod
    def first_time(at, lt):
        return at[1] if at[0] % 2 == 0 else lt - (at[1] + NGROUP - 1) + 1


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    models, fields = _models(c), _fields(c, seed)
    words = [seed_words(_seed(seed, i)) for i in range(len(models))]
    s = {"case": c, "kind": kind, "models": models}
    if kind in ("block", "uneven", "sweep"):
        b = PqmcBatch(models, fields, words, precision=1, meas=kind == "sweep")
        b.init()
        if kind == "sweep":
            b.set_measure(0)
        s |= {"batch": b, "loop": 1, "cursor": _Cursor(models[0].ntime)}
        if kind == "block":
            io = torch.empty((len(models), NGROUP, models[0].n_bf), dtype=torch.float64, pin_memory=True)
            s |= {"pinned": io, "io": io.numpy()}
        return s
    chains = [PqmcChain(m, field=f, rng_words=w) for m, f, w in zip(models, fields, words)]
    if kind == "grad":
        x = torch.from_numpy(np.stack([np.ascontiguousarray(f) for f in fields])).cuda().requires_grad_(True)
        return s | {"chains": chains, "x": x}
    ch = chains[0]
    if kind == "init":
        if not c["proj"]:
            ch.set_temperature(False)
        return s | {"chain": ch, "field": fields[0]}
    ch.init_expkv()
    ch.init_g(1)
    if kind == "global":
        ch.set_global(global_params(models[0], global_update_distance=0.05))
    return s | {"chain": ch, "loop": 1, "cursor": _Cursor(models[0].ntime)}


# ---- one pass ---------------------------------------------------------------
def _state_arrays(states):
    return {"ln_w": np.array([s["ln_cw"].real for s in states]),
            "accepts": np.array([[s["positive_accept"], s["negative_accept"]] for s in states]),
            "rng": np.array([s["rng"] for s in states])}


def run(s):
    kind = s["kind"]
    if kind == "block":
        b, at = s["batch"], s["cursor"].next()
        b.sweep_slices(*at, NGROUP)
        b.field_slices(_Cursor.first_time(at, s["models"][0].ntime), NGROUP, s["io"], False)
        return {"field": s["io"], **_state_arrays(b.states())}
    if kind == "uneven":
        b = s["batch"]
        b.sweep(s["loop"])
        s["loop"] += 1
        return {"field": np.concatenate([ch.field().ravel(order="F") for ch in b.chains]), **_state_arrays(b.states())}
    if kind == "sweep":
        b = s["batch"]
        b.sweep(s["loop"])
        s["loop"] += 1
        n = len(b.chains)
        return {"records": np.stack([b.records(i, 1)[0] for i in range(n)]), "field": np.stack([ch.field() for ch in b.chains]),
                "g": np.stack([ch.g() for ch in b.chains]), **_state_arrays(b.states())}
    if kind == "grad":
        w = log_weight(s["x"], s["chains"])
        (grad,) = torch.autograd.grad(w.sum(), s["x"])
        return {"w": w, "grad": grad}
    ch = s["chain"]
    if kind == "plain":
        at = s["cursor"].next()
        ch.sweep_slices(*at, NGROUP)
        return {"field": ch.get_field_slices(_Cursor.first_time(at, ch.m.ntime), NGROUP), "g": ch.g(), **_state_arrays([ch.state()])}
    if kind == "measured":
        records = ch.sweep(s["loop"], 1, warmup=0, cap=1)
        s["loop"] += 1
        return {"records": records, "field": ch.field(), "g": ch.g(), **_state_arrays([ch.state()])}
    if kind == "init":
        ch.set_field(s["field"])
        ch.init_expkv()
        ch.init_g(1)
        return {"g": ch.g(), "ln_w": ch.state()["ln_cw"].real}
    if kind == "global":
        n = ch.global_step(1)
        return {"accepted": n, "field": ch.field(), "g": ch.g(), **_state_arrays([ch.state()])}
    assert kind == "measure"
    rec, n = ch.begin_measure(False, ch.m.ntime // 2), len(M.FIELD_NAMES) * ch.m.lat.n_cell
    return {"scalars": rec[:-2 * n], "fields": rec[-2 * n:-n], "k_fields": rec[-n:]}


# ---- what a pass cannot do without ------------------------------------------
def _chain_work(c, m):
    """(bytes, flops) of one chain: complex FP64 in and out once, 8 flops per complex multiply-add."""
    ns, ne, nbf, lt = m.ns, m.nelec, m.n_bf, m.ntime
    kind = c["kind"]
    g, q, ekv = 16.0 * ns * ns, 16.0 * ns * ne, 2 * 16.0 * DIM * DIM * nbf     # G, one string block, a slice's propagators
    prop = 8.0 * NPF * DIM * ns * ne                                           # one slice applied to an Ns x nelec factor
    qr = 8.0 * (2 * ns * ne * ne - 2 * ne**3 / 3)                              # with Q formed
    get_g = 8.0 * (ns * ne * ne + ne**3 / 3 + ns * ne * ne + ns * ns * ne)
    slice_ = 8.0 * (NPF * 2 * DIM * ns * ns + 0.5 * nbf * DIM * ns * ns)       # wraps, and every second proposal accepted
    block_b, block_f = 2 * g + 3 * q + NGROUP * (16.0 * nbf + 2 * ekv), NGROUP * (slice_ + prop) + qr + get_g
    pairs = 8.0 * m.lat.n_cell**2 * (6 * 16 * 2 + 2 * 64 * 2 + 25 * 20)        # Wick contractions of every pair of cells
    record = 16.0 * M.record_width(m)
    if kind in ("block", "plain"):
        return block_b, block_f
    if kind in ("uneven", "sweep", "measured"):
        rec = kind != "uneven"
        return lt / NGROUP * block_b + rec * record, lt / NGROUP * block_f + rec * pairs
    if kind == "measure":
        return g + record, pairs
    if kind == "init":
        if not c["proj"]:   # square strings, Q and R kept
            return 8.0 * nbf * lt + 3 * lt * ekv + g * (2 + 2 * lt / NGROUP), lt * 8.0 * NPF * DIM * ns * ns + lt / NGROUP * 8.0 * ns**3 * 7 / 3 + 8.0 * ns**3 * 16 / 3
        return 8.0 * nbf * lt + 3 * lt * ekv + q * lt / NGROUP + g, lt * prop + lt / NGROUP * qr + get_g
    if kind == "global":    # three weights and one G
        return 4 * lt * (2 * ekv + 16.0 * nbf) + q * lt / NGROUP + g, 4 * (lt * prop + lt / NGROUP * qr) + get_g
    assert kind == "grad"   # left and right pass, G wrapped through every slice
    return 16.0 * nbf * lt + 4 * lt * ekv + 2 * q * lt / NGROUP, 2 * lt * prop + 2 * lt / NGROUP * qr + lt / NGROUP * get_g + lt * 8.0 * NPF * 2 * DIM * ns * ns


def work(case):
    per = [_chain_work(case, m) for m in _models(case)]
    return {"bytes": sum(b for b, _ in per), "flops": sum(f for _, f in per)}


# ---- the same in plain 64-bit arithmetic ------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _propagators(m, fields, want_derivative=False):
    """Per family (sites (n_pla, 4), E (chains, Lt, n_pla, 4, 4)[, dE/dx]): E = exp(-dtau (k K + x v V)), on
    plaquettes across the boundary times their phases; the derivative from the exponential of [[A, A'], [0, A]]."""
    x = torch.as_tensor(np.stack(fields), device=_device())                     # (chains, n_bf, Lt)
    out = []
    for f, t in enumerate(m.pf):
        phase = torch.as_tensor(np.where(t.crossing[:, None, None], t.bc_phases, 1.0 + 0j), device=x.device)
        a0 = -m.spec.delt * torch.as_tensor(m.k_coe[f] * m.kmat[f], device=x.device) * phase
        a1 = -m.spec.delt * torch.as_tensor(m.v_coe[f] * m.vmat[f], device=x.device) * phase
        xs = x[:, torch.as_tensor(t.bf_list, device=x.device)].permute(0, 2, 1)[..., None, None]
        a = a0 + xs * a1
        sites = torch.as_tensor(t.site_list, device=x.device)
        if want_derivative:
            big = torch.zeros(*a.shape[:-2], 2 * DIM, 2 * DIM, dtype=a.dtype, device=a.device)
            big[..., :DIM, :DIM], big[..., DIM:, DIM:], big[..., :DIM, DIM:] = a, a, a1.expand_as(a)
            big = torch.linalg.matrix_exp(big)
            out.append((sites, big[..., :DIM, :DIM], big[..., :DIM, DIM:]))
        else:
            out.append((sites, torch.linalg.matrix_exp(a.contiguous())))
    return out


def _apply(x, sites, e):
    """x(S, :) <- E x(S, :) on every plaquette; x (chains, Ns, n), e (chains, n_pla, 4, 4)."""
    y = x.clone()
    y[:, sites.reshape(-1)] = (e @ x[:, sites]).reshape(x.shape[0], -1, x.shape[2])
    return y


def _trial(m, n):
    return torch.as_tensor(np.ascontiguousarray(m.slater_q), device=_device()).expand(n, -1, -1)


def _finish_weight(m, ln):
    return (2.0 if m.spec.tr_weight else 1.0) * m.spec.ncopy * ln


def _exact_init(c, seed):
    m = _case_model(c)
    props = _propagators(m, _fields(c, seed))
    if c["proj"]:
        r = p = _trial(m, 1)
        ln = 2.0 * float(np.sum(np.log(np.abs(m.slater_d))))
        for t in range(m.ntime):
            for sites, e in props:
                r = _apply(r, sites, e[:, t])
            if (t + 1) % NGROUP == 0 or t + 1 == m.ntime:
                r, d = torch.linalg.qr(r)
                ln += float(torch.log(torch.abs(torch.diagonal(d[0]))).sum())
        lr = p.mH @ r
        g = r @ torch.linalg.solve(lr, p.mH)
        ln += float(torch.linalg.slogdet(lr)[1])
        return {"g": g[0].cpu().numpy(), "ln_w": _finish_weight(m, ln)}
    # (1 + B_n .. B_1)^-1 as the last block of the inverse of the cyclic matrix of the blocks, and its determinant
    n, nb = m.ns, m.ntime // NGROUP
    eye = torch.eye(n, dtype=torch.complex128, device=_device())
    cyc = torch.eye(n * nb, dtype=torch.complex128, device=_device())
    for b in range(nb):
        x = eye[None]
        for t in range(b * NGROUP, (b + 1) * NGROUP):
            for sites, e in props:
                x = _apply(x, sites, e[:, t])
        if nb == 1:
            cyc += x[0]
        elif b == 0:
            cyc[:n, (nb - 1) * n:] = x[0]
        else:
            cyc[b * n:(b + 1) * n, (b - 1) * n:b * n] = -x[0]
    rhs = torch.zeros(n * nb, n, dtype=torch.complex128, device=_device())
    rhs[-n:] = eye
    g = torch.linalg.solve(cyc, rhs)[-n:]
    ln = float(torch.linalg.slogdet(cyc)[1])
    return {"g": (eye - g).cpu().numpy(), "ln_w": _finish_weight(m, ln)}


def _exact_grad(c, seed):
    m = _case_model(c)
    fields = _fields(c, seed)
    n = len(fields)
    props = _propagators(m, fields, want_derivative=True)
    r = p = _trial(m, n)
    ln = torch.full((n,), 2.0 * float(np.sum(np.log(np.abs(m.slater_d)))), dtype=torch.float64, device=_device())
    right = []
    for t in range(m.ntime):
        for sites, e, _ in props:
            r = _apply(r, sites, e[:, t])
            right.append(r)
        if (t + 1) % NGROUP == 0 or t + 1 == m.ntime:
            r, d = torch.linalg.qr(r)
            ln = ln + torch.log(torch.abs(torch.diagonal(d, dim1=-2, dim2=-1))).sum(-1)
    ln = ln + torch.linalg.slogdet(p.mH @ r)[1]
    grad = torch.zeros(n, m.n_bf, m.ntime, dtype=torch.float64, device=_device())
    left = p                                                   # the left factor's conjugate transpose
    for t in reversed(range(m.ntime)):
        for f in reversed(range(len(props))):
            sites, e, de = props[f]
            r = right[t * len(props) + f]
            y = torch.linalg.solve(left.mH @ r, left.mH)       # G = r y just after family f
            block = r[:, sites] @ y[:, :, sites].permute(0, 2, 1, 3)
            tr = torch.einsum("bpij,bpji->bp", block, torch.linalg.solve(e[:, t], de[:, t], left=False))
            grad[:, torch.as_tensor(m.pf[f].bf_list, device=grad.device), t] += _finish_weight(m, tr.real)
            left = _apply(left, sites, e[:, t].mH)
        left = torch.linalg.qr(left)[0]
    return {"w": _finish_weight(m, ln), "grad": grad}


def _exact_measure(c, seed):
    """Every observable of one record: Wick contractions of cell pairs, summed over the pairs of each displacement."""
    m = _case_model(c)
    field = _fields(c, seed)[0]
    gh = _exact_init({**c, "proj": True}, seed)["g"]
    g = np.eye(m.ns) - gh
    tab, nc, hop, ep = M.meas_tables(m), m.lat.n_cell, m.spec.hop, m.spec.ep_parameter
    st, xn, yn = tab["cell_sites"], tab["cell_xnb"], tab["cell_ynb"]
    me, x = np.arange(nc), field[:, m.ntime // 2 - 1]
    xx, xy = x[tab["cell_bf"][:, 0]], x[tab["cell_bf"][:, 1]]

    def spin(nb):       # the two operators' sites: (4, nc) each, between a cell and its neighbour
        return (np.array([st[me, 0], st[me, 1], st[nb, 0], st[nb, 1]]), np.array([st[nb, 1], st[nb, 0], st[me, 1], st[me, 0]]))

    def straight(nb):   # the spin-diagonal bond
        return (np.array([st[me, 0], st[me, 1], st[nb, 0], st[nb, 1]]), np.array([st[nb, 0], st[nb, 1], st[me, 0], st[me, 1]]))

    def both(nb):
        a, b = spin(nb), straight(nb)
        return np.concatenate([a[0], b[0]]), np.concatenate([a[1], b[1]])

    def corr(l, r, vl, vr, hartree=False):   # (c1, c2)
        out = np.zeros((nc, nc), dtype=np.complex128)
        for i in range(len(l[0])):
            for j in range(len(r[0])):
                w = gh[l[1][i], l[0][i]][:, None] * gh[r[1][j], r[0][j]][None]
                if not hartree:
                    w = w + gh[np.ix_(r[1][j], l[0][i])].T * g[np.ix_(l[1][i], r[0][j])]
                out += vl[i][:, None] * w * vr[j]
        return out

    flat = lambda v: np.repeat(np.array(v, dtype=np.complex128)[:, None], nc, 1)   # noqa: E731  the boundary phases are 1 here
    vx, vy = [1j * hop, 1j * hop, -1j * hop, -1j * hop], [hop, -hop, -hop, hop]
    fx, fy, bx, by = flat(vx), flat(vy), spin(xn), spin(yn)
    pairs = [xx[:, None] * xx, xx[:, None] * xy, xy[:, None] * xy, (xx * xy)[:, None] * (xx * xy)]
    for h in (False, True):
        pairs += [corr(bx, bx, fx, fx, h), corr(bx, bx, fy, fy, h), corr(by, by, fx, fx, h), corr(by, by, fy, fy, h),
                  corr(bx, by, fx, fx, h), corr(bx, by, fy, fy, h)]
    pairs += [corr(bx, by, fx, fy, True), corr(bx, by, fy, fx, True)]
    u, d = st[:, 0], st[:, 1]
    mom = (np.array([u, u, d, d]), np.array([u, d, u, d]))
    dn, sz, sx, sy = (flat(v) for v in ([0.5, 0, 0, 0.5], [0.5, 0, 0, -0.5], [0, 0.5, 0.5, 0], [0, -0.5j, 0.5j, 0]))
    pairs += [corr(mom, mom, dn, dn), (gh[np.ix_(u, u)] * gh[np.ix_(d, d)] - gh[np.ix_(d, u)] * gh[np.ix_(u, d)]).T]
    pairs += [corr(mom, mom, v, v) for v in (sz, sx, sy)]
    for nb, v, xb in ((yn, fx, xy), (xn, fy, xx)):              # the physical current: the bond's own amplitude beside
        amp = np.concatenate([-v, ep * np.repeat(xb[None], 4, 0)])
        pairs.append(corr(both(nb), both(nb), amp, amp))
    fields = np.zeros((len(pairs), nc), dtype=np.complex128)
    for k, w in enumerate(pairs):
        np.add.at(fields[k], tab["rel_index"].T, w / nc)                        # rel_index[c2, c1]
    nxt = field[:, m.ntime // 2]
    dx = xx - nxt[tab["cell_bf"][:, 0]], xy - nxt[tab["cell_bf"][:, 1]]
    scal = [np.mean(0.5 * m.D * (xx**2 + xy**2)), np.mean(-0.5 * m.M * (dx[0]**2 + dx[1]**2) / m.spec.delt**2 + 1.0 / m.spec.delt), np.mean(xx + xy)]
    return {"scalars": np.array(scal, dtype=np.complex128), "fields": fields.ravel(), "k_fields": (fields @ m.lat.k_phase.T / nc).ravel()}


def exact(case, seed):
    """The chains that make Monte Carlo decisions have no closed answer."""
    c = dict(case)
    if c["kind"] == "init":
        return _exact_init(c, seed)
    if c["kind"] == "grad":
        return _exact_grad(c, seed)
    if c["kind"] == "measure":
        return _exact_measure(c, seed)
    return None
