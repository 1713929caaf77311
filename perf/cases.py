"""Workloads that a program linked against the RI library runs, with inputs made on the GPU from a seed.

Every case goes through the public entry points (``rerdmft_b200.ri``, ``mo``, ``scf``, ``integrals`` and,
for device copies of MO tensors, the C call ``rr_mo_copy_tensor``).  The three-centre tensors follow the
cube / Gaussian recipe of ``rerdmft_b200.synth`` (B[P, m, n] = c exp(-a (|r_m - r_P|^2 + |r_n - r_P|^2))) at
the sizes the benchmark and the tests use, with the box grown so that the density of centres stays the same.

* ``fock_nonrel`` / ``fock_x2c`` / ``fock_rkb``: one Fock build, the call an SCF loop makes in every iteration
* ``mo_nonrel`` / ``mo_ukb``: the MO three-index transforms that open the functional stage
* ``functional``: one orbital step of the functional stage (rotate the MO tensor, generalized Fock)
* ``integrals``: raw three-centre integrals and the aux metric of a water cluster, once per geometry
* ``scf_nonrel`` / ``scan_x2c``: whole SCF loops, one molecule and a geometry scan in lockstep
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from rerdmft_b200 import _lib as L
from rerdmft_b200 import basis as bs
from rerdmft_b200 import integrals, mo, ri, scf

DEV = "cuda"
F64, C128 = torch.float64, torch.complex128


# ------------------------------------------------------------------------------------------ the cases


def listed():
    return [
        # a light diatomic in a small basis: launches and latency count
        dict(name="fock_nonrel_small", kind="fock_nonrel", n=24, naux=129, nocc=5, host=False),
        # an ordinary molecule with odd sizes, called with host arrays as the reference's loop calls it
        dict(name="fock_nonrel_host", kind="fock_nonrel", n=203, naux=811, nocc=37, host=True),
        # the benchmark's shape, device arrays
        dict(name="fock_nonrel_large", kind="fock_nonrel", n=400, naux=1600, nocc=40, host=False),
        # a two-component build at the benchmark's X2C shape
        dict(name="fock_x2c", kind="fock_x2c", nl=200, naux=1000, ne=80, mixed=False),
        # the split-BF16 exchange that the mixed SCF loops use, odd sizes
        dict(name="fock_x2c_mixed", kind="fock_x2c", nl=131, naux=523, ne=54, mixed=True),
        # the four-component build at the benchmark's shape
        dict(name="fock_rkb", kind="fock_rkb", nl=200, ns=600, naux=1000, ne=40),
        # a new set of orbitals into an existing MO tensor, as each macro-iteration does it
        dict(name="mo_nonrel", kind="mo_nonrel", n=400, naux=1600),
        # the four-component MO tensor over the positive-energy spinors of a small molecule
        dict(name="mo_ukb", kind="mo_ukb", nl=101, ns=300, naux=500, nt=202),
        # one orbital step of a natural-orbital functional with pair terms, 120 spatial orbitals
        dict(name="functional", kind="functional", n=120, naux=480),
        # (H2O)_8 / cc-pVDZ with its automatic aux basis
        dict(name="integrals", kind="integrals", waters=8),
        # a whole closed-shell SCF from a core guess
        dict(name="scf_nonrel", kind="scf_nonrel", n=160, naux=640, nocc=21),
        # a geometry scan of uneven two-component problems
        dict(name="scan_x2c", kind="scan_x2c", count=12, nl_min=20, nl_max=72),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fock_nonrel", "fock_nonrel", "fock_x2c", "fock_x2c", "fock_rkb", "mo_nonrel", "mo_ukb",
                       "functional", "integrals", "scf_nonrel", "scan_x2c"])
    if kind == "fock_nonrel":
        n = _log(rng, 12, 400)
        return dict(kind=kind, n=n, naux=int(n * rng.uniform(3.0, 4.5)), nocc=max(1, int(n * rng.uniform(0.06, 0.3))),
                    host=rng.random() < 0.5)
    if kind == "fock_x2c":
        nl = _log(rng, 12, 200)
        return dict(kind=kind, nl=nl, naux=int(nl * rng.uniform(3.0, 5.0)), ne=2 * max(1, int(nl * rng.uniform(0.06, 0.2))),
                    mixed=rng.random() < 0.4)
    if kind == "fock_rkb":
        nl = _log(rng, 10, 180)
        return dict(kind=kind, nl=nl, ns=int(nl * rng.uniform(2.0, 3.0)), naux=int(nl * rng.uniform(3.0, 5.0)),
                    ne=2 * max(1, int(nl * rng.uniform(0.05, 0.1))))
    if kind == "mo_nonrel":
        n = _log(rng, 20, 380)
        return dict(kind=kind, n=n, naux=int(n * rng.uniform(3.0, 4.2)))
    if kind == "mo_ukb":
        nl = _log(rng, 10, 110)
        return dict(kind=kind, nl=nl, ns=int(nl * rng.uniform(2.0, 3.0)), naux=int(nl * rng.uniform(3.0, 5.0)),
                    nt=int(nl * rng.uniform(1.5, 2.0)))
    if kind == "functional":
        n = _log(rng, 10, 150)
        return dict(kind=kind, n=n, naux=int(n * rng.uniform(3.0, 4.5)))
    if kind == "integrals":
        return dict(kind=kind, waters=rng.randint(1, 9))
    if kind == "scf_nonrel":
        n = _log(rng, 24, 240)
        return dict(kind=kind, n=n, naux=int(n * rng.uniform(3.0, 4.5)), nocc=max(1, int(n * rng.uniform(0.06, 0.2))))
    return dict(kind=kind, count=rng.randint(3, 14), nl_min=rng.randint(12, 24), nl_max=rng.randint(40, 80))


# ------------------------------------------------------------------------------------------ inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _tensor(g, n, naux, box, alpha=0.3):
    """(naux, n*n) of the cube / Gaussian recipe, symmetric in its two AO indices."""
    r_ao, r_aux = box * _rand(g, n, 3), box * _rand(g, naux, 3)
    w = torch.exp(-alpha * ((r_aux[:, None, :] - r_ao[None, :, :]) ** 2).sum(-1))
    out = torch.empty(naux, n, n, device=DEV, dtype=F64)
    step = max(1, (1 << 25) // (n * n))
    for p in range(0, naux, step):
        c = _randn(g, min(step, naux - p), n, n)
        out[p:p + step] = (c + c.transpose(1, 2)) * 0.5 ** 0.5 * w[p:p + step, :, None] * w[p:p + step, None, :]
    return out.reshape(naux, n * n)


def _box(n):
    return 20.0 * (n / 400.0) ** (1.0 / 3.0)


def _b_scale(B):
    return 2.4 / math.sqrt(float(B.abs().max()) * math.sqrt(B.shape[0]))


def _inv_sqrt(s):
    w, u = torch.linalg.eigh(s)
    return (u / w.sqrt()) @ u.mH


def _overlap(g, n):
    a = _randn(g, n, n)
    return torch.eye(n, device=DEV, dtype=F64) + 0.05 * (a + a.T) / math.sqrt(n)


def _orthogonal(g, n):
    q, r = torch.linalg.qr(_randn(g, n, n))
    return q * torch.sign(torch.diagonal(r))


def _unitary(g, n):
    q, _ = torch.linalg.qr(torch.complex(_randn(g, n, n), _randn(g, n, n)))
    return q


def _kramers_even(m, blocks):
    nb = m.shape[0] // blocks
    i = torch.arange(m.shape[0], device=DEV)
    partner = (torch.div(i, nb, rounding_mode="floor") ^ 1) * nb + i % nb
    sign = torch.where(torch.div(i, nb, rounding_mode="floor") % 2 == 0, 1.0, -1.0).to(F64)
    return 0.5 * (m + torch.outer(sign, sign) * m[partner][:, partner].conj())


def _kramers_vectors(g, n, blocks):
    a = torch.complex(_randn(g, n, n), _randn(g, n, n))
    return torch.linalg.eigh(_kramers_even(0.5 * (a + a.mH), blocks))[1]


def _two(m):
    z = torch.zeros_like(m)
    return torch.cat([torch.cat([m, z], 1), torch.cat([z, m], 1)], 0).to(C128)


def _np(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _nonrel_inputs(c, seed):
    g = _gen(seed)
    n, nocc = c["n"], c["nocc"]
    B = _tensor(g, n, c["naux"], _box(n))
    S = _overlap(g, n)
    X = _inv_sqrt(S)
    C = X @ _orthogonal(g, n)[:, :nocc]
    h = _randn(g, n, n) * (12.0 / n)  # of the size of the two-electron part
    return dict(B=B, S=S, X=X, D=2.0 * C @ C.T, h=0.5 * (h + h.T))


def _x2c_inputs(c, seed):
    g = _gen(seed)
    nl, ne = c["nl"], c["ne"]
    B = _tensor(g, nl, c["naux"], _box(nl))
    B *= _b_scale(B)
    S_L = _overlap(g, nl)
    S, X = _two(S_L), _two(_inv_sqrt(S_L))
    C = X @ _kramers_vectors(g, 2 * nl, 2)[:, :ne]
    h = torch.complex(_randn(g, 2 * nl, 2 * nl), _randn(g, 2 * nl, 2 * nl)) * (0.6 / nl)
    return dict(B=B, S=S, X=X, P=_kramers_even(C @ C.mH, 2).contiguous(), h=_kramers_even(0.5 * (h + h.mH), 2).contiguous())


def _rkb_inputs(c, seed):
    g = _gen(seed)
    nl, ns, ne = c["nl"], c["ns"], c["ne"]
    nr, nu = 4 * nl, 2 * nl + 2 * ns
    BL = _tensor(g, nl, c["naux"], _box(nl))
    sc = _b_scale(BL)
    BL *= sc
    BS = _tensor(g, ns, c["naux"], _box(nl)) * (0.05 * sc)
    v = torch.zeros(nu, nr, device=DEV, dtype=C128)
    v[:2 * nl, :2 * nl] = torch.eye(2 * nl, device=DEV, dtype=C128)
    w = torch.complex(_randn(g, ns, nl), _randn(g, ns, nl)) / math.sqrt(ns)
    v[2 * nl:2 * nl + ns, 2 * nl:3 * nl] = w
    v[2 * nl + ns:, 3 * nl:] = w.conj()
    su = torch.eye(nu, device=DEV, dtype=C128)
    su[:2 * nl, :2 * nl] = _two(_overlap(g, nl))
    s = v.mH @ su @ v
    s = 0.5 * (s + s.mH)
    x = _inv_sqrt(s)
    C = x @ _kramers_vectors(g, nr, 4)[:, :ne]
    h = torch.complex(_randn(g, nr, nr), _randn(g, nr, nr)) * (0.3 / nr)
    return dict(BL=BL, BS=BS, v=v, s=s.contiguous(), x=x.contiguous(), P=_kramers_even(C @ C.mH, 4).contiguous(),
                h=_kramers_even(0.5 * (h + h.mH), 4).contiguous())


def _mo_inputs(c, seed):
    g = _gen(seed)
    return dict(B=_tensor(g, c["n"], c["naux"], _box(c["n"])), C=_orthogonal(g, c["n"]).contiguous())


def _ukb_inputs(c, seed):
    g = _gen(seed)
    nl, ns = c["nl"], c["ns"]
    BL = _tensor(g, nl, c["naux"], _box(nl))
    BS = _tensor(g, ns, c["naux"], _box(nl)) * 0.05
    return dict(BL=BL, BS=BS, C=_unitary(g, 2 * nl + 2 * ns)[:, :c["nt"]].contiguous())


def _functional_inputs(c, seed):
    g = _gen(seed)
    n = c["n"]
    B = _tensor(g, n, c["naux"], _box(n))
    B *= _b_scale(B)
    q = _orthogonal(g, n)
    Bmo = (q.T @ B.reshape(-1, n, n) @ q).reshape(-1, n * n).contiguous()
    nocc = max(1, n // 4)
    e = torch.cat([-3.0 + _rand(g, nocc), 0.5 + 3.0 * _rand(g, n - nocc)])
    qq = _orthogonal(g, n)
    h = _two((qq * e) @ qq.T).real.contiguous()
    o = torch.cat([0.97 - 0.05 * _rand(g, nocc), 0.05 * torch.exp(-torch.arange(n - nocc, device=DEV, dtype=F64) / 2.0)])
    occ = torch.cat([o, o])
    d = 2 * n
    pair = np.array([(i + 1) % d if i % 2 == 0 else i - 1 for i in range(d)], dtype=np.int64)
    k = 0.01 * _randn(g, n, n)
    u = torch.linalg.matrix_exp(k - k.T)
    return dict(Bmo=Bmo, h=h, occ=occ, h2=torch.outer(occ, occ), x2=torch.outer(occ, occ).sqrt(), pair=pair,
                l1=0.01 * _randn(g, d, d), l2=0.01 * _randn(g, d, d), U=_two(u).real.contiguous())


# The cc-pVDZ shells of O and H: (element, l, exponents, coefficients).
_O_CORE = [11720.0, 1759.0, 400.8, 113.7, 37.03, 13.27, 5.025, 1.013, 0.3023]
_SHELLS = [
    ("O", 0, _O_CORE, [0.00071, 0.00547, 0.027837, 0.1048, 0.283062, 0.448719, 0.270952, 0.015458, -0.002585]),
    ("O", 0, _O_CORE, [-0.00016, -0.001263, -0.006267, -0.025716, -0.070924, -0.165411, -0.116955, 0.557368, 0.572759]),
    ("O", 0, [0.3023], [1.0]),
    ("O", 1, [17.7, 3.854, 1.046, 0.2753], [0.043018, 0.228913, 0.508728, 0.460531]),
    ("O", 1, [0.2753], [1.0]),
    ("O", 2, [1.185], [1.0]),
    ("H", 0, [13.01, 1.962, 0.4446], [0.019685, 0.137977, 0.478148]),
    ("H", 0, [0.122], [1.0]),
    ("H", 1, [0.727], [1.0]),
]
_WATER = [("O", 0.0, 0.0, 0.0), ("H", 0.0, 1.430522676971576, 1.1073795095182872),
          ("H", 0.0, -1.430522676971576, 1.1073795095182872)]


def _water_cluster(waters, seed):
    """Water molecules 3 Angstrom apart on a cubic grid, each turned at random and shifted by up to 0.3 bohr."""
    r = np.random.default_rng(int(seed))
    k = int(math.ceil(waters ** (1.0 / 3.0) - 1e-9))
    geo = []
    for i in range(waters):
        at = np.array([i % k, (i // k) % k, i // (k * k)]) * 3.0 * bs.ANGSTROM_TO_BOHR + r.uniform(-0.3, 0.3, 3)
        q, _ = np.linalg.qr(r.standard_normal((3, 3)))
        geo += [bs.Atom(s, *map(float, q @ np.array(x) + at)) for s, *x in _WATER]
    sets = bs.basis_set_from_arrays([s[0] for s in _SHELLS], [s[1] for s in _SHELLS], [len(s[2]) for s in _SHELLS],
                                    [e for s in _SHELLS for e in s[2]], [e for s in _SHELLS for e in s[3]])
    orb = bs.build_molecular_basis(geo, sets)
    bs.normalize_cartesian_basis(orb)
    aux = bs.build_auto_auxiliary_basis(orb, "PAUTO")
    bs.normalize_cartesian_basis(aux)
    return orb, aux


def _scf_inputs(c, seed):
    g = _gen(seed)
    n, nocc = c["n"], c["nocc"]
    B = _tensor(g, n, c["naux"], _box(n))
    B *= _b_scale(B)
    e = torch.cat([-2.0 + 0.8 * _rand(g, nocc), -0.4 + 2.5 * _rand(g, n - nocc)])
    q = _orthogonal(g, n)
    h = (q * e) @ q.T
    S = _overlap(g, n)
    X = _inv_sqrt(S)
    C = X @ torch.linalg.eigh(X.T @ h @ X)[1][:, :nocc]
    return dict(B=B, h=_np(h), S=_np(S), X=_np(X), P0=_np(2.0 * C @ C.T))


def _scan_inputs(c, seed):
    g = _gen(seed)
    r = np.random.default_rng([c["count"], c["nl_min"], c["nl_max"]])  # the sizes belong to the case
    out = []
    for k in range(c["count"]):
        nl, ne = int(r.integers(c["nl_min"], c["nl_max"] + 1)), 4 if k % 2 == 0 else 14
        B = _tensor(g, nl, 4 * nl, _box(nl))
        B *= _b_scale(B)
        S_L = _overlap(g, nl)
        S, X = _two(S_L), _two(_inv_sqrt(S_L))
        e = torch.cat([-2.0 + 0.8 * _rand(g, ne // 2), 0.3 + 2.5 * _rand(g, nl - ne // 2)]).sort()[0].repeat_interleave(2)
        y = _kramers_vectors(g, 2 * nl, 2)
        sx = S @ X
        h = _kramers_even(sx @ ((y * e) @ y.mH) @ sx.mH, 2)
        C = X @ torch.linalg.eigh(X.mH @ h @ X)[1][:, :ne]
        P0 = _kramers_even(C @ C.mH, 2)
        out.append(dict(nl=nl, ne=ne, B=B, S=_np(S), X=_np(X), h=_np(h), P0=_np(P0)))
    return out


def prepare(case, seed):
    state = _prepare(case, seed)
    torch.cuda.synchronize()
    return state


def _store(src):
    torch.cuda.synchronize()  # the inputs are complete before the library copies them on its own stream
    src.store
    return src


def _prepare(case, seed):
    kind = case["kind"]
    if kind == "fock_nonrel":
        m = _nonrel_inputs(case, seed)
        host = _np if case["host"] else (lambda t: t.contiguous())
        src = ri.RiNonRelEriSource(case["n"], m["B"], host(m["X"]), host(m["S"]))
        _store(src)
        return dict(kind=kind, src=src, h=host(m["h"]), D=host(m["D"]))
    if kind == "fock_x2c":
        m = _x2c_inputs(case, seed)
        src = ri.RiX2cEriSource(case["nl"], m["B"], m["X"], m["S"])
        _store(src)
        return dict(kind=kind, src=src, h=m["h"], P=m["P"], precision="mixed" if case["mixed"] else "fp64")
    if kind == "fock_rkb":
        m = _rkb_inputs(case, seed)
        src = ri.RiDirectEriSource(case["nl"], case["ns"], m["BL"], m["BS"], m["v"], m["s"], m["x"])
        _store(src)
        return dict(kind=kind, src=src, h=m["h"], P=m["P"])
    if kind == "mo_nonrel":
        m = _mo_inputs(case, seed)
        src = ri.RiNonRelEriSource(case["n"], m["B"], None, None)
        _store(src)
        zero = torch.zeros(case["naux"], case["n"] ** 2, device=DEV, dtype=F64)
        torch.cuda.synchronize()
        return dict(kind=kind, src=src, C=m["C"], into=mo.RiNonRelSpinMoEri.from_tensor(zero, case["n"]))
    if kind == "mo_ukb":
        m = _ukb_inputs(case, seed)
        src = ri.RiDirectEriSource(case["nl"], case["ns"], m["BL"], m["BS"])
        _store(src)
        return dict(kind=kind, src=src, C=m["C"])
    if kind == "functional":
        m = _functional_inputs(case, seed)
        torch.cuda.synchronize()
        return dict(kind=kind, eri=mo.RiNonRelSpinMoEri.from_tensor(m["Bmo"], case["n"]), U=m["U"], pair=m["pair"],
                    **{k: _np(m[k]) for k in ("h", "occ", "h2", "x2", "l1", "l2")})
    if kind == "integrals":
        orb, aux = _water_cluster(case["waters"], seed)
        return dict(kind=kind, orb=orb, aux=aux)
    if kind == "scf_nonrel":
        m = _scf_inputs(case, seed)
        src = ri.RiNonRelEriSource(case["n"], m["B"], m["X"], m["S"])
        _store(src)
        return dict(kind=kind, src=src, ne=2 * case["nocc"], **{k: m[k] for k in ("h", "X", "P0")})
    problems = []
    for m in _scan_inputs(case, seed):
        src = ri.RiX2cEriSource(m["nl"], m["B"], m["X"], m["S"])
        _store(src)
        problems.append(dict(eri=src, h_x2c=m["h"], x_large=m["X"], initial_density=m["P0"], n_electrons=m["ne"]))
    return dict(kind=kind, problems=problems)


# ------------------------------------------------------------------------------------------ one pass


def _device_copy(eri):
    out = torch.empty(eri.naux, eri.n * eri.n, device=DEV, dtype=C128 if eri._kind == L.RR_MO_COMPLEX else F64)
    L.check(L.lib().rr_mo_copy_tensor(eri.handle, out.data_ptr(), ctypes.byref(L.opts(L.RR_MEM_DEVICE))))
    return out


def run(state):
    kind = state["kind"]
    if kind == "fock_nonrel":
        return ri.nonRelFockMatrix(state["h"], state["src"], state["D"])
    if kind == "fock_x2c":
        return ri.x2cFockMatrix(state["h"], state["src"], state["P"], precision=state["precision"])
    if kind == "fock_rkb":
        return ri.rkbFockMatrix(state["h"], state["src"], state["P"])
    if kind == "mo_nonrel":
        return _device_copy(mo.buildRiNonRelSpinMoEri(state["src"], state["src"].nl, state["C"], into=state["into"]))
    if kind == "mo_ukb":
        return _device_copy(mo.buildRiMoEri(state["src"], state["C"]))
    if kind == "functional":
        eri = state["eri"].rotated(state["U"])
        F = mo.hartreeExchangeFockMatrix(state["h"], eri, state["occ"], state["h2"], state["x2"], state["pair"],
                                         state["l1"], state["l2"])
        return F, _device_copy(eri)
    if kind == "integrals":
        return (integrals.threeCenterIntegralsRaw(state["orb"], state["aux"], device=True),
                integrals.auxMetric(state["aux"], device=True))
    if kind == "scf_nonrel":
        r = scf.runNonRelativisticHartreeFock(state["src"], state["h"], state["X"], state["P0"], state["ne"], orbitals=True)
        return r["energy"], r["P"], r["orbital_energies"], r["fock_matrix"]
    return [(r["energy"], r["P"]) for r in scf.runX2CHartreeFockScfBatch(state["problems"], mode="grouped")]


# ------------------------------------------------------------------------------------------ work


def _fock_work(blocks, naux, r, cplx):
    """(tensor elements, flops) of J and K: blocks = [(dimension, spin blocks)] per resident tensor, r occupied.
    Half-transforms, the exchange blocks on and above the diagonal, two passes over the symmetric half for J."""
    m = 4 if cplx else 1
    el = naux * sum(d * d for d, _ in blocks)
    sizes = [d for d, k in blocks for _ in range(k)]
    ht = sum(2.0 * naux * r * d * d for d in sizes) * (2 if cplx else 1)
    ex = sum((1.0 if i == j else 2.0) * naux * r * a * b for i, a in enumerate(sizes) for j, b in enumerate(sizes) if j >= i)
    return el, ht + m * ex + 2.0 * el


def _scf_steps(c):
    return 8  # iterations that such a loop takes, about


def work(case):
    kind = case["kind"]
    if kind in ("fock_nonrel", "scf_nonrel"):
        n = case["n"]
        el, fl = _fock_work([(n, 1)], case["naux"], case["nocc"], False)
        k = _scf_steps(case) if kind == "scf_nonrel" else 1
        return dict(bytes=8.0 * (el + 5 * n * n), flops=k * (fl + 8.0 * n ** 3))
    if kind == "fock_x2c":
        n = 2 * case["nl"]
        el, fl = _fock_work([(case["nl"], 2)], case["naux"], case["ne"], True)
        return dict(bytes=8.0 * el + 16.0 * 5 * n * n, flops=fl + 16.0 * n ** 3)
    if kind == "fock_rkb":
        nr, nu = 4 * case["nl"], 2 * case["nl"] + 2 * case["ns"]
        el, fl = _fock_work([(case["nl"], 2), (case["ns"], 2)], case["naux"], case["ne"], True)
        return dict(bytes=8.0 * el + 16.0 * (5 * nr * nr + nu * nr), flops=fl + 16.0 * nr ** 3 + 16.0 * nr * nr * nu)
    if kind == "mo_nonrel":
        n, p = case["n"], case["naux"]
        return dict(bytes=8.0 * (2 * p * n * n + n * n), flops=4.0 * p * n ** 3)
    if kind == "mo_ukb":
        nl, ns, p, t = case["nl"], case["ns"], case["naux"], case["nt"]
        nu = 2 * nl + 2 * ns
        return dict(bytes=8.0 * p * (nl * nl + ns * ns) + 16.0 * (p * t * t + nu * t),
                    flops=8.0 * p * t * (nl * nl + ns * ns) + 8.0 * p * t * t * nu)
    if kind == "functional":
        n, p = case["n"], case["naux"]
        return dict(bytes=8.0 * (2 * p * n * n + 6 * 4 * n * n), flops=4.0 * p * n ** 3 + 2.0 * p * 4 * n * n * 2 * n)
    if kind == "integrals":
        n, na = 25 * case["waters"], 357 * case["waters"]
        return dict(bytes=8.0 * (na * n * n + na * na), flops=200.0 * na * n * n / 2)
    sizes = np.linspace(case["nl_min"], case["nl_max"], case["count"])
    by = fl = 0.0
    for nl in sizes:
        el, f = _fock_work([(int(nl), 2)], 4 * int(nl), 9, True)
        by += 8.0 * el + 16.0 * 20 * nl * nl
        fl += _scf_steps(case) * (f + 20 * 8.0 * (2 * nl) ** 3)
    return dict(bytes=by, flops=fl)


# ------------------------------------------------------------------------------------------ in 64 bits


def _coulomb(tens, dens):
    gamma = sum(t @ d.reshape(-1) for t, d in zip(tens, dens))
    return [(gamma @ t).reshape(d.shape) for t, d in zip(tens, dens)]


def _occupied(X, S, P, scale, weighted):
    Z = S @ X
    w, y = torch.linalg.eigh(scale * (Z.mH @ P @ Z))
    keep = w > 0.5
    c = X @ y[:, keep]
    return c * w[keep].sqrt() if weighted else c


def _exchange(B, cf, cu):
    """sum_P B^P cf cu^dagger B^P for B (naux, m, m) real."""
    half = lambda c: torch.complex(B @ c.real, B @ c.imag) if c.is_complex() else B @ c  # noqa: E731
    v = [half(c).transpose(0, 1).reshape(B.shape[1], -1) for c in (cf, cu)]
    return v[0] @ v[1].mH


def _exchange2(Bf, Bu, cf, cu):
    half = lambda B, c: torch.complex(B @ c.real, B @ c.imag).transpose(0, 1).reshape(B.shape[1], -1)  # noqa: E731
    return half(Bf, cf) @ half(Bu, cu).mH


def exact(case, seed):
    kind = case["kind"]
    if kind == "fock_nonrel":
        m = _nonrel_inputs(case, seed)
        n = case["n"]
        c = _occupied(m["X"], m["S"], m["D"], 0.5, False)
        F = m["h"] + _coulomb([m["B"]], [m["D"]])[0] - _exchange(m["B"].reshape(-1, n, n), c, c)
        return _np(F) if case["host"] else F
    if kind == "fock_x2c":
        m = _x2c_inputs(case, seed)
        nl = case["nl"]
        c = _occupied(m["X"], m["S"], m["P"], 1.0, True)
        J = _coulomb([m["B"]], [(m["P"][:nl, :nl] + m["P"][nl:, nl:]).real.contiguous()])[0]
        B = m["B"].reshape(-1, nl, nl)
        F = m["h"] + _two(J)
        for f in range(2):
            for u in range(2):
                F[f * nl:(f + 1) * nl, u * nl:(u + 1) * nl] -= _exchange(B, c[f * nl:(f + 1) * nl], c[u * nl:(u + 1) * nl])
        return F
    if kind == "fock_rkb":
        m = _rkb_inputs(case, seed)
        nl, ns = case["nl"], case["ns"]
        c = m["v"] @ _occupied(m["x"], m["s"], m["P"], 1.0, True)
        Pu = m["v"] @ m["P"] @ m["v"].mH
        off = [0, nl, 2 * nl, 2 * nl + ns, 2 * nl + 2 * ns]
        sl = [slice(off[i], off[i + 1]) for i in range(4)]
        tens = [m["BL"].reshape(-1, nl, nl), m["BS"].reshape(-1, ns, ns)]
        J = _coulomb([m["BL"], m["BS"]], [(Pu[sl[0], sl[0]] + Pu[sl[1], sl[1]]).real.contiguous(),
                                          (Pu[sl[2], sl[2]] + Pu[sl[3], sl[3]]).real.contiguous()])
        G = torch.zeros(off[4], off[4], device=DEV, dtype=C128)
        for f in range(4):
            G[sl[f], sl[f]] += J[f // 2]
            for u in range(4):
                G[sl[f], sl[u]] -= _exchange2(tens[f // 2], tens[u // 2], c[sl[f]], c[sl[u]])
        return m["h"] + m["v"].mH @ G @ m["v"]
    if kind == "mo_nonrel":
        m = _mo_inputs(case, seed)
        n = case["n"]
        return (m["C"].T @ m["B"].reshape(-1, n, n) @ m["C"]).reshape(-1, n * n)
    if kind == "mo_ukb":
        m = _ukb_inputs(case, seed)
        nl, ns, t = case["nl"], case["ns"], case["nt"]
        out = torch.zeros(case["naux"], t, t, device=DEV, dtype=C128)
        off = 0
        for B, d in ((m["BL"], nl), (m["BL"], nl), (m["BS"], ns), (m["BS"], ns)):
            c = m["C"][off:off + d]
            B = B.reshape(-1, d, d)
            out += c.mH @ torch.complex(B @ c.real, B @ c.imag)
            off += d
        return out.reshape(-1, t * t)
    if kind == "functional":
        m = _functional_inputs(case, seed)
        n = case["n"]
        u = m["U"][:n, :n]
        rot = u.T @ m["Bmo"].reshape(-1, n, n) @ u
        b = torch.zeros(rot.shape[0], 2 * n, 2 * n, device=DEV, dtype=F64)
        b[:, :n, :n] = rot
        b[:, n:, n:] = rot
        pr = torch.as_tensor(m["pair"], device=DEV)
        F = m["occ"][None, :] * m["h"].T
        F = F + torch.einsum("pab,pa->ba", b, torch.diagonal(b, dim1=1, dim2=2) @ m["h2"])
        coef = 2.0 * (m["l1"][pr][:, pr] + m["l2"][pr])
        y = -m["x2"].T[None] * b.transpose(1, 2) + coef[None] * b[:, pr][:, :, pr]
        F = F + b.reshape(-1, 2 * n).T @ y.reshape(-1, 2 * n)
        return _np(F), rot.reshape(-1, n * n)
    # integrals: an independent program for contracted s, p, d and aux functions up to l = 6 would be needed;
    # the SCF loops stop at a tolerance, so their last iterate has no value of its own
    return None
