"""Performance cases of the block-sparse symmetric-tensor engine: the calls its users make.

A case is a dict of plain values whose ``"kind"`` names the call:

``matvec``      one compiled two-site effective-Hamiltonian matvec (``program.GraphMatvec``)
``lanczos``     one device Lanczos solve of a bond (``network.Env.solve``)
``sweep``       one two-site DMRG sweep of a converged chain (``network.sweep_``)
``tensordot``   a four-leg U(1) contraction (``tenet.einsum``)
``env_batch``   a batch of U(1) x U(1) x fZ2 environment updates (``batch.env_update_last``)
``heff_batch``  a batch of two-site matvecs (``batch.BatchedHeff2``)
``svd``         the truncated SVD of a two-site tensor (``linalg.svd_truncated``)
``ctm_move``    one Z2 corner-transfer-matrix move (``network.move``)
``lq``          the LQ of a site tensor (``linalg.lq``)
``dense``       a U(1) site-times-bond contraction with large sectors (``tenet.einsum``)

``listed()`` are the named cases, ``draw(rng)`` one more of the same ranges, ``prepare``
what a program holds before the call (seeded inputs on the GPU and the plan it keeps),
``run`` one call, ``work`` the bytes and flops the call cannot do without, ``exact`` the
same results in plain NumPy / torch FP64 where the result has one value (singular vectors
and Krylov vectors have a gauge; SU(2) and fermionic tensors would need the recoupling
this file does not restate).

Bonds are texts ``"label:multiplicity,..."`` (2j for SU(2), the charge for U(1)).
"""

from __future__ import annotations

import math
import sys
from itertools import product
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "tenet-py_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tenet  # noqa: E402
from tenet import batch, linalg, network, ops, program  # noqa: E402
from tenet.plan import adjoint_plan, repartition_plan, transpose_plan  # noqa: E402
from tenet.structure import IN, OUT, GradedSpace, Leg, TensorStructure, layout, \
    matrix_layout  # noqa: E402
from tenet.symmetry import SU2, U1, Z2, ProductSector, U1xU1xfZ2  # noqa: E402
from tenet.tensor import SymmetricTensor  # noqa: E402

# multiplets per spin of the L = 64 Heisenberg chain's mid bond at cutoff 1e-10, and of the
# synthetic bond of 256 multiplets (both the benchmark's)
_BOND_L64 = "0:8,2:14,4:7"
_BOND_256 = "1:60,3:56,5:46,7:36,9:25,11:16,13:10,15:5,17:2"


# ---------------------------------------------------------------------------------------
# the cases


def listed() -> list:
    return [
        # the smallest call of a DMRG run: one matvec of the L = 64 chain's mid bond, where
        # launches and dependent loads are all the time there is
        {"name": "matvec_L64", "kind": "matvec", "bond": _BOND_L64},
        # a bond's ground-state solve (20 Krylov vectors) at 256 multiplets on the bond
        {"name": "lanczos_256", "kind": "lanczos", "peak": 60.0, "width": 16.0, "side": 12,
         "ncv": 20},
        # the whole call a DMRG user waits for: a sweep of a short chain near convergence
        {"name": "sweep_L16", "kind": "sweep", "sites": 16, "chi": 64, "ncv": 20},
        # the four-leg U(1) contraction abcd,cdef->abef, seven charges, 40 states a leg
        {"name": "tensordot_u1", "kind": "tensordot", "scale": 12.0, "qmax": 3},
        # 64 Hubbard-chain environment updates in one call, in FP64 and in the 3xBF16 form
        {"name": "env_batch64", "kind": "env_batch", "n": 64, "lam": 24.0, "deg_seed": 1000,
         "precision": "f64"},
        {"name": "env_batch64_3xbf16", "kind": "env_batch", "n": 64, "lam": 24.0,
         "deg_seed": 1000, "precision": "3xbf16"},
        # many small solves served together: 32 matvecs of the L = 64 mid bond
        {"name": "heff_batch32", "kind": "heff_batch", "bond": _BOND_L64, "n": 32},
        # the truncation of a two-site tensor at 256 multiplets
        {"name": "svd_256", "kind": "svd", "group": "SU2", "bond": _BOND_256},
        # one CTMRG move of the Ising model at chi = 128
        {"name": "ctm_move_128", "kind": "ctm_move", "chi": 128},
        # canonising one U(1) site of 256 states a bond
        {"name": "lq_256", "kind": "lq", "scale": 77.0, "qmax": 3},
        # contractions whose sectors are dense matrices, in FP64 and on the tensor cores
        {"name": "dense_f64", "kind": "dense", "scale": 900.0, "qmax": 3, "precision": "f64"},
        {"name": "dense_3xbf16", "kind": "dense", "scale": 900.0, "qmax": 3,
         "precision": "3xbf16"},
    ]


def _log(rng, lo: float, hi: float) -> float:
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 3)


def _profile(peak: float, width: float, parity: int) -> dict:
    """Multiplets per spin of a Heisenberg chain's bond: ``peak (2j + 1) exp(-2j (2j + 2) /
    width)`` (the converged L = 64 mid bonds follow it to within a few multiplets)."""
    out = {}
    for tj in range(parity, 19, 2):
        m = round(peak * (tj + 1) * math.exp(-tj * (tj + 2) / width))
        if m:
            out[tj] = int(m)
    return out


def _text(bond: dict) -> str:
    return ",".join(f"{a}:{m}" for a, m in sorted(bond.items()))


def draw(rng) -> dict:
    kind = rng.choice(["matvec", "lanczos", "sweep", "tensordot", "env_batch", "heff_batch",
                       "svd", "ctm_move", "lq", "dense"])
    if kind == "matvec":
        return {"kind": kind, "bond": _text(_profile(_log(rng, 2.0, 60.0),
                                                     rng.uniform(10.0, 20.0), rng.randrange(2)))}
    if kind == "lanczos":
        return {"kind": kind, "peak": _log(rng, 12.0, 60.0), "width": round(rng.uniform(12.0, 18.0), 2),
                "side": 12, "ncv": rng.choice([8, 13, 20])}
    if kind == "sweep":
        return {"kind": kind, "sites": rng.randrange(8, 17, 2), "chi": rng.randrange(24, 64),
                "ncv": rng.choice([10, 15, 20])}
    if kind == "tensordot":
        return {"kind": kind, "scale": _log(rng, 2.0, 13.0), "qmax": rng.randrange(2, 4)}
    if kind == "env_batch":
        return {"kind": kind, "n": int(_log(rng, 4, 64)), "lam": round(rng.uniform(6.0, 24.0), 1),
                "deg_seed": rng.randrange(1000, 2000),
                "precision": rng.choice(["f64", "f64", "3xbf16", "tf32"])}
    if kind == "heff_batch":
        return {"kind": kind, "bond": _text(_profile(_log(rng, 3.0, 12.0),
                                                     rng.uniform(11.0, 18.0), 0)),
                "n": int(_log(rng, 4, 32))}
    if kind == "svd":
        if rng.randrange(2):
            bond = _profile(_log(rng, 4.0, 36.0), rng.uniform(11.0, 18.0), rng.randrange(2))
            return {"kind": kind, "group": "SU2", "bond": _text(bond)}
        s = _log(rng, 6.0, 60.0)
        bond = {q: max(1, round(s * math.exp(-q * q / 4))) for q in range(-4, 5)}
        return {"kind": kind, "group": "U1", "bond": _text(bond)}
    if kind == "ctm_move":
        return {"kind": kind, "chi": int(_log(rng, 12, 128))}
    if kind == "lq":
        return {"kind": kind, "scale": _log(rng, 6.0, 77.0), "qmax": rng.randrange(2, 5)}
    return {"kind": kind, "scale": _log(rng, 50.0, 900.0), "qmax": rng.randrange(1, 4),
            "precision": rng.choice(["f64", "f64", "3xbf16", "tf32"])}


# ---------------------------------------------------------------------------------------
# structures


def _space(provider, text: str) -> GradedSpace:
    pairs = (x.split(":") for x in text.split(","))
    return GradedSpace.new(provider, {provider.sector(int(a)): int(m) for a, m in pairs})


def _gauss(scale: float, qmax: int) -> dict:
    return {q: max(1, round(scale * math.exp(-q * q / 4))) for q in range(-qmax, qmax + 1)}


def _heff_structures(bond: str):
    """``(fl, w, fr, aa)`` of the SU(2) Heisenberg chain: an MPO bond of multiplets 0, 0, 2."""
    B, M, P = _space(SU2, bond), _space(SU2, "0:2,2:1"), _space(SU2, "1:1")
    return (TensorStructure((Leg(B, IN), Leg(M, OUT, True), Leg(B, OUT))),
            TensorStructure((Leg(M, IN, True), Leg(P, OUT), Leg(P, IN), Leg(M, OUT, True))),
            TensorStructure((Leg(B, OUT), Leg(M, IN, True), Leg(B, IN))),
            TensorStructure((Leg(B, OUT), Leg(P, OUT), Leg(P, OUT), Leg(B, IN))))


def _env_structures(case):
    """``(F, A, W)`` of a Hubbard chain's environment update: bond sectors (N, 2Sz) in [-4,
    4]^2 with Poisson degeneracies, an MPO leg of width 6, the site's four states."""
    rng = np.random.default_rng(case["deg_seed"])
    PS = ProductSector
    bond = {}
    for n in range(-4, 5):
        for sz in range(-4, 5):
            if (sz - n) % 2 == 0:
                bond[PS(n, sz, n % 2)] = int(np.clip(rng.poisson(case["lam"]), 1, 256))
    mpo = {PS(0, 0, 0): 2, PS(1, 1, 1): 1, PS(1, -1, 1): 1, PS(-1, -1, 1): 1, PS(-1, 1, 1): 1}
    phys = {PS(0, 0, 0): 1, PS(1, 1, 1): 1, PS(1, -1, 1): 1, PS(2, 0, 0): 1}
    V, M, P = (GradedSpace.new(U1xU1xfZ2, d) for d in (bond, mpo, phys))
    return (TensorStructure((Leg(V, IN), Leg(M, OUT, True), Leg(V, OUT))),
            TensorStructure((Leg(V, OUT), Leg(P, OUT), Leg(V, IN))),
            TensorStructure((Leg(M, IN, True), Leg(P, OUT), Leg(P, IN), Leg(M, OUT, True))))


def _u1_space(d: dict) -> GradedSpace:
    return GradedSpace.new(U1, {U1.sector(q): m for q, m in d.items()})


def _tensordot_structures(case):
    V = _u1_space(_gauss(case["scale"], case["qmax"]))
    return (TensorStructure(tuple(Leg(V, OUT) for _ in range(4))),
            TensorStructure((Leg(V, IN), Leg(V, IN), Leg(V, OUT), Leg(V, OUT))))


_SPIN1 = {-1: 1, 0: 1, 1: 1}
_SVD_CAP = 4096  # a cap as DMRG passes one; the cutoff decides


def _site_structure(case):
    """A U(1) site tensor ``(l OUT, p OUT, r IN)`` with three physical states."""
    V, P = _u1_space(_gauss(case["scale"], case["qmax"])), _u1_space(_SPIN1)
    return TensorStructure((Leg(V, OUT), Leg(P, OUT), Leg(V, IN)))


def _dense_structures(case):
    V = _u1_space(_gauss(case["scale"], case["qmax"]))
    return _site_structure(case), TensorStructure((Leg(V, OUT), Leg(V, IN)))


def _svd_structures(case):
    """``(two-site tensor, left factor, bond matrix, right factor)``."""
    if case["group"] == "SU2":
        B, P = _space(SU2, case["bond"]), _space(SU2, "1:1")
        mid = {}
        for a, m in ((s.two_j, m) for s, m in B.sectors):
            for c in (a - 1, a + 1):
                if c >= 0:
                    mid[c] = mid.get(c, 0) + m
        K = GradedSpace.new(SU2, {SU2.sector(c): max(1, m // 2) for c, m in mid.items()})
    else:
        B, P = _space(U1, case["bond"]), _u1_space({-1: 1, 1: 1})
        mid = {}
        for s, m in B.sectors:
            for c in (s.charge - 1, s.charge + 1):
                mid[c] = mid.get(c, 0) + m
        K = _u1_space({c: max(1, m // 2) for c, m in mid.items()})
    return (TensorStructure((Leg(B, OUT), Leg(P, OUT), Leg(P, OUT), Leg(B, IN))),
            TensorStructure((Leg(B, OUT), Leg(P, OUT), Leg(K, IN))),
            TensorStructure((Leg(K, OUT), Leg(K, IN))),
            TensorStructure((Leg(K, OUT), Leg(P, OUT), Leg(B, IN))))


def _ctm_structures(case):
    chi = case["chi"]
    V = GradedSpace.new(Z2, {Z2.sector(0): chi - chi // 2, Z2.sector(1): chi // 2})
    D = GradedSpace.new(Z2, {Z2.sector(0): 1, Z2.sector(1): 1})
    return (TensorStructure((Leg(V, OUT), Leg(V, IN))),
            TensorStructure((Leg(V, IN), Leg(V, OUT), Leg(D, IN))))


# ---------------------------------------------------------------------------------------
# inputs


def _gen(seed: int):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)


def _randn(s: TensorStructure, g, scale: float = 1.0) -> SymmetricTensor:
    a = torch.randn(layout(s).size, dtype=torch.float64, device="cuda", generator=g)
    return SymmetricTensor(s, arena=a * scale)


def _decay(s: TensorStructure, decades: float) -> torch.Tensor:
    """The arena of a diagonal bond matrix ``(K OUT, K IN)`` whose sectors' values fall from
    1 by ``decades`` decades (a converged state's Schmidt values)."""
    lay = layout(s)
    parts = []
    for b in range(len(lay.sizes)):
        n = int(lay.shapes[b][0])
        x = torch.arange(n, dtype=torch.float64, device="cuda") + 0.37 * (b + 1) / len(lay.sizes)
        parts.append(torch.diag(10.0 ** (-decades * x / max(n, 2))).reshape(-1))
    return torch.cat(parts)


def _chain_env(case, seed: int):
    """``(Env, bond, two-site structure)``: the Heisenberg chain's environments around the
    middle of ``2 side + 2`` sites, every site an isometry towards the middle, bonds growing
    from the ends as the spin-1/2 chain's do up to the case's profile."""
    m, L = case["side"], 2 * case["side"] + 2

    def growth(i, tj):
        k = (i - tj) // 2
        return math.comb(i, k) - (math.comb(i, k - 1) if k else 0) if k >= 0 else 0

    def bond(i):
        d = min(i, L - i)
        prof = _profile(case["peak"], case["width"], d % 2)
        out = {tj: min(mult, growth(d, tj)) for tj, mult in prof.items() if growth(d, tj)}
        return out or {d % 2: 1}

    sp = [GradedSpace.new(SU2, {SU2.sector(a): x for a, x in bond(i).items()})
          for i in range(L + 1)]
    P, g = _space(SU2, "1:1"), _gen(seed)
    legs = [TensorStructure((Leg(sp[i], OUT), Leg(P, OUT), Leg(sp[i + 1], IN)))
            for i in range(L)]
    psi = network.MPS([_randn(s, g) for s in legs])
    psi.canonize_()
    for i in range(m):
        psi[i] = linalg.svd_truncated(_randn(legs[i], g), ((0, 1), (2,)), cutoff=0.0)[0]
    env = network.Env(psi, network.heisenberg_mpo_su2(L))
    for i in range(L - 1, m + 1, -1):
        env.update_(i, to="first")
    for i in range(m):
        env.update_(i, to="last")
    s = TensorStructure((Leg(psi[m - 1].legs[2].space, OUT), Leg(P, OUT), Leg(P, OUT),
                         Leg(psi[m + 2].legs[0].space, IN)))
    return env, m, s, g


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    st = {"kind": kind, "case": case}
    if kind == "matvec":
        fl, w, fr, aa = _heff_structures(case["bond"])
        lf = network.fold_left(_randn(fl, g), _randn(w, g))
        rf = network.fold_right(_randn(w, g), _randn(fr, g))
        st["mv"] = program.GraphMatvec(program.heff2_folded_program(lf, rf, aa))
        st["x"] = _randn(aa, g)
    elif kind == "lanczos":
        env, n, s, g = _chain_env(case, seed)
        st.update(env=env, n=n, x=_randn(s, g))
        env.lanczos(n, s, case["ncv"])  # the bond's program, as a sweep keeps it
    elif kind == "sweep":
        L = case["sites"]
        rng = np.random.default_rng(seed)
        phys = GradedSpace.new(SU2, {SU2.sector(1): 1})
        bonds = [GradedSpace.new(SU2, {SU2.sector(j): 1 for j in
                                       range(i % 2, min(i, L - i, 6) + 1, 2)})
                 for i in range(L + 1)]
        psi = network.MPS.random(phys, bonds, seed=int(seed) % 10007).canonize_()
        h = network.heisenberg_mpo_su2(L, j=1.0 + 0.2 * float(rng.random()))
        env = network.Env(psi, h).setup_()
        for _ in range(6):
            network.sweep_(psi, h, env, chi=case["chi"], cutoff=1e-10, ncv=case["ncv"])
        st.update(psi=psi, h=h, env=env)
    elif kind == "tensordot":
        sa, sb = _tensordot_structures(case)
        st.update(a=_randn(sa, g), b=_randn(sb, g))
    elif kind == "env_batch":
        sf, sa, sw = _env_structures(case)

        def values(s, rows):
            return torch.randn((rows, layout(s).size), dtype=torch.float32, device="cuda",
                               generator=g).double()

        n = case["n"]
        st["f"] = batch.TensorBatch(sf, values(sf, n), n)
        st["a"] = batch.TensorBatch(sa, values(sa, n), n)
        st["w"] = batch.TensorBatch.broadcast(SymmetricTensor(sw, arena=values(sw, 1)[0]), n)
    elif kind == "heff_batch":
        fl, w, fr, aa = _heff_structures(case["bond"])
        n = case["n"]

        def stack(s):
            return batch.TensorBatch(s, torch.randn((n, layout(s).size), dtype=torch.float64,
                                                    device="cuda", generator=g), n)

        w1, w2 = (batch.TensorBatch.broadcast(_randn(w, g), n) for _ in range(2))
        st["prog"] = batch.BatchedHeff2(stack(fl), w1, w2, stack(fr), aa)
        st["x"] = stack(aa)
    elif kind == "svd":
        st["x"] = _svd_input(case, seed)
    elif kind == "ctm_move":
        bulk, c, e = _ctm_input(case, seed)
        st.update(absorb=network.Absorb(bulk), c=c, e=e)
    elif kind == "lq":
        st["x"] = _randn(_site_structure(case), g)
    else:
        sa, sb = _dense_structures(case)
        st.update(a=_randn(sa, g), b=_randn(sb, g))
    return st


def _svd_input(case, seed):
    """A two-site tensor as a solve leaves it: Schmidt values falling by three decades, then
    a tail of noise below the cutoff (so every seed keeps the same counts)."""
    saa, sx, sk, sy = _svd_structures(case)
    g = _gen(seed)
    x, y = _randn(sx, g), _randn(sy, g)
    mid = SymmetricTensor(sk, arena=_decay(sk, 3.0))
    t = ops.einsum("apx,xqr->apqr", ops.einsum("apx,xy->apy", x, mid), y)
    t = t / ops.norm(t)
    assert t.structure == saa
    return SymmetricTensor(saa, arena=t.arena + 1e-9 * torch.randn(
        t.arena.numel(), dtype=torch.float64, device="cuda", generator=g))


def _ctm_keep(case):
    """The bond the move keeps: twice the corner's significant values (``_ctm_input``)."""
    chi = case["chi"]
    return 2 * ((chi - chi // 2) // 2 + chi // 2 // 2)


def _ctm_input(case, seed):
    """A corner whose values fall by a decade over the first half of each sector and lie at
    rounding's edge in the second, as a converged corner's tail does: the enlarged corner
    then has twice as many significant values, the same count per parity for every seed."""
    sc, se = _ctm_structures(case)
    chi, g = case["chi"], _gen(seed)
    rng = np.random.default_rng(seed)
    bulk = network.ising_bulk(0.43 + 0.02 * float(rng.random()))
    c = []
    for n in (chi - chi // 2, chi // 2):
        x = torch.arange(n, dtype=torch.float64, device="cuda")
        x = 10.0 ** (-x / max(1, n // 2)) * (1.0 + 0.1 * torch.rand(
            n, dtype=torch.float64, device="cuda", generator=g))
        x[n // 2:] *= 1e-6
        c.append(torch.diag(x).reshape(-1))
    e = torch.randn(layout(se).size, dtype=torch.float64, device="cuda", generator=g)
    return bulk, SymmetricTensor(sc, arena=torch.cat(c)), SymmetricTensor(se, arena=e)


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "matvec":
        return state["mv"](state["x"]).arena
    if kind == "lanczos":
        energy, v = state["env"].solve(state["n"], state["x"], case["ncv"])
        return energy, v.arena
    if kind == "sweep":
        schmidt: dict = {}
        energy, _ = network.sweep_(state["psi"], state["h"], state["env"], schmidt,
                                   chi=case["chi"], cutoff=1e-10, ncv=case["ncv"])
        return energy, [np.array(schmidt[n]) for n in sorted(schmidt)]
    if kind == "tensordot":
        return tenet.einsum("abcd,cdef->abef", state["a"], state["b"]).arena
    if kind == "env_batch":
        prec = case["precision"]
        with ops.precision(prec, None if prec == "f64" else 0):
            return batch.env_update_last(state["f"], state["a"], state["w"]).arena
    if kind == "heff_batch":
        return state["prog"](state["x"]).arena
    if kind == "svd":
        u, s, vh = linalg.svd_truncated(state["x"], ((0, 1), (2, 3)),
                                        max_bond=_SVD_CAP, cutoff=1e-10)
        return u.arena, s.arena, vh.arena
    if kind == "ctm_move":
        c, e, _ = network.move(state["c"], state["e"], state["absorb"],
                               chi=_ctm_keep(case))
        return c.arena, e.arena
    if kind == "lq":
        left, q = linalg.lq(state["x"], ((0,), (1, 2)))
        return left.arena, q.arena
    with ops.precision(case["precision"]):
        return tenet.einsum("apc,cd->apd", state["a"], state["b"]).arena


# ---------------------------------------------------------------------------------------
# work: every input read once, every output written once, 2 M N K per sector product


def _einsum_s(eq, sa, sb):
    lhs, out = eq.split("->")
    ta, tb = lhs.split(",")
    shared = [x for x in ta if x in tb]
    axes = (tuple(ta.index(x) for x in shared), tuple(tb.index(x) for x in shared))
    ex = ops.contraction_exec(sa, sb, axes)
    free = [x for x in ta if x not in shared] + [x for x in tb if x not in shared]
    return transpose_plan(ex.out, tuple(free.index(x) for x in out))[0], ex.flops


def _heff_work(bond: str):
    """Bytes of the folded operands, input and output, and flops, of one two-site matvec in
    its two-contraction form."""
    fl, w, fr, aa = _heff_structures(bond)
    lf, _ = _einsum_s("axB,xPpm->aBPpm", fl, w)
    rf, _ = _einsum_s("mQqy,rys->mQqrs", w, fr)
    t, f0 = _einsum_s("apqr,mQqrs->apmQs", aa, rf)
    _, f1 = _einsum_s("apmQs,aBPpm->BPQs", t, lf)
    return 8 * (layout(lf).size + layout(rf).size), 16 * layout(aa).size, f0 + f1


def _sectors(s, outs, ins):
    return [matrix_layout(repartition_plan(s, outs, ins)[0]).shape[c]
            for c in matrix_layout(repartition_plan(s, outs, ins)[0]).sectors]


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        env, io, flops = _heff_work(case["bond"])
        return {"bytes": env + io, "flops": flops}
    if kind == "heff_batch":
        env, io, flops = _heff_work(case["bond"])
        return {"bytes": case["n"] * (env + io), "flops": case["n"] * flops}
    if kind == "lanczos":
        env, io, flops = _heff_work(_text(_profile(case["peak"], case["width"],
                                                   case["side"] % 2)))
        # the operands and the start vector once; each step's vector written and read
        return {"bytes": env + case["ncv"] * io, "flops": case["ncv"] * flops}
    if kind == "sweep":
        chi = case["chi"]
        peak = chi / 12.0  # the dense dimension sum (2j + 1) m of the profile is about 12 peak
        env, io, flops = _heff_work(_text(_profile(peak, 12.0, 0)))
        steps = 2 * (case["sites"] - 1)
        return {"bytes": steps * (env + case["ncv"] * io) / 2,
                "flops": steps * case["ncv"] * flops / 2}
    if kind in ("tensordot", "dense"):
        sa, sb = _tensordot_structures(case) if kind == "tensordot" else _dense_structures(case)
        so, flops = _einsum_s("abcd,cdef->abef" if kind == "tensordot" else "apc,cd->apd",
                              sa, sb)
        return {"bytes": 8 * sum(layout(s).size for s in (sa, sb, so)), "flops": flops}
    if kind == "env_batch":
        sf, sa, sw = _env_structures(case)
        t, f0 = _einsum_s("axB,apr->xBpr", sf, sa)
        t, f1 = _einsum_s("xPpm,xBpr->BrPm", sw, t)
        so, f2 = _einsum_s("BPs,BrPm->rms", adjoint_plan(sa)[0], t)
        per = 8 * (layout(sf).size + layout(sa).size + layout(so).size)
        return {"bytes": case["n"] * per + 8 * layout(sw).size, "flops": case["n"] * (f0 + f1 + f2)}
    if kind == "svd":
        s = _svd_structures(case)[0]
        flops = sum(14 * max(m, n) * min(m, n) ** 2 + 8 * min(m, n) ** 3
                    for m, n in _sectors(s, (0, 1), (2, 3)))
        return {"bytes": 3 * 8 * layout(s).size, "flops": flops}
    if kind == "ctm_move":
        chi = case["chi"]
        # two sectors of chi x chi (the enlarged corner) to factorise, the absorption and
        # the projection products: half of the dense products' flops by parity
        flops = 2 * 22 * chi ** 3 + (2 * chi ** 3 * (2 + 4 + 8) + 2 * chi ** 3 * (8 + 8)) / 2
        return {"bytes": 8 * (chi * chi / 2 + 2 * chi * chi / 2 * 2 + 4 * chi * chi / 2),
                "flops": flops}
    s = _site_structure(case)
    flops = sum(4 * max(m, n) * min(m, n) ** 2 for m, n in _sectors(s, (0,), (1, 2)))
    return {"bytes": 2 * 8 * layout(s).size, "flops": flops}


# ---------------------------------------------------------------------------------------
# exact: U(1) and Z2 tensors as dense arrays.  A block is one (OUT labels, IN labels) pair
# with equal fused charge, blocks sorted by those label tuples, C-order in leg order.


def _blocks(legs, z2=False):
    """``legs``: (degeneracies by label, is OUT, dual) each.  Yields each block's leg labels
    in block order."""
    def fused(leg, a):
        return -a if leg[2] and not z2 else a

    outs = [i for i, leg in enumerate(legs) if leg[1]]
    ins = [i for i, leg in enumerate(legs) if not leg[1]]
    total = (lambda t: sum(t) % 2) if z2 else sum
    by: dict = {}
    for it in sorted(product(*(sorted(fused(legs[i], a) for a in legs[i][0]) for i in ins))):
        by.setdefault(total(it), []).append(it)
    for ot in sorted(product(*(sorted(fused(legs[i], a) for a in legs[i][0]) for i in outs))):
        for it in by.get(total(ot), []):
            lab = [0] * len(legs)
            for i, a in (*zip(outs, ot), *zip(ins, it)):
                lab[i] = fused(legs[i], a)
            yield lab


def _slices(legs, lab):
    out = []
    for leg, a in zip(legs, lab):
        o = sum(m for b, m in leg[0].items() if b < a)
        out.append(slice(o, o + leg[0][a]))
    return tuple(out)


def _to_dense(arena, legs, z2=False):
    x = torch.zeros([sum(leg[0].values()) for leg in legs], dtype=torch.float64,
                    device=arena.device)
    o = 0
    for lab in _blocks(legs, z2):
        shape = [leg[0][a] for leg, a in zip(legs, lab)]
        n = math.prod(shape)
        x[_slices(legs, lab)] = arena[o:o + n].reshape(shape)
        o += n
    assert o == arena.numel()
    return x


def _from_dense(x, legs, z2=False):
    return torch.cat([x[_slices(legs, lab)].reshape(-1) for lab in _blocks(legs, z2)])


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind == "tensordot":
        d = _gauss(case["scale"], case["qmax"])
        la, lb = [(d, True, False)] * 4, [(d, False, False)] * 2 + [(d, True, False)] * 2
        sa, sb = _tensordot_structures(case)
        a, b = (_to_dense(_randn(s, g).arena, leg) for s, leg in ((sa, la), (sb, lb)))
        return _from_dense(torch.einsum("abcd,cdef->abef", a, b), la)
    if kind == "dense":
        d = _gauss(case["scale"], case["qmax"])
        la = [(d, True, False), (_SPIN1, True, False), (d, False, False)]
        lb = [(d, True, False), (d, False, False)]
        sa, sb = _dense_structures(case)
        a, b = (_to_dense(_randn(s, g).arena, leg) for s, leg in ((sa, la), (sb, lb)))
        return _from_dense(torch.einsum("apc,cd->apd", a, b), la)
    if kind == "lq":
        return _exact_lq(case, _randn(_site_structure(case), g).arena)
    if kind == "svd" and case["group"] == "U1":
        return _exact_svd(case, _svd_input(case, seed).arena)
    if kind == "ctm_move":
        return _exact_ctm(case, *_ctm_input(case, seed))
    return None


def _exact_lq(case, arena):
    """Per left charge the QR of the transposed sector matrix (columns: the pairs (p, r) with
    r - p the left charge, sorted by -p), LAPACK's signs."""
    d = _gauss(case["scale"], case["qmax"])
    x = _to_dense(arena, [(d, True, False), (_SPIN1, True, False), (d, False, False)]).cpu().numpy()
    off = {a: sum(m for b, m in d.items() if b < a) for a in d}
    L, Q = {}, {}
    for c in sorted(d):
        cols = [(p, c + p) for p in (1, 0, -1) if c + p in d]
        row = slice(off[c], off[c] + d[c])
        B = np.concatenate([x[row, p + 1, off[r]:off[r] + d[r]] for p, r in cols], axis=1)
        q, r = np.linalg.qr(B.T)
        L[c], at = r.T, 0
        for p, rr in cols:
            Q[c, p, rr], at = q.T[:, at:at + d[rr]], at + d[rr]
    # Q's legs are (bond OUT, p IN dual, r IN): blocks by (charge, -p, r)
    left = np.concatenate([L[c].ravel() for c in sorted(L)])
    right = np.concatenate([Q[k].ravel() for k in sorted(Q, key=lambda k: (k[0], -k[1], k[2]))])
    return torch.from_numpy(left), torch.from_numpy(right)


def _kept(values, max_bond, cutoff):
    """Kept counts per sector: the global descending order under a relative cutoff on the
    discarded squares and a cap on the number kept."""
    flat = sorted(((-float(s), c) for c, v in values.items() for s in v))
    total, dropped, n = sum(s * s for s, _ in flat), 0.0, len(flat)
    for s, _ in reversed(flat):
        if cutoff is None or dropped + s * s >= cutoff * total:
            break
        dropped, n = dropped + s * s, n - 1
    keep: dict = {}
    for _, c in flat[:min(n, max_bond)]:
        keep[c] = keep.get(c, 0) + 1
    return keep


def _exact_svd(case, arena):
    d = {int(a): int(m) for a, m in (x.split(":") for x in case["bond"].split(","))}
    p = {-1: 1, 1: 1}
    x = _to_dense(arena, [(d, True, False), (p, True, False), (p, True, False),
                          (d, False, False)]).cpu().numpy()
    off = {a: sum(m for b, m in d.items() if b < a) for a in d}
    values = {}
    for c in sorted({a + s for a in d for s in p}):
        rows = [(a, c - a) for a in d if c - a in p]
        cols = [(q, q + c) for q in p if q + c in d]
        if rows and cols:
            M = np.block([[x[off[a]:off[a] + d[a], (s + 1) // 2, (q + 1) // 2,
                             off[r]:off[r] + d[r]] for q, r in cols] for a, s in rows])
            values[c] = np.linalg.svd(M, compute_uv=False)
    keep = _kept(values, _SVD_CAP, 1e-10)
    s = [np.diag(values[c][:keep[c]]).ravel() for c in sorted(keep)]
    return None, torch.from_numpy(np.concatenate(s)), None


def _exact_ctm(case, bulk, c, e):
    """The new corner: the largest singular values of the enlarged corner, normalised."""
    chi = case["chi"]
    v, d = {0: chi - chi // 2, 1: chi // 2}, {0: 1, 1: 1}
    C = _to_dense(c.arena, [(v, True, False), (v, False, False)], True)
    E = _to_dense(e.arena, [(v, False, False), (v, True, False), (d, False, False)], True)
    B = _to_dense(bulk.arena, [(d, True, False)] * 2 + [(d, False, False)] * 2, True)
    t = torch.einsum("ab,ace->bce", C, E)
    t = torch.einsum("bce,fbg->cefg", t, E)
    t = torch.einsum("cefg,gehi->chfi", t, B)
    par = [(i >= v[0]) * 1 for i in range(chi)]
    M = t.reshape(2 * chi, 2 * chi).cpu().numpy()
    row = np.array([(a + b) % 2 for a in par for b in (0, 1)])
    values = {k: np.linalg.svd(M[np.ix_(row == k, row == k)], compute_uv=False) for k in (0, 1)}
    keep = _kept(values, _ctm_keep(case), None)
    nrm = math.sqrt(sum(float(x) ** 2 for k in keep for x in values[k][:keep[k]]))
    s = [np.diag(values[k][:keep[k]] / nrm).ravel() for k in sorted(keep)]
    return torch.from_numpy(np.concatenate(s)), None
