"""The chained batched environment update against the contraction-by-contraction form.

Every block map involved has one term of coefficient +-1 per block, so composing them moves
the same numbers: the two forms' tables must give equal results to the bit (the products
themselves are the same tables over the same packed operands)."""

import numpy as np
import pytest

import _emulate
from tenet import batch, ops
from tenet.structure import IN, OUT, GradedSpace, Leg, TensorStructure, layout
from tenet.symmetry import SU2, U1, Z2, U1xU1xfZ2, fZ2


def _structures(group):
    if group == "U1xU1xfZ2":
        import bench

        V, M, P = bench.config3_spaces(7, 2.5, 4)
    else:
        p = {"U1": U1, "Z2": Z2, "fZ2": fZ2, "SU2": SU2}[group]
        V, M, P = (GradedSpace.new(p, {p.sector(q): d for q, d in x.items()}) for x in {
            "U1": ({-1: 3, 0: 4, 2: 1}, {-1: 1, 0: 2, 1: 1}, {0: 1, 1: 2}),
            "Z2": ({0: 3, 1: 5}, {0: 2, 1: 1}, {0: 1, 1: 1}),
            "fZ2": ({0: 4, 1: 3}, {0: 2, 1: 2}, {0: 2, 1: 1}),
            "SU2": ({0: 2, 2: 3}, {0: 2, 2: 1}, {0: 1, 2: 1})}[group])
    return (TensorStructure((Leg(V, IN), Leg(M, OUT, True), Leg(V, OUT))),
            TensorStructure((Leg(V, OUT), Leg(P, OUT), Leg(V, IN))),
            TensorStructure((Leg(M, IN, True), Leg(P, OUT), Leg(P, IN), Leg(M, OUT, True))))


def _step(step, a, b):
    ap, bp, cp = (np.full(max(1, x), np.nan) for x in (step.a_size, step.b_size, step.c_size))
    _emulate.gather(step.pack, a, ap, b, bp)
    _emulate.gemm(step.gemm, ap, bp, cp)
    return cp


def _einsum(eq, sa, a, a_sh, sb, b, b_sh, n):
    axes, perm = ops._pair_plan(eq, sa.ndim, sb.ndim)
    bc = batch._contraction(sa, sb, axes, n, a_sh, b_sh, "f64", None, perm)
    ap = np.full(max(1, (1 if bc.a_shared else n) * bc.a_mat), np.nan)
    bp = np.full(max(1, (1 if bc.b_shared else n) * bc.b_mat), np.nan)
    cp, out = np.full(n * bc.c_mat, np.nan), np.full(n * bc.out_size, np.nan)
    _emulate.gather(bc.pack, a, ap, b, bp)
    _emulate.gemm(bc.gemm, ap, bp, cp)
    _emulate.gather(bc.unpack, cp, out)
    return bc.out, out


@pytest.mark.parametrize("group", ["U1", "Z2", "fZ2", "U1xU1xfZ2"])
@pytest.mark.parametrize("shared", [(0, 0, 1), (0, 0, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)])
def test_chain_tables(group, shared):
    sf, sa, sw = _structures(group)
    n, rng = 3, np.random.default_rng(2)
    f, a, w = (rng.standard_normal(layout(s).size * (1 if x else n))
               for s, x in zip((sf, sa, sw), shared))
    shared = tuple(bool(x) for x in shared)
    c = batch._env_update_chain(sf, sa, sw, n, shared, "f64", None, False)
    t = _step(c.bra, a, _step(c.mpo, w, _step(c.ket, f, a)))
    got = np.full(n * c.size, np.nan)
    _emulate.gather(c.unpack, t, got)
    # contraction by contraction
    m = 1 if shared[1] else n
    sbra, table = batch._unary(sa, "a", None, None, m)
    bra = a
    if table is not None:
        bra = np.full(m * layout(sbra).size, np.nan)
        _emulate.gather(table, a, bra)
    s1, t1 = _einsum("axB,apr->xBpr", sf, f, shared[0], sa, a, shared[1], n)
    s2, t2 = _einsum("xPpm,xBpr->BrPm", sw, w, shared[2], s1, t1, False, n)
    s3, t3 = _einsum("BPs,BrPm->rms", sbra, bra, shared[1], s2, t2, False, n)
    assert c.out == s3 and np.array_equal(got, t3)


def test_chain_leaves_other_calls_to_the_contractions():
    sf, sa, sw = _structures("SU2")
    assert batch._env_update_chain(sf, sa, sw, 2, (False,) * 3, "f64", None, False) is None
    uf, ua, uw = _structures("U1")
    for args in ((sf, ua, uw), (uf, ua, ua), (ua, ua, uw), (uf, uf, uw)):
        assert batch._env_update_chain(*args, 2, (False,) * 3, "f64", None, False) is None


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "3xbf16", "tf32"])
def test_env_update_chain_on_the_device(precision):
    import torch

    from tenet import _lib

    sf, sa, sw = _structures("U1xU1xfZ2")
    g = torch.Generator(device="cuda").manual_seed(3)
    n = 5

    def make(s, shared=False):
        rows = (layout(s).size,) if shared else (n, layout(s).size)
        return batch.TensorBatch(s, torch.randn(rows, dtype=torch.float64, device="cuda",
                                                generator=g), n, shared)

    f, a, w = make(sf), make(sa), make(sw, True)
    batch.AUTOTUNE = False
    try:
        with ops.precision(precision, 0):
            got = batch.env_update_last(f, a, w)
            t = batch.einsum("axB,apr->xBpr", f, a)
            t = batch.einsum("xPpm,xBpr->BrPm", w, t)
            want = batch.einsum("BPs,BrPm->rms", batch.adjoint(a), t)
    finally:
        batch.AUTOTUNE = True
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0
    assert got.structure == want.structure and torch.equal(got.arena, want.arena)
    with pytest.raises(ValueError):
        batch.env_update_last(f, a, batch.TensorBatch(sw, w.arena, n + 1, True))
