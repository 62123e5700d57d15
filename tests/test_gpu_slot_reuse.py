"""Slots that many loci pass through one after the other: what a locus leaves
in its slot (parameters, logits, history, target states, solver state) does
not reach the next.  Odd sizes, one slot and several, every form, also from a
given start point; by the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["gather", "tc", "dual"])
@pytest.mark.parametrize("N,L,batch", [(1, 9, 1), (63, 17, 2), (65, 40, 3), (129, 31, 7), (640, 25, 1)])
def test_slot_reuse(oracle_mod, form, N, L, batch):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    fm = dict(gather=_lib.FORM_GATHER, tc=_lib.FORM_TC, dual=_lib.FORM_DUAL)[form]
    rng = np.random.default_rng(N + 7 * L)
    st = rng.integers(0, 4, size=(N, L)).astype(np.uint8)
    w = rng.uniform(0.2, 1.0, size=N)
    order = np.concatenate([np.arange(L), np.arange(L)[::-1]]).astype(np.uint32)
    with Engine(N, L, form=fm, batch=batch) as E:
        E.set_alignment(st, w)
        lh, lJ, _ = E.lambdas()
        P = oracle_mod.Problem(st, w, lh, lJ)
        runs = [E.solve(order, want_x=True)]
        if form != "dual":
            runs.append(E.solve(order, want_x=True, x_init=rng.normal(size=(len(order), 16 * L + 4)) * 0.01))
    for res in runs:
        for k, r in enumerate(order):
            f64, g64 = P.objective(int(r), res.x[k])
            assert res.f[k] == pytest.approx(f64, rel=1e-6), (k, r)
            assert np.abs(g64).max() < 2e-3, (k, r)
