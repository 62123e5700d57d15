"""The plain form's gradient kernel at the edges of its tiles (64 loci, 64
sequences, two slots per block; odd slot counts and one slot): the first
iteration from a given start point against the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,batch", [(1, 1 + 1, 1), (63, 63, 2), (64, 64, 3), (65, 65, 1), (128, 129, 5), (130, 200, 33)])
def test_plain_gradient_tiles(oracle_mod, N, L, batch):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    rng = np.random.default_rng(N * 5 + L)
    st = rng.integers(0, 4, size=(N, L)).astype(np.uint8)
    w = rng.uniform(0.2, 1.0, size=N)
    with Engine(N, L, form=_lib.FORM_GATHER, batch=batch) as E:
        E.set_alignment(st, w)
        lh, lJ, _ = E.lambdas()
        P = oracle_mod.Problem(st, w, lh, lJ)
        loci = np.arange(L, dtype=np.uint32)[::max(1, L // 40)]
        res = E.solve(loci, want_x=True)
    for k, r in enumerate(loci):
        f, g = P.objective(int(r), res.x[k])
        # gnorm is the maximum of the kernel's gradient at the last iterate;
        # both stem from FP32 sums of N terms of at most 1: N roundings
        assert np.abs(g).max() == pytest.approx(res.gnorm[k], abs=2.0 ** -23 * (N + 64))
