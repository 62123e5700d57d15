"""The line searches of the plain and tensor-core forms, one cluster per slot:
sequence counts around a block's and a cluster's share, few slots (clusters of
eight) and enough for one block each.  The reported objective is the one at
the returned point and the gradient there is below the threshold, by the FP64
oracle; the searches' own counts are consistent."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("N,L,batch", [(1, 3, 1), (31, 20, 2), (256, 24, 5), (257, 24, 5), (513, 40, 40), (1024, 90, 80),
                                       (1025, 160, 160), (2049, 320, 320), (2300, 30, 3)])
def test_search_shapes(oracle_mod, form, N, L, batch):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    form = (_lib.FORM_GATHER, _lib.FORM_TC)[form]
    rng = np.random.default_rng(N + L)
    base = rng.integers(0, 2, size=(N, L)).astype(np.uint8)
    st = np.where(rng.uniform(size=(N, L)) < 0.1, rng.integers(0, 4, size=(N, L)), np.sort(base, axis=0)).astype(np.uint8)
    w = rng.uniform(0.2, 1.0, size=N)
    with Engine(N, L, form=form, batch=batch) as E:
        E.set_alignment(st, w)
        lh, lJ, _ = E.lambdas()
        loci = np.arange(L, dtype=np.uint32)
        res = E.solve(loci, want_x=True)
    P = oracle_mod.Problem(st, w, lh, lJ)
    for r in sorted({0, 1, L // 2, L - 1}):
        f64, g64 = P.objective(int(r), res.x[r])
        # the logits behind the reported value are sums of FP32 stretches of
        # 64 loci with parameters of order 1: 64 roundings of 2^-24 each
        assert res.f[r] == pytest.approx(f64, rel=64 * 2.0 ** -24)
        assert np.abs(g64).max() < 2e-3
    assert np.isin(res.status, (0, 2)).all()
    # every iteration takes at least one trial beyond its two bookkeeping evaluations
    assert (res.nfeval >= 1 + 2 * res.iterations).all()
    assert (res.iterations >= 0).all() and (res.iterations < 1000).all()
