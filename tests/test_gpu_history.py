"""History products and directions of the plain and tensor-core forms at the
edges of their tiles (4096 entries), with
every kind of history (FP32, BF16; one pair, three, ten) and few or many
slots: the solves reach the optimum, by the FP64 oracle, in the iterations a
working direction needs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("L,m,batch", [(2, 10, 1), (255, 10, 2), (256, 3, 7), (257, 1, 40), (513, 10, 130)])
def test_history_tiles(oracle_mod, form, bf16, L, m, batch):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    N = 90
    rng = np.random.default_rng(L + m)
    st = rng.integers(0, 4, size=(N, L)).astype(np.uint8)
    st[:, 1::2] = np.where(rng.uniform(size=(N, L // 2)) < 0.2, st[:, 1::2], st[:, 0:2 * (L // 2):2])
    w = rng.uniform(0.2, 1.0, size=N)
    loci = np.arange(L, dtype=np.uint32)[:min(L, 150)]
    with Engine(N, L, form=(_lib.FORM_GATHER, _lib.FORM_TC)[form], batch=batch, history=m, history_bf16=bf16) as E:
        E.set_alignment(st, w)
        lh, lJ, _ = E.lambdas()
        res = E.solve(loci, want_x=True)
    P = oracle_mod.Problem(st, w, lh, lJ)
    for k in sorted({0, 1, len(loci) // 2, len(loci) - 1}):
        f64, g64 = P.objective(int(loci[k]), res.x[k])
        assert res.f[k] == pytest.approx(f64, rel=1e-6)
        assert np.abs(g64).max() < 2e-3
    # ill-conditioned only through lambda: L-BFGS needs some tens of iterations, steepest descent thousands
    assert res.iterations.max() < 400
