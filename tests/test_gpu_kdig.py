"""The exact K rho product (k_kdig) at the edges of its tiles: 256-row pairs
(N), 17-slot groups (batch), 1536-sequence segments (N), and the largest N it
takes.  A wrong digit, segment or column would leave the solver at a point
where the oracle's gradient is not small."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,batch", [(256, 33, 17), (257, 40, 18), (64, 12, 1), (1536, 30, 16), (1537, 36, 35),
                                       (3201, 24, 5), (4000, 18, 18)])
def test_kdig_tile_edges(oracle_mod, N, L, batch):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    rng = np.random.default_rng(N + batch)
    base = rng.integers(0, 3, size=(1, L))
    states = np.where(rng.random((N, L)) < 0.3, rng.integers(0, 4, size=(N, L)), base).astype(np.uint8)
    w = rng.uniform(0.2, 1.0, N)
    loci = np.arange(min(L, 36))
    with Engine(N, L, form=_lib.FORM_DUAL, batch=batch) as E:
        E.set_alignment(states, w)
        res, (lh, lJ, _) = E.solve(loci, want_x=True), E.lambdas()
    assert np.all(res.status == 0), res.status
    P = oracle_mod.Problem(states, w, lh, lJ)
    for k, r in enumerate(loci):
        f, g = P.objective(int(r), res.x[k])
        assert np.abs(g).max() < 1.05e-3, (r, np.abs(g).max())
        assert abs(res.f[k] - f) <= 1e-6 * abs(f)
