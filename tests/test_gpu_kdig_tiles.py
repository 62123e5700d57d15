"""The exact K rho product (k_kdig) with more tiles (256-row pairs x 17-slot
groups) than its 76 CTA pairs: a pair then walks several tiles, its barrier
phases and its loads running on from one to the next.  With one, two and three
1536-sequence segments a tile (an odd count flips the accumulators' parity
between tiles), and a last slot group that is partly live.  All loci against
the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,batch,tiles", [(640, 450, 450, 81), (1000, 700, 700, 168), (1600, 200, 200, 84),
                                             (3201, 110, 110, 91)])
def test_kdig_more_tiles_than_pairs(oracle_mod, N, L, batch, tiles):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    assert (-(-N // 64) * 64 + 255) // 256 * -(-batch // 17) == tiles > 76
    rng = np.random.default_rng(N + batch)
    base = rng.integers(0, 3, size=(1, L))
    states = np.where(rng.random((N, L)) < 0.3, rng.integers(0, 4, size=(N, L)), base).astype(np.uint8)
    w = rng.uniform(0.2, 1.0, N)
    with Engine(N, L, form=_lib.FORM_DUAL, batch=batch) as E:
        E.set_alignment(states, w)
        res, (lh, lJ, _) = E.solve(np.arange(L), want_x=True), E.lambdas()
    assert np.all(res.status == 0), res.status
    P = oracle_mod.Problem(states, w, lh, lJ)
    for r in range(L):
        f, g = P.objective(r, res.x[r])
        assert np.abs(g).max() < 1.05e-3, (r, np.abs(g).max())
        assert abs(res.f[r] - f) <= 1e-6 * abs(f)
