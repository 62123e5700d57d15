"""The one-hot GEMM's persistent tiles (k_gemm): more subtile groups than SMs
(each CTA takes several tiles), one N tile with at most 64 live columns (two
accumulator buffers) and with more, several N tiles, a ragged last subtile and
last N tile, in the dual form (max-norm checks, digit planes) and the
tensor-core form (gradient, forward splits)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,batch,L", [("dual", 1, 9800), ("dual", 16, 10001), ("dual", 17, 10001), ("dual", 66, 9733),
                                          ("tc", 1, 10001), ("tc", 16, 9729), ("tc", 17, 10001), ("tc", 40, 9800)])
def test_gemm_tiles(oracle_mod, form, batch, L):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    N = 70
    rng = np.random.default_rng(L + batch)
    base = rng.integers(0, 3, size=(1, L))
    states = np.where(rng.random((N, L)) < 0.3, rng.integers(0, 4, size=(N, L)), base).astype(np.uint8)
    w = rng.uniform(0.3, 1.0, N)
    loci = rng.permutation(L)[:batch]
    loci[0] = L - 1
    with Engine(N, L, form=_lib.FORM_DUAL if form == "dual" else _lib.FORM_TC, batch=batch) as E:
        E.set_alignment(states, w)
        res, (lh, lJ, _) = E.solve(loci, want_x=True), E.lambdas()
    assert np.all(res.status == 0), res.status
    P = oracle_mod.Problem(states, w, lh, lJ)
    for k in list(range(min(batch, 6))) + [batch - 1]:
        f, g = P.objective(int(loci[k]), res.x[k])
        assert np.abs(g).max() < 2e-3, (loci[k], np.abs(g).max())
        assert abs(res.f[k] - f) <= 1e-6 * abs(f)
        assert np.isnan(res.scores[k][loci[k]]) and np.isfinite(np.delete(res.scores[k], loci[k])).all()
