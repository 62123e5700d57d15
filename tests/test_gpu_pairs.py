"""Sequence weights, the alignment transpose and the pair distances at the
edges of their kernels: 32-locus words and 64-word chunks, 32 x 32 and 64 x 64
pair blocks (the larger from 1537 sequences on), 16-byte and 4 x 4 byte pieces
of the transpose.  Weights are exact; a wrong transpose or agreement count
would leave the solver where the oracle's gradient is not small."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _states(N, L, seed):
    rng = np.random.default_rng(seed)
    base = rng.integers(0, 4, size=(max(1, N // 6), L))
    st = base[rng.integers(0, len(base), N)]
    return np.where(rng.random((N, L)) < 0.1, rng.integers(0, 4, size=(N, L)), st).astype(np.uint8)


@pytest.mark.parametrize("N,L", [(1, 2), (2, 31), (31, 32), (33, 33), (64, 63), (65, 65), (130, 2049), (300, 4095),
                                 (1600, 130), (1537, 2111)])
def test_weights_exact(N, L):
    from superdca_gb300.engine import Engine
    st = _states(N, L, N + L)
    mult = np.random.default_rng(1).integers(1, 4, N).astype(np.float64)
    d = np.zeros((N, N), dtype=np.int64)
    for k in range(4):
        m = (st == k).astype(np.float32)
        d += np.rint(m @ m.T).astype(np.int64)
    ident = d / L
    with Engine(N, L) as E:
        for thr, mu in ((0.8, None), (0.55, mult)):
            near = (ident >= thr) & ~np.eye(N, dtype=bool)
            m = np.ones(N) if mu is None else mu
            want = m / (m + near @ m)
            np.testing.assert_array_equal(E.compute_weights(st, thr, mu), want)


@pytest.mark.parametrize("N,L", [(63, 65), (64, 64), (129, 130), (130, 200), (1600, 67)])
def test_agreements_and_transpose(oracle_mod, N, L):
    from superdca_gb300 import _lib
    from superdca_gb300.engine import Engine
    st = _states(N, L, N * L)
    w = np.random.default_rng(2).uniform(0.3, 1.0, N)
    loci = np.unique([0, 1, L // 2, L - 2, L - 1])
    for form in (_lib.FORM_DUAL, _lib.FORM_GATHER):
        with Engine(N, L, form=form, batch=4) as E:
            E.set_alignment(st, w)
            res, (lh, lJ, _) = E.solve(loci, want_x=True), E.lambdas()
        P = oracle_mod.Problem(st, w, lh, lJ)
        for k, r in enumerate(loci):
            f, g = P.objective(int(r), res.x[k])
            assert res.status[k] == 0 and np.abs(g).max() < 2e-3, (form, r, np.abs(g).max())
            assert abs(res.f[k] - f) <= 1e-6 * abs(f)


def test_codes_out_of_range_are_refused():
    """A code >= 4 anywhere, the last locus of the last sequence included."""
    from superdca_gb300 import EngineError
    from superdca_gb300.engine import Engine
    st = _states(70, 131, 5)
    with Engine(70, 131) as E:
        for i, n, v in ((69, 130, 4), (0, 0, 255), (64, 64, 7)):
            bad = st.copy()
            bad[i, n] = v
            with pytest.raises(EngineError):
                E.set_alignment(bad, np.ones(70))
        E.set_alignment(st, np.ones(70))
