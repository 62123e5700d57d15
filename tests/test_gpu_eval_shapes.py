"""sdca_eval at the edges of its passes: 64-locus stretches and chunks that
end half way through one, partial logits in the gradient buffers or (few loci)
in their own, 16-locus blocks of the reference layout, handles of every form
and of several slots, no gradient wanted; against the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,form,batch", [(1, 2, 0, 1), (257, 3, 0, 2), (1000, 5, 2, 1), (33, 63, 0, 1), (64, 64, 1, 3),
                                            (255, 545, 2, 8), (300, 1057, 0, 1), (70, 20033, 0, 64), (520, 4097, 2, 2)])
def test_eval_shapes(oracle_mod, N, L, form, batch):
    from superdca_gb300.engine import Engine
    rng = np.random.default_rng(N * 3 + L)
    st = rng.integers(0, 4, size=(N, L)).astype(np.uint8)
    w = rng.uniform(0.0, 1.0, size=N)
    with Engine(N, L, form=form, batch=batch) as E:
        E.set_alignment(st, w)
        lh, lJ, _ = E.lambdas()
        P = oracle_mod.Problem(st, w, lh, lJ)
        for r in {0, L // 2, L - 1}:
            x = rng.normal(size=16 * L + 4) / np.sqrt(L)
            f, g = E.eval(r, x)
            f64, g64 = P.objective(int(r), x)
            assert f == pytest.approx(f64, rel=1e-6)
            np.testing.assert_allclose(g, g64, rtol=0, atol=1e-4 * max(1.0, np.abs(g64).max()))
            # (FP64 sums over blocks in any order)
            assert E.eval(r, x, grad=False) == pytest.approx(f, rel=1e-13)
            # the gradient comes in single precision, J_rr zero
            np.testing.assert_array_equal(g, g.astype(np.float32).astype(np.float64))
        # a solve after an evaluation is unaffected by the buffers it used
        res = E.solve([L - 1], want_x=True)
        assert np.abs(P.objective(L - 1, res.x[0])[1]).max() < 2e-3
