"""sdca_eval_noalloc in place: g is x, or holds the weights.  Both must give
the FP64 oracle's value and gradient, as with buffers apart, whether the
logits come in one slice or several and the gradient in one share or several."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shared", ["x", "weights"])
@pytest.mark.parametrize("N,L", [(1, 2), (33, 17), (257, 449), (600, 64), (900, 897), (70, 70001), (3000, 130)])
def test_eval_noalloc_in_place(engine_lib, oracle_mod, shared, N, L):
    import torch

    from superdca_gb300 import _lib

    rng = np.random.default_rng(N * 5 + L)
    st = rng.integers(0, 4, size=(N, L)).astype(np.uint8)
    w = rng.uniform(0.0, 1.0, size=N)
    dev = torch.device("cuda", 0)
    D = 16 * L + 4
    x = rng.normal(size=D) / np.sqrt(L)
    r = L // 2
    f64, g64 = oracle_mod.Problem(st, w, 0.3, 0.7).objective(r, x)
    d_states = torch.from_numpy(st).to(dev)
    d_g = torch.full((max(D, N),), float("nan"), dtype=torch.float64, device=dev)
    d_f = torch.full((1,), float("nan"), dtype=torch.float64, device=dev)
    d_x = d_g[:D] if shared == "x" else torch.empty(D, dtype=torch.float64, device=dev)
    d_w = d_g[:N] if shared == "weights" else torch.empty(N, dtype=torch.float64, device=dev)
    d_x.copy_(torch.from_numpy(x))
    d_w.copy_(torch.from_numpy(w))
    p = lambda t: C.c_void_p(t.data_ptr())
    assert engine_lib.sdca_eval_noalloc(p(d_states), N, L, p(d_w), 0.3, 0.7, r, p(d_x), p(d_f), p(d_g),
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream)) == _lib.SDCA_OK
    f, g = float(d_f.cpu()[0]), d_g[:D].cpu().numpy()
    # sums of at most 70,001 (logits) and 3000 (gradient) terms of order one in FP64
    assert f == pytest.approx(f64, rel=1e-12)
    np.testing.assert_allclose(g, g64, rtol=0, atol=1e-11 * max(1.0, np.abs(g64).max()))
