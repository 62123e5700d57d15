"""sdca_eval_noalloc at the edges of its passes: 16-locus steps and their
last quad, one to four sequences per thread and several sequence blocks, one
slice of logits (few loci) and many, one share of the gradient and several,
448-locus blocks, every alignment of the states' address, the first and last
locus as target; against the FP64 oracle to FP64 accuracy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,offset", [(1, 2, 0), (31, 15, 1), (32, 16, 2), (33, 17, 3), (256, 18, 0), (257, 449, 1),
                                        (600, 64, 2), (900, 897, 3), (1025, 130, 0), (2100, 3, 1), (5000, 2, 0),
                                        (70, 70001, 1)])
def test_eval_noalloc_shapes(engine_lib, oracle_mod, N, L, offset):
    import torch

    from superdca_gb300 import _lib

    rng = np.random.default_rng(N * 7 + L)
    st = rng.integers(0, 4, size=(N, L)).astype(np.uint8)
    w = rng.uniform(0.0, 1.0, size=N)
    dev = torch.device("cuda", 0)
    raw = torch.zeros(N * L + offset, dtype=torch.uint8, device=dev)
    d_states = raw[offset:]
    d_states.copy_(torch.from_numpy(st.reshape(-1)))
    D = 16 * L + 4
    x = rng.normal(size=D) / np.sqrt(L)
    d_w, d_x = torch.from_numpy(w).to(dev), torch.from_numpy(x).to(dev)
    d_f = torch.full((1,), float("nan"), dtype=torch.float64, device=dev)
    d_g = torch.full((D,), float("nan"), dtype=torch.float64, device=dev)
    P = oracle_mod.Problem(st, w, 0.3, 0.7)
    p = lambda t: C.c_void_p(t.data_ptr())
    for r in {0, L // 2, L - 1}:
        rc = engine_lib.sdca_eval_noalloc(p(d_states), N, L, p(d_w), 0.3, 0.7, r, p(d_x), p(d_f), p(d_g),
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == _lib.SDCA_OK
        f, g = float(d_f.cpu()[0]), d_g.cpu().numpy()
        f64, g64 = P.objective(int(r), x)
        # sums of at most 70,001 (logits) and 5000 (gradient) terms of order one in FP64
        assert f == pytest.approx(f64, rel=1e-12)
        np.testing.assert_allclose(g, g64, rtol=0, atol=1e-11 * max(1.0, np.abs(g64).max()))
