"""The start network's calls on several devices of one process.  Its kernels
need more dynamic shared memory than a launch gets by default, and the raised
limit belongs to one device: every device needs it, and a call that cannot
raise it has to say so each time, not only the first.  The library runs here
on the stand-in for the CUDA runtime (cuda_standin.py).  No GPU."""
import json

import pytest

import cuda_standin

CHILD = r"""
import ctypes as C, json, sys
import numpy as np
fake = C.CDLL(sys.argv[2], mode=C.RTLD_GLOBAL)
lib = C.CDLL(sys.argv[1])
M = 8
blob = np.zeros(lib.sdca_mlp_blob_size(), np.float32)
blob[0] = 1
X, T, out = np.zeros((M, 40), np.float32), np.zeros((M, 16), np.float32), np.zeros((M, 16), np.float32)
g, loss = np.zeros_like(blob), np.zeros(1)
p = lambda a: C.c_void_p(a.ctypes.data)
calls = {
    "grad": lambda: lib.sdca_mlp_grad(p(blob), p(X), p(T), C.c_int64(M), p(loss), p(g)),
    "predict": lambda: lib.sdca_mlp_predict(p(blob), p(X), C.c_int64(M), p(out)),
    "train": lambda: lib.sdca_mlp_train(p(blob), p(X), p(T), C.c_int64(M), 1, M, C.c_float(1e-3), C.c_uint64(1), p(loss)),
}
res = []
for refuse, device in json.loads(sys.argv[3]):
    fake.standin_refuse_limit(refuse)
    fake.standin_device(device)
    for name, call in calls.items():
        rc = call()
        res.append([refuse, device, name, rc, fake.standin_launches(), fake.cudaPeekAtLastError()])
print(json.dumps(res))
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory, engine_lib):
    from superdca_gb300 import _lib

    so = cuda_standin.build(tmp_path_factory.mktemp("runtime"))
    return lambda steps: json.loads(cuda_standin.run(so, CHILD, _lib.LIB_PATH, so, json.dumps(steps)))


def test_every_device_gets_the_limit(run):
    for refuse, device, name, rc, launches, pending in run([(0, 0), (0, 1), (0, 0)]):
        assert rc == 0 and launches > 0 and pending == 0, (device, name, rc, launches, pending)


def test_a_refused_limit_is_reported_by_every_call(run):
    from superdca_gb300 import _lib

    for refuse, device, name, rc, launches, pending in run([(1, 0), (1, 0), (0, 0), (1, 1)]):
        assert rc == (_lib.SDCA_E_CUDA if refuse else _lib.SDCA_OK), (refuse, device, name, rc)
        assert pending == 0, (refuse, device, name)
