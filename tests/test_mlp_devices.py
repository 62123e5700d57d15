"""The start network's calls on several devices of one process.  Its kernels
need more dynamic shared memory than a launch gets by default, and the raised
limit belongs to one device: every device needs it, and a call that cannot
raise it has to say so each time, not only the first.  The library runs here
on a stand-in for the CUDA runtime (preloaded: host memory, two devices, no
kernel runs) that refuses what the runtime refuses.  No GPU."""
import json
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>

struct Dim3 { unsigned x, y, z; };
struct Config { Dim3 grid, block; size_t smem; void *stream; };
static int device = 0, refuse_limit = 0, pending = 0, launches = 0;
static std::map<std::pair<int, const void *>, int> limit;
static Config config;

extern "C" {
void standin_device(int d) { device = d; }
void standin_refuse_limit(int r) { refuse_limit = r; }
int standin_launches() { const int n = launches; launches = 0; return n; }

int cudaGetDevice(int *d) { *d = device; return 0; }
int cudaDeviceGetAttribute(int *v, int, int) { *v = 152; return 0; }
int cudaMalloc(void **p, size_t n) { *p = std::calloc(1, n); return *p ? 0 : 2; }
int cudaFree(void *p) { std::free(p); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int) { std::memcpy(d, s, n); return 0; }
int cudaMemset(void *d, int v, size_t n) { std::memset(d, v, n); return 0; }
int cudaGetLastError() { const int e = pending; pending = 0; return e; }
int cudaPeekAtLastError() { return pending; }
const char *cudaGetErrorString(int) { return "refused"; }
int cudaFuncSetAttribute(const void *f, int, int value)
{
    if (refuse_limit) return pending = 1;
    limit[{device, f}] = value;
    return 0;
}
unsigned __cudaPushCallConfiguration(Dim3 g, Dim3 b, size_t smem, void *st)
{
    config = {g, b, smem, st};
    return 0;
}
int __cudaPopCallConfiguration(Dim3 *g, Dim3 *b, size_t *smem, void *st)
{
    *g = config.grid;
    *b = config.block;
    *smem = config.smem;
    *static_cast<void **>(st) = config.stream;
    return 0;
}
int __cudaGetKernel(const void **k, const void *f) { *k = f; return 0; }
static int launch(const void *f, size_t smem)
{
    const auto it = limit.find({device, f});
    if (smem > 48 * 1024 && (it == limit.end() || (size_t)it->second < smem)) return pending = 1;
    ++launches;
    return 0;
}
int __cudaLaunchKernel(const void *k, Dim3, Dim3, void **, size_t smem, void *) { return launch(k, smem); }
int cudaLaunchKernel(const void *k, Dim3, Dim3, void **, size_t smem, void *) { return launch(k, smem); }
}
"""

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

    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("runtime")
    (d / "standin.cpp").write_text(RUNTIME)
    so = str(d / "standin.so")
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", str(d / "standin.cpp"), "-o", so], check=True)

    def call(steps):
        out = subprocess.run([sys.executable, "-c", CHILD, _lib.LIB_PATH, so, json.dumps(steps)], capture_output=True,
                             text=True, env=dict(os.environ, LD_PRELOAD=so), timeout=120)
        assert out.returncode == 0, out.stderr[-2000:]
        return json.loads(out.stdout.strip().splitlines()[-1])

    return call


def test_every_device_gets_the_limit(run):
    for refuse, device, name, rc, launches, pending in run([(0, 0), (0, 1), (0, 0)]):
        assert rc == 0 and launches > 0 and pending == 0, (device, name, rc, launches, pending)


def test_a_refused_limit_is_reported_by_every_call(run):
    from superdca_gb300 import _lib

    for refuse, device, name, rc, launches, pending in run([(1, 0), (1, 0), (0, 0), (1, 1)]):
        assert rc == (_lib.SDCA_E_CUDA if refuse else _lib.SDCA_OK), (refuse, device, name, rc)
        assert pending == 0, (refuse, device, name)
