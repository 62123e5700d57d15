"""A stand-in for the CUDA runtime, preloaded under the engine library so that
its host code runs without a GPU: device memory is host memory, copies are
copies, launches are recorded and checked but run nothing.  It has two devices
and refuses what the runtime refuses (a launch with more dynamic shared memory
than the kernel's limit on the current device)."""
import os
import shutil
import subprocess
import sys

import pytest

RUNTIME = r"""
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>

struct Dim3 { unsigned x, y, z; };
struct Config { Dim3 grid, block; size_t smem; void *stream; };
static int device = 0, refuse_limit = 0, pending = 0, launches = 0, bad_padding = 0, transposes = 0;
static std::map<const void *, std::string> &names()
{
    static std::map<const void *, std::string> m;   // (filled by the library's static initialisers)
    return m;
}
static std::map<std::pair<int, const void *>, int> limit;
static Config config;

extern "C" {
void standin_device(int d) { device = d; }
void standin_refuse_limit(int r) { refuse_limit = r; }
int standin_launches() { const int n = launches; launches = 0; return n; }

int standin_bad_padding() { return bad_padding; }
int standin_transposes() { return transposes; }

int cudaGetDeviceCount(int *n) { *n = 2; return 0; }
int cudaSetDevice(int d) { device = d; return 0; }
int cudaGetDevice(int *d) { *d = device; return 0; }
int cudaDeviceGetAttribute(int *v, int, int) { *v = 152; return 0; }
// (fresh memory holds anything)
int cudaMalloc(void **p, size_t n) { *p = std::malloc(n); if (*p) std::memset(*p, 0xA5, n); return *p ? 0 : 2; }
int cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
int cudaFree(void *p) { std::free(p); return 0; }
int cudaFreeHost(void *p) { std::free(p); return 0; }
int cudaStreamCreateWithFlags(void **s, unsigned) { *s = &config; return 0; }
int cudaStreamSynchronize(void *) { return 0; }
int cudaStreamDestroy(void *) { return 0; }
int cudaEventCreate(void **e) { *e = &config; return 0; }
int cudaEventDestroy(void *) { return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *) { std::memcpy(d, s, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *) { std::memset(d, v, n); return 0; }
int cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t n, int, void *)
{
    for (size_t i = 0; i < n; ++i) std::memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return 0;
}
int cudaMemset2DAsync(void *d, size_t dp, int v, size_t w, size_t n, void *)
{
    for (size_t i = 0; i < n; ++i) std::memset((char *)d + i * dp, v, w);
    return 0;
}
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
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *,
                            int *)
{
    names()[host] = name;
}
static int launch(const void *f, void **args, size_t smem)
{
    if (names()[f].find("k_transpose") != std::string::npos) {
        // X [N][Lx]: whole rows are read, so nothing but zeros may follow the last locus
        const unsigned char *X = *static_cast<const unsigned char **>(args[0]);
        const long long Lx = *static_cast<long long *>(args[1]);
        const int N = *static_cast<int *>(args[2]), L = *static_cast<int *>(args[3]);
        for (int i = 0; i < N; ++i)
            for (long long n = L; n < Lx; ++n) bad_padding += X[i * Lx + n] != 0;
        ++transposes;
    }
    const auto it = limit.find({device, f});
    if (smem > 48 * 1024 && (it == limit.end() || (size_t)it->second < smem)) return pending = 1;
    ++launches;
    return 0;
}
int __cudaLaunchKernel(const void *k, Dim3, Dim3, void **args, size_t smem, void *) { return launch(k, args, smem); }
int cudaLaunchKernel(const void *k, Dim3, Dim3, void **args, size_t smem, void *) { return launch(k, args, smem); }
}
"""


def build(directory):
    """The stand-in as a shared library in `directory`."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    (directory / "standin.cpp").write_text(RUNTIME)
    so = str(directory / "standin.so")
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", str(directory / "standin.cpp"), "-o", so], check=True)
    return so


def run(so, code, *args):
    """`code` in a child process with the stand-in preloaded; its last line of output."""
    out = subprocess.run([sys.executable, "-c", code, *args], capture_output=True, text=True,
                         env=dict(os.environ, LD_PRELOAD=so), timeout=120)
    assert out.returncode == 0, out.stderr[-2000:]
    return out.stdout.strip().splitlines()[-1]
