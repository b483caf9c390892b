"""The kernels' opt-in to more than 48 KB of dynamic shared memory is made on every
device that a process uses, and made again where it failed: the launchers of the ghost
update, the cell update and the adjoint run in a process whose CUDA runtime is a fake
(no GPU, nothing launched) that refuses a launch beyond 48 KB on a device where the
kernel was not set up."""
import os
import re
import subprocess
import sys

import pytest

FAKE = r"""
#include <cstddef>
#include <map>
#include <utility>
struct dim3_ { unsigned x, y, z; };
static int dev = 0, refuse = 0, launches = 0, bad = 0, sets = 0;
static std::map<std::pair<int, const void*>, int> most;
static struct { dim3_ g, b; size_t smem; void* s; } cfg;
extern "C" {
int cudaGetDevice(int* d) { *d = dev; return 0; }
int cudaDeviceGetAttribute(int* v, int, int) { *v = 148; return 0; }
int cudaFuncSetAttribute(const void* f, int attr, int v) {
    ++sets;
    if (refuse > 0) { --refuse; return 1; }
    if (attr == 8) most[{dev, f}] = v; // cudaFuncAttributeMaxDynamicSharedMemorySize
    return 0;
}
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t smem, void* s) { cfg = {g, b, smem, s}; return 0; }
int __cudaPopCallConfiguration(dim3_* g, dim3_* b, size_t* smem, void** s) {
    *g = cfg.g; *b = cfg.b; *smem = cfg.smem; *s = cfg.s;
    return 0;
}
int cudaLaunchKernel(const void* f, dim3_, dim3_, void**, size_t smem, void*) {
    ++launches;
    auto it = most.find({dev, f});
    if (smem > 49152 && (it == most.end() || it->second < (int)smem)) { ++bad; return 1; }
    return 0;
}
int fake_set(int d, int r) { dev = d; refuse = r; return 0; }
int fake_counts(int* out) { out[0] = launches; out[1] = bad; out[2] = sets; launches = bad = sets = 0; return 0; }
}
"""

DRIVER = r"""
import ctypes as C, sys
fake, lib, adj, ghosts, rhs = sys.argv[1:]
F = C.CDLL(fake, mode=C.RTLD_GLOBAL)
L = C.CDLL(lib)
p, i, q = C.c_void_p, C.c_int, C.c_longlong
def call(dev, refuse=0):
    F.fake_set(dev, refuse)
    f = getattr(L, adj)
    f.restype = None
    f(p(), p(), i(0), i(1), q(1000), p(), i(4), p(), i(4), p(), i(4), p(), i(8), p(), i(8), *[p()] * 7, i(1))
    f = getattr(L, ghosts)
    f.restype = None
    f(p(), p(), p(), i(8), p(), i(8), p(), p(), i(0), C.c_bool(False))
    f = getattr(L, rhs)
    f.restype = None
    f(p(), p(), p(), i(4), i(0), i(0), p(), i(60000))
    n = (i * 3)()
    F.fake_counts(n)
    print(*n)
call(0)
call(1)
call(1)
call(0)
call(3, refuse=100)
call(3)
call(70)
"""


def _symbol(lib, name):
    out = subprocess.run(["nm", "-D", "--defined-only", lib], capture_output=True, text=True, check=True).stdout
    return re.search(r"\s(_ZN4rh3t\d+" + name + r"E\S+)", out).group(1)


@pytest.mark.parametrize("exact", [False, True])
def test_attributes_on_every_device(rh, tmp_path, exact):
    src, fake = tmp_path / "fake.cpp", tmp_path / "libfake.so"
    src.write_text(FAKE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", str(src), "-o", str(fake)], check=True)
    lib = rh.lib_path(exact)
    names = [_symbol(lib, n) for n in ("launch_adj_l", "launch_ghosts", "launch_rhs_stage")]
    env = dict(os.environ, LD_PRELOAD=str(fake))
    r = subprocess.run([sys.executable, "-c", DRIVER, str(fake), lib] + names, capture_output=True, text=True, env=env)
    assert r.returncode == 0, r.stderr
    first, other, again, back, refused, retried, far = [tuple(map(int, x.split())) for x in r.stdout.split("\n") if x]
    assert first[0] > 0 and first[1] == 0 and first[2] > 0
    assert other == first                          # another device is set up as the first was
    assert again == back == (first[0], 0, 0)       # once per device
    assert refused[1] > 0                          # an opt-in that fails shows as a failed launch
    assert retried[1] == 0                         # ... and is made again
    assert far[1] == 0
