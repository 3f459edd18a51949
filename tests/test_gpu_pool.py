"""The device blocks that the library keeps for reuse (sw_pool.h)."""
import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

POOL = """
import ctypes as C
from swb200 import abi
lib = abi.load_library()
cu = C.CDLL("libcuda.so.1")
malloc, free = lib._ZN3swb11pool_mallocEPPvm, lib._ZN3swb9pool_freeEPvm
malloc.argtypes, free.argtypes = [C.POINTER(C.c_void_p), C.c_size_t], [C.c_void_p, C.c_size_t]
GIB = 1 << 30

def take(n):
    p = C.c_void_p()
    return p, malloc(C.byref(p), n)

def room():
    a, b = C.c_size_t(), C.c_size_t()
    assert cu.cuMemGetInfo_v2(C.byref(a), C.byref(b)) == 0
    return a.value
"""

OUT_OF_MEMORY = """
p, e = take(GIB)                       # makes the primary context
assert e == 0
free(p, GIB)
dev, ctx, now = C.c_int(), C.c_void_p(), C.c_void_p()
assert cu.cuDeviceGet(C.byref(dev), 0) == 0 and cu.cuCtxCreate_v2(C.byref(ctx), 0, dev) == 0
p, e = take(GIB)
assert e == 0
free(p, GIB)                           # kept
before = room()
p, e = take(1 << 50)
assert e == 2 and not p.value          # cudaErrorMemoryAllocation
assert cu.cuCtxGetCurrent(C.byref(now)) == 0 and now.value == ctx.value, "another context"
assert room() >= before + GIB, "the context's own blocks were given back"
print("done")
"""

NEWEST = """
import numpy as np
from swb200 import Model, Parameter, model_setup
S = model_setup(Parameter(nx=1000, Ndays=1.0))
Model(S).close()                       # makes the primary context
lib.sw_trim_memory()
start = room()
sizes = [GIB + k * (64 << 20) for k in range(14)]
for n in sizes:                        # 19.7 GiB of blocks that nothing asks for again
    p, e = take(n)
    assert e == 0
    free(p, n)
assert start - room() <= 4 * GIB + (64 << 20), "the gradient's pool"
p, e = take(sizes[-1])
before = room()
free(p, sizes[-1])
assert e == 0 and room() == before, "the newest is kept"
model = lambda: Model(S).close()
before = room()
model()
assert room() < before, "a model's blocks are kept beside them"
before = room()
model()
assert room() == before
big, e = take(5 * GIB)
assert e == 0
before = room()
free(big, 5 * GIB)
assert room() >= before + 5 * GIB, "a block above the limit goes back at once"
lib.sw_trim_memory()
assert room() >= start - (64 << 20)
print("done")
"""


def child(code):
    r = subprocess.run([sys.executable, "-c", POOL + code], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": os.path.join(REPO, "shallowwaters.jl_b200")})
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]


def test_an_allocation_that_does_not_fit_leaves_the_context():
    """It gives back what is kept for the caller's CUDA context, and the
    caller's context stays the current one."""
    child(OUT_OF_MEMORY)


def test_the_newest_blocks_are_kept():
    """The gradient's blocks stay within their bound, the oldest go first, and
    they do not keep a model's blocks out."""
    child(NEWEST)
