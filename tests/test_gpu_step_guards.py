"""What the whole-step kernel's callers promise beside its values
(tests/test_gpu_step.py): a refused launch is an error; any CUDA context of
the process may use them."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import REPO, assert_bitwise, seeded_inputs
from swb200 import Model, Parameter, abi, initial_conditions, model_setup
from swb200.ensemble import Member, _batch_create, run_batched

pytestmark = pytest.mark.gpu


def members(n, **kw):
    return [Member(k, {**dict(nx=32, Ndays=0.1), **kw}, seed=k) for k in range(n)]


@pytest.mark.parametrize("nth", ["2", "3"])   # after the ghost points of the member's state: the even, the odd steps' launch
def test_a_refused_batch_launch_fails_the_run(nth, monkeypatch):
    """A step launch that CUDA refuses while the batch's graph is captured
    must not leave a graph without the step: the run reports the error."""
    lib = abi.load_library()
    monkeypatch.setenv("SWB200_TEST_FAIL_LAUNCH", nth)
    b, _, _ = _batch_create(members(2), lib)
    status = (abi.SwStatus * 2)()
    try:
        assert lib.sw_batch_run(b, 1 << 62, status) == abi.SW_ERR_CUDA
    finally:
        lib.sw_batch_destroy(b)
    monkeypatch.delenv("SWB200_TEST_FAIL_LAUNCH")
    rows = run_batched(members(2))
    assert all(r[3] == 0 for r in rows.values())


SECOND_CONTEXT = """
import ctypes as C, os, sys
import numpy as np
from swb200 import Model, Parameter, initial_conditions, model_setup
from swb200.ensemble import Member, run_batched

RUNS = [dict(nx=512), dict(nx=200, T=np.float64, topography="seamount"), dict(nx=128, time_scheme="SSPRK3"),
        dict(nx=64, adv_scheme="Sadourny", topography="flat"), dict(nx=128, storage="bf16"), dict(nx=128, storage="f16"),
        dict(nx=256, env=dict(SWB200_TMA="1"))]

def everything():
    out = []
    for kw in RUNS:
        kw = dict(kw)
        storage, env = kw.pop("storage", "native"), kw.pop("env", {})
        P = Parameter(**{**dict(Ndays=1.0, Uadv=1000, initial_cond="rest"), **kw})
        S = model_setup(P)
        eta = np.random.default_rng(1).normal(0, 0.01, (S.grid.ny, S.grid.nx))
        os.environ.update(env)
        with Model(S, storage=storage) as m:
            m.set_state(initial_conditions(P.Tprog, S, η0=eta))
            assert m.run(3).code == 0
            out += list(m.get_state())
        for k in env:
            del os.environ[k]
    _, final = run_batched([Member(k, dict(nx=[48, 200][k], Ndays=0.1), seed=k) for k in range(2)], return_states=True)
    return out + [f for k in sorted(final) for f in final[k]]

first = everything()
cu = C.CDLL("libcuda.so.1")
dev, ctx = C.c_int(), C.c_void_p()
assert cu.cuDeviceGet(C.byref(dev), 0) == 0 and cu.cuCtxCreate_v2(C.byref(ctx), 0, dev) == 0
second = everything()
assert len(first) == len(second) > 0
for k, (a, b) in enumerate(zip(first, second)):
    assert np.isfinite(a).all() and np.array_equal(a, b), k
print("equal")
"""


def test_a_second_cuda_context_in_the_process():
    """The shared memory that the kernels ask for is allowed per device and
    CUDA context, so a process may use the library in several."""
    r = subprocess.run([sys.executable, "-c", SECOND_CONTEXT], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": os.path.join(REPO, "shallowwaters.jl_b200")})
    assert r.returncode == 0 and "equal" in r.stdout, r.stderr[-2000:]


def stopped(kw, monkeypatch, refuse=0):
    """A context that a NaN check has stopped, and what it holds; the
    ``refuse``-th of its launches reports an error."""
    monkeypatch.setenv("SWB200_GRAPHS", "0")          # every launch is the context's own
    if refuse:
        monkeypatch.setenv("SWB200_TEST_FAIL_LAUNCH", str(refuse))
    S = model_setup(Parameter(**{**dict(nx=100, Ndays=2, Uadv=1000, tracer_advection=False, output_dt=0.5), **kw}))
    Prog = initial_conditions(S.parameters.Tprog, S, **seeded_inputs(S, 5))
    Prog.u[5, 7] = np.nan
    m = Model(S)
    m.set_state(Prog)
    assert m.run(S.grid.nt).code == abi.SW_NAN_DETECTED
    return m


@pytest.mark.parametrize("kw", [dict(), dict(time_scheme="SSPRK3")])
def test_a_failed_right_hand_side_leaves_the_stop_in_place(kw, monkeypatch):
    """sw_get_rhs_input lifts the NaN stop while it runs the earlier stages
    again; when one of them fails the context is still a stopped one."""
    with stopped(kw, monkeypatch) as m:
        n = m.kernel_launches
    with stopped(kw, monkeypatch, refuse=n + 1) as m:
        with pytest.raises(abi.SwError):
            m.get_rhs_input()
        before = m.get_state()
        m.run(2)                                       # returns at once: back at the same parity
        for x, y, name in zip(m.get_state(), before, ("u", "v", "η", "sst")):
            assert_bitwise(x, y, name)


@pytest.mark.parametrize("step", ["-1", "0"])
def test_the_right_hand_side_of_a_stopped_context(step, monkeypatch):
    """Steps asked of a stopped context evaluate nothing: the input of the
    last right-hand side stays that of the step the check stopped at."""
    monkeypatch.setenv("SWB200_STEP", step)
    with stopped({}, monkeypatch) as m:
        before = m.get_rhs_input()
    with stopped({}, monkeypatch) as m:
        for n in (2, 1, 3):
            m.run(n)
            for x, y, name in zip(m.get_rhs_input(), before, ("u", "v", "η")):
                assert_bitwise(x, y, name)
