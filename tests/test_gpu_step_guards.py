"""What the whole-step kernel's callers promise beside its values
(tests/test_gpu_step.py): a refused launch is an error."""
import pytest

from swb200 import abi
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
