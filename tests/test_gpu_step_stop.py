"""A tracer that stops the run while the next step runs beside it."""
import numpy as np
import pytest

from conftest import assert_bitwise, seeded_inputs
from swb200 import Model, Parameter, abi, initial_conditions, model_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw, storage", [(dict(), "native"), (dict(), "bf16"), (dict(T=np.float32, Tprog=np.float64), "native")])
def test_a_departure_beside_the_next_step_leaves_a_whole_state(kw, storage):
    """A NaN velocity has the first step's tracer report its departure points
    while the second step runs on several waves of blocks.  The state read
    back is one of whole steps (the block's last), not one that a part of the
    blocks wrote; later calls leave it, and a new state runs again."""
    kw = dict(nx=1400, Ndays=2.0, output_dt=24, **kw)
    block = 16

    def model(tracer):
        S = model_setup(Parameter(**kw, Uadv=1000, tracer_advection=tracer))
        return S, initial_conditions(S.parameters.Tprog, S, **seeded_inputs(S, 5))

    S, good = model(False)
    bad = initial_conditions(S.parameters.Tprog, S, **seeded_inputs(S, 5))
    bad.u[50, 700] = np.nan
    with Model(S, storage=storage) as m:
        m.set_state(bad)
        m.run(block)
        want = m.get_state()
        m.set_state(good)
        m.run(4 * block)
        want_good = m.get_state()
    S, good = model(True)
    assert S.grid.nadvstep == 1 and S.grid.nout > 6 * block
    with Model(S, storage=storage) as m:
        m.set_state(bad)
        for n in (4 * block, 2):
            with pytest.raises(abi.SwError, match="departure"):
                m.run(n)
            for x, y, name in zip(m.get_state(), want, ("u", "v", "η")):
                assert_bitwise(x, y, f"{name} after {n}")
        m.set_state(good)
        assert m.run(4 * block).code == 0
        for x, y, name in zip(m.get_state(), want_good, ("u", "v", "η")):
            assert_bitwise(x, y, name)
