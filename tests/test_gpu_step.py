"""The whole-step kernel (sw_step.cuh) and the blocks of steps in one graph.

* Every tile shape, at tile edges, remainders and tiles of two rows, against
  the CPU oracle, bit for bit: the kernel forms every value by the reference's
  expressions, so there is no tolerance.
* The same with two tile columns that a seam or a wall crosses, against the
  launches per stage (themselves pinned to the oracle), at sizes the oracle
  would be slow at.
* The input of the last right-hand side, which the kernel does not keep.
* The 16-bit storage form in every tile shape against its launches per stage.
* A run in blocks of steps against the same run step by step.
"""
import numpy as np
import pytest

import oracle as O
from conftest import assert_bitwise, seeded_inputs
from swb200 import Model, Parameter, initial_conditions, model_setup

pytestmark = pytest.mark.gpu

NAMES = ("u", "v", "η", "sst")
OPTIONS = [
    dict(diffusion="Smagorinsky"),                                                  # ridge: depth varies along x
    dict(topography="flat", bottom_drag="linear"),                                  # one depth per row
    dict(bc="nonperiodic", α=0.5, topography="seamount", diffusion="Smagorinsky", wind_forcing_x="double_gyre"),
    dict(bc="nonperiodic", α=2.0, topography="flat", bottom_drag="none", nstep_diff=2),
    dict(T=np.float64, topography="seamount", diffusion="Smagorinsky"),
    dict(T=np.float64, bc="nonperiodic", α=1.0, topography="flat"),
    dict(RKo=3, cfl=0.6, topography="flat", diffusion="Smagorinsky"),
    dict(RKo=2, cfl=0.3, bc="nonperiodic", α=0.0),
    dict(seasonal_wind_x=True, surface_relax=False),
]


def setup(kw, seed=3):
    P = Parameter(**{**dict(Ndays=0.5, Uadv=1000), **kw})
    S = model_setup(P)
    rng = np.random.default_rng(seed)
    G = S.grid
    inputs = seeded_inputs(S, seed)
    inputs["u0"] = 0.2 * np.sin(np.arange(G.nuy)[:, None] + 0.3 * np.arange(G.nux)) + rng.normal(0, 0.01, (G.nuy, G.nux))
    inputs["v0"] = 0.1 * np.cos(0.7 * np.arange(G.nvy)[:, None] + np.arange(G.nvx)) + rng.normal(0, 0.01, (G.nvy, G.nvx))
    return S, initial_conditions(P.Tprog, S, **inputs)


def run(S, Prog, n):
    with Model(S) as m:
        m.set_state(Prog)
        assert m.run(n).code == 0
        return m.get_state(), m.get_rhs_input()


# columns and rows around the tile widths (60, 124 and 32, 64 local columns; tiles hold 16 fewer, 20 at a seam) and
# heights (32, 56 and 64 rows), and the smallest grids
@pytest.mark.parametrize("shape", ["0", "1", "2", "3", "4"])
@pytest.mark.parametrize("size", [(4, 1), (28, 1), (56, 1), (57, 1), (61, 3), (121, 2), (125, 5)])
def test_tile_shapes_against_the_oracle(size, shape, monkeypatch):
    monkeypatch.setenv("SWB200_STEP", shape)
    nx, ratio = size
    for kw in OPTIONS:
        S, Prog = setup(dict(kw, nx=nx, L_ratio=ratio))
        o = O.Oracle(S)
        o.set_state(Prog)
        o.run(3)
        for x, y, name in zip(run(S, Prog, 3)[0], o.get_state(), NAMES):
            assert_bitwise(x, y, f"{name} {kw}")


@pytest.mark.parametrize("rows", ["2", "5", "15", "16", "38", "47"])
@pytest.mark.parametrize("shape", ["0", "1", "2", "3", "4"])
def test_tile_heights_against_the_launches_per_stage(shape, rows, monkeypatch):
    for kw in OPTIONS[:6]:
        S, Prog = setup(dict(kw, nx=211, L_ratio=2))
        monkeypatch.setenv("SWB200_STEP", "-1")
        ref, rhs = run(S, Prog, 2)
        monkeypatch.setenv("SWB200_STEP", shape)
        monkeypatch.setenv("SWB200_STEP_ROWS", rows)
        got, rhs_got = run(S, Prog, 2)
        for x, y, name in zip(got, ref, NAMES):
            assert_bitwise(x, y, f"{name} {kw}")
        for x, y, name in zip(rhs_got, rhs, NAMES):
            assert_bitwise(x, y, f"right-hand side's {name} {kw}")


@pytest.mark.parametrize("shape", ["0", "1", "2", "3", "4"])
@pytest.mark.parametrize("storage", ["bf16", "f16"])
def test_16bit_storage_against_the_launches_per_stage(storage, shape, monkeypatch):
    """The stored halves and the tracer; α = 0.5 keeps the launches per stage
    (its ghost increments are rounded on their own)."""
    options = [kw for kw in OPTIONS if kw.get("T") is None] + [dict(bc="nonperiodic", α=0.0), dict(nstep_diff=2)]
    for kw in options:
        for nx, ratio in ((61, 3), (125, 2), (211, 2)):
            S, Prog = setup(dict(kw, nx=nx, L_ratio=ratio))
            got = []
            for step in ("-1", shape):
                monkeypatch.setenv("SWB200_STEP", step)
                with Model(S, storage=storage, storage_scale_uv=8.0) as m:
                    m.set_state(Prog)
                    assert m.run(3).code == 0
                    got.append(m.get_state())
            for x, y, name in zip(*got, NAMES):
                assert_bitwise(x, y, f"{name} {kw}")


@pytest.mark.parametrize("n", [150, 60])   # 16-step blocks, then 4; single steps, then 16, 8 and 4
@pytest.mark.parametrize("kw", [dict(nx=100), dict(nx=64, Uadv=0.25), dict(nx=64, time_scheme="SSPRK3"),
                                dict(nx=64, bc="nonperiodic", T=np.float64), dict(nx=600, L_ratio=3)])
def test_blocks_of_steps_equal_single_steps(kw, n, monkeypatch):
    """n steps in one call (blocks, single steps between the NaN checks)
    against the same steps one call each and without graphs."""
    S, Prog = setup(dict(kw, output_dt=0.5))
    whole = run(S, Prog, n)
    monkeypatch.setenv("SWB200_GRAPHS", "0")
    single = run(S, Prog, n)
    for a, b in zip(whole, single):
        for x, y, name in zip(a, b, NAMES):
            assert_bitwise(x, y, name)


def test_nan_stop_inside_a_block():
    """The NaN check's step and state (those before the failing step) do not
    depend on the steps having run in blocks."""
    S, Prog = setup(dict(nx=60, Ndays=2, tracer_advection=False))
    Prog.u[5, 7] = np.nan
    o = O.Oracle(S)
    o.set_state(Prog)
    so = o.run(S.grid.nt)
    with Model(S) as m:
        m.set_state(Prog)
        sg = m.run(S.grid.nt)
        assert sg.code == so.code == 3 and sg.nan_step == so.nan_step
        for x, y, name in zip(m.get_state(), o.get_state(), NAMES):
            assert_bitwise(x, y, name)
