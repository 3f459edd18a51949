"""The whole-step kernel's SSP and Sadourny branches and its batches, which
tests/test_gpu_step.py and tests/test_ensemble.py reach in a shape or two:

* SSPRK2 with 2 to 4 sub-stages, SSPRK3, 4SSPRK3 and Sadourny's advection, in
  every tile shape, over tile edges and several tile columns that a seam or a
  wall crosses, against the CPU oracle and the launches per stage (the input of
  the last right-hand side too).
* Batches in every tile shape, and of more members than one launch takes.
* A run in blocks of steps against the same steps one call each.

All bit for bit: every value is formed by the reference's expressions.
"""
import numpy as np
import pytest

import oracle as O
from conftest import assert_bitwise
from swb200 import Model
from swb200.ensemble import COLUMNS, Member, member_setup, run_batched
from swb200.initial_conditions import remove_halo
from test_gpu_step import NAMES, run, setup

pytestmark = pytest.mark.gpu

SCHEMES = [
    dict(time_scheme="SSPRK2", RKs=2, cfl=0.5, topography="flat", diffusion="Smagorinsky"),
    dict(time_scheme="SSPRK2", RKs=3, bc="nonperiodic", α=0.5, topography="seamount", wind_forcing_x="double_gyre"),
    dict(time_scheme="SSPRK2", RKs=4, T=np.float64, bottom_drag="linear", nstep_diff=2),
    dict(time_scheme="SSPRK2", RKs=3, T=np.float64, adv_scheme="Sadourny", bc="nonperiodic", α=2.0, topography="flat"),
    dict(time_scheme="SSPRK3", RKn=2, diffusion="Smagorinsky"),
    dict(time_scheme="SSPRK3", RKn=2, T=np.float64, bc="nonperiodic", α=1.0, topography="seamount"),
    dict(time_scheme="SSPRK3", RKn=2, adv_scheme="Sadourny", topography="flat", bottom_drag="none"),
    dict(time_scheme="4SSPRK3", topography="flat", diffusion="Smagorinsky"),
    dict(time_scheme="4SSPRK3", bc="nonperiodic", α=0.0, adv_scheme="Sadourny", topography="seamount"),
    dict(time_scheme="4SSPRK3", T=np.float64, diffusion="Smagorinsky"),
    dict(adv_scheme="Sadourny", diffusion="Smagorinsky"),
    dict(adv_scheme="Sadourny", bc="nonperiodic", α=0.5, topography="flat"),
    dict(adv_scheme="Sadourny", T=np.float64, topography="seamount", RKo=3, cfl=0.6),
]


def launches(S, Prog, n):
    with Model(S) as m:
        m.set_state(Prog)
        before = m.kernel_launches
        assert m.run(n).code == 0
        return m.kernel_launches - before


@pytest.mark.parametrize("shape", ["0", "1", "2", "3", "4"])
@pytest.mark.parametrize("size", [(4, 1), (28, 1), (57, 1), (61, 3), (121, 2), (125, 5)])
def test_schemes_against_the_oracle(size, shape, monkeypatch):
    monkeypatch.setenv("SWB200_STEP", shape)
    nx, ratio = size
    for kw in SCHEMES:
        S, Prog = setup(dict(kw, nx=nx, L_ratio=ratio))
        o = O.Oracle(S)
        o.set_state(Prog)
        o.run(3)
        for x, y, name in zip(run(S, Prog, 3)[0], o.get_state(), NAMES):
            assert_bitwise(x, y, f"{name} {kw}")


@pytest.mark.parametrize("rows", ["2", "5", "12", "43", "0"])   # 0: the plan's own
@pytest.mark.parametrize("shape", ["0", "1", "2", "3", "4"])
def test_schemes_against_the_launches_per_stage(shape, rows, monkeypatch):
    for kw in SCHEMES:
        for nx, ratio in ((211, 2), (150, 1)):
            S, Prog = setup(dict(kw, nx=nx, L_ratio=ratio))
            monkeypatch.setenv("SWB200_STEP", "-1")
            ref, rhs = run(S, Prog, 2)
            monkeypatch.setenv("SWB200_STEP", shape)
            monkeypatch.setenv("SWB200_STEP_ROWS", rows)
            got, rhs_got = run(S, Prog, 2)
            for x, y, name in zip(got, ref, NAMES):
                assert_bitwise(x, y, f"{name} {kw}")
            for x, y, name in zip(rhs_got, rhs, NAMES):
                assert_bitwise(x, y, f"right-hand side's {name} {kw}")


@pytest.mark.parametrize("kw", SCHEMES)
def test_schemes_take_the_whole_step_kernel(kw, monkeypatch):
    """Two launches a step, the step and its tracer, in the widest tiles (which
    every scheme and size has)."""
    monkeypatch.setenv("SWB200_STEP", "4")
    S, Prog = setup(dict(kw, nx=211))
    assert launches(S, Prog, 4) == 8


def batch_equals_lone_runs(members, monkeypatch):
    info = {}
    table, states = run_batched(members, return_states=True, info=info)
    monkeypatch.setenv("SWB200_STEP", "-1")
    for m in members:
        P, S, Prog = member_setup(m)
        with Model(S) as model:
            model.set_state(Prog)
            st = model.run(S.grid.nt)
            ref = remove_halo(*model.get_state(), S)
        assert table[m.index][COLUMNS.index("steps")] == st.steps_done == S.grid.nt
        for x, y, name in zip(states[m.index], ref, NAMES):
            assert_bitwise(x, y, f"member {m.index}: {name}")
    return info["launches"]


@pytest.mark.parametrize("rows", ["0", "2", "7"])
@pytest.mark.parametrize("shape", ["0", "1", "2", "3", "4"])
def test_batches_in_every_tile_shape(shape, rows, monkeypatch):
    monkeypatch.setenv("SWB200_STEP", shape)
    monkeypatch.setenv("SWB200_STEP_ROWS", rows)
    sizes = [(24, 1), (57, 1), (125, 3), (211, 2), (150, 1), (40, 2)]
    members = [Member(k, dict(nx=nx, L_ratio=ratio, Ndays=0.05, Uadv=1000, bc=("periodic", "nonperiodic")[k % 2],
                              α=0.5, diffusion="Smagorinsky", topography=("ridge", "flat", "seamount")[k % 3]), seed=k)
               for k, (nx, ratio) in enumerate(sizes)]
    batch_equals_lone_runs(members, monkeypatch)


def test_a_batch_of_more_members_than_a_launch_takes(monkeypatch):
    """130 members of one group: launches of 64, 64 and 2."""
    members = [Member(k, dict(nx=20 + k % 23, Ndays=0.1, Fx0=0.05 + 0.001 * k, tracer_advection=False), seed=k)
               for k in range(130)]
    n = batch_equals_lone_runs(members, monkeypatch)
    steps = max(member_setup(m)[1].grid.nt for m in members)
    assert n >= 3 * steps


@pytest.mark.parametrize("kw", [dict(nx=100), dict(nx=64, time_scheme="SSPRK3"), dict(nx=64, bc="nonperiodic", T=np.float64)])
def test_blocks_of_steps_equal_one_call_per_step(kw):
    n = 150
    S, Prog = setup(dict(kw, output_dt=0.5))
    whole = run(S, Prog, n)
    with Model(S) as m:
        m.set_state(Prog)
        for _ in range(n):
            assert m.run(1).code == 0
        single = m.get_state(), m.get_rhs_input()
    for a, b in zip(whole, single):
        for x, y, name in zip(a, b, NAMES):
            assert_bitwise(x, y, name)
