"""The clearance tests in whole control steps of the gate race, where tiles clear from the start are
skipped: failure counts, plans and actions equal, without tolerance, those of the verification that
steps every sample to the end. The near states have failures, and in the far one the tables do end
whole tiles: no copy of theirs is waited for."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import helpers as H
from conftest import drb

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


def _gate(me, gap, toward):
    sc = H.small_gate(False, K=64, T=60, n_verif=1100, seed=3)
    sc.mppi.verif_horizon = 40
    sc.env.i_mppi = me
    sc.state = S.gate_state(sc.track, [0.31, 0.31 + gap] if me == 0 else [0.31 + gap, 0.31], me, [0, 0], speed=3.0)
    plan = H.toward_opponent_plan(sc) if toward else np.random.default_rng(2).normal(0, 1.0, (3, 60, 2)).astype(np.float32)
    return sc, plan


@pytest.mark.parametrize("me", [0, 1])
@pytest.mark.parametrize("gap,toward", [(0.016, True), (0.03, True), (0.05, False), (0.09, False)])
def test_gate_steps(gpu, me, gap, toward):
    sc, plan = _gate(me, gap, toward)
    out, failures = [], 0
    for table in (True, False):
        ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5, nominal=plan)
        ctl.set_ego_table(table)
        ctl.engine = object()
        r = []
        for _ in range(3):  # an eager step and replayed ones
            r += [ctl.getControl(sc.state).copy(), ctl.failCountNew.copy(), ctl.failCountOld.copy(), ctl.h_nominal.copy()]
            failures += int(r[-3].sum()) + int(r[-2].sum())
        out.append(r)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    if toward and gap < 0.02 and me == 0:  # (agent 1 is the slower one and does not catch up)
        assert failures > 0


@pytest.mark.parametrize("me", [0, 1])
@pytest.mark.parametrize("gap,ends", [(0.016, False), (0.45, True)])
def test_gate_tiles_that_are_clear_end_at_once(gpu, me, gap, ends):
    counts = []
    for table in (True, False):
        sc, plan = _gate(me, gap, not ends)
        ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5, nominal=plan)
        ctl.set_ego_table(table)
        out, info = np.zeros(2, np.float32), abi.dr_mppi_info()
        abi.check(abi.lib().dr_mppi_debug_stage_timeout(ctl.handle, 1, 128), "stage_timeout on")
        assert abi.lib().dr_gate_mppi_step(ctl.handle, C.byref(sc.state), abi.fptr(sc.belief()), abi.fptr(out), C.byref(info)) == abi.DR_ERR_TIMEOUT
        counts.append(info.verif_timeouts)
    tiles = 2 * -(-1100 // 512)  # both plans' verification
    assert counts[1] - counts[0] == (tiles if ends else 0)
