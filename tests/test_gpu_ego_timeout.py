"""The ego tables' bounded staging wait (mppi_ego_table) under dr_mppi_debug_stage_timeout: its CTAs
count their timeouts like the rollout's and the verification's, and a clearance block that was not
filled lets no verification tile end early (every tile still counts its own)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import drb

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


@pytest.mark.parametrize("nth,horizon", [(1, 7), (2, 40), (8, 33)])
def test_ego_table_timeouts_are_counted(gpu, nth, horizon):
    counts = []
    for table in (True, False):
        sc = S.circle_race(agent=0, seed=0, K=100, T=48, n_theta=nth, n_verif=1100)
        sc.mppi.verif_horizon = horizon
        ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5)
        ctl.set_ego_table(table)
        step = lambda: abi.lib().dr_mppi_step(ctl.handle, C.byref(sc.state), abi.fptr(sc.belief()), abi.fptr(out), C.byref(info))
        out, info = np.zeros(2, np.float32), abi.dr_mppi_info()
        assert step() == abi.DR_OK and info.verif_timeouts == 0
        abi.check(abi.lib().dr_mppi_debug_stage_timeout(ctl.handle, 1, 256), "stage_timeout on")
        assert step() == abi.DR_ERR_TIMEOUT
        counts.append(info.verif_timeouts)
        abi.check(abi.lib().dr_mppi_debug_stage_timeout(ctl.handle, 0, 0), "stage_timeout off")
        assert step() == abi.DR_OK and info.verif_timeouts == 0
    rows = 1 + nth * horizon  # of a plan, eight to a CTA; two plans a step
    assert counts[0] - counts[1] == 2 * ((rows + 7) // 8)
