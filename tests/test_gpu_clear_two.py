"""The clearance tests with two opponents, each with a witness and limits of its own: failure times,
counts and actions equal, without tolerance, those of the verification that steps every sample to the
end, from a state with failures to one where nothing can meet."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import drb
from test_gpu_grad import _multi_scenario

pytestmark = pytest.mark.gpu
abi = drb.abi


@pytest.mark.parametrize("horizon", [1, 17, 40])
@pytest.mark.parametrize("at,speeds", [((26, 42, 64), (3.0, 1.0, 1.0)), ((26, 44, 8), (1.0, 1.5, 2.0)), ((26, 70, 130), (3.0, 2.0, 1.0)), ((26, 190, 340), (1.0, 2.0, 2.0))])
def test_two_opponents(gpu, horizon, at, speeds):
    sc = _multi_scenario(2, 2, False)
    sc.mppi.n_verif_samples, sc.mppi.verif_horizon = 1100, horizon
    st, per = sc.state, sc.grids.track_length / 512
    for a, (i, v) in enumerate(zip(at, speeds)):
        t = sc.grids.t_grid[i]
        st.pos[2 * a], st.pos[2 * a + 1] = float(sc.grids.p_grid[i, 0]), float(sc.grids.p_grid[i, 1])
        st.vel[2 * a], st.vel[2 * a + 1] = v * float(t[0]), v * float(t[1])
        st.S[a], st.lat_dist[a] = float(np.float32(i * per)), 0.0
    plan = np.random.default_rng(horizon).normal(0, 0.7, (3, 40, 2)).astype(np.float32)
    out = []
    for table in (True, False):
        ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5)
        ctl.set_ego_table(table)
        for p in (0, 1):
            fc, ft = np.zeros(40, np.uint32), np.zeros(1100, np.int32)
            abi.check(abi.lib().dr_mppi_debug_verify(ctl.handle, C.byref(st), abi.fptr(sc.belief()), abi.fptr(plan), p, abi.uptr(fc), abi.iptr(ft), None), "verify")
            out.append((fc, ft))
        ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5, nominal=plan)
        ctl.set_ego_table(table)
        ctl.engine = object()
        out.append((ctl.getControl(st).copy(), ctl.failCountNew.copy(), ctl.failCountOld.copy()))
    for a, b in zip(out[:3], out[3:]):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
    if at == (26, 42, 64) and horizon > 1:
        assert out[0][0].sum() > 0
