"""The fast verification stops stepping samples that can no longer collide (clearOfEgo in
csrc/clear.cuh, from the ego tables of csrc/instance.cuh's clearance block). That changes
no result: per-sample failure times and counts equal, without tolerance, those of the
verification that moves the ego in every sample and steps all of them to the end, over horizons
around the table's step groups and over states from one in which nearly all samples collide to
one in which none can."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import drb

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


def _case(nth, H, gap, lat, seed, V=1100):
    T = max(H, 24)
    sc = S.circle_race(agent=1, seed=seed, K=64, T=T, n_theta=nth, n_verif=V)
    sc.mppi.verif_horizon = H
    rng = np.random.default_rng(seed)
    per = sc.grids.track_length / 512
    st = sc.state
    for a, i in enumerate((100, 100 + int(round(gap / per)))):
        t = sc.grids.t_grid[i]
        off = lat if a else -lat
        st.pos[2 * a] = float(sc.grids.p_grid[i, 0] - off * t[1])
        st.pos[2 * a + 1] = float(sc.grids.p_grid[i, 1] + off * t[0])
        v = 4.5 - 2.0 * a
        st.vel[2 * a], st.vel[2 * a + 1] = v * float(t[0]), v * float(t[1])
        st.S[a] = float(np.float32(i * per))
        st.lat_dist[a] = off
    plan = rng.normal(0, 3.0, (nth + 1, T, 2)).astype(np.float32)
    return sc, plan


def _verify(sc, plan, table):
    ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5)
    ctl.set_ego_table(table)
    V, T = sc.mppi.n_verif_samples, sc.mppi.n_timesteps
    fc, ft = np.zeros(T, np.uint32), np.zeros(V, np.int32)
    abi.check(abi.lib().dr_mppi_debug_verify(ctl.handle, C.byref(sc.state), abi.fptr(sc.belief()), abi.fptr(plan), 0, abi.uptr(fc), abi.iptr(ft), None),
              "debug_verify")
    return fc, ft


@pytest.mark.parametrize("nth,H", [(1, 1), (2, 15), (2, 16), (2, 17), (2, 40), (4, 41), (8, 33), (2, 81), (2, 200)])
@pytest.mark.parametrize("gap,lat", [(1.3, 0.0), (2.4, 0.2), (4.0, 0.6), (-3.0, 0.3), (9.0, 0.0)])
def test_clearance_changes_no_failure(gpu, nth, H, gap, lat):
    sc, plan = _case(nth, H, gap, lat, seed=nth * 100 + H)
    for a, b in zip(_verify(sc, plan, True), _verify(sc, plan, False)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("H", [5, 33, 64])
@pytest.mark.parametrize("limit", [0.6, 0.99, 1.0])
@pytest.mark.parametrize("gap", [-1.2, -1.6, -2.2])
def test_clearance_of_followers_near_their_limit(gpu, H, limit, gap):
    """An opponent behind the ego whose way the speed limit bounds before its acceleration does
    (clearAfter), while the ego coasts or brakes."""
    for brake in (0.0, 4.0):
        sc, plan = _case(2, H, gap, 0.1, seed=H)
        st = sc.state
        v = limit * float(sc.env.max_speed[1])
        n = float(np.hypot(st.vel[2], st.vel[3]))
        st.vel[2], st.vel[3] = st.vel[2] * v / n * 0.9999, st.vel[3] * v / n * 0.9999
        e = np.array([st.vel[0], st.vel[1]])
        plan[:] = -brake * e / np.hypot(*e)
        for a, b in zip(_verify(sc, plan, True), _verify(sc, plan, False)):
            assert np.array_equal(a, b)


def test_clear_tiles_of_whole_steps(gpu):
    """Whole control steps, where a tile clear from the start is skipped: the same failure
    counts, plans and actions with the tables and without, plain and persistent launches."""
    for gap in (1.5, 6.0, 12.0):
        out = []
        for table in (True, False):
            sc, plan = _case(2, 40, gap, 0.3, seed=3)
            ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5, nominal=plan)
            ctl.set_ego_table(table)
            batch = drb.controllers.MPPIBatch([ctl])
            r = []
            for k in range(4):
                if k == 2 and table:
                    batch.set_persistent(1, 1)
                r.append(batch.step([sc.state], sc.belief()[None, :]).copy())
                ctl._pull()
                r += [ctl.failCountNew.copy(), ctl.failCountOld.copy(), ctl.h_nominal]
            out.append(r)
        for a, b in zip(*out):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("me", [0, 1])
@pytest.mark.parametrize("Hv", [7, 8, 9, 40, 41, 60])
@pytest.mark.parametrize("gap,toward", [(0.016, True), (0.02, True), (0.02, False), (0.035, True), (0.05, False), (0.2, False)])
def test_gate_clearance_changes_no_failure(gpu, me, Hv, gap, toward):
    """The same on the gate race (gate_clear): an obstacle beside the track, either agent as the
    ego, horizons around the steps that a lane group takes."""
    import helpers as H

    sc = H.small_gate(False, K=64, T=60, n_verif=1100, seed=3)
    sc.mppi.verif_horizon = Hv
    sc.env.i_mppi = me
    u = [0.31, 0.31 + gap] if me == 0 else [0.31 + gap, 0.31]
    sc.state = S.gate_state(sc.track, u, me, [0, 0], speed=3.0)
    sc.env.n_round_obstacles = 1
    sc.env.round_obs_centers[0], sc.env.round_obs_centers[1], sc.env.round_obs_radius[0] = 2.0, 7.0, 0.4
    rng = np.random.default_rng(Hv)
    plan = H.toward_opponent_plan(sc) if toward else rng.normal(0, 3.0, (3, 60, 2)).astype(np.float32)
    out = []
    for table in (True, False):
        ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5)
        ctl.set_ego_table(table)
        fc, ft = np.zeros(60, np.uint32), np.zeros(1100, np.int32)
        abi.check(abi.lib().dr_gate_mppi_debug_verify(ctl.handle, C.byref(sc.state), abi.fptr(sc.belief()), abi.fptr(plan), 1, abi.uptr(fc),
                                                      abi.iptr(ft), None), "gate debug_verify")
        out.append((fc, ft))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
