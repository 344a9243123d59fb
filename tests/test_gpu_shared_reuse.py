"""CTAs that stage again over shared memory they have used: the ego tables of both plans in one
launch (verification beside the rollout off), and persistent launches whose CTAs go from one
controller's tiles to another's with other horizons, so that one tile's histogram and clearance
block lie where the next one's plan is staged. Failure counts, plans and actions equal, without
tolerance, those of one CTA per tile without the tables."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import drb

pytestmark = pytest.mark.gpu
S = drb.scenarios

# (T, verification horizon, samples verified, metres ahead of the ego), near enough to collide or not
RACES = [(24, 7, 900, 1.3), (64, 40, 1500, 2.4), (40, 40, 600, 1.6), (96, 81, 2100, 1.4), (33, 16, 1100, 9.0), (48, 33, 513, -1.5)]


def _run(shape):
    scs, ctls = [], []
    for i, (T, H, V, gap) in enumerate(RACES):
        sc = S.circle_race(agent=i, seed=i, K=300 + 64 * i, T=T, n_verif=V)
        sc.mppi.verif_horizon = H
        st, per = sc.state, sc.grids.track_length / 512
        for a, j in enumerate((100, 100 + int(round(gap / per)))):
            t = sc.grids.t_grid[j]
            st.pos[2 * a], st.pos[2 * a + 1] = float(sc.grids.p_grid[j, 0]), float(sc.grids.p_grid[j, 1])
            st.vel[2 * a], st.vel[2 * a + 1] = (4.0 - a) * float(t[0]), (4.0 - a) * float(t[1])
            st.S[a], st.lat_dist[a] = float(np.float32(j * per)), 0.0
        plan = np.random.default_rng(i).normal(0, 2.0, (sc.n_theta + 1, T, 2)).astype(np.float32)
        ctl = drb.controllers.MPPIController(sc.env, sc.mppi, 5 + i, nominal=plan)
        ctl.set_ego_table(shape is not None)
        scs.append(sc)
        ctls.append(ctl)
    batch = drb.controllers.MPPIBatch(ctls)
    if shape is not None:
        overlap, roll, verify, side = shape
        batch.set_overlap(overlap)
        batch.set_persistent(roll, verify)
        if side:
            batch.set_side_verify(side)
    out = []
    for _ in range(3):
        out.append(batch.step([s.state for s in scs], np.stack([s.belief() for s in scs])).copy())
        for c in ctls:
            c._pull()
            out += [c.failCountNew.copy(), c.failCountOld.copy(), c.h_nominal.copy()]
    batch.close()
    return out


@pytest.fixture(scope="module")
def plain(gpu):
    out = _run(None)
    assert sum(int(a.sum()) for a in out if a.dtype == np.uint32) > 0  # samples do collide
    return out


@pytest.mark.parametrize("shape", [(False, 0, 0, 0), (False, 1, 1, 0), (True, 1, 1, 1), (True, 2, 2, 0)])
def test_reused_shared_memory_changes_nothing(plain, shape):
    for a, b in zip(plain, _run(shape)):
        assert np.array_equal(a, b)
