"""The PR-MPPI kernels that step one ego per sample (egos that draw no noise; pr_rollout_shared
and pr_candidates_shared in csrc/prmppi_kernels.cu) give, without tolerance, what the general
kernels give. A batch takes the general kernels when any of its controllers' egos draws noise, so
the same controller is stepped once alone and once beside such a one: actions, plans, minima,
weights and candidate costs are equal step after step. Sampled hypotheses from one to the most,
samples that fill a tile in part, exactly and not at all, opponents with and without noise."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import drb

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


def _scenario(nth, P, K, noise, seed):
    sc = S.robust_race(agent=2, seed=4, K=K, T=40, P=P, n_theta=nth)
    if not noise:
        for th in range(nth):
            sc.env.opp_configs[th].action_noise[0] = 0.0
    st = sc.state
    for a in range(2):
        i = int(round(float(st.S[a]) / sc.grids.track_length * 512)) % 512
        t = sc.grids.t_grid[i]
        st.vel[2 * a], st.vel[2 * a + 1] = 3.5 * float(t[0]), 3.5 * float(t[1])
    sc.prmppi.final_opp_adv_weight = 15.0
    sc.seed = seed
    return sc


@pytest.mark.parametrize("noise", [True, False])
@pytest.mark.parametrize("nth,P,K", [(1, 1, 255), (2, 2, 161), (2, 3, 1), (4, 7, 64), (2, 9, 48), (2, 9, 49), (8, 10, 45), (8, 32, 30)])
def test_shared_ego_kernels_equal_the_general_ones(gpu, nth, P, K, noise):
    out = []
    for beside in (False, True):
        scs = [_scenario(nth, P, K, noise, 11)]
        if beside:
            other = _scenario(nth, 5, 33, noise, 12)
            other.env.action_noise_level = 0.1
            scs.append(other)
        ctls = [drb.controllers.PRMPPIController(s.env, s.prmppi, s.seed) for s in scs]
        batch = drb.controllers.PRMPPIBatch(ctls)
        beliefs = np.stack([s.belief() for s in scs])
        r = []
        for _ in range(3):
            r.append(batch.step([s.state for s in scs], beliefs)[0])
            r += list(ctls[0].nominals())
            i = batch.infos[0]
            r.append(np.array([i.use_nom_plan, i.reset_nom, *i.cand_cost, *i.min_costs, *i.nu, *i.inv_temperature, i.nonfinite_costs]))
        out.append(r)
        batch.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
