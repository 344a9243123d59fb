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


@pytest.mark.parametrize("noise", [True, False])
@pytest.mark.parametrize("me,P,K,tracked", [(0, 1, 70, False), (1, 3, 43, False), (0, 8, 29, True), (1, 9, 200, True), (0, 32, 7, False)])
def test_gate_shared_ego_kernels_equal_the_general_ones(gpu, me, P, K, tracked, noise):
    """The same on the gate race. An action noise of 1e-30 sends the ego's controller to the general
    kernels and moves nothing (it is far below the last bit of any action)."""
    import helpers as H

    out = []
    for level in (0.0, 1e-30):
        sc = H.small_gate(False, K=K, T=40, seed=9, noise=noise)
        sc.env.i_mppi = me
        u = [0.22, 0.24] if me == 0 else [0.24, 0.22]
        sc.state = S.gate_state(sc.track, u, me, [0, 0], speed=2.5)
        if tracked:
            for r in range(abi.DR_GATE_RACELINES):
                sc.state.S[me * abi.DR_GATE_RACELINES + r] = float(np.float32(u[me]))
        for th in range(2):
            sc.env.opp_pid[th].repulsion_factor = 0.3 * th
        sc.env.action_noise_level = level
        sc.prmppi = S.make_prmppi(K=K, T=40, P=P)
        sc.prmppi.final_opp_adv_weight = 15.0
        rng = np.random.default_rng(6)
        ctl = drb.controllers.PRMPPIController(sc.env, sc.prmppi, 5, nominal=rng.normal(0, 2.0, (40, 2)).astype(np.float32))
        ctl.engine = object()
        r = []
        for _ in range(3):
            r.append(ctl.getControl(sc.state))
            r += list(ctl.nominals())
            i = ctl.info
            r.append(np.array([i.use_nom_plan, i.reset_nom, *i.cand_cost, *i.min_costs, *i.nu, *i.inv_temperature, i.nonfinite_costs]))
        out.append(r)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
