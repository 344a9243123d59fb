"""The rollout of one opponent by lane pairs (csrc/pair_model.cuh) against the FP32 oracle on
identical perturbations and Philox noise: tiles that are empty, partial and full, one to eight
hypotheses (repeated ones among them), both control modes, every noise source on or off, and a
belief that has already committed. The tolerance is the one of the other rollout tests: host
and device round a few multiply-adds and exponentials differently, which moves the rare sample
that sits on a threshold."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import O, drb
from helpers import mppi_ctl

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


@pytest.mark.parametrize("noise", ["off", "opponent", "all"])
@pytest.mark.parametrize("nth,spl,K,certain", [(1, False, 1, False), (1, True, 257, False), (2, False, 63, False), (2, True, 65, False), (2, False, 640, True),
                                               (4, False, 97, False), (8, False, 47, False), (8, True, 33, False)])
def test_pair_rollout_matches_oracle(gpu, nth, spl, K, certain, noise):
    sc = S.circle_race(agent=1, seed=3, K=K, T=40, use_splines=spl, n_theta=nth, n_verif=64)
    st = sc.state
    for a in range(2):  # moving, a little off the centreline
        i = int(round(float(st.S[a]) / sc.grids.track_length * 512)) % 512
        t = sc.grids.t_grid[i]
        st.vel[2 * a], st.vel[2 * a + 1] = 3.0 * float(t[0]), 3.0 * float(t[1])
    if noise == "off":
        for th in range(nth):
            sc.env.opp_configs[th].action_noise[0] = 0.0
    if noise == "all":
        sc.env.action_noise_level, sc.env.pos_noise_level, sc.env.speed_noise_level = 0.2, 0.01, 0.05
    sc.mppi.final_opp_adv_weight = 20.0
    belief = sc.belief()
    if certain:
        belief[:] = (0.02, 0.98)
    rng = np.random.default_rng(5)
    ctl = mppi_ctl(sc, nominal=rng.normal(0, 1.0, (nth + 1, 40, 2)).astype(np.float32))
    ct = np.zeros((nth, K), np.float32)
    bu = np.zeros((nth, K), np.int32)
    bt = np.zeros((nth, K), np.int32)
    costs = np.zeros((nth + 1, K), np.float32)
    abi.check(abi.lib().dr_mppi_debug_rollout(ctl.handle, C.byref(sc.state), abi.fptr(belief), abi.fptr(ct), abi.iptr(bu), abi.iptr(bt), abi.fptr(costs)),
              "debug_rollout")
    B = O.spline_matrix(sc.mppi) if spl else None
    oct_, obu, obt = O.mppi_rollout(sc, belief, ctl.knots().copy(), O.mppi_noise(sc, 0), B, 0, prec=32)
    fin = np.isfinite(oct_)
    assert np.array_equal(fin, np.isfinite(ct))
    rel = np.abs(ct[fin] - oct_[fin]) / np.maximum(1.0, np.abs(oct_[fin]))
    assert np.mean(rel <= 1e-5) >= 0.97
    assert np.mean((bu == obu) & (bt == obt)) >= 0.97
    # the aggregation over hypotheses, from the rollout's own costs
    w = np.where(fin, belief[:, None], 0.0).astype(np.float64)
    mean = (w * np.where(fin, ct, 0.0)).sum(0) / w.sum(0)
    np.testing.assert_allclose(costs[0], mean, rtol=1e-5)
    assert np.array_equal(costs[1:][fin], ct[fin]) or np.allclose(costs[1:][fin], ct[fin], rtol=1e-6)


@pytest.mark.parametrize("M", [2, 3, 4, 5, 7, 8, 9])
def test_spline_sums_of_any_knot_count(gpu, M):
    """Knots are summed four at a time: counts that fill no, one and two groups, and remainders."""
    sc = S.circle_race(agent=1, seed=3, K=130, T=31, use_splines=True, n_theta=2, n_verif=64)
    sc.mppi = S.make_mppi(K=130, T=31, use_splines=True, M=M, n_verif_samples=64, verif_horizon=20)
    belief = sc.belief()
    ctl = mppi_ctl(sc, nominal=np.random.default_rng(M).normal(0, 1.0, (3, 31, 2)).astype(np.float32))
    ct, costs = np.zeros((2, 130), np.float32), np.zeros((3, 130), np.float32)
    bu, bt = np.zeros((2, 130), np.int32), np.zeros((2, 130), np.int32)
    abi.check(abi.lib().dr_mppi_debug_rollout(ctl.handle, C.byref(sc.state), abi.fptr(belief), abi.fptr(ct), abi.iptr(bu), abi.iptr(bt), abi.fptr(costs)),
              "debug_rollout")
    oct_, obu, obt = O.mppi_rollout(sc, belief, ctl.knots().copy(), O.mppi_noise(sc, 0), O.spline_matrix(sc.mppi), 0, prec=32)
    fin = np.isfinite(oct_)
    assert np.array_equal(fin, np.isfinite(ct))
    assert np.mean(np.abs(ct[fin] - oct_[fin]) <= 1e-5 * np.maximum(1.0, np.abs(oct_[fin]))) >= 0.97
    assert np.mean((bu == obu) & (bt == obt)) >= 0.97
