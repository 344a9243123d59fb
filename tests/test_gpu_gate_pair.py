"""The gate race's rollout by lane pairs (csrc/gate_pair.cuh) against the FP32 oracle, as
tests/test_gpu_gate.py compares it: partial and full tiles, either agent as the ego, a tracked
ego (each lane projects its own agent) and an untracked one (a raceline a lane), noise off and
on. The tolerance is the one of the other rollout tests."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import helpers as H
from conftest import O, drb

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


@pytest.mark.parametrize("spl,K,me,tracked,noise", [(False, 1, 0, False, True), (False, 63, 1, False, True), (False, 64, 0, True, False),
                                                    (True, 65, 0, False, True), (True, 130, 1, True, False), (False, 700, 0, False, False)])
def test_gate_pair_rollout_matches_oracle(gpu, spl, K, me, tracked, noise):
    sc = H.small_gate(spl, K=K, T=40, seed=9, noise=noise)
    sc.env.i_mppi = me
    u = [0.22, 0.25] if me == 0 else [0.25, 0.22]
    sc.state = S.gate_state(sc.track, u, me, [0, 0], speed=2.5)
    if tracked:  # the ego's arc lengths on both racelines
        for r in range(abi.DR_GATE_RACELINES):
            sc.state.S[me * abi.DR_GATE_RACELINES + r] = float(np.float32(u[me]))
    sc.mppi.final_opp_adv_weight = 20.0
    rng = np.random.default_rng(4)
    ctl = H.mppi_ctl(sc, nominal=H.random_nominal(sc, rng))
    belief = sc.belief()
    ct, bu, bt = np.zeros((2, K), np.float32), np.zeros((2, K), np.int32), np.zeros((2, K), np.int32)
    costs = np.zeros((3, K), np.float32)
    abi.check(abi.lib().dr_gate_mppi_debug_rollout(ctl.handle, C.byref(sc.state), abi.fptr(belief), abi.fptr(ct), abi.iptr(bu), abi.iptr(bt),
                                                   abi.fptr(costs)), "gate debug_rollout")
    B = O.spline_matrix(sc.mppi) if spl else None
    oct_, obu, obt = O.mppi_rollout(sc, belief, ctl.knots().copy(), O.mppi_noise(sc, 0), B, 0, prec=32)
    rel = np.abs(ct - oct_) / np.maximum(1.0, np.abs(oct_))
    assert np.mean(rel <= 1e-5) >= 0.97
    assert np.mean((bu == obu) & (bt == obt)) >= 0.97
