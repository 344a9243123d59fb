"""The PR-MPPI rollout's tiles are cut for the kernel that takes them: the general ones (two opponents,
noise on the ego, several hypothesis slots a thread) have 448 (gate race: 512) slots a CTA and launch no
more waves of CTAs than full tiles need, and a batch whose slot count changes gets the table of the
kernel that its rollouts then take, with the same results."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import helpers as H
from conftest import drb
from test_gpu_grad import _multi_scenario

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


def _tiles(batch) -> int:
    n = C.c_int()
    abi.check(abi.lib().dr_prmppi_batch_debug_rollout_tiles(batch._b, C.byref(n)), "rollout_tiles")
    return n.value


def _scenario(kind, P, K):
    if kind == "gate noise":
        sc = H.small_gate(False, K=K, T=30, seed=3)
        sc.env.action_noise_level = 0.1
    elif kind == "two opponents":
        sc = _multi_scenario(2, 2, True)
    else:
        sc = S.robust_race(agent=0, seed=1, K=K, T=30, P=P, n_theta=2)
        if kind == "noise":
            sc.env.speed_noise_level = 0.05
    sc.prmppi = S.make_prmppi(K=K, T=30, P=P)
    return sc


def _waves(tiles: int, opponents: int) -> int:
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return -(-tiles // (2 * sms if opponents == 1 else sms))


@pytest.mark.parametrize("kind,slots", [("noise", 448), ("two opponents", 448), ("gate noise", 512)])
@pytest.mark.parametrize("P,K", [(1, 60000), (2, 32768), (3, 149), (3, 20000), (8, 2048), (9, 50), (32, 4500), (32, 15)])
def test_general_rollouts_take_no_more_waves_than_full_tiles(gpu, kind, slots, P, K):
    sc = _scenario(kind, P, K)
    batch = drb.controllers.PRMPPIBatch([drb.controllers.PRMPPIController(sc.env, sc.prmppi, 3)])
    full, n = 2 * -(-K // (slots // P)), sc.env.n_opp if kind != "gate noise" else 1
    assert full <= _tiles(batch) and _waves(_tiles(batch), n) == _waves(full, n)
    batch.close()


@pytest.mark.parametrize("agents,K", [(1, 300), (4, 2048), (3, 5500)])
def test_tiles_follow_the_slots(gpu, agents, K):
    scs = [S.robust_race(agent=i, seed=2, K=K, T=30, P=8, n_theta=2) for i in range(agents)]
    make = lambda: drb.controllers.PRMPPIBatch([drb.controllers.PRMPPIController(s.env, s.prmppi, 3 + i) for i, s in enumerate(scs)])
    plain, changed = make(), make()
    shared = _tiles(plain)
    for slots in (1, 2, 4, 1):
        changed.set_rollout_slots(slots)
        full = agents * 2 * -(-K // 56)
        assert _tiles(changed) == shared if slots == 1 else _waves(_tiles(changed), 1) == _waves(full, 1)
        for _ in range(2):  # an eager step and a replayed one
            a, b = [x.step([s.state for s in scs], np.stack([s.belief() for s in scs])) for x in (plain, changed)]
            assert np.array_equal(a, b)
            for c, d in zip(plain.ctls, changed.ctls):
                assert all(np.array_equal(u, v) for u, v in zip(c.nominals(), d.nominals()))
    plain.close()
    changed.close()
