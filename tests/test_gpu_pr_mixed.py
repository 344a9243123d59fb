"""Controllers of different sampled hypotheses and horizons in one PR-MPPI batch: the widest sizes the
candidates' block and the longest the plans, and each controller's step is, without tolerance, the one it
takes alone."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import drb

pytestmark = pytest.mark.gpu
S = drb.scenarios


@pytest.mark.parametrize("sizes", [[(1, 12, 70), (32, 40, 9), (8, 25, 300)], [(9, 60, 49), (3, 7, 500)], [(17, 33, 20), (16, 64, 20), (2, 31, 161), (5, 48, 1)]])
@pytest.mark.parametrize("noise", [0.0, 0.1])
def test_mixed_batch_equals_single_controllers(gpu, sizes, noise):
    scs = [S.robust_race(agent=i, seed=4, K=K, T=T, P=P, n_theta=4) for i, (P, T, K) in enumerate(sizes)]
    for sc in scs:
        sc.env.action_noise_level = noise  # with it, the kernels that share no ego
    make = lambda: [drb.controllers.PRMPPIController(s.env, s.prmppi, 7 + i) for i, s in enumerate(scs)]
    alone, together = make(), make()
    one = [drb.controllers.PRMPPIBatch([c]) for c in alone]
    batch = drb.controllers.PRMPPIBatch(together)
    for _ in range(3):
        got = batch.step([s.state for s in scs], np.stack([s.belief() for s in scs]))
        for i, s in enumerate(scs):
            assert np.array_equal(one[i].step([s.state], s.belief()[None, :])[0], got[i])
            assert all(np.array_equal(a, b) for a, b in zip(alone[i].nominals(), together[i].nominals()))
            a, b = one[i].infos[0], batch.infos[i]
            for f in ("cand_cost", "min_costs", "nu", "inv_temperature"):
                assert list(getattr(a, f)) == list(getattr(b, f)), f
            assert a.use_nom_plan == b.use_nom_plan and a.reset_nom == b.reset_nom
    for b in [batch, *one]:
        b.close()
