"""The update and the PR-MPPI averages with their lanes split over a cluster of CTAs
(mppi_update, pr_weighted): the sums are defined by the reference's order (256 strided lanes,
each added in sample order, then a tree), so however many CTAs share the lanes the result is the
same bit for bit. A batch with enough controllers takes one CTA per block, a single controller of
the same samples up to eight: both give the same plans, minima and weights. Samples around the
numbers where the split changes and that fill no lane evenly."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import drb

pytestmark = pytest.mark.gpu
S = drb.scenarios


def _mppi(K, spl, seed):
    sc = S.circle_race(agent=1, seed=seed, K=K, T=24, use_splines=spl, n_theta=2, n_verif=256)
    if spl:
        sc.mppi = S.make_mppi(K=K, T=24, use_splines=True, M=5, inv_temperature=1.0, sampling_noise=1.0, n_verif_samples=256, verif_horizon=20)
    return sc


@pytest.mark.parametrize("spl", [True, False])
@pytest.mark.parametrize("K", [1, 255, 4096, 4097, 8191, 16640, 33000])
def test_update_is_the_same_for_every_split(gpu, K, spl):
    scs = [_mppi(K, spl, 3)] + [_mppi(300 + i, spl, 20 + i) for i in range(24)]
    out = []
    for n in (1, len(scs)):
        ctls = [drb.controllers.MPPIController(s.env, s.mppi, 7 + i) for i, s in enumerate(scs[:n])]
        b = drb.controllers.MPPIBatch(ctls)
        r = []
        for _ in range(2):
            r.append(b.step([s.state for s in scs[:n]], np.stack([s.belief() for s in scs[:n]]))[0])
            r += [ctls[0].knots(), ctls[0].h_nominal, np.array([b.infos[0].min_cost, b.infos[0].nu, b.infos[0].inv_temperature])]
        out.append(r)
        b.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("K", [1, 255, 2048, 2049, 8191, 16640])
def test_pr_averages_are_the_same_for_every_split(gpu, K):
    scs = [S.robust_race(agent=i, seed=3, K=K if i == 0 else 200 + i, T=24, P=3, n_theta=2) for i in range(14)]
    out = []
    for n in (1, len(scs)):
        ctls = [drb.controllers.PRMPPIController(s.env, s.prmppi, 7 + i) for i, s in enumerate(scs[:n])]
        b = drb.controllers.PRMPPIBatch(ctls)
        r = []
        for _ in range(2):
            r.append(b.step([s.state for s in scs[:n]], np.stack([s.belief() for s in scs[:n]]))[0])
            r += list(ctls[0].nominals())
            i = b.infos[0]
            r.append(np.array([*i.cand_cost, *i.min_costs, *i.nu, *i.inv_temperature]))
        out.append(r)
        b.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
