"""dr_mppi_batch_predict_device writes into the caller's device buffers, which need a float's
alignment and no more: outputs that start one float past a 16-byte boundary, beside outputs at one,
with the same values and nothing written around them."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import drb

pytestmark = pytest.mark.gpu
abi = drb.abi
S = drb.scenarios


@pytest.mark.parametrize("nth", [1, 2, 8])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_outputs_of_float_alignment(gpu, nth, shift):
    import torch

    scs = [S.circle_race(agent=a, seed=a, K=64, T=21 + 6 * a, n_theta=nth, n_verif=64) for a in range(2)]
    ctls = [drb.controllers.MPPIController(s.env, s.mppi, s.seed) for s in scs]
    batch = drb.controllers.MPPIBatch(ctls)
    st = torch.frombuffer(bytearray(bytes((type(scs[0].state) * 2)(*[s.state for s in scs]))), dtype=torch.uint8).cuda()
    bel = np.zeros((2, abi.DR_MAX_THETA), np.float32)
    for i, s in enumerate(scs):
        bel[i, :nth] = s.belief()
    bel = torch.from_numpy(bel).cuda()
    act0, infos = torch.zeros((2, 2), device="cuda"), torch.zeros(2 * C.sizeof(abi.dr_mppi_info), dtype=torch.uint8, device="cuda")
    batch.step_device(st.data_ptr(), bel.data_ptr(), act0.data_ptr(), infos.data_ptr())
    T, rows = 30, 2 * nth
    sizes = (rows * T * 4, rows * T * 2, rows * abi.DR_PREDICT_RECORD, rows)
    out = []
    for off in (0, shift):
        bufs = [torch.full((n + 8,), -7, dtype=d, device="cuda") for n, d in zip(sizes, (torch.float32, torch.float32, torch.int32, torch.float32))]
        abi.check(abi.lib().dr_mppi_batch_predict_device(batch._b, st.data_ptr(), bel.data_ptr(), *[b.data_ptr() + 4 * off for b in bufs], T), "predict_device")
        torch.cuda.synchronize()
        for b, n in zip(bufs, sizes):
            assert bool((b[:off] == -7).all()) and bool((b[off + n :] == -7).all())
        out.append([b[off : off + n].cpu().numpy() for b, n in zip(bufs, sizes)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
