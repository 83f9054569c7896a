"""The frame on packed records unpacks its eval records and its train batches in one launch
(UnpackNRCInput, shader/src/NRCRecord.glsl:97-125): bit for bit the outputs, weights and
optimizer entries of the separate unpack calls followed by the same frame, at record counts
around a warp's group, a block and the resident grid, with uneven and empty batches."""
import numpy as np
import pytest

from gpu_util import count, dev, host

pytestmark = pytest.mark.gpu


# eval records, their capacity, train capacity, train counts
@pytest.mark.parametrize("q,qcap,r,counts", [
    (1, 1, 1, (1, 1, 1, 1)),
    (31, 64, 33, (33, 32, 31, 1)),
    (300, 257, 129, (0, 129, 200, 1)),  # counts past their capacities
    (0, 70, 64, (64, 0, 0, 64)),
    (70001, 70001, 2500, (2500, 1, 0, 2499)),
    (1000, 1000, 40000, (40000, 39999, 0, 17)),  # more train records than eval records
    (1000, 1000, 0, (0, 0, 0, 0)),
])
@pytest.mark.parametrize("prepared", [False, True])
def test_frame_packed_one_unpack_launch(cuda, q, qcap, r, counts, prepared):
    import torch

    from vknrc_gb300 import Cache, nrc, synthetic as S

    sc = S.scene(S.rng_for(70))
    ds = nrc.DeviceScene(sc).prepare() if prepared else nrc.DeviceScene(sc)
    ev = dev(S.eval_records(S.rng_for(71), sc, qcap, bad_fraction=0.02).view(np.int32))
    tr = [dev(S.packed_train_records(S.rng_for(72, b), sc, max(r, 1)).view(np.int32)) for b in range(4)]
    res = []
    for packed in (True, False):
        with Cache(seed=73, learning_rate=1e-3, beta2=0.99) as c:
            out = torch.full((qcap, 3), -1.0, dtype=torch.float32, device="cuda")
            for _ in range(2):
                n, cnt = count(q), [count(k) for k in counts]
                if packed:
                    c.frame_packed(ds, ev, n, out, tr, cnt, eval_capacity=qcap, train_capacity=r)
                else:
                    inputs = torch.zeros((qcap, 14), dtype=torch.float32, device="cuda")
                    nrc.unpack_eval(ds, ev, n, inputs)
                    us = [torch.zeros((max(r, 1), 20), dtype=torch.float32, device="cuda") for _ in range(4)]
                    for t, u, k in zip(tr, us, cnt):
                        nrc.unpack_train(ds, t, k, u, capacity=r)
                    c.frame_overlapped(inputs, n, out, us, cnt, eval_capacity=qcap, train_capacity=r)
            res.append((host(out), c.get_weights(0), c.get_optimizer()[1]))
            assert c.error() == 0
    for a, b in zip(res[0], res[1]):
        np.testing.assert_array_equal(a, b)
