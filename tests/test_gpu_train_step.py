"""A single training step (two launches: the gradient pass, the optimizer step)
against the same step as one cooperative launch of the same CTA count
(nrc_train_many), bit for bit, at the edges of the tiles and of the grid: no
record, part of a tile, one tile more than the CTAs, a count past the capacity
and one past the batch size."""
import numpy as np
import pytest

from gpu_util import count, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("n,capacity,batch",
                         [(0, 256, 16384), (1, 1, 16384), (127, 128, 16384), (129, 129, 16384), (10240, 10240, 16384),
                          (19456, 19456, 65536), (19457, 19457, 65536), (500, 300, 16384), (5000, 5000, 4000)])
def test_single_step_equals_fused_launch(cuda, precision, n, capacity, batch):
    from vknrc_gb300 import Cache, nrc
    from vknrc_gb300 import synthetic as S

    prec = nrc.PRECISION_BF16 if precision == "bf16" else nrc.PRECISION_FP16
    rec = dev(S.train_records(S.rng_for(300 + n), capacity, target="field", sigma=0.5))
    with Cache(seed=301, precision=prec, train_batch_size=batch) as a, \
            Cache(seed=301, precision=prec, train_batch_size=batch) as b:
        for step in range(3):
            ca, cb = count(n), count(n)
            a.train(rec, ca, write_use=step != 1, capacity=capacity)
            nrc.train_many([nrc.train_job(b, [rec], [cb], write_use_last=step != 1, capacity=capacity)], ctas=[152])
            assert int(host(ca)[0]) == int(host(cb)[0]) == min(n, batch)
            assert np.array_equal(a.get_weights(0), b.get_weights(0)), step
            assert np.array_equal(a.get_weights(1), b.get_weights(1)), step
        assert a.get_optimizer()[0] == b.get_optimizer()[0]
        assert np.array_equal(a.get_optimizer()[1], b.get_optimizer()[1])
        assert a.error() == 0 and b.error() == 0
