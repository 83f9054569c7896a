"""A single training step is applied as a whole or not at all, and a time-out of
an earlier call does not stop later steps. No wait runs out here: the words that
a time-out leaves are written by the test (the error word and, after it, the
trainer's words, which sit behind the step state in the cache's block: two barrier
counters, then from the fifth word on the number of the step in flight, that of the
last step that failed, the state to write and the number of steps launched)."""
import ctypes

import numpy as np
import pytest

from gpu_util import count, dev, host

pytestmark = pytest.mark.gpu

STATE_TO_ERROR, ERROR_TO_TRAINER = 256, 64  # bytes


class _Words:
    def __init__(self, address, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (address, False), "version": 3}


def _words(address, n):
    import torch

    return torch.as_tensor(_Words(address, n), device="cuda")


def _same(a, b):
    return (a.get_optimizer()[0] == b.get_optimizer()[0] and np.array_equal(a.get_optimizer()[1], b.get_optimizer()[1]) and
            np.array_equal(a.get_weights(0), b.get_weights(0)) and np.array_equal(a.get_weights(1), b.get_weights(1)))


def _train_records(n):
    from vknrc_gb300 import synthetic as S

    return dev(S.train_records(S.rng_for(500 + n), n, target="field", sigma=0.5))


@pytest.mark.parametrize("word", [1, 3, -1])
def test_steps_go_on_after_a_timeout(cuda, word):
    from vknrc_gb300 import Cache

    rec = _train_records(3000)
    with Cache(seed=501) as a, Cache(seed=501) as b:
        err = _words(b.device_buffers()[3] + STATE_TO_ERROR, 1)
        err.fill_(word)
        for _ in range(2):
            a.train(rec, count(3000))
            b.train(rec, count(3000))
        assert a.get_optimizer()[0][0] == 2 and _same(a, b)
        assert a.error() == 0 and b.error() != 0 and b.error() == 0


@pytest.mark.parametrize("word", [2, 3, -1])
def test_noalloc_does_not_read_its_error_word(cuda, word):
    import torch

    from vknrc_gb300 import Cache, nrc

    rec, cfg = _train_records(1000), nrc.default_config()
    with Cache(seed=502) as a, Cache(seed=502) as b:
        for c, err in ((a, None), (b, torch.full((1,), word, dtype=torch.int32, device="cuda"))):
            w, use, ent, st = c.device_buffers()
            assert nrc.lib().nrc_train_noalloc(w, use, ent, st, rec.data_ptr(), count(1000).data_ptr(), 1000, ctypes.byref(cfg),
                                               None if err is None else err.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream) == 0
        assert a.get_optimizer()[0][0] == 1 and _same(a, b)
        assert int(host(err)[0]) == word


@pytest.mark.parametrize("n", [0, 3000])
def test_failed_gradient_pass_changes_nothing(cuda, n):
    from vknrc_gb300 import Cache

    rec = _train_records(3000)
    with Cache(seed=503) as a, Cache(seed=503) as b, Cache(seed=503) as untouched:
        words = _words(b.device_buffers()[3] + STATE_TO_ERROR + ERROR_TO_TRAINER, 13)
        assert not host(words).any()
        words[5] = 1  # what a CTA of the first step's gradient pass that gave up leaves
        b.train(rec, count(n))
        assert _same(b, untouched) and host(words)[[0, 1, 4, 5, 12]].tolist() == [0, 0, 1, 1, 1]
        a.train(rec, count(3000))
        b.train(rec, count(3000))
        assert a.get_optimizer()[0][0] == 1 and _same(a, b) and host(words)[[0, 1, 4, 5, 12]].tolist() == [0, 0, 2, 1, 2]
