"""Scenes far from the origin, against the oracle's brute-force hits: coordinates
past the +-1e15 that the tree's boxes keep, and rays whose origin over a component
of their direction overflows."""
import numpy as np
import pytest

from gpu_util import host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("far", [2.0 ** 53, -2.0 ** 53, 2.0 ** 62])
def test_hits_equal_brute_force_far_from_the_origin(cuda, oracle, far, axis):
    from vknrc_gb300 import nrc, synthetic as S

    n, unit = 200, abs(far) * 2.0 ** -23  # a few representable steps of the far coordinate
    rng = S.rng_for(int(axis))
    t = (rng.uniform(-4, 4, (n, 1, 3)) + rng.uniform(-1, 1, (n, 3, 3))) * unit
    # the far coordinate, across the view
    t[:, :, axis] = far + unit * (rng.integers(0, 4, (n, 1)) + rng.integers(0, 2, (n, 3)))
    sc = S.scene(rng, vertices=3 * n, primitives=n, instances=1)
    sc["vertices"] = t.reshape(-1, 3).astype(np.float32)
    sc["vertex_indices"] = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    sc["transforms"][0] = np.eye(3, 4, dtype=np.float32)
    sc["instance_ranges"] = np.array([[0, n]], np.uint32)
    P = oracle.TraceParams()
    w, h = 63, 41  # odd: the middle column and row have a zero component
    look = np.zeros(3)
    look[2 if axis == 1 else 1] = 1.0
    side, up = np.zeros(3), np.zeros(3)
    side[axis], up[3 - axis - (2 if axis == 1 else 1)] = 0.5, 0.4
    origin = -8 * unit * look
    origin[axis] = far + 2 * unit
    for k, v in {"origin": origin, "look": look, "side": side, "up": up}.items():
        getattr(P, k)[:] = v.tolist()
    P.width, P.height, P.seed, P.left_method, P.right_method, P.train_probability = w, h, 11, 0, 0, 0.0
    ref = oracle.path_trace(sc, P, w * h + 65536)
    img = ref["bias_factor_r"].reshape(-1, 4)
    hits = (~(img == img[0, :]).all(1)).sum()
    ds = nrc.DeviceScene(sc)
    bvh = nrc.Bvh(ds)
    buf = nrc.TraceBuffers(w, h)
    buf.reset()
    nrc.path_trace(ds, bvh, nrc.TraceParams.from_buffer_copy(bytes(P)), buf)
    assert hits > 100
    assert np.array_equal(host(buf.bias_factor_r), ref["bias_factor_r"], equal_nan=True)
    assert np.array_equal(host(buf.factor_gb), ref["factor_gb"], equal_nan=True)
    bvh.close()
