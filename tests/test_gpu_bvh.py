"""The path tracer's tree over scenes whose shape is hard on it, against the
oracle's brute-force hits (equal bit for bit, as in test_trace.py): from no
triangle to just past each node and leaf size, runs of identical triangles, a
chain of shrinking triangles (a tall tree), one triangle far larger than the
rest, and triangles that can never be hit."""
import numpy as np
import pytest

from gpu_util import host

pytestmark = pytest.mark.gpu


def _triangles(kind, n, rng):
    """(n, 3, 3) float32 triangles around the origin."""
    if kind == "random":
        return rng.uniform(-1, 1, (n, 3, 3))
    if kind == "identical":
        return np.repeat(rng.uniform(-1, 1, (1, 3, 3)) * 1.5, n, 0)
    if kind == "chain":
        s = 0.93 ** np.arange(n)[:, None, None]
        return rng.uniform(-0.5, 0.5, (n, 3, 3)) * s + s * np.array([2.0, 0.4, 0.0])
    t = rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-0.1, 0.1, (n, 3, 3))
    if kind == "wall":
        t[n // 2] = [[-40, -40, 1.2], [40, -40, 1.3], [0, 60, 1.1]]
    else:  # "never hit": NaN, infinite and zero-area triangles among the rest
        t[::5, 1, 0] = np.nan
        t[1::5, 2, 1] = np.inf
        t[2::5, 2] = t[2::5, 1]
    return t


@pytest.mark.parametrize("kind,n", [("random", k) for k in (0, 1, 2, 3, 4, 5, 7, 13, 17, 257)] +
                         [("identical", 2), ("identical", 300), ("chain", 400), ("wall", 500), ("never hit", 300)])
def test_hits_equal_brute_force(cuda, oracle, kind, n):
    from vknrc_gb300 import nrc, synthetic as S

    rng = S.rng_for(n + len(kind))
    sc = S.scene(rng, vertices=max(3 * n, 3), primitives=max(n, 1), instances=1)
    if n > 0:
        sc["vertices"] = _triangles(kind, n, rng).reshape(-1, 3).astype(np.float32)
        sc["vertex_indices"] = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    sc["transforms"][0] = np.eye(3, 4, dtype=np.float32)
    sc["instance_ranges"] = np.array([[0, n]], np.uint32)
    w, h = 64, 40
    P = oracle.TraceParams()
    for k, v in {"origin": (0.0, 0.3, -4.0), "look": (0.0, 0.0, 1.0), "side": (0.5, 0.0, 0.0),
                 "up": (0.0, 0.4, 0.0)}.items():
        getattr(P, k)[:] = v
    P.width, P.height, P.seed, P.left_method, P.right_method, P.train_probability = w, h, 11, 0, 1, 0.3
    ref = oracle.path_trace(sc, P, w * h + 65536)
    ds = nrc.DeviceScene(sc)
    bvh = nrc.Bvh(ds)
    assert bvh.info() == (n, max(n - 1, 0))
    buf = nrc.TraceBuffers(w, h)
    buf.reset()
    nrc.path_trace(ds, bvh, nrc.TraceParams.from_buffer_copy(bytes(P)), buf)
    assert np.array_equal(host(buf.bias_factor_r), ref["bias_factor_r"])
    assert np.array_equal(host(buf.factor_gb), ref["factor_gb"])
    assert int(host(buf.eval_count)[0]) == ref["eval_count"]
    assert [int(host(c)[0]) for c in buf.train_counts] == ref["train_counts"]
    bvh.close()
