"""Trees built by the clustering's launches (more than 512 triangles), against the
oracle's brute-force hits, equal bit for bit: either side of the one-block limit
and of a launch's blocks, past 256 blocks, a batch of passes that leaves one
cluster, runs of identical triangles, and scenes on which the nearest-neighbour
search alone merges one pair a pass: triangles nested in one another, in a plane
(a tree higher than the traversal's stack) and along an axis, and growing gaps."""
import numpy as np
import pytest

from gpu_util import host

pytestmark = pytest.mark.gpu


def _triangles(kind, n, rng):
    """(n, 3, 3) triangles around the origin."""
    if kind == "identical":
        return np.repeat(np.array([[[-1.0, -1.0, 0.0], [1.0, -1.0, 0.2], [0.0, 1.0, 0.1]]]), n, 0)
    size = 2.5 * n ** -0.4
    t = rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-size, size, (n, 3, 3))
    if kind == "random":
        return t
    if kind == "wall":
        t[n // 2] = [[-40, -40, 1.2], [40, -40, 1.3], [0, 60, 1.1]]
        return t
    if kind == "never hit":
        t[::5, 1, 0] = np.nan
        t[1::5, 2, 1] = np.inf
        t[2::5, 2] = t[2::5, 1]
        return t
    i = np.arange(n)
    if kind == "gaps":
        x = np.cumsum(1.001 ** i)
        x = (x / x[-1] * 3.0 - 1.5)[:, None]
        return np.stack([np.concatenate([x, 0 * x - 1, 0 * x], 1), np.concatenate([x + 1e-4, 0 * x + 1, 0 * x], 1),
                         np.concatenate([x, 0 * x + 1, 0 * x + 0.01], 1)], 1)
    s = 1.0005 ** i
    z = np.zeros(n)
    t = np.stack([np.stack([s, z, z], 1), np.stack([-s, s, z], 1), np.stack([z, -s, z], 1)], 1) * (2.0 / s[-1])
    if kind == "nested along z":
        t[:, :, 2] = -0.5 * i[:, None] / n
    return t


def _compare(oracle, tri, w, h):
    from vknrc_gb300 import nrc, synthetic as S

    n = len(tri)
    sc = S.scene(S.rng_for(n), vertices=300, primitives=100, instances=1)
    for k in ("texcoord_indices", "material_ids"):
        sc[k] = np.resize(sc[k], (n,) + sc[k].shape[1:])
    sc["vertices"] = tri.reshape(-1, 3).astype(np.float32)
    sc["vertex_indices"] = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    sc["transforms"][0] = np.eye(3, 4, dtype=np.float32)
    sc["instance_ranges"] = np.array([[0, n]], np.uint32)
    P = oracle.TraceParams()
    for k, v in {"origin": (0.0, 0.3, -4.0), "look": (0.0, 0.0, 1.0), "side": (0.5, 0.0, 0.0),
                 "up": (0.0, 0.4, 0.0)}.items():
        getattr(P, k)[:] = v
    P.width, P.height, P.seed, P.left_method, P.right_method, P.train_probability = w, h, 11, 0, 1, 0.3
    ref = oracle.path_trace(sc, P, w * h + 65536)
    ds = nrc.DeviceScene(sc)
    bvh = nrc.Bvh(ds)
    assert bvh.info() == (n, n - 1)
    buf = nrc.TraceBuffers(w, h)
    buf.reset()
    nrc.path_trace(ds, bvh, nrc.TraceParams.from_buffer_copy(bytes(P)), buf)
    assert np.array_equal(host(buf.bias_factor_r), ref["bias_factor_r"])
    assert np.array_equal(host(buf.factor_gb), ref["factor_gb"])
    assert int(host(buf.eval_count)[0]) == ref["eval_count"]
    assert [int(host(c)[0]) for c in buf.train_counts] == ref["train_counts"]
    assert len(np.unique(ref["bias_factor_r"].reshape(-1, 4), axis=0)) > 20
    bvh.close()


@pytest.mark.parametrize("kind,n", [("random", k) for k in (511, 512, 513, 769, 1023, 1024, 1025, 3000, 8192, 8193)] +
                         [("identical", 513), ("identical", 3000), ("wall", 2000), ("never hit", 2000), ("gaps", 4000),
                          ("nested", 8000), ("nested along z", 4000)])
def test_hits_equal_brute_force(cuda, oracle, kind, n):
    from vknrc_gb300 import synthetic as S

    _compare(oracle, _triangles(kind, n, S.rng_for(n + len(kind))), 64, 40)


def test_hits_equal_brute_force_past_256_blocks(cuda, oracle):
    from vknrc_gb300 import synthetic as S

    _compare(oracle, _triangles("random", 70000, S.rng_for(70)), 32, 20)


def test_build_time_is_bounded(cuda):
    """Triangles whose boxes grow along the order take a bounded number of passes: one
    merge a pass is some hundred times as long as an ordinary scene's build."""
    import time

    import torch

    from vknrc_gb300 import nrc, synthetic as S

    n, best = 60000, []
    for kind in ("random", "nested along z"):
        sc = S.scene(S.rng_for(3), vertices=300, primitives=100, instances=1)
        for k in ("texcoord_indices", "material_ids"):
            sc[k] = np.resize(sc[k], (n,) + sc[k].shape[1:])
        sc["vertices"] = _triangles(kind, n, S.rng_for(n)).reshape(-1, 3).astype(np.float32)
        sc["vertex_indices"] = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
        sc["instance_ranges"] = np.array([[0, n]], np.uint32)
        ds, times = nrc.DeviceScene(sc), []
        for _ in range(4):
            torch.cuda.synchronize()
            t = time.perf_counter()
            nrc.Bvh(ds).close()
            times.append(time.perf_counter() - t)
        best.append(min(times))
    assert best[1] < 15 * best[0], best
