"""Which triangles a ray hits does not depend on how the tree groups them: the same
triangles with and without others far away, which no ray reaches but which change
the order and the boxes, give the same image bit for bit. The scenes are slivers
seen from so far away that the rounding of the intersection test accepts points
off the triangle."""
import numpy as np
import pytest

from gpu_util import host

pytestmark = pytest.mark.gpu


def _image(tri, distance, w=192, h=120):
    from vknrc_gb300 import nrc, synthetic as S

    n = len(tri)
    sc = S.scene(S.rng_for(5), vertices=300, primitives=100, instances=1)
    for k in ("texcoord_indices", "material_ids"):
        sc[k] = np.resize(sc[k], (n,) + sc[k].shape[1:])
    sc["vertices"] = tri.reshape(-1, 3).astype(np.float32)
    sc["vertex_indices"] = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    sc["transforms"][0] = np.eye(3, 4, dtype=np.float32)
    sc["instance_ranges"] = np.array([[0, n]], np.uint32)
    ds = nrc.DeviceScene(sc)
    buf = nrc.TraceBuffers(w, h)
    buf.reset()
    look = np.array([0.6, -0.5, 0.62]) / np.linalg.norm([0.6, -0.5, 0.62])
    side = np.cross(look, [0, 1, 0]) / np.linalg.norm(np.cross(look, [0, 1, 0]))
    P = nrc.TraceParams()
    for k, v in {"origin": -look * distance, "look": look, "side": side * 1.2 / distance,
                 "up": np.cross(side, look) * 1.2 / distance}.items():
        getattr(P, k)[:] = v.tolist()
    P.width, P.height, P.seed = w, h, 3
    bvh = nrc.Bvh(ds)
    nrc.path_trace(ds, bvh, P, buf)
    out = host(buf.bias_factor_r).view(np.uint32).copy()
    bvh.close()
    return out


@pytest.mark.parametrize("n,distance", [(1000, 4e4), (300, 1e5), (1000, 4.0)])
def test_hits_do_not_depend_on_grouping(cuda, n, distance):
    rng = np.random.default_rng(17)
    c = rng.uniform(-1, 1, (n, 1, 3))
    a = rng.standard_normal((n, 3))
    a = (0.3 * a / np.linalg.norm(a, axis=1, keepdims=True))[:, None]
    b = 0.01 * rng.standard_normal((n, 1, 3))
    t = np.concatenate([c - a, c + a, c + b], 1)
    far = rng.uniform(-1, 1, (n, 1, 3)) * [5, 40, 5] + [0, 300, 0] + rng.uniform(-0.5, 0.5, (n, 3, 3))
    alone = _image(t, distance)
    assert len(np.unique(alone.reshape(-1, 4), axis=0)) > 100
    assert np.array_equal(alone, _image(np.concatenate([t, far]), distance))


def test_tree_memory(cuda):
    """A tree holds less than 140 bytes a triangle (one box, one copy of the
    vertices and a third of a 128-byte node each)."""
    import torch

    from vknrc_gb300 import nrc, synthetic as S

    ds = nrc.DeviceScene(S.terrain_scene(S.rng_for(1), 512))
    nrc.Bvh(ds).close()  # whatever the first build loads
    free = torch.cuda.mem_get_info()[0]
    bvh = nrc.Bvh(ds)
    held = free - torch.cuda.mem_get_info()[0]
    triangles = bvh.info()[0]
    bvh.close()
    assert held <= 140 * triangles + (4 << 20), held / triangles
