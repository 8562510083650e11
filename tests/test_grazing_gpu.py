"""Forms of the closest hit where the order of visits decides it
(grazing_cases.py): every form of a call agrees with the loop that it stands
for, bit for bit."""
import numpy as np
import pytest

import grazing_cases as G
from renderingengine_b200 import _native as N
from renderingengine_b200.traversal import Scene

pytestmark = pytest.mark.gpu


def _rays(o, d, tmax=1.0):
    r = np.zeros(len(o), N.RAY_DTYPE)
    r["origin_tmin"][:, :3], r["origin_tmin"][:, 3] = o, 1e-4
    r["direction_tmax"][:, :3], r["direction_tmax"][:, 3] = d, tmax
    return r


@pytest.mark.parametrize("build", [N.BUILD_FLATTENED_SAH, N.BUILD_LBVH], ids=["sah", "lbvh"])
@pytest.mark.parametrize("seed,side,clutter", [(1, 4, 70), (2, 6, 30), (3, 10, 6), (4, 10, 14)])
def test_grazing_batches_equal_child_pair_loop(native, build, seed, side, clutter):
    """Counted batches always walk the child pairs; the others take the form of
    their size, before and after a batch of 2^18 rays."""
    data, o, _, d = G.scene(seed, side, clutter)
    scene = Scene(data.triangles, 5, 1, build)
    one = _rays(o, d)
    many = np.resize(one, 1 << 18)
    for rays in (one, many, one):
        for any_hit in (False, True):
            want, _ = scene.trace(rays, any_hit=any_hit, counters=True)
            got = scene.trace(rays, any_hit=any_hit)
            assert (want["metadata"][:, 1] == N.HIT_KIND_TRIANGLE).mean() > 0.9
            differ = (got.view(np.uint32).reshape(len(rays), -1) != want.view(np.uint32).reshape(len(rays), -1)).any(1)
            assert not differ.any(), f"{differ[:len(one)].sum()} of {len(one)} rays, any-hit {any_hit}"
