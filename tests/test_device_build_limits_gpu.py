"""Device builds of forests that want more nodes than the build's pool holds:
splits with an empty child, repeated down to the depth limit in many small
geometries. The build is refused, nothing is written or read past the pool, and
the context goes on with builds that fit."""

import numpy as np
import pytest

from helpers import Scene, scenes, single_mesh_scene
from rendiation_gb300 import native
from test_device_build_gpu import assert_arrays_equal, assert_same_traces

pytestmark = pytest.mark.gpu


def stuck_soup(n, seed):
    """Triangles whose boxes' areas are beyond the float range: no split candidate is below infinity, so the first one
    is taken although its left side is empty."""
    rng = np.random.default_rng(seed)
    tri = rng.uniform(2e19, 3e19, (n, 3, 3))
    tri[:, 0] = rng.uniform(0, 1e18, (n, 3))
    tri[:, 1] = rng.uniform(2.9e19, 3e19, (n, 3))
    return tri.astype(np.float32).reshape(-1, 3)


# g geometries of t triangles: a pool of 2 g t + 2 g + 64 nodes; at the default depth limit of 50 they want
# g (1 + 2 * 50), so up to 49 triangles each do not fit (the last level that is begun fits in part or not at all).
@pytest.mark.parametrize("geoms,tris", [(1000, 5), (37, 9), (4, 10)])
def test_pool_overflow_is_refused(geoms, tris, cuda):
    assert geoms * 101 > 2 * geoms * tris + 2 * geoms + 64
    sc = Scene([[(stuck_soup(tris, k), None, 1)] for k in range(geoms)], [[{"blas": k}] for k in range(geoms)])
    P = sc.build_product()  # the host build takes such a forest
    for _ in range(2):
        with pytest.raises(native.RdnError, match="more nodes"):
            P.build(blas_bin_size=4, tlas_bin_size=10, device_build=True)
    P.build(blas_bin_size=4, tlas_bin_size=10, blas_max_depth=2, device_build=True)
    assert_arrays_equal(P, S=sc.build_oracle(blas_max_depth=2))
    good = single_mesh_scene(scenes.triangle_soup(3000, seed=geoms))
    Q = good.build_product(device_build=True)
    assert_arrays_equal(Q, S=good.build_oracle())
    assert_same_traces(Q, good.build_product(), scenes.sphere_rays(500, (0, 0, 0), (1, 1, 1), seed=2))
    assert Q.check_errors() == (0, 0)


@pytest.mark.parametrize("geoms,tris,depth", [(1, 30, 20), (4, 300, 50)])
def test_stuck_forest_that_fits(geoms, tris, depth, cuda):
    assert geoms * (1 + 2 * depth) <= 2 * geoms * tris + 2 * geoms + 64
    sc = Scene([[(stuck_soup(tris, k), None, 1)] for k in range(geoms)], [[{"blas": k}] for k in range(geoms)])
    P = sc.build_product(device_build=True, blas_max_depth=depth)
    assert_arrays_equal(P, S=sc.build_oracle(blas_max_depth=depth))
