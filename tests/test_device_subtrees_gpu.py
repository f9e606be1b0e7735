"""Device build at the sizes where a node goes from level rounds to a block of
its own (256 primitives), against the oracle: every array of the reference
layout byte-identical."""

import numpy as np
import pytest

from helpers import Scene, rt, scenes, single_mesh_scene
from test_device_build_gpu import assert_arrays_equal, assert_same_traces, degenerate_soup

pytestmark = pytest.mark.gpu


def check(sc, **options):
    S = sc.build_oracle(**options)
    P = sc.build_product(device_build=True, **options)
    assert_arrays_equal(P, S=S)
    a, b = P.build_stats(), S.build_stats()
    assert a["sah_splits"] == b["sah_splits"] and a["median_fallbacks"] == b["median_fallbacks"]
    return P


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 255, 256, 257, 511, 513, 1025])
@pytest.mark.parametrize("bins", [1, 4])
def test_sizes(n, bins, cuda):
    sc = single_mesh_scene(scenes.triangle_soup(n, seed=n), bins=bins)
    P = check(sc)
    assert_same_traces(P, sc.build_product(), scenes.sphere_rays(500, (0, 0, 0), (1, 1, 1), seed=n))


@pytest.mark.parametrize("n", [7, 256, 300, 2000])
def test_median_splits(n, cuda):
    check(single_mesh_scene(degenerate_soup(n, seed=n), bins=1))
    same = scenes.Mesh(np.tile(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), (n, 1)), None)
    check(single_mesh_scene(same, bins=1))


@pytest.mark.parametrize("depth", [1, 4, 9])
@pytest.mark.parametrize("bins", [300, 100])
def test_depth_limit_and_large_leaves(depth, bins, cuda):
    check(single_mesh_scene(scenes.triangle_soup(3000, seed=6), bins=bins), blas_max_depth=depth)


def test_many_sizes_in_one_build(cuda):
    sizes = [0, 1, 256, 257, 5, 3000, 255, 0, 700]
    blas = [[(scenes.triangle_soup(max(n, 1), seed=k).positions[: 3 * n], None, 1)] for k, n in enumerate(sizes)]
    check(Scene(blas, [[{"blas": k} for k in range(len(sizes))]]))


@pytest.mark.parametrize("n", [200, 300])
def test_empty_children(n, cuda):
    """Areas beyond the float range: no candidate is below infinity, so the
    first one is taken although its side is empty, down to the depth limit."""
    rng = np.random.default_rng(n)
    tri = rng.uniform(2e19, 3e19, (n, 3, 3))
    tri[:, 0] = rng.uniform(0, 1e18, (n, 3))
    tri[:, 1] = rng.uniform(2.9e19, 3e19, (n, 3))
    P = check(single_mesh_scene(scenes.Mesh(tri.astype(np.float32).reshape(-1, 3), None), bins=4), blas_max_depth=12)
    nodes = np.frombuffer(P.built_array("tri_bvh_forest"), np.uint32).reshape(-1, 12)
    assert (nodes[:, 8] == nodes[:, 9]).any()  # content_range: an empty leaf
