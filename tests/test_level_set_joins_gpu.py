"""Joins of a level set's edges by several blocks a share of vertices and, on a
mesh with more shares than the launch wants blocks, by one: the noise in a
corner of a large constant field gives what the same window gives by itself
(which test_level_set_sizes_gpu compares with the numpy restatement)."""
import numpy as np
import pytest

from ftk2_b200 import api
from oracle import contour_oracle as co
from test_contour_gpu import as_dict, assert_same

pytestmark = pytest.mark.gpu
Q = 2.0 ** 20


@pytest.mark.parametrize("dims", [[9, 8, 7], [40, 30, 3], [5, 4, 6, 3], [13, 12, 11, 3]])
def test_noise_against_the_restatement(ctx, dims):
    f = np.random.default_rng(21).standard_normal(tuple(dims[::-1]))
    r = ctx.contour(api.regular_mesh_desc(dims), f, 0.0, Q)
    assert_same(as_dict(r), co.contour(f, 0.0, dims, q=Q))


@pytest.mark.parametrize("big,window", [([2300, 2201, 2], [50, 40, 2]), ([61, 57, 53, 60], [12, 11, 10, 5])])
def test_window_of_a_large_mesh(ctx, big, window):
    off = [b - w for b, w in zip(big, window)]
    noise = np.random.default_rng(22).standard_normal(tuple(window[::-1])).astype(np.float32)
    edge = np.ones_like(noise, dtype=bool)  # a rim of the constant around the noise
    edge[tuple(slice(1 if o else 0, None) for o in off[::-1])] = False
    noise[edge] = 1.0
    f = np.ones(tuple(big[::-1]), np.float32)
    f[tuple(slice(o, None) for o in off[::-1])] = noise
    whole = ctx.contour(api.regular_mesh_desc(big), f, 0.0, Q)
    part = ctx.contour(api.regular_mesh_desc(window, off, big), noise, 0.0, Q)
    assert len(part.track_id) > 1000
    assert_same(as_dict(whole), as_dict(part))


def _labels(n, cells):
    """Smallest member of every node's component under the cells."""
    label = np.arange(n)
    while True:
        low = label[cells].min(1)
        new = label.copy()
        for j in range(cells.shape[1]):
            np.minimum.at(new, cells[:, j], low)
            np.minimum.at(new, label[cells[:, j]], low)
        while not np.array_equal(new, new[new]):
            new = new[new]
        if np.array_equal(new, label):
            return label
        label = new


@pytest.mark.parametrize("dims,above", [([270, 230, 5], False), ([340, 270, 6], True), ([32, 30, 28, 9], True)])
def test_tracks_around_the_hooked_size(ctx, dims, above):
    """Tracks of noise below and above the 2^20 edges from which the trees are
    hooked and flattened ahead, against the components of the call's own cells
    (compared with the restatement elsewhere)."""
    f = np.random.default_rng(23).standard_normal(tuple(dims[::-1])).astype(np.float32)
    r = ctx.contour(api.regular_mesh_desc(dims), f, 0.6, Q)
    assert (len(r.track_id) >= 1 << 20) == above
    assert np.array_equal(r.track_id, _labels(len(r.track_id), r.cells.astype(np.int64)))
    assert r.n_tracks == len(np.unique(r.track_id)) > 1
