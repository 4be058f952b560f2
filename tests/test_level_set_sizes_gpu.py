"""Level sets and fiber surfaces on meshes whose vertices end at, before and
after a word (32) and a block's share (1024) of the kernels, with layers of one
vertex, arrays larger than the mesh, and values that are mostly one sign or
noise: level sets against the numpy restatement, fiber surfaces against a plain
enumeration of the mesh's triangles and pentatopes (engine.hpp:1388-1413)."""
import itertools

import numpy as np
import pytest

from ftk2_b200 import api
from oracle import contour_oracle as co
from test_contour_gpu import as_dict, assert_same

pytestmark = pytest.mark.gpu
Q = 2.0 ** 20


def _field(dims, seed, kind, dtype, pad=0):
    rng = np.random.default_rng(seed)
    shape = tuple(d + pad for d in reversed(dims))
    f = rng.standard_normal(shape)
    if kind == "smooth":
        g = np.indices(shape).sum(0) / (sum(shape) - len(shape) + 1) - 0.5
        f = g + 0.02 * f
    if kind == "ties":
        f = rng.integers(-1, 2, shape) / Q
    return f.astype(dtype)


@pytest.mark.parametrize("kind", ["noise", "smooth", "ties"])
@pytest.mark.parametrize("dims,pad,dtype", [([2, 2, 2], 0, np.float64), ([31, 1, 2], 0, np.float32),
                                            ([8, 4, 1], 0, np.float64), ([11, 31, 3], 0, np.float64),
                                            ([32, 16, 2], 3, np.float32), ([25, 41, 2], 0, np.float32),
                                            ([1, 2, 3, 4], 0, np.float64), ([5, 3, 2, 2], 2, np.float64),
                                            ([8, 8, 8, 2], 0, np.float32), ([7, 9, 5, 4], 0, np.float64),
                                            ([41, 5, 5, 2], 0, np.float32)])
def test_level_set(ctx, dims, pad, dtype, kind):
    f = _field(dims, 3, kind, dtype, pad)
    r = ctx.contour(api.regular_mesh_desc(dims), f, 0.0, Q)
    inner = np.ascontiguousarray(f[tuple(slice(0, d) for d in reversed(dims))])
    want = co.contour(inner, 0.0, dims, q=Q)
    assert_same(as_dict(r), want)
    assert r.n_tracks == len(set(r.track_id.tolist()))


def _fiber_surface(f0, f1, dims):
    """Feature rows, cells and track ids of the origin's fiber surface."""
    ids = np.arange(np.prod(dims)).reshape(dims[::-1])
    quant = [(f.astype(np.float64) * Q + np.where(f > 0, 0.5, -0.5)).astype(np.int64).ravel() for f in (f0, f1)]
    q = np.stack(quant, 1)

    def inside(v):
        s = []
        for a, b, tie in ((0, 1, 1), (1, 2, 1), (2, 0, -1)):
            d = int(q[v[a], 0]) * int(q[v[b], 1]) - int(q[v[a], 1]) * int(q[v[b], 0])
            s.append((d > 0) - (d < 0) or tie)
        return s[0] == s[1] == s[2]

    stride = np.cumprod([1] + list(dims[:-1]))
    rank = {}
    for c in itertools.product(*(range(d) for d in reversed(dims))):
        c = c[::-1]
        v = int(ids[c[::-1]])
        off = {e: sum(int(stride[k]) for k in range(4) if e >> k & 1) for e in range(16)}
        for a in range(1, 16):
            for b in range(a + 1, 16):
                if a & b != a or any(b >> k & 1 and c[k] + 1 >= dims[k] for k in range(4)):
                    continue
                t = (v, v + off[a], v + off[b])
                if inside(t):
                    rank[t] = len(rank)
    parent = list(range(len(rank)))

    def root(x):
        while parent[x] != x:
            x = parent[x]
        return x

    cells = set()
    for c in itertools.product(*(range(d - 1) for d in dims)):
        base = sum(int(x * s) for x, s in zip(c, stride))
        for p in itertools.permutations(range(4)):
            path = [base]
            for k in p:
                path.append(path[-1] + int(stride[k]))
            found = sorted((rank[t], t) for t in itertools.combinations(path, 3) if t in rank)
            for out in path:
                face = [r for r, t in found if out not in t]
                for r in face[1:]:
                    hs, ht = found[0][0], face[0]
                    if hs == ht or hs == r:
                        continue
                    cells.add(tuple(sorted((hs, ht, r))))
                    for x in (ht, r):
                        a, b = sorted((root(hs), root(x)))
                        parent[b] = a
    rows = np.array(sorted(rank, key=rank.get), np.uint64).reshape(-1, 3)
    return rows, np.array(sorted(cells), np.uint32).reshape(-1, 3), np.array([root(i) for i in range(len(rank))],
                                                                             np.uint64)


@pytest.mark.parametrize("kind", ["noise", "smooth", "ties"])
@pytest.mark.parametrize("dims,pad,dtype", [([2, 2, 2, 2], 0, np.float64), ([31, 2, 1, 2], 0, np.float32),
                                            ([4, 4, 4, 4], 1, np.float64), ([8, 8, 8, 2], 0, np.float32),
                                            ([41, 5, 5, 1], 0, np.float64), ([7, 5, 6, 5], 0, np.float32)])
def test_fiber_surface(ctx, dims, pad, dtype, kind):
    f = [_field(dims, 5 + k, kind, dtype, pad) for k in range(2)]
    if kind == "smooth":
        f[1] = np.ascontiguousarray(f[1][::-1, :, ::-1])
    keep: list = []
    r = ctx.fiber_surface(api.regular_mesh_desc(dims), api.field_desc(f, api.LAYOUT_SEPARATE, 2, keep=keep),
                          (0.0, 0.0), Q)
    cut = tuple(slice(0, d) for d in reversed(dims))
    rows, cells, track = _fiber_surface(f[0][cut], f[1][cut], dims)
    assert np.array_equal(r.simplices, rows)
    assert np.array_equal(r.cells, cells)
    assert np.array_equal(r.track_id, track)
    assert r.n_tracks == len(set(track.tolist()))
