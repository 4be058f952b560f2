"""Performance cases: the feature extractions a program asks this library for.

A case is a dict of plain values; ``prepare`` makes its seeded inputs and the
handles a program keeps (context, mesh, predicate), ``run`` is one call through
the public Python API with the whole result on the host, ``exact`` recomputes
the barycentrics with plain torch in 64 bits.

kinds: "cp" (critical points of one field, regular mesh), "batch" (many fields
of uneven sizes in one call), "stream" (regular mesh pushed one timestep at a
time), "extruded" (tet mesh over a jittered plane, one call or a stream),
"contour" (level set), "fiber" (2D+t points or 3D+t surfaces of two scalars).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ftk2_b200 import api, generate, synthetic

Q = 2.0 ** 20  # lattice scale of every case


# ---------------------------------------------------------------------------
# cases


def listed():
    return [
        # the smallest call: the 64 x 64 x 10 double field of the 2D examples,
        # device-resident, where launches and host work count
        dict(name="cp2d_small", kind="cp", dims="64,64", nt=10, f64=True, separate=False, scalar=False,
             classify=False, refined=False, host=False, blobs=24, lo=4.0, hi=12.0, scale=1.0, noise=0.0),
        # a 2D simulation's separate component arrays of odd sizes, with the
        # scalar interpolated at the points and their types classified
        dict(name="cp2d_separate_typed", kind="cp", dims="1021,765", nt=12, f64=False, separate=True, scalar=True,
             classify=True, refined=False, host=False, blobs=48, lo=8.0, hi=64.0, scale=1.0, noise=0.0),
        # the headline 3D flow workload: 128^3 x 16 double
        dict(name="cp3d_f64", kind="cp", dims="128,128,128", nt=16, f64=True, separate=False, scalar=False,
             classify=False, refined=False, host=False, blobs=32, lo=4.0, hi=12.0, scale=1.0, noise=0.0),
        # the largest: 256^3 x 8 float with measurement noise, refined positions
        dict(name="cp3d_noise_refined", kind="cp", dims="256,256,256", nt=8, f64=False, separate=False, scalar=False,
             classify=False, refined=True, host=False, blobs=64, lo=16.0, hi=48.0, scale=256.0, noise=1e-3),
        # a served request: a two-timestep 3D slab of odd sizes from pinned host memory
        dict(name="cp3d_slab_host", kind="cp", dims="121,97,83", nt=2, f64=False, separate=False, scalar=False,
             classify=False, refined=False, host=True, blobs=32, lo=4.0, hi=16.0, scale=1.0, noise=0.0),
        # 256 independent 2D and 3D fields of uneven sizes in one call
        dict(name="batch_256", kind="batch", n=256, spec=2024, f64=False),
        # an in-situ run: one timestep at a time, tracks so far at the end
        dict(name="stream3d", kind="stream", dims="96,101,88", nt=8, f64=False, separate=False, scalar=False,
             classify=False, refined=False, host=False, blobs=32, lo=4.0, hi=12.0, scale=1.0, noise=0.0),
        # the served unstructured stream: 100 x 100 plane x 40 layers of tets, 16 timesteps
        dict(name="extruded_stream", kind="extruded", nx=100, ny=100, layers=40, nt=16, f64=False, stream=True,
             blobs=48, lo=3.0, hi=9.0),
        # a one-shot extraction on a smaller unstructured tet mesh, double
        dict(name="extruded_once", kind="extruded", nx=61, ny=47, layers=23, nt=5, f64=True, stream=False,
             blobs=24, lo=3.0, hi=9.0),
        # a moving iso-surface of a 3D scalar
        dict(name="contour3d", kind="contour", dims="96,96,96", nt=6, f64=True, threshold=0.125, blobs=32,
             lo=4.0, hi=12.0),
        # points where two 2D scalars meet their thresholds, float, odd sizes
        dict(name="fiber2d", kind="fiber", dims="401,323", nt=16, f64=False, threshold=0.0625, blobs=32, lo=8.0,
             hi=24.0),
        # fiber surfaces of two 3D scalars, 96^3 x 8 double
        dict(name="fiber3d", kind="fiber", dims="96,96,96", nt=8, f64=True, threshold=0.0, blobs=32, lo=4.0, hi=12.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, d, lo, hi, nt, most):
    """d log-uniform sides whose product with nt is at most ``most``."""
    s = [_log(rng, lo, hi) for _ in range(d)]
    while math.prod(s) * nt > most:
        k = s.index(max(s))
        s[k] = max(lo, s[k] * 4 // 5)
    return ",".join(map(str, s))


def draw(rng):
    kind = rng.choice(["cp", "cp", "cp", "batch", "stream", "extruded", "contour", "fiber"])
    d = rng.choice([2, 3])
    f64 = rng.random() < 0.5
    blobs = rng.randint(8, 64)
    if kind in ("cp", "stream"):
        nt = rng.randint(2, 16)
        host = kind == "cp" and rng.random() < 0.25
        separate = rng.random() < 0.4
        noisy = d == 3 and rng.random() < 0.25
        most = 4_000_000 if host else 8_000_000 if kind == "stream" else 32_000_000
        return dict(kind=kind, dims=_sides(rng, d, 32 if d == 2 else 16, 2048 if d == 2 else 256, nt, most), nt=nt,
                    f64=f64, separate=separate, scalar=separate and kind == "cp" and rng.random() < 0.5,
                    classify=rng.random() < 0.25, refined=not f64 and rng.random() < 0.5, host=host, blobs=blobs,
                    lo=16.0 if noisy else 4.0, hi=48.0 if noisy else 16.0, scale=256.0 if noisy else 1.0,
                    noise=1e-3 if noisy else 0.0)
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 4, 128), spec=rng.randint(1, 9999), f64=f64)
    if kind == "extruded":
        return dict(kind=kind, nx=_log(rng, 16, 100), ny=_log(rng, 16, 100), layers=_log(rng, 4, 40),
                    nt=rng.randint(2, 12), f64=f64, stream=rng.random() < 0.5, blobs=blobs, lo=3.0, hi=9.0)
    nt = rng.randint(2, 16)
    threshold = rng.choice([0.0, 0.0625, 0.125, 0.25])
    most = 5_000_000 if kind == "contour" else 6_000_000
    return dict(kind=kind, dims=_sides(rng, d, 24 if d == 2 else 12, 512 if d == 2 else 128, nt, most), nt=nt, f64=f64,
                threshold=threshold, blobs=blobs, lo=4.0, hi=16.0)


# ---------------------------------------------------------------------------
# inputs


def _dims(case):
    return tuple(int(v) for v in case["dims"].split(","))


def _dtype(case):
    return torch.float64 if case["f64"] else torch.float32


def _inputs(case, seed):
    """The case's arrays on the GPU, from the seed alone (batches: a list of
    (mesh dims, components, array); extruded: (components, nt, vertices))."""
    kind = case["kind"]
    if kind == "batch":
        out = []
        for i, (dims, nt, nb, _) in enumerate(generate.batch_specs(case["n"], case["spec"])):
            f = generate.gaussian_field_fast(dims, nt, seed * 1009 + i, nb, dtype=_dtype(case))
            out.append((list(dims) + [nt], len(dims), f))
        return out
    if kind == "extruded":
        coords, _ = _plane(case)
        v = generate.gaussian_at_device(coords, case["nt"], seed=seed, n_blobs=case["blobs"], dtype=_dtype(case),
                                        sigma=(case["lo"], case["hi"]), drift=0.8)
        return v.view(3, case["nt"], -1)
    sigma = (case["lo"], case["hi"])
    if kind in ("contour", "fiber"):
        n = 1 if kind == "contour" else 2
        return [generate.gaussian_potential_device(_dims(case), case["nt"], seed=seed * 2 + k, n_blobs=case["blobs"],
                                                   sigma=sigma).to(_dtype(case)) for k in range(n)]
    f = generate.gaussian_field_device(_dims(case), case["nt"], seed=seed, n_blobs=case["blobs"], dtype=_dtype(case),
                                       sigma=sigma, scale=case["scale"], noise=case["noise"])
    if not case["separate"]:
        return [f]
    arrays = [f[..., j].contiguous() for j in range(len(_dims(case)))]
    if case["scalar"]:
        arrays.append(generate.gaussian_potential_device(_dims(case), case["nt"], seed=seed, n_blobs=case["blobs"],
                                                         sigma=sigma).to(_dtype(case)))
    return arrays


def _plane(case):
    return synthetic.extruded_tet_mesh(case["nx"], case["ny"], case["layers"])


def _threshold(case):
    return float(case["threshold"])


def prepare(case, seed):
    kind = case["kind"]
    data = _inputs(case, seed)
    ctx = api.Context(0)
    s = dict(case=case, ctx=ctx, keep=[data])
    keep = s["keep"]
    if kind == "batch":
        s["meshes"] = [api.regular_mesh_desc(d) for d, _, _ in data]
        s["fields"] = [api.field_desc(f, api.LAYOUT_MULTICOMPONENT, m, keep=keep) for _, m, f in data]
        s["params"] = [api.params(Q) for _ in data]
        return s
    if kind == "extruded":
        coords, cells = _plane(case)
        if case["stream"]:
            s["mesh"] = api.extruded_mesh_desc(coords.shape[0], cells, 1, keep)
            s["steps"] = [api.field_desc([data[j, t] for j in range(3)], api.LAYOUT_PER_VERTEX, 3, keep=keep)
                          for t in range(case["nt"])]
            return s
        base = api.UnstructuredSimplicialMesh(3, 3, coords, cells)
        pred = api.CriticalPointPredicate(3, var_names=["u", "v", "w"], use_multicomponent=False, sos_q=Q)
        s["engine"] = api.SimplicialEngine(api.ExtrudedSimplicialMesh(base, case["nt"] - 1), pred, ctx)
        s["data"] = {n: data[j].reshape(-1) for j, n in enumerate("uvw")}
        return s
    dims = _dims(case)
    m = len(dims)
    if kind == "stream":
        layout = api.LAYOUT_SEPARATE if case["separate"] else api.LAYOUT_MULTICOMPONENT
        s["mesh"] = api.regular_mesh_desc([*dims, 1])
        s["prm"] = api.params(Q, precision=api.PRECISION_REFINED if case["refined"] else api.PRECISION_EXACT,
                              classify=case["classify"])
        s["steps"] = []
        for t in range(case["nt"]):
            a = [x[t] for x in data]
            s["steps"].append(api.field_desc(a if case["separate"] else a[0], layout, m, keep=keep))
        return s
    mesh = api.RegularSimplicialMesh([*dims, case["nt"]])
    if kind == "contour":
        pred = api.ContourPredicate("s", _threshold(case), Q)
        s["data"] = {"s": data[0]}
    elif kind == "fiber":
        pred = api.FiberPredicate(["a", "b"], (_threshold(case), _threshold(case)), Q)
        s["data"] = {"a": data[0], "b": data[1]}
    else:
        if case["host"]:  # pinned host arrays, as a program that feeds a GPU keeps them
            keep.append([x.cpu().pin_memory() for x in data])
            keep.pop(0)
            data = [x.numpy() for x in keep[0]]
        more = dict(sos_q=Q, precision=api.PRECISION_REFINED if case["refined"] else api.PRECISION_EXACT,
                    classify=case["classify"])
        if case["separate"]:
            names = ["u", "v", "w"][:m]
            pred = api.CriticalPointPredicate(m, var_names=names, use_multicomponent=False,
                                              scalar_var_name="s" if case["scalar"] else "", **more)
            s["data"] = dict(zip(names + ["s"], data))
        else:
            pred = api.CriticalPointPredicate(m, vector_var_name="v", **more)
            s["data"] = {"v": data[0]}
    s["engine"] = api.SimplicialEngine(mesh, pred, ctx)
    return s


# ---------------------------------------------------------------------------
# one pass

CP_FIELDS = ("simplices", "lam", "bary", "track_id", "type", "cp_class", "scalar", "edges", "n_tracks")
LEVEL_FIELDS = ("simplices", "lam", "bary", "track_id", "scalar", "cells", "n_tracks")


def _rows(case):
    """More features (and edges or cells, by a factor) than any seed's fields
    of this case give."""
    if case["kind"] == "batch":
        return 4096 * case["n"]
    if case["kind"] == "extruded":
        return 1 << 16
    nv = math.prod(_dims(case)) * case["nt"]
    if case["kind"] in ("contour", "fiber"):
        return max(1 << 14, nv if case["kind"] == "contour" else nv // 4)
    return max(1 << 14, min(nv // 8, 1 << 18))


def _pad(a, rows):
    """a with zero rows up to ``rows`` (how many features a field holds
    depends on the seed, and outputs are compared shape by shape)."""
    if len(a) > rows:
        raise ValueError(f"{len(a)} rows, room for {rows}")
    if isinstance(a, torch.Tensor):
        return torch.cat([a, a.new_zeros((rows - len(a),) + tuple(a.shape[1:]))])
    out = np.zeros((rows,) + a.shape[1:], a.dtype)
    out[:len(a)] = a
    return out


class Out(dict):
    """A pass's result arrays, whole; one is padded when it is read, so that
    no pass pays for it."""

    def __init__(self, case, arrays):
        super().__init__(arrays)
        self.case = case

    def __getitem__(self, name):
        a = super().__getitem__(name)
        if isinstance(a, int) or name == "counts":
            return a
        n = _rows(self.case)
        if self.case["kind"] == "batch":  # raveled rows of up to four values
            n *= 4
        return _pad(a, n * {"cells": 7, "edges": 2}.get(name, 1))


def _out(case, r):
    names = LEVEL_FIELDS if isinstance(r, api.ContourResult) else CP_FIELDS
    out = {n: getattr(r, n) for n in names}
    out["n"] = len(r.track_id)
    return Out(case, out)


def run(s):
    if "engine" in s:
        s["engine"].execute(s["data"])
        return _out(s["case"], s["engine"].get_complex())
    if "steps" in s:
        with api.Stream(s["ctx"], s["mesh"], s["steps"][0], s.get("prm") or api.params(Q)) as stream:
            for f in s["steps"]:
                stream.push(f)
            return _out(s["case"], stream.result())
    every = s["ctx"].extract_batch(s["meshes"], s["fields"], s["params"])
    out = {n: np.concatenate([getattr(r, n).ravel() for r in every]) for n in CP_FIELDS[:-1]}
    out["counts"] = np.array([(len(r.track_id), len(r.edges), r.n_tracks) for r in every])
    return Out(s["case"], out)


# ---------------------------------------------------------------------------
# work: the input read once; level sets, whose results are of the input's
# order, with the results the generator's fields give per vertex, written once


def work(case):
    es = 8 if case["f64"] else 4
    if case["kind"] == "batch":
        n = sum(math.prod(d) * nt * len(d) for d, nt, _, _ in generate.batch_specs(case["n"], case["spec"]))
        return {"bytes": n * es, "flops": 0}
    if case["kind"] == "extruded":
        return {"bytes": case["nx"] * case["ny"] * case["layers"] * case["nt"] * 3 * es, "flops": 0}
    d = _dims(case)
    nv = math.prod(d) * case["nt"]
    if case["kind"] == "contour":
        # a crossing edge is 52 bytes (ids, barycentrics, track, value), a cell
        # 4 bytes a vertex
        feat = 0.25
        cells = feat * (5.7 if len(d) == 3 else 2)
        return {"bytes": int(nv * (es + feat * 52 + cells * 4 * (len(d) + 1))), "flops": 0}
    if case["kind"] == "fiber":
        return {"bytes": nv * 2 * es, "flops": 0}
    return {"bytes": nv * es * (len(d) + (1 if case["scalar"] else 0)), "flops": 0}


# ---------------------------------------------------------------------------
# the same barycentrics in 64 bits, with plain torch


def _chains(d, m):
    """Corner masks 0 < k1 < .. < km of every m-simplex of the Kuhn d-cube."""
    out = [(0,)]
    for _ in range(m):
        out = [c + (k,) for c in out for k in range(c[-1] + 1, 1 << d) if k & c[-1] == c[-1]]
    return out


def _rows_regular(word, dims, m):
    """Vertex ids (n, m + 1) of the grid's m-simplices over whose vertices no
    bit of ``word`` survives (word: shaped as the reversed dims)."""
    d = len(dims)
    ids = torch.arange(word.numel(), device=word.device).view(word.shape)
    rows = []
    for c in _chains(d, m):
        def corner(a, k):
            """The view of a at corner k of every hypercube holding the chain."""
            cut = [slice((k >> x) & 1, dims[x] - ((c[-1] >> x) & 1) + ((k >> x) & 1)) for x in range(d)]
            return a[tuple(reversed(cut))]
        w = corner(word, 0)
        for k in c[1:]:
            w = w & corner(word, k)
        pick = (w == 0).nonzero(as_tuple=True)
        rows.append(torch.stack([corner(ids, k)[pick] for k in c], 1))
    return torch.cat(rows)


def _sorted_rows(rows):
    for k in reversed(range(rows.shape[1])):
        rows = rows[torch.argsort(rows[:, k], stable=True)]
    return rows


def _signs(v):
    """Strict sign bits of every component, (n, M) -> (n,) uint8."""
    w = torch.zeros(v.shape[0], dtype=torch.uint8, device=v.device)
    for j in range(v.shape[1]):
        w |= (v[:, j] > 0).to(torch.uint8) << j
        w |= (v[:, j] < 0).to(torch.uint8) << (3 + j)
    return w


def _quant(v):
    return (v * Q + torch.where(v > 0, 0.5, -0.5)).to(torch.int64)


def _first_sign(levels):
    """The sign of the first non-zero level, +1 where all are zero."""
    s = torch.zeros_like(levels[0])
    for x in levels:
        s = torch.where(s == 0, torch.sign(x), s)
    return torch.where(s == 0, torch.ones_like(s), s)


def _inside(q):
    """Whether the perturbed origin lies inside the simplex of integer rows
    q (n, M + 1, M): simulation of simplicity, M = 2 or 3."""
    if q.shape[2] == 2:
        s = []
        for a, b, tie in ((0, 1, 1), (1, 2, 1), (2, 0, -1)):
            det = q[:, a, 0] * q[:, b, 1] - q[:, a, 1] * q[:, b, 0]
            s.append(_first_sign([det, torch.full_like(det, tie)]))
        return (s[0] == s[1]) & (s[1] == s[2])
    s = []
    for r in ((1, 3, 2), (0, 2, 3), (0, 3, 1), (0, 1, 2)):
        a, b, c = (q[:, i] for i in r)

        def two(x, y, i, j):
            return x[:, i] * y[:, j] - x[:, j] * y[:, i]

        def det(a, bc):
            return a[:, 0] * bc[0] - a[:, 1] * bc[1] + a[:, 2] * bc[2]
        bc = [two(b, c, 1, 2), two(b, c, 0, 2), two(b, c, 0, 1)]
        whole = det(a, bc)  # exact modulo 2^64
        near = det(a.double(), [x.double() for x in bc])
        whole = torch.where(near.abs() < 2.0 ** 62, whole, torch.sign(near).to(torch.int64))
        s.append(_first_sign([whole, bc[2], -bc[1], bc[0], -two(a, c, 0, 1), c[:, 0], -c[:, 1], two(a, c, 0, 2),
                              c[:, 2], -two(a, c, 1, 2), two(a, b, 0, 1), -b[:, 0], b[:, 1], a[:, 0]]))
    return (s[0] == s[1]) & (s[1] == s[2]) & (s[2] == s[3])


def _solve(v):
    """Barycentrics of the origin in the simplices v (n, M + 1, M), and where
    they exist and lie in [0, 1] to rounding."""
    n, m = v.shape[0], v.shape[2]
    a = (v[:, :m] - v[:, m:]).transpose(1, 2).clone()
    x = -v[:, m].clone()
    ok = torch.ones(n, dtype=torch.bool, device=v.device)
    row = torch.arange(n, device=v.device)
    for i in range(m):
        p = a[:, i:, i].abs().argmax(1) + i
        for t in (a, x):
            t[row, p], t[:, i] = t[:, i].clone(), t[row, p].clone()
        ok &= a[:, i, i].abs() >= 1e-12
        for j in range(i + 1, m):
            f = a[:, j, i] / a[:, i, i]
            a[:, j] -= f[:, None] * a[:, i]
            x[:, j] -= f * x[:, i]
    for i in reversed(range(m)):
        x[:, i] = (x[:, i] - (a[:, i, i + 1:] * x[:, i + 1:]).sum(1)) / a[:, i, i]
    lam = torch.cat([x, 1 - x.sum(1, keepdim=True)], 1)
    ok &= ((lam >= -1e-9) & (lam <= 1 + 1e-9)).all(1)
    return lam, ok


def _points(rows, v, centroid):
    """Sorted feature rows and their barycentrics."""
    lam, ok = _solve(v[rows])
    keep = _inside(_quant(v[rows]))
    if centroid:
        lam = torch.where(ok[:, None], lam, 1.0 / 3.0)
    else:
        keep &= ok
    both = _sorted_rows(torch.cat([rows, torch.arange(rows.shape[0], device=rows.device)[:, None]], 1)[keep])
    return both[:, :-1], lam[both[:, -1]]


def _exact_cp(f, dims):
    """One multicomponent field f of (mesh) dims incl. time."""
    m = len(dims) - 1
    v = f.double().reshape(-1, m)
    rows = _rows_regular(_signs(v).view(tuple(dims[::-1])), dims, m)
    return _points(rows, v, False)


def _exact_extruded(case, data):
    _, cells = _plane(case)
    cells = torch.sort(torch.from_numpy(cells.astype(np.int64)).cuda(), 1).values
    nv, nt = data.shape[2], case["nt"]
    v = data.double().reshape(3, -1).T.contiguous()
    w, rows = _signs(v), []
    for t in range(nt):
        for j in range(4):
            if t + 1 == nt:  # the last layer holds spatial simplices only
                top = [cells + t * nv]
                if j:
                    continue
            else:
                five = torch.cat([cells[:, :j + 1], cells[:, j:] + nv], 1) + t * nv
                top = [torch.cat([five[:, :k], five[:, k + 1:]], 1) for k in range(5)]
            for r in top:
                keep = (w[r[:, 0]] & w[r[:, 1]] & w[r[:, 2]] & w[r[:, 3]]) == 0
                rows.append(r[keep])
    return _points(torch.unique(torch.cat(rows), dim=0), v, False)


def _exact_out(case, lam, scalar=None):
    out = Out(case, {"lam": lam, "bary": lam})
    out = {n: out[n] for n in out}
    if scalar is not None:
        out["scalar"] = _pad(scalar, _rows(case))
    return out


def exact(case, seed):
    data = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        got = [_exact_cp(f, dims)[1] for dims, _, f in data]
        lam = torch.cat([x.reshape(-1) for x in got])
        return _exact_out(case, lam)
    if kind == "extruded":
        return _exact_out(case, _exact_extruded(case, data)[1])
    dims = [*_dims(case), case["nt"]]
    thr = case.get("threshold", 0.0)
    if kind == "contour":
        x = data[0].reshape(-1).double() - thr
        q = _quant(x)
        odd = torch.arange(x.numel(), device=x.device) & 1
        pos = torch.where(q != 0, q > 0, odd == 0)
        word = torch.where(pos, 1, 2).to(torch.uint8).view(data[0].shape)
        rows = _sorted_rows(_rows_regular(word, dims, 1))
        v0, v1 = x[rows[:, 0]], x[rows[:, 1]]
        l0 = -v1 / (v0 - v1)
        l0 = torch.where(((v0 - v1).abs() < 1e-12) | (l0 < -1e-9) | (l0 > 1 + 1e-9), 0.5, l0)
        return _exact_out(case, torch.stack([l0, 1 - l0], 1))
    if kind == "fiber":
        v = torch.stack([x.reshape(-1).double() - thr for x in data], 1)
        # ties keep simplices that span quantised zeros: signs of the quantised values
        word = _signs(_quant(v)).view(data[0].shape)
        return _exact_out(case, _points(_rows_regular(word, dims, 2), v, True)[1])
    f = torch.stack(data[:len(dims) - 1], -1) if case["separate"] else data[0]
    rows, lam = _exact_cp(f, dims)
    scalar = (data[-1].reshape(-1).double()[rows] * lam).sum(1) if case["scalar"] else None
    return _exact_out(case, lam, scalar)
