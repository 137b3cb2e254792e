"""The treelet traversal (aurora_gb300/csrc/aur_wide.cuh) on the CPU against
the oracle's walk of intersect() / intersectAny(): the header the kernels
compile is built for the host (tests/wide_model.cpp) and traced over NMHs the
oracle builds. Closest hits (t, u, v, prim id), the first occluder and the
occluded flag must be equal bit for bit, over every shape of the heap's bottom
levels and the inputs that stress a box or slab test."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
from aurora_gb300 import scenes, types as T

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("wide") / "wide_model.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-fno-fast-math", "-std=c++17", "-shared", "-fPIC",
                           "-Wno-attributes", "-I" + cuda + "/include", "-o", so,
                           os.path.join(HERE, "wide_model.cpp")])
    lib = ctypes.CDLL(so)
    lib.wide_model_create.restype = ctypes.c_void_p
    lib.wide_model_create.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32]
    lib.wide_model_destroy.argtypes = [ctypes.c_void_p]
    lib.wide_model_trace.restype = ctypes.c_long
    lib.wide_model_trace.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_int] + [ctypes.c_void_p] * 3
    return lib


def _rays(o, d, tmax=1.0e6):
    r = np.zeros(len(o), T.ray_dtype)
    r["ox"], r["oy"], r["oz"] = np.asarray(o, np.float32).T
    r["dx"], r["dy"], r["dz"] = np.asarray(d, np.float32).T
    r["tmax"] = tmax
    return r


def _random_rays(n, seed, tmax=1.0e6):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    return _rays(rng.random((n, 3)), d / np.linalg.norm(d, axis=1, keepdims=True), tmax)


def _check(lib, V, rays):
    V = oracle.pad_even(np.ascontiguousarray(V, np.float32).reshape(-1, 9))
    perm, _ = oracle.nmh_build(V)
    verts = oracle.gather9(V, perm)
    n = len(rays)
    ohits, _, _ = oracle.trace_closest(verts, perm, rays)
    oocc, _, _ = oracle.trace_any(verts, perm, rays)
    rays = np.ascontiguousarray(rays)
    verts = np.ascontiguousarray(verts, np.float32)
    perm = np.ascontiguousarray(perm, np.uint32)
    m = lib.wide_model_create(verts.ctypes.data, perm.ctypes.data, len(perm))
    tuv, prim, steps = np.zeros((n, 3), np.float32), np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    changed = []
    try:
        for mode in range(5 if len(perm) <= 64 else 3):
            changed.append(lib.wide_model_trace(m, rays.ctypes.data, n, mode, tuv.ctypes.data, prim.ctypes.data,
                                                steps.ctypes.data))
            assert changed[-1] >= 0, "the traversal does not end"
            if mode in (0, 3):
                assert np.array_equal(prim, ohits["prim"])
                for q, f in enumerate("tuv"):
                    assert np.array_equal(tuv[:, q].view(np.uint32), ohits[f].view(np.uint32)), f
            elif mode in (1, 4):
                assert np.array_equal(prim, (oocc != T.NO_HIT).astype(np.uint32))
            else:
                assert np.array_equal(prim, oocc)
    finally:
        lib.wide_model_destroy(m)
    return ohits, changed


@pytest.mark.parametrize("n_tris", [1, 2, 3, 4, 5, 6, 7, 9, 12, 13, 14, 15, 16, 27, 30, 31, 62, 63, 100, 126, 128, 253,
                                    1000, 4099, 20000])
def test_every_heap_shape(model, n_tris):
    V = scenes.random_soup(n_tris, seed=n_tris) if n_tris > 4000 else None
    if V is None:
        rng = np.random.default_rng(n_tris)
        c = rng.random((n_tris, 3, 1))
        V = (c + rng.normal(size=(n_tris, 3, 3)) * 0.2).astype(np.float32).reshape(-1, 9)
    hits, _ = _check(model, V, _random_rays(3000, n_tris))
    assert n_tris < 4 or (hits["prim"] != T.NO_HIT).any()


def test_ties_and_short_rays(model):
    V = scenes.random_soup(3000, seed=5)
    V[2000:2100] = V[100:200]           # coincident copies: equal t
    V[2100:2200] = V[100:200]
    c = np.stack([V[100:200, 0:3].mean(1), V[100:200, 3:6].mean(1), V[100:200, 6:9].mean(1)], 1)
    rng = np.random.default_rng(0)
    o = np.repeat(c, 20, axis=0) + rng.normal(size=(2000, 3)) * 0.1
    d = np.repeat(c, 20, axis=0) - o
    length = np.linalg.norm(d, axis=1)
    for scale in (1.0e6, 1.0, 0.999999, 0.5):    # past, at, just short of and well short of the copies
        _check(model, V, _rays(o, d / length[:, None], 1.0e6 if scale == 1.0e6 else length * scale))


def test_axis_aligned_walls(model):
    """The Cornell box: flat triangles on slab planes, rays through shared
    edges and corners, axis-parallel rays with +0 and -0 components."""
    sd = scenes.cornell()
    V = sd.vertices.reshape(-1, 9)
    P = np.concatenate([V[:, 0:3], V[:, 3:6], V[:, 6:9]], 0).reshape(3, -1, 3).transpose(1, 2, 0).reshape(-1, 3)
    rng = np.random.default_rng(1)
    o = rng.uniform(P.min(0), P.max(0), (4000, 3)).astype(np.float32)
    aim = P[rng.integers(0, len(P), 4000)]
    mid = 0.5 * (aim + P[rng.integers(0, len(P), 4000)])
    for target in (aim, mid, rng.uniform(P.min(0), P.max(0), (4000, 3))):
        d = target - o
        _check(model, V, _rays(o, d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-6)))
    d = np.zeros((4000, 3), np.float32)
    d[np.arange(4000), rng.integers(0, 3, 4000)] = rng.choice([-1.0, 1.0], 4000)
    d[d == 0] = np.where(rng.random((d == 0).sum()) < 0.5, 0.0, -0.0)
    _check(model, V, _rays(o, d))
    on = P[rng.integers(0, len(P), 4000)].copy()      # starting in the walls' planes
    on[:, 0] = o[:, 0]
    _check(model, V, _rays(on, d))


def test_lattice_planes(model):
    rng = np.random.default_rng(3)
    n = 4000
    c = rng.integers(0, 32, size=(n, 3)).astype(np.float32) / 32.0
    e = rng.integers(1, 4, size=(n, 2)).astype(np.float32) / 128.0
    flat = rng.integers(0, 3, size=n)
    V = np.zeros((n, 3, 3), np.float32)
    for k in range(n):
        a, b = [x for x in range(3) if x != flat[k]]
        p = np.tile(c[k], (3, 1))
        p[1, a] += e[k, 0]
        p[2, b] += e[k, 1]
        if rng.random() < 0.5:
            p[[1, 2]] = p[[2, 1]]
        V[k] = p.T
    o = rng.integers(0, 64, size=(4000, 3)).astype(np.float32) / 64.0
    t = rng.integers(0, 64, size=(4000, 3)).astype(np.float32) / 64.0
    d = t - o
    d[np.all(d == 0, axis=1)] = (1.0, 0.0, 0.0)
    _check(model, V.reshape(-1, 9), _rays(o, d))
    _check(model, V.reshape(-1, 9), _rays(o, d / np.linalg.norm(d, axis=1, keepdims=True)))


@pytest.mark.parametrize("n_tris", [2, 33, 64])
@pytest.mark.parametrize("scale,shift", [(1.0, 0.0), (1.0, 1000.0), (1e-4, 0.0), (1e4, -3e5), (1e13, 0.0), (1e18, 1e19)])
def test_few_triangles_over_coordinate_ranges(model, n_tris, scale, shift):
    """Edges, vertices and grazing rays of a few triangles: the filter in front
    of the exact tests keeps every triangle they accept."""
    rng = np.random.default_rng(n_tris)
    V = (rng.random((n_tris, 3, 1)) + rng.normal(size=(n_tris, 3, 3)) * 0.3) * scale + shift
    V = V.astype(np.float32)
    P = V[rng.integers(0, n_tris, 3000)].astype(np.float64)      # triangle, axis, corner
    a, b = rng.random((2, 3000))
    a[:1000] = np.round(a[:1000])                                  # on edges and vertices
    b = b * (1 - a)
    target = P[:, :, 0] + a[:, None] * (P[:, :, 1] - P[:, :, 0]) + b[:, None] * (P[:, :, 2] - P[:, :, 0])
    o = target + rng.normal(size=(3000, 3)) * scale * rng.choice([1e-3, 1.0, 100.0], (3000, 1))
    e = P[:, :, 1] - P[:, :, 0]
    o[2000:] = target[2000:] - e[2000:] + 1e-4 * (o[2000:] - target[2000:])
    d = target - o
    _check(model, V.reshape(-1, 9), _rays(o, d / np.linalg.norm(d, axis=1, keepdims=True), 1.0e30))


@pytest.mark.parametrize("scale,shift", [(1.0, 1000.0), (1e-3, 0.0), (1e4, -3e4), (1e-6, 1.0), (1e18, 0.0)])
def test_coordinate_ranges(model, scale, shift):
    V = scenes.random_soup(3000, seed=6) * np.float32(scale) + np.float32(shift)
    r = _random_rays(2000, 7)
    for f in ("ox", "oy", "oz"):
        r[f] = r[f] * np.float32(scale) + np.float32(shift)
    _check(model, V, r)


def test_float_range_and_non_finite_rays(model):
    """Coordinates whose extent overflows, and rays with NaN, infinite, zero
    or tiny components."""
    rng = np.random.default_rng(8)
    V = (rng.uniform(-3.2e38, 3.2e38, (64, 9))).astype(np.float32)
    _check(model, V, _random_rays(200, 1))
    V = scenes.random_soup(500, seed=8)
    r = _random_rays(1200, 9)
    fields = ("ox", "oy", "oz", "dx", "dy", "dz", "tmax")
    values = (np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-38, 1e-42, 1e30)
    for j in range(0, 1200, 2):
        r[fields[j // 2 % 7]][j] = values[j // 14 % 8]
    _check(model, V, r)
