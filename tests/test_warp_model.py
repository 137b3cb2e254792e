"""The traversals a warp runs together (wide_packet, and wide_warp with its
triangle queue: aurora_gb300/csrc/aur_wide.cuh) on the CPU, compiled from the
header the kernels compile with 32 lanes in lockstep (tests/warp_model.cpp),
against the oracle's walk of intersect() / intersectAny(): closest hit, the
first occluder and the occluded flag, bit for bit. The lanes must also meet
every warp intrinsic together, with and without a ray of their own."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
from aurora_gb300 import scenes, types as T
from test_packet_model import _camera_chunks, _octant_chunks
from test_short_directions import _short_rays
from test_wide_model import model  # noqa: F401  (the module's fixture)

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def warp(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("warp") / "warp_model.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-fno-fast-math", "-std=c++17", "-shared", "-fPIC",
                           "-Wno-attributes", "-I" + cuda + "/include", "-o", so, os.path.join(HERE, "warp_model.cpp")])
    lib = ctypes.CDLL(so)
    lib.warp_model_trace.restype = ctypes.c_long
    lib.warp_model_trace.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32] + [ctypes.c_int] * 3 + \
        [ctypes.c_void_p] * 2
    return lib


def _check(model, warp, V, rays, packets):
    V = oracle.pad_even(np.ascontiguousarray(V, np.float32).reshape(-1, 9))
    perm, _ = oracle.nmh_build(V)
    verts = np.ascontiguousarray(oracle.gather9(V, perm), np.float32)
    perm = np.ascontiguousarray(perm, np.uint32)
    rays = np.ascontiguousarray(rays)
    n = len(rays)
    ohits, _, _ = oracle.trace_closest(verts, perm, rays)
    oocc, _, _ = oracle.trace_any(verts, perm, rays)
    m = model.wide_model_create(verts.ctypes.data, perm.ctypes.data, len(perm))
    try:
        for mode in range(3):
            for backwards in range(2):
                tuv, prim = np.zeros((n, 3), np.float32), np.zeros(n, np.uint32)
                apart = warp.warp_model_trace(m, rays.ctypes.data, n, packets, mode, backwards, tuv.ctypes.data,
                                              prim.ctypes.data)
                assert apart == -1, "the lanes of the chunk at ray %d did not stay together" % apart
                if mode == 0:
                    assert np.array_equal(prim, ohits["prim"])
                    for q, f in enumerate("tuv"):
                        assert np.array_equal(tuv[:, q].view(np.uint32), ohits[f].view(np.uint32)), f
                elif mode == 1:
                    assert np.array_equal(prim != T.NO_HIT, oocc != T.NO_HIT)
                else:
                    assert np.array_equal(prim, oocc)
    finally:
        model.wide_model_destroy(m)
    return ohits


def _unit(n, rng):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _random(n, rng, tmax=1.0e6):
    rays = np.zeros(n, T.ray_dtype)
    rays["ox"], rays["oy"], rays["oz"] = rng.random((3, n)).astype(np.float32)
    rays["dx"], rays["dy"], rays["dz"] = _unit(n, rng).astype(np.float32).T
    rays["tmax"] = tmax
    return rays


@pytest.mark.parametrize("n_tris", [1, 2, 3, 7, 8, 63, 300, 5000])
def test_packets_equal_the_walk(model, warp, n_tris):  # noqa: F811
    """Close and spread origins, diverging directions, a camera's rays; the
    last chunk is partial."""
    rng = np.random.default_rng(n_tris)
    V = scenes.random_soup(n_tris, seed=n_tris)
    if n_tris < 1000:      # large enough to be hit
        V = V.reshape(-1, 3, 3)
        V = (V.mean(2, keepdims=True) + (V - V.mean(2, keepdims=True)) * 30.0).reshape(-1, 9)
    rays = np.concatenate([_octant_chunks(rng, 10, 0.004), _octant_chunks(rng, 5, 1.0), _camera_chunks(rng, 6)])[:-13]
    hits = _check(model, warp, V, rays, 1)
    assert n_tris < 8 or (hits["prim"] != T.NO_HIT).any()


@pytest.mark.parametrize("n_tris", [1, 3, 8, 300, 5000])
def test_queue_equals_the_walk(model, warp, n_tris):  # noqa: F811
    rng = np.random.default_rng(n_tris)
    V = scenes.random_soup(n_tris, seed=n_tris).reshape(-1, 3, 3)
    V = (V.mean(2, keepdims=True) + (V - V.mean(2, keepdims=True)) * 20.0).reshape(-1, 9).astype(np.float32)
    rays = _random(32 * 16 - 5, rng)
    rays["tmax"][::5] = 0.2
    _check(model, warp, V, rays, 0)


@pytest.mark.parametrize("packets", [0, 1])
def test_ties_zero_components_and_short_segments(model, warp, packets):  # noqa: F811
    rng = np.random.default_rng(3)
    V = scenes.random_soup(3000, seed=5)
    V[2000:2200] = V[100:300]                       # coincident copies: ties in t
    V[2200:2400] = V[100:300]
    c = np.stack([V[100:132, 0:3].mean(1), V[100:132, 3:6].mean(1), V[100:132, 6:9].mean(1)], 1)
    ax = np.zeros(96, T.ray_dtype)                  # axis-parallel through the copies, +0 and -0 alternating
    for a in range(3):
        s = slice(32 * a, 32 * a + 32)
        o = c.copy()
        o[:, a] -= 2.0
        ax["ox"][s], ax["oy"][s], ax["oz"][s] = o.astype(np.float32).T
        z = np.where(np.arange(32) % 2, -0.0, 0.0).astype(np.float32)
        comps = [z, z, z]
        comps[a] = np.ones(32, np.float32)
        ax["dx"][s], ax["dy"][s], ax["dz"][s] = comps
    ax["tmax"] = 1e6
    ends = _octant_chunks(rng, 4, 0.004)
    ends["tmax"] = rng.random(128).astype(np.float32) * 0.05    # most end before a hit
    _check(model, warp, V, np.concatenate([_octant_chunks(rng, 6, 0.01), ax, ends]), packets)


@pytest.mark.parametrize("packets", [0, 1])
def test_rays_that_hit_nothing_among_others(model, warp, packets):  # noqa: F811
    """Lanes with a NaN, infinite or zero component, no range, or nothing at
    all beside lanes that traverse; chunks of such rays only."""
    rng = np.random.default_rng(9)
    V = scenes.random_soup(500, seed=8).reshape(-1, 3, 3)
    V = (V.mean(2, keepdims=True) + (V - V.mean(2, keepdims=True)) * 10.0).reshape(-1, 9).astype(np.float32)
    rays = _octant_chunks(rng, 12, 0.01)[:-7]
    fields = ("ox", "oy", "oz", "tmax") if packets else ("ox", "oy", "oz", "dx", "dy", "dz", "tmax")
    values = (np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-42, 1e30, 1e-9)
    for j in range(0, 320, 3):
        rays[fields[j // 3 % len(fields)]][j] = values[j // 7 % 8]
    rays["tmax"][320:352] = 0.0
    _check(model, warp, V, rays, packets)


@pytest.mark.parametrize("packets", [0, 1])
@pytest.mark.parametrize("n_tris", [70, 400])
def test_short_directions_among_others(model, warp, n_tris, packets):  # noqa: F811
    """Directions of length 1e-21 to 1e-6 in one chunk."""
    V, rays = _short_rays(n_tris, 1e-13, n_tris)
    rng = np.random.default_rng(n_tris)
    if packets:                     # one octant per chunk
        key = (rays["dx"] < 0) * 1 + (rays["dy"] < 0) * 2 + (rays["dz"] < 0) * 4
        groups = [np.flatnonzero(key == o) for o in range(8)]
        rays = rays[np.concatenate([g[:len(g) // 32 * 32][:64] for g in groups])]
    else:
        rays = rays[rng.permutation(len(rays))[:300]]
    scale = 10.0 ** rng.uniform(-8.0, 7.0, len(rays))
    for f in ("dx", "dy", "dz"):
        rays[f] = (rays[f].astype(np.float64) * scale).astype(np.float32)
    hits = _check(model, warp, V, rays, packets)
    assert (hits["prim"] != T.NO_HIT).any()
