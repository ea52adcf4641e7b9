"""Which rays the ray queries trace over the wide BVH (pt_scene.cuh wide_ray), compiled for the host by
tests/native/host_queries.cu: every ray it admits must find over the wide BVH what it finds over the
BVH2, bit for bit -- small scenes far from the world's origin, directions from unit length down to 1e-12
and up to 1e12, components that are zero or far below the others, origins at the world's origin, near
the scene and beyond it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle_ctypes as oc

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "open_rendering_framework_b200", "csrc")
SO = os.path.join(HERE, "native", "_build", "libhost_queries.so")
SRC = [os.path.join(HERE, "native", "host_queries.cu"), os.path.join(CSRC, "pt_bvh.cu")]
HDR = [os.path.join(CSRC, f) for f in ("pt_scene.cuh", "pt_math.cuh", "pt_bvh.h")]


@pytest.fixture(scope="module")
def lib():
    newest = max(os.path.getmtime(p) for p in SRC + HDR)
    if not os.path.exists(SO) or os.path.getmtime(SO) < newest:
        os.makedirs(os.path.dirname(SO), exist_ok=True)
        subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "--fmad=false", "-Wno-deprecated-gpu-targets",
                        "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off", "-shared"] + SRC + ["-o", SO], check=True)
    L = ctypes.CDLL(SO)
    L.hq_build.restype = ctypes.c_void_p
    L.hq_build.argtypes = [ctypes.c_void_p, ctypes.c_uint]
    L.hq_free.argtypes = [ctypes.c_void_p]
    L.hq_bary_at.restype = ctypes.c_ulonglong
    L.hq_bary_at.argtypes = [ctypes.c_uint]
    L.hq_rays_per_warp.restype = ctypes.c_uint
    L.hq_rays_per_warp.argtypes = [ctypes.c_uint, ctypes.c_uint]
    L.hq_trace.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long] + [ctypes.c_void_p] * 7
    return L


def trace(lib, tp, rays):
    n = len(rays)
    h = lib.hq_build(oc.fp(tp), len(tp))
    assert h
    out = [np.empty(n, t) for t in (np.int32, np.int32, np.float32, np.int32, np.int32, np.float32, np.int32)]
    lib.hq_trace(h, oc.fp(rays), n, *[oc.fp(a) for a in out])
    lib.hq_free(h)
    return out


def soup(rng, n, half, center):
    """n random triangles of about a fifth of the scene's size around `center`, and two making a wall."""
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    p = c + 0.2 * rng.uniform(-1.0, 1.0, (n, 3, 3))
    p[0] = [(0, -1, -1), (0, 1, -1), (0, 1, 1)]
    p[1] = [(0, -1, -1), (0, 1, 1), (0, -1, 1)]
    return np.ascontiguousarray((p * half + np.asarray(center)).reshape(n, 9), np.float32)


def agree(out):
    wide, p, t, a, p2, t2, a2 = out
    bad = np.flatnonzero((p != p2) | (t.view(np.uint32) != t2.view(np.uint32)) | (a != a2))
    return bad


@pytest.mark.parametrize("half", [1e-3, 1e-5, 1e-6])
def test_small_wall_far_from_the_origin_with_short_directions(lib, half):
    """A wall at x = 1000 seen along directions of length 1e-9 with zero components: the hits lie at t = 1e12,
    beyond what the wide BVH's box tests cover for a zero component."""
    rng = np.random.default_rng(3)
    tp = soup(rng, 2, half, (1000.0, 0.0, 0.0))
    n = 20_000
    rays = np.zeros((n, 8), np.float32)
    rays[:, 1:3] = rng.uniform(-half, half, (n, 2))
    rays[:, 4] = 1e-9
    rays[:, 7] = 1e27
    out = trace(lib, tp, rays)
    assert (out[4] >= 0).mean() > 0.99  # the BVH2 finds the wall
    assert agree(out).size == 0


@pytest.mark.parametrize("offset", [0.0, 1.0, 30.0, 1e3, 3e4])
@pytest.mark.parametrize("half", [1e-4, 1e-2, 1.0, 50.0])
def test_admitted_rays_find_the_same_over_both_trees(lib, half, offset):
    rng = np.random.default_rng(int(offset) % 1000 + int(half * 1e4) % 997)
    total_wide, total = 0, 0
    for axis in range(3):
        center = np.zeros(3)
        center[axis] = offset
        tp = soup(rng, 60, half, center)
        n = 8000
        target = tp.reshape(-1, 3, 3)[rng.integers(0, len(tp), n)]
        target = (target * rng.dirichlet([1.0, 1.0, 1.0], n)[:, :, None]).sum(axis=1)
        kind = rng.integers(0, 4, n)
        o = np.where((kind == 0)[:, None], rng.uniform(-half, half, (n, 3)),                          # about the world's origin
                     np.where((kind == 1)[:, None], center + rng.uniform(-1, 1, (n, 3)) * 3 * half,   # near the scene
                              center + rng.normal(size=(n, 3)) * (offset + half)))                    # beyond it
        zero = rng.integers(0, 4, n)                   # a component exactly zero: the origin takes the target's coordinate
        o = o.astype(np.float32)
        target = target.astype(np.float32)
        for k in range(3):
            o[zero == k, k] = target[zero == k, k]
        d = target.astype(np.float64) - o
        d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-300)
        d *= 10.0 ** rng.uniform(-12.0, 12.0, (n, 1)) * np.where(rng.random((n, 1)) < 0.3, 0.0, 1.0) + np.where(rng.random((n, 1)) < 0.3, 1.0, 0.0)
        small = rng.random(n) < 0.2                    # a component far below the others
        d[small, rng.integers(0, 3)] *= 1e-20
        rays = np.concatenate([o, np.zeros((n, 1)), d, np.full((n, 1), 1e27)], 1).astype(np.float32)
        out = trace(lib, tp, np.ascontiguousarray(rays))
        total_wide += int(out[0].sum())
        total += n
        bad = agree(out)
        assert bad.size == 0, (bad.size, rays[bad[0]])
    # ordinary rays keep the wide BVH: all but those of tiny directions
    assert total_wide > 0.6 * total or offset > 30.0 * half


def test_every_unit_direction_near_an_ordinary_scene_is_admitted(lib):
    rng = np.random.default_rng(9)
    tp = soup(rng, 40, 1.0, (0.0, 0.0, 0.0))
    n = 4000
    d = rng.normal(size=(n, 3))
    d[: n // 2, 0] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([rng.uniform(-100, 100, (n, 3)), np.full((n, 1), 1e-4), d, np.full((n, 1), 1e27)], 1).astype(np.float32)
    assert trace(lib, tp, np.ascontiguousarray(rays))[0].all()


@pytest.mark.parametrize("i", [0, 1, 2 ** 31 - 1, 2 ** 31, 2 ** 32 - 1])
def test_query_indexes_hold_for_every_ray_count(lib, i):
    """Ray i's barycentrics lie at 2 i and the warps' runs cover all of n = i rays, past 2^31 too."""
    assert lib.hq_bary_at(i) == 2 * i
    for warps in (32, 4736):
        per = lib.hq_rays_per_warp(i, warps)
        assert per == max(32, -(-i // warps)) and per * warps >= i
