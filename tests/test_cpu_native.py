"""Host code and index arithmetic that the kernels share, compiled alone (g++, no GPU) and driven at
its limits by small programs under tests/native."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from orion_gb300 import build

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    """native(name, *sources): path of tests/native/<name>.cpp compiled with the library's `sources`."""
    out = tmp_path_factory.mktemp("native")

    def compile_one(name, *sources):
        exe = str(out / name)
        if os.path.exists(exe):
            return exe
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", build.CSRC, "-I",
                        os.path.join(build.CUDA_HOME, "include"), os.path.join(NATIVE, name + ".cpp"),
                        *(os.path.join(build.CSRC, s) for s in sources), "-o", exe, "-lpthread", "-ldl"], check=True)
        return exe

    return compile_one


def _run(exe, *args):
    p = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip().endswith("ok"), (p.returncode, p.stdout, p.stderr)


@pytest.mark.parametrize("photons,dealt", [(2**31 - 1, 2**31 - 200_001), (2**31 - 155_000, 2**31 - 160_000),
                                           (100_000, 0), (31, 0)])
def test_photons_near_the_largest_count_are_dealt_once(native, photons, dealt):
    """k_sppm_photons' warps overshoot the last photon by up to 32 each: all of them stop, and each photon
    is started once, up to the largest count that orion_gpu_render_sppm accepts."""
    _run(native("photon_deal"), photons, dealt)


INT32_MAX = 2**31 - 1


@pytest.mark.parametrize("pixels,spp,wave,exact", [
    (740 * 1451, 4000, INT32_MAX, 0),  # a wave rounded up to whole chunks would pass INT32_MAX paths
    (740 * 1451, 4000, INT32_MAX, 1), (2 * 2**27 + 2, 8, INT32_MAX - 7, 0), (1, INT32_MAX, INT32_MAX, 0),
    (1, 7, 3, 1), (33 * 6, 255, 64, 0), (33 * 6, 255, 1000, 1), (1920 * 1080, 128, 1 << 25, 0),
    (1024 * 1024, 64, 1 << 25, 0), (257, 1, 100, 0), (7 * 41, 257, 7 * 41 * 257, 0)])
def test_waves_cover_the_film_within_their_capacity(native, pixels, spp, wave, exact):
    _run(native("wave_plan"), pixels, spp, wave, exact)


@pytest.mark.parametrize("spp", [0, -3])
def test_no_samples_make_no_waves(native, spp):
    _run(native("wave_plan"), 64 * 48, spp, 1, 0)


@pytest.mark.parametrize("width,height", [
    (1, 1), (7, 3), (8, 4), (9, 5), (33, 6), (1, 97), (641, 359), (1 << 28, 3), ((1 << 28) + 1, 7), (1 << 29, 4),
    (1 << 30, 1),  # a tile row of 2^32 pixels
    (1 << 30, 4), (INT32_MAX, 1), (INT32_MAX, 9), (65536, 65536), (3, 1 << 29)])
def test_tile_order_visits_each_pixel_once(native, width, height):
    _run(native("tile_pixel"), width, height)


@pytest.mark.parametrize("kind", ["plain", "pooled"])
def test_allocations_out_of_memory_trim_the_pools_and_retry(native, kind):
    _run(native("device_buffers"), kind, 1, "retried")


@pytest.mark.parametrize("kind", ["plain", "pooled"])
def test_refused_allocations_leave_no_error_behind(native, kind):
    """The autotuners skip a configuration that does not fit; the launches after it must not fail over it."""
    _run(native("device_buffers"), kind, 2, "refused")


@pytest.mark.parametrize("triangles,threads", [(2000, 0), (5000, 0), (5000, 2), (100_000, 0), (100_000, 3)])
def test_bvh_build_does_without_threads(native, triangles, threads):
    """A process at its thread limit builds the same tree on the threads it has."""
    _run(native("bvh_threads", "bvh_build.cpp"), "threads", triangles, threads)


@pytest.mark.parametrize("triangles", [5000, 100_000])
def test_bvh_build_hands_a_threads_exception_on(native, triangles):
    """Out of memory on a worker thread: the caller gets the exception, once, and can build again."""
    _run(native("bvh_threads", "bvh_build.cpp"), "memory", triangles)


def _soup(n, seed=5):
    """n small triangles in the unit cube (n x 3 x 3)."""
    g = np.random.RandomState(seed)
    return g.uniform(size=(n, 1, 3)) + 0.01 * g.uniform(size=(n, 3, 3))


def _bvh_of(native, tmp_path, positions):
    path = str(tmp_path / "positions.bin")
    with np.errstate(over="ignore"):
        positions.astype(np.float32).reshape(-1).tofile(path)
    _run(native("bvh_inputs", "bvh_build.cpp"), path)


@pytest.mark.parametrize("n", [1, 2, 3, 7, 64, 1000, 70000])
@pytest.mark.parametrize("extent", [(1, 1, 1), (1e-39,) * 3, (3e-38,) * 3, (1, 1, 1e-42), (1, 1, 0), (0, 0, 0)])
def test_bvh_of_any_extent(native, tmp_path, n, extent):
    """Extents down to denormal ones, where bins per unit of length overflow a float, and flat ones."""
    _bvh_of(native, tmp_path, _soup(n) * np.array(extent))


def test_bvh_of_mixed_magnitudes(native, tmp_path):
    g = np.random.RandomState(6)
    _bvh_of(native, tmp_path, _soup(5000) * 10.0 ** g.uniform(-44, 30, size=(5000, 1, 1)))


@pytest.mark.parametrize("n", [1, 2, 3, 7, 64, 1000, 70000])
@pytest.mark.parametrize("kind", ["nan corner", "nan", "infinite", "all nan", "huge"])
def test_bvh_with_corners_that_are_not_finite(native, tmp_path, n, kind):
    """Triangles with NaN or infinite corners are in the tree and widen no box; finite ones whose extent
    overflows a float have boxes that hold them."""
    p = _soup(n)
    if kind == "nan corner":
        p[::7, 1, 2] = np.nan
    elif kind == "nan":
        p[::7] = np.nan
    elif kind == "infinite":
        p[::5, 0, 0] = np.inf
        p[1::5, 0, 1] = -np.inf
    elif kind == "all nan":
        p[:] = np.nan
    else:
        p = np.clip((p - 0.5) * 6.8e38, -np.finfo(np.float32).max, np.finfo(np.float32).max)
    _bvh_of(native, tmp_path, p)


@pytest.mark.parametrize("kind,radius", [
    ("plain", 0.505 * 3 ** 0.5), ("infinite", 0.505 * 3 ** 0.5), ("nan", 0.505 * 3 ** 0.5), ("none", 0), ("wide", 1e18),
    ("far", 0)])
def test_world_sphere_is_finite(native, tmp_path, kind, radius):
    """Corners that are not finite, and extents whose square overflows a float, leave the sphere that distant and
    environment lights stand on finite (a ray to a point at infinity passes every box of the tree)."""
    p = _soup(1000).astype(np.float64)
    p[0], p[1] = 0.0, 1.01  # the corners of the bounds
    if kind == "infinite":
        p[2, 0, 0], p[3, 1, 2] = np.inf, -np.inf
    elif kind == "nan":
        p[2] = np.nan
    elif kind == "none":
        p[:] = np.inf
    elif kind == "wide":
        p = (p - 0.5) * 4e38
    elif kind == "far":
        p = 3.2e38 + p * 1e37
    path = str(tmp_path / "positions.bin")
    p.astype(np.float32).reshape(-1).tofile(path)
    _run(native("world_bounds", "scene_prep.cpp"), path, radius)
