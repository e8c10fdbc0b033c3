"""GPU path vs the CPU oracle at sizes the oracle finishes in seconds.

* 1M seeded rays, through the test hook and through the renderer's own
  persistent trace kernels: closest-hit primitive equal except ties, t within
  1e-5 relative or the float rounding bound of helpers.t_tolerance, occlusion equal to
  the oracle's (the oracle's BVH is checked equal to a brute-force loop in the
  CPU suite).
* images: the GPU and the oracle trace the same Sobol sample per path, so
  per-pixel sums match except where FP32 rounding sends a path down another
  branch; at least IMAGE_IDENTICAL of the pixels must match to 1e-4 relative.
* statistics: a 1024-spp FP64 GPU render against the reference's 65,536-spp
  FP64 per-pixel means, |difference| <= 3 sigma for >= 95% of the tested
  pixels; relative RMSE is printed.
"""
from __future__ import annotations

import os

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

# Path-for-path image bars (fraction of pixels identical to 1e-4; relative RMSE of the film sums).
# Measured on GB300: 0.9966 (displaced) to 0.9999 (Cornell) of pixels, RMSE 1.3e-6 to 1.4e-3.
IMAGE_IDENTICAL = 0.995
IMAGE_RMSE = 5e-3


@pytest.fixture(scope="module")
def port(built):
    from oracle import port as p
    p.lib()
    return p


def _bounds(host):
    p = host.arrays()["positions"].reshape(-1, 3)
    return p.min(0), p.max(0)


@pytest.mark.parametrize("name,kw", [("cornell", {}), ("displaced", dict(res=64, spp=4, subdiv=6))])
@pytest.mark.parametrize("kernel", ["hook", "production"])
def test_million_rays_match_oracle(ctx, port, tmp_path, name, kw, kernel):
    """1M seeded rays (origins in the scene's padded box, uniform directions) against the oracle's closest
    hit. kernel "hook": orion_gpu_trace (one ray per thread, traverse()); "production": orion_gpu_trace_wave,
    the renderer's own persistent k_trace / k_trace_sh launched on the rays as a wave's extension and shadow
    rays. Same primitive unless the two are at equal distance (a tie), t within t_tolerance; a hit where
    the oracle misses (or the reverse) only on rays through a shared edge, where the two triangle tests
    round differently: at most 10 per million."""
    import orion_gb300 as og
    path = helpers.write_scene(name, str(tmp_path / name), **kw)
    host = og.HostScene.load(path)
    lo, hi = _bounds(host)
    n = 1 << 20
    rays = helpers.random_rays(n, lo, hi, seed=17)
    finite = np.zeros(n, bool)
    finite[: n // 8] = True  # the renderer's closest-hit rays are unbounded: finite tfar only for occlusion
    rays[finite, 7] = (helpers.splitmix_uniform(n // 8, 18) * float(np.max(hi - lo))).astype(np.float32)
    sid = ctx.upload(host)
    trace = ctx.trace if kernel == "hook" else ctx.trace_wave
    closest = rays.copy()
    if kernel == "production":
        closest[:, 7] = helpers.FLT_MAX
    t, u, v, prim = trace(sid, closest)
    _, _, _, occ = trace(sid, rays, any_hit=True)
    ctx.release(sid)
    sc = port.Scene(host)
    rt, ru, rv, rprim = sc.trace(closest)
    _, _, _, rocc = sc.trace(rays) if kernel == "production" else (rt, ru, rv, rprim)
    hit = rprim >= 0
    miss_mismatch = np.count_nonzero((prim >= 0) != hit)
    assert miss_mismatch <= n * 1e-5, f"hit/miss differs on {miss_mismatch} rays"
    occ_mismatch = np.count_nonzero((occ >= 0) != (rocc >= 0))
    assert occ_mismatch <= n * 1e-5, f"occlusion differs on {occ_mismatch} rays"
    both = hit & (prim >= 0)
    tol = helpers.t_tolerance(closest, rt, rprim, host.arrays()["positions"])
    t_ok = np.abs(t.astype(np.float64) - rt) <= tol
    same = prim == rprim
    rel = np.abs(t - rt)[both] / np.maximum(np.abs(rt[both]), 1e-30)
    print(f"{name} ({kernel}): {n} rays, {hit.mean():.3f} hit, primitive identical on {same[both].mean():.6f} "
          f"of hits (rest are ties), t beyond 1e-5 relative on {np.count_nonzero(rel > 1e-5)} rays (max "
          f"{rel.max():.2e}), all within the rounding bound: {bool(t_ok[both].all())}; hit/miss differs on "
          f"{miss_mismatch}, occlusion on {occ_mismatch}")
    assert t_ok[both].all(), f"t outside the tolerance on {np.count_nonzero(both & ~t_ok)} rays"
    if kernel == "production":  # barycentrics of the same primitive (grazing hits round them further)
        ok = same & both
        uv_ok = (np.abs(u[ok] - ru[ok]) <= 1e-4) & (np.abs(v[ok] - rv[ok]) <= 1e-4)
        assert uv_ok.mean() >= 0.9999, f"u, v differ beyond 1e-4 on {np.count_nonzero(~uv_ok)} hits"


def test_traversal_stack_overflow_is_reported(ctx, tmp_path):
    """A traversal whose stack would overflow writes nothing out of bounds and the call fails with
    ORION_ERR_DEVICE; the context keeps working (test kernels with a 2-entry stack)."""
    import orion_gb300 as og
    path = helpers.write_scene("displaced", str(tmp_path / "d"), res=32, spp=1, subdiv=6)
    host = og.HostScene.load(path)
    sid = ctx.upload(host)
    lo, hi = _bounds(host)
    rays = helpers.random_rays(1 << 14, lo, hi, seed=23)
    try:
        good = ctx.trace_wave(sid, rays)
        ref, _ = ctx.render(sid, 32, 32)
        ctx.set_test_limits(stack_entries=2)
        with pytest.raises(og.OrionError, match="overflowed its stack") as e:
            ctx.trace_wave(sid, rays)
        assert e.value.code == -7
        with pytest.raises(og.OrionError, match="overflowed its stack"):
            ctx.render(sid, 32, 32)
        ctx.set_test_limits()
        again = ctx.trace_wave(sid, rays)
        img, _ = ctx.render(sid, 32, 32)
        assert all(np.array_equal(a, b) for a, b in zip(good, again))
        assert np.array_equal(img, ref)
    finally:
        ctx.set_test_limits()
        ctx.release(sid)


@pytest.mark.parametrize("name,kw", [
    ("cornell", dict(res=96, spp=8)),
    ("zoo", dict(res=64, spp=8, beckmann=True)),
    ("mixed", dict(width=96, height=54, spp=8, subdivs=(2, 2, 2, 2, 2, 2, 2, 2))),
    ("displaced", dict(res=64, spp=8, subdiv=5)),
    ("envlit", dict(res=64, spp=8)),
    ("textured", dict(res=64, spp=8)),
])
def test_image_matches_oracle_path_for_path(ctx, port, tmp_path, name, kw):
    import orion_gb300 as og
    path = helpers.write_scene(name, str(tmp_path / name), **kw)
    host = og.HostScene.load(path)
    sc = port.Scene(host)
    ref, _ = sc.render()
    sid = ctx.upload(host)
    gpu, cnt = ctx.render(sid, sc.width, sc.height)
    ctx.release(sid)
    assert (cnt == sc.spp).all()
    close = (np.abs(gpu.astype(np.float64) - ref) <= 1e-4 * np.abs(ref) + 1e-5).all(2).mean()
    rmse = float(np.sqrt(np.mean((gpu.astype(np.float64) - ref) ** 2)) / max(np.sqrt(np.mean(ref.astype(np.float64) ** 2)), 1e-12))
    print(f"{name}: {close:.4f} of pixels identical path-for-path, relative RMSE {rmse:.2e}")
    assert close >= IMAGE_IDENTICAL
    assert rmse < IMAGE_RMSE


def test_render_statistics_within_3_sigma_of_reference(ctx, tmp_path):
    """Cornell box at the benchmark resolution: GPU FP64 film vs the reference's 64k-spp FP64 pixel means."""
    import orion_gb300 as og
    g = helpers.golden("stats_cornell.npz")
    path = helpers.write_scene("cornell", str(tmp_path / "c"))
    assert helpers.scene_hash(path) == bytes(g["hash"]).decode()
    host = og.HostScene.load(path)
    sid = ctx.upload(host)
    n = 1024
    ref_spp = int(g["spp"])
    s, q = ctx.render(sid, 256, 256, spp=n, first_pass=ref_spp, fp64=True)  # sample passes disjoint from the reference's
    ctx.release(sid)
    pix = g["pix"]
    s, q = s[pix[:, 1], pix[:, 0]], q[pix[:, 1], pix[:, 0]]
    mean = s / n
    var = np.maximum(q / n - mean ** 2, 0)
    rmean = g["sum"] / ref_spp
    rvar = np.maximum(g["sumsq"] / ref_spp - rmean ** 2, 0)
    sigma = np.sqrt(var / n + rvar / ref_spp) + 1e-7
    z = np.abs(mean - rmean) / sigma
    frac = (z <= 3).all(1).mean()
    rmse = float(np.sqrt(np.mean((mean - rmean) ** 2)) / np.sqrt(np.mean(rmean ** 2)))
    print(f"{len(pix)} pixels: {frac:.3f} within 3 sigma, relative RMSE {rmse:.4f} vs {ref_spp}-spp FP64 reference")
    assert frac >= 0.95
    assert rmse < 0.05


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 4097, 70001])
def test_ray_queries_at_ragged_sizes(ctx, port, tmp_path, n):
    """Ray counts that leave warps and their pieces of the list partly empty: unbounded rays equal the
    renderer's trace kernels bit for bit; rays with a near and a far bound (hits in (tnear, tfar]) agree with
    the oracle in hit or miss but for edge rays (10 per million, one at least) and in distance within
    t_tolerance."""
    import orion_gb300 as og
    path = helpers.write_scene("zoo", str(tmp_path / "zoo"), res=32, spp=1)
    host = og.HostScene.load(path)
    lo, hi = _bounds(host)
    rays = helpers.random_rays(n, lo, hi, seed=29)
    sid = ctx.upload(host)
    for a, b in zip(ctx.trace(sid, rays), ctx.trace_wave(sid, rays)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    size = float(np.max(hi - lo))
    rays[:, 6] = (helpers.splitmix_uniform(n, 30) * 0.2 * size).astype(np.float32)
    rays[:, 7] = rays[:, 6] + (helpers.splitmix_uniform(n, 31) * size).astype(np.float32)
    t, _, _, prim = ctx.trace(sid, rays)
    ctx.release(sid)
    rt, _, _, rprim = port.Scene(host).trace(rays)
    edge = max(1, int(n * 1e-5))
    assert np.count_nonzero((prim >= 0) != (rprim >= 0)) <= edge
    both = (prim >= 0) & (rprim >= 0)
    tol = helpers.t_tolerance(rays, rt, rprim, host.arrays()["positions"])
    assert np.count_nonzero(both & ~(np.abs(t.astype(np.float64) - rt) <= tol)) <= edge
    assert (t[prim >= 0] > rays[prim >= 0, 6]).all() and (t[prim >= 0] <= rays[prim >= 0, 7]).all()


@pytest.mark.parametrize("n", [63, 8193, 100001])
def test_ray_queries_that_begin_behind_the_origin(ctx, port, tmp_path, n):
    """Negative near bounds (three rays of four, among others whose hits all lie ahead), some with negative far
    bounds too: the least t in (tnear, tfar], as the oracle finds it, and the same rays hit something in
    orion_gpu_trace's any-hit form; edge rays (10 per million, one at least) excepted."""
    import orion_gb300 as og
    host = og.HostScene.load(helpers.write_scene("zoo", str(tmp_path / "zoo"), res=32, spp=1))
    lo, hi = _bounds(host)
    size = float(np.max(hi - lo))
    rays = helpers.random_rays(n, lo, hi, seed=41)
    behind = np.arange(n) % 4 != 0
    rays[behind, 6] = (-helpers.splitmix_uniform(n, 42) * size)[behind].astype(np.float32)
    rays[:, 7] = rays[:, 6] + (helpers.splitmix_uniform(n, 43) * size).astype(np.float32)
    sid = ctx.upload(host)
    t, _, _, prim = ctx.trace(sid, rays)
    _, _, _, occ = ctx.trace(sid, rays, any_hit=True)
    ctx.release(sid)
    rt, _, _, rprim = port.Scene(host).trace(rays)
    edge = max(1, int(n * 1e-5))
    assert n < 100 or np.count_nonzero((rprim >= 0) & (rt < 0)) > n // 10
    assert np.count_nonzero((prim >= 0) != (rprim >= 0)) <= edge
    assert np.count_nonzero((occ >= 0) != (rprim >= 0)) <= edge
    both = (prim >= 0) & (rprim >= 0)
    tol = helpers.t_tolerance(rays, rt, rprim, host.arrays()["positions"])
    assert np.count_nonzero(both & ~(np.abs(t.astype(np.float64) - rt) <= tol)) <= edge
    assert (t[prim >= 0] > rays[prim >= 0, 6]).all() and (t[prim >= 0] <= rays[prim >= 0, 7]).all()


@pytest.mark.parametrize("n", [2**59, 2**60, 2**63 - 1])
def test_ray_queries_beyond_any_memory_are_refused(ctx, tmp_path, n):
    """Counts whose buffers' bytes wrap 64 bits: ORION_ERR_NOMEM before any device work."""
    import ctypes
    import orion_gb300 as og
    host = og.HostScene.load(helpers.write_scene("cornell", str(tmp_path / "c"), res=32, spp=1))
    sid = ctx.upload(host)
    rays = np.zeros((1, 8), np.float32)
    out = [np.zeros(1, np.float32) for _ in range(3)] + [np.zeros(1, np.int32)]
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    for any_hit in (0, 1):
        assert og.library().orion_gpu_trace(ctx._h, sid, n, ptr(rays), any_hit, *(ptr(a) for a in out)) == -5
    assert (ctx.trace(sid, rays)[3] == -1).all()
    ctx.release(sid)


@pytest.mark.parametrize("name,kw", [
    ("caustics", dict(res=48, iterations=8, photons=20000, radius=0.08, max_depth=5)),
    ("envlit_sppm", dict(res=32, iterations=4, photons=10000, radius=0.08)),
    ("textured_sppm", dict(res=32, iterations=4, photons=10000, radius=0.08)),
])
def test_sppm_matches_oracle(ctx, port, tmp_path, name, kw):
    """SPPM on the GPU against the oracle (pinned bit-exact to the reference's single-thread SPPM).

    The same sample indices drive both; photon flux adds up in another order on the GPU (atomics) and
    device transcendental functions round differently, so a pixel agrees to FP32 rounding unless one of
    its photons took another path: most pixels within 1e-3 relative, the image within 1% RMSE."""
    import orion_gb300 as og
    path = helpers.write_scene(name, str(tmp_path / "c"), **kw)
    host = og.HostScene.load(path)
    ref, _ = port.Scene(host).render_sppm()
    sid = ctx.upload(host)
    gpu, cnt = ctx.render_sppm(sid, kw["res"], kw["res"])
    st = ctx.last_stats()
    ctx.release(sid)
    assert (cnt == kw["iterations"]).all() and np.isfinite(gpu).all()
    rel = np.abs(gpu.astype(np.float64) - ref) / np.maximum(np.abs(ref), 1e-3)
    close = (rel <= 1e-3).all(2).mean()
    rmse = float(np.sqrt(np.mean((gpu.astype(np.float64) - ref) ** 2)) / np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    print(f"{name}: {close:.4f} of pixels within 1e-3, relative RMSE {rmse:.2e}, {st['rays']} rays, "
          f"{st['device_ms']:.2f} ms")
    assert close >= 0.9
    assert rmse < 0.01


@pytest.mark.parametrize("width,height,iterations,photons,radius,max_depth",
                         [(33, 5, 2, 1, 0.08, 3), (37, 21, 2, 6001, 0.3, 4),
                          (9, 3, 3, 31, 0.08, 1), (40, 40, 2, 20000, 0.02, 6)])
def test_sppm_at_ragged_sizes(ctx, port, width, height, iterations, photons, radius, max_depth):
    """(Not a film of one pixel: its grid spans exactly two radii, so whether it has one cell or two per
    axis, and a photon counts once or eight times, hangs on the last bit of the visible point.)
    Films smaller than a tile or a block, photon counts that leave warps partly empty, cells of many
    more hits than lanes (large radius) and of few: film counts exact, the image within the 1% RMSE of
    the test above (a photon that takes another path on the CPU, 3 in 10,000, moves a pixel of hundreds of
    photons by less)."""
    from orion_gb300 import scenegen
    s = scenegen.caustics(64, subdiv=2)
    s.width, s.height = width, height
    host = scenegen.to_host_scene(s)
    kw = dict(iterations=iterations, photons=photons, radius=radius, max_depth=max_depth)
    ref, _ = port.Scene(host).render_sppm(**kw)
    sid = ctx.upload(host)
    gpu, cnt = ctx.render_sppm(sid, width, height, **kw)
    ctx.release(sid)
    assert (cnt == iterations).all() and np.isfinite(gpu).all()
    ref = ref.astype(np.float64).reshape(gpu.shape)
    assert np.sqrt(np.mean((gpu - ref) ** 2)) <= 0.01 * np.sqrt(np.mean(ref ** 2))


@pytest.mark.parametrize("width,height", [(3, 3), (4, 3)])
def test_sppm_hash_cells_of_many_hits(ctx, port, width, height):
    """A film of few pixels has as few hash cells, so each holds far more photon hits than the gather adds up
    together (2^14; about 50,000 here) and turns up many times in one sphere: cells one by one, the image
    within 1% RMSE as above (thousands of photons a pixel). How often a photon counts hangs on which cells a
    sphere reaches, and films this small easily have one that ends at a cell's edge: the oracle's own film
    must not hang on the last bits of the camera."""
    from orion_gb300 import scenegen

    def scene(shift=(0.0, 0.0, 0.0)):
        s = scenegen.caustics(64, subdiv=2)
        s.width, s.height = width, height
        s.eye = tuple(e + d for e, d in zip((0.113, 0.071, 3.437), shift))
        return scenegen.to_host_scene(s)

    kw = dict(iterations=1, photons=500_000, radius=0.37, max_depth=5)
    rms = lambda a: np.sqrt(np.mean(a ** 2))
    ref = port.Scene(scene()).render_sppm(**kw)[0].astype(np.float64)
    for axis in range(3):
        moved, _ = port.Scene(scene([1e-5 * (axis == k) for k in range(3)])).render_sppm(**kw)
        assert rms(moved - ref) < 1e-3 * rms(ref)
    sid = ctx.upload(scene())
    gpu, cnt = ctx.render_sppm(sid, width, height, **kw)
    ctx.release(sid)
    assert (cnt == 1).all() and np.isfinite(gpu).all()
    assert rms(gpu - ref.reshape(gpu.shape)) <= 0.01 * rms(ref)


def test_sppm_of_more_cells_than_one_scan_pass_takes(ctx, port):
    """4.2 million pixels, as many hash cells: the scan of their counts has more block sums than its last
    pass adds up by itself (kScanRaw). Each visible point has about 60 photons, and 3 in 10,000 take another
    path on the CPU (above), so about 2% of the pixels may differ by a photon: 95% within 1e-3, of pixels of
    which photons light most."""
    from orion_gb300 import scenegen
    s = scenegen.caustics(64, subdiv=0)
    s.width, s.height = 2100, 2000
    host = scenegen.to_host_scene(s)
    kw = dict(iterations=1, radius=0.047, max_depth=2)
    oracle = port.Scene(host)
    close = lambda a, b: (np.abs(a - b) <= 1e-3 * np.abs(b) + 1e-6).all(-1).mean()
    ref = oracle.render_sppm(photons=200_000, threads=0, **kw)[0].astype(np.float64)
    without = oracle.render_sppm(photons=1, threads=0, **kw)[0].astype(np.float64)
    assert close(without, ref) < 0.2
    sid = ctx.upload(host)
    gpu, cnt = ctx.render_sppm(sid, 2100, 2000, photons=200_000, **kw)
    ctx.release(sid)
    assert (cnt == 1).all()
    assert close(gpu, ref) > 0.95


def test_sppm_parameters_and_errors(ctx, tmp_path):
    import orion_gb300 as og
    path = helpers.write_scene("caustics", str(tmp_path / "c"), res=24, iterations=2, photons=-1, radius=0.1)
    host = og.HostScene.load(path)
    sid = ctx.upload(host)
    try:
        a, ca = ctx.render_sppm(sid, 24, 24)                       # the scene's parameters (photons = W*H)
        b, cb = ctx.render_sppm(sid, 24, 24, photons=24 * 24)       # the same, explicitly
        assert np.allclose(a, b, rtol=1e-4, atol=1e-6) and (ca == 2).all()  # photon sums: atomics, any order
        c, cc = ctx.render_sppm(sid, 24, 24, iterations=3)
        assert (cc == 3).all()
        with pytest.raises(og.OrionError, match="radius"):
            ctx.render_sppm(sid, 24, 24, radius=0.0)
    finally:
        ctx.release(sid)
