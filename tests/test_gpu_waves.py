"""Wave scheduling: a render is split into waves of path slots, and consecutive
waves run on two streams. Every pixel's film sum is taken in sample order
(RenderTarget::acumulate, src/texture/rendertarget.cpp:22-27), so the film
must be bit-identical whatever the wave size, whether waves overlap on two
streams or run on one (profiled renders), and from run to run."""
from __future__ import annotations

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(ctx, tmp_path_factory):
    import orion_gb300 as og
    path = helpers.write_scene("zoo", str(tmp_path_factory.mktemp("waves") / "zoo"), res=48, spp=12)
    host = og.HostScene.load(path)
    sid = ctx.upload(host)
    yield sid
    ctx.release(sid)


def test_film_independent_of_waves_and_streams(ctx, scene):
    total = 48 * 48 * 12
    ref, cnt = ctx.render(scene, 48, 48, wave_paths=total)  # one wave, one stream
    assert (cnt == 12).all()
    cfg = ctx.get_config()
    try:
        for streams in (1, 2, 3, 4):
            ctx.set_config(streams=streams)
            for wave in (4096, 3001, 48 * 48):
                img, c = ctx.render(scene, 48, 48, wave_paths=wave)  # several waves on `streams` streams
                assert np.array_equal(c, cnt)
                assert np.array_equal(img.view(np.uint32), ref.view(np.uint32)), f"wave {wave}, {streams} streams"
    finally:
        ctx.set_config(**cfg)
    # FP64 sums of squares are grouped by wave (rounding depends on the wave size), so the FP64
    # film is compared at one wave size: two streams against one.
    s1, q1 = ctx.render(scene, 48, 48, wave_paths=5000, fp64=True)
    ctx.set_profiling(True)
    try:
        img, _ = ctx.render(scene, 48, 48, wave_paths=4096)  # profiled: one stream
        s2, q2 = ctx.render(scene, 48, 48, wave_paths=5000, fp64=True)
    finally:
        ctx.set_profiling(False)
    assert np.array_equal(s1, s2) and np.array_equal(q1, q2)
    assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))
    ctx.render(scene, 48, 48, wave_paths=4096)
    st = ctx.last_stats()
    again, _ = ctx.render(scene, 48, 48, wave_paths=4096)
    assert np.array_equal(again.view(np.uint32), ref.view(np.uint32))
    assert ctx.last_stats()["rays"] == st["rays"]


def test_traversal_work_counts(ctx, scene):
    """A counting render traces the same rays into the same film and reports
    per-kind BVH work: every ray visits the root node at least."""
    import orion_gb300 as og
    ref, _ = ctx.render(scene, 48, 48, wave_paths=4096)
    assert all(v == 0 for k in ctx.traversal_work().values() for v in k.values())
    ctx.set_profiling(og.PROFILE_TRAVERSAL)
    try:
        img, _ = ctx.render(scene, 48, 48, wave_paths=4096)
        st = ctx.last_stats()
        work = ctx.traversal_work()
        ctx.set_profiling(og.PROFILE_STAGES | og.PROFILE_TRAVERSAL)
        both, _ = ctx.render(scene, 48, 48, wave_paths=4096)
        assert ctx.stage_times()["trace_ext"]["launches"] > 0
        assert ctx.traversal_work()["ext"]["rays"] == work["ext"]["rays"]
    finally:
        ctx.set_profiling(False)
    assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(both.view(np.uint32), ref.view(np.uint32))
    assert work["ext"]["rays"] == st["ext_rays"]
    assert work["shadow"]["rays"] == st["shadow_rays"]
    assert work["mis"]["rays"] == st["mis_rays"]
    for kind, w in work.items():
        if w["rays"]:
            assert w["nodes"] >= w["rays"], kind
            assert w["triangles"] > 0, kind
            assert w["nodes"] < 10_000 * w["rays"], kind
    ctx.render(scene, 48, 48, wave_paths=4096)
    assert ctx.traversal_work()["ext"]["nodes"] == 0


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (3, 5, 7), (9, 4, 1), (33, 6, 255), (7, 41, 257), (64, 48, 3),
                                              (8, 3, 700)])
def test_pixel_order_at_ragged_sizes(ctx, width, height, spp):
    """Slots run pixel after pixel through tiles of 8 x 4 pixels, each pixel's passes in order, and the
    film adds up to 256 samples of a pixel at a go: films with cut-off tiles, chunks and sample runs
    equal the batch engine's, which has kernels of its own (FP64 sums, 1e-5 as its tests: the two
    engines' FP32 paths are compiled apart), and do not depend on the wave size."""
    from orion_gb300 import scenegen
    s = scenegen.zoo(subdiv=1, spp=spp, max_depth=3)
    s.width, s.height = width, height
    host = scenegen.to_host_scene(s)
    sid = ctx.upload(host)
    try:
        (want, _, _), = ctx.render_batch([dict(sid=sid, width=width, height=height, first_pass=5)])[0]
        got, _ = ctx.render(sid, width, height, first_pass=5, fp64=True)
        assert np.allclose(got, want, rtol=1e-5, atol=1e-7)
        ref, cnt = ctx.render(sid, width, height, first_pass=5)
        assert (cnt == spp).all()
        for wave in (width * height * spp, 1000, 64):
            img, c = ctx.render(sid, width, height, first_pass=5, wave_paths=wave)
            assert np.array_equal(c, cnt)
            assert np.array_equal(img.view(np.uint32), ref.view(np.uint32)), f"wave {wave}"
    finally:
        ctx.release(sid)


@pytest.mark.parametrize("paths", [(1 << 19) - 4096, 1 << 19, (1 << 19) + 4096])
def test_appended_and_compacted_queues_agree(ctx, paths):
    """Waves of up to 2^19 paths append to their queues, larger ones list them in slot order; the order
    of a queue never changes a path's result."""
    from orion_gb300 import scenegen
    s = scenegen.zoo(subdiv=2, spp=paths // 4096, max_depth=4)
    s.width = s.height = 64
    sid = ctx.upload(scenegen.to_host_scene(s))
    try:
        one, cnt = ctx.render(sid, 64, 64, wave_paths=paths)
        many, c = ctx.render(sid, 64, 64, wave_paths=1 << 16)
        assert np.array_equal(c, cnt) and (cnt == paths // 4096).all()
        assert np.array_equal(one.view(np.uint32), many.view(np.uint32))
    finally:
        ctx.release(sid)


@pytest.mark.parametrize("spp", [1, 7, 8, 9, 31, 255, 256, 257])
def test_batch_film_adds_every_run_of_samples(ctx, spp):
    """A batch wave's film kernel takes 256 slots at a time and adds up each pixel's run of samples in
    pieces of 8: runs of one sample to more than 256, cut at block ends and (behind a job of 3 samples
    a pixel, 13 x 7 pixels) at odd slots, with squares and without. Sums and squares as
    the plain FP64 render's to FP32 rounding (1e-5, as the batch tests), counts exactly."""
    from orion_gb300 import scenegen
    s = scenegen.zoo(subdiv=1, spp=spp, max_depth=2)
    s.width, s.height = 13, 7
    sid = ctx.upload(scenegen.to_host_scene(s))
    try:
        jobs = [dict(sid=sid, width=13, height=7, spp=3), dict(sid=sid, width=13, height=7, spp=spp, first_pass=2)]
        films = ctx.render_batch(jobs)[0]
        for job, (got, sq, count) in zip(jobs, films):
            want, want_sq = ctx.render(sid, 13, 7, spp=job["spp"], first_pass=job.get("first_pass", 0), fp64=True)
            assert (count == job["spp"]).all()
            assert np.allclose(got, want, rtol=1e-5, atol=1e-7)
            assert np.allclose(sq, want_sq, rtol=1e-5, atol=1e-7)
        only_sums = ctx.render_batch(jobs, sumsq=False)[0]
        for a, b in zip(films, only_sums):
            assert np.allclose(a[0], b[0], rtol=1e-12, atol=1e-12)
    finally:
        ctx.release(sid)


def test_a_render_of_no_samples_is_black(ctx):
    """A scene of 0 samples a pixel renders to a film of zeros and no counts, whatever the context rendered
    before."""
    from orion_gb300 import scenegen
    s = scenegen.zoo(subdiv=1, spp=2, max_depth=2)
    s.width, s.height = 20, 12
    some = ctx.upload(scenegen.to_host_scene(s))
    s.spp = 0
    none = ctx.upload(scenegen.to_host_scene(s))
    try:
        img, cnt = ctx.render(some, 20, 12)
        assert img.any() and (cnt == 2).all()
        ctx.render(some, 20, 12, fp64=True)
        img, cnt = ctx.render(none, 20, 12)
        assert not img.any() and not cnt.any()
        for sums in ctx.render(none, 20, 12, fp64=True):
            assert not sums.any()
        assert ctx.last_stats()["paths"] == 0
    finally:
        ctx.release(some)
        ctx.release(none)
