"""GPU checks of batch runs (many rooms as one wavefront, pach_batch_begin) and of the graph-mode
device loop: every room of a batch traces exactly as a single run with the same primary numbering."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from pachydermacoustic_universal_gb300 import _capi, rooms, tracer  # noqa: E402

pytestmark = pytest.mark.gpu


def _rooms():
    hall = rooms.irregular_hall_c2(target_tris=2000)
    return [rooms.shoebox_c1(), rooms.proposal_room_c4(3), hall]


def test_batch_rooms_match_single_runs():
    ws = _rooms()
    ds = [tracer.DeviceScene(w.scene) for w in ws]
    rays = [3000, 2000, 700]
    seed = 11
    hb, sb = tracer.trace_batch(ws, dscenes=ds, rays=rays, seed=seed)
    off = 0
    seg = 0
    for i, w in enumerate(ws):
        hs, ss = tracer.trace(w, dscene=ds[i], rays=rays[i], seed=seed, ray_begin=off)
        T = hs["energy"].shape[-1]
        for name in ("energy", "pressure", "dir_pos", "dir_neg", "analysis"):
            a, b = hb[i][name][..., :T], hs[name]
            assert np.allclose(a, b, rtol=1e-9, atol=1e-30), (i, name)
        seg += ss["segments"]
        off += rays[i]
    assert sb["segments"] == seg
    assert sb["primaries"] == sum(rays)


def test_batch_scaling_is_per_room():
    ws = _rooms()[:2]
    ds = [tracer.DeviceScene(w.scene) for w in ws]
    rays = [1500, 500]
    raw, _ = tracer.trace_batch(ws, dscenes=ds, rays=rays, seed=3)
    sc, _ = tracer.trace_batch(ws, dscenes=ds, rays=rays, seed=3, scaled=True)
    for i in range(2):
        ns = len(ws[i].sources)
        assert np.allclose(sc[i]["energy"], raw[i]["energy"] * ns / rays[i], rtol=1e-9)


def test_graph_loop_matches_host_loop():
    w = rooms.shoebox_c1()
    ds = tracer.DeviceScene(w.scene)
    hg, sg = tracer.trace(w, dscene=ds, rays=4000, seed=9)
    hh, sh = tracer.trace(w, dscene=ds, rays=4000, seed=9, kernel_timing=True)
    assert sg["segments"] == sh["segments"]
    assert np.allclose(hg["energy"], hh["energy"], rtol=1e-9, atol=1e-30)
    assert sh["trace_ms"] > 0 and sg["trace_ms"] == 0


def test_batch_of_c3_rooms_runs():
    ws = rooms.batched_rooms_c3(n_rooms=16, max_rays=20_000)
    h, s = tracer.trace_batch(ws, rays=[min(w.rays, 600) for w in ws], seed=5)
    assert len(h) == 16
    for i, w in enumerate(ws):
        assert h[i]["energy"].shape[0] == len(w.receivers)
        assert np.all(np.isfinite(h[i]["energy"]))
        assert h[i]["energy"].sum() > 0
    assert s["queue_overflows"] == 0


def test_autotune_picks_and_caches(tmp_path):
    ws = _rooms()[:2]
    ds = [tracer.DeviceScene(w.scene) for w in ws]
    cache = str(tmp_path / "tune.txt")
    t1 = tracer.autotune(ws, dscenes=ds, rays=[2000, 2000], sample_rays=600, cache_path=cache)
    assert t1["from_cache"] == 0 and t1["trials"] >= 5 and t1["segments_per_s"] > 0
    assert t1["wave_kilo_items"] in (2048, 4096, 8192, 16384) and t1["block_threads"] in (128, 256)
    assert t1["blocks_per_sm"] in (4, 6) and t1["traversal"] in (1, 2, 3)
    t2 = tracer.autotune(ws, dscenes=ds, rays=[2000, 2000], sample_rays=600, cache_path=cache)
    assert t2["from_cache"] == 1
    assert all(t2[k] == t1[k] for k in tracer.TUNE_KNOBS)
    # the tuned knobs change scheduling only: same histograms as the defaults
    ha, _ = tracer.trace_batch(ws, dscenes=ds, rays=[800, 400], seed=2, tune=t1)
    hb, _ = tracer.trace_batch(ws, dscenes=ds, rays=[800, 400], seed=2)
    for i in range(2):
        assert np.allclose(ha[i]["energy"], hb[i]["energy"], rtol=1e-9, atol=1e-30)


def test_quantised_nodes_trace_the_same_rays():
    """64-byte nodes hold conservative boxes of the 128-byte ones: the same nearest hits, except that
    the walk order decides exact FP32 ties (a ray through an edge shared by two walls), which sends a
    few rays in a million down the other wall's path."""
    for w in (rooms.shoebox_c1(), rooms.irregular_hall_c2(target_tris=4000)):
        ds = tracer.DeviceScene(w.scene)
        ha, sa = tracer.trace(w, dscene=ds, rays=1500, seed=21, bvh_format=1)
        hb, sb = tracer.trace(w, dscene=ds, rays=1500, seed=21, bvh_format=2)
        assert abs(sa["segments"] - sb["segments"]) <= 1e-4 * sa["segments"]
        assert hb["energy"].sum() == pytest.approx(ha["energy"].sum(), rel=1e-3)


def test_fused_walk_traces_the_same_rays():
    """traversal 3 walks the rays inside the shading kernel with the same walk as the trace kernel's
    one-leaf-at-a-time variant: identical hits, identical histograms."""
    for w in (rooms.shoebox_c1(), rooms.irregular_hall_c2(target_tris=3000)):
        ds = tracer.DeviceScene(w.scene)
        ha, sa = tracer.trace(w, dscene=ds, rays=1500, seed=8, traversal=1)
        hb, sb = tracer.trace(w, dscene=ds, rays=1500, seed=8, traversal=3)
        assert sa["segments"] == sb["segments"]
        assert np.allclose(ha["energy"], hb["energy"], rtol=1e-9, atol=1e-30)


def test_scenes_built_together_equal_scenes_built_one_by_one():
    """pach_scenes_create (parallel host builds) gives the scenes pach_scene_create gives."""
    ws = rooms.batched_rooms_c3(max_rays=20_000)[:6]
    many = tracer.DeviceScene.many([w.scene for w in ws], threads=4)
    one = [tracer.DeviceScene(w.scene) for w in ws]
    for a, b in zip(many, one):
        ia, ib = a.info(), b.info()
        assert ia["n_triangles"] == ib["n_triangles"]
        np.testing.assert_array_equal(ia["poly_area"], ib["poly_area"])
    ha, sa = tracer.trace_batch(ws, dscenes=many, rays=[200] * len(ws), seed=9)
    hb, sb = tracer.trace_batch(ws, dscenes=one, rays=[200] * len(ws), seed=9)
    assert sa["segments"] == sb["segments"] and sa["accel"] == sb["accel"]
    for x, y in zip(ha, hb):
        np.testing.assert_allclose(x["energy"], y["energy"], rtol=1e-12, atol=1e-300)


@pytest.mark.parametrize("rays,ring_log2,feed_batch", [([1, 255, 256, 257, 900], 0, 0), ([300, 40, 700, 256, 513], 20, 0),
                                                       ([257, 600, 1, 300, 256], 0, 100)])
def test_batch_feed_order_traces_every_primary_once(rays, ring_log2, feed_batch):
    """Pilots first (several rooms at a time where the plan lets them), then the rest, with rooms below,
    at and above a pilot's size, a ring that takes few pilots at once and feeds smaller than a pilot:
    each room equals its single run (FP64 sums of the same terms in another order: 1e-9)."""
    ws = [rooms.proposal_room_c4(10 + i) for i in range(len(rays))]
    for w in ws:
        w.cutoff_s = 0.4
    ds = [tracer.DeviceScene(w.scene) for w in ws]
    kw = dict(seed=4, ring_log2=ring_log2, feed_batch=feed_batch)
    hb, sb = tracer.trace_batch(ws, dscenes=ds, rays=rays, **kw)
    assert sb["primaries"] == sum(rays) and sb["queue_overflows"] == 0
    off = 0
    for i, w in enumerate(ws):
        hs, _ = tracer.trace(w, dscene=ds[i], rays=rays[i], seed=4, ray_begin=off)
        for name in ("energy", "pressure", "dir_pos", "dir_neg", "analysis"):
            np.testing.assert_allclose(hb[i][name], hs[name], rtol=1e-9, atol=1e-30, err_msg=f"{i} {name}")
        off += rays[i]


@pytest.mark.parametrize("big,alpha,ring_log2,capture", [(4, 0.25, 20, 0), (4, 0.25, 19, 1), (2, 0.2, 20, 0), (40, 0.15, 0, 0)])
def test_rooms_that_outgrow_the_first_are_traced_in_the_ring_they_fit(big, alpha, ring_log2, capture):
    """A room of small trees first (alpha 0.6: 170 live rays a primary at most), then rooms of 9 to 30 times larger
    ones: the plan from the first room lets the others' pilots in together, which fills the ring, given or (40
    rooms) the three loops' own.  Each room alone fits, so the run starts over with the pilots one at a time and
    every room equals its single run (FP64 sums in another order: 1e-9; FP32 capture sums 1e-4)."""
    ws = [rooms.shoebox_c1() for _ in range(big + 1)]
    for i, w in enumerate(ws):
        w.scene.absorption = np.full_like(w.scene.absorption, alpha if i else 0.6)
        w.cutoff_s = 1.0
    ds = [tracer.DeviceScene(w.scene) for w in ws[:2]]
    ds += [ds[1]] * (big - 1)
    n = [256] * (big + 1)
    p = tracer._batch_params(ws, n, 4, ring_log2=ring_log2, capture=capture)
    run = tracer.BatchRun(ds, ws, n, p)
    run.wait()
    hb, sb = run.room_histograms(), run.stats()
    assert sb["primaries"] == sum(n) and sb["queue_overflows"] == 0
    cap = run.capture() if capture else None
    run.close()
    seg = det = 0
    for i, w in enumerate(ws):
        hs, ss = tracer.trace(w, dscene=ds[i], rays=256, seed=4, ray_begin=256 * i, capture=capture)
        seg, det = seg + ss["segments"], det + ss["detections"]
        for name in ("energy", "pressure", "dir_pos", "dir_neg", "analysis"):
            np.testing.assert_allclose(hb[i][name], hs[name], rtol=1e-9, atol=1e-30, err_msg=f"{i} {name}")
        if capture:
            R = len(w.receivers)
            np.testing.assert_allclose(cap[R * i:R * i + R].sum(axis=2), hs["capture"].sum(axis=2), rtol=1e-4)
    assert sb["segments"] == seg and sb["detections"] == det


def test_peak_of_several_loops_is_of_one_time():
    """The most rays that three loops hold at once: no more than the run's rays or the rings hold, and no less than a
    third of a run of one loop that is fed the same pilot (each of the three pilots is a third of it or more)."""
    w = rooms.shoebox_c1()
    w.cutoff_s = 0.4
    ds = tracer.DeviceScene(w.scene)
    for rays in (300, 5000):
        _, s3 = tracer.trace(w, dscene=ds, rays=rays, seed=6)
        _, s1 = tracer.trace(w, dscene=ds, rays=rays, seed=6, ring_log2=24)
        assert s3["kernel_launches"] != s1["kernel_launches"] and s3["octave_rays"] == s1["octave_rays"]
        assert s1["peak_live_rays"] / 3 <= s3["peak_live_rays"] <= min(s3["octave_rays"], 3 << 22)


@pytest.mark.parametrize("kind", ["box", "hall"])
def test_a_cancelled_run_has_traced_the_first_of_its_primaries(kind):
    """However many loops shared them: what a cancelled run leaves equals a run of its first rays_done primaries, and
    the run that goes on at ray_begin + rays_done adds the rest (FP64 sums in another order: 1e-9)."""
    w = rooms.shoebox_c1() if kind == "box" else rooms.irregular_hall_c2(target_tris=2000)
    w.cutoff_s = 0.4
    ds = tracer.DeviceScene(w.scene)
    p = dict(cutoff_length_m=w.cutoff_length_m, hist_cotime_ms=400.0, seed=6)
    run = tracer.Run(ds, w.sources, w.receivers, tracer.make_params(rays=4_000_000, ray_begin=100, **p))
    while run.poll()["rays_done"] < 3000:
        pass
    run.cancel()
    with pytest.raises(_capi.PachError):
        run.wait()
    n = run.poll()["rays_done"]
    h = run.histograms()
    assert 3000 <= n < 4_000_000 and run.stats()["primaries"] == n
    run.close()
    first, _ = tracer.trace(w, dscene=ds, rays=n, seed=6, ray_begin=100)
    for name in ("energy", "pressure", "dir_pos", "dir_neg", "analysis"):
        np.testing.assert_allclose(h[name], first[name], rtol=1e-9, atol=1e-30, err_msg=name)
    rest, _ = tracer.trace(w, dscene=ds, rays=500, seed=6, ray_begin=100 + n)
    both, _ = tracer.trace(w, dscene=ds, rays=n + 500, seed=6, ray_begin=100)
    np.testing.assert_allclose(h["energy"] + rest["energy"], both["energy"], rtol=1e-9, atol=1e-30)


def _l_room():
    """An L-shaped room (8 planes, not convex) of quads in two triangles."""
    x = [(0, 0), (8, 0), (8, 3), (4, 3), (4, 7), (0, 7)]
    b = rooms._Builder()
    lo, hi = [b.vertex((*p, 0.0)) for p in x], [b.vertex((*p, 3.0)) for p in x]
    for i in range(6):
        j = (i + 1) % 6
        b.quad_tris(lo[i], lo[j], hi[j], hi[i])
    for v in (lo, hi):
        b.quad_tris(v[0], v[1], v[2], v[3])
        b.quad_tris(v[0], v[3], v[4], v[5])
    v, offs, idx = b.arrays()
    n = offs.size - 1
    rng = np.random.default_rng(6)
    scene = rooms.SceneArrays(v, offs, idx, rng.uniform(0.1, 0.4, (n, 8)), np.full((n, 8), 0.3), np.zeros((n, 8)))
    return rooms.Workload("l_room", scene, [rooms.SourceSpec((1.0, 1.0, 1.5))],
                          [rooms.ReceiverSpec(p) for p in ((7.0, 1.0, 1.2), (1.0, 6.0, 1.6))], 1000, 0.8)


@pytest.mark.parametrize("ring_log2,rays", [(0, 700), (20, 60), (0, 1)])
@pytest.mark.parametrize("kind", ["box", "l", "diffusers"])
def test_rays_kept_over_interactions_equal_one_walk_per_launch(kind, ring_log2, rays):
    """Small scenes (rays kept in registers, the walk over planes where there are at most 8, the BVH for the
    diffusers' 12 + 36 triangles) against the BVH walk in a launch of its own: the same hits, so the same terms in
    every bin.  The small ring leaves few interactions a wave; ties go to the BVH in both."""
    if kind == "box":
        w = rooms.shoebox_c1()
    elif kind == "l":
        w = _l_room()
    else:
        w = rooms.shoebox_c1()
        w.scene = rooms._jittered_room(np.random.default_rng(2), (10.0, 8.0, 4.0), 12, 3, 0.0, (0.1, 0.4), (0.1, 0.5))
        assert 12 < w.scene.n_triangles <= 64
    w.cutoff_s = 0.8
    ds = tracer.DeviceScene(w.scene)
    ha, sa = tracer.trace(w, dscene=ds, rays=rays, seed=8, ring_log2=ring_log2)
    hb, sb = tracer.trace(w, dscene=ds, rays=rays, seed=8, traversal=1)
    assert sa["segments"] == sb["segments"] and sa["detections"] == sb["detections"] and sa["queue_overflows"] == 0
    for name in ("energy", "pressure", "dir_pos", "dir_neg", "analysis"):
        np.testing.assert_allclose(ha[name], hb[name], rtol=1e-9, atol=1e-30, err_msg=name)


@pytest.mark.parametrize("offset", [40.0, 150.0, 1000.0, 3000.0])
@pytest.mark.parametrize("kind", ["box", "l"])
def test_small_rooms_off_the_origin_walk_as_the_bvh_does(kind, offset):
    """A room that lies many times its extent from the origin: FP32 coordinates there are rounded by more than the
    margin of a room at the origin.  The walk over planes (up to 16 extents out) and what is used beyond find the
    BVH walk's hits; at 16 extents the BVH's own boxes are rounded by a tenth of their padding, so a hit may
    differ in 1e5 segments."""
    w = rooms.shoebox_c1() if kind == "box" else _l_room()
    s = np.array([offset, -0.7 * offset, 0.1 * offset])
    w.scene.vertices = w.scene.vertices + s
    w.sources = [rooms.SourceSpec(tuple(np.add(x.origin, s)), x.power_db, x.kind) for x in w.sources]
    w.receivers = [rooms.ReceiverSpec(tuple(np.add(x.origin, s)), x.radius) for x in w.receivers]
    w.cutoff_s = 0.5
    ds = tracer.DeviceScene(w.scene)
    ha, sa = tracer.trace(w, dscene=ds, rays=300, seed=8)
    hb, sb = tracer.trace(w, dscene=ds, rays=300, seed=8, traversal=1)
    assert abs(sa["segments"] - sb["segments"]) <= 1e-5 * sb["segments"]
    assert ha["energy"].sum() == pytest.approx(hb["energy"].sum(), rel=1e-4)
    assert sa["lost_energy"] == pytest.approx(sb["lost_energy"], rel=1e-3, abs=1e-5 * sb["initial_energy"])


@pytest.mark.parametrize("kind", ["hall", "map", "capture", "batch"])
@pytest.mark.parametrize("rays", [256, 257, 1001])
def test_primaries_shared_out_to_several_loops_equal_one_loop(kind, rays):
    """Above 256 primaries a run is shared out to loops with rings of their own; a given feed size keeps one.  The
    same rays, so the same terms in every bin (FP64 sums in another order: 1e-9; a primary's captures are FP32 sums
    of at most a thousand detections: 2 x 1000 x 2^-24)."""
    if kind == "batch":
        ws = [rooms.proposal_room_c4(20 + i) for i in range(4)]
        n = [rays, 1, rays // 2, 2]
    else:
        ws = [rooms.irregular_hall_c2(target_tris=2000)]
    kw = {}
    if kind == "map":
        lo, hi = ws[0].scene.bounds()
        org = rooms.audience_plane(lo[:2] + 2.0, hi[:2] - 2.0, 1.2, 2.0)
        kw["map_receivers"] = tracer.MapReceivers(org, 2.0, 400.0)
    elif kind == "capture":
        kw["capture"] = 2
    for w in ws:
        w.cutoff_s = 0.4
    ds = [tracer.DeviceScene(w.scene) for w in ws]
    got = []
    for feed in (0, 64):
        if kind == "batch":
            got.append(tracer.trace_batch(ws, dscenes=ds, rays=n, seed=6, feed_batch=feed))
        else:
            h, s = tracer.trace(ws[0], dscene=ds[0], rays=rays, seed=6, feed_batch=feed, **kw)
            got.append(([{**h, **{"map " + k: v for k, v in h.get("map", {}).items()}}], s))
    (ha, sa), (hb, sb) = got
    for name in ("primaries", "segments", "octave_rays", "end_traces", "detections", "queue_overflows"):
        assert sa[name] == sb[name], name
    assert sa["segments"] > 0 and sa["queue_overflows"] == 0
    for a, b in zip(ha, hb):
        assert "map energy" in a or kind != "map"
        for name, x in a.items():
            if isinstance(x, np.ndarray):
                rtol = 1.2e-4 if name == "capture" else 1e-9
                np.testing.assert_allclose(x, b[name], rtol=rtol, atol=1e-30, err_msg=name)


@pytest.mark.parametrize("bvh_format", [1, 2])
@pytest.mark.parametrize("tris,rays", [(84, 1), (84, 300), (2000, 5), (2000, 260), (5000, 40)])
def test_speculative_walk_finds_the_hits_of_the_plain_one(bvh_format, tris, rays):
    """Lanes that take rays together, from fewer rays than a warp to many, and both node forms: the same nearest hits
    as one leaf at a time, up to exact ties between triangles (a few rays in a million, as between the formats)."""
    w = rooms.irregular_hall_c2(target_tris=tris) if tris > 1000 else rooms.shoebox_c1()
    if tris <= 1000:
        w.scene = rooms._jittered_room(np.random.default_rng(2), (10.0, 8.0, 4.0), tris, 3, 0.0, (0.1, 0.4), (0.1, 0.5))
        assert w.scene.n_triangles > 64
    w.cutoff_s = 0.4
    ds = tracer.DeviceScene(w.scene)
    ha, sa = tracer.trace(w, dscene=ds, rays=rays, seed=3, bvh_format=bvh_format, traversal=1)
    hb, sb = tracer.trace(w, dscene=ds, rays=rays, seed=3, bvh_format=bvh_format, traversal=2)
    assert sb["primaries"] == rays and sb["queue_overflows"] == 0
    assert abs(sa["segments"] - sb["segments"]) <= 1e-4 * sa["segments"]
    assert hb["energy"].sum() == pytest.approx(ha["energy"].sum(), rel=1e-3)
