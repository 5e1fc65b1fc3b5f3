"""The node test of the traversal (near and far planes picked by the direction's sign) where it
can go wrong: directions with zero, negative-zero and vanishing components, origins on box
planes, rays without a direction, and trees whose last nodes have unused child slots. The BVH
only prunes, so closest and any-hit answers must equal the oracle's scans bit for bit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 1


def _edge_rays(tris, n, seed):
    rng = np.random.default_rng(seed)
    v = tris.reshape(-1, 3)
    o = v[rng.integers(0, len(v), n)].astype(np.float64)
    o[rng.random((n, 3)) < 0.5] += 0.75                      # the others stay on a vertex's (and a box's) plane
    o += rng.choice([0.0, -3.0, 3.0], (n, 3))
    d = rng.normal(0, 1, (n, 3))
    kind = rng.integers(0, 5, n)
    for k in range(n):
        if kind[k] == 0:                                     # one axis only, the others +0 or -0
            a = rng.integers(0, 3)
            d[k] = rng.choice([0.0, -0.0], 3)
            d[k, a] = rng.choice([-1.0, 1.0])
        elif kind[k] == 1:                                   # one zero component
            d[k, rng.integers(0, 3)] = rng.choice([0.0, -0.0])
        elif kind[k] == 2:                                   # one vanishing component, denormals among them
            d[k, rng.integers(0, 3)] = rng.choice([1e-30, -1e-38, 1e-42])
        elif kind[k] == 3 and k % 8 == 0:                    # no direction at all
            d[k] = 0.0
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 9, 17, 400])
def test_axis_parallel_and_degenerate_rays(rn, oracle, n):
    rng = np.random.default_rng(100 + n)
    # vertices on a coarse grid: many boxes share planes, many triangles are flat in one axis
    tris = rng.integers(-4, 5, (n, 9)).astype(np.float32)
    rays = _edge_rays(tris, 6000, n)
    tmax = np.where(rng.random(len(rays)) < 0.3, rng.uniform(0.5, 6.0, len(rays)), 1e30).astype(np.float32)
    acc = rn.LinearAccel(tris)
    tri, t = rn.closest(acc, rays, tmax)
    rtri, rt = oracle.closest_scan(tris, rays, tmax, threads=THREADS)
    assert np.array_equal(tri, rtri), int((tri != rtri).sum())
    assert np.array_equal(t, rt)
    assert np.array_equal(rn.occluded(acc, rays, tmax) != 0, tri >= 0)


@pytest.mark.parametrize("spp", [1, 16, 40])
def test_frontier_groups_against_the_scan(rn, oracle, spp):
    """AO-only walks start from the warp's frontier, tested in groups of four with the last one
    padded: against the oracle's trace on a scene dense enough to fill it."""
    import scene as scenes
    sc = scenes.build_synthetic_scene(3, 60, 10, grid=20, half=8.0, subdiv=2)
    cam = (6.0, 4.0, 5.0, 0.0, 0.5, 0.0, 0.0, 1.0, 0.0, 0.9)
    _, pos, nrm, mask = oracle.rasterize(sc.tris, sc.normals, cam, 75, 53)
    acc = rn.LinearAccel(sc.tris)
    for radius in (0.05, 1.0):
        ao = rn.compute_rtao(rn.GBuffer(pos, nrm, mask), acc, spp, radius)
        ref = oracle.trace(pos, nrm, mask, sc.tris, spp, radius, threads=THREADS)
        ref = ref[0] if isinstance(ref, tuple) else ref
        assert np.array_equal(ao, ref), int((ao != ref).sum())


@pytest.mark.parametrize("spp", [1, 63, 64, 65, 130])
def test_sieve_chunks_against_the_scan(rn, oracle, spp):
    """Sample counts around the sieve's 64-sample chunks (the sun's slot falls into the last one
    or opens another), in a frame whose packets are ragged at the right and lower edge."""
    import scene as scenes
    sc = scenes.build_test_scene()
    _, pos, nrm, mask = oracle.rasterize(sc.tris, sc.normals, sc.camera, 61, 43)
    acc = rn.LinearAccel(sc.tris)
    g = rn.GBuffer(pos, nrm, mask)
    ao, sky, sun = rn.compute_rt_visibility(g, acc, spp, 2.0, to_light=sc.to_light)
    rao, rsky, rsun = oracle.trace(pos, nrm, mask, sc.tris, spp, 2.0, to_light=sc.to_light, threads=THREADS)
    assert np.array_equal(ao, rao) and np.array_equal(sky, rsky) and np.array_equal(sun, rsun)
    assert np.array_equal(rn.compute_rtao(g, acc, spp, 2.0), rao)


@pytest.mark.parametrize("spp", [15, 16, 17, 31, 32, 33, 37, 65, 130, 257])
@pytest.mark.parametrize("small", [True, False])
def test_small_frames_share_a_pixels_samples(rn, oracle, small, spp):
    """Frames of few packets give a pixel's samples to two lanes (from 16 samples) or four (from
    32), a run each, the last one shorter, the sun ray with the first: the oracle's AO, sky and sun
    bit for bit, on a small tree and a deeper one, in ragged frames and packets of 4, 8 and 16
    columns."""
    import scene as scenes
    if small:
        sc = scenes.build_test_scene()
        cam = sc.camera
    else:
        sc = scenes.build_synthetic_scene(5, 60, 10, grid=20, half=8.0, subdiv=2)
        cam = (6.0, 4.0, 5.0, 0.0, 0.5, 0.0, 0.0, 1.0, 0.0, 0.9)
    tl = (0.3, 0.8, -0.5)
    acc = rn.LinearAccel(sc.tris)
    saved = rn.tune_get("trace_packet")
    try:
        for (w, h), packet in (((61, 43), 8), ((17, 9), 4), ((33, 3), 16)):
            rn.tune_set("trace_packet", packet)
            _, pos, nrm, mask = oracle.rasterize(sc.tris, sc.normals, cam, w, h)
            g = rn.GBuffer(pos, nrm, mask)
            want = oracle.trace(pos, nrm, mask, sc.tris, spp, 1.0, to_light=tl, threads=THREADS)
            got = rn.compute_rt_visibility(g, acc, spp, 1.0, to_light=tl)
            for a, b in zip(got, want):
                assert np.array_equal(a, b), (w, h, int((a != b).sum()))
            assert np.array_equal(rn.compute_rtao(g, acc, spp, 1.0), want[0])
    finally:
        rn.tune_set("trace_packet", saved)


@pytest.mark.parametrize("scale", [1.0, 1e-4, 1e5])
@pytest.mark.parametrize("length", [1.0, 2e-3, 1e-3, 5e-4, 1e-25])
def test_rays_along_axes_and_planes(rn, oracle, scale, length):
    """Directions with one or two zero components (and of every size around the node test's line
    for short ones) from origins on and off vertices' coordinates, over a soup of several levels at
    three scales: closest and any-hit answers are the oracle's scans."""
    rng = np.random.default_rng(7)
    tris = (oracle.soup(3000, 11) * np.float32(scale)).astype(np.float32)
    v = tris.reshape(-1, 3)
    n = 3000
    o = v[rng.integers(0, len(v), n)].copy()
    off = rng.random((n, 3)) < 0.5
    o[off] += (rng.normal(0, 2.0, (n, 3)) * scale).astype(np.float32)[off]
    d = rng.normal(0, 1, (n, 3))
    d[np.arange(n), rng.integers(0, 3, n)] = 0.0
    two = rng.random(n) < 0.5
    d[two, rng.integers(0, 3, n)[two]] = -0.0
    d /= np.maximum(np.abs(d).max(1, keepdims=True), 1e-6)
    rays = np.concatenate([o, d * length], 1).astype(np.float32)
    tmax = np.where(rng.random(n) < 0.3, 3.0 * scale / length, 1e30).astype(np.float32)
    acc = rn.LinearAccel(tris)
    tri, t = rn.closest(acc, rays, tmax)
    rtri, rt = oracle.closest_scan(tris, rays, tmax, threads=THREADS)
    assert np.array_equal(tri, rtri), int((tri != rtri).sum())
    assert np.array_equal(t, rt)
    assert np.array_equal(rn.occluded(acc, rays, tmax) != 0, oracle.occluded_scan(tris, rays, tmax, threads=THREADS) != 0)


@pytest.mark.parametrize("log2", [34, 40, 42])
@pytest.mark.parametrize("length", [1.0, 5e-4])
def test_rays_along_axes_far_from_the_origin(rn, oracle, log2, length):
    """The same at coordinates of 2e11 to 6e13, where a coordinate times the reciprocal of a zero
    component leaves float's range. The scales are powers of two: the vertices stay exact."""
    scale = np.float32(2.0 ** log2)
    rng = np.random.default_rng(9)
    tris = oracle.soup(2000, 12) * scale
    n = 3000
    o = tris.reshape(-1, 3)[rng.integers(0, 3 * len(tris), n)].copy()
    off = rng.random((n, 3)) < 0.5
    o[off] += (rng.normal(0, 2.0, (n, 3)) * scale).astype(np.float32)[off]
    d = rng.normal(0, 1, (n, 3))
    d[np.arange(n), rng.integers(0, 3, n)] = 0.0
    two = rng.random(n) < 0.5
    d[two, rng.integers(0, 3, n)[two]] = -0.0
    d /= np.maximum(np.abs(d).max(1, keepdims=True), 1e-6)
    rays = np.concatenate([o, d * length], 1).astype(np.float32)
    tmax = np.where(rng.random(n) < 0.3, 3.0 * scale / length, 1e30).astype(np.float32)
    acc = rn.LinearAccel(tris)
    tri, t = rn.closest(acc, rays, tmax)
    rtri, rt = oracle.closest_scan(tris, rays, tmax, threads=THREADS)
    assert (rtri >= 0).sum() > n // 20
    assert np.array_equal(tri, rtri), int((tri != rtri).sum())
    assert np.array_equal(t, rt)
    assert np.array_equal(rn.occluded(acc, rays, tmax) != 0, oracle.occluded_scan(tris, rays, tmax, threads=THREADS) != 0)


@pytest.mark.parametrize("log2", [34, 40])
def test_frame_far_from_the_origin(rn, oracle, log2):
    """AO, sky and a sun with a zero component over the built-in scene at such coordinates: the
    oracle's planes bit for bit. The positions lie 1/16 off the surface: on it the rounding of t alone
    decides whether a ray hits its own triangle."""
    import scene as scenes
    sc = scenes.build_test_scene()
    _, pos, nrm, mask = oracle.rasterize(sc.tris, sc.normals, sc.camera, 61, 43)
    scale = np.float32(2.0 ** log2)
    tris, pos = sc.tris * scale, (pos + nrm / 16) * scale
    acc = rn.LinearAccel(tris)
    g = rn.GBuffer(pos, nrm, mask)
    for sun in ((0.9, 0.5, 0.0), (0.0, 0.5, 0.9)):
        want = oracle.trace(pos, nrm, mask, tris, 65, 2.0 * scale, to_light=sun, accel="scan", threads=THREADS)
        assert (want[2][mask != 0] == 0).sum() > 10
        got = rn.compute_rt_visibility(g, acc, 65, 2.0 * scale, to_light=sun)
        for a, b in zip(got, want):
            assert np.array_equal(a, b), int((a != b).sum())
    saved = {k: rn.tune_get(k) for k in ("trace_pool", "trace_frontier")}
    try:
        for pool in (0, 24):
            for frontier in (0, 1):
                rn.tune_set("trace_pool", pool)
                rn.tune_set("trace_frontier", frontier)
                assert np.array_equal(rn.compute_rtao(g, acc, 65, 2.0 * scale), want[0]), (pool, frontier)
    finally:
        for k, v in saved.items():
            rn.tune_set(k, v)


def _chain(n):
    """Triangles around the origin, each 1.5 times as large as the last: a tree of one interior child a
    node, n / 3 levels deep."""
    s = 1.5 ** (np.arange(n) - n + 5.0)
    tris = np.zeros((n, 3, 3))
    for k in range(3):
        tris[:, k, k] = s
    return tris.reshape(n, 9).astype(np.float32)


@pytest.mark.parametrize("n", [24, 30, 33, 60, 75, 78, 80, 81, 90])
def test_deep_trees_trace_from_the_frontier(rn, oracle, n):
    """Trees of 8 to 30 levels, around the depths at which the frontier's entries and the walk's own
    no longer fit into stacks of 48 (past 10 levels) and 96 (past 26, where walks start at the
    root): the oracle's scan bit for bit, and fewer node visits than from the root wherever the
    frontier runs."""
    tris = _chain(n)
    rng = np.random.default_rng(n)
    h, w = 13, 29
    pos = (rng.uniform(0.6, 1.0, (h, w, 1)) * np.ones(3) * 1.5 ** 4).astype(np.float32)
    nrm = np.full((h, w, 3), -1 / np.sqrt(3), np.float32)
    mask = np.ones((h, w), np.uint8)
    g = rn.GBuffer(pos, nrm, mask)
    acc = rn.LinearAccel(tris)
    keys = ("trace_stack", "trace_frontier", "trace_frontier_min_spp", "trace_pool")
    saved = {k: rn.tune_get(k) for k in keys}
    try:
        rn.tune_set("trace_frontier_min_spp", 1)
        for radius in (0.5, 3.0):
            want = oracle.trace(pos, nrm, mask, tris, 15, radius, accel="scan", threads=THREADS)
            nodes = {}
            for stack in (48, 96):
                for frontier in (0, 1):
                    for pool in (0, 24):
                        rn.tune_set("trace_stack", stack)
                        rn.tune_set("trace_frontier", frontier)
                        rn.tune_set("trace_pool", pool)
                        assert np.array_equal(rn.compute_rtao(g, acc, 15, radius), want), (stack, frontier, pool)
                    nodes[frontier] = rn.trace_stats(g, acc, 15, radius)["nodes"]
            if n <= 80:
                assert nodes[1] < nodes[0], nodes
            else:
                assert nodes[1] == nodes[0], nodes
    finally:
        for k, v in saved.items():
            rn.tune_set(k, v)


@pytest.mark.parametrize("spp", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("small", [True, False])
def test_few_samples_against_the_scan(rn, oracle, small, spp):
    """One and two samples a pixel run without the sieve, and up to three cap the frontier at four
    entries a sample: the oracle's AO, sky and sun bit for bit, in ragged frames, packets of 4, 8
    and 16 columns, with the frontier on and off, and as a view of a batch."""
    import scene as scenes
    import torch
    if small:
        sc = scenes.build_test_scene()
        cam = sc.camera
    else:
        sc = scenes.build_synthetic_scene(5, 60, 10, grid=20, half=8.0, subdiv=2)
        cam = (6.0, 4.0, 5.0, 0.0, 0.5, 0.0, 0.0, 1.0, 0.0, 0.9)
    tl = (0.3, 0.8, -0.5)
    acc = rn.LinearAccel(sc.tris)
    keys = ("trace_packet", "trace_frontier", "trace_frontier_min_spp")
    saved = {k: rn.tune_get(k) for k in keys}
    try:
        rn.tune_set("trace_frontier_min_spp", 1)
        for (w, h), packet in (((61, 43), 8), ((17, 9), 4), ((33, 3), 16)):
            rn.tune_set("trace_packet", packet)
            _, pos, nrm, mask = oracle.rasterize(sc.tris, sc.normals, cam, w, h)
            g = rn.GBuffer(pos, nrm, mask)
            want = oracle.trace(pos, nrm, mask, sc.tris, spp, 1.0, to_light=tl, threads=THREADS)
            for frontier in (0, 1):
                rn.tune_set("trace_frontier", frontier)
                got = rn.compute_rt_visibility(g, acc, spp, 1.0, to_light=tl)
                for a, b in zip(got, want):
                    assert np.array_equal(a, b), (w, h, frontier, int((a != b).sum()))
                assert np.array_equal(rn.compute_rtao(g, acc, spp, 1.0), want[0]), (w, h, frontier)
            dg = rn.GBuffer(*[torch.from_numpy(t).cuda() for t in (pos, nrm, mask)])
            dacc = rn.LinearAccel(torch.from_numpy(sc.tris).cuda())
            batch = rn.Batch(dacc, [dict(g=dg, spp=spp, radius=1.0, ssao=False)])
            batch.run()
            assert np.array_equal(batch.outputs[0]["ao"].cpu().numpy(), want[0]), (w, h)
            batch.close()
    finally:
        for k, v in saved.items():
            rn.tune_set(k, v)


@pytest.mark.parametrize("spp", [1, 4, 5, 7, 8, 9])
@pytest.mark.parametrize("boxes", [0, 8, 60, 900])
def test_few_samples_within_a_short_reach(rn, oracle, boxes, spp):
    """AO from the frontier at the largest numbers of samples that run without the sieve (4, and 8 in
    trees of six levels and more) and the smallest beyond, for radii from nothing within reach to
    the whole scene, nodes of fewer than four children among those fetched: the oracle's AO bit for
    bit."""
    import scene as scenes
    if boxes == 0:
        sc = scenes.build_test_scene()
        cam = sc.camera
    else:
        sc = scenes.build_synthetic_scene(5, boxes, boxes // 6, grid=20, half=8.0, subdiv=2)
        cam = (6.0, 4.0, 5.0, 0.0, 0.5, 0.0, 0.0, 1.0, 0.0, 0.9)
    acc = rn.LinearAccel(sc.tris)
    _, pos, nrm, mask = oracle.rasterize(sc.tris, sc.normals, cam, 61, 43)
    g = rn.GBuffer(pos, nrm, mask)
    keys = ("trace_frontier", "trace_frontier_min_spp")
    saved = {k: rn.tune_get(k) for k in keys}
    try:
        rn.tune_set("trace_frontier", 1)
        rn.tune_set("trace_frontier_min_spp", 1)
        for radius in (0.005, 0.05, 0.4, 40.0):
            want = oracle.trace(pos, nrm, mask, sc.tris, spp, radius, threads=THREADS)
            assert np.array_equal(rn.compute_rtao(g, acc, spp, radius), want), radius
    finally:
        for k, v in saved.items():
            rn.tune_set(k, v)
