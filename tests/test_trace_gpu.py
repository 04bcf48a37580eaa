"""Parity of the CUDA ray-tracing path with the oracle (GPU).

Every comparison is bit-exact: hit triangle ids, hit distances (as bit
patterns) and image bytes. The oracle itself is pinned against the reference
(test_oracle_golden.py), and the full-size cases are also checked against the
digests the reference produced (tests/golden/golden_hashes.json)."""
import json
import os

import numpy as np
import pytest

from golden_util import sha
from nostrum_pray_gb300 import native, scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    native.lib()
    torch.cuda.set_device(0)


def render(sc, setup):
    h, w = setup.height, setup.width
    rgb = torch.empty((h, w, 3), dtype=torch.uint8, device="cuda")
    ids = torch.empty((h, w), dtype=torch.int32, device="cuda")
    ts = torch.empty((h, w), dtype=torch.float32, device="cuda")
    cnt = torch.zeros(2, dtype=torch.int64, device="cuda")
    sc.render_rt(setup, rgb, ids, ts, cnt)
    torch.cuda.synchronize()
    return rgb.cpu().numpy(), ids.cpu().numpy().reshape(-1), ts.cpu().numpy().reshape(-1), cnt.cpu().numpy()


def trace(sc, rays, eps):
    r = torch.from_numpy(np.ascontiguousarray(rays, np.float32)).cuda()
    n = rays.shape[0]
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    ts = torch.empty(n, dtype=torch.float32, device="cuda")
    sc.trace_closest(r, eps, ids, ts)
    torch.cuda.synchronize()
    return ids.cpu().numpy(), ts.cpu().numpy()


def check_frame(oracle, mesh, setup, traversal=native.TRAVERSAL_AUTO):
    sc = native.Scene.from_setup(mesh, setup)
    sc.set_traversal(traversal)
    img, ids, ts, cnt = render(sc, setup)
    orc = oracle.OracleScene.from_setup(mesh, setup)
    want_img, want_sh = orc.render_rt(setup)
    rays = oracle.primary_rays(setup.width, setup.height, setup.fov, setup.cam_pos, setup.cam_look)
    want_ids, want_t = orc.trace(rays, setup.det_eps)
    mism = int((ids != want_ids.astype(np.int32)).sum())
    assert mism == 0, f"{mism} hit ids differ"
    np.testing.assert_array_equal(ts.view(np.uint32), want_t.view(np.uint32))
    np.testing.assert_array_equal(img, want_img)
    assert int(cnt[0]) == setup.width * setup.height
    assert int(cnt[1]) == want_sh
    # host-memory entry point gives the same frame
    himg, rays_cast = sc.render_rt_host(setup)
    np.testing.assert_array_equal(himg, want_img)
    assert int(rays_cast[1]) == want_sh
    return img, ids, ts


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_soup_frame(oracle, seed):
    check_frame(oracle, scenes.soup(10_000, seed), scenes.soup_setup())


@pytest.mark.parametrize("traversal", [native.TRAVERSAL_LANES, native.TRAVERSAL_PACKETS,
                                       native.TRAVERSAL_PRIMARY_PACKETS])
@pytest.mark.parametrize("scene", ["soup", "sphere", "sah_soup", "far_camera"])
def test_frame_traversals(oracle, traversal, scene):
    """Each traversal of the ray-traced frame (per lane; warp packets over a
    pixel tile for the primary and occlusion rays, or for the primary rays
    only) gives the oracle's frame: hit ids, distances, image. The distant
    camera's rays take the exact node copy, which packet warps leave to the
    per-lane walk."""
    if scene == "soup":
        m, st = scenes.soup(10_000, 3), scenes.soup_setup(256, 192)
    elif scene == "sphere":
        m, st = scenes.icosphere(6), scenes.icosphere_setup(320, 240)
    elif scene == "sah_soup":
        m, st = scenes.soup(10_000, 4), scenes.soup_setup(320, 240)
        st.tree, st.leaf_size, st.max_depth, st.sah_ct = "sah", 32, 20, 1.0
    else:
        m, st = scenes.soup(10_000, 5), scenes.soup_setup(160, 120)
        st.cam_pos, st.fov = (0.5, 0.5, -30.0), 3
    check_frame(oracle, m, st, traversal)


def test_traversal_choice():
    """AUTO picks one of the traversals on the first frame and keeps it; an
    explicit choice is kept as given."""
    m, st = scenes.soup(2_000, 1), scenes.soup_setup(64, 64)
    sc = native.Scene.from_setup(m, st)
    assert sc.traversal() == native.TRAVERSAL_AUTO
    sc.render_rt_host(st)
    assert sc.traversal() in (native.TRAVERSAL_LANES, native.TRAVERSAL_PACKETS, native.TRAVERSAL_PRIMARY_PACKETS)
    sc.set_traversal(native.TRAVERSAL_PACKETS)
    sc.render_rt_host(st)
    assert sc.traversal() == native.TRAVERSAL_PACKETS
    with pytest.raises(native.PrayError):
        sc.set_traversal(5)


def test_soup_sah_default_constants(oracle):
    st = scenes.soup_setup(320, 240)
    st.tree, st.leaf_size, st.max_depth = "sah", 32, 20
    check_frame(oracle, scenes.soup(10_000, 4), st)


@pytest.mark.parametrize("eps", [0.0, 1e-4])
def test_icosphere_level5(oracle, golden, eps):
    hashes, small = golden
    st = scenes.icosphere_setup(480, 270, det_eps=eps)
    img, ids, ts = check_frame(oracle, scenes.icosphere(5), st)
    key = f"ico5_eps{eps:g}"
    assert sha(img) == hashes[key]["image"]  # the reference's own frame
    assert sha(ids) == hashes[key]["ids"] and sha(ts) == hashes[key]["t"]


@pytest.mark.parametrize("name", ["cube", "head_fov30", "plant"])
def test_examples(oracle, golden, name):
    hashes, small = golden
    info = small[f"ex_{name}_info"]
    m = scenes.Mesh(small[f"ex_{name}_verts"], small[f"ex_{name}_colors"], small[f"ex_{name}_emit"])
    st = scenes.RenderSetup(width=160, height=120, fov=int(info[2]), cam_pos=tuple(info[6:9]),
                            cam_look=tuple(info[9:12]), lights=[tuple(l) for l in small[f"ex_{name}_lights"]],
                            background=tuple(info[12:15]), tree="median")
    img, _, _ = check_frame(oracle, m, st)
    np.testing.assert_array_equal(img, small[f"ex_{name}_image160"])


def test_random_rays_inside_scene(oracle):
    """Rays from inside the soup in random directions, including exact axis
    directions and zero components (infinite inverse directions)."""
    m = scenes.soup(10_000, 5)
    st = scenes.soup_setup()
    sc = native.Scene.from_setup(m, st)
    orc = oracle.OracleScene.from_setup(m, st)
    rng = np.random.default_rng(0)
    n = 200_000
    o = rng.uniform(-0.2, 1.2, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[: n // 10, 1:] = 0.0          # +-x axis rays
    d[n // 10: n // 5, 0] = 0.0      # rays in the yz plane
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    with np.errstate(divide="ignore"):
        inv = (1.0 / d).astype(np.float32)
    rays = np.concatenate([o, d, inv], 1)
    for eps in (1e-4, 0.0):
        ids, ts = trace(sc, rays, eps)
        wid, wt = orc.trace(rays, eps)
        assert int((ids != wid.astype(np.int32)).sum()) == 0
        np.testing.assert_array_equal(ts.view(np.uint32), wt.view(np.uint32))


@pytest.mark.parametrize("tree", ["median", "sah"])
def test_occlusion_rays(oracle, tree):
    """pray_trace_occluded against the reference's shadow test on the
    oracle's closest hits (occluded iff a hit with dist2 > t * t,
    src/pray.cpp:39-43): random rays inside the soup with distances around
    their closest hits, including dist2 exactly t * t (not occluded), the
    next float above it (occluded), zero, negative and infinite."""
    m = scenes.soup(10_000, 6)
    st = scenes.soup_setup()
    st.tree = tree
    sc = native.Scene.from_setup(m, st)
    orc = oracle.OracleScene.from_setup(m, st)
    rng = np.random.default_rng(3)
    n = 120_000
    o = rng.uniform(-0.2, 1.2, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[: n // 20, 1:] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    with np.errstate(divide="ignore"):
        inv = (1.0 / d).astype(np.float32)
    rays = np.concatenate([o, d, inv], 1).astype(np.float32)
    for eps in (1e-4, 0.0):
        wid, wt = orc.trace(rays, eps)
        hit = wid >= 0
        tt = np.where(hit, wt, 1.0).astype(np.float32)
        t2 = (tt * tt).astype(np.float32)
        kind = rng.integers(0, 7, n)
        dist2 = np.select([kind == 0, kind == 1, kind == 2, kind == 3, kind == 4, kind == 5],
                          [t2, np.nextafter(t2, np.float32(np.inf)), np.float32(0), np.float32(-1),
                           np.float32(np.inf), t2 * np.float32(0.25)],
                          rng.uniform(0, 4, n).astype(np.float32) * t2).astype(np.float32)
        want = (hit & (dist2 > t2)).astype(np.uint8)
        r = torch.from_numpy(rays).cuda()
        dd = torch.from_numpy(dist2).cuda()
        occ = torch.empty(n, dtype=torch.uint8, device="cuda")
        sc.trace_occluded(r, dd, eps, occ)
        torch.cuda.synchronize()
        got = occ.cpu().numpy()
        assert int((got != want).sum()) == 0, f"{int((got != want).sum())} occlusion answers differ"
        assert 0 < int(want.sum()) < n


def test_ties_duplicated_triangles(oracle):
    """Coincident copies of each triangle: equal distances, so the first in
    the reference's depth-first order must win."""
    base = scenes.soup(3_000, 9)
    m = scenes.Mesh(np.concatenate([base.verts, base.verts[::-1]]), np.concatenate([base.colors, base.colors]),
                    np.zeros(6_000, np.uint8))
    for tree in ("median", "sah"):
        st = scenes.soup_setup(256, 256)
        st.tree = tree
        check_frame(oracle, m, st)


def test_empty_and_tiny_scenes(oracle):
    st = scenes.soup_setup(33, 17)  # ragged size: partial 8x4 tiles
    st.background = (0.25, 0.5, 1.0)
    empty = scenes.Mesh(np.zeros((0, 9), np.float32), np.zeros((0, 3), np.float32), np.zeros(0, np.uint8))
    sc = native.Scene.from_setup(empty, st)
    img, _ = sc.render_rt_host(st)
    want = np.array([int(np.float32(c) * np.float32(255) + np.float32(0.5)) for c in st.background], np.uint8)
    assert (img == want).all()
    one = scenes.Mesh(np.array([[0, 0, 0, 1, 0, 0, 0, 1, 0]], np.float32) + np.float32(0.5) * 0,
                      np.array([[0.5, 0.6, 0.7]], np.float32), np.zeros(1, np.uint8))
    st2 = scenes.RenderSetup(width=64, height=48, fov=60, cam_pos=(0.2, 0.2, -2.0), cam_look=(0, 0, 1),
                             lights=[(0.2, 0.2, -1.0, 1, 1, 1)])
    check_frame(oracle, one, st2)


def test_invalid_arguments_raise():
    st = scenes.soup_setup(16, 16)
    m = scenes.soup(100, 0)
    with pytest.raises(native.PrayError):
        native.Scene(m, native.tree_options(st, max_depth=31))
    sc = native.Scene.from_setup(m, st)
    bad = scenes.soup_setup(0, 16)
    with pytest.raises(native.PrayError):
        sc.render_rt_host(bad)


@pytest.mark.slow
def test_icosphere_level8_full(oracle, golden):
    """The 1.31M-triangle displaced sphere at 1920x1080 with the SAH tree:
    GPU frame == oracle frame == the reference's frame (digests)."""
    hashes, _ = golden
    m = scenes.icosphere(8)
    for eps in (0.0, 1e-4):
        st = scenes.icosphere_setup(det_eps=eps)
        img, ids, ts = check_frame(oracle, m, st)
        key = f"ico8_eps{eps:g}"
        assert sha(img) == hashes[key]["image"]
        assert sha(ids) == hashes[key]["ids"] and sha(ts) == hashes[key]["t"]


def test_rays_through_vertices_and_edges(oracle):
    """Rays aimed at triangle vertices, edge midpoints and edge thirds (u or v
    at or next to 0 and 1, u + v at 1): the intersector's early outs must
    decide exactly as the reference's full computation."""
    m = scenes.soup(4_000, 12)
    st = scenes.soup_setup()
    sc = native.Scene.from_setup(m, st)
    orc = oracle.OracleScene.from_setup(m, st)
    rng = np.random.default_rng(5)
    v = m.verts.reshape(-1, 3, 3).astype(np.float64)
    tri = rng.integers(0, m.n, 60_000)
    which = rng.integers(0, 6, tri.size)
    a, b, c = v[tri, 0], v[tri, 1], v[tri, 2]
    targets = np.where((which == 0)[:, None], a, np.where((which == 1)[:, None], b, np.where(
        (which == 2)[:, None], c, np.where((which == 3)[:, None], (a + b) / 2, np.where(
            (which == 4)[:, None], (b + c) / 2, a + (c - a) / 3)))))
    o = rng.uniform(-1.0, 2.0, (tri.size, 3))
    d = targets - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d = d.astype(np.float32)
    with np.errstate(divide="ignore"):
        rays = np.concatenate([o.astype(np.float32), d, (1.0 / d).astype(np.float32)], 1)
    for eps in (1e-4, 0.0):
        ids, ts = trace(sc, rays, eps)
        wid, wt = orc.trace(rays, eps)
        assert int((ids != wid.astype(np.int32)).sum()) == 0
        np.testing.assert_array_equal(ts.view(np.uint32), wt.view(np.uint32))


@pytest.mark.parametrize("dist", [0.3, 1.5, 3.5, 6.0, 100.0, 3000.0])
def test_distant_origins(oracle, dist):
    """Rays from origins `dist` scene diagonals from the scene's centre (from
    inside the scene to far beyond the reach of the padded culling boxes,
    where the exact node copy serves them), aimed at a cluster of small
    triangles next to the world origin inside a scene of large ones: the
    float error of a slab test grows with the distance travelled, not with
    the small boxes' coordinates."""
    rng = np.random.default_rng(int(dist * 10))
    small = scenes.soup(20_000, 7)
    big = scenes.soup(300, 8, spread=0.05)
    m = scenes.Mesh(np.concatenate([small.verts * np.float32(0.02), big.verts * np.float32(2) - np.float32(1)]),
                    np.concatenate([small.colors, big.colors]), np.zeros(20_300, np.uint8))
    st = scenes.room_setup(64, 64)
    sc = native.Scene.from_setup(m, st)
    orc = oracle.OracleScene.from_setup(m, st)
    v = m.verts.reshape(-1, 3).astype(np.float64)
    lo, hi = v.min(0), v.max(0)
    centre, diag = (lo + hi) / 2, float(np.linalg.norm(hi - lo))
    n = 60_000
    u = rng.normal(size=(n, 3))
    o = centre + dist * diag * u / np.linalg.norm(u, axis=1, keepdims=True)
    tgt = np.where((rng.random(n) < 0.7)[:, None], rng.uniform(-0.001, 0.021, (n, 3)), rng.uniform(lo, hi, (n, 3)))
    o = o.astype(np.float32)
    d = (tgt - o.astype(np.float64))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    rays = np.concatenate([o, d, (1.0 / d).astype(np.float32)], 1)
    ids, ts = trace(sc, rays, 0.0)
    wid, wt = orc.trace(rays, 0.0)
    assert (wid >= 0).sum() > n // 3
    assert int((ids != wid.astype(np.int32)).sum()) == 0
    np.testing.assert_array_equal(ts.view(np.uint32), wt.view(np.uint32))


def test_host_rays_from_many_threads(oracle):
    """pray_trace_closest_host, the entry point behind the reference-side
    SpatialDatabase::intersect binding: host rays in, host ids and distances
    out, called concurrently from eight host threads on one scene (the
    reference's renderers query the database from OpenMP threads), with
    batches of one ray up to whole frames; bit-exact against the oracle."""
    from concurrent.futures import ThreadPoolExecutor
    mesh = scenes.soup(10_000, 2)
    st = scenes.soup_setup(96, 80)
    sc = native.Scene.from_setup(mesh, st)
    rays = oracle.primary_rays(st.width, st.height, st.fov, st.cam_pos, st.cam_look)
    want_ids, want_t = oracle.OracleScene.from_setup(mesh, st).trace(rays, st.det_eps)
    sizes = [1, 7, 64, 1000, rays.shape[0]]

    def job(k):
        n = sizes[k % len(sizes)]
        lo = (k * 977) % (rays.shape[0] - n + 1)
        ids, ts = sc.trace_closest_host(rays[lo:lo + n], st.det_eps)
        return lo, n, ids, ts

    with ThreadPoolExecutor(8) as ex:
        results = list(ex.map(job, range(64)))
    for lo, n, ids, ts in results:
        np.testing.assert_array_equal(ids, want_ids[lo:lo + n].astype(np.int32))
        np.testing.assert_array_equal(ts.view(np.uint32), want_t[lo:lo + n].view(np.uint32))
    assert int((want_ids >= 0).sum()) > 500
    ids, ts = sc.trace_closest_host(rays[:0], st.det_eps)
    assert ids.size == 0
    sc.close()


def _hard_rays(mesh, seed, n):
    """Rays that culling gets wrong first: at vertices, edge midpoints and
    interior points of triangles (ties at shared edges) from around and inside
    the scene, near-axis and axis-parallel directions, and random ones."""
    rng = np.random.default_rng(seed)
    v = mesh.verts.reshape(-1, 3, 3).astype(np.float64)
    lo, hi = v.min((0, 1)), v.max((0, 1))
    size = max(float(np.linalg.norm(hi - lo)), 1e-3)
    t = v[rng.integers(0, len(v), n)]
    w = rng.dirichlet((1, 1, 1), n)
    kind = rng.integers(0, 4, n)
    w[kind == 0] = np.eye(3)[rng.integers(0, 3, (kind == 0).sum())]
    w[kind == 1] = (0.5, 0.5, 0.0)
    p = np.einsum("nk,nkc->nc", w, t)
    o = rng.uniform(lo - size, hi + size, (n, 3))
    d = p - o
    d[kind == 3] = rng.normal(size=((kind == 3).sum(), 3))
    axis = rng.integers(0, 8, n) == 0  # nearly or exactly parallel to an axis
    d[axis] = np.eye(3)[rng.integers(0, 3, axis.sum())] * size
    d[axis] += rng.normal(size=(axis.sum(), 3)) * rng.choice([0.0, 1e-7, 1e-3], (axis.sum(), 1)) * size
    o[axis] = p[axis] - 1.5 * d[axis]
    d32 = (d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)).astype(np.float32)
    with np.errstate(divide="ignore"):
        return np.concatenate([o.astype(np.float32), d32, np.float32(1.0) / d32], 1)


def _well_posed(mesh, rays):
    """Rays within the culling pad's bound (host/flatten.cpp): sin a sin b of at
    least 1/50 (a the smallest angle, b the ray's angle to the plane) for
    every triangle that the ray's line passes through or within a hundredth
    of its size, and no zero-area triangle within that of the line. Outside it
    a reported distance can lie anywhere, and any walk that skips boxes beyond
    the best hit may miss the reference's choice."""
    v = mesh.verts.reshape(-1, 3, 3).astype(np.float64)
    a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = np.cross(e1, e2)
    area = np.linalg.norm(n, axis=1)
    e = np.sort(np.stack([np.linalg.norm(x, axis=1) for x in (e1, e2, e2 - e1)]), 0)
    sin_a = area / np.maximum(e[1] * e[2], 1e-300)
    ok = np.ones(len(rays), bool)
    for i in range(0, len(rays), 500):
        o, d = rays[i:i + 500, 0:3].astype(np.float64), rays[i:i + 500, 3:6].astype(np.float64)
        sin_b = np.abs(d @ n.T) / np.maximum(area, 1e-300)
        # distance of the line to the triangle's plane section: barycentrics of the line's closest approach
        p = np.cross(d[:, None], e2[None])
        det = np.einsum("rtc,tc->rt", p, e1)
        t = o[:, None] - a[None]
        u = np.einsum("rtc,rtc->rt", t, p)
        w = np.einsum("rc,rtc->rt", d, np.cross(t, e1[None]))
        # the line's distance to the triangle's centroid against its size
        c = v.mean(1)[None] - o[:, None]
        dist = np.linalg.norm(c - np.einsum("rtc,rc->rt", c, d)[..., None] * d[:, None], axis=2)
        near = dist <= e[2] * (2 / 3) * 1.01
        with np.errstate(divide="ignore", invalid="ignore"):
            u, w = u / det, w / det
            inside = (u > -0.01) & (w > -0.01) & (u + w < 1.01)
        posed = sin_a * sin_b >= 1 / 50
        ok[i:i + 500] = ~(near & ~posed & (inside | (sin_b < 1 / 50) | (sin_a[None] < 1 / 50))).any(1)
    return ok


def _hard_mesh(name):
    rng = np.random.default_rng(5)
    if name == "one":
        v = rng.uniform(-1, 1, (1, 9))
    elif name == "copies":  # one triangle 40 times (equal centres), a few others
        v = np.concatenate([np.repeat(rng.uniform(-1, 1, (1, 9)), 40, 0), rng.uniform(-1, 1, (9, 9))])
    elif name == "layers":  # a quad grid twice in the same plane: every hit is a tie
        g = scenes._quad_grid((-1, -1, 0), (2, 0, 0), (0, 2, 0), 9)
        v = np.concatenate([g, g[::-1]])
    elif name == "flat":  # zero-area triangles among others
        v = rng.uniform(-1, 1, (60, 9))
        v[::3, 6:9] = v[::3, 3:6]
    elif name == "offset":
        v = scenes.icosphere(3).verts + np.tile([300.0, -200.0, 100.0], 3)
    elif name == "room":
        return scenes.room(grid=3)
    else:
        return scenes.soup(700, 2)
    v = np.asarray(v, np.float32)
    return scenes.Mesh(v, np.full((len(v), 3), 0.5, np.float32), np.zeros(len(v), np.uint8))


@pytest.mark.parametrize("tree", ["median", "sah"])
@pytest.mark.parametrize("name", ["one", "copies", "layers", "flat", "offset", "room", "soup"])
def test_culling_hierarchy_matches_reference_walk(oracle, name, tree):
    """The culling hierarchy (triangles once each, hits checked against the
    reference's leaves that own them) gives the oracle's ids and distances bit
    for bit, and its occlusion answers, for every leaf size and both trees, on
    the rays that use it (finite inverse directions) within the error bound
    that it rests on."""
    m = _hard_mesh(name)
    st = scenes.soup_setup()
    st.det_eps = 0.0
    st.tree, st.leaf_size, st.sah_ct = tree, 4, 1.0
    rays = _hard_rays(m, 3, 6000)
    rays = np.ascontiguousarray(rays[_well_posed(m, rays) & np.isfinite(rays[:, 6:9]).all(1)])
    assert len(rays) > 1000
    want, want_t = oracle.OracleScene.from_setup(m, st).trace(rays, st.det_eps)
    rng = np.random.default_rng(9)
    d2 = np.where(rng.random(len(rays)) < 0.5, np.minimum(want_t, 1e3) ** 2, 1.0) * rng.choice([0.9, 1.0, 1.1], len(rays))
    d2 = d2.astype(np.float32)
    with np.errstate(over="ignore"):
        want_occ = (want >= 0) & (want_t * want_t < d2)
    for refine in (8, 3, 1):
        sc = native.Scene.from_setup(m, st, leaf_refine=refine)
        ids, ts = trace(sc, rays, st.det_eps)
        np.testing.assert_array_equal(ids, want.astype(np.int32))
        np.testing.assert_array_equal(ts.view(np.uint32), want_t.view(np.uint32))
        occ = torch.empty(len(rays), dtype=torch.uint8, device="cuda")
        sc.trace_occluded(torch.from_numpy(rays).cuda(), torch.from_numpy(d2).cuda(), st.det_eps, occ)
        np.testing.assert_array_equal(occ.cpu().numpy(), want_occ.astype(np.uint8))


def _edges(warps_per_sm):
    """Item counts at which a launch over few rays or pixels changes its lanes
    per warp: half of the resident warps times 1, 2, 4; all of them times 8."""
    w = torch.cuda.get_device_properties(0).multi_processor_count * warps_per_sm
    return [w // 2, w, 2 * w, 8 * w]


@pytest.mark.parametrize("edge", [-1, 0, 1, 2, 3])
def test_rays_per_warp(oracle, edge):
    """Closest hits and occlusion of ray counts on both sides of each edge (and
    of 1, 3, 33 rays): every ray is answered, none beyond the last is written."""
    m, st = scenes.soup(2_000, 8), scenes.soup_setup()
    sc = native.Scene.from_setup(m, st)
    orc = oracle.OracleScene.from_setup(m, st)
    counts = [1, 3, 33] if edge < 0 else [_edges(36)[edge] + k for k in (-1, 0, 1)]
    rng = np.random.default_rng(edge + 9)
    n = max(counts)
    o = rng.uniform(-0.2, 1.2, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d, (1.0 / d).astype(np.float32)], 1)
    wid, wt = orc.trace(rays, 1e-4)
    d2 = rng.uniform(0.0, 1.0, n).astype(np.float32)
    want = (wid >= 0) & (d2 > (wt * wt).astype(np.float32))
    r, dd = torch.from_numpy(rays).cuda(), torch.from_numpy(d2).cuda()
    for k in counts:
        ids = torch.full((n + 40,), -7, dtype=torch.int32, device="cuda")
        ts = torch.full((n + 40,), -7.0, dtype=torch.float32, device="cuda")
        occ = torch.full((n + 40,), 9, dtype=torch.uint8, device="cuda")
        sc.trace_closest(r[:k], 1e-4, ids[:k], ts[:k])
        sc.trace_occluded(r[:k], dd[:k], 1e-4, occ[:k])
        torch.cuda.synchronize()
        assert (ids[k:] == -7).all() and (ts[k:] == -7).all() and (occ[k:] == 9).all()
        np.testing.assert_array_equal(ids[:k].cpu().numpy(), wid[:k].astype(np.int32))
        np.testing.assert_array_equal(ts[:k].cpu().numpy().view(np.uint32), wt[:k].view(np.uint32))
        np.testing.assert_array_equal(occ[:k].cpu().numpy(), want[:k].astype(np.uint8))


@pytest.mark.parametrize("traversal", [native.TRAVERSAL_LANES, native.TRAVERSAL_PACKETS,
                                       native.TRAVERSAL_PRIMARY_PACKETS])
@pytest.mark.parametrize("warps", [32, 40])
def test_pixels_per_warp(oracle, traversal, warps):
    """Frames of ragged sizes on both sides of each edge."""
    m = scenes.soup(2_000, 9)
    for w, h in [(1, 1), (9, 5)] + [(97, e // 97 + k) for e in _edges(warps) for k in (-2, 3)]:
        check_frame(oracle, m, scenes.soup_setup(w, h), traversal)


@pytest.mark.parametrize("scale,squash", [(1.0, 1.0), (1e-6, 1.0), (1e6, 1.0), (1.0, 1e-3), (37.0, 30.0)])
def test_grid_boxes_match_reference_walk(oracle, scale, squash):
    """Ray queries, which test boxes on a scene-wide grid, over scenes of
    different sizes and proportions: ids and distances are the oracle's, also
    for directions so close to an axis that an inverse is up to 1e37 (the grid
    serves those up to 1e30)."""
    m = scenes.soup(700, 4)
    m.verts[:] = (m.verts.reshape(-1, 3, 3) * np.float32([scale, scale, scale * squash])).reshape(m.verts.shape)
    st = scenes.soup_setup()
    st.det_eps = 0.0
    rays = _hard_rays(m, 6, 6000)
    rng = np.random.default_rng(7)
    k = len(rays) // 3
    d = (10.0 ** rng.uniform(-37, -20, (k, 3)) * rng.choice([-1, 1], (k, 3))).astype(np.float32)
    d[np.arange(k), rng.integers(0, 3, k)] = rng.choice([-1, 1], k)
    rays[:k, 3:6], rays[:k, 6:9] = d, 1.0 / d
    rays = np.ascontiguousarray(rays[_well_posed(m, rays) & np.isfinite(rays[:, 6:9]).all(1)])
    assert len(rays) > 1000
    ids, ts = trace(native.Scene.from_setup(m, st), rays, 0.0)
    want, want_t = oracle.OracleScene.from_setup(m, st).trace(rays, 0.0)
    np.testing.assert_array_equal(ids, want.astype(np.int32))
    np.testing.assert_array_equal(ts.view(np.uint32), want_t.view(np.uint32))
