"""Host side of the culling hierarchy (host/cull_bvh.cpp, host/flatten.cpp),
checked by a small C++ program built from the same sources."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "nostrum_pray_gb300", "csrc", "host")


@pytest.fixture(scope="session")
def cull_check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cull") / "cull_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-pthread", "-I", HOST, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "cull_check.cpp"), os.path.join(HOST, "cull_bvh.cpp"),
                    os.path.join(HOST, "flatten.cpp"), os.path.join(HOST, "kdtree.cpp"), "-ldl"], check=True)

    def run(*args):
        return subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=300)

    return run


@pytest.mark.parametrize("limit", [0, 1, 3])
def test_build_survives_a_thread_limit(cull_check, limit):
    """A system that gives fewer threads than were asked for costs time, not the
    process: the hierarchy is the same."""
    r = cull_check("threads", limit)
    assert r.returncode == 0, (r.returncode, r.stderr)
    assert r.stdout.split() == ["same", "1"]


@pytest.mark.parametrize("n", [1, 2, 5])
def test_build_threads_bounds_the_whole_build(cull_check, n):
    """build_threads counts everything a scene's creation runs at once: the
    reference's tree, the culling hierarchy beside it and the caller. (A
    thread that has given its place back may still be ending when the next
    starts: room for that where there is more than one.)"""
    r = cull_check("budget", n)
    assert r.returncode == 0, r.stderr
    most = int(r.stdout.split()[1])
    assert most <= 2 * n - 1


@pytest.mark.parametrize("n", [40, 200, 100_000])
def test_owners_of_a_large_triangle(cull_check, n):
    """A hit on a floor that thousands of leaves hold finds the first leaf whose
    box the ray passes, with the box tests of a walk down a tree and not of
    all the leaves."""
    r = cull_check("owners", n)
    assert r.returncode == 0, r.stdout + r.stderr
    v = dict(zip(r.stdout.split()[::2], map(float, r.stdout.split()[1::2])))
    assert v["wrong"] == 0 and v["hits"] > 0
    assert v["leaves"] > 0 if n < 100_000 else v["leaves"] > 1000
    assert v["mean"] < 40 and v["most"] < 160


@pytest.mark.parametrize("half", [50, 1000, 30_000])
def test_fine_detail_in_a_large_scene(cull_check, half):
    """The pads of the culling boxes follow the origins served: rays near a fine
    object test hardly more triangles on a large floor than on a small one."""
    def run(h):
        r = cull_check("mixed", h)
        assert r.returncode == 0, r.stderr
        return dict(zip(r.stdout.split()[::2], map(float, r.stdout.split()[1::2])))
    small, large = run(2), run(half)
    assert large["served"] == 1.0
    assert large["tris"] < 4 * small["tris"]


@pytest.mark.parametrize("refs,tris,fits", [(2 ** 30, 2 ** 28, 1), (2 ** 30 + 2 ** 29, 2 ** 29 - 1, 1),
                                            (2 ** 29, 2 ** 29, 0), (2 ** 31 - 2 ** 20, 2 ** 20, 0)])
def test_large_scenes_are_culled(cull_check, refs, tris, fits):
    """The culling copy's limit is its own triangles', not that of all records:
    its records come first."""
    assert cull_check("fits", refs, tris).stdout.split() == ["fits", str(fits)]


@pytest.mark.parametrize("leaf", [8, 32, 10 ** 6])
@pytest.mark.parametrize("strips", [40, 300, 2000])
def test_thin_triangles(cull_check, strips, leaf):
    """A thin triangle's box is its own, grown by the error of its hits, and not
    that of the leaves that hold it: a line through cylinders of strips meets a
    few strips on each wall it crosses, whatever the leaf size."""
    r = cull_check("slivers", strips, leaf)
    assert r.returncode == 0, r.stderr
    assert float(r.stdout.split()[1]) < 40


@pytest.mark.parametrize("half,made", [(1, True), (3, True), (300, False), (30_000, False)])
def test_grid_only_where_it_fits_the_boxes(cull_check, half, made):
    """Grid pairs are made where the scene's 16-bit steps are fine enough for its
    boxes, and then cost a ray hardly any more triangles."""
    r = cull_check("grid", half)
    assert r.returncode == 0, r.stderr
    v = dict(zip(r.stdout.split()[::2], map(float, r.stdout.split()[1::2])))
    assert bool(v["made"]) == made and v["ratio"] < 1.5


@pytest.mark.parametrize("tree", ["median", "sah"])
@pytest.mark.parametrize("refine", [0, 1, 4, 8])
def test_device_layout_holds_every_triangle(tree, refine):
    """The culling hierarchy of a device layout holds every triangle once and
    has nodes of its own; with refinement off there is none."""
    from nostrum_pray_gb300 import native, scenes
    st = scenes.soup_setup()
    st.tree = tree
    m = scenes.soup(2000, 1)
    h = native.HostTree(m, native.tree_options(st))
    nodes, refs, tris, cull = (int(x) for x in h.device_layout(refine))
    stats = [int(x) for x in h.tree_stats()]
    assert refs == stats[4]
    if refine == 0:
        assert (tris, cull) == (0, 0)
    else:
        assert tris == m.n and 2 * m.n // min(refine, 4) <= cull <= 2 * m.n and nodes > cull
