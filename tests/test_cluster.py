"""Scenes stepped on chip patch by patch (fw_cluster.cuh) against the gather and
stream steps: same bits, at the sizes where the patches, halos, corner slots
and cluster sizes change, and through every gate decision."""

import numpy as np
import pytest

import flatworld_b200 as fw
from flatworld_b200 import _native
from flatworld_b200.batch import BatchedLoop
from tests import scenes

pytestmark = pytest.mark.gpu


def _rectangle(nx, ny, mat, ground, cell=0.02, **kw):
    conn, coords = fw.structured_rectangle(nx, ny, nx * cell, ny * cell, origin=(0.0, 0.0), jitter=0.1, seed=nx)
    fem = fw.FemDomain(fw.Mesh(2, conn, coords), fw.SolidProp(mat), [fw.Gravity([0.0, -9.8])],
                       initials=[fw.InitialVel("ALL", [0.1, -1.0])], **kw)
    return [ground, fem] if ground is not None else [fem]


def _plane(y=-0.005):
    return fw.GroundDomain(2, [0.0, y], [0.0, 1.0])


def _bump(lo, hi):
    xs = np.linspace(lo, hi, 64)
    return fw.HeightFieldDomain(2, (0.01 * np.sin(40 * xs) - 0.015).astype(np.float32), lb=[lo, -1.0], ub=[hi, 1.0])


MATS = {"elastic": fw.Elastic(5e4, 0.3, 500.0), "neohookean": fw.HyperElastic(5e4, 0.3, 500.0),
        "mises": fw.MisesPlastic(5e4, 0.3, 500.0, sigma_y=300.0, H=5e3)}


def _disk():
    """A fan around one node (24 corners on it) inside a ring: more corner slots than a structured mesh needs."""
    n = 24
    a = 2 * np.pi * np.arange(n) / n
    pts = np.concatenate([[[0.0, 0.0]], *[r * np.stack([np.cos(a), np.sin(a)], 1) for r in (0.05, 0.1, 0.15)]])
    tri = [[0, 1 + i, 1 + (i + 1) % n] for i in range(n)]
    for ring in range(2):
        for i in range(n):
            p, q = 1 + ring * n + i, 1 + ring * n + (i + 1) % n
            tri += [[p, p + n, q], [q, p + n, q + n]]
    mesh = fw.Mesh(2, np.asarray(tri, np.int32), (pts + [0.0, 0.151]).astype(np.float32))
    return [_plane(0.0), fw.FemDomain(mesh, fw.SolidProp(MATS["neohookean"]), [fw.Gravity([0.0, -9.8])])]


SINGLE = {
    "one patch": lambda: _rectangle(3, 2, MATS["elastic"], _plane()),
    "two patches": lambda: _rectangle(15, 8, MATS["neohookean"], _plane()),
    "a thread per triangle, J2": lambda: _rectangle(60, 31, MATS["mises"], _plane()),
    "a thread per triangle, 640 threads": lambda: _rectangle(200, 160, MATS["neohookean"], _plane(), cell=0.005),
    "two triangles per thread": lambda: _rectangle(200, 200, MATS["mises"], _plane(), cell=0.005),
    "several triangles per thread": lambda: _rectangle(260, 251, MATS["neohookean"], _plane(), cell=0.004),
    "records in L2": lambda: _rectangle(640, 500, MATS["neohookean"], _plane(-0.0005), cell=0.002),
    "records in L2, J2": lambda: _rectangle(520, 440, MATS["mises"], _plane(-0.0005), cell=0.002),
    "nodes of many corners": _disk,
    "no pairs": lambda: _rectangle(40, 17, MATS["mises"], None),
    "seven bodies": lambda: scenes.multi_block_scene(fw, 7),
    "boundary conditions": lambda: scenes.bcs_scene(fw),
    "forces from outside the gate box": lambda: _rectangle(40, 30, MATS["neohookean"], _bump(0.25, 0.55)),
    "nodes below the gate box": lambda: _rectangle(20, 20, MATS["elastic"], _plane(0.12)),
    "voxels": lambda: scenes.voxel_disk_scene(fw),
}


def _same(a, b, energy=True):
    pa, pb = a._packed, b._packed
    na, nb = a._native, b._native
    for field in (_native.FW_FIELD_X, _native.FW_FIELD_V):
        assert np.array_equal(na.read_nodes(field, 0, pa.N), nb.read_nodes(field, 0, pb.N), equal_nan=True)
    for u, v in zip(na.read_plastic(pa.E), nb.read_plastic(pb.E)):
        assert np.array_equal(u, v, equal_nan=True)
    assert np.array_equal(na.read_aabb(pa.B), nb.read_aabb(pb.B))
    assert np.array_equal(na.read_counters(pa.S), nb.read_counters(pb.S))


@pytest.mark.parametrize("name", SINGLE)
def test_single_scene_bitwise(name):
    a = fw.ExplicitLoop(0.0, SINGLE[name](), damping=0.02)
    b = fw.ExplicitLoop(0.0, SINGLE[name](), damping=0.02, path="gather")
    assert a._native.get_option(_native.FW_OPT_CLUSTER) == 1 and a.path == 2
    for lp in (a, b):
        lp.enable_cfl_monitor()
        lp.advance()
        for n in (2, 17, 150):
            lp.advance_n(n)
    _same(a, b)
    assert a.currentStableTime() == b.currentStableTime()
    for lp in (a, b):  # positions set between calls: the next gates still use the last substep's boxes
        x = lp._native.read_nodes(_native.FW_FIELD_X, 0, lp._packed.N)
        lp._native.write_nodes(_native.FW_FIELD_X, 0, x + np.float32([0.0, 0.01]))
        lp.advance_n(3)
    _same(a, b)


def test_moduli_per_triangle_and_set_later():
    def build(path="auto"):
        doms = _rectangle(40, 20, MATS["neohookean"], _plane())
        doms[1].elementYoung = np.linspace(4e4, 6e4, doms[1].nelements).astype(np.float32)
        return fw.ExplicitLoop(1e-4, doms, useAdapativeDT=False, path=path)

    a, b = build(), build("gather")
    u, v = (fw.ExplicitLoop(1e-4, _rectangle(40, 20, MATS["mises"], _plane()), useAdapativeDT=False, path=p)
            for p in ("auto", "gather"))
    for lp in (a, b, u, v):
        lp.advance_n(40)
        lp._native.set_element_young(np.linspace(6e4, 4e4, lp._packed.E).astype(np.float32))
        lp.advance_n(40)
    assert all(lp._native.get_option(_native.FW_OPT_CLUSTER) == 1 for lp in (a, u))
    _same(a, b)
    _same(u, v)


def _graded(nx, ny):
    """A body whose triangles each have their own Young's modulus."""
    doms = _rectangle(nx, ny, MATS["neohookean"], _plane(), cell=0.01)
    doms[1].elementYoung = np.linspace(2e4, 8e4, doms[1].nelements).astype(np.float32)
    return doms


@pytest.mark.parametrize("sizes,covered", [([(9, 9), (30, 20), (60, 40)], 1), ([(9, 9), (200, 160), (30, 20)], 2)],
                         ids=["on chip", "one too large"])
def test_moduli_per_triangle_in_batches(sizes, covered):
    """The same bits however the substeps are cut into calls: the on-chip, the stream and the gather kernels."""
    def build(**kw):
        return BatchedLoop([_graded(*size) for size in sizes] + _batch([(12, 7)]), dt=5e-5, useAdapativeDT=False, **kw)

    a, b, c, d = build(), build(), build(stream_patch=64), build(path="gather")
    assert a._native.get_option(_native.FW_OPT_CLUSTER) == covered
    for lp in (a, b, c, d):
        lp._packed = lp.packed
    for _ in range(24):
        b.advance(1)
    for lp in (a, c, d):
        lp.advance(24)
    for lp in (b, c, d):
        _same(a, lp)
    for lp in (a, c, d):  # and changed later, with the batch's graphs made
        lp.advance(24)
        lp._native.set_element_young(np.linspace(8e4, 2e4, lp.packed.E).astype(np.float32))
        lp.advance(24)
    for lp in (c, d):
        _same(a, lp)


def test_moduli_per_triangle_in_arenas():
    from flatworld_b200.serve import Arena

    ar = Arena(60_000, 120_000, 16, 16, 64, 1 << 16, 1 << 16)
    build = [lambda: _batch([(12, 7)])[0], lambda: _graded(30, 20), lambda: _graded(200, 160), lambda: _graded(9, 9)]
    dt = np.float32(5e-5)
    ran, sc = [], []
    for b in build:  # the first scene is resident before one with several moduli comes
        sc.append(ar.insert(b()))
        ran.append(0)
        for n in (1, 1, 1, 9, 2):
            ar.native.step_served_n(np.where(np.isin(np.arange(ar.S), sc), dt, np.float32(0.0)), n)
            ran = [r + n for r in ran]
    ar.native.synchronize()
    for s, b, n in zip(sc, build, ran):
        lp = fw.ExplicitLoop(5e-5, b(), useAdapativeDT=False, path="gather")
        lp.advance_n(n - 1)  # the first substep of a committed scene is its construction step
        nn = lp._packed.N
        assert np.array_equal(ar.coords(s), lp.femSpringManager.coords.numpy()[:nn])
        assert np.array_equal(ar.velocities(s), lp.femSpringManager.V.numpy()[:nn])
    ar.close()


def _batch(sizes):
    out = []
    for k, (nx, ny) in enumerate(sizes):
        mat = list(MATS.values())[k % 3]
        out.append(_rectangle(nx, ny, mat, _plane() if k % 2 else _bump(-1.0, 6.0),
                              cell=0.01))
    return out


@pytest.mark.parametrize("sizes,covered", [
    ([(4, 3), (9, 9), (30, 20), (60, 40), (100, 60), (130, 90)], 1),  # clusters of 1 to 16
    ([(9, 9), (200, 160), (30, 20)], 2),  # one scene too large for a cluster: the stream kernels step it
    ([(8, 5 + k % 7) for k in range(70)], 1),
], ids=["cluster sizes", "one too large", "many small"])
def test_batch_bitwise(sizes, covered):
    a = BatchedLoop(_batch(sizes), dt=5e-5, useAdapativeDT=False)
    b = BatchedLoop(_batch(sizes), dt=5e-5, useAdapativeDT=False, stream_patch=64)
    assert a._native.get_option(_native.FW_OPT_CLUSTER) == covered
    assert b._native.get_option(_native.FW_OPT_CLUSTER) == 0
    frozen = np.ones(len(sizes), np.int32)
    frozen[::3] = 0
    for lp in (a, b):
        lp._packed = lp.packed
        lp.advance(1)
        lp._set_active(frozen)
        lp.advance(7)
        lp._set_active(np.ones(len(sizes), np.int32))
        lp.advance(64)
        lp.advanceWithTime(3.3e-4)
    _same(a, b)
    a._native.set_option(_native.FW_OPT_CLUSTER, 0)  # the path's own kernels go on from the same state
    for lp in (a, b):
        lp.advance(9)
    _same(a, b)


@pytest.mark.parametrize("n", [20, 530])
def test_short_calls_of_one_scene_equal_the_gather_kernels(n):
    """Calls on both sides of the length from which a scene is stepped on chip, small and above 2500 triangles per SM."""
    a, b = (fw.ExplicitLoop(0.0, _rectangle(n, 380, MATS["neohookean"], _plane(-0.0005), cell=0.002), path=p)
            for p in ("auto", "gather"))
    for lp in (a, b):
        for k in (1, 2, 3, 1, 4, 5, 2, 1, 9, 3):
            lp.advance_n(k)
    _same(a, b)


@pytest.mark.parametrize("n,least", [(20, 3), (150, 4), (420, 4)])
def test_least_substeps_of_an_on_chip_call(n, least):
    """Shorter calls are two plain launches a substep: 15,200, 114,000 and 319,200 triangles."""
    lp = fw.ExplicitLoop(0.0, _rectangle(n, 380, MATS["neohookean"], _plane(-0.0005), cell=0.002))
    for k in range(1, 6):
        before = lp._native.launch_count()
        lp.advance_n(k)
        assert lp._native.launch_count() - before == (1 if k >= least else 2 * k)


def test_short_calls_with_new_and_repeated_step_sizes():
    """Launched one by one at first, as a graph when repeated: the same bits, and the launches of the substeps."""
    a, b = (fw.ExplicitLoop(5e-5, _rectangle(20, 30, MATS["mises"], _plane()), useAdapativeDT=False, path=p)
            for p in ("auto", "gather"))
    for n, dt in ((2, 5e-5), (2, 5e-5), (2, 5e-5), (2, 4e-5), (2, 5e-5), (3, 3e-5), (2, 3e-5), (2, 4e-5), (2, 4e-5)):
        before = a._native.launch_count()
        a.advance_n(n, dt)
        assert a._native.launch_count() - before == (4 if n == 2 else 1)
        for _ in range(n):
            b.advance_n(1, dt)
    _same(a, b)


@pytest.mark.parametrize("bodies", [4, 34])
def test_short_calls_equal_the_stream_kernels(bodies):
    """Calls on both sides of the length from which a batch is stepped on chip, below and above 1500 triangles per SM."""
    a = BatchedLoop(_batch([(60, 58)] * bodies), dt=5e-5, useAdapativeDT=False)
    b = BatchedLoop(_batch([(60, 58)] * bodies), dt=5e-5, useAdapativeDT=False, stream_patch=64)
    for lp in (a, b):
        lp._packed = lp.packed
        for n in (1, 2, 3, 4, 5, 1, 8, 2):
            lp.advance(n)
        lp.advanceWithTime(2e-4)
        lp.advanceWithTime(1e-3)
    _same(a, b)


@pytest.mark.parametrize("sizes,least", [([(8, 8)] * 20, 3), ([(60, 60)] * 8, 3), ([(40, 40)] * 16, 4),
                                         ([(60, 60)] * 40, 5)])
def test_least_substeps_of_an_on_chip_batch(sizes, least):
    """Shorter calls are two launches a substep; one more substep where the wide clusters take turns on the SMs."""
    lp = BatchedLoop([_rectangle(nx, ny, MATS["elastic"], _plane(), cell=0.01) for nx, ny in sizes], dt=5e-5,
                     useAdapativeDT=False)
    for k in range(1, 7):
        before = lp.launch_count()
        lp.advance(k)
        assert lp.launch_count() - before == (1 if k >= least else 2 * k)


@pytest.mark.parametrize("size,scenes,least", [((8, 8), 20, 3), ((8, 8), 320, 6), ((50, 50), 20, 7), ((50, 50), 40, 16)])
def test_least_substeps_of_an_on_chip_arena(size, scenes, least):
    """Shorter calls are two launches a substep (and one that carries an odd call's state back), by the scenes and by
    the SMs that their wide clusters take; the same bits on both sides."""
    from flatworld_b200.serve import Arena
    from flatworld_b200.world import PackedWorld, SceneLayout

    lay = SceneLayout(_rectangle(*size, MATS["mises"], _plane(), cell=0.01))
    ar = Arena(400_000, 800_000, 512, 512, 512, 1, 1)
    pk = ar.pack(lay, PackedWorld([lay]))
    sc = [ar.insert_pack(lay, pk) for _ in range(scenes)]
    dts = np.zeros(ar.S, np.float32)
    dts[sc] = 2e-5
    ran = 0
    for n in (1, 2, 3, 4, 5, 6, 7, 15, 16, 17, 3):
        before = ar.native.launch_count()
        ar.native.step_served_n(dts, n)
        ran += n
        assert ar.native.launch_count() - before == (1 if n >= least else 2 * n + n % 2)
    lp = fw.ExplicitLoop(2e-5, _rectangle(*size, MATS["mises"], _plane(), cell=0.01), useAdapativeDT=False, path="gather")
    lp.advance_n(ran - 1)
    for s in (sc[0], sc[-1]):
        assert np.array_equal(ar.coords(s), lp.femSpringManager.coords.numpy()[: lp._packed.N])
    pk.close()
    ar.close()


@pytest.mark.parametrize("patch,on_chip", [(0, 1), (64, 0)])
def test_tuning_keeps_the_on_chip_step(patch, on_chip, tmp_path, monkeypatch):
    from flatworld_b200 import autotune

    monkeypatch.setenv("FLATWORLD_B200_CACHE", str(tmp_path))
    lp = BatchedLoop(_batch([(20, 9), (7, 30)]), dt=5e-5, useAdapativeDT=False, stream_patch=patch)
    best = autotune.tune_batched(lp, steps=4)
    assert best["path"] == "stream" and best["minb"] > 0 and bool(best.get("on_chip")) == bool(on_chip)
    assert lp._native.get_option(_native.FW_OPT_CLUSTER) == on_chip


@pytest.mark.parametrize("build,bad", [
    (lambda: _rectangle(20, 100, MATS["neohookean"], _plane(0.005)), range(32, 64)),
    (lambda: scenes.multi_block_scene(fw, 2), [121]),
], ids=["a warp of boundary nodes", "a warp of two bodies"])
def test_nan_nodes_leave_the_contact_of_the_others(build, bad):
    """Nodes that are NaN widen no box: the others' gates are the same on every path."""
    loops = [fw.ExplicitLoop(2e-5, build(), useAdapativeDT=False, path=p) for p in ("auto", "gather")]
    loops.append(fw.ExplicitLoop(2e-5, build(), useAdapativeDT=False, front_warps=6))
    loops += [BatchedLoop([build()], dt=2e-5, useAdapativeDT=False, **kw) for kw in ({}, {"stream_patch": 64})]
    for lp in loops:
        lp._packed = lp.packed if isinstance(lp, BatchedLoop) else lp._packed
        x = lp._native.read_nodes(_native.FW_FIELD_X, 0, lp._packed.N)
        x[list(bad)] = np.nan
        lp._native.write_nodes(_native.FW_FIELD_X, 0, x)
        (lp.advance if isinstance(lp, BatchedLoop) else lp.advance_n)(8)
    for lp in loops[1:]:
        _same(loops[0], lp)


@pytest.mark.parametrize("sizes,covered", [([(20, 9), (7, 30)], 1), ([(20, 9), (200, 160)], 2)])
def test_tuning_shapes_the_stream_kernels_of_short_calls(sizes, covered, tmp_path, monkeypatch):
    """The scenes on chip stay there, also beside one too large for it; the stream kernels get the shape."""
    from flatworld_b200 import autotune

    monkeypatch.setenv("FLATWORLD_B200_CACHE", str(tmp_path))
    a, b = (BatchedLoop(_batch(sizes), dt=5e-5, useAdapativeDT=False) for _ in range(2))
    best = autotune.tune_batched(a, steps=4)
    assert a._native.get_option(_native.FW_OPT_CLUSTER) == covered and best["on_chip"]
    assert (best["minb"], best["bulk"]) in [(c["minb"], c["bulk"]) for c in best["candidates"]]
    a.set_stream_shape(16, True)
    assert a._native.get_option(_native.FW_OPT_CLUSTER) == covered
    assert a._native.get_option(_native.FW_OPT_STREAM_MINB) == 16
    for lp in (a, b):
        lp._packed = lp.packed
        for n in (1, 2, 9, 1, 20):
            lp.advance(n)
    _same(a, b)


def test_tuning_a_single_scene_times_the_default_too(tmp_path, monkeypatch):
    import json

    from flatworld_b200 import autotune

    monkeypatch.setenv("FLATWORLD_B200_CACHE", str(tmp_path))
    kw = autotune.tune_resident(SINGLE["two patches"], fronts=(4, 6), patches=(0, 2), steps=50)
    (entry,) = json.loads((tmp_path / "autotune.json").read_text()).values()
    shapes = [(c["front_warps"], c["patches"]) for c in entry["candidates"]]
    assert shapes == [(0, 0), (4, 0), (4, 2), (6, 0), (6, 2)]
    best = min(entry["candidates"], key=lambda c: c["ms"])
    assert kw == {"front_warps": best["front_warps"], "patches": best["patches"]}
    a, b = fw.ExplicitLoop(0.0, SINGLE["two patches"](), **kw), fw.ExplicitLoop(0.0, SINGLE["two patches"]())
    assert a._native.get_option(_native.FW_OPT_CLUSTER) == (1 if kw == {"front_warps": 0, "patches": 0} else 0)
    for lp in (a, b):
        lp.advance_n(50)
    _same(a, b)


def test_wait_runs_out_and_the_context_recovers():
    lp = fw.ExplicitLoop(0.0, SINGLE["two patches"]())
    lp.advance_n(20)
    lp._native.set_option(_native.FW_OPT_WAIT_LIMIT, 4096)
    lp._native.set_option(_native.FW_OPT_TEST_WITHHOLD, 1)
    lp.advance_n(10)
    with pytest.raises(RuntimeError, match="gave up"):
        lp.synchronize()
    lp._native.set_option(_native.FW_OPT_TEST_WITHHOLD, -1)
    lp.advance_n(10)
    lp.synchronize()
    b = BatchedLoop(_batch([(60, 40), (9, 9), (61, 41)]), dt=5e-5, useAdapativeDT=False)
    b.advance(20)
    b._native.set_option(_native.FW_OPT_WAIT_LIMIT, 4096)
    b._native.set_option(_native.FW_OPT_TEST_WITHHOLD, 1)
    b.advance(10)
    with pytest.raises(RuntimeError, match="gave up"):
        b.synchronize()
    b._native.set_option(_native.FW_OPT_TEST_WITHHOLD, -1)
    b.advance(10)
    b.synchronize()


@pytest.mark.parametrize("name", ["two patches", "records in L2"])
def test_a_wait_that_ran_out_is_reported_whatever_ran_after(name):
    """A call whose waits gave up, then calls on the gather kernels, or the on-chip step given up for good (the large
    mesh then has the gather kernels only): the next synchronisation still reports it, and once."""
    for after in ("short call", "off"):
        lp = fw.ExplicitLoop(0.0, SINGLE[name]())
        lp.advance_n(5)
        lp.advance_n(1)
        lp.synchronize()
        lp._native.set_option(_native.FW_OPT_WAIT_LIMIT, 4096)
        lp._native.set_option(_native.FW_OPT_TEST_WITHHOLD, 1)
        lp.advance_n(10)
        lp._native.set_option(_native.FW_OPT_TEST_WITHHOLD, -1)
        if after == "off":
            lp._native.set_option(_native.FW_OPT_CLUSTER, 0)
            assert lp._native.get_path()[0] == (2 if name == "two patches" else 1)
        else:
            lp.advance_n(1)
        with pytest.raises(RuntimeError, match="gave up"):
            lp.synchronize()
        lp.advance_n(1)
        lp.synchronize()


def _terrain_scene(nx, ny, kind):
    """A block on (and partly inside) a voxel grid of nx x ny cells: solid, solid with cells of neither state, or
    random."""
    rng = np.random.default_rng(nx * 100 + ny)
    if kind == "random":
        occ = (rng.random((nx, ny)) < 0.4).astype(np.int32)
    else:
        top = rng.integers(ny // 2, ny + 1, nx)
        occ = (np.arange(ny)[None, :] < top[:, None]).astype(np.int32)
        if kind == "marked":
            occ[rng.random((nx, ny)) < 0.1] = 5
    lb = np.array([0.1, -0.02 * ny + 0.03], np.float32)
    vox = fw.VoxelGridDomain(2, nx, ny, lb, lb + np.float32([0.02 * nx, 0.02 * ny]), occupancy_np=occ)
    return _rectangle(24, 11, MATS["elastic"], vox, cell=0.03)


@pytest.mark.parametrize("kind", ["solid", "marked", "random"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (37, 1), (1, 29), (31, 64), (130, 33)])
def test_voxel_contact_matches_the_oracle(nx, ny, kind):
    import oracle

    o = oracle.OracleLoop(_terrain_scene(nx, ny, kind), 0.0, useAdapativeDT=True, threads=4)
    loops = [fw.ExplicitLoop(0.0, _terrain_scene(nx, ny, kind), path=p) for p in ("auto", "gather")]
    loops.append(fw.ExplicitLoop(0.0, _terrain_scene(nx, ny, kind), front_warps=6))
    o.advance(60)
    x, v, _ = o.state()
    for lp in loops:
        lp.advance_n(60)
        n = lp._packed.N
        assert np.array_equal(lp.femSpringManager.coords.numpy()[:n].astype(np.float64), x)
        assert np.array_equal(lp.femSpringManager.V.numpy()[:n].astype(np.float64), v)


def _long_terrain_scene(nx, ny, at):
    """A block lying in a long solid grid with its middle at cell ``at`` of the long side."""
    along = nx > ny
    cell = (0.001, 0.02) if along else (0.02, 0.001)
    vox = fw.VoxelGridDomain(2, nx, ny, np.float32([0.0, 0.0]), np.float32([nx * cell[0], ny * cell[1]]),
                             occupancy_np=np.ones((nx, ny), np.int32))
    origin = (at * 0.001 - 0.05, ny * 0.02 - 0.01) if along else (nx * 0.02 - 0.01, at * 0.001 - 0.05)
    conn, coords = fw.structured_rectangle(10, 10, 0.1, 0.1, origin=origin, jitter=0.1, seed=3)
    return [vox, fw.FemDomain(fw.Mesh(2, conn, coords), fw.SolidProp(MATS["elastic"]), [fw.Gravity([0.0, -9.8])])]


@pytest.mark.parametrize("nx,ny", [(65535, 4), (65536, 4), (70000, 4), (4, 65535), (2, 70000)])
@pytest.mark.parametrize("at", [65400, 65535])
def test_voxel_contact_on_long_grids(nx, ny, at):
    """Sides on both sides of the cell table's 16 bits; nodes on both sides of cell 65535."""
    import oracle

    def build():
        return _long_terrain_scene(nx, ny, at)

    o = oracle.OracleLoop(build(), 0.0, useAdapativeDT=True, threads=4)
    loops = [fw.ExplicitLoop(0.0, build(), path=p) for p in ("auto", "gather")]
    loops.append(fw.ExplicitLoop(0.0, build(), front_warps=6))
    batch = BatchedLoop([build(), build()], dt=loops[0].dt, useAdapativeDT=False, stream_patch=64)
    o.advance(10)
    x, v, _ = o.state()
    assert np.abs(v).max() > 2 * 9.8 * 10 * loops[0].dt  # pushed out: faster than a free fall
    for lp in loops:
        lp.advance_n(10)
        n = lp._packed.N
        assert np.array_equal(lp.femSpringManager.coords.numpy()[:n].astype(np.float64), x)
        assert np.array_equal(lp.femSpringManager.V.numpy()[:n].astype(np.float64), v)
    batch.advance(10)
    assert np.array_equal(batch.coords(1).astype(np.float64), x)


def test_voxel_cells_take_a_table_only_where_there_is_room():
    """An arena without voxel grounds takes no memory for them beyond the cells, and one whose cell table the device
    cannot hold (192 GiB here) walks the grids: the same bits as a scene of its own."""
    import torch

    from flatworld_b200.serve import Arena

    torch.cuda.init()
    before = torch.cuda.mem_get_info()[0]
    ar = Arena(20_000, 40_000, 8, 8, 32, 1 << 10, 1 << 30)
    assert before - torch.cuda.mem_get_info()[0] < 3 << 30
    ar.close()
    ar = Arena(20_000, 40_000, 8, 8, 32, 1 << 10, 24 << 30)
    dt = np.float32(5e-5)
    build = [lambda: _rectangle(12, 7, MATS["elastic"], _plane()), lambda: _terrain_scene(31, 64, "marked"),
             lambda: _terrain_scene(130, 33, "solid")]
    sc = [ar.insert(b()) for b in build]
    for n in (1, 2, 18):
        ar.native.step_served_n(np.where(np.isin(np.arange(ar.S), sc), dt, np.float32(0.0)), n)
    for s, b in zip(sc, build):
        lp = fw.ExplicitLoop(5e-5, b(), useAdapativeDT=False)
        lp.advance_n(20)
        assert np.array_equal(ar.coords(s), lp.femSpringManager.coords.numpy()[: lp._packed.N])
    ar.close()


@pytest.mark.parametrize("n,ground", [(3, "plane"), (16, "plane"), (41, "bump"), (70, "bump"), (150, "plane")])
def test_reverse_pass_matches_the_gather_reverse(n, ground):
    """One patch, several, and meshes whose patches hold more than 512 triangles; contact on."""
    from flatworld_b200.diff import DiffSim

    def build():
        g = _plane(0.1 / n) if ground == "plane" else _bump(-1.0, 6.0)  # a quarter of a cell deep, whatever the mesh
        return _rectangle(n, n, MATS["neohookean"], g, cell=0.4 / n)

    dt = 0.05 * (0.4 / n) / 10.0
    a, b = DiffSim(build(), dt, 37, 15, damping=0.01), DiffSim(build(), dt, 37, 15, damping=0.01, path="gather")
    rng = np.random.default_rng(n)
    young = (5e4 * np.exp(0.1 * rng.standard_normal(a.E))).astype(np.float32)
    v0 = rng.standard_normal((a.N, 2)).astype(np.float32)
    seed = rng.standard_normal((a.N, 2)).astype(np.float32)
    xa, xb = a.forward(young, v0), b.forward(young, v0)
    assert np.array_equal(xa, xb)
    for u, v in zip(a.backward(seed, 0.1 * seed), b.backward(seed, 0.1 * seed)):
        assert np.abs(v).max() > 0 and np.array_equal(u, v)
