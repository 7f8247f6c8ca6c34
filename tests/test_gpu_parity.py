"""GPU parity of the FP64 path against the oracle (bit-exact) and of the mixed path
(per-grain volume within 1e-3 relative).

Cases are seeded Voronoi microstructures small enough for the oracle to finish in
seconds.  Stage tests check each batched kernel on the GPU's own inputs against the
oracle's single-box restatement; loop tests run both implementations side by side
and compare every step.
"""
import os

import numpy as np
import pytest

from gragles_3d_b200 import microstructure as msgen

pytestmark = pytest.mark.gpu

CASES = {
    "tiny": dict(N=32, G=20, border=5, seed=1032),
    "vanish": dict(N=40, G=150, border=5, seed=1040),
    "border10": dict(N=48, G=60, border=10, seed=1048),
}


def _case(name):
    c = CASES[name]
    ms = msgen.voronoi(c["N"], c["G"], seed=c["seed"])
    ext, counts = ms.grain_extents()
    return c, ms, ext, counts


def _default_lists_from(gh):
    """CSR of the GPU's default lists, fed to the oracle so both start identically."""
    G = gh.G
    off = np.zeros(G + 2, np.int64)
    ids = []
    for g in range(1, G + 1):
        l = gh.comparison_list(g)
        ids.extend(l.tolist())
        off[g + 1] = off[g] + len(l)
    return off, np.array(ids, np.uint32)


def _pair(gpu, oracle, name, precision=0):
    c, ms, ext, counts = _case(name)
    gh = gpu.GrainHandler(c["N"], c["border"], 0.2, c["G"], precision=precision)
    gh.load(ms.labels, ext, counts)
    gh.default_lists()
    lists = _default_lists_from(gh)
    osim = oracle.OracleSim(c["N"], c["border"], 0.2, ms.labels, ext, counts, lists=lists)
    return c, gh, osim


def test_convolution_kernel_bitexact(gpu, oracle):
    rng = np.random.default_rng(7)
    sides = [5, 8, 13, 20, 33, 34, 47]
    boxes = [rng.uniform(-0.1, 0.1, (n, n, n)) for n in sides]
    got = gpu.convolve_boxes_f64(boxes, 128, 0.2)
    for b, g in zip(boxes, got):
        want = oracle.convolve_box(b, 128, 0.2)
        assert np.array_equal(g, want), f"side {b.shape[0]}: max diff {np.abs(g - want).max()}"


@pytest.mark.parametrize("sides", [[1, 2, 3, 4], [7, 8, 9, 6, 15, 16, 17], [23, 24, 25, 39, 40, 41], [55, 56, 57, 40],
                                   [63, 64, 31], [65, 66, 8], [97, 81, 3]])
def test_convolution_kernel_bitexact_at_fragment_edges(gpu, oracle, sides):
    """Sides around the matrix instruction's 8 x 8 x 4 fragments (lines, frequencies and chain
    lengths with every remainder), around pass B's switch to two line buffers (above 64) and
    up to the largest side, the large ones beside small ones; the chains' order makes the
    result equal to the oracle's bit for bit."""
    rng = np.random.default_rng(17)
    boxes = [rng.uniform(-0.1, 0.1, (n, n, n)) for n in sides]
    got = gpu.convolve_boxes_f64(boxes, 100, 0.2)
    for b, g in zip(boxes, got):
        assert np.array_equal(g, oracle.convolve_box(b, 100, 0.2)), f"side {b.shape[0]}"


def test_mixed_convolution_kernel_accuracy(gpu, oracle):
    """The mixed path's convolution (tcgen05 with operands split into FP16 hi + lo, three MMAs per
    K-step, when all sides are <= 64; FP32 SIMT otherwise) against the FP64 specified DFT: FP32-level error, far below plain TF32's
    ~5e-4.  Side sets with repeated and alternating sides exercise the kernel's switch
    between its two C_n buffers."""
    rng = np.random.default_rng(8)
    for sides in ([5, 8, 13, 20, 33, 47, 64], [40, 40, 17, 40, 17, 17, 64, 1, 2, 64, 33] * 3, [96, 100]):
        boxes = [rng.uniform(-0.1, 0.1, (n, n, n)).astype(np.float32) for n in sides]
        got = gpu.convolve_boxes_mixed(boxes, 128, 0.2)
        for b, g in zip(boxes, got):
            want = oracle.convolve_box(b.astype(np.float64), 128, 0.2)
            err = np.abs(g.astype(np.float64) - want).max() / np.abs(b).max()
            assert err <= 4e-6, f"side {b.shape[0]}: relative max error {err:.3g}"


@pytest.mark.parametrize("sides", [[65, 20], [95, 97, 1], [128, 33], [139]])
def test_mixed_convolution_large_sides(gpu, oracle, sides):
    """The FP32 kernels for sides above 64: one to five 32-wide column groups, row groups with
    every remainder, smaller boxes in the same call, and the largest side, whose plane is
    staged by halves; FP32-level error as above."""
    rng = np.random.default_rng(18)
    boxes = [rng.uniform(-0.1, 0.1, (n, n, n)).astype(np.float32) for n in sides]
    for b, g in zip(boxes, gpu.convolve_boxes_mixed(boxes, 100, 0.2)):
        want = oracle.convolve_box(b.astype(np.float64), 100, 0.2)
        err = np.abs(g.astype(np.float64) - want).max() / np.abs(b).max()
        assert err <= 4e-6, f"side {b.shape[0]}: relative max error {err:.3g}"


def test_initial_sdf_bitexact(gpu, oracle):
    c, gh, osim = _pair(gpu, oracle, "tiny")
    for g in range(1, c["G"] + 1):
        ob, osdf = osim.sdf(g)
        gb, gsdf = gh.sdf(g, which=1)
        assert ob == gb
        assert np.array_equal(osdf, gsdf), f"grain {g}"


def test_stages_bitexact_on_gpu_inputs(gpu, oracle):
    """Each stage on the GPU's own inputs equals the oracle's restatement of it."""
    c, gh, _ = _pair(gpu, oracle, "border10")
    G, M, gb, N = c["G"], c["N"] + 2 * c["border"], c["border"], c["N"]
    h, delta = 1.0 / N, gb / float(N)
    for _ in range(2):
        # convolution
        gh.stage("convolution")
        conv = {}
        for g in range(1, G + 1):
            bi, sin = gh.sdf(g, which=0)
            bo, sout = gh.sdf(g, which=1)
            assert bi == bo
            want = oracle.convolve_box(sin, N, 0.2)
            assert np.array_equal(sout, want), f"convolution grain {g}"
            conv[g] = (bo, sout)
        ids_before = {g: gh.idlocal(g) for g in range(1, G + 1)}
        gh.stage("update_lists")
        lists = {g: gh.comparison_list(g) for g in range(1, G + 1)}
        gh.stage("comparison")
        for g in range(1, G + 1):
            box, sconv = conv[g]
            l = lists[g]
            # IDLocal follows the box by flat-prefix resize before the comparison
            ob_, oid = ids_before[g]
            n = int(np.prod([box[1] - box[0], box[3] - box[2], box[5] - box[4]]))
            idl = np.zeros(n, np.uint32)
            k = min(n, oid.size)
            idl[:k] = oid[:k]
            out, idl = oracle.compare_box(box, [conv[i][0] for i in l], l, [conv[i][1] for i in l], idl, M, gb, h)
            res, newbox = oracle.set_compare_box(box, sconv, out, delta, M, gb)
            gbx, gres = gh.sdf(g, which=0)
            assert gbx == box
            assert np.array_equal(gres, res), f"comparison grain {g}"
            ib, gid = gh.idlocal(g)
            assert ib == box and np.array_equal(gid, idl.ravel()), f"IDLocal grain {g}"
        cmp_state = {g: gh.sdf(g, which=0) for g in range(1, G + 1)}
        id_state = {g: gh.idlocal(g) for g in range(1, G + 1)}
        gh.stage("level_set")
        st = gh.stats()
        for g in range(1, G + 1):
            box, sdf = cmp_state[g]
            ntri, vol, sur, nbrs = oracle.mc_box(box, sdf, id_state[g][1], g, h)
            assert st.exists[g] == (ntri > 0)
            if ntri > 0:
                assert st.volume[g] == vol, f"volume grain {g}"
                assert st.surface[g] == sur, f"surface grain {g}"
                assert np.array_equal(gh.neighbors(g), nbrs), f"neighbours grain {g}"
        gh.stage("redistancing")
        for g in range(1, G + 1):
            if not st.exists[g]:
                continue
            ib, sin = cmp_state[g]
            ob, sout = gh.sdf(g, which=1)
            want = oracle.redistance_box(ib, sin, ob, h, delta)
            assert np.array_equal(sout, want), f"redistancing grain {g}"


@pytest.mark.parametrize("name,steps", [("tiny", 6), ("vanish", 45), ("border10", 12)])
def test_loop_fp64_bitexact(gpu, oracle, name, steps):
    c, gh, osim = _pair(gpu, oracle, name)
    G = c["G"]
    for s in range(steps):
        cnt_o = osim.step()
        rep = gh.step()
        assert rep["grain_count"] == cnt_o, f"step {s}: grain count"
        assert rep["voxel_updates"] == osim.last_voxels(), f"step {s}: voxel updates"
        st = gh.stats()
        for g in range(1, G + 1):
            inf = osim.info(g)
            assert bool(st.exists[g]) == inf["exists"], f"step {s} grain {g}: exists"
            if not inf["exists"]:
                continue
            assert tuple(st.boxes[g]) == inf["box"], f"step {s} grain {g}: box"
            assert st.volume[g] == inf["volume"], f"step {s} grain {g}: volume"
            assert st.surface[g] == inf["surface"], f"step {s} grain {g}: surface"
            assert np.array_equal(gh.neighbors(g), osim.neighbors(g)), f"step {s} grain {g}: neighbours"
            assert np.array_equal(gh.comparison_list(g), osim.comparison_list(g)), f"step {s} grain {g}: list"
    for g in range(1, G + 1):
        if osim.info(g)["exists"]:
            ob, osdf = osim.sdf(g)
            gb_, gsdf = gh.sdf(g, which=1)
            assert ob == gb_ and np.array_equal(osdf, gsdf), f"final SDF grain {g}"


@pytest.mark.parametrize("border", [4, 7])
@pytest.mark.parametrize("lists", ["reversed", "thinned"])
def test_comparison_of_ties_and_unlisted_neighbours_bitexact(gpu, oracle, border, lists):
    """A lattice of equal cubes, whose fields tie along every symmetry plane (the earliest
    list position decides), with lists in descending order, or with 40% of their members
    left out and some lists empty (unlisted candidates and voxels no listed neighbour
    covers keep their IDLocal): the fields and IDs equal the oracle's bit for bit."""
    n, c = 4, 6
    N, G = n * c, n ** 3
    ax = np.arange(N) // c
    lab = (1 + ax[None, None, :] + n * ax[None, :, None] + n * n * ax[:, None, None]).astype(np.uint32)
    cube = np.array([[x * c, x * c + c - 1, y * c, y * c + c - 1, z * c, z * c + c - 1]
                     for z in range(n) for y in range(n) for x in range(n)], np.int32)
    counts = np.full(G, c ** 3, np.int64)
    gh = gpu.GrainHandler(N, border, 0.2, G, precision=0)
    gh.load(lab, cube, counts)
    gh.default_lists()
    rng = np.random.default_rng(5)
    rows = []
    for g in range(1, G + 1):
        r = gh.comparison_list(g)
        rows.append(r[::-1] if lists == "reversed" else (r[rng.random(r.size) < 0.6] if g % 9 else r[:0]))
    off = np.concatenate([[0, 0], np.cumsum([r.size for r in rows])]).astype(np.int64)
    ids = np.concatenate(rows).astype(np.uint32)
    gh.set_lists(off, ids)
    osim = oracle.OracleSim(N, border, 0.2, lab, cube, counts, lists=(off, ids))
    for s in range(3):
        assert gh.step()["grain_count"] == osim.step(), f"step {s}"
        st = gh.stats()
        for g in range(1, G + 1):
            inf = osim.info(g)
            assert bool(st.exists[g]) == inf["exists"], f"step {s} grain {g}"
            assert np.array_equal(gh.comparison_list(g), osim.comparison_list(g)), f"step {s} grain {g}: list"
            if inf["exists"]:
                assert tuple(st.boxes[g]) == inf["box"] and st.volume[g] == inf["volume"], f"step {s} grain {g}"
                ob, oid = osim.idlocal(g)
                gb, gid = gh.idlocal(g)
                assert ob == gb and np.array_equal(oid, gid), f"step {s} grain {g}: IDLocal"
                assert np.array_equal(osim.sdf(g)[1], gh.sdf(g)[1]), f"step {s} grain {g}: field"


@pytest.mark.parametrize("G", [40, 220, 420])
def test_contour_at_every_cta_size_bitexact(gpu, oracle, G):
    """The marching-cubes kernel's CTA size goes with the number of grains (few, some, many
    against the SMs): volumes, surfaces and neighbours in first-seen order equal the oracle's."""
    ms = msgen.voronoi(38, G, seed=3000 + G)
    ext, counts = ms.grain_extents()
    gh = gpu.GrainHandler(38, 5, 0.2, G, precision=0)
    gh.load(ms.labels, ext, counts)
    gh.default_lists()
    osim = oracle.OracleSim(38, 5, 0.2, ms.labels, ext, counts, lists=_default_lists_from(gh))
    for s in range(2):
        assert gh.step()["grain_count"] == osim.step()
    st = gh.stats()
    for g in range(1, G + 1):
        inf = osim.info(g)
        assert bool(st.exists[g]) == inf["exists"], f"grain {g}"
        if inf["exists"]:
            assert st.volume[g] == inf["volume"] and st.surface[g] == inf["surface"], f"grain {g}"
            assert np.array_equal(gh.neighbors(g), osim.neighbors(g)), f"grain {g}"


def test_redistancing_at_class_edges_bitexact(gpu, oracle):
    """Output boxes at the edges of the redistancing's size classes beside each other in one step:
    56 | 57 (two classes), 63 and 64 (the last bits of the 64-bit sign masks), 65 to 67 (runtime
    pitch) and small ones; every field equals the oracle's bit for bit.  Eight slabs of 8
    layers, each with one square grain and four in the rest."""
    n, border = 64, 5
    lab = np.zeros((n, n, n), np.int64)
    G = 0
    for k, a in enumerate((47, 48, 54, 55, 56, 57, 58, 30)):
        for ys, xs in ((slice(0, a), slice(0, a)), (slice(0, 32), slice(a, n)), (slice(32, n), slice(a, n)),
                       (slice(a, n), slice(0, a // 2)), (slice(a, n), slice(a // 2, a))):
            G += 1
            lab[8 * k:8 * k + 8, ys, xs] = G
    ms = msgen.Microstructure(lab.astype(np.uint32), np.zeros((G, 3)), np.zeros(G), np.zeros((G, 3)))
    ext, counts = ms.grain_extents()
    gh = gpu.GrainHandler(n, border, 0.2, G, precision=0)
    gh.load(ms.labels, ext, counts)
    gh.default_lists()
    osim = oracle.OracleSim(n, border, 0.2, ms.labels, ext, counts, lists=_default_lists_from(gh))
    for s in range(3):
        assert gh.step()["grain_count"] == osim.step()
        st = gh.stats()
        sides = set(int(b[1] - b[0]) for g, b in enumerate(st.boxes) if st.exists[g])
        assert {33, 56, 57, 63, 64, 65, 66, 67} <= sides
        for g in range(1, G + 1):
            inf = osim.info(g)
            assert bool(st.exists[g]) == inf["exists"] and tuple(st.boxes[g]) == inf["box"], f"step {s} grain {g}"
            assert np.array_equal(osim.sdf(g)[1], gh.sdf(g)[1]), f"step {s} grain {g}: field"


def test_loop_mixed_volume_tolerance(gpu, oracle):
    c, gh, osim = _pair(gpu, oracle, "border10", precision=1)
    worst = 0.0
    for s in range(12):
        osim.step()
        gh.step()
        st = gh.stats()
        for g in range(1, c["G"] + 1):
            inf = osim.info(g)
            if inf["exists"] and st.exists[g]:
                worst = max(worst, abs(st.volume[g] - inf["volume"]) / inf["volume"])
    assert worst <= 1e-3, f"max relative volume error {worst}"


def test_long_isotropic_run_mixed_tracks_fp64(gpu):
    """Over 150 isotropic steps (80^3, 400 grains, about one in eight vanish) the mixed
    path's per-grain volumes stay with the FP64 path's: median below 1e-5, 99th percentile
    below 1e-4, all but 1% of grains within 1e-3 (a grain that is shrinking to nothing can
    pass it for a step), and the same grains alive up to a grain or two whose vanishing
    step a rounding can move."""
    N, G, S = 80, 400, 150
    ms = msgen.voronoi(N, G, seed=1080)
    ext, counts = ms.grain_extents()
    hs = []
    for prec in (1, 0):
        gh = gpu.GrainHandler(N, 10, 0.2, G, precision=prec)
        gh.load(ms.labels, ext, counts)
        gh.default_lists()
        hs.append(gh)
    for s in range(1, S + 1):
        for gh in hs:
            gh.step()
        if s % 50:
            continue
        sm, sd = hs[0].stats(), hs[1].stats()
        assert int((sm.exists[1:] != sd.exists[1:]).sum()) <= 2, f"step {s}: grains alive differ"
        both = sm.exists & sd.exists
        both[0] = False
        rel = np.abs(sm.volume[both] - sd.volume[both]) / sd.volume[both]
        assert np.median(rel) < 1e-5, f"step {s}: median {np.median(rel)}"
        assert np.quantile(rel, 0.99) <= 1e-4, f"step {s}: 99th percentile {np.quantile(rel, 0.99)}"
        assert (rel > 1e-3).mean() <= 0.01, f"step {s}: {(rel > 1e-3).sum()} grains above 1e-3"
    assert int(sd.exists[1:].sum()) < 0.95 * G


def _container_from_oracle(osim, N, border, G):
    """LSbox::copyDataToContainer (box.cpp:3008-3032) over the oracle's grains in
    ascending ID order: a voxel takes the ID of the last grain whose output SDF is >= 0
    there.  Grains whose hull vanished must hold no such voxel (the GPU leaves them out)."""
    want = np.zeros((N, N, N), np.uint32)
    for g in range(1, G + 1):
        inf = osim.info(g)
        if not inf["present"]:
            continue
        (x0, x1, y0, y1, z0, z1), sdf = osim.sdf(g)
        if sdf.size == 0:
            continue
        inside = sdf >= 0
        if not inf["exists"]:
            assert not inside.any(), f"grain {g}: vanished hull with voxels >= 0"
            continue
        zs, ys, xs = np.nonzero(inside)
        zs, ys, xs = zs + z0 - border, ys + y0 - border, xs + x0 - border
        ok = (zs >= 0) & (ys >= 0) & (xs >= 0) & (zs < N) & (ys < N) & (xs < N)
        want[zs[ok], ys[ok], xs[ok]] = g
    return want


@pytest.mark.parametrize("precision", [0, 1])
def test_voxel_container_matches_oracle(gpu, oracle, precision):
    """saveNetworkAsVoxelContainer's label volume: exact on the FP64 path at every
    checked step, including steps where grains vanish; the mixed path's differs only
    where an SDF sits within its rounding of 0."""
    c, gh, osim = _pair(gpu, oracle, "vanish", precision=precision)
    N, G = c["N"], c["G"]
    for s in range(30):
        osim.step()
        gh.step()
        if s % 6 != 5:
            continue
        got = gh.voxel_container()
        want = _container_from_oracle(osim, N, c["border"], G)
        if precision == 0:
            assert np.array_equal(got, want), f"step {s}: {(got != want).sum()} voxels differ"
        else:
            assert (got != want).mean() < 1e-3, f"step {s}: {(got != want).sum()} voxels differ"


def test_c1_fp64_matches_reference_golden(gpu):
    """The plain-method configuration at full length: 64^3, 200 Voronoi grains, 10-voxel
    border, 50 timesteps (51 loop iterations), started from the library's R-tree lists
    (gg_rtree_lists), which must equal the reference's own (tests/golden/c1.npz, written by
    the compiled reference).  Every
    loop: existence, boxes, volumes and surfaces bit for bit, hull neighbours in
    first-seen order, and the grain-count trajectory; the comparison lists of the last
    loop in order."""
    d = dict(np.load(os.path.join(os.path.dirname(__file__), "golden", "c1.npz")))
    N, G, border = int(d["N"]), int(d["G"]), int(d["border"])
    ms = msgen.voronoi(N, G, seed=int(d["seed"]))
    ext, counts = ms.grain_extents()
    gh = gpu.GrainHandler(N, border, 0.2, G, precision=gpu.PRECISION_FP64)
    gh.load(ms.labels, ext, counts)
    # the library's own R-tree lists are the reference's initial lists, in order
    gh.rtree_lists()
    for g in range(1, G + 1):
        want = d["init_list_ids"][d["init_list_off"][g]:d["init_list_off"][g + 1]]
        assert np.array_equal(gh.comparison_list(g), want), f"grain {g}: initial list"
    nb_base = np.concatenate([[0], np.cumsum(d["nb_len"])])
    li_base = np.concatenate([[0], np.cumsum(d["list_len"])])
    loops = d["exists"].shape[0]
    assert loops == int(d["steps"]) + 1
    for s in range(loops):
        gh.step()
        st = gh.stats()
        assert int(st.exists[1:].sum()) == int(d["exists"][s, 1:].sum()), f"loop {s}: grain count"
        nb_ids = d["nb_ids"][nb_base[s]:nb_base[s + 1]]
        for g in range(1, G + 1):
            assert bool(st.exists[g]) == bool(d["exists"][s, g]), f"loop {s} grain {g}: exists"
            if not st.exists[g]:
                continue
            assert tuple(st.boxes[g]) == tuple(d["box"][s, g]), f"loop {s} grain {g}: box"
            assert st.volume[g] == d["volume"][s, g], f"loop {s} grain {g}: volume"
            assert st.surface[g] == d["surface"][s, g], f"loop {s} grain {g}: surface"
            want = nb_ids[d["nb_off"][s][g]:d["nb_off"][s][g + 1]]
            assert np.array_equal(gh.neighbors(g), want), f"loop {s} grain {g}: neighbours"
    li_ids = d["list_ids"][li_base[loops - 1]:li_base[loops]]
    for g in range(1, G + 1):
        want = li_ids[d["list_off"][loops - 1][g]:d["list_off"][loops - 1][g + 1]]
        if want.size:
            assert np.array_equal(gh.comparison_list(g), want), f"grain {g}: final comparison list"
    gh.close()


def test_autotuned_launches_give_the_same_bits(gpu, oracle):
    """The autotuner (gg_params.autotune) times five launch configurations on loops 1-5 and
    keeps each stage's fastest; every stage kernel's results are independent of its grid,
    so the FP64 run stays bit-identical to an untuned one (and the oracle's)."""
    N, G, border = 40, 150, 5
    ms = msgen.voronoi(N, G, seed=1040)
    ext, counts = ms.grain_extents()
    runs = []
    for tune in (False, True):
        gh = gpu.GrainHandler(N, border, 0.2, G, precision=gpu.PRECISION_FP64, autotune=tune)
        gh.load(ms.labels, ext, counts)
        gh.rtree_lists()
        hist = []
        for _ in range(9):
            gh.step()
            st = gh.stats()
            hist.append((st.exists.copy(), st.volume.copy(), st.boxes.copy()))
        cfg, done = gh.launch_config()
        assert done
        if tune:
            assert all(c in (2, 4, 8, 16, 32) for c in cfg), cfg
        runs.append(hist)
        gh.close()
    for (ea, va, ba), (eb, vb, bb) in zip(*runs):
        assert np.array_equal(ea, eb) and np.array_equal(va, vb) and np.array_equal(ba, bb)


@pytest.mark.parametrize("correction", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_autotuner_leaves_entries_alone_that_no_kernel_reads(gpu, precision, correction):
    """The convolutions and the redistancing size their own grids: the autotuner reports the
    default for the redistancing, and for the convolution's stage without the correction."""
    N, G = 32, 60
    ms = msgen.voronoi(N, G, seed=1032)
    ext, counts = ms.grain_extents()
    cfg = {}
    for tune in (False, True):
        with gpu.GrainHandler(N, 5, 0.2, G, precision=precision, autotune=tune, correction=correction,
                              unique_energies=False, mobility_model=True) as gh:
            gh.load(ms.labels, ext, counts)
            gh.default_lists()
            gh.set_orientations(ms.euler)
            for _ in range(6):
                gh.step()
            cfg[tune], done = gh.launch_config()
            assert done
    assert cfg[True][4] == cfg[False][4]
    if not correction:
        assert cfg[True][0] == cfg[False][0]
    assert all(c in (2, 4, 8, 16, 32) for c in cfg[True])


def test_cpp_host_runs_the_reference_mode4_case(gpu, tmp_path):
    """The C++ host (gragles_3d_b200/gg_run, the reference's mode-4 main over the C ABI) reads
    the reference's own input files and parameters.xml and reproduces the compiled
    reference's run of the plain-method configuration: every loop's sum of the existing
    grains' volumes, summed in grain order, equals the reference's bit for bit."""
    import subprocess

    d = dict(np.load(os.path.join(os.path.dirname(__file__), "golden", "c1.npz")))
    N, G, border, steps = int(d["N"]), int(d["G"]), int(d["border"]), int(d["steps"])
    ms = msgen.voronoi(N, G, seed=int(d["seed"]))
    msgen.write_mode4(ms, str(tmp_path))
    params = os.path.join(str(tmp_path), "parameters.xml")
    msgen.write_parameters(params, n_grains=G, border=border, steps=steps)
    runner = os.path.join(os.path.dirname(gpu.LIB_PATH), "gg_run")
    stats = os.path.join(str(tmp_path), "stats.txt")
    proc = subprocess.run([runner, params, "--stats", stats], capture_output=True, text=True, timeout=600)
    assert proc.returncode == 0, proc.stderr
    rows = [line.split("\t") for line in open(stats).read().splitlines()]
    assert len(rows) == steps + 1
    for s, r in enumerate(rows):
        want = 0.0
        for g in range(1, G + 1):
            if d["exists"][s, g]:
                want += d["volume"][s, g]
        assert int(r[0]) == s and float(r[3]) == want, f"loop {s}: {r[3]} vs {want!r}"
