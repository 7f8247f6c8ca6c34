"""Capacity errors of the device pool and the list rows, raised on the host side of the
C ABI and by the kernels' own checks (nothing faults: an over-capacity kernel skips
the access and sets an error bit that the host turns into a status code).

The reference has no such limits (its boxes, lists and hulls are std::vectors); the
device pool and the fixed-capacity rows here replace them, so running out is an error
the caller must see, with a message naming the capacity, and the context must still
answer read-back calls afterwards.
"""
import numpy as np
import pytest

from gragles_3d_b200 import microstructure as msgen

pytestmark = pytest.mark.gpu


def _case(N=40, G=60, seed=7):
    ms = msgen.voronoi(N, G, seed=seed)
    ext, counts = ms.grain_extents()
    return ms, ext, counts


def test_pool_smaller_than_the_initial_boxes(gpu):
    ms, ext, counts = _case()
    G = ms.n_grains
    with gpu.GrainHandler(ms.n, 6, 0.2, G, precision=gpu.PRECISION_FP64) as big:
        big.load(ms.labels, ext, counts)
        st = big.stats()
        need = sum((int(b[1] - b[0]) ** 3 + 31) // 32 * 32 for g, b in enumerate(st.boxes) if g and st.exists[g])
    with gpu.GrainHandler(ms.n, 6, 0.2, G, precision=gpu.PRECISION_FP64, pool_voxels=need - 32) as gh:
        with pytest.raises(gpu.GGError) as ei:
            gh.load(ms.labels, ext, counts)
        assert ei.value.code == gpu.GG_ERR_POOL_EXHAUSTED
        assert f"pool holds {need - 32}" in str(ei.value) and f"need {need} voxels" in str(ei.value)
    # exactly enough: loads and steps
    with gpu.GrainHandler(ms.n, 6, 0.2, G, precision=gpu.PRECISION_FP64, pool_voxels=need) as gh:
        gh.load(ms.labels, ext, counts)
        gh.default_lists()
        gh.step()
        assert gh.stats().exists[1:].any()


def test_hull_capacity_exhausted_in_the_loop(gpu):
    """The correction's hull capture holds hull_capacity triangles per grain; a hull
    with more stops the step with GG_ERR_POOL_EXHAUSTED, and nothing past the capture
    arrays is written (read-back still works)."""
    ms, ext, counts = _case()
    G = ms.n_grains
    with gpu.GrainHandler(ms.n, 6, 0.2, G, precision=gpu.PRECISION_FP64, correction=True, unique_energies=False,
                          mobility_model=True, hull_capacity=8) as gh:
        gh.load(ms.labels, ext, counts)
        gh.default_lists()
        gh.set_orientations(ms.euler)
        with pytest.raises(gpu.GGError) as ei:
            gh.step()
        assert ei.value.code == gpu.GG_ERR_POOL_EXHAUSTED
        assert "hull_capacity" in str(ei.value)
        st = gh.stats()
        assert st.exists.shape == (G + 1,)
        assert np.isfinite(st.volume).all()


def test_list_capacity_exhausted(gpu):
    """Comparison lists longer than list_capacity: refused by gg_set_lists on the host,
    and flagged by the device-built default lists."""
    ms, ext, counts = _case()
    G = ms.n_grains
    with gpu.GrainHandler(ms.n, 6, 0.2, G, precision=gpu.PRECISION_FP64) as ref:
        ref.load(ms.labels, ext, counts)
        ref.default_lists()
        lens = [len(ref.comparison_list(g)) for g in range(1, G + 1)]
    cap = max(lens) - 1
    assert cap > 0
    with gpu.GrainHandler(ms.n, 6, 0.2, G, precision=gpu.PRECISION_FP64, list_capacity=cap) as gh:
        gh.load(ms.labels, ext, counts)
        with pytest.raises(gpu.GGError) as ei:
            gh.default_lists()
        assert ei.value.code == gpu.GG_ERR_LIST_OVERFLOW
        assert "list capacity" in str(ei.value)
        assert gh.stats().exists[1:].any()
        # the same lists from the host are refused before anything is copied
        off = np.zeros(G + 2, np.int64)
        ids = np.concatenate([np.arange(1, n + 1, dtype=np.uint32) % G + 1 for n in lens])
        off[2:] = np.cumsum(lens)
        with pytest.raises(gpu.GGError) as ei:
            gh.set_lists(off, ids)
        assert ei.value.code == gpu.GG_ERR_LIST_OVERFLOW
        assert f"has {max(lens)} entries" in str(ei.value)


def test_element_build_overflow_is_named_whatever_it_runs_beside(gpu):
    """A capacity of the element build runs out (one cube of 20^3 among 4^3 cubes: fewer than 256
    neighbours, more than 256 distinct neighbour lists): the step fails with the same code and
    text, the capacity named, whether the overflow happens before or after the redistancing's
    plan is checked, and the read-back calls still answer."""
    n, c = 36, 4
    ax = np.arange(n) // c
    cells = n // c
    lab = 2 + ax[None, None, :] + cells * ax[None, :, None] + cells * cells * ax[:, None, None]
    lab[8:28, 8:28, 8:28] = 1
    _, lab = np.unique(lab, return_inverse=True)
    lab = (1 + lab.reshape(n, n, n)).astype(np.uint32)
    G = int(lab.max())
    ms = msgen.Microstructure(labels=lab, euler=np.zeros((G, 3)), stored_energy=np.zeros(G), seeds=np.zeros((G, 3)))
    ext, counts = ms.grain_extents()
    texts = set()
    for precision in (gpu.PRECISION_FP64, gpu.PRECISION_MIXED):
        for beside in (0, 1, -1, -1):
            with gpu.GrainHandler(n, 5, 0.2, G, precision=precision, correction=True, unique_energies=False,
                                  mobility_model=True) as gh:
                gh.set_work_split(elements_beside=beside)
                gh.load(lab, ext, counts)
                gh.default_lists()
                with pytest.raises(gpu.GGError) as ei:
                    gh.step()
                assert ei.value.code == gpu.GG_ERR_POOL_EXHAUSTED
                texts.add(str(ei.value))
                assert gh.stats().exists.shape == (G + 1,)
                assert len(gh.neighbors(1)) <= 256
    (text,) = texts
    assert "redistancing plan: more than 256 distinct neighbour lists" in text
