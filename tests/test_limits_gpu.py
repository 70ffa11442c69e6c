"""GPU: calls at the limits of the kernels' counts and of the caller's memory."""
import ctypes
import mmap

import numpy as np
import pytest

from test_deposit_gpu import adeco, check_cells  # noqa: F401  (adeco: the fixture)

pytestmark = pytest.mark.gpu


def folded_patches(m, count):
    """Patch 0 folds its cubes onto the unit cube (vertex i at i mod 2) and
    leaves 11 of them, 66 tets, alive; the others are padding."""
    v = m + 1
    p = np.full((count, v, v, v, 3), 666.0, np.float32)
    z, y, x = np.meshgrid(*[np.arange(v)] * 3, indexing="ij")
    own = np.stack([x % 2, y % 2, z % 2], -1).astype(np.float32)
    p[0, :2] = own[:2]            # the 9 cubes of the lowest layer
    p[0, 2, :2, :3] = own[2, :2, :3]  # and 2 of the next
    return p.reshape(-1)


def test_wave_of_more_than_2_31_pairs(adeco):
    """66 tets of one block that each cover a grid of 322^3 cells: 2.2e9
    candidate pairs in one wave (2000 patches, so that each is one unit of
    work), against the FP64 path.

    A partial cell's share comes from FP32 coordinates of up to 644 cells,
    rounded by 4e-5 of a cell (6e-8 relative): under 1e-3 of the mean cell.
    Cells cut by a face are a few in a hundred, and a sum's quantum, 2^-43, is
    5e-6 of a cube's mass in a cell, rounded the same way in most cells: the
    total holds to 1e-5."""
    m, count, dims = 3, 2000, 322
    box = np.array([0.25, 0.75] * 3, np.float32)
    pos = folded_patches(m, count)
    got = adeco.deposit_tets_ex(pos, m, box, dims, num_patches=count)
    want = adeco.deposit_tets_ex(pos, m, box, dims, num_patches=1, precision=1)  # the padding adds nothing
    # the reference's corner order covers a cube once on average, not evenly
    assert abs(want.mean() / (66.0 * (0.5 / dims) ** 3) - 1.0) < 1e-2
    assert abs(got.sum() / want.sum() - 1.0) < 1e-5
    assert np.abs(got - want).max() < 1e-3 * want.mean()


@pytest.mark.parametrize("precision", [0, 1], ids=["mixed", "plain_fp64"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("box", [(0.5, 4.5), (-9.0, 3.0), (40.0, 44.0)], ids=["whole", "part", "empty"])
def test_grid_off_its_cells_alignment(adeco, box, dtype, precision):
    """A caller's grid that starts between two cells gains what an aligned one
    does: the sums come back and are added by the host.  (Bit for bit; the FP64
    path's atomic sums differ by their order, some 100 adds a cell: 1e-13.)"""
    dims, m = 21, 5
    rng = np.random.default_rng(5)
    v = np.stack(np.meshgrid(*[np.arange(m + 1.0)] * 3, indexing="ij"), -1)[..., ::-1]
    pos = (v + rng.uniform(-0.3, 0.3, v.shape)).astype(np.float32).reshape(-1)
    bb = np.array(box * 3, np.float32)
    n, size = dims ** 3, np.dtype(dtype).itemsize
    pre = rng.uniform(0.5, 2.0, n).astype(dtype)
    want = adeco.deposit_tets_ex(pos, m, bb, dims, data=pre.copy(), precision=precision)
    for offset in (1, 2, size - 1, size + 2):
        room = np.full(n * size + 32, 7, np.uint8)
        room[offset:offset + n * size] = pre.view(np.uint8)
        got = room[offset:offset + n * size].view(dtype)
        assert not got.flags.aligned and got.flags.c_contiguous
        adeco.deposit_tets_ex(pos, m, bb, dims, data=got, precision=precision)
        got = np.array(got)
        assert np.array_equal(got, want) if precision == 0 else np.allclose(got, want, rtol=1e-13 if size == 8 else 1e-6)
        assert np.all(room[:offset] == 7) and np.all(room[offset + n * size:] == 7)
    assert (want.sum() > pre.sum()) == (box[0] < 40.0)


@pytest.mark.parametrize("shift,rows", [(0.0, (0, 3)), (50.0, (23, 28)), (-200.0, None)], ids=["corner", "slab", "outside"])
def test_only_the_pages_of_the_box_become_resident(adeco, shift, rows):
    """A 64 MB grid that the caller never touched: a call that meets some
    layers of cells makes the pages of those resident, a call beside the grid
    none."""
    dims, m = 256, 4
    page = mmap.PAGESIZE
    rng = np.random.default_rng(3)
    v = np.stack(np.meshgrid(*[np.arange(m + 1.0)] * 3, indexing="ij"), -1)[..., ::-1] + rng.uniform(-0.2, 0.2, (m + 1,) * 3 + (3,))
    v[..., 2] += shift
    box = np.array([0.5, 512.5] * 3, np.float32)  # cells of 2
    mem = mmap.mmap(-1, 4 * dims ** 3, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    mem.madvise(mmap.MADV_NOHUGEPAGE)
    grid = np.frombuffer(mem, np.float32)
    adeco.deposit_tets_ex(v.astype(np.float32).reshape(-1), m, box, dims, data=grid)
    vec = (ctypes.c_ubyte * (len(mem) // page))()
    libc = ctypes.CDLL(None, use_errno=True)
    assert libc.mincore(ctypes.c_void_p(grid.ctypes.data), ctypes.c_size_t(len(mem)), vec) == 0
    resident = np.flatnonzero(np.frombuffer(vec, np.uint8) & 1) * page // (4 * dims * dims)  # their layers
    if rows is None:
        assert resident.size == 0
    else:
        assert resident.size > 0 and resident.min() >= rows[0] and resident.max() <= rows[1]
        assert grid.sum() > 0
    assert (grid.sum() == 0) == (rows is None)


def test_leaf_lists_of_repeated_builds(adeco):
    """Builds of growing and shrinking size in one session: the leaves' lists
    that come back from the device are the host builder's, whichever built
    them, and so are the leaves' sums.  (The host builder's lists go to the
    device and come back with the leaves' cubes behind them.)"""
    from adeco_gb300.synthetic import zeldovich_lattice
    pos = zeldovich_lattice(64, L=64.0, seed=12, rms_disp=2.0)
    with adeco.Session(pos) as s:
        for max_tets in (60000, 1500, 20000, 400, 1500):
            lists, grids = [], []
            for builder in ("device", "host"):
                info = s.build_octree(max_tets, 8, leaf_dims=2, builder=builder)
                lists.append([s.leaf_meta(q) for q in range(len(info.leaves))])
                grids.append(s.deposit_leaves()[0])
            assert len(lists[0]) == len(lists[1])
            assert all(np.array_equal(a, b) for a, b in zip(*lists))
            assert np.array_equal(*grids)


@pytest.mark.parametrize("dims", [63, 64, 73, 74, 80, 81, 102, 138])
def test_results_copied_by_one_or_several_threads(adeco, dims):
    """Results of 2.0 to 21 MB, around where the copy to the caller takes its
    second, third, fourth and fifth thread: whole, the same each time, and the same
    when they start at another place of the batch's block."""
    from adeco_gb300.synthetic import zeldovich_lattice
    pos = zeldovich_lattice(24, L=24.0, seed=5, rms_disp=1.0)
    req = ((11.0, 12.0, 13.0), 18.0, dims)
    with adeco.Session(pos) as s:
        b = s.submit([req])
        s.wait(b)
        first, again = s.result(b, 0, dims), s.result(b, 0, dims)
        s.release(b)
        b = s.submit([((12.0, 12.0, 12.0), 5.0, 3), req])
        s.wait(b)
        third = s.result(b, 1, dims)
        s.release(b)
    assert np.array_equal(first, again) and np.array_equal(first, third)
    assert (first.reshape(-1)[-dims:] > 0).any() and (first > 0).mean() > 0.9


@pytest.mark.parametrize("order", [0, 1], ids=["ref", "conforming"])
@pytest.mark.parametrize("dims", [1, 2, 3, 8])
def test_whole_tets_on_coarse_grids(adeco, oracle, dims, order):
    """Grids much coarser than the tets, where most lanes of a warp add a whole
    tet to the same few cells: one cell that holds everything gains exactly a
    mass per tet; others are within the mixed path's bar of the FP64 oracle.
    The same through a session's zoom request and leaves."""
    from adeco_gb300.synthetic import zeldovich_lattice
    m = 14
    pos = zeldovich_lattice(m + 1, L=15.0, seed=6, rms_disp=0.3)
    lo, hi = float(pos.min()) - 0.25, float(pos.max()) + 0.25
    box = np.array([lo, hi] * 3, np.float32)
    n_tets = 6 * m ** 3
    got = adeco.deposit_tets_ex(pos.reshape(-1), m, box, dims, tet_order=order)
    ref = oracle.deposit_patches(pos.reshape(-1), m, box, dims, fp64=True, order=order)
    check_cells(got, ref, n_tets=n_tets)
    side, mid = float(box[1] - box[0]), 0.5 * float(box[0] + box[1])
    with adeco.Session(pos, tet_order=order) as s:
        b = s.submit([((mid, mid, mid), 1.02 * side, dims)])
        s.wait(b)
        zoom = s.result(b, 0, dims)
        s.release(b)
        s.build_octree(10 ** 9, 0, leaf_dims=dims)
        leaf = s.deposit_leaves()[0]
    # the request's box is not the grid's: its total, and that of the leaf (the particles' own box), only
    tol = 1e-9 * n_tets + 3e-7 * np.sqrt(n_tets)
    assert abs(zoom.sum() - n_tets) <= tol and abs(leaf.sum() - n_tets) <= tol
    if dims == 1:
        assert got.sum() == n_tets and zoom.sum() == n_tets


@pytest.mark.parametrize("precision", [0, 1], ids=["mixed", "plain_fp64"])
def test_calls_beside_and_inside_the_grid_in_turn(adeco, oracle, precision):
    """A launch whose vertices cannot meet the grid ends at once: only that
    one.  Boxes beside the patches, touching them by a face, holding one
    corner, and a NaN vertex among patches that lie outside otherwise."""
    m = 4
    rng = np.random.default_rng(9)
    v = np.stack(np.meshgrid(*[np.arange(m + 1.0)] * 3, indexing="ij"), -1)[..., ::-1] + rng.uniform(-0.2, 0.2, (m + 1,) * 3 + (3,))
    v[0, 0, 0] = 0.0
    v = np.maximum(v, 0.0).astype(np.float32)
    tol = dict(rel=1e-5, abs_=1e-7) if precision == 0 else dict(rel=1e-10, abs_=1e-12)
    for lo, hi, meets in ((9.0, 11.0, False), (1.0, 3.0, True), (-2.0, 0.0, False), (-2.0, 0.5, True), (50.0, 52.0, False)):
        box = np.array([lo, hi] * 3, np.float32)
        got = adeco.deposit_tets_ex(v.reshape(-1), m, box, 6, precision=precision)
        check_cells(got, oracle.deposit_patches(v.reshape(-1), m, box, 6, fp64=True), n_tets=6 * m ** 3, **tol)
        assert (got.sum() > 0) == meets
    odd = v.copy()
    odd[m, m, m, 1] = np.nan
    got = adeco.deposit_tets_ex(odd.reshape(-1), m, np.array([1.0, 2.5] * 3, np.float32), 6, precision=precision)
    want = adeco.deposit_tets_ex(v.reshape(-1), m, np.array([1.0, 2.5] * 3, np.float32), 6, precision=precision)
    assert np.allclose(got, want, rtol=1e-13)  # the tets of that vertex lie outside this box
