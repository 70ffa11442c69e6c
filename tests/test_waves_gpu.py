"""GPU: the edges of the deposit kernels' work splitting, against the FP64
oracle or the other path to the same result.

* Patches of 1 cube (6 tets) to 9^3 cubes in several patches: waves with a
  remainder, an item shared by many CTAs, more partial pairs in a wave than the
  pair list holds (few tets over many cells), tets wide enough for rows of
  cells, and lattices squashed so that every tet is ill-conditioned.
  Tolerances are those of test_deposit_gpu.py: 1e-5 relative + 1e-7 tet masses
  for the mixed path, 1e-10 + 1e-12 for plain FP64.
* Sums added into the caller's grid wherever it lies in memory, results of
  requests of any size, and leaf work made on the device or by the host are
  compared bit for bit.
"""
import numpy as np
import pytest

from test_deposit_gpu import ABS, REL, adeco, check_cells  # noqa: F401  (adeco: the fixture)

pytestmark = pytest.mark.gpu


def patches(m, count, squash, seed):
    """count patches of m^3 cubes along x, jittered; z scaled by squash."""
    rng = np.random.default_rng(seed)
    v = m + 1
    z, y, x = np.meshgrid(*[np.arange(v, dtype=np.float64)] * 3, indexing="ij")
    out = []
    for k in range(count):
        p = np.stack([x + k * m, y, z], -1) + rng.uniform(-0.3, 0.3, (v, v, v, 3))
        p[..., 2] *= squash
        out.append(p.reshape(-1))
    return np.concatenate(out).astype(np.float32)


@pytest.mark.parametrize("squash", [1.0, 0.01], ids=["cubic", "flat"])
@pytest.mark.parametrize("m,count,dims", [(1, 1, 5), (1, 1, 70), (2, 3, 33), (3, 1, 64), (7, 1, 24), (8, 2, 9), (9, 1, 17)])
@pytest.mark.parametrize("precision", [0, 1], ids=["mixed", "plain_fp64"])
def test_patch_shapes_vs_oracle(adeco, oracle, precision, m, count, dims, squash):
    pos = patches(m, count, squash, seed=100 * m + dims)
    side = np.float32(m * count + 1)  # cubic box around the patches
    box = np.array([-0.5, side - 0.5, -0.5, side - 0.5, -0.5, side - 0.5], np.float32)
    got = adeco.deposit_tets_ex(pos, m, box, dims, num_patches=count, precision=precision)
    ref = oracle.deposit_patches(pos, m, box, dims, fp64=True, num_patches=count)
    tol = dict(rel=REL, abs_=ABS) if precision == 0 else dict(rel=1e-10, abs_=1e-12)
    check_cells(got, ref, n_tets=6 * count * m ** 3 if precision == 0 else 0, **tol)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_sums_added_at_any_address(adeco, dtype, offset):
    """A caller's grid that starts at an odd element of a buffer gains what an
    aligned one does, and its neighbours in the buffer nothing."""
    dims, m = 21, 5
    pos = patches(m, 1, 1.0, seed=5)
    box = np.array([0.5, 4.5] * 3, np.float32)
    n = dims ** 3
    pre = np.random.default_rng(6).uniform(0.5, 2.0, n).astype(dtype)
    want = adeco.deposit_tets_ex(pos, m, box, dims, data=pre.copy())
    room = np.full(n + 8, 7, dtype)
    room[offset:offset + n] = pre
    adeco.deposit_tets_ex(pos, m, box, dims, data=room[offset:offset + n])
    assert np.array_equal(room[offset:offset + n], want)
    assert np.all(room[:offset] == 7) and np.all(room[offset + n:] == 7)


def test_requests_of_any_size_same_alone_and_together(adeco):
    """Requests of 1^3 to 66^3 cells, their results starting anywhere in the
    batch's: each is what the request gives alone."""
    from adeco_gb300.synthetic import zeldovich_lattice
    pos = zeldovich_lattice(40, L=40.0, seed=3, rms_disp=2.0)
    reqs = [((14.0 + k, 20.0, 17.0), 3.0 + k, d) for k, d in enumerate((1, 2, 7, 33, 5, 66, 3))]
    with adeco.Session(pos) as s:
        b = s.submit(reqs)
        s.wait(b)
        together = [s.result(b, k, r[2]) for k, r in enumerate(reqs)]
        s.release(b)
        for r, got in zip(reqs, together):
            b = s.submit([r])
            s.wait(b)
            assert np.array_equal(s.result(b, 0, r[2]), got)
            assert got.sum() > 0
            s.release(b)


@pytest.mark.parametrize("n,max_tets,leaf_dims", [(15, 6 * 14 ** 3, 8), (16, 500, 4), (50, 3000, 8)])
def test_leaf_work_from_either_builder(adeco, n, max_tets, leaf_dims):
    """The leaves' sums are the same whether the octree, and with it the list of
    work items, was built on the device or by the host: one leaf holding
    everything, lattices that are and are not whole meta-cells."""
    from adeco_gb300.synthetic import zeldovich_lattice
    pos = zeldovich_lattice(n, L=30.0, seed=8, rms_disp=1.5)
    grids = []
    for builder in ("device", "host"):
        with adeco.Session(pos) as s:
            s.build_octree(max_tets, 8, leaf_dims=leaf_dims, builder=builder)
            grids.append(s.deposit_leaves()[0])
    assert np.array_equal(grids[0], grids[1])
    assert grids[0].sum() > 0
