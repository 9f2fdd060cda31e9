"""The far field of many directions (k_ff_part) against the sum over the dipoles
in NumPy, on both sides of the rule's thresholds and at the edges of its 32- and
64-direction blocks, with one to three right-hand sides (pairs and a remainder),
permuted dipoles and requests beyond the context's workspace."""
import numpy as np
import pytest

import dda_b200
from tests.pairs import scrambled_arrays

pytestmark = pytest.mark.gpu


def _sum(p, pol, dirs):
    g = p.geometry
    r = g.positions.astype(np.float64) - (np.array(p.box) - 1) / 2
    k = p.wave_num
    ph = np.exp(-1j * p.kd * (dirs @ r.T))
    out = np.empty((len(dirs), len(pol), 3), dtype=np.complex128)
    for b in range(len(pol)):
        P = pol[b].reshape(3, p.nvs)[:, :p.nv]
        S = ph @ P.T
        out[:, b] = 1j * k * k * (S - dirs * np.einsum("ij,ij->i", dirs, S)[:, None])
    return out


@pytest.mark.parametrize("ndir", [1, 31, 32, 33, 63, 64, 65, 200, 1023, 1024, 1057])
@pytest.mark.parametrize("target", ["scrambled", "sphere"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_far_field_of_many_directions(prec, target, ndir):
    if target == "scrambled":  # 30 lines, workspace of a few KB
        g = dda_b200.Geometry.from_arrays(*scrambled_arrays())
        mats = [1.5 + 0.1j, 1.3 + 0.0j]
    else:  # 400 lines
        g = dda_b200.Geometry.sphere("1um", "0.1um")
        mats = [1.5 + 0.1j]
    p = dda_b200.DDAParams(g, mats, "0.9um")
    mv = dda_b200.CudaMatVec(p, prec, max_rhs=3)
    rng = np.random.default_rng(ndir)
    dirs = rng.normal(size=(ndir, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    pol = rng.uniform(-1, 1, (3, p.vec_size)) + 1j * rng.uniform(-1, 1, (3, p.vec_size))
    if prec == "fp32":
        pol = pol.astype(np.complex64).astype(np.complex128)  # the context's precision: exact
    want = _sum(p, pol, dirs)
    for n in (1, 2, 3):
        got = mv.far_field(dirs, nrhs=n, pol=pol[:n])
        # sums of 120 to 4 200 terms of phases up to 20 rad in FP64, in another order
        assert np.abs(got - want[:, :n]).max() < 1e-12 * np.abs(want).max()
    mv.close()


def test_splits_of_a_small_target_take_one_launch():
    # 400 lines, 2 978 directions: 25 splits of the lines want 25 sets of
    # partial sums, beyond the Krylov vectors' room; all directions still go in
    # one launch (and one that adds the sums)
    g = dda_b200.Geometry.sphere("1um", "0.1um")
    p = dda_b200.DDAParams(g, [1.5 + 0.1j], "0.9um")
    rng = np.random.default_rng(1)
    dirs = rng.normal(size=(2978, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    for nrhs in (1, 2):
        mv = dda_b200.CudaMatVec(p, "fp64", max_rhs=nrhs)
        pol = rng.uniform(-1, 1, (nrhs, p.vec_size)) + 1j * rng.uniform(-1, 1, (nrhs, p.vec_size))
        want = _sum(p, pol, dirs)
        n = mv.launches
        got = mv.far_field(dirs, nrhs=nrhs, pol=pol)
        assert mv.launches - n == 2
        assert np.abs(got - want).max() < 1e-12 * np.abs(want).max()
        mv.close()


def test_directions_beyond_the_room_go_in_blocks():
    # one set of partial sums is 67 MB, above the 64 MB of a request that
    # allocates: two blocks of directions
    g = dda_b200.Geometry.from_arrays(*scrambled_arrays())
    p = dda_b200.DDAParams(g, [1.5 + 0.1j, 1.3 + 0.0j], "0.9um")
    mv = dda_b200.CudaMatVec(p, "fp64", max_rhs=2)
    rng = np.random.default_rng(2)
    dirs = rng.normal(size=(700000, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    pol = rng.uniform(-1, 1, (2, p.vec_size)) + 1j * rng.uniform(-1, 1, (2, p.vec_size))
    n = mv.launches
    got = mv.far_field(dirs, nrhs=2, pol=pol)
    assert mv.launches - n == 4
    for at in (slice(0, 100), slice(699000, 699100), slice(-100, None)):  # the second block begins at 699 050
        want = _sum(p, pol, dirs[at])
        assert np.abs(got[at] - want).max() < 1e-12 * np.abs(want).max()
    mv.close()


def test_kernel_of_a_request():
    # k_farfield is one launch, k_ff_part two: the rule's lines for a small
    # target, a long one and one of more than 256 lines
    torch = pytest.importorskip("torch")
    wave = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    long_box = np.stack([v.ravel() for v in np.meshgrid(np.arange(100), np.arange(8), np.arange(8), indexing="ij")],
                        axis=1).astype(np.uint32)
    long_box = long_box[np.lexsort((long_box[:, 0], long_box[:, 1], long_box[:, 2]))]
    small = dda_b200.Geometry.from_arrays(*scrambled_arrays())
    cases = [(small, 2, wave // 2), (small, 1, wave),
             (dda_b200.Geometry.from_arrays(long_box, np.zeros(len(long_box), np.uint8), "0.1um"), 1, 63),
             (dda_b200.Geometry.sphere("1um", "0.1um"), 2, 31)]
    rng = np.random.default_rng(3)
    for g, nrhs, last_few in cases:
        p = dda_b200.DDAParams(g, [1.5 + 0.1j, 1.3 + 0.0j] if g is small else [1.5 + 0.1j], "0.9um")
        mv = dda_b200.CudaMatVec(p, "fp64", max_rhs=nrhs)
        pol = rng.uniform(-1, 1, (nrhs, p.vec_size)) + 1j * rng.uniform(-1, 1, (nrhs, p.vec_size))
        for ndir, launches in ((last_few, 1), (last_few + 1, 2)):
            dirs = rng.normal(size=(ndir, 3))
            dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
            n = mv.launches
            got = mv.far_field(dirs, nrhs=nrhs, pol=pol)
            assert mv.launches - n == launches, (nrhs, ndir)
            want = _sum(p, pol, dirs)
            assert np.abs(got - want).max() < 1e-12 * np.abs(want).max()
        mv.close()
