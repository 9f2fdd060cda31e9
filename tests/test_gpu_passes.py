"""The y/z passes as three kernels (matvec_pass.cuh), the plane kernel of small
planes and the planned x passes against the oracle, at FP64 1e-12 and FP32 2e-6 relative in the 2-norm as for
the other matvec paths: two- and three-stage plans on every axis, odd and even
first radices, last radices 2 to 8, boxes of half the grid and of less, one
right-hand side (W = 1), a pair, and a pair with an idle lane."""
import numpy as np
import pytest

from tests.pairs import Pair, rel

pytestmark = pytest.mark.gpu

BOXES = {
    (4, 4, 4): (8, 8, 8),
    (5, 7, 9): (10, 14, 18),
    (9, 15, 27): (18, 30, 54),
    (11, 13, 11): (24, 28, 24),        # less than half of every edge
    (35, 49, 21): (70, 98, 42),
    (33, 45, 81): (70, 90, 162),       # odd first radices
    (140, 6, 5): (280, 12, 10),        # three stages along x
    (6, 125, 8): (12, 250, 16),        # ... y
    (5, 6, 150): (10, 12, 300),        # ... z
    (20, 21, 21): (40, 42, 42),        # the largest small plane
    (5, 21, 22): (10, 42, 48),     # ... and one beyond it
    (8, 110, 128): (16, 224, 256),
    (4, 63, 126): (8, 126, 252),
}


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 2e-6)])
@pytest.mark.parametrize("box", list(BOXES))
def test_passes_match_oracle(box, prec, tol):
    rng = np.random.default_rng(box[0])
    z, y, x = np.meshgrid(*[np.arange(n) for n in box[::-1]], indexing="ij")
    keep = rng.random(x.shape) < 0.7
    keep[0, 0, 0] = keep[-1, -1, -1] = True  # the box's corners
    pos = np.stack([x[keep], y[keep], z[keep]], axis=1).astype(np.uint32)
    mat = (rng.random(len(pos)) < 0.4).astype(np.uint8)
    pr = Pair("arrays", (pos, mat, "0.1um"), [1.5 + 0.1j, 1.3 + 0.02j], "1.1um", prec, max_rhs=3)
    assert pr.p.grid == BOXES[box] and pr.mv.passes == (max(pr.p.grid[1:]) > 42)
    assert pr.mv.layout["yz_path"] == ("passes" if pr.mv.passes else "fused")
    xs = [pr.rand_vec(40 + r) for r in range(3)]
    want = []
    for r, pol in enumerate((1, 2, 1)):
        pr.set_cc((0.36, 0.48, 0.8) if r else (0, 0, 1), pol, "ldr", rhs=r)
        want.append(pr.op.matvec(xs[r]))
    n = pr.p.vec_size
    three = pr.mv.apply(np.concatenate(xs)).reshape(3, n)
    for r in range(3):
        assert rel(three[r], want[r]) < tol, r
    # alone and as a pair: the same bits
    assert np.array_equal(pr.mv.apply(xs[0]), three[0])
    assert np.array_equal(pr.mv.apply(np.concatenate(xs[:2])).reshape(2, n), three[:2])
    pr.mv.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("box,nrhs", [((4, 25, 24), 6),    # room for two entries of one frequency
                                      ((4, 25, 24), 1),    # ... for several frequencies of one
                                      ((30, 40, 35), 5)])  # ... for some frequencies of all
def test_small_work_buffer_gives_identical_results(box, nrhs, prec):
    # chunks of frequencies and of right-hand sides change no bit
    import dda_b200
    from dda_b200 import api
    z, y, x = np.meshgrid(*[np.arange(n) for n in box[::-1]], indexing="ij")
    pos = np.stack([v.ravel() for v in (x, y, z)], axis=1).astype(np.uint32)
    g = dda_b200.Geometry.from_arrays(pos, np.zeros(len(pos), np.uint8), "0.1um")
    p = dda_b200.DDAParams(g, [1.4 + 0.05j], "2um")
    rng = np.random.default_rng(nrhs)
    v = rng.uniform(-1, 1, (nrhs, 3, p.nvs)) + 1j * rng.uniform(-1, 1, (nrhs, 3, p.nvs))
    v[:, :, p.nv:] = 0
    out, launches, held = [], [], []
    for flags in (0, api.FLAG_SMALL_WORK):
        mv = dda_b200.CudaMatVec(p, prec, max_rhs=nrhs, flags=flags)
        assert mv.passes
        for r in range(nrhs):
            mv.set_couple_constants(dda_b200.CoupleConstants(p, (0, 0.6, 0.8), 1 + r % 2, "ldr"), rhs=r)
        n = mv.launches
        out.append(mv.apply(v.ravel()))
        launches.append(mv.launches - n)
        held.append(mv.layout["device_bytes"])
        mv.close()
    assert np.array_equal(out[0], out[1])
    assert launches[1] > launches[0] and held[1] < held[0]


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("box", [(28, 28, 28), (9, 28, 28), (64, 28, 28), (32, 32, 32), (75, 32, 32)])
def test_one_wave_of_planes(box, prec):
    # 56 x 56 planes (FP32: 64 x 64 too) run the plane kernel for the batches
    # of which they are one wave, the passes for others: the same bits
    import dda_b200
    from dda_b200 import api
    z, y, x = np.meshgrid(*[np.arange(n) for n in box[::-1]], indexing="ij")
    pos = np.stack([v.ravel() for v in (x, y, z)], axis=1).astype(np.uint32)
    g = dda_b200.Geometry.from_arrays(pos, np.zeros(len(pos), np.uint8), "0.1um")
    p = dda_b200.DDAParams(g, [1.4 + 0.05j], "2um")
    gx, small = p.grid[0], p.grid[1] == 56 or prec != "fp64"
    assert p.grid[1:] == (2 * box[1], 2 * box[2])
    wave = [small and 56 <= gx * n <= 148 for n in range(1, 5)]
    rng = np.random.default_rng(2)
    v = rng.uniform(-1, 1, (4, 3, p.nvs)) + 1j * rng.uniform(-1, 1, (4, 3, p.nvs))
    v[:, :, p.nv:] = 0
    v = v.reshape(4, -1)

    def products(max_rhs, flags=0):
        mv = dda_b200.CudaMatVec(p, prec, max_rhs=max_rhs, flags=flags)
        assert flags or mv.passes == (not wave[max_rhs - 1])
        for r in range(max_rhs):
            mv.set_couple_constants(dda_b200.CoupleConstants(p, (0, 0.6, 0.8), 1 + r % 2, "ldr"), rhs=r)
        out = []
        for n in range(1, max_rhs + 1):
            k = mv.launches
            out.append(mv.apply(v[:n].ravel()))
            # (an apply in mixed precision is FP64)
            if not flags and prec != "mixed":
                assert mv.launches - k == (3 if wave[n - 1] else 5) + (4 if prec == "fp32" else 0), n
        mv.close()
        return out

    want = products(4, api.FLAG_YZ_GROUPS2 if p.grid[0] in (56, 64, 128) else 0)  # (tuned lengths)
    for max_rhs in (1, 2, 4):
        for a, b in zip(products(max_rhs), want):
            assert np.array_equal(a, b)
