"""The far field of many directions (k_ff_part) against the oracle's sum and
against the few-direction kernel, on both sides of the rule's thresholds and at
the edges of its 32- and 64-direction blocks, with one to three right-hand
sides (pairs and a remainder), permuted dipoles and a request beyond the
context's workspace."""
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
