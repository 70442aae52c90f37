"""Gradient task lists and kernels: two-float classes with the block's warps in step,
finer tasks of short lists, against the plain FP64 kernels."""
import numpy as np
import pytest

import oracle as O
from gbhf import _lib, basis as B, molecules as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters,basis", [(1, "6-31g"), (2, "6-31g"), (4, "sto-3g"), (2, "6-31g*"), (7, "6-31g"),
                                          (12, "6-31g")])
def test_gradient_against_fp64_lists(ctx, waters, basis):
    """A function of exponent 1e-9 without density keeps every quartet in FP64; without
    it most are two-float.  The gradient adds some 1e3 of magnitudes with 2^-43 of
    each at worst: 1e-10 absolute."""
    xyz = M.water_cluster(waters, np.random.default_rng(waters))
    atoms = B.make_atoms(M.water_labels(waters), xyz, basis)
    fb = B.flatten(atoms)
    rng = np.random.default_rng(5)
    pos = fb.xyz[fb.cgf_atom]
    r = np.linalg.norm(pos[:, None] - pos[None], axis=2)
    m = rng.standard_normal((2, fb.n_cgf, fb.n_cgf)) * 0.15
    d, w = (x + x.T for x in m * np.exp(-r / 1.6))
    d += np.diag(rng.uniform(0.3, 2.0, fb.n_cgf))
    ctx.set_basis(fb)
    got = ctx.gradient(O.square_to_tri(d), O.square_to_tri(w), schwarz=0.0)
    at = int(np.searchsorted(fb.cgf_atom, 1, side="right"))     # the functions of atoms 0 and 1 come first
    atoms[1].basis = atoms[1].basis + [B.CGF(((1e-7, 1e-9),), "S")]
    ctx.set_basis(B.flatten(atoms))
    d, w = (np.insert(np.insert(x, at, 0, axis=0), at, 0, axis=1) for x in (d, w))
    ref = ctx.gradient(O.square_to_tri(d), O.square_to_tri(w), schwarz=0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-10)
