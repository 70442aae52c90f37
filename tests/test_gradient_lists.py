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


@pytest.mark.parametrize("waters,basis", [(1, "6-31g*"), (5, "sto-3g"), (6, "sto-3g"), (11, "sto-3g")])
def test_one_electron_terms_against_differences(ctx, waters, basis):
    """3, 15, 18 and 33 nuclei (on 4, 16 and 32 lanes, and in two rounds).  The
    one-electron terms are odd in (D, W), the rest is even; tr D H - tr W S by fourth-order
    central differences: rounding 1e3 * 2^-53 / 1e-3, truncation 1e-12 / 30 times a fifth
    derivative of up to 1e5: 1e-7 absolute."""
    xyz = M.water_cluster(waters, np.random.default_rng(waters))
    labels = M.water_labels(waters)
    fb = B.flatten(B.make_atoms(labels, xyz, basis))
    rng = np.random.default_rng(7)
    d, w = (O.square_to_tri(m + m.T) for m in rng.standard_normal((2, fb.n_cgf, fb.n_cgf)) * 0.1)
    off = np.full(fb.n_cgf * (fb.n_cgf + 1) // 2, 2.0)
    off[np.cumsum(np.concatenate([[0], np.arange(fb.n_cgf, 1, -1)]))] = 1.0    # diagonal of the flat triangle
    ctx.set_basis(fb)
    got = 0.5 * (ctx.gradient(d, w) - ctx.gradient(-d, -w))

    def value(coords):
        ctx.set_basis(B.flatten(B.make_atoms(labels, coords, basis)))
        return off @ (d * ctx.hcore(_lib.MODE_EXACT) - w * ctx.overlap(_lib.MODE_EXACT))

    step = 1e-3
    for atom, x in ((0, 0), (1, 2), (3 * waters - 1, 1)):
        f = []
        for k in (-2, -1, 1, 2):
            c = np.array(xyz, float)
            c[atom, x] += k * step
            f.append(value(c))
        assert abs((f[0] - 8 * f[1] + 8 * f[2] - f[3]) / (12 * step) - got[atom, x]) < 1e-7


@pytest.mark.parametrize("open_shell", [False, True])
def test_gradient_of_densities_outside_the_fp32_range(ctx, open_shell):
    """The two-electron gradient is quadratic in the density, also where block maxima
    leave the FP32 range beside blocks that are zero (1e-12 of its largest component:
    the order of the FP64 atomics differs)."""
    xyz = M.water_cluster(3, np.random.default_rng(3))
    fb = B.flatten(B.make_atoms(M.water_labels(3), xyz, "6-31g"))
    ctx.set_basis(fb)
    rng = np.random.default_rng(2)
    d = rng.standard_normal((fb.n_cgf, fb.n_cgf))
    at = fb.cgf_atom
    some = rng.random((fb.n_atoms, fb.n_atoms)) < 0.5   # about a third of the atom blocks is zero
    d = (d + d.T) * (some | some.T | np.eye(fb.n_atoms, dtype=bool))[at[:, None], at[None]]
    zero = np.zeros(fb.n_cgf * (fb.n_cgf + 1) // 2)

    def two_electron(scale):
        def grad(sign):
            t = O.square_to_tri(d * (sign * scale))
            return ctx.gradient_uhf(t, -0.5 * t, zero, schwarz=0.0) if open_shell else ctx.gradient(t, zero, schwarz=0.0)
        return 0.5 * (grad(1.0) + grad(-1.0)) / scale ** 2

    nuc = ctx.gradient(zero, zero)
    one, far = two_electron(1.0) - nuc, two_electron(2.0 ** 200)
    np.testing.assert_allclose(far, one, rtol=0, atol=1e-12 * np.abs(one).max())


@pytest.mark.parametrize("waters,basis,before", [(2, "6-31g", 1.1e-13), (4, "sto-3g", 6.9e-13), (2, "6-31g*", 1.1e-13)])
def test_translational_invariance_to_rounding(ctx, waters, basis, before):
    """The gradient adds up to zero over the atoms.  The quartets on one atom add
    nothing but the rounding of their terms; with them the sum was `before` (rms over
    densities and directions), without them it stays below two thirds of it."""
    xyz = M.water_cluster(waters, np.random.default_rng(waters))
    fb = B.flatten(B.make_atoms(M.water_labels(waters), xyz, basis))
    ctx.set_basis(fb)
    pos = fb.xyz[fb.cgf_atom]
    r = np.linalg.norm(pos[:, None] - pos[None], axis=2)

    def density(seed):
        rng = np.random.default_rng(seed)
        d = rng.standard_normal((fb.n_cgf, fb.n_cgf)) * 0.15
        return O.square_to_tri((d + d.T) * np.exp(-r / 1.6) + np.diag(rng.uniform(0.3, 2.0, fb.n_cgf)))

    sums = [ctx.gradient(density(s), 0.2 * density(s + 10), schwarz=0.0).sum(axis=0) for s in (1, 2, 3) for _ in range(4)]
    assert np.sqrt(np.mean(np.square(sums))) < 2.0 / 3.0 * before
