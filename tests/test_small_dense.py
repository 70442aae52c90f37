"""Dense steps of small matrices: the one-launch cluster forms (small_dense.cu, up
to 56 functions) and the tiled product above, at the edges of their 8 x 8 tiles and
cluster sizes."""
import numpy as np
import pytest
from scipy.linalg import eigh

import oracle as O
from gbhf import _lib, basis as B, molecules as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 16, 17, 31, 32, 33, 39, 40, 41, 64, 65, 71, 130])
def test_error_matrix(ctx, n):
    """e = X^T (F D S - S D F) X: four products of n terms, each rounded at 2^-53 of
    its magnitudes: 8 n 2^-53 of the product of the norms."""
    rng = np.random.default_rng(n)
    f, s, d = (a + a.T for a in rng.standard_normal((3, n, n)))
    x = rng.standard_normal((n, n))     # no symmetry
    got = ctx.diis_error(*(O.square_to_tri(a) for a in (f, s, d)), x)
    m = f @ d @ s
    scale = np.linalg.norm(x) ** 2 * np.linalg.norm(f) * np.linalg.norm(d) * np.linalg.norm(s)
    np.testing.assert_allclose(got, x.T @ (m - m.T) @ x, rtol=0, atol=8 * n * 2.0 ** -53 * scale)


@pytest.mark.parametrize("name,waters,basis", [
    ("He", 0, "6-31g"), ("H2", 0, "sto-3g"), ("w1", 1, "sto-3g"), ("w1", 1, "6-31g"), ("w1", 1, "6-31g*"),
    ("w2", 2, "6-31g"), ("w4", 4, "6-31g"), ("w8", 8, "sto-3g"), ("w3", 3, "6-31g*"), ("w5", 5, "6-31g"),
    ("w11", 11, "sto-3g"), ("w16", 16, "sto-3g")])
def test_density_of_converged_scf(ctx, name, waters, basis):
    """2 to 112 functions: S^(-1/2) and the purified density of the last Fock matrix
    against a diagonalisation; the SCF stops at an rms density change of 1e-8 or less."""
    if waters:
        atoms = B.make_atoms(M.water_labels(waters), M.water_cluster(waters, np.random.default_rng(waters)), basis)
    elif name == "H2":
        atoms = B.make_atoms(["H", "H"], np.array([[0, 0, 0], [0, 0, 1.4]]), basis)
    else:
        atoms = B.make_atoms(["He"], np.zeros((1, 3)), basis)
    fb = B.flatten(atoms)
    ctx.set_basis(fb)
    r = ctx.scf(_lib.baseline_opts())
    assert r["converged"]
    s = O.tri_to_square(ctx.overlap(_lib.MODE_EXACT))
    f, d = O.tri_to_square(r["fock"]), O.tri_to_square(r["density"])
    nocc = int(round(fb.charge.sum())) // 2
    c = eigh(f, s)[1][:, :nocc]
    np.testing.assert_allclose(d, 2 * c @ c.T, rtol=0, atol=1e-6)
    np.testing.assert_allclose(d @ s @ d, 2 * d, rtol=0, atol=1e-10)     # idempotent whatever the SCF's state
    assert abs(np.trace(d @ s) - 2 * nocc) < 1e-10
