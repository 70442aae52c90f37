"""Reference-mode integrals with a warp per function pair or quartet: terms in
parallel, added in the reference's order.  Contractions of 1, 3 and 6 primitives
(1 to 1296 terms, below and above a warp), with d functions, against the oracle."""
import numpy as np
import pytest

import oracle as O
from gbhf import _lib, basis as B, molecules as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("labels,coords,basis", [
    (["H"], [[0, 0, 0]], "6-31g"),                                  # 2 functions, 3 and 1 primitives
    (["O"], [[0.1, 0.2, 0.3]], "6-31g*"),                           # one centre, s p d
    (["O", "H", "H"], [[0, 0, 0], [1.4, 0, 1.1], [-1.4, 0, 1.1]], "6-31g*")])
def test_reference_terms_against_oracle(ctx, labels, coords, basis):
    """Values up to ~35 from up to 1296 terms of 2^-53 each: 1e-12 absolute."""
    fb = B.flatten(B.make_atoms(labels, np.asarray(coords, float), basis))
    ob = O.OracleBasis(fb)
    ctx.set_basis(fb)
    ctx.set_boys_grid(O.boys_ref_grid())
    np.testing.assert_allclose(ctx.overlap(_lib.MODE_REFERENCE), ob.overlap(True), rtol=0, atol=1e-12)
    np.testing.assert_allclose(ctx.hcore(_lib.MODE_REFERENCE), ob.hcore(True), rtol=0, atol=1e-12)
    np.testing.assert_allclose(ctx.eri_canonical(_lib.MODE_REFERENCE), ob.eri_canonical(True), rtol=0, atol=1e-12)


def test_canonical_tables_follow_the_basis(ctx):
    """The pair tables stay with the context: smaller, larger and again smaller bases."""
    ctx.set_boys_grid(O.boys_ref_grid())
    for basis in ("sto-3g", "6-31g", "sto-3g"):
        fb = B.flatten(M.water_atoms(basis, "text"))
        ctx.set_basis(fb)
        np.testing.assert_allclose(ctx.eri_canonical(_lib.MODE_REFERENCE), O.OracleBasis(fb).eri_canonical(True),
                                   rtol=0, atol=1e-12)
