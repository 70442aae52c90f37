"""The kernels whose warps go through a primitive quartet in step (two-float (ps|pp),
(pp|pp) and (p.|p.) gradients): blocks with fewer tasks than warps, batches of
different lengths, warps that run out of work early."""
import numpy as np
import pytest

import oracle as O
from gbhf import _lib, basis as B, molecules as M
from test_two_float import _density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters,basis", [(3, "sto-3g"), (2, "6-31g"), (5, "6-31g"), (9, "sto-3g")])
def test_repeated_builds_agree(ctx, waters, basis):
    """Twenty builds and gradients of one density: who takes which task changes, and the
    order of the FP64 atomics with it (1e-13 of elements up to ~30), nothing else.  The
    first Fock matrix against the oracle's (1e-13 of its largest element)."""
    xyz = M.water_cluster(waters, np.random.default_rng(waters))
    fb = B.flatten(B.make_atoms(M.water_labels(waters), xyz, basis))
    ctx.set_basis(fb)
    d, w = _density(fb, waters), 0.1 * _density(fb, waters + 1)
    h = np.zeros_like(d)
    ref, _ = O.OracleBasis(fb).fock_direct(h, d, 0.0, False)
    f = [ctx.fock(h, d, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0) for _ in range(20)]
    g = [ctx.gradient(d, w, schwarz=0.0) for _ in range(20)]
    tol = 1e-13 * max(1.0, np.abs(ref).max())
    np.testing.assert_allclose(f[0], ref, rtol=0, atol=tol)
    for x in f[1:]:
        np.testing.assert_allclose(x, f[0], rtol=0, atol=tol)
    for x in g[1:]:
        np.testing.assert_allclose(x, g[0], rtol=0, atol=1e-11)   # some 1e3 of magnitudes cancel
