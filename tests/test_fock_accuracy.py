"""How far an FP64 Fock matrix is from its exact value."""
import numpy as np
import pytest

import oracle as O
from gbhf import _lib, basis as B, molecules as M
from test_two_float import _density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters,basis,plain", [(4, "sto-3g", 2.3e-15), (8, "6-31g", 7.8e-15)])
def test_two_float_lists_cost_no_digits(ctx, waters, basis, plain):
    """Against an extended-precision build the library's FP64 build without two-float
    lists has an rms error of `plain`, the oracle's 1.6e-15 and 4.5e-15 (eight threads;
    more of them, less).  With the lists the difference from the oracle stays below
    what these two make together."""
    xyz = M.water_cluster(waters, np.random.default_rng(waters))
    fb = B.flatten(B.make_atoms(M.water_labels(waters), xyz, basis))
    ob = O.OracleBasis(fb)
    ctx.set_basis(fb)
    err = []
    for seed in (1, 2, 3):
        d = _density(fb, seed)
        h = np.zeros_like(d)
        ref, _ = ob.fock_direct(h, d, 0.0, False)
        err += [ctx.fock(h, d, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0) - ref for _ in range(4)]
    oracle = 1.6e-15 if waters == 4 else 4.5e-15
    assert np.sqrt(np.mean(np.square(err))) < np.hypot(plain, oracle)
