"""Batched purification (a launch per step, 8 x 8 tiles, molecules in order of size):
densities of batches whose members differ in size and converge at different steps
against the single-molecule path."""
import numpy as np
import pytest

from gbhf import _lib, basis as B, molecules as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(1, "sto-3g")], [(1, "sto-3g"), (1, "6-31g")],
                                   [(2, "6-31g"), (1, "sto-3g"), (3, "6-31g"), (5, "sto-3g"), (1, "6-31g*")]])
def test_batch_energies_match_single(ctx, sizes):
    """Same thresholds, same FP64 builds: energies to 1e-8 hartree (the SCF's own
    convergence), gradients to 1e-5 (density converged to 1e-8 or better)."""
    flats = []
    for k, (w, basis) in enumerate(sizes):
        flats.append(B.flatten(B.make_atoms(M.water_labels(w), M.water_cluster(w, np.random.default_rng(k)), basis)))
    opts = _lib.baseline_opts()
    energies, _, converged, grads = ctx.scf_batch(flats, opts, gradients=True)
    assert converged.all()
    for k, fb in enumerate(flats):
        ctx.set_basis(fb)
        ref = ctx.scf(opts)
        assert abs(energies[k] - ref["energy"]) < 1e-8
        np.testing.assert_allclose(grads[k], ctx.gradient(), rtol=0, atol=1e-5)
