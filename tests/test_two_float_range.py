"""Which primitive pairs may enter the two-float lists (ff_pair_range in
csrc/gbhf_ff.cuh): products of steep shells leave the FP32 range, and an FP64 build
then keeps them in FP64."""
import math
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from gbhf import _lib, basis as B, molecules as M
from test_two_float import CSRC, _density


def test_range_rule_against_long_double(tmp_path):
    """Every class at the rule's edge: finite, ERIs within 2^-38 of the largest
    component plus 2^-45; the steep p shells that overflow are refused."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "ff_range_check"
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC),
                    str(Path(__file__).resolve().parent / "host" / "ff_range_check.cpp"), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    rows = [line.split() for line in subprocess.run([str(exe)], check=True, capture_output=True,
                                                    text=True).stdout.splitlines()]
    classes = [r for r in rows if r[0] != "steep"]
    assert len(classes) == 27
    for name, bad, n, worst in classes:
        assert int(bad) == 0, name
        assert name.startswith("grad_") or (int(n) > 1000 and float(worst) < 1.0), name
    steep = [tuple(int(x) for x in r[1:]) for r in rows if r[0] == "steep"]
    assert any(not finite for _, finite, _ in steep)       # the case exists,
    assert all(finite or not taken for _, finite, taken in steep)   # and is refused


def _steep(momentum, exponent):
    """A contracted p or d shell with a small share of a steep primitive."""
    labels = {1: ("Px", "Py", "Pz"), 2: ("Dxx", "Dxy", "Dxz", "Dyy", "Dyz", "Dzz")}[momentum]
    norm = [(2 * e / math.pi) ** 0.75 * (4 * e) ** (momentum / 2) for e in (exponent, 0.9)]
    return [B.CGF(((0.01 * norm[0], exponent), (norm[1], 0.9)), t) for t in labels]


@pytest.mark.gpu
@pytest.mark.parametrize("momentum,exponent", [(1, 1e5), (1, 1e7), (2, 1e4), (2, 1e6)])
def test_steep_shells_stay_in_fp64(ctx, momentum, exponent):
    """FP64 Fock matrix against the oracle (1e-13 of its largest element, as without
    the steep primitive), and the gradient against the basis that an exponent of 1e-9
    keeps in FP64 (1e-10, as in the gradient list tests)."""
    xyz = M.water_cluster(3, np.random.default_rng(3))
    atoms = B.make_atoms(M.water_labels(3), xyz, "6-31g")
    atoms[0].basis = atoms[0].basis + _steep(momentum, exponent)
    fb = B.flatten(atoms)
    ob = O.OracleBasis(fb)
    ctx.set_basis(fb)
    d = O.tri_to_square(_density(fb, 4))
    h = np.zeros(fb.n_cgf * (fb.n_cgf + 1) // 2)
    ref = O.fock_canonical(h, O.square_to_tri(d), ob.eri_canonical(False))
    got = ctx.fock(h, O.square_to_tri(d), _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-13 * np.abs(ref).max())
    w = 0.1 * d
    grad = ctx.gradient(O.square_to_tri(d), O.square_to_tri(w), schwarz=0.0)
    at = int(np.searchsorted(fb.cgf_atom, 1, side="right"))
    atoms[1].basis = atoms[1].basis + [B.CGF(((1e-7, 1e-9),), "S")]
    ctx.set_basis(B.flatten(atoms))
    d, w = (np.insert(np.insert(x, at, 0, axis=0), at, 0, axis=1) for x in (d, w))
    ref = ctx.gradient(O.square_to_tri(d), O.square_to_tri(w), schwarz=0.0)
    np.testing.assert_allclose(grad, ref, rtol=0, atol=1e-10 * max(1.0, np.abs(ref).max()))


@pytest.mark.gpu
def test_small_coefficients_keep_their_digits(ctx):
    """All coefficients times 1e-9: integrals near 1e-36, where FP32 products lose
    their low parts.  The FP64 Fock matrix is that of the unscaled basis times 1e-36."""
    xyz = M.water_cluster(3, np.random.default_rng(3))
    out = []
    for scale in (1.0, 1e-9):
        atoms = B.make_atoms(M.water_labels(3), xyz, "6-31g")
        for a in atoms:
            a.basis = [B.CGF(tuple((c * scale, e) for c, e in f.primitives), f.funtype) for f in a.basis]
        fb = B.flatten(atoms)
        ctx.set_basis(fb)
        d = _density(fb, 4)
        out.append(ctx.fock(np.zeros_like(d), d, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0) / scale ** 4)
    np.testing.assert_allclose(out[1], out[0], rtol=0, atol=1e-13 * np.abs(out[0]).max())
