"""Two-float gradients: the generated code on the host by kind of quartet, and the
open-shell kernels (spin density without a Coulomb term) on the GPU."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from gbhf import _lib, basis as B, molecules as M
from test_two_float import CSRC, _density


def test_gradient_code_by_kind_of_quartet(tmp_path):
    """2^-42 rms and 2^-36 at worst of the largest component: the bounds of the ERI
    classes, 2^-43 and 2^-40, with one order more and the difference of two terms."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "ff_grad_check"
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC),
                    str(Path(__file__).resolve().parent / "host" / "ff_grad_check.cpp"), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    rows = [line.split() for line in subprocess.run([str(exe)], check=True, capture_output=True,
                                                    text=True).stdout.splitlines()]
    assert {r[0] for r in rows} == {"ssss", "ssps", "sspp", "psss", "psps", "pspp", "ppss", "ppps", "pppp", "ssds",
                                    "ssdp", "psds", "dsss", "dsps"}
    assert all((c, str(k)) in {(r[0], r[1]) for r in rows} for c in ("ssss", "pppp", "dsps") for k in range(3))
    for cls, kind, worst, rms in rows:
        assert float(worst) < 2.0 ** -36 and float(rms) < 2.0 ** -42, (cls, kind, worst, rms)


@pytest.mark.gpu
@pytest.mark.parametrize("waters,basis", [(2, "6-31g"), (4, "sto-3g"), (2, "6-31g*"), (7, "6-31g")])
def test_open_shell_gradient_against_fp64_lists(ctx, waters, basis):
    """As the closed-shell test of the gradient lists: a function of exponent 1e-9
    without density keeps every quartet in FP64 (1e-10)."""
    xyz = M.water_cluster(waters, np.random.default_rng(waters))
    atoms = B.make_atoms(M.water_labels(waters), xyz, basis)
    fb = B.flatten(atoms)
    da, db, w = (O.tri_to_square(_density(fb, s)) * f for s, f in ((1, 0.5), (2, 0.4), (3, 0.1)))
    ctx.set_basis(fb)
    got = ctx.gradient_uhf(*(O.square_to_tri(x) for x in (da, db, w)), schwarz=0.0)
    at = int(np.searchsorted(fb.cgf_atom, 1, side="right"))
    atoms[1].basis = atoms[1].basis + [B.CGF(((1e-7, 1e-9),), "S")]
    ctx.set_basis(B.flatten(atoms))
    wide = [O.square_to_tri(np.insert(np.insert(x, at, 0, axis=0), at, 0, axis=1)) for x in (da, db, w)]
    ref = ctx.gradient_uhf(*wide, schwarz=0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-10)


@pytest.mark.gpu
def test_open_shell_energy_with_two_float_lists(ctx):
    """The FP64 energy of a water dimer cation in 6-31G*: the Coulomb and exchange build
    of the total density and the exchange build of the spin density run in two floats.
    The oracle's Fock matrices of the densities found give the same energy (1e-9: the
    last density step, 1e-9 rms, enters squared)."""
    fb = B.flatten(M.cluster_atoms("batch256", "6-31g*", index=7))
    ctx.set_basis(fb)
    r = ctx.scf_uhf(2, _lib.baseline_opts(charge=1.0, conv_energy=1e-11, conv_density=1e-9, max_iter=200))
    ob = O.OracleBasis(fb)
    h = O.tri_to_square(ob.hcore(False))
    da, db = O.tri_to_square(r["density_alpha"]), O.tri_to_square(r["density_beta"])
    eri = O.eri_tensor(ob, fb.n_cgf)
    j = np.einsum("abcd,cd->ab", eri, da + db)
    fa = h + j - np.einsum("acbd,cd->ab", eri, da)
    fbm = h + j - np.einsum("acbd,cd->ab", eri, db)
    e = 0.5 * (np.sum((da + db) * h) + np.sum(da * fa) + np.sum(db * fbm)) + O.nuclear_rep(fb.xyz, fb.charge)
    assert abs(e - r["energy"]) < 1e-9
