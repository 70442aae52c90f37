"""Two-float arithmetic (csrc/gbhf_ff.cuh) of the direct builds: its generated
integral code on the host against long double, and builds that use it on the
GPU against the oracle and under scaling of the density."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from gbhf import _lib, basis as B, molecules as M

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "haskell-abinitio_gb300" / "csrc"


def test_two_float_code_against_long_double(tmp_path):
    """1/sqrt to 2^-45; F_0..F_9 to 2^-41 (nine recursion steps, each a few
    2^-46); primitive quartets to 2^-43 rms and 2^-40 at worst of the largest
    component (a few dozen operations of 2^-46 with partial cancellation)."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "ff_check"
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC),
                    str(Path(__file__).resolve().parent / "host" / "ff_check.cpp"), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    rows = [line.split() for line in subprocess.run([str(exe)], check=True, capture_output=True,
                                                     text=True).stdout.splitlines()]
    res = {r[0]: (float(r[1]), float(r[2])) for r in rows}
    assert res["rsqrt"][0] < 2.0 ** -45
    assert res["boys"][0] < 2.0 ** -41
    eri = [k for k in res if k not in ("rsqrt", "boys") and not k.startswith("grad_")]
    assert len(eri) == 13
    for k in eri:
        assert res[k][0] < 2.0 ** -40 and res[k][1] < 2.0 ** -43, (k, res[k])
    for k in res:
        if k.startswith("grad_"):   # derivatives of one-centre quartets cancel
            assert res[k][0] < 1e-8, (k, res[k])


def _density(fb, seed):
    """Symmetric, falling off with distance, with the large core diagonal of a density."""
    rng = np.random.default_rng(seed)
    pos = fb.xyz[fb.cgf_atom]
    r = np.linalg.norm(pos[:, None] - pos[None], axis=2)
    d = rng.standard_normal((fb.n_cgf, fb.n_cgf)) * 0.15
    d = (d + d.T) * np.exp(-r / 1.6) + np.diag(rng.uniform(0.3, 2.0, fb.n_cgf))
    return O.square_to_tri(d)


@pytest.mark.gpu
@pytest.mark.parametrize("waters,basis", [(3, "6-31g"), (4, "sto-3g"), (2, "6-31g*")])
def test_fp64_fock_with_two_float_quartets(ctx, waters, basis):
    """Unscreened FP64 builds large enough for the two-float lists: elements up
    to ~30, sums of ~1e5 rounding errors of 2^-53 and of 2^-50 (2^-45 of quartets
    below 2^-5 of the largest, a random walk): 1e-13 absolute."""
    xyz = M.water_cluster(waters, np.random.default_rng(waters))
    fb = B.flatten(B.make_atoms(M.water_labels(waters), xyz, basis))
    ob = O.OracleBasis(fb)
    ctx.set_basis(fb)
    h, d = ob.hcore(False), _density(fb, waters)
    ref = O.fock_canonical(h, d, ob.eri_canonical(False))
    got = ctx.fock(h, d, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-13 * max(1.0, np.abs(ref).max()))


@pytest.mark.gpu
@pytest.mark.parametrize("power", [-300, 300])
def test_fock_is_linear_far_outside_the_fp32_range(ctx, power):
    """The two-float density is scaled by a power of two: densities of any size
    give the same digits (1e-13: the order of the FP64 atomics differs)."""
    xyz = M.water_cluster(3, np.random.default_rng(3))
    fb = B.flatten(B.make_atoms(M.water_labels(3), xyz, "6-31g"))
    ctx.set_basis(fb)
    d = _density(fb, 9)
    h = np.zeros_like(d)
    one = ctx.fock(h, d, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0)
    far = ctx.fock(h, d * 2.0 ** power, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0) * 2.0 ** -power
    np.testing.assert_allclose(far, one, rtol=0, atol=1e-13 * np.abs(one).max())


@pytest.mark.gpu
def test_exponents_outside_the_fp32_range_stay_in_fp64(ctx):
    """A basis with an exponent of 1e-9 is outside the two-float range: its FP64
    build still matches the oracle."""
    xyz = M.water_cluster(3, np.random.default_rng(3))
    atoms = B.make_atoms(M.water_labels(3), xyz, "6-31g")
    atoms[1].basis = atoms[1].basis + [B.CGF(((1e-7, 1e-9),), "S")]
    fb = B.flatten(atoms)
    ob = O.OracleBasis(fb)
    ctx.set_basis(fb)
    h, d = ob.hcore(False), _density(fb, 4)
    ref = O.fock_canonical(h, d, ob.eri_canonical(False))
    got = ctx.fock(h, d, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-13 * np.abs(ref).max())


def _one_atom_pair(shells):
    """Two atoms with one-primitive shells of the given angular momenta."""
    lab = {0: ("S",), 1: ("Px", "Py", "Pz"), 2: ("Dxx", "Dxy", "Dxz", "Dyy", "Dyz", "Dzz")}
    fns = [B.CGF(((1.0, 0.7 + 0.4 * i),), t) for i, l in enumerate(shells) for t in lab[l]]
    return B.flatten([B.AtomData((0.0, 0.0, 0.0), fns, 8.0), B.AtomData((0.0, 0.3, 1.9), fns, 8.0)])


@pytest.mark.gpu
@pytest.mark.parametrize("shells", [(0,), (0, 0), (1, 0), (2,), (2, 0), (2, 0, 0), (2, 1), (2, 2, 0, 0), (2, 1, 0)],
                         ids=lambda s: "".join("spd"[l] for l in s))
def test_every_class_alone_and_with_zero_density(ctx, shells):
    """Unscreened builds over few shells: a zero density gives exactly the core
    matrix, a random one the stored-integral Fock matrix (1e-12: sums of a few
    hundred rounding errors of elements of order one to ten)."""
    fb = _one_atom_pair(shells)
    ctx.set_basis(fb)
    ntri = fb.n_cgf * (fb.n_cgf + 1) // 2
    h = np.arange(ntri, dtype=float)
    np.testing.assert_array_equal(ctx.fock(h, np.zeros(ntri), _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0), h)
    d = np.random.default_rng(1).standard_normal(ntri)
    ref = O.fock_canonical(np.zeros(ntri), d, O.OracleBasis(fb).eri_canonical(False))
    got = ctx.fock(np.zeros(ntri), d, _lib.MODE_EXACT, _lib.PREC_FP64, 0.0, 0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12)


@pytest.mark.gpu
def test_queued_batches_of_a_large_system(ctx):
    """(H2O)10/6-31G: 4 095 pairs, ket ranges longer than a batch and batches cut by
    the density screening; FP64 against the oracle's screened build and mixed
    against FP64 (the bounds of the library's own Fock tests)."""
    xyz = M.water_cluster(10, np.random.default_rng(10))
    fb = B.flatten(B.make_atoms(M.water_labels(10), xyz, "6-31g"))
    ob = O.OracleBasis(fb)
    ctx.set_basis(fb)
    h, d = ob.hcore(False), _density(fb, 10)
    ref, _ = ob.fock_direct(h, d, 1e-12)
    got = ctx.fock(h, d, _lib.MODE_EXACT, _lib.PREC_FP64, 1e-12, 0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-10)
    mix = ctx.fock(h, d, _lib.MODE_EXACT, _lib.PREC_MIXED, 1e-12, 1e-4)
    assert 0 < np.max(np.abs(mix - got)) < 1e-6
