"""The FP64 Fock build's two forms of a quartet (FP64 at or above a Schwarz bound of 1/8, pairs of floats
below it) and its launches with several lanes per quartet, against the stored integrals of the same
context, which are computed in FP64 throughout and contracted in FP64."""
import numpy as np
import pytest

from conftest import rand_density

# sizes on both sides of the launch rules: a few hundred quartets (one warp each), a few thousand in some
# classes, and classes split into both forms; s/p, and d shells through the fixtures
MOLECULES = [("water", 1), ("water", 2), ("water", 3), ("water", 6), ("alkane", 1), ("alkane", 3)]


def _bound(b, pmax):
    """Every integral of a quartet below the cut of 1/8 carries at most 2^-45 of it (a few operations of
    2^-48 on every value that enters); a G element sums N^2 products with the density, each integral
    reached by at most three of them (J once, twice over, and K)."""
    return 3.0 * b.norb ** 2 * 0.125 * 2.0 ** -45 * pmax


@pytest.mark.gpu
@pytest.mark.parametrize("uhf", [False, True])
@pytest.mark.parametrize("basis", ["STO-3G", "6-31G"])
@pytest.mark.parametrize("system,n", MOLECULES)
def test_split_build_matches_stored_integrals(gpu, system, n, basis, uhf):
    from unomol_gb300 import molecules, native
    from unomol_gb300.basis import Basis
    atoms = molecules.water_cluster(n, 5) if system == "water" else molecules.alkane(n)
    b = Basis(text=molecules.patin_text(atoms, basis))
    Ps = [rand_density(b.norb, 11 + k) for k in range(2 if uhf else 1)]
    t = native.TwoElectronInts(b)
    direct = t.form_g_uhf(*Ps) if uhf else [t.form_g(Ps[0])]
    t.store_integrals(native.STORE_UHF if uhf else native.STORE_RHF)
    stored = t.form_g_uhf(*Ps) if uhf else [t.form_g(Ps[0])]
    for g, w in zip(direct, stored):
        assert np.abs(g - w).max() <= _bound(b, max(np.abs(p).max() for p in Ps))


@pytest.mark.gpu
def test_split_build_far_from_the_origin(gpu):
    """A molecule 4096 bohr from the origin (its coordinates, multiples of 2^-20 bohr, are exact there):
    the pairs of floats hold coordinates relative to the molecule, so G moves by no more than FP64
    coordinates of that size make it move (2^-41 bohr on the products' centres)."""
    from unomol_gb300 import molecules, native
    from unomol_gb300.basis import Basis
    b = Basis(text=molecules.patin_text(molecules.water_cluster(3, 5), "6-31G"))
    b.centers = np.round(np.asarray(b.centers) * 2.0 ** 20) / 2.0 ** 20
    P = rand_density(b.norb, 3)
    G = native.TwoElectronInts(b).form_g(P)
    b.centers = b.centers + 4096.0
    H = native.TwoElectronInts(b).form_g(P)
    assert np.abs(G - H).max() <= _bound(b, 1.0) + 3.0 * b.norb ** 2 * 2.0 ** -41


@pytest.mark.gpu
@pytest.mark.parametrize("basis", ["STO-3G", "6-31G"])
@pytest.mark.parametrize("system,n", MOLECULES)
def test_screened_fp64_build_matches_stored_integrals(gpu, system, n, basis):
    """The density-screened FP64 build with nothing skipped: its part of every class in the group kernels or one
    lane per quartet, by the number of quartets."""
    from unomol_gb300 import molecules, native
    from unomol_gb300.basis import Basis
    atoms = molecules.water_cluster(n, 5) if system == "water" else molecules.alkane(n)
    b = Basis(text=molecules.patin_text(atoms, basis))
    P = rand_density(b.norb, 11)
    t = native.TwoElectronInts(b)
    t.set_precision(native.PREC_MIXED, 0.0)
    t.set_density_screening(0.0)
    G = t.form_g(P)
    t.store_integrals(native.STORE_RHF)
    assert np.abs(G - t.form_g(P)).max() <= _bound(b, np.abs(P).max())


@pytest.mark.gpu
def test_two_root_regime_edge(gpu):
    """The reference's two-root form starts above T = 15, where it departs from the exact one by 3.5e-4.  Two
    centres at distances that put T of their (ps|ps) quartets within a few 2^-24 of 15 on both sides: the pairs
    of floats and the FP64 integrals take the same side, whatever the parts of T."""
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    worst = 0.0
    for a, c in ((0.5, 0.5), (0.37, 0.61), (0.83, 0.29)):
        p, q = 2 * a, 2 * c  # both pairs on one centre each
        for k in range(-12, 13):
            R = np.sqrt(15.0 * (1.0 + (k + 0.5) * 2.0 ** -25) * (p + q) / (p * q))
            d = np.array([0.36, 0.48, 0.8]) * R
            text = "\n".join(["4 8 2 1", "2 50", "1e-10", "0 0", "2 1 0", "0 0 0", "1.0 0.0 0.0 0.0",
                              f"1.0 {d[0]!r} {d[1]!r} {d[2]!r}"]
                             + [f"1 {l} {x}\n{e!r} 1.0" for x, e in ((0, a), (1, c)) for l in (0, 1)]) + "\n"
            text = text.replace("np.float64(", "").replace(")", "")
            b = Basis(text=text)
            P = rand_density(b.norb, 4)
            t = native.TwoElectronInts(b)
            t.set_precision(native.PREC_MIXED, 0.0)  # the screened FP64 build: its quartets in both forms
            t.set_density_screening(0.0)
            G = t.form_g(P)
            t.store_integrals(native.STORE_RHF)
            worst = max(worst, float(np.abs(G - t.form_g(P)).max()))
    assert worst <= 1e-10
