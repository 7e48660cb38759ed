"""Quartets in pairs of floats whose T lies on both sides of the two-root form's edges (15, 40) and of the ends of the
one-, two- and three-root tables (41, 48, 55), within 2^-22 of it, against the stored integrals of the same context,
which are computed in FP64 throughout."""
import numpy as np
import pytest

from conftest import rand_density

EXPONENTS = [(0.008, 0.008), (0.0061, 0.0079), (0.0047, 0.0066)]
DIRECTION = np.array([0.36, 0.48, 0.8])


def _text(a, c, m, edge):
    """Two groups of m centres, an s and a p shell on each, exponents a in one group and c in the other.  The centres
    of a group lie so close together that every quartet of one pair in each group has T within 2^-22 of `edge`; the
    steps leave no T nearer than 2^-33 to it, far more than either arithmetic's rounding."""
    p, q = 2 * a, 2 * c
    R = np.sqrt(edge * (p + q) / (p * q))
    step = R * 2.0 ** -22 / m ** 2
    one = [-(i - m // 2) * step for i in range(m)]
    two = [R + ((j - m // 2) * m + 0.125) * step for j in range(m)]
    cen = [x * DIRECTION for x in one + two]
    lines = [f"{4 * m} {8 * m} {2 * m} 1", "2 50", "1e-10", "0 0", "2 1 0", "0 0 0"]
    lines += [f"1.0 {float(x)!r} {float(y)!r} {float(z)!r}" for x, y, z in cen]
    lines += [f"1 {l} {i}\n{a if i < m else c!r} 1.0" for i in range(2 * m) for l in (0, 1)]
    return "\n".join(lines) + "\n"


def _tolerance(b, P):
    """A quartet below 1/8 carries at most 2^-45 of it; a G element sums N^2 products with the density, each integral
    reached at most three times."""
    return 3.0 * b.norb ** 2 * 0.125 * 2.0 ** -45 * np.abs(P).max()


# the number of centres sets the lanes per quartet of the (ps|ps) class: a warp, four lanes, one lane
@pytest.mark.gpu
@pytest.mark.parametrize("m", [5, 8, 12])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("edge", [15.0, 40.0, 41.0, 48.0, 55.0])
def test_quartets_at_the_edges_of_the_root_tables(gpu, edge, exact, m, tmp_path):
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    for a, c in EXPONENTS:
        one = native.TwoElectronInts(Basis(text=_text(a, c, 1, edge)))
        one.write_records(str(tmp_path / "r"))
        # the largest integral is a Schwarz bound squared: every quartet takes pairs of floats
        assert 1e-3 < np.abs(np.fromfile(tmp_path / "r", dtype=native.RECORD_DTYPE)["val"]).max() < 0.125
        b = Basis(text=_text(a, c, m, edge))
        P = rand_density(b.norb, 4)
        t = native.TwoElectronInts(b)
        t.set_rys_mode(native.RYS_EXACT if exact else native.RYS_REFERENCE)
        plain = t.form_g(P)
        t.set_precision(native.PREC_MIXED, 0.0)  # the screened FP64 build, nothing skipped: kernels of its own
        t.set_density_screening(0.0)
        screened = t.form_g(P)
        t.set_precision(0)
        t.store_integrals(native.STORE_RHF)
        want = t.form_g(P)
        assert np.abs(plain - want).max() <= _tolerance(b, P)
        assert np.abs(screened - want).max() <= _tolerance(b, P)


@pytest.mark.gpu
@pytest.mark.parametrize("edge", [15.0, 48.0])
def test_batches_at_the_edges_of_the_root_tables(gpu, edge):
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    bases = [Basis(text=_text(a, c, 6, edge)) for a, c in EXPONENTS]
    Ps = [rand_density(b.norb, 4 + k) for k, b in enumerate(bases)]
    bat = native.Batch(bases)
    for mixed in (False, True):
        if mixed:
            bat.set_precision(native.PREC_MIXED, 0.0, 0.0)
        bat.set_densities(Ps)
        bat.fock()
        for b, P, g in zip(bases, Ps, bat.get_focks()):
            t = native.TwoElectronInts(b)
            t.store_integrals(native.STORE_RHF)
            assert np.abs(g - t.form_g(P)).max() <= _tolerance(b, P)


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(10))
def test_batch_of_256_molecules_matches_each_ones_stored_integrals(gpu, seed):
    """The batching workload's mix (half alkanes, half water clusters, STO-3G or 6-31G) at ten sets of geometries."""
    from unomol_gb300 import molecules, native
    from unomol_gb300.basis import Basis
    rng = np.random.default_rng(256)
    texts = []
    for i in range(256):
        basis = "STO-3G" if rng.integers(2) == 0 else "6-31G"
        if i < 128:
            atoms = molecules.perturb(molecules.alkane(int(rng.integers(1, 9))), 0.05, 1000 * seed + i)
        else:
            atoms = molecules.water_cluster(int(rng.integers(1, 7)), 1000 * seed + i)
        texts.append(molecules.patin_text(atoms, basis))
    bases = [Basis(text=t) for t in texts]
    Ps = [rand_density(b.norb, seed + 3 * k) for k, b in enumerate(bases)]
    want = []
    for b, P in zip(bases, Ps):
        t = native.TwoElectronInts(b)
        t.store_integrals(native.STORE_RHF)
        want.append(t.form_g(P))
        t.close()
    bat = native.Batch(bases)
    bat.set_densities(Ps)
    bat.fock()
    plain = bat.get_focks()
    bat.set_precision(native.PREC_MIXED, 0.0, 0.0)
    bat.fock()
    for g, s, w in zip(plain, bat.get_focks(), want):
        assert np.abs(g - w).max() <= 1e-10  # the suite's tolerance of G
        assert np.abs(s - w).max() <= 1e-10
    bat.close()
