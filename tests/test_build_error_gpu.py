"""Rounding error of the FP64 build's G against the oracle in long double: no larger than that of a build with every
quartet in FP64, one accumulator per element of T and the light classes first."""
import numpy as np
import pytest

from conftest import rand_density


def core_density(b):
    """The density of the core Hamiltonian's lowest orbitals: the size, decay and signs of a molecule's own density."""
    from unomol_gb300 import native
    S, _, H = native.one_electron(b)
    tri = np.tril_indices(b.norb)

    def square(v):
        m = np.zeros((b.norb, b.norb))
        m[tri] = v
        return m + np.tril(m, -1).T

    s, U = np.linalg.eigh(square(S))
    X = U / np.sqrt(s)
    C = X @ np.linalg.eigh(X.T @ square(H) @ X)[1][:, :b.nelec // 2]
    return np.ascontiguousarray((C @ C.T)[tri])


def error(b, P):
    """rms over G of two builds' errors."""
    from oracle import orc
    from unomol_gb300 import native
    (exact,) = orc.fock_long(b, [P])
    t = native.TwoElectronInts(b)
    e = np.concatenate([np.asarray(t.form_g(P).astype(np.longdouble) - exact, np.float64) for _ in range(2)])
    return float(np.sqrt((e ** 2).mean()))


# the errors of that build, measured (1e-15)
@pytest.mark.gpu
@pytest.mark.parametrize("system,n,basis,seed,density,most", [
    ("alkane", 7, "STO-3G", 3, "random", 2.24), ("alkane", 7, "STO-3G", 5, "random", 2.39),
    ("alkane", 4, "6-31G", 3, "core", 2.38), ("water", 5, "6-31G", 3, "core", 2.31),
])
def test_rounding_error_of_a_build(gpu, system, n, basis, seed, density, most):
    from unomol_gb300 import molecules
    from unomol_gb300.basis import Basis
    atoms = molecules.water_cluster(n, seed) if system == "water" else molecules.perturb(molecules.alkane(n), 0.05, seed)
    b = Basis(text=molecules.patin_text(atoms, basis))
    P = rand_density(b.norb, seed) if density == "random" else core_density(b)
    assert error(b, P) <= most * 1e-15
