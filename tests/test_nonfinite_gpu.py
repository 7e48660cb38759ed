"""Integrals that overflow show in G: the degeneracy factor, applied to the exponent field, leaves infinities and NaN."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("l", [0, 2])  # the templated kernels and the warp-per-quartet ones
def test_overflowing_integrals_stay_non_finite(gpu, l):
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    n = (l + 1) * (l + 2) // 2
    b = Basis(text=f"1 {n} 1 {l}\n2 50\n1e-10\n0 0\n2 1 0\n0 0 0\n2.0 0.0 0.0 0.0\n1 {l} 0\n0.8 1.0\n")
    P = np.zeros(b.no2)
    P[[i * (i + 1) // 2 + i for i in range(n)]] = 0.5
    assert np.isfinite(native.TwoElectronInts(b).form_g(P)).all()
    b.coef[0] = np.inf
    G = native.TwoElectronInts(b).form_g(P)
    assert not np.isfinite(G[0])  # (00|00), one shell pair with itself, is the only quartet
