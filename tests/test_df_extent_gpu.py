"""Molecules of two fragments far apart: the pairs of floats keep the precision of each fragment's own quartets, against
the stored integrals of the same context, which are computed in FP64 throughout."""
import numpy as np
import pytest

from conftest import rand_density


def _text(half, bits, seed):
    """Four centres around each of the two points (+-half, +-half, +-half), an s and a p shell on each.  Exponents are
    powers of two and coordinates multiples of 2^-bits, so that FP64 computes every product's centre exactly."""
    rng = np.random.default_rng(seed)
    lines = ["16 32 8 1", "2 50", "1e-10", "0 0", "2 1 0", "0 0 0"]
    for side in (-1, 1):
        for k in range(4):
            x = side * half + np.array([2.0 * (k & 1), 2.0 * (k >> 1), 0.0]) + rng.uniform(-0.4, 0.4, 3)
            x = np.round(x * 2.0 ** bits) / 2.0 ** bits
            lines.append("1.0 " + " ".join(repr(float(v)) for v in x))
    lines += [f"1 {l} {c}\n0.5 1.0" for c in range(8) for l in (0, 1)]
    return "\n".join(lines) + "\n"


def _tolerance(b, P):
    """A quartet below 1/8 carries at most 2^-45 of it; a G element sums N^2 products with the density, each integral
    reached at most three times."""
    return 3.0 * b.norb ** 2 * 0.125 * 2.0 ** -45 * np.abs(P).max()


@pytest.mark.gpu
@pytest.mark.parametrize("half,bits", [(8.0, 33), (512.0, 33), (262144.0, 33)])
def test_two_fragments_far_apart(gpu, half, bits):
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    for seed in range(4):
        b = Basis(text=_text(half, bits, seed))
        P = rand_density(b.norb, 9)
        t = native.TwoElectronInts(b)
        direct = t.form_g(P)
        t.set_precision(native.PREC_MIXED, 0.0)
        t.set_density_screening(0.0)
        screened = t.form_g(P)
        t.set_precision(0)
        t.store_integrals(native.STORE_RHF)
        want = t.form_g(P)
        assert np.abs(direct - want).max() <= _tolerance(b, P)
        assert np.abs(screened - want).max() <= _tolerance(b, P)
