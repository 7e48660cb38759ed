"""The warp-per-quartet kernels (classes with more than 81 function quartets, f and g shells) against the stored
integrals of the same context, computed one lane per quartet with the recurrences of the other kernels."""
import numpy as np
import pytest

from conftest import rand_density

TOL_G = 1e-10  # the suite's tolerance of G


def _text(shells):
    """Two centres, every (l, primitives) of `shells` on both; `primitives` geometric exponents from 0.4."""
    sh = [(l, k, c) for c in (1, 2) for l, k in shells]
    norb = sum((l + 1) * (l + 2) // 2 for l, _, _ in sh)
    out = [f"{len(sh)} {norb} 2 {max(l for l, _, _ in sh)}", "2 50", "1e-10", "0 0", "2 1 0", "0 0 0",
           "1.0 0.1 0.2 -0.3", "1.0 0.9 -0.4 1.1"]
    for l, k, c in sh:
        out.append(f"{k} {l} {c - 1}")
        out += [f"{0.4 * 2.1 ** i:.6f} {1.0 / (i + 1):.6f}" for i in range(k)]
    return "\n".join(out) + "\n"


# 6 primitives: 36 x 36 primitive quartets, several rounds of the 32-wide screen; 1: a single one.  The kernels'
# register budgets change at 128, 224, 384 and 672 function quartets: (ds|dp) 108, (dd|ds) 216, (dp|dp) 324,
# (fd|ds) 360, (dd|dp) 648, (dd|dd) 1296; g shells: (gs|gs) 225, (gd|ds) 540, (gg|ss) 225
@pytest.mark.gpu
@pytest.mark.parametrize("uhf", [False, True])
@pytest.mark.parametrize("shells", [[(2, 1)], [(2, 6), (0, 1)], [(2, 2), (1, 3)], [(3, 1), (2, 1), (0, 2)],
                                    [(4, 1), (0, 1)], [(4, 1), (2, 1), (1, 1), (0, 3)]])
def test_coop_classes_match_stored_integrals(gpu, shells, uhf):
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    b = Basis(text=_text(shells))
    Ps = [rand_density(b.norb, 5 + k) for k in range(2 if uhf else 1)]
    t = native.TwoElectronInts(b)
    t.set_screening(0.0)
    direct = t.form_g_uhf(*Ps) if uhf else [t.form_g(Ps[0])]
    # the density-screened FP64 build (nothing skipped) takes the same kernels over its own work lists
    t.set_precision(native.PREC_MIXED, 0.0)
    t.set_density_screening(0.0)
    screened = t.form_g_uhf(*Ps) if uhf else [t.form_g(Ps[0])]
    t.set_precision(native.PREC_FP64)
    t.store_integrals(native.STORE_UHF if uhf else native.STORE_RHF)
    stored = t.form_g_uhf(*Ps) if uhf else [t.form_g(Ps[0])]
    for g, s, w in zip(direct, screened, stored):
        assert np.abs(g - w).max() <= TOL_G
        assert np.abs(s - w).max() <= TOL_G
