"""Launches of the warp-per-quartet kernels: from several threads at once, and above one row of CTAs."""
import threading

import numpy as np
import pytest

from conftest import rand_density


def _text(shells, ncen, spread, seed):
    """ncen centres in a cube of `spread` bohr; `shells`: (l, exponent, centres that carry it)."""
    rng = np.random.default_rng(seed)
    sh = [(l, a, c) for l, a, cs in shells for c in cs]
    norb = sum((l + 1) * (l + 2) // 2 for l, _, _ in sh)
    lines = [f"{len(sh)} {norb} {ncen} {max(l for l, _, _ in sh)}", "2 50", "1e-10", "0 0", "2 1 0", "0 0 0"]
    lines += ["1.0 " + " ".join(f"{x:.6f}" for x in rng.uniform(0, spread, 3)) for _ in range(ncen)]
    lines += [f"1 {l} {c}\n{a} 1.0" for l, a, c in sh]
    return "\n".join(lines) + "\n"


@pytest.mark.gpu
def test_builds_of_several_threads(gpu):
    """Classes of one register budget with different amounts of shared memory ((dd|dd) 70 KB, (fp|fp) 56, (ff|pp) 60),
    launched by four threads, each with a context of its own."""
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    bases = [Basis(text=_text([(2, 0.8, range(2))], 2, 2.0, 1)), Basis(text=_text([(3, 0.7, range(2)), (1, 0.9, range(2))], 2, 2.0, 2))] * 2
    Ps = [rand_density(b.norb, 3) for b in bases]
    want = [native.TwoElectronInts(b).form_g(P) for b, P in zip(bases, Ps)]
    failed = []

    def work(b, P, w):
        try:
            t = native.TwoElectronInts(b)
            for _ in range(400):
                assert np.abs(t.form_g(P) - w).max() <= 1e-10
        except Exception as e:  # noqa: BLE001 (reported below)
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(bases, Ps, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:2]


@pytest.mark.gpu
def test_more_quartets_than_one_row_of_ctas(gpu):
    """One f shell and 165 s shells: 165 (fs| pairs with 13695 |ss) pairs are 2.26 million quartets, more than 2^21."""
    from unomol_gb300 import native
    from unomol_gb300.basis import Basis
    b = Basis(text=_text([(3, 0.5, [0]), (0, 0.4, range(165))], 165, 6.0, 5))
    P = rand_density(b.norb, 3)
    t = native.TwoElectronInts(b)
    direct = t.form_g(P)
    t.set_precision(native.PREC_MIXED, 0.0)  # the screened build's list, nothing skipped
    t.set_density_screening(0.0)
    screened = t.form_g(P)
    t.set_precision(0)
    t.store_integrals(native.STORE_RHF)
    want = t.form_g(P)
    for g in (direct, screened):
        assert np.abs(g - want).max() <= 1e-12 * np.abs(want).max()
