"""Shell offsets that leave elements of the lower triangle without a shell pair (shells out of order, or one that lies
inside another) are refused before any GPU work."""
import pytest


def _basis():
    from unomol_gb300 import molecules
    from unomol_gb300.basis import Basis
    return Basis(text=molecules.patin_text(molecules.water_cluster(1, 0), "STO-3G"))


@pytest.mark.parametrize("change", ["inside", "order"])
def test_bad_shell_offsets_are_refused(change):
    """Water in STO-3G: shells s, s, p on the oxygen and an s on either hydrogen, at 0, 1, 2, 5, 6."""
    from unomol_gb300 import native
    b = _basis()
    assert list(b.shell_offset) == [0, 1, 2, 5, 6]
    b.shell_offset = {"inside": [0, 1, 2, 3, 6], "order": [1, 0, 2, 5, 6]}[change]
    with pytest.raises(native.UnomolError, match="do not cover|beyond norb"):
        native.one_electron_gpu(b)
