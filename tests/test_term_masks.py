"""Masks and phases of many strings at once equal each string's own."""
import numpy as np
import pytest

from qrusty_gb300.pyqrusty import Pauli, _term_masks

PREFIXES = ["", "+", "-", "i", "-i", "j", "1j", "-1i"]


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 62, 63, 64])
def test_masks_equal_each_string(n):
    rng = np.random.default_rng(n)
    paulis = [Pauli(p + "".join(rng.choice(list("IXYZ"), n))) for p in PREFIXES * 4]
    paulis += [Pauli(c * n) for c in "IXYZ"]
    x, z, ph, bp = _term_masks(paulis)
    assert (x.dtype, z.dtype, ph.dtype, bp.dtype) == (np.uint64, np.uint64, np.uint8, np.uint8)
    for k, p in enumerate(paulis):
        assert (int(x[k]), int(z[k])) == (p.x_indices(), p.z_indices())
        assert (int(ph[k]), int(bp[k])) == (p.phase(), p.base_phase())


class Other(Pauli):
    def x_indices(self):
        return 0


def test_other_types_keep_their_methods():
    x, _, _, _ = _term_masks([Pauli("XX"), Other("XX")])
    assert x.tolist() == [3, 0]
