"""What complex_lu_solve_batched refuses before it hands any memory to the library, and what it hands over."""
import types

import numpy as np
import pytest

from refeff_gb300 import fms


class _Library:
    calls = 0

    def refeff_complex_lu_solve_batched(self, *args):
        self.calls += 1
        return 0


def _context():
    return types.SimpleNamespace(_lib=_Library(), handle=None, last_error=lambda: "")


@pytest.mark.parametrize("a,b,error", [((3, 4, 4), (2, 4, 1), IndexError), ((2, 4, 4), (2, 3, 1), ValueError),
                                       ((2, 4, 4), (2, 5, 1), ValueError), ((2, 4, 3), (2, 4, 1), ValueError)])
def test_shapes_that_do_not_fit_reach_no_memory(a, b, error):
    ctx = _context()
    with pytest.raises(error):
        fms.complex_lu_solve_batched(ctx, np.ones(a), np.ones(b))
    assert ctx._lib.calls == 0


def test_right_hand_sides_beyond_the_systems_are_left_out():
    ctx = _context()
    X, st, _ = fms.complex_lu_solve_batched(ctx, np.ones((2, 4, 4)), np.ones((5, 4, 3)))
    assert X.shape == (2, 4, 3) and st.shape == (2,) and ctx._lib.calls == 1
