"""The result array of the host-pointer steps: of the caller's qnew only the ghost cells
are carried over where the step writes the rest, whatever the array's order and type; an
array of another shape than the step's is copied whole."""
import numpy as np
import pytest

from pyclaw_b200.classic2 import _prep


@pytest.mark.parametrize("mx,my", [(1, 1), (2, 1), (1, 7), (5, 3)])
@pytest.mark.parametrize("form", ["F", "C", "f4", "strided", "list"])
def test_ghost_cells_are_the_callers(mx, my, form):
    r = np.random.default_rng(mx * 10 + my)
    base = r.integers(-99, 99, (3, mx + 4, my + 4)).astype(float)  # exact in every type
    qnew = {"F": np.asfortranarray(base), "C": base.copy(), "f4": base.astype(np.float32),
            "strided": np.repeat(base, 2, axis=1)[:, ::2], "list": base.tolist()}[form]
    qold = np.zeros_like(base)
    old, out, method, mthlim = _prep(qold, qnew, [1, 2, 2, 0, 0, 0, 0], [4, 4], 2, mx, my)
    assert out.dtype == np.float64 and out.flags.f_contiguous and out.shape == base.shape
    assert not np.shares_memory(out, qnew if form != "list" else base) and not np.shares_memory(out, old)
    ghost = np.ones(base.shape, dtype=bool)
    ghost[:, 2:-2, 2:-2] = False
    assert np.array_equal(out[ghost], base[ghost])


def test_in_place_and_other_shapes():
    q = np.asfortranarray(np.random.default_rng(0).random((3, 9, 8)))
    old, out, _, _ = _prep(q, q, [1], [4], 2, 5, 4)
    assert out is q and old is q
    wide = np.random.default_rng(1).random((3, 9, 9))
    _, out, _, _ = _prep(q, wide, [1], [4], 2, 5, 4)  # not the step's shape: all of it
    assert np.array_equal(out, wide)
