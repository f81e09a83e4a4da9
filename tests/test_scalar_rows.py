"""The binding's residues of integer constants (Context.lincomb), in bulk and one at a time."""
import random
from types import SimpleNamespace

import numpy as np


def test_scalar_rows_match_single_residues():
    import fides_b200 as F
    rng = random.Random(4)
    ctx = SimpleNamespace(q=[(1 << 60) - 93, (1 << 50) - 27, (1 << 62) - 57, 12289])
    ctx._scalars = lambda v, l: F.Context._scalars(ctx, v, l)
    ends = [0, -1, (1 << 63) - 1, -(1 << 63), 12289, -12289]
    for extra in ([], [1 << 63], [-(1 << 100)], [[1, 2, 3, 4]], [np.int64(-5)]):
        rows = ends + [rng.randrange(-(1 << 63), 1 << 63) for _ in range(20)] + extra
        got = F.Context._scalar_rows(ctx, rows, 4)
        want = np.stack([ctx._scalars(v, 4) for v in rows])
        assert got.dtype == want.dtype == np.uint64 and got.flags.c_contiguous
        assert np.array_equal(got, want)


def test_scalar_rows_of_any_iterable():
    """The constants may come from an iterator or a view, which can be walked once or not be indexed."""
    import fides_b200 as F
    ctx = SimpleNamespace(q=[(1 << 60) - 93, 12289])
    ctx._scalars = lambda v, l: F.Context._scalars(ctx, v, l)
    for rows in ([5, -7, 1 << 40], [5, -(1 << 100)], [[1, 2], 3]):
        want = np.stack([ctx._scalars(v, 2) for v in rows])
        for it in (iter(rows), (v for v in rows), map(lambda v: v, rows), dict(enumerate(rows)).values(), tuple(rows)):
            assert np.array_equal(F.Context._scalar_rows(ctx, it, 2), want)


def test_no_constants_are_refused():
    """The library reads one row of residues per ciphertext: an empty list must not reach it."""
    import pytest

    import fides_b200 as F
    ctx = SimpleNamespace(q=[(1 << 60) - 93, 12289])
    ctx._scalars = lambda v, l: F.Context._scalars(ctx, v, l)
    for none in ([], (), iter(())):
        with pytest.raises(ValueError):
            F.Context._scalar_rows(ctx, none, 2)
