"""The searches' selection from ranks against the reference's loop (CPU only).

The run search, the search of wide windows and the test of the proposals keep an
err_diff as a rank, 0 below zero and err_diff + 1 from there on, and select by the
smallest rank at its first position; where a window holds an err_diff < 0 or = 0, by the
first position of rank 0 or 1 and the last row that holds a rank 0. A window may be
taken in slabs of rows whose statistics are merged. The selection counts where its
m is at most the threshold."""
import numpy as np

from test_selection_rule import INVALID, random_window, reference_loop

NO_RANK = 0xFFFF


def rank(e):
    return NO_RANK if e is INVALID else max(e, -1) + 1


def by_ranks(rows, thr, slab):
    n = len(rows[0])
    best, first, last = None, None, None  # (rank, position), position, (row, position)
    for r0 in range(0, len(rows), slab):
        window = [(rank(e), r, r * n + c) for r in range(r0, min(r0 + slab, len(rows))) for c, e in enumerate(rows[r])]
        b = min(((v, p) for v, _, p in window))
        if b[0] <= 1:  # else no position of the slab has an err_diff <= 0
            le0 = [p for v, _, p in window if v <= 1]
            first = min(le0) if first is None else first
            for v, r, p in window:
                if v == 0 and (last is None or r > last[0]):
                    last = (r, p)
        best = b if best is None else min(best, b)
    if best[0] <= 1:
        pos = last[1] if last is not None and last[0] > first // n else first
        return divmod(pos, n) if thr >= 0 else None
    return divmod(best[1], n) if best[0] != NO_RANK and best[0] - 1 <= thr else None


def test_ranks_equal_reference_loop():
    rng = np.random.default_rng(77)
    for _ in range(20000):
        rows = random_window(rng, int(rng.integers(1, 7)), int(rng.integers(1, 9)))
        thr = int(rng.choice([-3, -1, 0, 1, 2, 5, 70000, 0x7FFFFFFE]))
        sel, m = reference_loop(rows)
        want = sel if sel is not None and m <= thr else None
        for slab in (1, 2, 3, len(rows)):
            assert by_ranks(rows, thr, slab) == want, (rows, thr, slab)


def test_the_largest_err_diff_has_a_rank():
    assert rank(65025) == 65026 < NO_RANK
    assert by_ranks([[INVALID, 65025]], 65025, 1) == (0, 1)
    assert by_ranks([[INVALID, 65025]], 65024, 1) is None
    assert by_ranks([[INVALID, INVALID]], 0x7FFFFFFE, 1) is None
