"""Windows of the CSR stream kernel (csr_stream.cu: stream_windows and the
walk of stream_window), restated in numpy: every nonzero belongs to exactly
one window, rows start and end where row_offset says, and every window that
meets a split row leaves exactly one piece of it, in window order."""
import bisect

import numpy as np
import pytest

OVER = 32  # kOver


def windows(rp, T):
    """(first, end, row ordinal, flags) per window, and the split rows' (first
    window, last window, ordinal)."""
    m, nnz = len(rp) - 1, int(rp[-1])
    rp = [int(v) for v in rp]
    pos = np.concatenate([[0], np.cumsum(np.diff(rp) > 0)])
    out, rows = [], []
    for w in range(-(-nnz // T)):
        a, b = w * T, min(w * T + T, nnz)
        r, r2 = bisect.bisect_left(rp, a, 0, m), bisect.bisect_left(rp, b, 0, m)
        split = lambda i: rp[i + 1] > (rp[i] // T + 1) * T + OVER  # noqa: E731
        eA, first, flags = rp[r], pos[r] if r < m else r, 0
        if eA > a and split(r - 1):
            flags, eA, first = 1, a, pos[r - 1]
        if r2 > r:
            if split(r2 - 1):
                flags |= 2
                eB = b
                rows.append((w, (rp[r2] - 1) // T, int(pos[r2 - 1])))
            else:
                eB = rp[r2]
        elif flags & 1:
            eB = min(rp[r], b)
            flags |= 2 if rp[r] > b else 0
        else:
            eB = eA
        out.append((eA, eB, int(first), flags))
    return out, rows


def row_offsets(lens):
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)


rng = np.random.default_rng(3)
CASES = {
    "one": [1],
    "one_long": [5000],
    "window": [256, 256, 512, 1],
    "window_edges": [255, 1, 256, 257, 0, 0, 511, 1, 512, 2],
    "over_edges": [1, 511, 1, 512, 1, 513, 200, 312, 1, 100, 669, 3],
    "empty_ends": [0, 0, 3, 0, 700, 0, 0, 2000, 0, 0],
    "short": rng.integers(0, 12, 3000),
    "uniform32": [32] * 500,
    "zipf": np.minimum(rng.zipf(1.5, 800), 6000),
    "long_runs": [3, 4000, 5, 0, 1300, 900, 300, 10000, 1],
}


@pytest.mark.parametrize("T", [224, 480, 992, 1248])
@pytest.mark.parametrize("case", list(CASES))
def test_windows_cover_every_row_once(case, T):
    rp = row_offsets(CASES[case])
    nnz = int(rp[-1])
    nonempty = np.flatnonzero(np.diff(rp))
    ends = np.zeros(nnz, bool)
    ends[rp[nonempty + 1] - 1] = True
    covered, pieces, written = np.zeros(nnz, int), {}, {}
    recs, split = windows(rp, T)
    for w, (eA, eB, row, flags) in enumerate(recs):
        assert 0 <= eA <= eB <= nnz and eB <= (w + 1) * T + OVER
        covered[eA:eB] += 1
        head_split = bool(flags & 1)
        start = eA
        for e in range(eA, eB):
            if ends[e]:
                i = nonempty[row]
                if head_split:
                    head_split = False
                    pieces.setdefault(row, []).append(("head", w))
                else:
                    assert (start, e + 1) == (rp[i], rp[i + 1])  # a whole row
                    written[row] = written.get(row, 0) + 1
                row += 1
                start = e + 1
        if flags & 2:
            pieces.setdefault(row, []).append(("tail", w))
        else:
            assert start == eB  # nothing left open
    assert np.all(covered == 1)
    for w0, w1, row in split:
        # tail pieces of w0 .. w1 - 1, then the head piece of w1
        assert pieces.pop(row) == [("tail", w) for w in range(w0, w1)] + [("head", w1)]
        written[row] = written.get(row, 0) + 1
    assert not pieces
    assert sorted(written) == list(range(len(nonempty))) and set(written.values()) <= {1}
