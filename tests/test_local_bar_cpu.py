"""CPU model of the local-alignment bar of the wavefront kernel: several records
stream through a group of threads, each a step behind its left neighbour, and a
row counts only if it beats the thread's own best, the left columns' best up to
the step before and the right columns' best in the rows they have reached."""
import numpy as np
import pytest

from test_recurrence_cpu import blosum_like, sw_matrix, sw_reference_end

RPS = 4  # rows per step


def pipeline_ends(records, Q, G, K):
    """(score, row, column) per record (its H rows), as the kernel's threads find them."""
    steps = [max(1, -(-len(H) // RPS)) for H in records]
    begin = np.cumsum([0] + steps)  # thread 0's first step of each record
    total = int(begin[-1]) + G
    best, right, out_b, left = [0] * G, [0] * G, [0] * G, [0] * G
    row_of, saved = [-1] * G, [None] * G
    found = [[None] * G for _ in records]
    for s in range(total):
        sent_right = [max(b, r) for b, r in zip(best, right)]
        sent_left = list(out_b)
        for t in range(G):
            k = int(np.searchsorted(begin, s - t, side="right")) - 1
            if s < t or k >= len(records):
                continue
            q4 = (s - t - int(begin[k])) * RPS
            if q4 == 0:
                best[t] = left[t] = 0
                row_of[t], saved[t] = -1, None
            msg_b = sent_left[t - 1] if t else 0
            right[t] = 0 if t == G - 1 or q4 < 2 * RPS else sent_right[t + 1]
            thr = max(best[t], left[t], right[t])
            for row in range(q4, min(q4 + RPS, len(records[k]))):
                cols = records[k][row][t * K:min(Q, (t + 1) * K)]
                cm = max(cols) if cols else 0
                if cm > thr:
                    thr = best[t] = cm
                    row_of[t], saved[t] = row, list(cols)
            out_b[t], left[t] = max(best[t], msg_b), msg_b
            found[k][t] = (best[t], row_of[t], t * K + saved[t].index(best[t]) if saved[t] else 0x7FFF)
    ends = []
    for per_thread in found:
        acc = (0, -1, 0x7FFF)
        for b, r, c in per_thread:  # columns to the left win ties
            if b > acc[0] or (b == acc[0] and b > 0 and r < acc[1]):
                acc = (b, r, c)
        ends.append(acc if acc[0] > 0 else (0, -1, 0))
    return ends


@pytest.mark.parametrize("G", [1, 2, 4, 8])
def test_ends_with_the_whole_groups_bar(G):
    rng = np.random.default_rng(70 + G)
    for trial in range(40):
        A = 3 if trial % 2 else 6  # small alphabets: many equal maxima
        M = blosum_like(rng, A)
        Q = int(rng.integers(1, 30))
        K = -(-Q // G)
        q = rng.integers(0, A, Q)
        op, ex = [(3, 1), (5, 2), (2, 1)][trial % 3]
        rows = []
        for length in rng.integers(0, 45, 5):
            r = rng.integers(0, A, int(length))
            if trial % 3 == 0 and len(r) > Q:  # a copy of the query: a high best just before the next record
                pos = int(rng.integers(0, len(r) - Q + 1))
                r[pos:pos + Q] = q
            rows.append(sw_matrix(q, r, M, op, ex))
        assert pipeline_ends(rows, Q, G, K) == [sw_reference_end(H) for H in rows], (G, trial)
