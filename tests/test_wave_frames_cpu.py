"""CPU model of the wavefront kernel's semi-global arithmetic (no GPU needed):
unsigned 16-bit values raised by a bias and by row and column frames, the
profile added to both records' halves as one 32-bit integer.  Every sum must
stay inside its half (no borrow from the high half, no carry into it), and the
scores must be plain Gotoh's, at the largest scores, penalties and record
lengths that the fast regime admits.
"""
import numpy as np
import pytest

from test_recurrence_cpu import gotoh_rows

ENDS = [0, 1, 4, 5, 8, 12, 13]


def halves(w):
    return w & 0xFFFF, w >> 16


def add32(w, x):
    """w + x with both halves of the result checked to be the halves' own sums."""
    r = (w + x) & 0xFFFFFFFF
    lo = x & 0xFFFF
    lo -= 0x10000 if lo >= 0x8000 else 0
    hi = ((x - lo) >> 16) & 0xFFFF
    hi -= 0x10000 if hi >= 0x8000 else 0
    a, b = halves(w)
    assert 0 <= a + lo <= 0xFFFF and 0 <= b + hi <= 0xFFFF
    assert halves(r) == (a + lo, b + hi)
    return r


def max2(x, y):
    return max(x & 0xFFFF, y & 0xFFFF) | (max(x >> 16, y >> 16) << 16)


def addmax(x, c, y):
    """u16x2 add-max: c added per half, modulo 2^16; the sums must not wrap."""
    (a, b), (ca, cb) = halves(x), halves(c)
    sa, sb = a + ca - (0x10000 if ca >= 0x8000 else 0), b + cb - (0x10000 if cb >= 0x8000 else 0)
    assert 0 <= sa <= 0xFFFF and 0 <= sb <= 0xFFFF
    return max2(sa | (sb << 16), y)


def both(v):
    return (v & 0xFFFF) | ((v & 0xFFFF) << 16)


def wave_pair(q, recs, M, op, ex, ends, G, K, max_len):
    """H(i, Q-1) of both records of a pair, row by row, as the kernel holds them."""
    Q, d = len(q), G * K - len(q)
    R = 1
    while R < (1 << 20) and 2 * R * max(ex, 1) <= 2048:
        R *= 2
    qs, ts = ends & 1, ends & 4
    low = 2 * op if ts else 3 * op + ex * max_len
    bias = low + 8 * ex + 256
    ppad = 0 if ts else -(op + ex)
    n = G * K
    # one thread with all columns: the pipeline only delays the same values
    H = [both(bias + c * ex + (0 if (qs or c < d) else -op - ex * (c - d))) for c in range(n)]
    E = [(h + (ex - op) * 0x10001) & 0xFFFFFFFF for h in H]
    left0, left_ext = (bias * 0x10001, ex * 0x10001) if ts else (op * 0x10001, 0)
    eo = both(ex - op)
    out = []
    for i in range(max(len(r) for r in recs)):
        f = (i & (R - 1)) * ex
        if i and (i & (R - 1)) == 0:
            H = [add32(h, -R * ex * 0x10001) for h in H]
            E = [add32(e, -R * ex * 0x10001) for e in E]
        diag = left0 + (i & (R - 1)) * left_ext - left_ext
        F = 0
        codes = [r[min(i, len(r) - 1)] for r in recs]
        new = []
        for c in range(n):
            pa, pb = ((ppad if c < d else int(M[x][q[c - d]])) + 2 * ex for x in codes)
            dp = add32(diag if c == 0 else H[c - 1], pb * 65536 + pa)
            h = max2(max2(dp, E[c]), F)
            E[c] = addmax(h, eo, E[c])
            F = addmax(h, eo, F)
            new.append(h)
        H = new
        out.append([x - bias - f - n * ex for x in halves(H[-1])])
    return out


@pytest.mark.parametrize("case", ["plain", "top", "deep", "long_gap", "fixed_long"])
@pytest.mark.parametrize("ends", ENDS)
def test_framed_values_stay_in_their_halves(case, ends):
    rng = np.random.default_rng(100 * ENDS.index(ends) + len(case))
    G, K, op, ex, alpha, lens = {
        "plain": (2, 6, 3, 1, 5, (23, 17)),
        # (Q + 1) * max(M) just below 30,000
        "top": (2, 118, 11, 3, 4, (240, 239)),
        # 2 * open + ext * (padded Q + 3) + |min M| + 64 just below 30,000
        "deep": (2, 10, 9999, 400, 4, (19, 26)),
        "long_gap": (2, 26, 600, 512, 4, (41, 38)),
        # the longest records a fixed target start admits with these penalties
        "fixed_long": (1, 9, 500, 120, 4, (205, 180)),
    }[case]
    Q = G * K - 1
    M = rng.integers(-128, 128, (alpha, alpha))
    if case == "top":
        M = np.where(np.eye(alpha, dtype=bool), 127, -128)
    q = rng.integers(0, alpha, Q)
    recs = [rng.integers(0, alpha, n) for n in lens]
    if case == "top":
        recs[0] = np.concatenate([q, q])[:lens[0]]
    base = 2 * op + ex * (G * K + 3) + 128 + 64
    assert base <= 30000 and (Q + 1) * 127 <= 30000
    if not ends & 4:
        room = (30000 - base - op) // ex
        lens = tuple(min(n, room) for n in lens)
        if min(lens) < 1:
            pytest.skip("no record is short enough for a fixed start with these penalties")
        recs = [r[:n] for r, n in zip(recs, lens)]
    got = wave_pair(q, recs, M, op, ex, ends, G, K, max(lens))
    for x, r in enumerate(recs):
        want = [H[-1] for _, H in gotoh_rows(q, r, M, op, ex, ends)]
        assert [row[x] for row in got[:len(r)]] == want
