"""Bucket 0 gets the blocked hands' term of every river card and, between two of them, the staged sums
of the card before: in a pass with one CTA per root two warps add them, one after the other. The order
is that of a split pass, where one thread adds all terms, so regrets and average sums of the same roots
agree bit for bit, in every run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLOP = (1 << 6) | (1 << 21) | (1 << 44)
N, CHUNK = 300, 60  # CHUNK roots are split over CTAs, N are not


def _pass(P, tables, boards, bets, reg, ranges, average):
    b = P.Builder()
    for c, x in zip(boards, bets):
        b.add(c, float(x))
    if average:
        b.enable_average()
    b.set_regrets(reg)
    for p in range(2):
        if average:
            b.upload_own_all(ranges[1 - p])
        b.upload_all(ranges[p])
        b.evaluate(tables, p)
    got = b.regrets(), b.average_sums() if average else np.zeros(0, np.float32)
    b.close()
    return got


@pytest.mark.parametrize("average", [False, True])
def test_whole_and_split_passes_add_in_one_order(average):
    import pokerrust_b200 as P
    tables = P.build_flop_tables(FLOP)
    rng = np.random.default_rng(12)
    turns = [c for c in range(52) if not FLOP >> c & 1]
    boards = [FLOP | (1 << turns[i % len(turns)]) for i in range(N)]
    bets = rng.integers(1, 20, N).astype(np.float32)
    reg = np.maximum(rng.random((N, 26, 256), dtype=np.float32) * 100 - 30, 0)
    ranges = rng.random((2, N, 1326), dtype=np.float32)
    whole = _pass(P, tables, boards, bets, reg, ranges, average)
    again = _pass(P, tables, boards, bets, reg, ranges, average)
    parts = [_pass(P, tables, boards[i:i + CHUNK], bets[i:i + CHUNK], reg[i:i + CHUNK], ranges[:, i:i + CHUNK], average)
             for i in range(0, N, CHUNK)]
    P.free_eval(tables)
    for k in range(1 + average):
        assert np.array_equal(whole[k], again[k])
        assert np.array_equal(whole[k], np.concatenate([x[k] for x in parts]))
