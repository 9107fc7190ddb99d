"""Every number of CTAs per root that a river pass takes (the counts of roots below reach them all on 148
SMs), and that it is the split form that ran: values, regrets and average sums of CFR passes, with and
without average sums, and the values of best responses have the bits of the whole pass, which many roots
and passes under capture run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLOP = (1 << 2) | (1 << 27) | (1 << 40)
MOST = 260  # roots that are never split


@pytest.fixture(scope="module")
def tables():
    import pokerrust_b200 as P
    t = P.build_flop_tables(FLOP)
    yield t
    P.free_eval(t)


def _builder(P, n, average):
    rng = np.random.default_rng(21)
    turns = [c for c in range(52) if not FLOP >> c & 1]
    bets = rng.integers(1, 20, MOST)
    b = P.Builder()
    for i in range(n):
        b.add(FLOP | (1 << turns[i % len(turns)]), float(bets[i]))
    if average:
        b.enable_average()
    b.set_regrets(np.maximum(rng.random((MOST, 26, 256), dtype=np.float32)[:n] * 100 - 30, 0))
    return b, rng.random((2, MOST, 1326), dtype=np.float32)[:, :n]


def _cfr(P, tables, n, average):
    b, ranges = _builder(P, n, average)
    splits, out = set(), []
    for p in range(2):
        if average:
            b.upload_own_all(ranges[1 - p])
        b.upload_all(ranges[p])
        b.evaluate(tables, p)
        splits.add(b.splits)
        out.append(b.download_all())
    out.append(b.regrets())
    if average:
        out.append(b.average_sums())
    b.close()
    return splits, out


def _best(P, tables, n):
    b, ranges = _builder(P, n, False)
    assert b.splits == 0
    out = [b.best_response_f64(tables, 1, ranges[1].astype(np.float64))]
    splits = {b.splits}
    b.upload_all(ranges[0])
    b.evaluate(tables, 0, True)
    out.append(b.download_all())
    splits.add(b.splits)
    b.close()
    return splits, out


@pytest.fixture(scope="module")
def whole(tables):
    import pokerrust_b200 as P
    got = {avg: _cfr(P, tables, MOST, avg) for avg in (False, True)}
    got["best"] = _best(P, tables, MOST)
    assert all(s == {1} for s, _ in got.values())
    return {k: v for k, (_, v) in got.items()}


# roots of a CFR pass -> CTAs per root on 148 SMs
FORMS = {1: 48, 5: 24, 8: 16, 10: 12, 13: 8, 20: 6, 28: 4, 40: 3, 74: 2, 149: 6, 172: 6}


@pytest.mark.parametrize("n", FORMS)
@pytest.mark.parametrize("average", [False, True])
def test_cfr_forms(tables, whole, n, average):
    import torch

    import pokerrust_b200 as P
    splits, got = _cfr(P, tables, n, average)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert len(splits) == 1 and min(splits) > 1 and (sms != 148 or splits == {FORMS[n]})
    for x, w in zip(got, whole[average]):
        assert np.array_equal(x, w[:n])


@pytest.mark.parametrize("n", [1, 10, 74, 98, 111, 149, 197, 198, 240])
def test_best_response_forms(tables, whole, n):
    import pokerrust_b200 as P
    splits, got = _best(P, tables, n)
    assert len(splits) == 1 and min(splits) > 1
    for x, w in zip(got, whole["best"]):
        assert np.array_equal(x, w[:n])
