"""A river root's values do not depend on how its pass runs: a pass over few roots (river cards spread
over several CTAs), one over many, and one recorded into a CUDA graph (never split) add a hand's 48
river cards in the same order, so that they agree bit for bit, in CFR and best-response passes and in
double precision. Counts at both ends of the ranges that are split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLOP = (1 << 9) | (1 << 18) | (1 << 50)
MOST = 260  # roots that are never split


def _roots(seed):
    rng = np.random.default_rng(seed)
    turns = [c for c in range(52) if not FLOP >> c & 1]
    boards = [FLOP | (1 << turns[i % len(turns)]) for i in range(MOST)]
    bets = rng.integers(1, 20, MOST).astype(np.float32)
    reg = np.maximum(rng.random((MOST, 26, 256), dtype=np.float32) * 100 - 30, 0)
    return boards, bets, reg, rng.random((2, MOST, 1326), dtype=np.float32)


def _builder(P, n, roots):
    boards, bets, reg, _ = roots
    b = P.Builder()
    for c, x in zip(boards[:n], bets[:n]):
        b.add(c, float(x))
    b.set_regrets(reg[:n])
    return b


def _values(P, tables, n, roots):
    """Values of a CFR pass and of best responses in single and double precision, per player."""
    out = []
    b = _builder(P, n, roots)
    for p in range(2):
        ranges = roots[3][p][:n]
        out.append(b.best_response_f64(tables, p, ranges.astype(np.float64)))
        for exploit in (True, False):
            b.upload_all(ranges)
            b.evaluate(tables, p, exploit)
            out.append(b.download_all())
    b.close()
    return out


@pytest.fixture(scope="module")
def whole():
    import pokerrust_b200 as P
    tables = P.build_flop_tables(FLOP)
    roots = _roots(5)
    yield tables, roots, _values(P, tables, MOST, roots)
    P.free_eval(tables)


@pytest.mark.parametrize("n", [1, 2, 10, 25, 49, 74, 149, 240])
def test_values_have_the_bits_of_the_whole_pass(whole, n):
    import pokerrust_b200 as P
    tables, roots, want = whole
    for got, w in zip(_values(P, tables, n, roots), want):
        assert np.array_equal(got, w[:n])


def test_values_under_capture(whole):
    import torch

    import pokerrust_b200 as P
    tables, roots, _ = whole
    n = 20
    d_in = torch.zeros((n, 1328), device="cuda")
    d_in[:, :1326] = torch.tensor(roots[3][0][:n])
    outs = []
    for captured in (False, True):
        b = _builder(P, n, roots)
        out = torch.zeros((n, 1328), device="cuda")
        b.regrets()  # device state is in place before the capture
        torch.cuda.synchronize()
        if captured:
            g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.graph(g, stream=s):
                b.evaluate_device(tables, 0, False, d_in.data_ptr(), out.data_ptr(), s.cuda_stream)
            g.replay()
        else:
            b.evaluate_device(tables, 0, False, d_in.data_ptr(), out.data_ptr())
        torch.cuda.synchronize()
        outs.append(out)
        b.close()
    assert torch.equal(*outs)
