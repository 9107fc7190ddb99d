"""Passes over few river roots spread each root's river cards over several CTAs (launch_river): the
regrets and average sums they leave have the bits of the one-CTA pass, which runs when the same roots
are part of a larger set, and the values differ by the rounding of sums over 48 river cards (at most
48 half-ulps of the largest partial sum; 1e-5 of the largest value in single precision, 1e-13 in
double)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLOP = 0b111


def _roots(n, seed):
    rng = np.random.default_rng(seed)
    turns = rng.integers(3, 52, n)
    boards = [FLOP | (1 << int(t)) for t in turns]
    bets = rng.integers(1, 20, n).astype(np.float32)
    reg = np.maximum(rng.random((n, 26, 256), dtype=np.float32) * 100 - 30, 0)
    ranges = rng.random((2, n, 1326), dtype=np.float32)
    return boards, bets, reg, ranges


def _builder(P, boards, bets, reg, average):
    b = P.Builder()
    for c, x in zip(boards, bets):
        b.add(c, float(x))
    if average:
        b.enable_average()
    b.set_regrets(reg)
    return b


def _passes(P, tables, n, boards, bets, reg, ranges, average):
    """Values of a CFR pass per player, a best response, regrets and average sums."""
    b = _builder(P, boards[:n], bets[:n], reg[:n], average)
    out = []
    for p in range(2):
        if average:
            b.upload_own_all(ranges[1 - p][:n])
        b.upload_all(ranges[p][:n])
        b.evaluate(tables, p)
        out.append(b.download_all())
    b.upload_all(ranges[0][:n])
    b.evaluate(tables, 0, True)
    out.append(b.download_all())
    br64 = b.best_response_f64(tables, 1, ranges[1][:n].astype(np.float64))
    res = out, br64, b.regrets(), b.average_sums() if average else None
    b.close()
    return res


@pytest.fixture(scope="module")
def whole():
    """The passes over 260 roots: more than are ever split."""
    import pokerrust_b200 as P
    tables = P.build_flop_tables(FLOP)
    roots = _roots(260, 5)
    got = {avg: _passes(P, tables, 260, *roots, avg) for avg in (False, True)}
    yield tables, roots, got
    P.free_eval(tables)


@pytest.mark.parametrize("n,average", [(1, False), (1, True), (3, False), (4, True), (13, False), (25, False),
                                       (49, False), (74, True), (75, False), (148, False), (149, True), (240, False)])
def test_split_pass_has_the_whole_pass_bits(whole, n, average):
    import pokerrust_b200 as P
    tables, roots, got = whole
    out, br64, reg, avg = _passes(P, tables, n, *roots, average)
    w_out, w_br64, w_reg, w_avg = got[average]
    assert np.array_equal(reg, w_reg[:n])
    if average:
        assert np.array_equal(avg, w_avg[:n])
    for a, b in zip(out, w_out):
        assert np.abs(a - b[:n]).max() <= 1e-5 * np.abs(b[:n]).max()
    assert np.abs(br64 - w_br64[:n]).max() <= 1e-13 * np.abs(w_br64[:n]).max()


def test_split_passes_on_two_streams(whole):
    """Best responses of one builder queued on two streams at once do not share scratch."""
    import torch

    import pokerrust_b200 as P
    tables, (boards, bets, reg, ranges), _ = whole
    n = 20
    b = _builder(P, boards[:n], bets[:n], reg[:n], False)
    d_in = [torch.zeros((n, 1328), device="cuda") for _ in range(2)]
    for p in range(2):
        d_in[p][:, :1326] = torch.tensor(ranges[p][:n])
    one = [torch.zeros((n, 1328), device="cuda") for _ in range(2)]
    for p in range(2):
        b.evaluate_device(tables, p, True, d_in[p].data_ptr(), one[p].data_ptr())
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    many = [[torch.zeros((n, 1328), device="cuda") for _ in range(10)] for _ in range(2)]
    torch.cuda.synchronize()
    for i in range(10):
        for p in range(2):
            b.evaluate_device(tables, p, True, d_in[p].data_ptr(), many[p][i].data_ptr(), streams[p].cuda_stream)
    torch.cuda.synchronize()
    for p in range(2):
        for t in many[p]:
            assert torch.equal(t, one[p])
    b.close()


def test_split_pass_under_capture(whole):
    """A pass recorded into a caller's CUDA graph takes no memory of its own and gives the same bits."""
    import torch

    import pokerrust_b200 as P
    tables, (boards, bets, reg, ranges), got = whole
    n = 3
    b = _builder(P, boards[:n], bets[:n], reg[:n], False)
    d_in = torch.zeros((n, 1328), device="cuda")
    d_in[:, :1326] = torch.tensor(ranges[0][:n])
    out = torch.zeros((n, 1328), device="cuda")
    b.regrets()  # device state is in place before the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        b.evaluate_device(tables, 0, False, d_in.data_ptr(), out.data_ptr(), s.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    want = got[False][0][0][:n]
    assert np.abs(out.cpu().numpy()[:, :1326] - want).max() <= 1e-5 * np.abs(want).max()
    b.close()
