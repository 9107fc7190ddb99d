"""Device memory that passes over few roots take for themselves: one bounded pool per device, whatever
the number of builders, given back with the last of them; and none of it stands in the way of a stream
that is being captured elsewhere."""
import pytest

pytestmark = pytest.mark.gpu

FLOP = (1 << 9) | (1 << 18) | (1 << 50)
TURNS = [c for c in range(52) if not FLOP >> c & 1]


def _builder(P, n):
    b = P.Builder()
    for i in range(n):
        b.add(FLOP | (1 << TURNS[i % len(TURNS)]), 2.0 + i)
    b.regrets()  # device state is in place
    return b


def test_many_builders_hold_one_pool():
    import torch

    import pokerrust_b200 as P
    tables = P.build_flop_tables(FLOP)
    n = 70
    builders = [_builder(P, n) for _ in range(8)]
    d_in = torch.rand((n, 1328), device="cuda")
    d_out = torch.zeros((n, 1328), device="cuda")

    def held():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    free = held()
    for b in builders:
        b.evaluate_device(tables, 0, False, d_in.data_ptr(), d_out.data_ptr())
    used = free - held()
    assert all(b.splits > 1 for b in builders)
    # the pool keeps 256 MB at most (64 MB to spare for the kernels, loaded on first use)
    assert used <= 320 << 20, used >> 20
    for b in builders:
        b.close()
    assert held() >= free
    P.free_eval(tables)


def test_first_pass_beside_a_capture():
    """The pass that makes the pool, on one stream while another is being captured."""
    import torch

    import pokerrust_b200 as P
    tables = P.build_flop_tables(FLOP)
    n = 3
    d_in = torch.rand((n, 1328), device="cuda")
    d_out = [torch.zeros((n, 1328), device="cuda") for _ in range(2)]
    x = torch.ones(4, device="cuda")
    side = torch.cuda.Stream()
    for k in range(2):
        b = _builder(P, n)
        torch.cuda.synchronize()
        if k == 0:
            b.evaluate_device(tables, 0, False, d_in.data_ptr(), d_out[k].data_ptr(), side.cuda_stream)
        else:
            g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.graph(g, stream=s):
                y = x + 1
                b.evaluate_device(tables, 0, False, d_in.data_ptr(), d_out[k].data_ptr(), side.cuda_stream)
            g.replay()
            torch.cuda.synchronize()
            assert (y == 2).all()
        torch.cuda.synchronize()
        b.close()  # and with it the pool
    assert torch.equal(*d_out)
    P.free_eval(tables)
