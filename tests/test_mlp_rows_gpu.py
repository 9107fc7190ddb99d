"""pr_mlp_forward over few samples runs only the 128-row tiles that hold them, with narrower column
tiles the fewer there are, and writes the output from the last layer's epilogue. Every output value
sums over the same terms in the same order whatever the tile, so it has the bits of the same sample in
a full batch. Counts at the edges of the row tiles and of the tile widths' ranges; inputs and outputs
that start on 4-byte addresses only; nothing is written past the last sample."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 3072


def test_few_rows_have_the_bits_of_a_full_batch():
    import torch
    import pokerrust_b200 as P
    net = P.ValueNet(rows=ROWS, seed=6)
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    ranges = torch.rand((ROWS, 2, 1326), generator=g, device="cuda") / 600.0
    boards = torch.full((ROWS,), 0b1111 << 20, dtype=torch.int64, device="cuda")
    scalars = torch.rand((ROWS, 2), generator=g, device="cuda")
    want = torch.zeros((ROWS, 2652), device="cuda")
    net.forward(ranges, boards, scalars, want)
    for count in (1, 127, 128, 129, 384, 385, 768, 769, 1152, 1153, 2304, 2305, ROWS):
        out = torch.full((count + 1, 2652), 9.0, device="cuda")
        net.forward(ranges[:count], boards[:count], scalars[:count], out[:count])
        assert torch.equal(out[:count], want[:count]), count
        assert (out[count] == 9.0).all(), count
    count = 130
    flat_in = torch.zeros(count * 2652 + 1, device="cuda")
    flat_in[1:] = ranges[:count].reshape(-1)
    flat_out = torch.full((count * 2652 + 2,), 9.0, device="cuda")
    out = flat_out[1:-1].reshape(count, 2652)
    net.forward(flat_in[1:].reshape(count, 2, 1326), boards[:count], scalars[:count], out)
    assert torch.equal(out, want[:count])
    assert flat_out[0] == 9.0 and flat_out[-1] == 9.0
    net.close()
