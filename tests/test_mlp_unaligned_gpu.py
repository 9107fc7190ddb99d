"""pr_mlp_train_step on inputs and targets that start on 4-byte addresses only (read one by one, not as
quads): the loss, every gradient and every updated weight have the bits of the aligned step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 130, 256])
def test_unaligned_step_has_the_aligned_bits(count):
    import torch

    import pokerrust_b200 as P
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    ranges = torch.rand((count, 2, 1326), generator=g, device="cuda") / 600.0
    targets = torch.rand((count, 2652), generator=g, device="cuda") - 0.5
    boards = torch.full((count,), 0b1111 << 20, dtype=torch.int64, device="cuda")
    scalars = torch.rand((count, 2), generator=g, device="cuda")
    got = []
    for off in (0, 1):
        flat_r, flat_t = (torch.zeros(count * 2652 + 1, device="cuda") for _ in range(2))
        r = flat_r[off:off + count * 2652].view(count, 2, 1326).copy_(ranges)
        t = flat_t[off:off + count * 2652].view(count, 2652).copy_(targets)
        assert r.data_ptr() % 16 == t.data_ptr() % 16 == 4 * off
        net = P.ValueNet(rows=256, seed=9)
        loss = net.train_step(r, boards, scalars, t, lr=1e-3)
        got.append((loss, [net.grad(l) for l in range(5)], [net.layer(l) for l in range(5)]))
        net.close()
    assert got[0][0] == got[1][0]
    for which in (1, 2):
        for a, b in zip(got[0][which], got[1][which]):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))
