"""Backward pass: the replay over event lists (rn_bwd_lists.cu, rn_apply.cu), which runs where the heads fill the chip, against
the sweep that runs for a few heads (checked against the oracle's autograd elsewhere): the same problem in one call and head
by head."""
import pytest
import torch

from tests.gpu_common import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,A,T,C,K,pool,dtype,masked,ma", [
    (160, 256, 129, 36, (4, 6), 256, torch.float32, False, False),   # one owner, a block and one token, partial channel group
    (40, 2048, 127, 64, (8, 8), 2048, torch.bfloat16, True, False),  # two owners
    (24, 4096, 257, 64, (16, 16), 4096, torch.bfloat16, True, True),  # four
    (40, 4096, 140, 32, (16, 16), 24, torch.float32, True, True),    # 24 hot slots: steps cut short
    (40, 4096, 70, 32, (16, 16), 40, torch.float32, False, False),   # 40 slots
    (20, 9000, 50, 32, (12, 12), 9000, torch.float32, False, False),  # eight owners
    (40, 4096, 70, 32, (32, 5), 4096, torch.float16, False, False),  # four addresses a thread
    (160, 37, 40, 4, (5, 2), 37, torch.float32, True, False),        # slots not a power of two, four channels
])
def test_replay_over_lists_equals_the_sweep(heads, A, T, C, K, pool, dtype, masked, ma):
    ops()
    KT, eps = K[0] + K[1], 1e-6
    g = torch.Generator().manual_seed(A + T)
    slots = torch.randperm(A, generator=g)[:pool]
    idx = slots[torch.randint(pool, (1, T, heads, KT), generator=g)].to(torch.int32).cuda()
    val = torch.rand(1, T, heads, KT, generator=g).cuda() * 0.4 + 0.01
    val[:, ::5, :, 1] = 0.0
    val[:, ::3, :, K[0]] = 0.0
    x = torch.randn(1, T, heads, C, generator=g).to(dtype).cuda()
    gamma = (torch.randn(1, heads, T, generator=g) * 0.5).to(dtype).cuda()
    slot, mass = torch.randn(1, heads, A, C, generator=g).cuda(), (torch.rand(1, heads, A, generator=g) + 0.05).cuda()
    mask = (torch.rand(1, T, generator=g) > 0.2).cuda() if masked else None
    d_y = torch.randn(1, T, heads, C, generator=g).to(dtype).cuda()
    d_slot, d_mass = torch.randn(1, heads, A, C, generator=g).cuda() * 0.1, torch.randn(1, heads, A, generator=g).cuda() * 0.1

    def run(h):
        return torch.ops.ramnet_ops.gsu_backward(
            idx[:, :, h].permute(0, 2, 3, 1), val[:, :, h].permute(0, 2, 3, 1), x[:, :, h].transpose(1, 2), gamma[:, h],
            slot[:, h].contiguous(), mass[:, h].contiguous(), mask, d_y[:, :, h].transpose(1, 2),
            d_slot[:, h].contiguous(), d_mass[:, h].contiguous(), K[0], K[1], ma, eps)

    whole = run(slice(0, heads))
    # float32 sums in another order: some C terms a dot product, T * K / pool updates of a row; x and gamma gradients rounded to their type
    hits = max(8, 3 * T * KT // min(pool, T * KT))
    tol = (C + 16 * hits) * 2.0 ** -23
    half = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    for h in range(0, heads, max(1, heads // 4)):
        for name, a, b in zip(("d_val", "d_x", "d_gamma", "d_slot", "d_mass"), whole, run(slice(h, h + 1))):
            a = a[:, h:h + 1].double()
            assert a.shape == b.shape, name
            limit = tol + (half if name == "d_x" else 0.0)
            assert float((a - b.double()).norm()) <= limit * float(b.double().norm()), name
