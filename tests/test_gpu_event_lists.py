"""The event-list prefill kernels (rn_lists.cu, rn_apply.cu) against a token-by-token fp32 reference.

Addresses are given directly, so that blocks can be driven to their edges: one token more or less than a block, slots hit
by every token (lists that do not fit are cut into shorter steps), the same slot several times in one token, numbers of
slots that give one, two, four and eight owners, a partial channel group, dead events and masked tokens."""
import pytest
import torch

from tests.gpu_common import ops

pytestmark = pytest.mark.gpu


def _reference(idx, val, x, gamma, slot, mass, mask, Kw, mass_aware, eps):
    """idx / val (B,H,K,T), x (B,H,T,C), gamma (B,H,T); float64 state, writes of a token in order, then its reads."""
    B, H, K, T = idx.shape
    slot, mass, y = slot.double(), mass.double(), torch.zeros_like(x, dtype=torch.float64)
    rows = torch.arange(B)[:, None], torch.arange(H)[None, :]
    for t in range(T):
        live = torch.ones(B, H, dtype=torch.bool) if mask is None else mask[:, t, None].expand(B, H)
        g = gamma[..., t].double()
        for k in range(Kw):
            a, w = idx[:, :, k, t].long(), val[:, :, k, t].double().abs()
            on = live & (w != 0)
            m = mass[rows[0], rows[1], a]
            alpha = (1 - w) / ((1 - w) + g.exp() * w)
            m1 = torch.where(on, alpha * m + w, m)
            gain = torch.where(on, w / (m1 + eps), torch.zeros_like(w))
            s = slot[rows[0], rows[1], a]
            slot[rows[0], rows[1], a] = s + gain[..., None] * (x[:, :, t].double() - s)
            mass[rows[0], rows[1], a] = m1
        r = val[:, :, Kw:, t].double().abs() * live[..., None]
        a = idx[:, :, Kw:, t].long()
        if mass_aware:
            u = r * mass[rows[0][..., None], rows[1][..., None], a]
            r = u * r.sum(-1, keepdim=True) / (u.sum(-1, keepdim=True) + eps)
        y[:, :, t] = (r[..., None] * slot[rows[0][..., None], rows[1][..., None], a]).sum(2)
    return y, slot, mass


@pytest.mark.parametrize("A,T,C,K,pool,dtype,masked,ma", [
    (256, 129, 36, (4, 6), 256, torch.float32, False, False),     # one owner, a block and one token, partial channel group
    (2048, 127, 16, (16, 3), 2048, torch.bfloat16, True, False),  # two owners would do at 16 channels
    (4096, 257, 64, (16, 16), 4096, torch.bfloat16, False, True),
    (4096, 200, 32, (16, 16), 24, torch.float32, True, True),     # 24 hot slots: steps cut short
    (4096, 140, 32, (16, 16), 3, torch.float32, False, False),    # three slots, every one several times in a token
    (16384, 70, 32, (12, 12), 16384, torch.float32, False, False),  # eight owners
    (16384, 40, 8, (128, 128), 2, torch.float32, True, True),     # 128 writes of a token on two slots
    (37, 140, 4, (5, 2), 37, torch.float16, False, False),        # slots not a power of two
])
def test_event_lists_match_a_sequential_reference(A, T, C, K, pool, dtype, masked, ma):
    ops()
    B, H, KT, eps = 2, 2, K[0] + K[1], 1e-6
    g = torch.Generator().manual_seed(A + T)
    slots = torch.randperm(A, generator=g)[:pool]
    idx = slots[torch.randint(pool, (B, T, H, KT), generator=g)].to(torch.int32).permute(0, 2, 3, 1)
    val = (torch.rand(B, T, H, KT, generator=g) * 0.4 + 0.01).permute(0, 2, 3, 1).contiguous()
    val[:, :, 1, ::5] = 0.0
    val[:, :, K[0]:] *= -1
    x = torch.randn(B, H, T, C, generator=g).to(dtype)
    gamma = (torch.randn(B, H, T, generator=g) * 0.5).to(dtype)
    slot, mass = torch.randn(B, H, A, C, generator=g), torch.rand(B, H, A, generator=g) + 0.05
    mask = torch.rand(B, T, generator=g) > 0.2 if masked else None
    val = val.permute(0, 3, 1, 2).contiguous().permute(0, 2, 3, 1)  # token-major, as the decode leaves it
    idx = idx.permute(0, 3, 1, 2).contiguous().permute(0, 2, 3, 1)
    y, s, m = torch.ops.ramnet_ops.gsu_forward(idx.cuda(), val.cuda(), x.cuda(), gamma.cuda(), slot.cuda(), mass.cuda(),
                                               None if mask is None else mask.cuda(), K[0], K[1], ma, eps)
    ry, rs, rm = _reference(idx, val, x.float(), gamma.float(), slot.clone(), mass.clone(), mask, K[0], ma, eps)
    # A row goes through at most T * Kw updates of three roundings each, all of them convex combinations, so its relative
    # error stays below T * Kw * 3 ulp; hot slots take the largest number
    hits = max(8, T * K[0] * 3 // min(pool, T * K[0]))
    tol = hits * 3 * 2.0 ** -24
    assert float((s.cpu().double() - rs).abs().max()) <= 8 * tol * float(rs.abs().max())
    assert float((m.cpu().double() - rm).abs().max()) <= 8 * tol * float(rm.abs().max())
    out = {torch.float32: 64 * tol, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10}[dtype]
    assert float((y.cpu().double() - ry).norm() / ry.norm()) <= out


@pytest.mark.parametrize("T", [1, 40, 129])
def test_in_place_moves_touched_rows_only_and_leaves_the_others(T):
    """Few events on a large state updated in place: the same results as the copying form, untouched rows bit for bit."""
    ops()
    B, H, A, C, K = 2, 3, 4096, 64, 6
    g = torch.Generator().manual_seed(T)
    idx = torch.randint(A, (B, T, H, 2 * K), generator=g).to(torch.int32).permute(0, 2, 3, 1).cuda()
    val = (torch.rand(B, T, H, 2 * K, generator=g) * 0.4 + 0.01).permute(0, 2, 3, 1).cuda()
    x, gamma = torch.randn(B, H, T, C, generator=g).cuda(), torch.randn(B, H, T, generator=g).cuda()
    slot, mass = torch.randn(B, H, A, C, generator=g).cuda(), (torch.rand(B, H, A, generator=g) + 0.1).cuda()
    for ma in (False, True):
        want = torch.ops.ramnet_ops.gsu_forward(idx, val, x, gamma, slot, mass, None, K, K, ma, 1e-6)
        s, m = slot.clone(), mass.clone()
        y = torch.ops.ramnet_ops.gsu_forward_(idx, val, x, gamma, s, m, None, K, K, ma, 1e-6)
        assert torch.equal(y, want[0]) and torch.equal(s, want[1]) and torch.equal(m, want[2])
