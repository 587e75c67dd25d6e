"""Several decode steps in one launch (DecodeGraph): against the same steps one by one."""
import pytest
import torch

from tests.gpu_common import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,U,P,K,C,dtype,masked,mass_aware", [
    # a pair of warps per (batch, head): one pair, several pairs per warp (more than 13 an SM), two rows per lane
    (1, 1, 2, 64, 16, 128, torch.bfloat16, False, False),
    (125, 16, 2, 64, 16, 128, torch.float16, True, True),
    (3, 5, 2, 64, 16, 256, torch.bfloat16, True, False),
    # decoders ahead: rows of several 128-channel pieces, ragged rows, rows that are no multiple of four, K over 32
    (2, 3, 3, 8, 8, 256, torch.float32, False, True),
    (2, 3, 2, 32, 8, 36, torch.bfloat16, True, False),
    (3, 2, 2, 16, 4, 30, torch.float16, False, True),
    (1, 2, 2, 64, 40, 128, torch.float32, False, False),
    # more pairs than that kernel takes: one launch per step; sixteen pairs per block
    (160, 4, 3, 8, 8, 64, torch.float16, True, True),
    (160, 4, 2, 16, 4, 128, torch.float32, False, False),
])
def test_steps_in_one_launch_equal_single_steps(B, H, U, P, K, C, dtype, masked, mass_aware):
    ops()
    import ramnet_ops
    n, A = 5, P ** U
    g = torch.Generator(device="cuda").manual_seed(5)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)  # noqa: E731
    # peaked logits on few digits: the steps read and write the same slots again
    w, r = draw(n, B, H, U, P) * 3, draw(n, B, H, U, P) * 3
    w[..., :3] += 6
    r[..., :3] += 6
    x, gate = draw(n, B, H, C), draw(n, B, H, C)
    gamma = torch.sigmoid(torch.randn(n, B, H, generator=g, device="cuda")).to(dtype)
    slot = torch.randn(B, H, A, C, generator=g, device="cuda") * 0.1
    mass = torch.rand(B, H, A, generator=g, device="cuda")
    pos = torch.randint(0, 3 * A, (B,), generator=g, device="cuda", dtype=torch.int32)
    mask = torch.rand(B, generator=g, device="cuda") > 0.3 if masked else torch.empty(0, dtype=torch.bool, device="cuda")
    nw = torch.linspace(0.5, 1.5, C, device="cuda")
    E, rho = H // 2, 0.5

    e_slot, e_mass, e_pos, eager = slot.clone(), mass.clone(), pos.clone(), []
    for j in range(n):
        eager.append(torch.ops.ramnet_ops.decode_fused_(w[j], r[j], x[j], gamma[j], e_slot, e_mass, mask, E, e_pos, K, K, rho,
                                                        rho, mass_aware, 1e-12, nw, gate[j], 1e-6))
        e_pos += 1
    graph = ramnet_ops.DecodeGraph(w, r, x, gamma, slot, mass, pos, embed_num=E, top_k=K, w_re_norm=rho, r_re_norm=rho,
                                   mass_aware=mass_aware, mask=mask if masked else None, norm_weight=nw, gate_logits=gate)
    outs = graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(pos, e_pos)
    # float32 sums of the same terms: 2^-24 a rounding, some 2 K of them per row and step; the outputs rounded to their type
    tol = 2 * K * n * 2.0 ** -24
    half = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 0.0}[dtype]
    assert float((slot - e_slot).abs().max()) <= tol * float(e_slot.abs().max())
    assert float((mass - e_mass).abs().max()) <= tol * float(e_mass.abs().max())
    for a, b in zip(outs, eager):
        assert float((a.float() - b.float()).abs().max()) <= (8 * tol + half) * float(b.float().abs().max())
