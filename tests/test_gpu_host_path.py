"""The native host path of the public calls against the Python front end on the same inputs.

Both end in the same kernels, so results (and gradients) are equal bit for bit; calls the native path has to decline
(a broadcast shape, a tensor subclass, another time axis, a dispatch mode) still give the front end's result."""
import pytest
import torch

from tests.gpu_common import ops, randn

pytestmark = pytest.mark.gpu


def _args(B, T, H, U, P, K, C, dtype, state, mask, pos, scalar_gate=False):
    A = P ** U
    kw = dict(w_addr=randn((B, T, H, U, P), 1, dtype), r_addr=randn((B, T, H, U, P), 2, dtype), values=randn((B, T, H, C), 3, dtype),
              gamma=0.25 if scalar_gate else torch.sigmoid(randn((B, T, H), 4)).to(dtype), top_k=K, embed_num=H // 2)
    if state:
        kw["init_ram"] = (randn((B, H, A, C), 5), torch.rand(B, H, A, generator=torch.Generator().manual_seed(6)) + 0.1)
    if mask:
        kw["mask"] = torch.rand(B, T, generator=torch.Generator().manual_seed(7)) > 0.3
    if pos is not None:
        kw["position_ids"] = (torch.arange(T).view(1, T) * 3 + torch.arange(B if pos == "rows" else 1).view(-1, 1) + 5)
    move = lambda v: v.cuda() if isinstance(v, torch.Tensor) else tuple(t.cuda() for t in v) if isinstance(v, tuple) and isinstance(v[0], torch.Tensor) else v  # noqa: E731
    return {k: move(v) for k, v in kw.items()}


def _call(monkeypatch, native, kw, grads=False):
    import ramnet_ops
    from ramnet_ops import ram_attn
    kw = {k: (tuple(t.clone() for t in v) if k == "init_ram" else v.clone() if isinstance(v, torch.Tensor) else v) for k, v in kw.items()}
    leaves = []
    if grads:
        leaves = [kw[k] for k in ("w_addr", "r_addr", "values", "gamma") if isinstance(kw[k], torch.Tensor)] + list(kw.get("init_ram", ()))
        for t in leaves:
            t.requires_grad_(True)
    with monkeypatch.context() as m:
        m.setattr(ram_attn, "_native", lambda: native)
        y, (slot, mass) = ramnet_ops.random_access_memory_attention(**kw)
    out = [y, slot, mass]
    if grads:
        ups = [torch.full_like(y, 0.5), slot.detach() * 0.1, mass.detach() * 0.1] if grads == "all" else [torch.full_like(y, 0.5)]
        out += torch.autograd.grad(out[:len(ups)], leaves[:4 if grads == "y" and "init_ram" not in kw else None], ups)
    return [t.detach() for t in out]


@pytest.mark.parametrize("shape,dtype,opts", [
    ((3, 1, 4, 2, 64, 16, 128), torch.bfloat16, dict(state=True, mask=False, pos="rows")),
    ((3, 1, 4, 2, 64, 16, 128), torch.bfloat16, dict(state=False, mask=True, pos=None)),
    ((2, 1, 3, 3, 8, 8, 64), torch.float16, dict(state=True, mask=True, pos="one", scalar_gate=True)),
    ((1, 1, 2, 2, 6, (3, 5), 10), torch.float32, dict(state=True, mask=False, pos=None)),
    ((2, 70, 4, 2, 16, 4, 64), torch.float32, dict(state=False, mask=False, pos=None)),
    ((2, 70, 4, 2, 64, 16, 128), torch.bfloat16, dict(state=True, mask=True, pos="rows")),
    ((1, 33, 2, 3, 4, (8, 3), 7), torch.float16, dict(state=False, mask=True, pos="one")),
    ((1, 33, 2, 3, 32, 8, 16), torch.bfloat16, dict(state=False, mask=False, pos="rows", scalar_gate=True)),  # state in global memory
])
def test_same_bits_as_the_front_end(monkeypatch, shape, dtype, opts):
    ops()
    kw = _args(*shape, dtype, **opts)
    kw["top_k_re_norm"] = (0.5, 0.25)
    for inplace in (False, True) if opts["state"] else (False,):
        kw["inplace"] = kw["mass_aware"] = inplace
        for a, b in zip(_call(monkeypatch, True, kw), _call(monkeypatch, False, kw)):
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


@pytest.mark.parametrize("shape,dtype,opts,grads", [
    ((2, 70, 4, 2, 16, 4, 64), torch.float32, dict(state=True, mask=True, pos="rows"), "all"),
    ((2, 70, 4, 2, 64, 16, 128), torch.bfloat16, dict(state=False, mask=False, pos=None), "y"),
    ((1, 1, 2, 2, 16, 4, 8), torch.float32, dict(state=True, mask=False, pos=None), "all"),
    ((1, 40, 2, 2, 16, 4, 8), torch.float16, dict(state=True, mask=False, pos="one"), "all"),
])
def test_same_gradients_as_the_front_end(monkeypatch, shape, dtype, opts, grads):
    ops()
    kw = _args(*shape, dtype, **opts)
    for a, b in zip(_call(monkeypatch, True, kw, grads), _call(monkeypatch, False, kw, grads)):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


def test_declined_calls_and_addresses(monkeypatch):
    C_ = ops()
    import ramnet_ops
    from torch.utils._python_dispatch import TorchDispatchMode
    kw = _args(2, 40, 4, 2, 16, 4, 64, torch.float32, True, False, "rows")
    want = _call(monkeypatch, False, kw)
    one = dict(kw, r_addr=kw["r_addr"][:1].clone())       # broadcast over the batch
    for a, b in zip(_call(monkeypatch, True, dict(one, r_addr=one["r_addr"])), _call(monkeypatch, False, one)):
        assert torch.equal(a, b)
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Watch():
        got = _call(monkeypatch, True, kw)
    assert any("ramnet_ops" in name for name in seen)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    names = ("w_addr", "r_addr", "values", "gamma", "init_ram", "mask", "embed_num", "position_ids", "top_k", "top_k_re_norm",
             "mass_aware", "eps", "t_dim", "inplace", "impl_backend")
    full = dict(dict(mask=None, top_k_re_norm=0.0, mass_aware=False, eps=1e-12, t_dim=1, inplace=False, impl_backend=None), **kw)
    args = [full[n] for n in names]
    assert C_.host.attention(*args) is not None
    for name, bad in (("t_dim", 0), ("eps", 0.0), ("embed_num", 9), ("top_k", 0), ("top_k", "4"), ("top_k_re_norm", 1.5),
                      ("impl_backend", "torch"), ("values", kw["values"].half()), ("init_ram", (None, 0.5)), ("w_addr", kw["w_addr"].cpu())):
        assert C_.host.attention(*[bad if n == name else v for n, v in zip(names, args)]) is None, name

    addr = randn((2, 40, 4, 3, 8), 9, torch.bfloat16).cuda().permute(0, 2, 3, 4, 1)
    pos = (torch.arange(40).view(1, 40) + torch.arange(2).view(2, 1) * 100).cuda()
    outs = []
    for native in (True, False):
        with monkeypatch.context() as m:
            m.setattr(ramnet_ops.ram_attn, "_native", lambda native=native: native)
            outs.append(ramnet_ops.topk_addr(addr, 2, pos, 8, 0.5, True, False))
    assert all(torch.equal(a, b) and a.stride() == b.stride() for a, b in zip(*outs))
