"""Gradients of the output in the layouts autograd makes them (slices of a concatenation, misaligned starts, expanded sums,
permuted), and expanded keys and values: the gradients of the contiguous copies, on the tcgen05 kernels."""
import pytest
import torch

import fa_b200_capi as capi

pytestmark = pytest.mark.gpu


def _douts(out):
    """(name, function of the output whose gradient has that layout, the same gradient written out)"""
    b, s, h, d = out.shape
    wide = [torch.randn(b, s, n + h * d + m, device="cuda").to(out.dtype) for n, m in ((0, 1), (0, 4), (4, 0), (1, 0), (8, 0))]
    for (n, m), w in zip(((0, 1), (0, 4), (4, 0), (1, 0), (8, 0)), wide):
        x, y = (torch.randn(b, s, c, device="cuda").to(out.dtype) for c in (n, m))
        yield f"cat{n}-{m}", (lambda o, x=x, y=y, w=w: (torch.cat([x, o.flatten(-2), y], -1) * w).sum()), w[..., n:n + h * d].unflatten(-1, (h, d))
    w = torch.randn(b, h, d, device="cuda").to(out.dtype)
    yield "sum over tokens", lambda o: (o.sum(1) * w).sum(), w[:, None].expand(b, s, h, d)
    w2 = torch.randn(b, s, d, device="cuda").to(out.dtype)
    yield "sum over heads", lambda o: (o.sum(2) * w2).sum(), w2[:, :, None].expand(b, s, h, d)
    w3 = torch.randn(h, b, s, d, device="cuda").to(out.dtype)
    yield "permuted", lambda o: (o.permute(2, 0, 1, 3) * w3).sum(), w3.permute(1, 2, 0, 3)


@pytest.mark.parametrize("route", ["direct", "op"])
@pytest.mark.parametrize("version,packed", [(2, False), (2, True), (3, False), (3, True)])
@pytest.mark.parametrize("d", [32, 64, 72, 96, 128, 136, 256])
def test_output_gradients_in_any_layout(d, version, packed, route, monkeypatch):
    import flash_attn_npu as fa2
    import flash_attn_npu_3 as fa3
    from flash_attn_npu import flash_attn_npu_interface as i2
    from flash_attn_npu_3 import flash_attn_npu_interface as i3
    fa = fa2 if version == 2 else fa3
    if route == "op":
        for m in (i2, i3):
            monkeypatch.setattr(m, "_plain", lambda *t: False)
    b, s, h = 2, 131, 3
    x = [torch.randn(b, s, h, d, device="cuda").bfloat16().requires_grad_(True) for _ in range(3)]
    cu = torch.tensor([0, s, 2 * s], dtype=torch.int32, device="cuda")

    def forward():
        if packed:
            return fa.flash_attn_varlen_func(*[t.flatten(0, 1) for t in x], cu, cu, s, s, causal=True).unflatten(0, (b, s))
        return fa.flash_attn_func(*x, causal=True)

    for name, f, dout in _douts(forward()):
        got = torch.autograd.grad(f(forward()), x)
        kernel = capi.last_kernel()
        want = torch.autograd.grad(forward(), x, dout.contiguous())
        torch.cuda.synchronize()
        assert kernel.startswith("sm100"), (name, kernel)
        assert all(torch.equal(a, w) for a, w in zip(got, want)), name
    assert capi.lib.fa_debug_get(2) == 0


@pytest.mark.parametrize("d", [96, 128])
def test_expanded_keys_and_values(d):
    from flash_attn_npu import flash_attn_npu as ext
    b, s, h = 2, 200, 4
    q, dout = (torch.randn(b, s, h, d, device="cuda").half() for _ in range(2))
    k, v = (torch.randn(b, s, 1, d, device="cuda").half().expand(b, s, h, d) for _ in range(2))
    out, lse, _, _ = ext.fwd(q, k.contiguous(), v.contiguous(), None, None, 0.0, d ** -0.5, True, -1, -1, 0.0, False, None)

    def run(k, v):
        g = ext.bwd(dout, q, k, v, out, lse, None, None, None, None, 0.0, d ** -0.5, True, -1, -1, 0.0, False, None, None)[:3]
        torch.cuda.synchronize()
        assert capi.last_kernel().startswith("sm100")
        return g

    assert all(torch.equal(x, y) for x, y in zip(run(k, v), run(k.contiguous(), v.contiguous())))
