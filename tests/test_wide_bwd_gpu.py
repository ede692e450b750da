"""Backward at head dims above 128 on the tcgen05 kernels: edges of the 128-row tiles, padded head dims, groups, windows,
packed sequences, several launches; against the float64 oracle, larger shapes against the general kernels."""
import pytest
import torch

from oracle import attention_oracle as orc
from parity import assert_within

pytestmark = pytest.mark.gpu

# (dtype, B, H, Hkv, Sq, Sk, D, causal, wl, wr, softcap)
CASES = [
    (torch.bfloat16, 2, 2, 2, 128, 128, 256, False, -1, -1, 0.0),
    (torch.float16, 1, 4, 2, 129, 127, 192, True, -1, -1, 0.0),
    (torch.bfloat16, 1, 6, 2, 1, 300, 136, True, -1, -1, 0.0),
    (torch.float16, 1, 2, 1, 300, 1, 256, False, -1, -1, 0.0),
    (torch.bfloat16, 1, 2, 2, 700, 513, 248, True, -1, -1, 0.0),
    (torch.bfloat16, 1, 4, 1, 520, 520, 256, True, 100, 0, 0.0),
    (torch.float16, 2, 2, 2, 260, 300, 160, False, 40, 70, 0.0),
    (torch.bfloat16, 1, 2, 1, 300, 300, 200, True, -1, -1, 5.0),
]


def _grads(q, k, v, do, scale, causal, window, cap, slopes=None):
    import fa_b200_capi as capi
    from flash_attn_npu import flash_attn_npu as ext
    out, lse, _, _ = ext.fwd(q, k, v, None, slopes, 0.0, scale, causal, *window, cap, False, None)
    g = [torch.full_like(t, 777.0) for t in (q, k, v)]
    ext.bwd(do, q, k, v, out, lse, *g, slopes, 0.0, scale, causal, *window, cap, False, None, None)
    torch.cuda.synchronize()
    assert capi.lib.fa_debug_get(2) == 0
    return g, capi.last_kernel()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(x).replace("torch.", "") for x in c))
def test_wide_backward_against_the_oracle(case):
    dt, b, h, hkv, sq, sk, d, causal, wl, wr, cap = case
    q, do = ((torch.rand(b, sq, h, d) * 2 - 1).to(dt) for _ in range(2))
    k, v = ((torch.rand(b, sk, hkv, d) * 2 - 1).to(dt) for _ in range(2))
    scale = d ** -0.5
    _, lse = orc.attention_fwd(q.float(), k.float(), v.float(), scale, causal, (wl, wr), cap, data_type=torch.float32)
    lp = orc.attention_bwd(q, k, v, do, lse, scale, causal, (wl, wr), cap)
    f32 = orc.attention_bwd(q.float(), k.float(), v.float(), do.float(), lse, scale, causal, (wl, wr), cap)
    got, name = _grads(q.cuda(), k.cuda(), v.cuda(), do.cuda(), scale, causal, (wl, wr), cap)
    assert name == "sm100_wide_tcgen05_bwd"
    for n, g, a, r in zip(("dq", "dk", "dv"), got, lp, f32):
        assert_within(n, g.cpu(), a, r, roundings=3)


@pytest.mark.parametrize("d", [192, 256])
def test_wide_packed_backward_against_the_oracle(d):
    import fa_b200_capi as capi
    from flash_attn_npu import flash_attn_npu as ext
    lq, lk, h, hkv, dt = [300, 0, 129, 64], [260, 70, 400, 1], 4, 2, torch.bfloat16
    q, do = (torch.randn(sum(lq), h, d).to(dt) for _ in range(2))
    k, v = (torch.randn(sum(lk), hkv, d).to(dt) for _ in range(2))
    cu = [torch.tensor([0] + torch.tensor(x).cumsum(0).tolist(), dtype=torch.int32) for x in (lq, lk)]
    scale = d ** -0.5
    _, lse32 = orc.attention_varlen_fwd(q.float(), k.float(), v.float(), *cu, scale, True, data_type=torch.float32)
    lp = orc.attention_varlen_bwd(q, k, v, do, lse32, *cu, scale, True)
    f32 = orc.attention_varlen_bwd(q.float(), k.float(), v.float(), do.float(), lse32, *cu, scale, True)
    qg, kg, vg, dog, cq, ck = (t.cuda() for t in (q, k, v, do, *cu))
    out, lse, _, _ = ext.varlen_fwd(qg, kg, vg, None, cq, ck, None, None, None, None, max(lq), max(lk), 0.0, scale, False, True,
                                    -1, -1, 0.0, False, None)
    g = [torch.full_like(t, 777.0) for t in (qg, kg, vg)]
    ext.varlen_bwd(dog, qg, kg, vg, out, lse, *g, cq, ck, None, max(lq), max(lk), 0.0, scale, False, True, -1, -1, 0.0, False,
                   None, None)
    torch.cuda.synchronize()
    assert capi.last_kernel() == "sm100_wide_tcgen05_bwd" and capi.lib.fa_debug_get(2) == 0
    for n, x, a, r in zip(("dq", "dk", "dv"), g, lp, f32):
        assert_within(n, x.cpu(), a, r, roundings=3)


@pytest.mark.parametrize("b,sq,sk,h,hkv,causal", [(9, 1024, 1100, 8, 8, True), (2, 2048, 2048, 8, 2, True), (3, 1000, 900, 6, 3, False)])
def test_wide_backward_over_several_launches(b, sq, sk, h, hkv, causal):
    """More KV heads than one launch's tiles hold, long walks: against the general kernels.  Both round P, dS and the
    result to the input type once and sum in fp32, in another order: three half-ulp roundings of the largest value."""
    import fa_b200_capi as capi
    dt, d = torch.bfloat16, 256
    q, do = (torch.randn(b, sq, h, d, device="cuda", dtype=dt) for _ in range(2))
    k, v = (torch.randn(b, sk, hkv, d, device="cuda", dtype=dt) for _ in range(2))
    slopes = torch.rand(h, device="cuda") * 0.2
    got, name = _grads(q, k, v, do, 0.07, causal, (-1, -1), 0.0, slopes)
    assert name == "sm100_wide_tcgen05_bwd"
    again, _ = _grads(q, k, v, do, 0.07, causal, (-1, -1), 0.0, slopes)
    capi.lib.fa_set_kernel_policy(1)
    try:
        ref, name = _grads(q, k, v, do, 0.07, causal, (-1, -1), 0.0, slopes)
        assert name == "generic_mma_bwd"
    finally:
        capi.lib.fa_set_kernel_policy(0)
    for n, x, y, r in zip(("dq", "dk", "dv"), got, again, ref):
        assert torch.equal(x, y), n
        assert (x.float() - r.float()).abs().max().item() <= 3 * 2.0 ** -8 * r.float().abs().max().item(), n


@pytest.mark.parametrize("packed", [False, True])
def test_wide_backward_without_room_for_the_tiles(packed, monkeypatch):
    """The allocator refuses the workspace with the tiles: the call runs on the least one, with the general kernels' bits."""
    import fa_b200_capi as capi
    from flash_attn_npu import flash_attn_npu as ext
    s, h, hkv, d = 600, 4, 2, 256
    shape = (lambda n: (2 * s, n, d)) if packed else (lambda n: (2, s, n, d))
    q, do = (torch.randn(*shape(h), device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(*shape(hkv), device="cuda").bfloat16() for _ in range(2))
    cu = torch.tensor([0, s, 2 * s], dtype=torch.int32, device="cuda")
    if packed:
        out, lse, _, _ = ext.varlen_fwd(q, k, v, None, cu, cu, None, None, None, None, s, s, 0.0, 0.1, False, True, -1, -1, 0.0, False, None)
    else:
        out, lse, _, _ = ext.fwd(q, k, v, None, None, 0.0, 0.1, True, -1, -1, 0.0, False, None)

    def run():
        if packed:
            g = ext.varlen_bwd(do, q, k, v, out, lse, None, None, None, cu, cu, None, s, s, 0.0, 0.1, False, True, -1, -1, 0.0, False, None, None)
        else:
            g = ext.bwd(do, q, k, v, out, lse, None, None, None, None, 0.0, 0.1, True, -1, -1, 0.0, False, None, None)
        torch.cuda.synchronize()
        return g[:3], capi.last_kernel()

    assert run()[1] == "sm100_wide_tcgen05_bwd"
    capi.lib.fa_set_kernel_policy(1)
    try:
        want, _ = run()
    finally:
        capi.lib.fa_set_kernel_policy(0)
    real, sizes = capi.workspace, []

    def small(n, device):
        sizes.append(n)
        if n > 1 << 20:
            raise torch.OutOfMemoryError("no room")
        return real(n, device)

    monkeypatch.setattr(capi, "workspace", small)
    got, name = run()
    assert name == "generic_mma_bwd" and len(sizes) == 2 and sizes[1] < 1 << 20 < sizes[0]
    assert all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("d", [136, 256])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("causal,win,cap,alibi", [(True, (-1, -1), 0.0, False), (False, (-1, -1), 0.0, False), (False, (70, 40), 0.0, True), (True, (-1, -1), 3.0, False)])
def test_non_finite_values_stay_in_their_packed_sequence(d, bad, causal, win, cap, alibi):
    import fa_b200_capi as capi
    from flash_attn_npu import flash_attn_npu as ext
    lens, h, hkv = [200, 77, 130, 300], 4, 2
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    q, do = (torch.randn(sum(lens), h, d, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(sum(lens), hkv, d, device="cuda").bfloat16() for _ in range(2))
    slopes = torch.rand(h, device="cuda") * 0.1 if alibi else None
    tail = (cu, cu, slopes, 300, 300, 0.0, d ** -0.5, False, causal, *win, cap, False, None, None)
    out, lse, _, _ = ext.varlen_fwd(q, k, v, None, cu, cu, None, None, None, slopes, 300, 300, 0.0, d ** -0.5, False, causal, *win, cap, False, None)

    def run():
        g = ext.varlen_bwd(do, q, k, v, out, lse, None, None, None, *tail)[:3]
        torch.cuda.synchronize()
        assert capi.last_kernel() == "sm100_wide_tcgen05_bwd" and capi.lib.fa_debug_get(2) == 0
        return g

    want = run()
    for t in (q, k, v, do, out):
        t[200:277] = bad
    got = run()
    for x, y in zip(got, want):
        for s in (slice(0, 200), slice(277, None)):
            assert torch.equal(x[s], y[s])


@pytest.mark.parametrize("cap", [0.5, 30.0, 2e4, 1e6])
def test_capped_scores_keep_their_precision(cap):
    """A large cap multiplies whatever absolute error tanh has: with the oracle's LSE the gradients stay within the roundings of
    P, dS and the result."""
    import fa_b200_capi as capi
    from flash_attn_npu import flash_attn_npu as ext
    d, dt = 256, torch.float16
    q, k, v, do = ((torch.rand(1, 260, 2, d) * 2 - 1).to(dt) for _ in range(4))
    scale = d ** -0.5
    out, lse = orc.attention_fwd(q.float(), k.float(), v.float(), scale, True, (-1, -1), cap, data_type=torch.float32)
    lp = orc.attention_bwd(q, k, v, do, lse, scale, True, (-1, -1), cap)
    f32 = orc.attention_bwd(q.float(), k.float(), v.float(), do.float(), lse, scale, True, (-1, -1), cap)
    got = ext.bwd(*(t.cuda() for t in (do, q, k, v, out.to(dt), lse)), None, None, None, None, 0.0, scale, True, -1, -1, cap, False, None, None)[:3]
    torch.cuda.synchronize()
    assert capi.last_kernel() == "sm100_wide_tcgen05_bwd"
    for n, g, a, r in zip(("dq", "dk", "dv"), got, lp, f32):
        assert_within(n, g.cpu(), a, r, roundings=3)


@pytest.mark.parametrize("dt,d,causal,win,cap", [
    (torch.float16, 256, False, (60, 30), 0.0), (torch.bfloat16, 192, True, (100, 0), 0.0), (torch.float16, 160, True, (-1, -1), 4.0),
    (torch.bfloat16, 256, False, (-1, -1), 0.0), (torch.float16, 248, False, (0, 150), 2.0)])
def test_wide_packed_backward_with_windows_and_caps(dt, d, causal, win, cap):
    import fa_b200_capi as capi
    from flash_attn_npu import flash_attn_npu as ext
    lq, lk, h, hkv = [300, 0, 129, 64, 1], [260, 70, 400, 1, 130], 4, 2
    q, do = ((torch.rand(sum(lq), h, d) * 2 - 1).to(dt) for _ in range(2))
    k, v = ((torch.rand(sum(lk), hkv, d) * 2 - 1).to(dt) for _ in range(2))
    cu = [torch.tensor([0] + torch.tensor(x).cumsum(0).tolist(), dtype=torch.int32) for x in (lq, lk)]
    scale = d ** -0.5
    out, lse = orc.attention_varlen_fwd(q.float(), k.float(), v.float(), *cu, scale, causal, win, cap, data_type=torch.float32)
    lp = orc.attention_varlen_bwd(q, k, v, do, lse, *cu, scale, causal, win, cap)
    f32 = orc.attention_varlen_bwd(q.float(), k.float(), v.float(), do.float(), lse, *cu, scale, causal, win, cap)
    qg, kg, vg, dog, og, lg, cq, ck = (t.cuda() for t in (q, k, v, do, out.to(dt), lse, *cu))
    g = [torch.full_like(t, 777.0) for t in (qg, kg, vg)]
    ext.varlen_bwd(dog, qg, kg, vg, og, lg, *g, cq, ck, None, max(lq), max(lk), 0.0, scale, False, causal, *win, cap, False, None, None)
    torch.cuda.synchronize()
    assert capi.last_kernel() == "sm100_wide_tcgen05_bwd" and capi.lib.fa_debug_get(2) == 0
    for n, x, a, r in zip(("dq", "dk", "dv"), g, lp, f32):
        assert_within(n, x.cpu(), a, r, roundings=3)
