"""dQ from stored dS tiles: packed sequences (the numbering of their query blocks, empty sequences, sequences without keys or
whose first queries see none) and dense calls with two query blocks a CTA (odd counts, neighbours with different key ranges),
against the general kernels.  Both round P, dS and the result to the input type once and sum in fp32, in another order:
three half-ulp roundings of the largest value."""
import pytest
import torch

pytestmark = pytest.mark.gpu


STORED_DS = 3                            # fa_debug_get(8): dQ came from stored dS tiles


def _compare(run, dt, name):
    import fa_b200_capi as capi
    got = run()
    assert capi.last_kernel() == name and capi.lib.fa_debug_get(8) == STORED_DS and capi.lib.fa_debug_get(2) == 0
    again = run()
    capi.lib.fa_set_kernel_policy(1)
    try:
        ref = run()
        assert capi.last_kernel() == "generic_mma_bwd"
    finally:
        capi.lib.fa_set_kernel_policy(0)
    bits = 8 if dt == torch.bfloat16 else 11
    for n, x, y, r in zip(("dq", "dk", "dv"), got, again, ref):
        assert torch.equal(x, y), n
        assert (x.float() - r.float()).abs().max().item() <= 3 * 2.0 ** -bits * r.float().abs().max().item(), n


PACKED = [
    ([128, 256, 1, 0, 127, 129, 640], None, 128, 4, 2, True, (-1, -1), torch.bfloat16),
    ([300, 0, 129, 64, 500], [260, 70, 400, 0, 130], 64, 2, 2, True, (-1, -1), torch.float16),
    ([1, 1, 1, 2, 1500], None, 96, 2, 1, False, (-1, -1), torch.bfloat16),
    ([700, 900, 333], None, 128, 4, 4, True, (100, 0), torch.float16),
    ([400, 513], [900, 40], 128, 2, 2, False, (30, 60), torch.bfloat16),
]


@pytest.mark.parametrize("case", PACKED, ids=lambda c: str(c[0]))
def test_packed_backward(case):
    from flash_attn_npu import flash_attn_npu as ext
    lq, lk, d, h, hkv, causal, win, dt = case
    lk = lk or lq
    q, do = (torch.randn(sum(lq), h, d, device="cuda", dtype=dt) for _ in range(2))
    k, v = (torch.randn(sum(lk), hkv, d, device="cuda", dtype=dt) for _ in range(2))
    cq, ck = (torch.tensor([0] + torch.tensor(x).cumsum(0).tolist(), dtype=torch.int32, device="cuda") for x in (lq, lk))
    out, lse, _, _ = ext.varlen_fwd(q, k, v, None, cq, ck, None, None, None, None, max(lq), max(lk), 0.0, d ** -0.5, False,
                                    causal, *win, 0.0, False, None)

    def run():
        g = [torch.full_like(t, 777.0) for t in (q, k, v)]
        ext.varlen_bwd(do, q, k, v, out, lse, *g, cq, ck, None, max(lq), max(lk), 0.0, d ** -0.5, False, causal, *win, 0.0,
                       False, None, None)
        torch.cuda.synchronize()
        return g

    _compare(run, dt, "sm100_tcgen05_bwd")


def test_packed_backward_without_room_for_the_tiles(monkeypatch):
    """The allocator refuses the workspace with the dS tiles: the call runs on the least one, within the roundings of the
    other path."""
    import fa_b200_capi as capi
    from flash_attn_npu import flash_attn_npu as ext
    lens, h, d = [300, 77, 513], 4, 128
    q, k, v, do = (torch.randn(sum(lens), h, d, device="cuda").bfloat16() for _ in range(4))
    cu = torch.tensor([0, 300, 377, 890], dtype=torch.int32, device="cuda")
    out, lse, _, _ = ext.varlen_fwd(q, k, v, None, cu, cu, None, None, None, None, 513, 513, 0.0, 0.1, False, True, -1, -1, 0.0, False, None)
    args = (do, q, k, v, out, lse, None, None, None, cu, cu, None, 513, 513, 0.0, 0.1, False, True, -1, -1, 0.0, False, None, None)
    a = ext.varlen_bwd(*args)
    real, sizes = capi.workspace, []

    def small(n, device):
        sizes.append(n)
        if n > 1 << 20:
            raise torch.OutOfMemoryError("no room")
        return real(n, device)

    monkeypatch.setattr(capi, "workspace", small)
    b = ext.varlen_bwd(*args)
    torch.cuda.synchronize()
    assert len(sizes) == 2 and sizes[1] < sizes[0] and capi.lib.fa_debug_get(8) == 0 and capi.lib.fa_debug_get(2) == 0
    for x, y in zip(a[:3], b[:3]):
        assert (x.float() - y.float()).abs().max().item() <= 2 * 2.0 ** -8 * y.float().abs().max().item()


@pytest.mark.parametrize("b,sq,sk,h,hkv,d,causal,win", [
    (4, 2432, 2432, 16, 4, 128, True, (-1, -1)), (4, 2370, 1100, 16, 16, 64, True, (-1, -1)),
    (2, 4700, 4700, 16, 8, 128, True, (150, 0)), (3, 3000, 500, 18, 6, 96, False, (200, 100))])
def test_dense_backward_with_two_query_blocks_a_cta(b, sq, sk, h, hkv, d, causal, win):
    from flash_attn_npu import flash_attn_npu as ext
    dt = torch.bfloat16
    assert b * h * ((sq + 127) // 128) >= 8 * torch.cuda.get_device_properties(0).multi_processor_count
    q, do = (torch.randn(b, sq, h, d, device="cuda", dtype=dt) for _ in range(2))
    k, v = (torch.randn(b, sk, hkv, d, device="cuda", dtype=dt) for _ in range(2))
    out, lse, _, _ = ext.fwd(q, k, v, None, None, 0.0, d ** -0.5, causal, *win, 0.0, False, None)

    def run():
        g = [torch.full_like(t, 777.0) for t in (q, k, v)]
        ext.bwd(do, q, k, v, out, lse, *g, None, 0.0, d ** -0.5, causal, *win, 0.0, False, None, None)
        torch.cuda.synchronize()
        return g

    _compare(run, dt, "sm100_tcgen05_bwd_5gemm")
