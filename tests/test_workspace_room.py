"""Large workspaces are only asked for where they can be had."""
import pytest
import torch

import fa_b200_capi as capi

GIB = 1 << 30


@pytest.mark.parametrize("nbytes,held,free,fits,asked", [
    (1 << 20, 0, 0, True, 0),                                # small ones are not looked at
    (3 * GIB, 4 * GIB, 0, True, 1),                          # the allocator holds enough: the driver is not asked
    (3 * GIB, 2 * GIB, 2 * GIB, True, 2),
    (3 * GIB, 1 * GIB, 1 * GIB, False, 2),
    (3 * GIB, None, 0, True, 1),
])
def test_what_fits(nbytes, held, free, fits, asked, monkeypatch):
    calls = []
    stats = {} if held is None else {"reserved_bytes": {"all": {"current": 5 * GIB + held}}, "allocated_bytes": {"all": {"current": 5 * GIB}}}
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda.memory, "memory_stats_as_nested_dict", lambda device=None: calls.append("stats") or stats)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: calls.append("driver") or (free, 180 * GIB))
    assert capi.workspace_fits(nbytes, 0) is fits and len(calls) == asked
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert capi.workspace_fits(nbytes, 0)


def test_an_allocator_without_counts_is_simply_asked(monkeypatch):
    """A pluggable allocator refuses the question with a RuntimeError."""
    def refuse(device=None):
        raise RuntimeError("not supported")
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda.memory, "memory_stats_as_nested_dict", refuse)
    assert capi.workspace_fits(3 * GIB, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("d,kernel", [(128, "sm100_tcgen05_bwd"), (256, "generic_mma_bwd")])
def test_backward_does_not_try_what_cannot_fit(d, kernel, monkeypatch):
    from flash_attn_npu import flash_attn_npu as ext
    q, k, v, do = (torch.randn(1, 700, 4, d, device="cuda").bfloat16() for _ in range(4))
    out, lse, _, _ = ext.fwd(q, k, v, None, None, 0.0, 0.1, True, -1, -1, 0.0, False, None)
    args = (do, q, k, v, out, lse, None, None, None, None, 0.0, 0.1, True, -1, -1, 0.0, False, None, None)
    want = ext.bwd(*args)[:3]
    real, sizes = capi.workspace, []
    monkeypatch.setattr(capi, "workspace", lambda n, device: sizes.append(n) or real(n, device))
    monkeypatch.setattr(capi, "_LARGE_WORKSPACE", 1 << 20)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (0, 180 * GIB))
    stats = torch.cuda.memory.memory_stats_as_nested_dict
    monkeypatch.setattr(torch.cuda.memory, "memory_stats_as_nested_dict", lambda device=None: {
        key: {"all": {"current": stats(device)["allocated_bytes"]["all"]["current"]}} for key in ("reserved_bytes", "allocated_bytes")})
    got = ext.bwd(*args)[:3]
    torch.cuda.synchronize()
    assert capi.last_kernel() == kernel and len(sizes) == 1 and sizes[0] < 1 << 20 and capi.lib.fa_debug_get(2) == 0
    for x, y in zip(got, want):                              # roundings of P, dS and the result
        assert (x.float() - y.float()).abs().max().item() <= 3 * 2.0 ** -8 * y.float().abs().max().item()


@pytest.mark.gpu
@pytest.mark.parametrize("d,packed,kernel", [(128, False, "sm100_tcgen05_bwd"), (128, True, "sm100_tcgen05_bwd"), (256, False, "generic_mma_bwd"), (192, True, "generic_mma_bwd")])
def test_a_workspace_aligned_for_floats_only_holds_no_tiles(d, packed, kernel, monkeypatch):
    """Bulk copies want 16-byte addresses; a C caller's workspace may start on any float."""
    from flash_attn_npu import flash_attn_npu as ext
    s, h = 300, 4
    q, k, v, do = (torch.randn(*((2 * s, h, d) if packed else (2, s, h, d)), device="cuda").bfloat16() for _ in range(4))
    cu = torch.tensor([0, s, 2 * s], dtype=torch.int32, device="cuda")
    if packed:
        out, lse, _, _ = ext.varlen_fwd(q, k, v, None, cu, cu, None, None, None, None, s, s, 0.0, 0.1, False, True, -1, -1, 0.0, False, None)
        run = lambda: ext.varlen_bwd(do, q, k, v, out, lse, None, None, None, cu, cu, None, s, s, 0.0, 0.1, False, True, -1, -1, 0.0, False, None, None)[:3]  # noqa: E731
    else:
        out, lse, _, _ = ext.fwd(q, k, v, None, None, 0.0, 0.1, True, -1, -1, 0.0, False, None)
        run = lambda: ext.bwd(do, q, k, v, out, lse, None, None, None, None, 0.0, 0.1, True, -1, -1, 0.0, False, None, None)[:3]  # noqa: E731
    want = run()
    real = capi.workspace
    monkeypatch.setattr(capi, "workspace", lambda n, device: real(n + 16, device)[4:4 + n])
    got = run()
    torch.cuda.synchronize()
    assert capi.last_kernel() == kernel and capi.lib.fa_debug_get(8) == 0 and capi.lib.fa_debug_get(2) == 0
    for x, y in zip(got, want):                              # roundings of P, dS and the result
        assert (x.float() - y.float()).abs().max().item() <= 3 * 2.0 ** -8 * y.float().abs().max().item()
