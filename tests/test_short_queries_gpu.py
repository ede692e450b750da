"""At most 128 query rows a block: both softmax groups work on the same rows, on even and odd key tiles.  One, two and three
key tiles, rows that see keys of one group only or none, windows, alibi, packed queries, stacked heads with split keys."""
import pytest
import torch

from oracle import attention_oracle as orc
from parity import assert_lse, assert_within, fwd_refs

pytestmark = pytest.mark.gpu

SHORT_QUERIES = 1                        # fa_debug_get(8): both softmax groups worked on the same rows

# (dtype, B, H, Hkv, Sq, Sk, D, causal, wl, wr, alibi)
CASES = [
    (torch.bfloat16, 2, 2, 2, 1, 1, 128, False, -1, -1, False),
    (torch.float16, 1, 2, 2, 128, 128, 64, True, -1, -1, False),
    (torch.bfloat16, 1, 2, 1, 127, 129, 128, True, -1, -1, False),
    (torch.float16, 1, 2, 2, 128, 256, 96, False, -1, -1, False),
    (torch.bfloat16, 2, 4, 2, 33, 300, 128, True, -1, -1, True),
    (torch.bfloat16, 1, 8, 1, 5, 1025, 64, True, -1, -1, True),
    (torch.float16, 1, 2, 2, 100, 900, 128, True, 60, 0, False),
    (torch.bfloat16, 1, 2, 2, 128, 40, 128, True, -1, -1, False),
    (torch.float16, 1, 4, 1, 16, 777, 128, False, 200, 100, False),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(x).replace("torch.", "") for x in c))
def test_short_dense_queries(case):
    import fa_b200_capi as capi
    import flash_attn_npu as fa
    dt, b, h, hkv, sq, sk, d, causal, wl, wr, alibi = case
    q, k, v = (torch.randn(b, s, n, d).to(dt) for s, n in ((sq, h), (sk, hkv), (sk, hkv)))
    slopes = torch.rand(h) * 0.3 if alibi else None
    (lp_o, _), (f_o, f_l) = fwd_refs(q, k, v, d ** -0.5, causal, (wl, wr), 0.0, slopes)
    out, lse, _ = fa.flash_attn_func(q.cuda(), k.cuda(), v.cuda(), causal=causal, window_size=(wl, wr),
                                     alibi_slopes=None if slopes is None else slopes.cuda(), return_attn_probs=True)
    torch.cuda.synchronize()
    rows = sq * (h // hkv if sq < 128 else 1)                # a group of heads is stacked into the tile rows
    assert capi.last_kernel() == "sm100_tcgen05_2q" and capi.lib.fa_debug_get(2) == 0
    assert capi.lib.fa_debug_get(8) == (SHORT_QUERIES if rows <= 128 and sk > 128 else 0)      # one key tile is not shared out
    assert_within("out", out.cpu(), lp_o, f_o)
    assert_lse(lse.cpu(), f_l)


def test_short_packed_queries_and_a_growing_maximum():
    """Packed queries of at most 128 a sequence; keys whose scores grow from tile to tile, so that the two groups end on
    different exponent bases and each moves its own."""
    import flash_attn_npu as fa
    lq, lk, d = [128, 0, 1, 77], [700, 130, 0, 513], 64
    q, k, v = torch.zeros(sum(lq), 1, d), torch.zeros(sum(lk), 1, d), torch.randn(sum(lk), 1, d)
    q[..., 0] = 8.0
    k[:, 0, 0] = torch.arange(sum(lk)) // 128 * 3.0
    q, k, v = (t.half() for t in (q, k, v))
    cu = [torch.tensor([0] + torch.tensor(x).cumsum(0).tolist(), dtype=torch.int32) for x in (lq, lk)]
    lp_o, _ = orc.attention_varlen_fwd(q, k, v, *cu, 1.0, False)
    f_o, f_l = orc.attention_varlen_fwd(q.float(), k.float(), v.float(), *cu, 1.0, False, data_type=torch.float32)
    out, lse, _ = fa.flash_attn_varlen_func(q.cuda(), k.cuda(), v.cuda(), cu[0].cuda(), cu[1].cuda(), 128, 700, softmax_scale=1.0,
                                            return_attn_probs=True)
    import fa_b200_capi as capi
    assert capi.lib.fa_debug_get(8) == SHORT_QUERIES
    assert_within("out", out.cpu(), lp_o, f_o)
    assert_lse(lse.cpu(), f_l)


@pytest.mark.parametrize("page", [0, 64, 256])
@pytest.mark.parametrize("sq,h,splits", [(4, 16, 0), (4, 16, 1), (3, 16, 3), (32, 8, 0), (100, 2, 2)])
def test_short_chunks_against_a_cache(page, sq, h, splits):
    import fa_b200_capi as capi
    import flash_attn_npu as fa
    hkv, d, lens, cap, dt = 2, 128, [5, 256, 1000, 1290], 1536, torch.bfloat16
    b = len(lens)
    q = torch.randn(b, sq, h, d).to(dt)
    if page:
        per = cap // page
        table = torch.randperm(b * per).to(torch.int32).reshape(b, per)
        kc, vc = (torch.randn(b * per, page, hkv, d).to(dt) for _ in range(2))
    else:
        table, (kc, vc) = None, (torch.randn(b, cap, hkv, d).to(dt) for _ in range(2))
    lens_t = torch.tensor(lens, dtype=torch.int32)
    lp, _ = orc.kvcache_fwd(q, kc.clone(), vc.clone(), lens_t, d ** -0.5, block_table=table, causal=True)
    f, fl = orc.kvcache_fwd(q.float(), kc.float(), vc.float(), lens_t, d ** -0.5, block_table=table, causal=True)
    out, lse = fa.flash_attn_with_kvcache(q.cuda(), kc.cuda(), vc.cuda(), cache_seqlens=lens_t.cuda(), causal=True, num_splits=splits,
                                          block_table=None if table is None else table.cuda(), return_softmax_lse=True)
    torch.cuda.synchronize()
    assert capi.last_kernel() == "sm100_tcgen05_2q" and capi.lib.fa_debug_get(8) == SHORT_QUERIES and capi.lib.fa_debug_get(2) == 0
    assert_within("out", out.cpu(), lp, f)
    assert_lse(lse.cpu(), fl)
