"""Capped scores without alibi on the kernel with one query tile a CTA: tile edges, padded head dims, windows, scores on both
sides of the range of the tanh polynomial (|score * scale| <= 0.8 cap), a moving exponent base, packed and cached keys."""
import pytest
import torch

from oracle import attention_oracle as orc
from parity import assert_lse, assert_within, fwd_refs

pytestmark = pytest.mark.gpu

ONE_TILE = ("sm100_tcgen05_2q", 2)       # fa_last_kernel(), fa_debug_get(8)


def _ran():
    import fa_b200_capi as capi
    return capi.last_kernel(), capi.lib.fa_debug_get(8)


# (dtype, B, H, Hkv, Sq, Sk, D, causal, wl, wr, cap, spread of q)
CASES = [
    (torch.bfloat16, 2, 2, 2, 128, 128, 128, False, -1, -1, 30.0, 1.0),
    (torch.float16, 1, 4, 2, 129, 127, 64, True, -1, -1, 30.0, 1.0),
    (torch.bfloat16, 1, 2, 1, 1, 300, 128, False, -1, -1, 2.0, 1.0),
    (torch.float16, 1, 2, 2, 257, 1, 64, False, -1, -1, 30.0, 1.0),
    (torch.bfloat16, 1, 2, 2, 300, 513, 96, True, -1, -1, 50.0, 1.0),
    (torch.float16, 1, 2, 1, 260, 260, 8, False, 40, 70, 1.0, 4.0),
    (torch.bfloat16, 1, 4, 4, 700, 700, 128, True, 100, 0, 30.0, 40.0),
    (torch.float16, 1, 2, 2, 520, 1100, 64, False, -1, -1, 60.0, 40.0),
    (torch.bfloat16, 1, 2, 2, 400, 300, 128, True, -1, -1, 0.5, 20.0),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(x).replace("torch.", "") for x in c))
def test_capped_forward_against_the_oracle(case):
    import fa_b200_capi as capi
    import flash_attn_npu as fa
    dt, b, h, hkv, sq, sk, d, causal, wl, wr, cap, spread = case
    q = (torch.randn(b, sq, h, d) * spread).to(dt)
    k, v = (torch.randn(b, sk, hkv, d).to(dt) for _ in range(2))
    scale = d ** -0.5
    (lp_o, _), (f_o, f_l) = fwd_refs(q, k, v, scale, causal, (wl, wr), cap)
    out, lse, _ = fa.flash_attn_func(q.cuda(), k.cuda(), v.cuda(), causal=causal, window_size=(wl, wr), softcap=cap, return_attn_probs=True)
    torch.cuda.synchronize()
    assert capi.lib.fa_debug_get(2) == 0 and _ran() == ONE_TILE
    assert_within("out", out.cpu(), lp_o, f_o)
    assert_lse(lse.cpu(), f_l)


def test_capped_forward_row_maximum_grows_along_the_keys():
    """Every key tile raises the row maximum by more than the threshold at which the exponent base moves, in one half of the
    tile and then in the other; not-a-number scores stay in their own rows."""
    import flash_attn_npu as fa
    sk, d = 640, 64
    q, k, v = torch.zeros(1, 130, 1, d), torch.zeros(1, sk, 1, d), torch.randn(1, sk, 1, d)
    q[..., 0] = 8.0
    k[0, :, 0, 0] = torch.tensor([(3.0 * (i // 64)) for i in range(sk)])
    q, k, v = (t.half() for t in (q, k, v))
    (lp_o, _), (f_o, f_l) = fwd_refs(q, k, v, 1.0, False, (-1, -1), 300.0)
    qn = q.clone()
    qn[0, 5] = float("nan")
    for x in (q, qn):
        out, lse, _ = fa.flash_attn_func(x.cuda(), k.cuda(), v.cuda(), softmax_scale=1.0, softcap=300.0, return_attn_probs=True)
        assert _ran() == ONE_TILE
        keep = torch.arange(130) != 5 if x is qn else slice(None)
        assert_within("out", out.cpu()[:, keep], lp_o[:, keep], f_o[:, keep])
        assert_lse(lse.cpu()[..., keep], f_l[..., keep])
    assert torch.isnan(out[0, 5]).all()


@pytest.mark.parametrize("page", [0, 64, 128])
@pytest.mark.parametrize("sq,splits", [(70, 1), (200, 3), (9, 2)])
def test_capped_prefill_against_a_cache(page, sq, splits):
    import fa_b200_capi as capi
    import flash_attn_npu as fa
    b, h, hkv, d, lens, cap = 2, 8, 2, 128, [333, 700], 5.0
    dt = torch.bfloat16
    q = torch.randn(b, sq, h, d).to(dt)
    if page:
        per = 768 // page
        table = torch.randperm(b * per).to(torch.int32).reshape(b, per)
        kc, vc = (torch.randn(b * per, page, hkv, d).to(dt) for _ in range(2))
    else:
        table, (kc, vc) = None, (torch.randn(b, 768, hkv, d).to(dt) for _ in range(2))
    args = dict(block_table=table, causal=True, softcap=cap)
    lp, _ = orc.kvcache_fwd(q, kc.clone(), vc.clone(), torch.tensor(lens), d ** -0.5, **args)
    f, fl = orc.kvcache_fwd(q.float(), kc.float(), vc.float(), torch.tensor(lens), d ** -0.5, **args)
    out, lse = fa.flash_attn_with_kvcache(q.cuda(), kc.cuda(), vc.cuda(), cache_seqlens=torch.tensor(lens, dtype=torch.int32).cuda(),
                                          block_table=None if table is None else table.cuda(), causal=True, softcap=cap, num_splits=splits,
                                          return_softmax_lse=True)
    torch.cuda.synchronize()
    assert capi.lib.fa_debug_get(2) == 0 and _ran() == ONE_TILE
    assert_within("out", out.cpu(), lp, f)
    assert_lse(lse.cpu(), fl)


@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("d,causal,win", [(64, False, (-1, -1)), (128, True, (-1, -1)), (128, True, (90, 0))])
def test_infinite_scores_are_capped(d, causal, win, sign):
    """The cap makes a finite score of an infinite one: such a row averages the values it sees, and its LSE is sign * cap + ln(keys)."""
    import math
    import fa_b200_capi as capi
    import flash_attn_npu as fa
    b, s, h, cap = 1, 300, 2, 200.0
    q, k, v = (torch.randn(b, s, h, d) for _ in range(3))
    q[:, ::3], k[..., 1:], k[..., 0] = 0.0, 0.0, 1.0
    q[:, ::3, :, 0] = sign * math.inf
    q, k, v = (t.bfloat16() for t in (q, k, v))
    out, lse, _ = fa.flash_attn_func(q.cuda(), k.cuda(), v.cuda(), causal=causal, window_size=win, softcap=cap, return_attn_probs=True)
    torch.cuda.synchronize()
    assert capi.lib.fa_debug_get(2) == 0 and _ran() == ONE_TILE
    for i in range(0, s, 3):
        lo, hi = (max(0, i - win[0]) if win[0] >= 0 else 0), (i if causal else s - 1)
        want = v[:, lo:hi + 1].float().mean(1)
        assert (out[:, i].cpu().float() - want).abs().max() <= 2.0 ** -7 * max(1.0, want.abs().max().item()), i
        assert (lse[..., i].cpu() - (sign * cap + math.log(hi - lo + 1))).abs().max() <= 1e-3, i
