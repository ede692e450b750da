"""Append + rotary in 16-byte pieces against the oracle bit for bit, at the edges of its rule (rotary_dim that is and is not a
multiple of 16, rows with an odd number of chunks, rows that land outside the cache); the combine of few splits at the edges
of its own (2, 4 and 8 splits, one more, head dims off the vector width, empty splits, unaligned outputs)."""
import pytest
import torch

from oracle import attention_oracle as orc
from parity import assert_lse, assert_within

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("d,rd", [(64, 64), (128, 128), (128, 64), (72, 32), (72, 0), (128, 40), (256, 256), (8, 0), (24, 16)])
@pytest.mark.parametrize("sq", [1, 5, 130])
def test_append_and_rotary_bits(d, rd, interleaved, sq):
    import flash_attn_npu as fa
    b, h, hkv, page, dt = 3, 4, 2, 64, torch.bfloat16
    lens = [0, 61, 250]
    per = 7
    table = torch.randperm(b * per).to(torch.int32).reshape(b, per)
    q, kn, vn = (torch.randn(b, sq, n, d).to(dt) for n in (h, hkv, hkv))
    kc, vc = (torch.randn(b * per, page, hkv, d).to(dt) for _ in range(2))
    cos, sin = orc.rotary_tables(400, rd, dtype=dt) if rd else (None, None)
    kr, vr = kc.clone(), vc.clone()
    ro, _ = orc.kvcache_fwd(q, kr, vr, lens, d ** -0.5, k_new=kn, v_new=vn, rotary_cos=cos, rotary_sin=sin,
                            rotary_interleaved=interleaved, block_table=table, causal=True)
    kg, vg = kc.cuda(), vc.cuda()
    cu = (lambda t: None if t is None else t.cuda())
    out = fa.flash_attn_with_kvcache(q.cuda(), kg, vg, kn.cuda(), vn.cuda(), rotary_cos=cu(cos), rotary_sin=cu(sin),
                                     cache_seqlens=torch.tensor(lens, dtype=torch.int32).cuda(), block_table=table.cuda(),
                                     causal=True, rotary_interleaved=interleaved)
    assert torch.equal(kg.cpu().view(torch.int16), kr.view(torch.int16))
    assert torch.equal(vg.cpu().view(torch.int16), vr.view(torch.int16))
    assert (out.cpu().float() - ro.float()).abs().max().item() <= 2 ** -5      # two roundings of values up to about 4


def test_append_outside_the_cache_changes_nothing():
    import flash_attn_npu as fa
    q, kn = torch.randn(2, 3, 2, 64).half().cuda(), torch.randn(2, 3, 2, 64).half().cuda()
    kc = torch.randn(2, 128, 2, 64).half().cuda()
    vc = kc.clone()
    k0 = kc.clone()
    fa.flash_attn_with_kvcache(q, kc, vc, kn, kn, cache_seqlens=torch.tensor([126, 500], dtype=torch.int32).cuda(), causal=True)
    torch.cuda.synchronize()
    k0[0, 126:128] = kn[0, :2]
    assert torch.equal(kc, k0) and torch.equal(vc, k0)


@pytest.mark.parametrize("nsplit", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("dv", [8, 64, 128, 130, 256])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_combine_of_few_splits(nsplit, dv, dtype):
    import flash_attn_npu_3 as fa3
    rows = 37
    op, lp = torch.randn(nsplit, 1, rows, 1, dv), torch.randn(nsplit, 1, rows, 1) * 3
    lp[0, 0, 3] = -float("inf")
    lp[:, 0, 5] = -float("inf")
    dead = torch.isneginf(lp)
    ref_o, ref_l = orc.combine_partials(torch.where(dead[..., None], torch.zeros(()), op).reshape(nsplit, rows, dv), lp.reshape(nsplit, rows), torch.float32)
    op[dead] = float("nan")                                  # never read
    out, lse = fa3.flash_attn_combine(op.cuda(), lp.cuda(), out_dtype=dtype)
    out = out.cpu().float().reshape(rows, dv)
    # eight products and sums in fp32, then one rounding to the output type
    tol = 2e-6 * nsplit + {torch.float32: 0.0, torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}[dtype] * ref_o.abs().max().item()
    assert (out - ref_o).abs().max().item() <= tol
    assert_lse(lse.cpu().reshape(rows), ref_l)
