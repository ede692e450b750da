"""Key splits of prefill chunks against a cache: the counts that the planner chooses between, and shapes where the wrong one was
measurably slower."""
import pytest
import torch

import fa_b200_capi as capi

pytestmark = pytest.mark.gpu


def _splits(b, sq, hq, hkv, d, sk, cap=0.0):
    q = torch.empty(b, sq, hq, d, device="cuda", dtype=torch.bfloat16)
    kv = torch.empty(b, 8, hkv, d, device="cuda", dtype=torch.bfloat16)      # the planner only looks at strides
    lens = torch.zeros(b, dtype=torch.int32, device="cuda")
    p = capi.FwdParams()
    p.q, p.o = capi.tensor4(q), capi.tensor4(q)
    p.k, p.v = capi.tensor4(kv), capi.tensor4(kv)
    p.k.stride_b = p.v.stride_b = sk * hkv * d
    p.kv_entries, p.seqused_k = b, lens.data_ptr()
    p.b, p.sq, p.sk, p.hq, p.hkv, p.d, p.dv = b, sq, sk, hq, hkv, d, d
    p.scale, p.softcap, p.causal, p.window_left, p.window_right, p.dtype = d ** -0.5, cap, 1, -1, -1, 1
    return capi.lib.fa_fwd_num_splits(p)


def _ctas(b, sq, hq, hkv):
    g = hq // hkv
    stacked = sq < 128 and g > 1 and g & (g - 1) == 0
    return b * (hkv if stacked else hq) * -(-sq * (g if stacked else 1) // 256)


SMS = 148


@pytest.mark.parametrize("d", [64, 128])
def test_counts(d):
    for b, sq, hq, hkv in ((1, 64, 32, 8), (1, 512, 32, 8), (2, 256, 16, 16), (4, 512, 32, 8), (8, 300, 16, 4), (3, 1000, 16, 2), (8, 64, 8, 1)):
        for sk in (2048, 4096, 11264, 16000, 32768):
            for cap in (0.0, 30.0):
                ctas = _ctas(b, sq, hq, hkv)
                most = max(1, min(-(-2 * SMS // ctas), -(-sk // 2048)))
                n = _splits(b, sq, hq, hkv, d, sk, cap)
                whole = lambda k: -(-(-(-sk // 64)) // ((-(-(-(-sk // 64)) // k) + 1) // 2 * 2))     # splits of whole 128-key tiles  # noqa: E731
                assert n in {whole(k) for k in (1, min(most, max(1, SMS // ctas)), most)}, (b, sq, hq, hkv, sk, cap, n)


@pytest.mark.parametrize("shape,n", [
    ((1, 64, 32, 8, 128, 32768), 16), ((1, 256, 8, 8, 128, 28672), 14),       # one wave holds the most: 15 and 13 were slower
    ((4, 512, 32, 8, 64, 32768, 30.0), 2), ((4, 512, 32, 8, 128, 32768, 30.0), 2),         # two CTAs an SM
    ((4, 512, 32, 8, 128, 16128), 1), ((1, 512, 32, 8, 128, 16000), 2), ((2, 256, 16, 16, 64, 16128), 4)])
def test_choices(shape, n):
    if torch.cuda.get_device_properties(0).multi_processor_count != SMS:
        pytest.skip("measured on 148 SMs")
    assert _splits(*shape) == n
