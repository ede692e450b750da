"""The tanh polynomial of the capped-score forward, its coefficients read from the source and evaluated in fp32 with fused
multiply-adds as the kernel does."""
import os
import re

import numpy as np

import fa_b200_capi as capi


def test_error_of_the_polynomial():
    text = open(os.path.join(os.path.dirname(capi.__file__), "csrc", "fwd_single_sm100.cu")).read()
    body = text[text.index("float2 tanh_small2"):text.index("float tanh_any")]
    c = [np.float32(x) for x in re.findall(r"c2\((-?[\d.]+)f\)", body)]
    top = np.float32(re.search(r"kTanhSmall = ([\d.]+)f", text).group(1))
    assert len(c) == 6
    y = np.unique(np.concatenate([np.linspace(1e-6, top, 400001), np.geomspace(1e-6, top, 100001)]).astype(np.float32))
    y = y[y <= top]
    t, q = (y * y).astype(np.float32), np.full_like(y, c[0])
    for x in c[1:]:                                          # the products are exact in float64, one rounding each
        q = (q.astype(np.float64) * t.astype(np.float64) + np.float64(x)).astype(np.float32)
    got, want = (q * y).astype(np.float32), np.tanh(y.astype(np.float64))
    assert np.abs(got / want - 1).max() < 1.6e-7 and np.abs(got - want).max() < 1.01e-7
    # the other form, 1 - 2 / (1 + e^2y), with every step exact but for its rounding to fp32, is further off
    one, two = np.float32(1), np.float32(2)
    e = np.exp2((two * y * np.float32(np.log2(np.e))).astype(np.float64)).astype(np.float32)
    assert np.abs((one - two / (one + e)) - want).max() > 1.1e-7
