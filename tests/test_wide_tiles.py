"""Backward above head dim 128: the tiles that its kernels store and read stay inside the workspace that the stated longest
lengths ask for, also when a packed sequence is longer than stated; and they are the tiles that hold visible pairs."""
import ctypes as C
import os
import random
import subprocess

import pytest
import torch

import fa_b200_capi as capi

HARNESS = r"""
#include "bwd_wide_tiles.h"
using namespace fa;
extern "C" void key_rule(const int* t, int sq, int sk, int n, int* r) {
    const BlockRange x = wide_query_blocks({t[0], t[1], t[2], t[3], t[4]}, sq, sk, n); r[0] = x.lo; r[1] = x.hi;
}
extern "C" void query_rule(const int* t, int sq, int sk, int m, int* r) {
    const BlockRange x = wide_key_blocks({t[0], t[1], t[2], t[3], t[4]}, sq, sk, m); r[0] = x.lo; r[1] = x.hi;
}
extern "C" size_t tile(const int* t, int group, int pair, int g, int n, int m) {
    return wide_tile_at({t[0], t[1], t[2], t[3], t[4]}, group, pair, g, n, m);
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("wide_tiles")
    src, so = d / "h.cpp", d / "h.so"
    src.write_text(HARNESS)
    inc = os.path.join(os.path.dirname(capi.__file__), "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", inc, str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.tile.restype = C.c_size_t
    return lib


def _visible_blocks(sq, sk, causal, wl, wr):
    """(key block, query block) pairs that hold a visible pair, row by row."""
    wr = 0 if causal else wr
    pairs = set()
    for i in range(sq):
        lo = max(0, i + sk - sq - wl) if wl >= 0 else 0
        hi = min(sk - 1, i + sk - sq + wr) if wr >= 0 else sk - 1
        pairs.update((n, i // 128) for n in range(lo // 128, hi // 128 + 1) if lo <= hi)
    return pairs


def test_every_tile_lies_in_the_workspace_and_none_is_missing(rules):
    rng = random.Random(5)
    for trial in range(400):
        sq, sk = (rng.choice([0, 1, 127, 128, 129, rng.randint(0, 900)]) for _ in range(2))
        causal, wl, wr = rng.random() < 0.5, rng.choice([-1, 0, 100, 300]), rng.choice([-1, 0, 50, 400])
        stated = rng.choice([(sq, sk), (max(1, sq // 3), max(1, sk // 2)), (1, 1), (2 * sq + 1, sk + 400)])
        nqb, nkb = ((x + 127) // 128 for x in stated)
        t, r = (C.c_int * 5)(nkb, nqb, int(causal), wl, wr), (C.c_int * 2)()
        group, pairs = rng.choice([1, 3]), rng.choice([1, 2])
        size = pairs * group * nkb * nqb * 128 * 128 * 2
        stored, read = set(), set()
        for n in range(nkb):                                 # the grids run over the stated blocks
            if n * 128 < sk:
                rules.key_rule(t, sq, sk, n, r)
                stored.update((n, m) for m in range(r[0], r[1]))
        for m in range(nqb):
            if m * 128 < sq:
                rules.query_rule(t, sq, sk, m, r)
                read.update((n, m) for n in range(r[0], r[1]))
        assert stored == read
        for n, m in stored:
            assert n < nkb and m < nqb
            for pair in range(pairs):
                for g in range(group):
                    assert rules.tile(t, group, pair, g, n, m) + 128 * 128 * 2 <= size
        # whole key blocks at a time: a superset of the visible blocks, all of them inside the stated lengths
        assert {(n, m) for n, m in _visible_blocks(sq, sk, causal, wl, wr) if n < nkb and m < nqb} <= stored
    assert len({rules.tile(t, 3, p, g, n, m) for p in range(2) for g in range(3) for n in range(nkb) for m in range(nqb)}) == 6 * nkb * nqb


@pytest.mark.gpu
@pytest.mark.parametrize("d,hkv", [(192, 2), (256, 1)])
def test_understated_longest_length_stays_inside_the_workspace(d, hkv, monkeypatch):
    """The workspace lies in a larger allocation filled with a pattern: the pattern is there afterwards, and the sequences
    that are as long as stated or shorter get the gradients of a call that states the true length."""
    from flash_attn_npu import flash_attn_npu as ext
    lens, h = [100, 1100, 90, 700], 4
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    q, do = (torch.randn(sum(lens), h, d, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(sum(lens), hkv, d, device="cuda").bfloat16() for _ in range(2))
    out, lse, _, _ = ext.varlen_fwd(q, k, v, None, cu, cu, None, None, None, None, 1100, 1100, 0.0, 0.1, False, True, -1, -1, 0.0, False, None)
    held, guard = [], 8 << 20

    def guarded(n, device):
        held.append(torch.full((n + 2 * guard,), 0xA5, dtype=torch.uint8, device=device))
        return held[-1][guard:guard + n]

    monkeypatch.setattr(capi, "workspace", guarded)

    def run(most):
        g = ext.varlen_bwd(do, q, k, v, out, lse, None, None, None, cu, cu, None, most, most, 0.0, 0.1, False, True, -1, -1, 0.0, False,
                           None, None)[:3]
        torch.cuda.synchronize()
        assert capi.last_kernel() == "sm100_wide_tcgen05_bwd" and capi.lib.fa_debug_get(2) == 0
        return g

    full, short = run(1100), run(128)
    for buf in held:
        assert (buf[:guard] == 0xA5).all() and (buf[-guard:] == 0xA5).all()
    for a, b in zip(full, short):
        for s in (slice(0, 100), slice(1200, 1290)):
            assert torch.equal(a[s], b[s])
