"""The extension module of the v2 API: `fwd`, `varlen_fwd`, `fwd_kvcache`, `bwd`,
`varlen_bwd` with the positional signatures and return lists of the reference's pybind
module (csrc/ascend910/flash_attn_npu/flash_api.cpp:1330-1338), implemented as calls
into libfa_b200.so.  torch allocates outputs and workspaces; the library computes.

Argument errors are raised as RuntimeError like the reference's TORCH_CHECKs
(flash_api.cpp:386-420, :658-682, :884-934).  Unlike the reference, alibi slopes,
rotary embedding, in-place append of new k/v, paged varlen and forced split counts are
implemented rather than rejected; dropout, return_softmax, leftpad_k stay rejected.
"""
from typing import List, Optional

import torch
import torch.nn.functional as F

import ctypes

import fa_b200_capi as capi


def _dtype_code(t):
    if t.dtype not in capi.DTYPES:
        raise RuntimeError("FlashAttention only supports FP16 and BF16 data types")
    return capi.DTYPES[t.dtype]


def _common_checks(q, k, v, softcap, what="key"):
    capi.require_cuda(q, k, v)
    if k.dtype != q.dtype:
        raise RuntimeError(f"query and {what} must have the same dtype")
    if v.dtype != q.dtype:
        raise RuntimeError("query and value must have the same dtype")
    for t in (q, k, v):
        if t.stride(-1) != 1:
            raise RuntimeError("Input tensor must have contiguous last dimension")
    if softcap < 0.0:
        raise RuntimeError("softcap must be non-negative (0.0 disables softcap)")


def _alibi(alibi_slopes, batch, nheads):
    """-> (tensor to keep alive, pointer, batch stride)"""
    if alibi_slopes is None:
        return None, 0, 0
    a = alibi_slopes.to(torch.float32).contiguous()
    if a.shape not in ((nheads,), (batch, nheads)):
        raise RuntimeError("alibi_slopes must have shape (nheads,) or (batch_size, nheads)")
    return a, a.data_ptr(), 0 if a.dim() == 1 else a.stride(0)


def _leaves(t, packed=False):
    """The four leaves of an fa_tensor: (B,S,H,D), or packed (T,H,D) without a batch stride."""
    s = t.stride()
    if s[-1] != 1:
        raise RuntimeError("last dimension must be contiguous")
    return (t.data_ptr(), 0, s[0], s[1]) if packed else (t.data_ptr(), s[0], s[1], s[2])


_NO_TENSOR = (0, 0, 0, 0)


def _ptr(t):
    return 0 if t is None else t.data_ptr()


def _i32(x):
    return x if -2 ** 31 <= x < 2 ** 31 else ctypes.c_int32(x).value


def _pad8(t):
    d = t.size(-1)
    return t if d % 8 == 0 else F.pad(t, [0, 8 - d % 8])


def fwd(q, k, v, out_, alibi_slopes_, p_dropout, softmax_scale, is_causal, window_size_left,
        window_size_right, softcap, return_softmax, gen_) -> List[torch.Tensor]:
    """mha_fwd (flash_api.cpp:639-846). q (B,Sq,H,D), k/v (B,Sk,Hkv,D) ->
    [out, softmax_lse (B,H,Sq) fp32, p (empty), rng_state (int64[2])]."""
    out, lse = dense_forward(q, k, v, out_, alibi_slopes_, p_dropout, softmax_scale, is_causal, window_size_left,
                             window_size_right, softcap, return_softmax)
    return [out, lse, *_unused(q)]


def _unused(q):
    return (torch.empty((0,), dtype=q.dtype, device=q.device), torch.zeros((2,), dtype=torch.int64, device=q.device))


def dense_forward(q, k, v, out_, alibi_slopes_, p_dropout, softmax_scale, is_causal, window_size_left,
                  window_size_right, softcap, return_softmax):
    """fwd without the two results that carry nothing here (dropout mask and generator state)."""
    _common_checks(q, k, v, softcap)
    if p_dropout != 0.0:
        raise RuntimeError("FlashAttention on B200 does not support dropout.")
    if return_softmax:
        raise RuntimeError("FlashAttention on B200 does not support return_softmax.")
    batch, sq, hq, d_og = q.shape
    sk, hkv = k.shape[1], k.shape[2]
    if batch <= 0:
        raise RuntimeError("batch size must be positive")
    if d_og > 256:
        raise RuntimeError("FlashAttention only supports head dimension at most 256")
    if hq % hkv != 0:
        raise RuntimeError("Number of heads in key/value must divide number of heads in query")
    q, k, v = _pad8(q), _pad8(k), _pad8(v)
    d = q.size(-1)
    device = q.device
    out = torch.empty_like(q) if (out_ is None or d != d_og) else out_
    lse = torch.empty((batch, hq, sq), dtype=torch.float32, device=device)
    keep, alibi, alibi_sb = _alibi(alibi_slopes_, batch, hq)
    buf = capi.FWD_BLOCK.new(
        *_leaves(q), *_leaves(k), *_leaves(v), *_leaves(out), lse.data_ptr(), *lse.stride(),
        0, 0, 0,                                             # cu_seqlens_q, cu_seqlens_k, seqused_k
        0, 0, 0, 0, alibi, alibi_sb,                         # block_table, its stride, page_size, cache_batch_idx
        batch, sq, sk, 0, 0, hq, hkv, d, v.size(-1), softmax_scale, softcap,
        int(is_causal), _i32(window_size_left), _i32(window_size_right), _dtype_code(q),
        *_NO_TENSOR, *_NO_TENSOR, 0, 0, 0, 0, 0, 0,          # new keys and values, rotary
        1, 0, 0, 0, 0, 0, 0, 0, 0, 0,                        # num_splits .. kv_entries
        capi.raw_stream(device))
    capi.launch(capi._call_fwd, buf, device)
    del keep
    if d != d_og:
        out = out[..., :d_og]
        if out_ is not None:
            out_.copy_(out)
            out = out_
    return out, lse


def varlen_fwd(q, k, v, out_, cu_seqlens_q, cu_seqlens_k, seqused_k_, leftpad_k_, block_table_,
               alibi_slopes_, max_seqlen_q, max_seqlen_k, p_dropout, softmax_scale, zero_tensors,
               is_causal, window_size_left, window_size_right, softcap, return_softmax, gen_):
    """mha_varlen_fwd (flash_api.cpp:848-1089). q (Tq,H,D), k/v (Tk,Hkv,D) or a paged cache
    (blocks,page,Hkv,D) with block_table -> [out, softmax_lse (H,Tq), p, rng_state]."""
    out, lse = packed_forward(q, k, v, out_, cu_seqlens_q, cu_seqlens_k, seqused_k_, leftpad_k_, block_table_, alibi_slopes_,
                              max_seqlen_q, max_seqlen_k, p_dropout, softmax_scale, zero_tensors, is_causal,
                              window_size_left, window_size_right, softcap, return_softmax)
    return [out, lse, *_unused(q)]


def packed_forward(q, k, v, out_, cu_seqlens_q, cu_seqlens_k, seqused_k_, leftpad_k_, block_table_, alibi_slopes_,
                   max_seqlen_q, max_seqlen_k, p_dropout, softmax_scale, zero_tensors, is_causal, window_size_left,
                   window_size_right, softcap, return_softmax):
    """varlen_fwd without the two results that carry nothing here."""
    _common_checks(q, k, v, softcap)
    if p_dropout != 0.0:
        raise RuntimeError("FlashAttention on B200 does not support dropout.")
    if return_softmax:
        raise RuntimeError("FlashAttention on B200 does not support return_softmax.")
    if leftpad_k_ is not None:
        raise RuntimeError("FlashAttention on B200 does not support leftpad_k.")
    if cu_seqlens_q.dtype != torch.int32 or (cu_seqlens_k is not None and cu_seqlens_k.dtype != torch.int32):
        raise RuntimeError("cu_seqlens must have dtype int32")
    total_q, hq, d_og = q.shape
    paged = block_table_ is not None
    hkv = k.shape[-2]
    if d_og > 256:
        raise RuntimeError("FlashAttention only supports head dimension at most 256")
    if hq % hkv != 0:
        raise RuntimeError("Number of heads in key/value must divide number of heads in query")
    q, k, v = _pad8(q), _pad8(k), _pad8(v)
    d = q.size(-1)
    batch = cu_seqlens_q.numel() - 1
    out = torch.empty_like(q) if (out_ is None or d != d_og) else out_
    if zero_tensors:
        out.zero_()
    device = q.device
    lse = torch.full((hq, total_q), float("inf"), dtype=torch.float32, device=device)
    table = (0, 0, 0)
    if paged:
        if block_table_.dtype != torch.int32 or block_table_.stride(-1) != 1:
            raise RuntimeError("block_table must be int32 with contiguous last dimension")
        table = (block_table_.data_ptr(), block_table_.stride(0), k.shape[1])
    keep, alibi, alibi_sb = _alibi(alibi_slopes_, batch, hq)
    lse_sh, lse_ss = lse.stride()
    buf = capi.FWD_BLOCK.new(
        *_leaves(q, True), *_leaves(k, not paged), *_leaves(v, not paged), *_leaves(out, True), lse.data_ptr(), 0, lse_sh, lse_ss,
        cu_seqlens_q.data_ptr(), _ptr(cu_seqlens_k), _ptr(seqused_k_) if paged else 0, *table, 0, alibi, alibi_sb,
        batch, max_seqlen_q, max_seqlen_k, total_q, 0 if paged else k.shape[0], hq, hkv, d, v.size(-1), softmax_scale, softcap,
        int(is_causal), _i32(window_size_left), _i32(window_size_right), _dtype_code(q),
        *_NO_TENSOR, *_NO_TENSOR, 0, 0, 0, 0, 0, 0,
        0 if paged else 1, 0, 0, 0, 0, 0, 0, 0, 0, min(k.shape[0], v.shape[0]) if paged else 0,
        capi.raw_stream(device))
    nbytes = capi._fwd_bytes(buf)
    if nbytes:
        ws = capi.workspace(nbytes, device)
        capi.set_workspace(capi.FWD_BLOCK, buf, ws, nbytes)
    capi.launch(capi._call_varlen_fwd, buf, device)
    del keep
    if d != d_og:
        out = out[..., :d_og]
        if out_ is not None:
            out_.copy_(out)
            out = out_
    return out, lse


def kvcache_forward(q, kcache, vcache, k_, v_, seqlens_k_, rotary_cos_, rotary_sin_, cache_batch_idx_,
                    block_table_, alibi_slopes_, out_, softmax_scale, is_causal, window_size_left,
                    window_size_right, softcap, is_rotary_interleaved, num_splits,
                    cu_seqlens_q=None, max_seqlen_q=None, kv_range=None, partials=None, sched_meta=None):
    """Shared by the v2 and v3 kvcache entry points.  q (B,Sq,H,D) or packed (Tq,H,D) with
    cu_seqlens_q.  kv_range=(begin,end) and partials=(o fp32, lse fp32) select the
    cross-device KV-sharded mode, where fp32 partial results are left for a later combine.
    sched_meta: the device blob of get_scheduler_metadata (uint8 or int32 view); the split-KV decode kernels take
    every sequence's keys per split from it (a blob built for another batch, split count or for other lengths is
    ignored on the device, so a stale blob costs balance, never correctness)."""
    _common_checks(q, kcache, vcache, softcap, what="key_cache")
    packed_q = cu_seqlens_q is not None
    if packed_q:
        total_q, hq, d_og = q.shape
        batch = cu_seqlens_q.numel() - 1
        sq = int(max_seqlen_q)
    else:
        batch, sq, hq, d_og = q.shape
        total_q = 0
    paged = block_table_ is not None
    hkv = kcache.shape[2]
    if batch <= 0:
        raise RuntimeError("batch size must be positive")
    if d_og > 256:
        raise RuntimeError("FlashAttention only supports head dimension at most 256")
    if hq % hkv != 0:
        raise RuntimeError("Number of heads in key/value must divide number of heads in query")
    if seqlens_k_ is not None and seqlens_k_.dtype != torch.int32:
        raise RuntimeError("seqlens_k must have dtype int32")
    if paged and (block_table_.dtype != torch.int32 or block_table_.stride(-1) != 1):
        raise RuntimeError("block_table must have dtype int32 and contiguous last dimension")
    if d_og % 8 != 0:
        if k_ is not None:
            raise RuntimeError("appending k/v needs a head dimension that is a multiple of 8")
        q, kcache, vcache = _pad8(q), _pad8(kcache), _pad8(vcache)
    d = q.size(-1)
    device = q.device
    out = torch.empty_like(q) if (out_ is None or d != d_og) else out_
    if packed_q:
        lse = torch.full((hq, total_q), float("inf"), dtype=torch.float32, device=device)
        lse_strides = (0, *lse.stride())
    else:
        lse = torch.empty((batch, hq, sq), dtype=torch.float32, device=device)
        lse_strides = lse.stride()
    new_kv, s_new = _NO_TENSOR + _NO_TENSOR, 0
    if k_ is not None:
        if v_ is None:
            raise RuntimeError("k and v must be passed together")
        if seqlens_k_ is None:
            raise RuntimeError("seqlens_k must be passed when appending k and v")
        if k_.dtype != q.dtype or v_.dtype != q.dtype:
            raise RuntimeError("new k/v must have the query's dtype")
        new_kv, s_new = _leaves(k_) + _leaves(v_), k_.shape[1]
    if paged:
        table = (block_table_.data_ptr(), block_table_.stride(0), kcache.shape[1])
        sk = block_table_.shape[1] * kcache.shape[1]
    else:
        table, sk = (0, 0, 0), kcache.shape[1]
    rotary = (0, 0, 0, 0, 0)
    if rotary_cos_ is not None:
        if k_ is None:
            raise RuntimeError("rotary embedding is only applied when k and v are passed in")
        rc = rotary_cos_.to(q.dtype).contiguous()
        rs = rotary_sin_.to(q.dtype).contiguous()
        rotary = (rc.data_ptr(), rs.data_ptr(), rc.shape[1] * 2, int(is_rotary_interleaved), rc.shape[0])
    kv_begin, kv_end = (0, 0) if kv_range is None else (int(kv_range[0]), int(kv_range[1]))
    part = (0, 0, 0) if partials is None else (1, partials[0].data_ptr(), partials[1].data_ptr())
    if sched_meta is not None:
        capi.require_cuda(sched_meta)
        if sched_meta.dtype not in (torch.uint8, torch.int32) or not sched_meta.is_contiguous():
            raise RuntimeError("scheduler_metadata must be the contiguous uint8 / int32 tensor get_scheduler_metadata returned")
        if sched_meta.numel() * sched_meta.element_size() < 4 * capi.lib.fa_scheduler_metadata_ints(batch) or sched_meta.data_ptr() % 4:
            raise RuntimeError("scheduler_metadata is too small for this batch size")
    keep, alibi, alibi_sb = _alibi(alibi_slopes_, batch, hq)
    buf = capi.FWD_BLOCK.new(
        *_leaves(q, packed_q), *_leaves(kcache), *_leaves(vcache), *_leaves(out, packed_q), lse.data_ptr(), *lse_strides,
        cu_seqlens_q.data_ptr() if packed_q else 0, 0, _ptr(seqlens_k_), *table, _ptr(cache_batch_idx_), alibi, alibi_sb,
        batch, sq, sk, total_q, 0, hq, hkv, d, vcache.size(-1), softmax_scale, softcap,
        int(is_causal), _i32(window_size_left), _i32(window_size_right), _dtype_code(q),
        *new_kv, s_new, *rotary, num_splits, kv_begin, kv_end, *part, 0, 0, _ptr(sched_meta),
        min(kcache.shape[0], vcache.shape[0]), capi.raw_stream(device))
    nbytes = capi._fwd_bytes(buf)
    if nbytes:
        ws = capi.workspace(nbytes, device)
        capi.set_workspace(capi.FWD_BLOCK, buf, ws, nbytes)
    capi.launch(capi._call_kvcache, buf, device)
    del keep
    if d != d_og:
        out = out[..., :d_og]
        if out_ is not None:
            out_.copy_(out)
            out = out_
    return out, lse


def fwd_kvcache(q, kcache, vcache, k_, v_, seqlens_k_, rotary_cos_, rotary_sin_, cache_batch_idx_,
                leftpad_k_, block_table_, alibi_slopes_, out_, softmax_scale, is_causal,
                window_size_left, window_size_right, softcap, is_rotary_interleaved, num_splits):
    """mha_fwd_kvcache (flash_api.cpp:356-637) -> [out, softmax_lse (B,H,Sq)]."""
    if leftpad_k_ is not None:
        raise RuntimeError("FlashAttention on B200 does not support leftpad_k")
    if num_splits < 0:
        raise RuntimeError("num_splits must be >= 0")
    out, lse = kvcache_forward(q, kcache, vcache, k_, v_, seqlens_k_, rotary_cos_, rotary_sin_,
                               cache_batch_idx_, block_table_, alibi_slopes_, out_, softmax_scale, is_causal,
                               window_size_left, window_size_right, softcap, is_rotary_interleaved, num_splits)
    return [out, lse]


def _bwd_common(dout, q, k, v, out, softmax_lse, dq_, dk_, dv_, alibi_slopes_, p_dropout, softmax_scale,
                is_causal, wl, wr, softcap, deterministic, cu_q=None, cu_k=None, max_sq=0, max_sk=0):
    """The three gradients."""
    capi.require_cuda(dout, q, k, v, out, softmax_lse)
    if softcap < 0.0:
        raise RuntimeError("softcap must be non-negative (0.0 disables softcap)")
    if p_dropout != 0.0:
        raise RuntimeError("FlashAttention on B200 does not support dropout.")
    packed = cu_q is not None
    d_og = q.size(-1)
    if d_og % 8 != 0:
        raise RuntimeError("backward needs a head dimension that is a multiple of 8 (the Python API pads it)")
    device = q.device
    dq = torch.empty_like(q) if dq_ is None else dq_
    dk = torch.empty_like(k) if dk_ is None else dk_
    dv = torch.empty_like(v) if dv_ is None else dv_
    # The caller of a backward does not choose how autograd lays out the gradient of the output (a slice of a concatenation):
    # what 16-byte loads cannot read in place is copied.  So are expanded inputs (the gradient of a sum, keys shared by heads),
    # which tile copies cannot read.
    s = dout.stride()
    if s[-1] == 1 and (dout.data_ptr() % 16 or (s[0] | s[1] | s[-2]) % 8):
        dout = dout.clone(memory_format=torch.contiguous_format)
    leaves, copies = [], []
    for t in (dout, q, k, v, out, dq, dk, dv):
        s = t.stride()
        if s[-1] != 1:
            raise RuntimeError("Input tensor must have contiguous last dimension")
        if 0 in s and len(leaves) < 20:                      # one of the five inputs
            t = t.clone(memory_format=torch.contiguous_format)
            copies.append(t)
            s = t.stride()
        leaves += (t.data_ptr(), 0, s[0], s[1]) if packed else (t.data_ptr(), s[0], s[1], s[2])
    if packed:
        total_q, hq, _ = q.shape
        total_k, hkv, _ = k.shape
        if softmax_lse.dim() != 2:
            raise RuntimeError("mha_varlen_bwd: softmax_lse for TND must be a 2D tensor.")
        if softmax_lse.shape != (hq, total_q):
            raise RuntimeError("mha_varlen_bwd: softmax_lse must have shape (nheads, total_q)")
        batch, sq, sk = cu_q.numel() - 1, max_sq, max_sk
        lse_strides = (0, *softmax_lse.stride())
        cu = (cu_q.data_ptr(), cu_k.data_ptr())
    else:
        batch, sq, hq, _ = q.shape
        sk, hkv = k.shape[1], k.shape[2]
        if softmax_lse.shape != (batch, hq, sq):
            raise RuntimeError("softmax_lse must have shape (batch, nheads, seqlen_q)")
        total_q = total_k = 0
        lse_strides = softmax_lse.stride()
        cu = (0, 0)
    if softmax_lse.dtype != torch.float32:
        raise RuntimeError("softmax_lse must be fp32")
    if hq % hkv != 0:
        raise RuntimeError("Number of heads in key/value must divide number of heads in query")
    keep, alibi, alibi_sb = _alibi(alibi_slopes_, batch, hq)
    buf = capi.BWD_BLOCK.new(
        *leaves, softmax_lse.data_ptr(), *lse_strides, *cu, batch, sq, sk, total_q, total_k, hq, hkv, q.size(-1), v.size(-1),
        softmax_scale, softcap, int(is_causal), _i32(wl), _i32(wr), _dtype_code(q), int(deterministic), 0, 0,
        capi.raw_stream(device), alibi, alibi_sb)
    nbytes = capi._bwd_bytes(buf)
    try:                                                     # without room for P and dS tiles the kernels recompute them
        ws = capi.workspace(nbytes if capi.workspace_fits(nbytes, device) else capi._bwd_min_bytes(buf), device)
    except torch.OutOfMemoryError:
        ws = capi.workspace(capi._bwd_min_bytes(buf), device)
    capi.set_workspace(capi.BWD_BLOCK, buf, ws, ws.numel())
    capi.launch(capi._call_varlen_bwd if packed else capi._call_bwd, buf, device)
    del keep, copies
    return dq, dk, dv


def bwd(dout, q, k, v, out, softmax_lse, dq_, dk_, dv_, alibi_slopes_, p_dropout, softmax_scale, is_causal,
        window_size_left, window_size_right, softcap, deterministic, gen_, rng_state):
    """mha_bwd (flash_api.cpp:1279-1328) -> [dq, dk, dv, softmax_d]."""
    dq, dk, dv = _bwd_common(dout, q, k, v, out, softmax_lse, dq_, dk_, dv_, alibi_slopes_, p_dropout, softmax_scale,
                             is_causal, window_size_left, window_size_right, softcap, deterministic)
    batch, sq, hq, _ = q.shape
    return [dq, dk, dv, torch.empty((batch, hq, (sq + 127) // 128 * 128), dtype=torch.float32, device=q.device)]


def varlen_bwd(dout, q, k, v, out, softmax_lse, dq_, dk_, dv_, cu_seqlens_q, cu_seqlens_k, alibi_slopes_,
               max_seqlen_q, max_seqlen_k, p_dropout, softmax_scale, zero_tensors, is_causal,
               window_size_left, window_size_right, softcap, deterministic, gen_, rng_state):
    """mha_varlen_bwd (flash_api.cpp:1092-1277) -> [dq, dk, dv, softmax_d]."""
    dq, dk, dv = _bwd_common(dout, q, k, v, out, softmax_lse, dq_, dk_, dv_, alibi_slopes_, p_dropout, softmax_scale,
                             is_causal, window_size_left, window_size_right, softcap, deterministic,
                             cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k)
    total_q, hq, _ = q.shape
    return [dq, dk, dv, torch.empty((hq, total_q + 128 * (cu_seqlens_q.numel() - 1)), dtype=torch.float32, device=q.device)]
