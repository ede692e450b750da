// Argument block shared by the tcgen05 forward kernels: two query tiles a CTA and head dims above 128 (fwd_sm100.cu),
// capped scores (fwd_single_sm100.cu).
#pragma once
#include "fa_utils.cuh"
#include "fa_internal.h"
#include "sm100_ptx.cuh"

namespace fa {

struct alignas(64) Sm100FwdArgs {
    CUtensorMap tq, tk, tv;
    void* o;
    float* lse;
    int64_t o_sb, o_ss, o_sh;
    int64_t lse_sb, lse_sh, lse_ss;
    const int32_t* cu_q;
    const int32_t* cu_k;
    // KV-cache calls: device-resident lengths, page table, cache row of a batch entry
    const int32_t* seqused_k;
    const int32_t* block_table;
    const int32_t* cache_batch_idx;
    int64_t bt_stride;
    int page_size, s_new;
    int b, sq, sk, hq, hkv;
    int d;                               // the call's head dim (a multiple of 8): the kernels run the next of 64 / 128 / 192 / 256, the tile copies
                                         // zero-fill the columns past d and the epilogue stores d columns
    float scale_log2;
    int causal, wl, wr;
    // score transforms of the BIAS instantiation: softcap (0 = off) and alibi slopes ((hq) or (b,hq), null = off)
    float softcap, cap_in;               // cap_in = scale / softcap
    const float* alibi;
    int64_t alibi_sb;
    int kv_box;                          // rows of one K/V copy: 128, or 64 when pages are an odd multiple of 64 tokens
    int gq;                              // two-tile kernel: 1, or the query group size when a KV head's heads are stacked into the tile rows
    // split-KV (two-tile kernel, cache calls): split s of a sequence takes keys [s * keys_per_split, (s + 1) * ...) and
    // leaves a normalised fp32 partial output and its LSE for the combine kernel (nsplit = 1: final output directly)
    int nsplit, keys_per_split;          // keys_per_split is a multiple of 128
    float* o_part;                       // (nsplit, rows_all, D), rows_all = batch * sq * hq, row = (b * sq + qpos) * hq + head
    float* lse_part;                     // (nsplit, rows_all)
    int64_t rows_all;
    int chunk, nheads_grid;              // grid order, see the kernels: (batch entry, head) pairs a chunk; heads of the grid
};

// capped scores, head dims up to 128: one query tile a CTA, two CTAs an SM (fwd_single_sm100.cu)
int launch_fwd_single_sm100(const fa_fwd_params& p, Sm100FwdArgs& a);
int fwd_single_error_flag(bool clear);

}  // namespace fa
