// Forward attention with capped scores (softcap, no alibi) on the tcgen05 tensor cores, head dims up to 128, ONE 128-row
// query tile a CTA and TWO CTAs an SM, sm_100a.
//
// With the cap the softmax, not the tensor core, bounds the kernel: tanh by its exponential and a division makes three
// special-function operations a score.  The two-tile kernel (fwd_sm100.cu), two softmax warps a scheduler with 128 scores
// a thread and the cap branch on every score, took 432 us at B1 S8192 H16/8 D128 window 1024 bf16; this one 135.  What
// makes the difference:
//  - two threads share a score row (64 scores each: warps 0-3 keys 0-63 of the tile, warps 4-7 keys 64-127), so that four
//    softmax warps of two independent CTAs run on each scheduler, and the start and the end of a CTA run beside the other's
//    tiles.  Without the cap the same kernel is slower than the two-tile one (D = 64 full attention 872 against 799 us,
//    D = 128 1160 against 998): its instructions a score are more, and there they count.
//  - tanh as an odd polynomial on the FMA pipe where all scores of a warp are at most 0.8 of the cap, which leaves one
//    special-function operation a score; above that the exponential form.  Evaluated in fp32 the polynomial is within
//    1.6e-7 of tanh, relative, and 1.0e-7 absolute; 1 - 2 / (1 + e^2y) is within 1.2e-7 absolute with exact steps, 1.8e-7
//    with the approximate exponential and division, and not relative: at small scores, which a large cap multiplies, the
//    polynomial is far better, at 0.8 of the cap the two are close.
//
//   warps 0-7  softmax (thread = row warp % 4 * 32 + lane, half = warp / 4), epilogue
//   warp 8     TMA producer, tensor-memory allocation
//   warp 9     MMA issue
// Tensor memory (256 columns a CTA).  Head dim 64: S 0-127, P 128-191, O 192-255; the scores of the next tile are
// multiplied as soon as these have been read into registers, so that the chain from tile to tile is the softmax alone.
// Head dim 128: S 0-127, O 128-255, and a thread writes its half of P over its own half of S (keys 0-63 to columns 0-31,
// keys 64-127 to columns 64-95).  P V is issued in two groups, the first 32 keys of both halves and then the second.
//
// The exponent base of a row moves when the row maximum has outgrown it by 2^8, as in the two-tile kernel.  The two
// warps that share 32 rows agree on that with one barrier reduction a tile; only when it says yes do they exchange
// maxima through shared memory and rescale O.
//
// Same arithmetic, features and bounded waits as the two-tile kernel.
#include "fwd_sm100_common.cuh"

namespace fa {

using namespace sm100;

__device__ int g_fwd_single_error = 0;

int fwd_single_error_flag(bool clear) {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_fwd_single_error, sizeof(int));
    if (clear) { int z = 0; cudaMemcpyToSymbol(g_fwd_single_error, &z, sizeof(int)); }
    return v;
}

namespace {

template <int D>
struct FwdSingleSmem {
    static constexpr int kSub = 128 * 128;
    static constexpr int kTile = (D / 64) * kSub;            // a Q, K or V tile
    static constexpr int kStages = D == 64 ? 2 : 1;          // K and V buffers: two CTAs have to fit into an SM's 227 KB
    static constexpr int oQ = 0;
    static constexpr int oK = oQ + kTile;
    static constexpr int oV = oK + kStages * kTile;
    static constexpr int oMax = oV + kStages * kTile;        // [2 halves][128 rows] floats: row maxima
    static constexpr int oSum = oMax + 2 * 128 * 4;          // the same for the row sums at the end
    static constexpr int oBar = oSum + 2 * 128 * 4;
    static constexpr int kBytes = oBar + 256;
};
static_assert(2 * (FwdSingleSmem<64>::kBytes + 1024 + 1024) <= 228 * 1024 && 2 * (FwdSingleSmem<128>::kBytes + 1024 + 1024) <= 228 * 1024, "two CTAs an SM");

// F/E: K or V buffer full / free; S: scores done; SR: scores read; P0, P1: first / second 32 keys of both halves of P
// stored; PV: P V of a tile done; O: the last of them
enum { N_Q = 0, N_KF0, N_KF1, N_KE0, N_KE1, N_VF0, N_VF1, N_VE0, N_VE1, N_S, N_SR, N_P0, N_P1, N_PV, N_O, N_DRAIN, N_COUNT };

// true in every thread of the 64 that name barrier `id` when `pred` holds in any of them
__device__ __forceinline__ bool pair_any(int id, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %2, 0;\n\t"
        "barrier.cta.red.or.pred p, %1, 64, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r) : "r"(id), "r"((uint32_t)pred) : "memory");
    return r != 0;
}

// tanh(y) as y times a polynomial in y^2, fitted for the least maximum relative error on |y| <= kTanhSmall: 6.7e-8 with these
// coefficients in exact arithmetic, 1.6e-7 evaluated in fp32
constexpr float kTanhSmall = 0.8f;
__device__ __forceinline__ float2 tanh_small2(float2 y) {
    const float2 t = mul2(y, y);
    auto c2 = [](float c) { return make_float2(c, c); };
    float2 q = fma2(t, c2(-0.004355299286544323f), c2(0.01909329928457737f));
    q = fma2(q, t, c2(-0.05311431363224983f));
    q = fma2(q, t, c2(0.13321048021316528f));
    q = fma2(q, t, c2(-0.3333267569541931f));
    q = fma2(q, t, c2(0.9999999403953552f));
    return mul2(q, y);
}
// tanh(y) for any y2e = 2 y log2(e): 1 - 2 / (1 + e^(2y)), absolute error about 1.8e-7
__device__ __forceinline__ float tanh_any(float y2e) { return 1.f - __fdividef(2.f, 1.f + ex2_approx(y2e)); }

template <typename T, int D>
__global__ void __launch_bounds__(320, 2) fwd_single_sm100_kernel(const __grid_constant__ Sm100FwdArgs a) {
    using L = FwdSingleSmem<D>;
    constexpr int NSUB = D / 64;
    constexpr int KSTEPS = D / 16;
    constexpr int NST = L::kStages;
    constexpr bool kOwnP = D == 64;                          // P has columns of its own (see the head of the file)
    constexpr uint32_t TMEM_COLS = 256, COL_P = kOwnP ? 128 : 0, COL_O = kOwnP ? 192 : 128;
    constexpr uint32_t P_HALF = kOwnP ? 32 : 64;             // columns from the first to the second half of P
    constexpr int FMT = Elem<T>::kDtype == FA_BF16 ? 1 : 0;
    constexpr uint32_t IDESC_QK = umma_idesc(FMT, 128, 128, 0, 0);
    constexpr uint32_t IDESC_PV = umma_idesc(FMT, 128, D, 0, 1);
    constexpr float kRescaleThreshold = 8.f;

    extern __shared__ unsigned char smem_raw[];
    const uint32_t sbase = (smem_addr(smem_raw) + 1023u) & ~1023u;
    unsigned char* sgen = smem_raw + (sbase - smem_addr(smem_raw));
    const uint32_t sQ = sbase + L::oQ, sK = sbase + L::oK, sV = sbase + L::oV;
    const uint32_t bars = sbase + L::oBar;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + L::oBar + 8 * N_COUNT);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sgen + L::oBar + 8 * N_COUNT + 8);
    auto bar = [&](int i) { return bars + 8u * i; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // Grid order and tile rows as in the two-tile kernel (see there)
    const int pair = blockIdx.z * a.chunk + blockIdx.x;
    if (pair >= a.b * a.nheads_grid) return;
    const int b = pair / a.nheads_grid, hg = pair % a.nheads_grid;
    const int gq = a.gq;
    const int qpt = 128 / gq;                                // query positions of the tile
    const int hk = gq > 1 ? hg : hg / (a.hq / a.hkv);
    const int h0 = gq > 1 ? hk * gq : hg;                    // head of tile row 0
    const int split = (int)blockIdx.y % a.nsplit;
    const int mblk = (int)gridDim.y / a.nsplit - 1 - (int)blockIdx.y / a.nsplit;
    int q_off = 0, k_off = 0, sq = a.sq, sk = a.sk;
    if (a.cu_q) { q_off = a.cu_q[b]; sq = a.cu_q[b + 1] - q_off; k_off = a.cu_k[b]; sk = a.cu_k[b + 1] - k_off; }
    if (a.seqused_k) sk = (int)max(0LL, min((long long)a.seqused_k[b] + a.s_new, (long long)a.sk));
    const int m0 = mblk * qpt;                               // first query position of the CTA
    if (m0 >= sq) return;
    if (g_fwd_single_error) return;
    const int wl = a.wl, wr = a.causal ? 0 : a.wr;
    const int rows = min(128, (sq - m0) * gq);               // tile rows in use

    int lo_first, hi_first, lo_last, hi_last;
    window_bounds(m0, sq, sk, wl, wr, lo_first, hi_first);
    window_bounds(m0 + (rows - 1) / gq, sq, sk, wl, wr, lo_last, hi_last);
    int t_lo = lo_first / 128, t_hi = hi_last < 0 ? 0 : hi_last / 128 + 1;
    if (sk <= 0 || lo_first >= sk) { t_lo = 0; t_hi = 0; }
    if (a.nsplit > 1) {                                      // this split's share of the key tiles
        t_lo = max(t_lo, split * (a.keys_per_split / 128));
        t_hi = min(t_hi, (split + 1) * (a.keys_per_split / 128));
    }
    const int ntiles = max(0, t_hi - t_lo);

    // output row, LSE slot and row in the partial buffers of tile row t
    auto out_row = [&](int t) -> T* {
        return reinterpret_cast<T*>(a.o) + (a.cu_q ? 0 : (int64_t)b * a.o_sb) + (int64_t)(q_off + m0 + t / gq) * a.o_ss + (int64_t)(h0 + t % gq) * a.o_sh;
    };
    auto lse_slot = [&](int t) -> float* {
        return a.lse + (a.cu_q ? 0 : (int64_t)b * a.lse_sb) + (int64_t)(h0 + t % gq) * a.lse_sh + (int64_t)(q_off + m0 + t / gq) * a.lse_ss;
    };
    auto part_row = [&](int t) -> int64_t {
        return (int64_t)split * a.rows_all + ((int64_t)b * a.sq + m0 + t / gq) * a.hq + h0 + t % gq;
    };

    if (ntiles == 0) {
        if (tid < rows) {
            if (a.nsplit > 1) {                              // an empty split: weight zero in the combine, O never read
                a.lse_part[part_row(tid)] = -INFINITY;
            } else {
                const uint4 z = make_uint4(0, 0, 0, 0);
                T* orow = out_row(tid);
#pragma unroll
                for (int c = 0; c < D / 8; ++c)
                    if (c * 8 < a.d) reinterpret_cast<uint4*>(orow)[c] = z;
                if (a.lse) *lse_slot(tid) = INFINITY;
            }
        }
        return;
    }

    if (tid == 0) {
        for (int i = 0; i < N_COUNT; ++i) mbar_init(bar(i), (i == N_P0 || i == N_P1 || i == N_SR) ? 256u : 1u);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 8) {
        tmem_alloc(smem_addr(tmem_slot), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    int* err = &g_fwd_single_error;

    if (warp == 8) {
        if (lane == 0) {
            tma_prefetch_desc(&a.tq); tma_prefetch_desc(&a.tk); tma_prefetch_desc(&a.tv);
            mbar_expect_tx(bar(N_Q), L::kTile);
#pragma unroll
            for (int s = 0; s < NSUB; ++s) tma_load_4d(sQ + s * L::kSub, &a.tq, bar(N_Q), s * 64, h0, (a.cu_q ? q_off : 0) + m0, a.cu_q ? 0 : b);
            // where key tile j lives: as in the two-tile kernel
            const int32_t* btab = a.block_table ? a.block_table + (int64_t)b * a.bt_stride : nullptr;
            const int kbatch = a.cu_q ? 0 : (a.cache_batch_idx ? a.cache_batch_idx[b] : b);
            auto load = [&](uint32_t dst, const CUtensorMap* map, uint32_t full, int krow, int kouter, int krow2, int kouter2) {
                mbar_expect_tx(full, L::kTile);
#pragma unroll
                for (int s = 0; s < NSUB; ++s) {
                    tma_load_4d(dst + s * L::kSub, map, full, s * 64, hk, krow, kouter);
                    if (a.kv_box == 64) tma_load_4d(dst + s * L::kSub + 64 * 128, map, full, s * 64, hk, krow2, kouter2);
                }
            };
            bool ok = true;
            for (int j = 0; j < ntiles && ok; ++j) {
                const int st = j % NST, use = j / NST;
                int krow = (a.cu_q ? k_off : 0) + (t_lo + j) * 128, kouter = kbatch, krow2 = 0, kouter2 = 0;
                if (btab) {
                    const int pos = (t_lo + j) * 128;
                    kouter = btab[pos / a.page_size];
                    krow = pos % a.page_size;
                    if (a.kv_box == 64) {
                        const bool in_table = (pos + 64) / a.page_size < a.bt_stride;
                        kouter2 = in_table ? btab[(pos + 64) / a.page_size] : kouter;
                        krow2 = in_table ? (pos + 64) % a.page_size : krow;
                    }
                }
                if (use > 0) ok = mbar_wait(bar(N_KE0 + st), (use - 1) & 1, abort_flag, err, 81);
                if (!ok) break;
                load(sK + st * L::kTile, &a.tk, bar(N_KF0 + st), krow, kouter, krow2, kouter2);
                if (use > 0) ok = mbar_wait(bar(N_VE0 + st), (use - 1) & 1, abort_flag, err, 82);
                if (!ok) break;
                load(sV + st * L::kTile, &a.tv, bar(N_VF0 + st), krow, kouter, krow2, kouter2);
            }
        }
    } else if (warp == 9) {
        const uint64_t dQ = umma_desc(sQ, 16, 1024), dK = umma_desc(sK, 16, 1024), dV = umma_desc(sV, L::kSub, 1024);
        auto issue_qk = [&](int j) {
            umma_ss_scores<KSTEPS, L::kSub>(tmem, dQ, umma_desc_at(dK, (j % NST) * L::kTile), IDESC_QK);
            umma_commit_w(bar(N_S));
            umma_commit_w(bar(N_KE0 + j % NST));
        };
        bool ok = mbar_wait(bar(N_Q), 0, abort_flag, err, 83);
        if (ok) ok = mbar_wait(bar(N_KF0), 0, abort_flag, err, 84);
        if (ok) { tc_fence_after(); issue_qk(0); }
        for (int j = 0; j < ntiles && ok; ++j) {
            const int st = j % NST;
            const bool more = j + 1 < ntiles;
            if (kOwnP && more) {                             // the next scores as soon as these have been read
                ok = mbar_wait(bar(N_KF0 + (j + 1) % NST), ((j + 1) / NST) & 1, abort_flag, err, 87);
                if (ok) ok = mbar_wait(bar(N_SR), j & 1, abort_flag, err, 88);
                if (!ok) break;
                tc_fence_after();
                issue_qk(j + 1);
            }
            // the copies are waited for first, so that only the MMAs stand between "P is ready" and the tensor core
            ok = mbar_wait(bar(N_VF0 + st), (j / NST) & 1, abort_flag, err, 86);
            if (!kOwnP && ok && more) ok = mbar_wait(bar(N_KF0 + (j + 1) % NST), ((j + 1) / NST) & 1, abort_flag, err, 87);
            if (!ok) break;
            if (a.seqused_k && (t_lo + j) * 128 + 128 > sk) {
                // cache rows past the sequence may hold NaN patterns and 0 x NaN is NaN: the V rows that the copy fetched
                // are cleared (rows past the capacity of a dense cache were zero-filled by the copy)
                const int first = max(0, sk - (t_lo + j) * 128);
                const int last = a.block_table ? 128 : min(128, a.sk - (t_lo + j) * 128);
#pragma unroll
                for (int sub = 0; sub < NSUB; ++sub)
                    for (int idx = first * 8 + lane; idx < last * 8; idx += 32)
                        *reinterpret_cast<uint4*>(sgen + L::oV + st * L::kTile + sub * L::kSub + idx * 16) = make_uint4(0, 0, 0, 0);
                fence_proxy_async_smem();
                __syncwarp();
            }
            ok = mbar_wait(bar(N_P0), j & 1, abort_flag, err, 85);
            if (!ok) break;
            tc_fence_after();
            // 16 keys = 8 columns of P and 2048 bytes of V a step; keys 0-31 and 64-95, then 32-63 and 96-127
            const uint64_t bv = umma_desc_at(dV, st * L::kTile);
            umma_ts_quad<0, 8, P_HALF, P_HALF + 8, 0, 128, 512, 640>(tmem + COL_O, tmem + COL_P, bv, IDESC_PV, j > 0);
            ok = mbar_wait(bar(N_P1), j & 1, abort_flag, err, 91);
            if (!ok) break;
            tc_fence_after();
            umma_ts_quad<16, 24, P_HALF + 16, P_HALF + 24, 256, 384, 768, 896>(tmem + COL_O, tmem + COL_P, bv, IDESC_PV, 1);
            if (!kOwnP && more) issue_qk(j + 1);             // over S and P of tile j, behind the P V that reads P
            if (kOwnP && more) umma_commit_w(bar(N_PV));
            if (!more) umma_commit_w(bar(N_O));
            umma_commit_w(bar(N_VE0 + st));
        }
        // no arrive of a commit may land after the CTA has left: wait for a last one (see the two-tile kernel)
        if (ok) {
            umma_commit_w(bar(N_DRAIN));
            ok = mbar_wait(bar(N_DRAIN), 0, abort_flag, err, 93);
        }
    } else {
        const int quarter = warp & 3, half = warp >> 2;
        const int r = quarter * 32 + lane;
        const int bid = 1 + quarter;                         // named barrier of the two warps that share these rows
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t t_s = tmem + lane_base + half * 64;
        const uint32_t t_p = tmem + lane_base + COL_P + half * P_HALF;
        const uint32_t t_o = tmem + lane_base + COL_O + half * (D / 2);     // the half of O this thread rescales and stores
        float* s_max = reinterpret_cast<float*>(sgen + L::oMax);
        float* s_sum = reinterpret_cast<float*>(sgen + L::oSum);
        const int qi = m0 + r / gq;
        int klo = 1, khi = 0;
        if (r < rows) window_bounds(qi, sq, sk, wl, wr, klo, khi);
        // key range that every / any row of this warp sees (rows past the end see nothing and only lose the fast path)
        const int wfirst = quarter * 32, wlast = min(wfirst + 31, rows - 1);
        int all_lo = 1, all_hi = 0, any_lo = 1, any_hi = 0;
        if (wfirst < rows) {
            int tl, th;
            window_bounds(m0 + wfirst / gq, sq, sk, wl, wr, any_lo, all_hi);
            window_bounds(m0 + wlast / gq, sq, sk, wl, wr, tl, th);
            all_lo = tl; any_hi = th;
        }
        float m_used = -INFINITY, l_run = 0.f;
        const float cap_out = a.softcap * kLog2e;
        const float cap_in2 = a.cap_in * 2.f * kLog2e;
        bool ok = true;
        for (int j = 0; j < ntiles; ++j) {
            const int n0 = (t_lo + j) * 128 + half * 64;     // first key of this thread's 64
            ok = ok && mbar_wait(bar(N_S), j & 1, abort_flag, err, 89);
            tc_fence_after();
            // warp-uniform: every row of the warp sees every key / no row sees any key of chunk c
            const bool full = n0 >= all_lo && n0 + 63 <= all_hi;
            auto dead = [&](int c) { return n0 + c * 32 > any_hi || n0 + c * 32 + 31 < any_lo; };
            uint32_t sreg[2][32];
            tmem_ld32(t_s, sreg[0]);
            tmem_ld32(t_s + 32, sreg[1]);
            tmem_wait_ld();
            if constexpr (kOwnP) { tc_fence_before(); mbar_arrive_relaxed(bar(N_SR)); }
            float a0 = 0.f, a1 = 0.f;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    a0 = fmaxf(fmaxf(a0, fabsf(__uint_as_float(sreg[c][i]))), fabsf(__uint_as_float(sreg[c][i + 1])));
                    a1 = fmaxf(fmaxf(a1, fabsf(__uint_as_float(sreg[c][i + 2]))), fabsf(__uint_as_float(sreg[c][i + 3])));
                }
            }
            // every score of the warp is in the range of the tanh polynomial
            const bool small = __all_sync(0xffffffffu, fmaxf(a0, a1) * a.cap_in <= kTanhSmall);
            auto seen = [&](int c, int i) { const int col = n0 + c * 32 + i; return col >= klo && col <= khi; };
            if (!full) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (!seen(c, i)) sreg[c][i] = 0xff800000u;     // -inf
                }
            }
            float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    mx0 = fmaxf(fmaxf(mx0, __uint_as_float(sreg[c][i])), __uint_as_float(sreg[c][i + 1]));
                    mx1 = fmaxf(fmaxf(mx1, __uint_as_float(sreg[c][i + 2])), __uint_as_float(sreg[c][i + 3]));
                    mx2 = fmaxf(fmaxf(mx2, __uint_as_float(sreg[c][i + 4])), __uint_as_float(sreg[c][i + 5]));
                    mx3 = fmaxf(fmaxf(mx3, __uint_as_float(sreg[c][i + 6])), __uint_as_float(sreg[c][i + 7]));
                }
            }
            float m_loc = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
            // the cap is monotone; log2 domain.  It makes a finite score of an infinite one, so that -inf only stands for a row
            // that sees none of these keys.
            m_loc = klo <= khi && klo <= n0 + 63 && khi >= n0 ? cap_out * tanh_any(m_loc * cap_in2) : -INFINITY;
            // one of the 64 threads moves its base (or gave up waiting): both warps take the slow way
            if (pair_any(bid, !ok || m_loc > m_used + kRescaleThreshold)) {
                s_max[half * 128 + r] = m_loc;
                if (pair_any(bid, !ok)) { ok = false; break; }
                const float m_row = fmaxf(m_loc, s_max[(half ^ 1) * 128 + r]);
                if (m_used == -INFINITY) m_used = m_row;
                if (j > 0 && __any_sync(0xffffffffu, m_row > m_used + kRescaleThreshold)) {
                    if constexpr (kOwnP) {                   // P V of the last tile may still be running
                        ok = ok && mbar_wait(bar(N_PV), (j - 1) & 1, abort_flag, err, 92);
                        tc_fence_after();
                    }
                    const float m_next = fmaxf(m_used, m_row);
                    const float alpha = m_used == -INFINITY ? 1.f : ex2_approx(m_used - m_next);
                    m_used = m_next;
                    l_run *= alpha;
#pragma unroll
                    for (int c = 0; c < D / 32; ++c) {
                        uint32_t oreg[16];
                        tmem_ld16(t_o + c * 16, oreg);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) oreg[i] = __float_as_uint(__uint_as_float(oreg[i]) * alpha);
                        tmem_st16(t_o + c * 16, oreg);
                    }
                }
            }
            const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
            const float2 nm2 = make_float2(neg_m, neg_m);
            float2 sum_a = make_float2(0.f, 0.f), sum_b = make_float2(0.f, 0.f);
            // exponentials of the 64 keys; SMALL: the tanh polynomial holds for all of them; MASK: keys that the row does not
            // see become exact zeros
            auto exp_phase = [&](auto small_c, auto mask_c) {
                constexpr bool SMALL = decltype(small_c)::value, MASK = decltype(mask_c)::value;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t preg[16];
                    if (MASK && dead(c)) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) preg[i] = 0u;
                    } else {
                        static_for<0, 16>([&](auto pi) {
                            constexpr int i = 2 * pi.value;
                            const float2 s = make_float2(__uint_as_float(sreg[c][i]), __uint_as_float(sreg[c][i + 1]));
                            const float2 th = SMALL ? tanh_small2(mul2(s, make_float2(a.cap_in, a.cap_in)))
                                                    : make_float2(tanh_any(s.x * cap_in2), tanh_any(s.y * cap_in2));
                            const float2 xv = fma2(th, make_float2(cap_out, cap_out), nm2);
                            float2 pv = make_float2(ex2_approx(xv.x), ex2_approx(xv.y));
                            if constexpr (MASK) {            // the cap has made a finite score of the mask's -inf
                                pv.x = seen(c, i) ? pv.x : 0.f;
                                pv.y = seen(c, i + 1) ? pv.y : 0.f;
                            }
                            if constexpr (pi.value & 1) sum_b = add2(sum_b, pv); else sum_a = add2(sum_a, pv);
                            preg[pi.value] = Elem<T>::pack(pv.x, pv.y);
                        });
                    }
                    if (kOwnP && c == 0 && j > 0) {          // P of the last tile has been read
                        ok = ok && mbar_wait(bar(N_PV), (j - 1) & 1, abort_flag, err, 94);
                        tc_fence_after();
                    }
                    tmem_st16(t_p + c * 16, preg);
                    tmem_wait_st();
                    tc_fence_before();
                    mbar_arrive_relaxed(bar(c ? N_P1 : N_P0));
                }
            };
            if (full && small) exp_phase(std::true_type{}, std::false_type{});
            else if (full) exp_phase(std::false_type{}, std::false_type{});
            else if (small) exp_phase(std::true_type{}, std::true_type{});
            else exp_phase(std::false_type{}, std::true_type{});
            l_run += (sum_a.x + sum_b.x) + (sum_a.y + sum_b.y);
        }
        // the two halves of the row sum (after a break both warps come here with `ok` false)
        s_sum[half * 128 + r] = l_run;
        ok = !pair_any(bid, !ok);
        const float l_tot = s_sum[r] + s_sum[128 + r];
        if (ok) ok = mbar_wait(bar(N_O), 0, abort_flag, err, 90);
        if (ok) {
            tc_fence_after();
            const float inv = l_tot > 0.f ? 1.f / l_tot : 0.f;
            T* orow = out_row(r) + half * (D / 2);
            float* prow = a.nsplit > 1 ? a.o_part + part_row(r) * a.d + half * (D / 2) : nullptr;
            const int left = a.d - half * (D / 2);           // columns of the call's head dim from here on
#pragma unroll
            for (int c = 0; c < D / 64; ++c) {
                uint32_t oreg[32];
                tmem_ld32(t_o + c * 32, oreg);
                tmem_wait_ld();
                if (r < rows && prow) {
#pragma unroll
                    for (int v = 0; v < 8; ++v)
                        if (c * 32 + v * 4 < left)
                            reinterpret_cast<float4*>(prow + c * 32)[v] = make_float4(__uint_as_float(oreg[4 * v]) * inv, __uint_as_float(oreg[4 * v + 1]) * inv,
                                                                                     __uint_as_float(oreg[4 * v + 2]) * inv, __uint_as_float(oreg[4 * v + 3]) * inv);
                } else if (r < rows) {
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        uint4 pk;
                        pk.x = Elem<T>::pack(__uint_as_float(oreg[8 * v + 0]) * inv, __uint_as_float(oreg[8 * v + 1]) * inv);
                        pk.y = Elem<T>::pack(__uint_as_float(oreg[8 * v + 2]) * inv, __uint_as_float(oreg[8 * v + 3]) * inv);
                        pk.z = Elem<T>::pack(__uint_as_float(oreg[8 * v + 4]) * inv, __uint_as_float(oreg[8 * v + 5]) * inv);
                        pk.w = Elem<T>::pack(__uint_as_float(oreg[8 * v + 6]) * inv, __uint_as_float(oreg[8 * v + 7]) * inv);
                        if (c * 32 + v * 8 < left) reinterpret_cast<uint4*>(orow + c * 32)[v] = pk;
                    }
                }
            }
            if (half == 0 && r < rows && prow) a.lse_part[part_row(r)] = l_tot > 0.f ? (m_used + log2f(l_tot)) * kLn2 : -INFINITY;
            else if (half == 0 && r < rows && a.lse) *lse_slot(r) = l_tot > 0.f ? (m_used + log2f(l_tot)) * kLn2 : INFINITY;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

template <typename T, int D>
int launch_t(const fa_fwd_params& p, Sm100FwdArgs& a) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(p.stream);
    auto kern = fwd_single_sm100_kernel<T, D>;
    const int smem = FwdSingleSmem<D>::kBytes + 1024;
    if (int e = cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "cudaFuncSetAttribute")) return e;
    if (int e = cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared), "cudaFuncSetAttribute")) return e;
    const int qpc = 128 / a.gq;                              // query positions of a CTA
    const unsigned nbx = (unsigned)(((p.sq + qpc - 1) / qpc) * a.nsplit);
    a.nheads_grid = a.gq > 1 ? p.hkv : p.hq;
    a.chunk = grid_chunk((int64_t)p.b * a.nheads_grid, (int64_t)p.sk * p.d * 4);
    dim3 grid(a.chunk, nbx, (unsigned)(((int64_t)p.b * a.nheads_grid + a.chunk - 1) / a.chunk));
    kern<<<grid, 320, smem, st>>>(a);
    mark_kernel(st);
    return cuda_ok(cudaGetLastError(), "fwd_single_sm100 launch");
}
}  // namespace

int launch_fwd_single_sm100(const fa_fwd_params& p, Sm100FwdArgs& a) {
    if (p.dtype == FA_F16) return p.d <= 64 ? launch_t<__half, 64>(p, a) : launch_t<__half, 128>(p, a);
    return p.d <= 64 ? launch_t<__nv_bfloat16, 64>(p, a) : launch_t<__nv_bfloat16, 128>(p, a);
}

}  // namespace fa
