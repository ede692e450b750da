// Backward attention for head dims above 128 (kernels for 192 and 256) on the tcgen05 tensor cores, sm_100a.
//
// The dK/dV kernel of the smaller head dims keeps dK and dV in tensor memory; at 256 columns each they would fill it
// and leave no room for scores.  So the two halves of the backward are separated:
//
//  score kernel     S^T = K Q^T and dP^T = V dO^T of whole 128 x 128 tiles, P^T = exp(S^T - LSE) and
//                   dS^T = P^T o (dP^T - D) rounded to the input type, both written to a workspace as 32 KiB tiles.
//                   Nothing is accumulated, so a CTA may take any run of query blocks of its key block.
//  gradient kernel  one CTA per 128-row block of dV, dK or dQ sums one product of stored tiles and input rows:
//                   dV = sum P^T dO, dK = scale sum dS^T Q, dQ = scale sum dS K.
//
// Ten 128^3 products a tile at head dim 256, none of them twice.  The mma.sync kernels that served these head dims
// recompute the scores for dQ and reached 43 TFLOP/s counted: 1397 us with the delta pass at B2 S2048 H8/4 D256 causal
// bf16, against 133 us for this pair (648 TFLOP/s; 1002 us = 686 at B1 S8192 H8, 1945 us = 707 at B2 S4096 H16/4 full).
// Both kernels are bound by what an SM can read from L2: the score kernel loads 128 KiB and stores 64 KiB a tile for
// 2048 cycles of MMA, the gradient kernel loads 96 KiB for 1024 (8.3 TB/s over the GPU).  From HBM that would be slower
// still, so KV heads are processed in groups whose tiles stay in L2 (kWideGroupBytes).
//
// Math and rounding points as in bwd_sm100.cu (fag_kernel.cpp:400-465, fag_epilogue_op.hpp:1287-1322, :1394,
// :1447-1480, fag_epilogue_post.hpp:149-200).  No atomics, fixed order of sums; all waits are bounded.
#include "bwd_sm100_common.cuh"
#include "bwd_wide_tiles.h"

namespace fa {

using namespace sm100;

__device__ int g_bwd_wide_error = 0;

int bwd_wide_error_flag(bool clear) {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_bwd_wide_error, sizeof(int));
    if (clear) { int z = 0; cudaMemcpyToSymbol(g_bwd_wide_error, &z, sizeof(int)); }
    return v;
}

namespace {

constexpr int kSub = 128 * 128;                              // bytes of a [128 rows x 64 columns] sub-tile

struct alignas(64) WideBwdArgs {
    CUtensorMap tq, tdo, tk, tv;
    void *dq, *dk, *dv;
    int64_t dq_sb, dq_ss, dq_sh, dk_sb, dk_ss, dk_sh, dv_sb, dv_ss, dv_sh;
    const float* lse;
    int64_t lse_sb, lse_sh, lse_ss;
    const float* delta;                  // [token][head]
    const int32_t* cu_q;
    const int32_t* cu_k;
    int b, sq, sk, hq, hkv, d;           // d: the call's head dim, a multiple of 8 (tile copies zero-fill the columns past it)
    float scale, scale_log2;
    WideGrid grid;                       // blocks a head and the masks that say which of them meet
    float softcap, cap_in, cap_out;      // cap_in = scale / softcap, cap_out = softcap log2(e)
    const float* alibi;
    int64_t alibi_sb;
    // stored tiles of the (batch entry, KV head) pairs unit0 .. of this launch: tile (pair, head of the group, key block,
    // query block) = 128 keys x 128 queries as [16 chunks of 8 queries][128 keys][8 queries]
    unsigned char *p_tiles, *ds_tiles;
    int unit0, steps_per_cta;
};

struct Geometry {
    int b, hk, q_off, k_off, sq, sk;
    __device__ Geometry(const WideBwdArgs& a, int unit) : b(unit / a.hkv), hk(unit % a.hkv), q_off(0), k_off(0), sq(a.sq), sk(a.sk) {
        if (a.cu_q) { q_off = a.cu_q[b]; sq = a.cu_q[b + 1] - q_off; k_off = a.cu_k[b]; sk = a.cu_k[b + 1] - k_off; }
    }
};

// ------------------------------------------------------------------------------------------------------
// Scores.  K and V of the key block stay in shared memory; Q and dO arrive as [128 x 64] sub-tiles through one ring
// (each is read by four MMAs and released), so the ring holds five sub-tiles however wide the head is.  S^T and dP^T
// have two buffers each in tensor memory: the products of step s + 1 run during the element-wise work of step s.
//   warps 0-15 element-wise (thread = key row, 32 query columns), warp 16 TMA, warp 17 MMA, warp 18 completes the block
// ------------------------------------------------------------------------------------------------------
constexpr int kRing = 5;
enum { WB_K = 0, WB_V, WB_RF0, WB_RE0 = WB_RF0 + kRing, WB_S0 = WB_RE0 + kRing, WB_S1, WB_DP0, WB_DP1, WB_TE0, WB_TE1, WB_COUNT };

template <int D>
struct ScoreSmem {
    static constexpr int kTile = (D / 64) * kSub;
    static constexpr int oK = 0, oV = kTile, oRing = 2 * kTile;
    static constexpr int oVec = oRing + kRing * kSub;        // per element-wise warp: 2 x (32 -lse2 + 32 -delta)
    static constexpr int oBar = oVec + 16 * 128 * 4;
    static constexpr int kBytes = oBar + 8 * WB_COUNT + 16;
};

template <typename T, int D, bool BIAS>
__global__ void __launch_bounds__(608, 1) bwd_wide_scores_kernel(const __grid_constant__ WideBwdArgs a) {
    using L = ScoreSmem<D>;
    constexpr int NSUB = D / 64;
    constexpr uint32_t TMEM_COLS = 512, COL_S = 0, COL_DP = 256;     // two 128-column buffers each
    constexpr int FMT = Elem<T>::kDtype == FA_BF16 ? 1 : 0;
    constexpr uint32_t IDESC = umma_idesc(FMT, 128, 128, 0, 0);

    extern __shared__ unsigned char smem_raw[];
    const uint32_t sbase = (smem_addr(smem_raw) + 1023u) & ~1023u;
    unsigned char* sgen = smem_raw + (sbase - smem_addr(smem_raw));
    const uint32_t bars = sbase + L::oBar;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + L::oBar + 8 * WB_COUNT);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sgen + L::oBar + 8 * WB_COUNT + 8);
    auto bar = [&](int i) { return bars + 8u * i; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int local = blockIdx.x, nb = blockIdx.y;
    const Geometry geo(a, a.unit0 + local);
    const int b = geo.b, hk = geo.hk, sq = geo.sq, sk = geo.sk, n0 = nb * 128;
    if (n0 >= sk) return;
    if (g_bwd_wide_error) return;
    const int G = a.hq / a.hkv;
    const int wl = a.grid.wl, wr = a.grid.causal ? 0 : a.grid.wr;
    const int diff = sk - sq;
    const BlockRange qr = wide_query_blocks(a.grid, sq, sk, nb);
    const int mb_lo = qr.lo, nmb = qr.hi - qr.lo;
    const int s_begin = blockIdx.z * a.steps_per_cta;
    const int steps = min(nmb * G - s_begin, a.steps_per_cta);
    if (steps <= 0) return;

    if (tid == 0) {
        for (int i = 0; i < WB_COUNT; ++i) mbar_init(bar(i), i >= WB_TE0 ? 512u : 1u);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 16) { tmem_alloc(smem_addr(tmem_slot), TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    int* err = &g_bwd_wide_error;
    const int bb = a.cu_q ? 0 : b;
    const int q_row0 = a.cu_q ? geo.q_off : 0;

    if (warp == 16) {
        if (lane == 0) {
            tma_prefetch_desc(&a.tq); tma_prefetch_desc(&a.tdo); tma_prefetch_desc(&a.tk); tma_prefetch_desc(&a.tv);
            const int krow = (a.cu_q ? geo.k_off : 0) + n0;
            auto fixed = [&](const CUtensorMap* map, uint32_t dst, int full) {
                mbar_expect_tx(bar(full), L::kTile);
#pragma unroll
                for (int c = 0; c < NSUB; ++c) tma_load_4d(dst + c * kSub, map, bar(full), c * 64, hk, krow, bb);
            };
            bool ok = true;
            int it = 0;                                       // sub-tile count: ring stage it % kRing
            auto stream = [&](const CUtensorMap* map, int h, int qrow) {
#pragma unroll 1
                for (int c = 0; c < NSUB && ok; ++c, ++it) {
                    const int st = it % kRing;
                    if (it >= kRing) ok = mbar_wait(bar(WB_RE0 + st), (it / kRing - 1) & 1, abort_flag, err, 61);
                    if (!ok) break;
                    mbar_expect_tx(bar(WB_RF0 + st), kSub);
                    tma_load_4d(sbase + L::oRing + st * kSub, map, bar(WB_RF0 + st), c * 64, h, qrow, bb);
                }
            };
            fixed(&a.tk, sbase + L::oK, WB_K);
            for (int s = 0; s < steps && ok; ++s) {
                const int h = hk * G + (s_begin + s) / nmb;
                const int qrow = q_row0 + (mb_lo + (s_begin + s) % nmb) * 128;
                stream(&a.tq, h, qrow);
                if (s == 0) fixed(&a.tv, sbase + L::oV, WB_V);
                stream(&a.tdo, h, qrow);
            }
        }
    } else if (warp == 17) {
        const uint64_t dK0 = umma_desc(sbase + L::oK, 16, 1024), dV0 = umma_desc(sbase + L::oV, 16, 1024);
        const uint64_t dR0 = umma_desc(sbase + L::oRing, 16, 1024);
        bool ok = mbar_wait(bar(WB_K), 0, abort_flag, err, 62);
        int it = 0;
        // [128 keys x 128 queries] = fixed operand x the next NSUB sub-tiles of the ring
        auto product = [&](uint32_t d_t, uint64_t fixed0) {
#pragma unroll 1
            for (int c = 0; c < NSUB && ok; ++c, ++it) {
                const int st = it % kRing;
                ok = mbar_wait(bar(WB_RF0 + st), (it / kRing) & 1, abort_flag, err, 63);
                if (!ok) break;
                tc_fence_after();
                umma_ss_group4<0, 2, 4, 6, 0, 2, 4, 6>(d_t, umma_desc_at(fixed0, c * kSub), umma_desc_at(dR0, st * kSub), IDESC, c > 0);
                umma_commit_w(bar(WB_RE0 + st));
            }
        };
        for (int s = 0; s < steps && ok; ++s) {
            const int buf = s & 1;
            if (s >= 2) ok = mbar_wait(bar(WB_TE0 + buf), ((s >> 1) - 1) & 1, abort_flag, err, 64);
            if (!ok) break;
            tc_fence_after();
            product(tmem + COL_S + buf * 128, dK0);
            if (!ok) break;
            umma_commit_w(bar(WB_S0 + buf));
            if (s == 0) ok = mbar_wait(bar(WB_V), 0, abort_flag, err, 65);
            if (!ok) break;
            product(tmem + COL_DP + buf * 128, dV0);
            if (!ok) break;
            umma_commit_w(bar(WB_DP0 + buf));
        }
        // The last release of a ring stage has no waiter, but the element-wise warps wait for the last WB_DP commit, which
        // was issued after it: commits complete in order, so nothing arrives after the CTA has left.
    } else if (warp < 16) {
        const int cg = warp >> 2;
        const int r = (warp & 3) * 32 + lane;                // TMEM lane = key row of the tile
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const int n = n0 + r;
        int qi_lo = 0, qi_hi = sq - 1;                       // query rows that see key n
        if (wr >= 0) qi_lo = max(0, n - diff - wr);
        if (wl >= 0) qi_hi = min(sq - 1, n + wl - diff);
        if (n >= sk) { qi_lo = 1; qi_hi = 0; }
        float* vec0 = reinterpret_cast<float*>(sgen + L::oVec) + warp * 128;
        bool ok = true;
        // -LSE (log2 domain) and -delta of the warp's 32 query columns, one per lane, fetched one step ahead
        auto fetch_vec = [&](int s, float& nl, float& nd) {
            const int h = hk * G + (s_begin + s) / nmb;
            const int i = (mb_lo + (s_begin + s) % nmb) * 128 + cg * 32 + lane;
            nl = -INFINITY; nd = 0.f;
            if (i < sq) {
                const int64_t tok = (int64_t)geo.q_off + i;
                nl = -a.lse[(a.cu_q ? 0 : (int64_t)b * a.lse_sb) + (int64_t)h * a.lse_sh + tok * a.lse_ss] * kLog2e;
                nd = -a.delta[((a.cu_q ? tok : (int64_t)b * a.sq + i)) * a.hq + h];
            }
        };
        float st_l, st_d;
        fetch_vec(0, st_l, st_d);
        const float2 sc2 = make_float2(a.scale_log2, a.scale_log2);
        for (int s = 0; s < steps && ok; ++s) {
            const int buf = s & 1;
            const int g = (s_begin + s) / nmb, m = mb_lo + (s_begin + s) % nmb;
            const int i0 = m * 128 + cg * 32;                // first query row of this thread's 32 columns
            float* vec = vec0 + buf * 64;
            vec[lane] = st_l;
            vec[32 + lane] = st_d;
            __syncwarp();
            if (s + 1 < steps) fetch_vec(s + 1, st_l, st_d);
            // thread's 16-byte chunk of chunk row c: 8 queries of key r (a warp stores 512 contiguous bytes)
            const size_t off = wide_tile_at(a.grid, G, local, g, nb, m) + ((size_t)(cg * 4) * 128 + r) * 16;
            uint4* p_dst = reinterpret_cast<uint4*>(a.p_tiles + off);
            uint4* ds_dst = reinterpret_cast<uint4*>(a.ds_tiles + off);
            ok = mbar_wait(bar(WB_S0 + buf), (s >> 1) & 1, abort_flag, err, 66);
            if (!ok) break;
            tc_fence_after();
            uint32_t pr[32], w[16];
            tmem_ld32(tmem + lane_base + COL_S + buf * 128 + cg * 32, pr);
            tmem_wait_ld();
            const bool inside = __all_sync(0xffffffffu, i0 >= qi_lo && i0 + 31 <= qi_hi);
            // a packed sequence ends inside the tile: how many of the thread's 32 columns are its own
            const bool past_end = a.cu_q && (n0 + 128 > sk || (m + 1) * 128 > sq);
            const int own = n < sk ? sq - i0 : 0;
            float slope = 0.f;
            if constexpr (BIAS) { if (a.alibi) slope = a.alibi[(int64_t)b * a.alibi_sb + hk * G + g] * kLog2e; }
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 nl = *reinterpret_cast<const float4*>(vec + i);
                float2 x01, x23;
                float fac[4] = {1.f, 1.f, 1.f, 1.f};                      // d(capped score) / d(scaled score)
                if constexpr (BIAS) {
                    float xv[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float v = __uint_as_float(pr[i + e]);
                        if (a.softcap > 0.f) {
                            // not by the exponential: its absolute error of 1.8e-7, times the cap, moves the exponent of P
                            // (0.5 % at a cap of 20000)
                            const float th = tanhf(v * a.cap_in);
                            v = a.cap_out * th;
                            fac[e] = 1.f - th * th;
                        } else {
                            v *= a.scale_log2;
                        }
                        xv[e] = v - slope * fabsf((float)(i0 + i + e + sk - sq - n));
                    }
                    x01 = make_float2(xv[0] + nl.x, xv[1] + nl.y);
                    x23 = make_float2(xv[2] + nl.z, xv[3] + nl.w);
                } else {
                    x01 = fma2(make_float2(__uint_as_float(pr[i]), __uint_as_float(pr[i + 1])), sc2, make_float2(nl.x, nl.y));
                    x23 = fma2(make_float2(__uint_as_float(pr[i + 2]), __uint_as_float(pr[i + 3])), sc2, make_float2(nl.z, nl.w));
                }
                float2 p01 = make_float2(ex2_approx(x01.x), ex2_approx(x01.y));
                float2 p23 = make_float2(ex2_approx(x23.x), ex2_approx(x23.y));
                if (!inside) {
                    const int qi = i0 + i;
                    p01.x = (qi >= qi_lo && qi <= qi_hi) ? p01.x : 0.f;
                    p01.y = (qi + 1 >= qi_lo && qi + 1 <= qi_hi) ? p01.y : 0.f;
                    p23.x = (qi + 2 >= qi_lo && qi + 2 <= qi_hi) ? p23.x : 0.f;
                    p23.y = (qi + 3 >= qi_lo && qi + 3 <= qi_hi) ? p23.y : 0.f;
                }
                pr[i] = __float_as_uint(p01.x * fac[0]); pr[i + 1] = __float_as_uint(p01.y * fac[1]);
                pr[i + 2] = __float_as_uint(p23.x * fac[2]); pr[i + 3] = __float_as_uint(p23.y * fac[3]);
                w[i / 2] = Elem<T>::pack(p01.x, p01.y);
                w[i / 2 + 1] = Elem<T>::pack(p23.x, p23.y);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) p_dst[c * 128] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
            ok = mbar_wait(bar(WB_DP0 + buf), (s >> 1) & 1, abort_flag, err, 67);
            if (!ok) break;
            tc_fence_after();
            uint32_t dr[32];
            tmem_ld32(tmem + lane_base + COL_DP + buf * 128 + cg * 32, dr);
            tmem_wait_ld();
            tc_fence_before();
            mbar_arrive_relaxed(bar(WB_TE0 + buf));          // both buffers of this step have been read
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 nd = *reinterpret_cast<const float4*>(vec + 32 + i);
                float2 d01 = mul2(make_float2(__uint_as_float(pr[i]), __uint_as_float(pr[i + 1])),
                                        add2(make_float2(__uint_as_float(dr[i]), __uint_as_float(dr[i + 1])), make_float2(nd.x, nd.y)));
                float2 d23 = mul2(make_float2(__uint_as_float(pr[i + 2]), __uint_as_float(pr[i + 3])),
                                        add2(make_float2(__uint_as_float(dr[i + 2]), __uint_as_float(dr[i + 3])), make_float2(nd.z, nd.w)));
                if (past_end) {
                    // selected, not multiplied: the rows that a tile copy fetched past the end of a packed sequence are its
                    // neighbour's, and 0 x NaN is NaN
                    d01 = make_float2(i < own ? d01.x : 0.f, i + 1 < own ? d01.y : 0.f);
                    d23 = make_float2(i + 2 < own ? d23.x : 0.f, i + 3 < own ? d23.y : 0.f);
                }
                w[i / 2] = Elem<T>::pack(d01.x, d01.y);
                w[i / 2 + 1] = Elem<T>::pack(d23.x, d23.y);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) ds_dst[c * 128] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

// ------------------------------------------------------------------------------------------------------
// Gradients: out[128 x D] = sum over steps of A B with A a stored tile and B 128 rows of dO, Q or K.
// grid (pair of this launch, block): blocks 0 .. 2 nkb - 1 are dV and dK of key block y / 2, the rest dQ of (head of the
// group, query block).  Two 96 KiB stages (tile + rows); at the L2 rate of this GPU a stage takes longer to arrive than
// to multiply, so the kernel is bound by those reads.
//   warp 0 copies, warp 1 MMA (owns the tensor memory), warps 2-5 epilogue (thread = output row)
// ------------------------------------------------------------------------------------------------------
enum { GB_F0 = 0, GB_F1, GB_E0, GB_E1, GB_ACC, GB_COUNT };

template <int D>
struct GradSmem {
    static constexpr int kRows = (D / 64) * kSub;
    static constexpr int kStage = (int)kWideTileBytes + kRows;
    static constexpr int kBytes = 2 * kStage + 8 * GB_COUNT + 16;
};

template <typename T, int D>
__global__ void __launch_bounds__(192, 1) bwd_wide_grads_kernel(const __grid_constant__ WideBwdArgs a) {
    using L = GradSmem<D>;
    constexpr int NSUB = D / 64;
    constexpr uint32_t TMEM_COLS = 256;
    constexpr int FMT = Elem<T>::kDtype == FA_BF16 ? 1 : 0;
    // B is read across its rows in every mode (MN-major); A is K-major for dV and dK (M = keys, K = queries), MN-major
    // for dQ (M = queries, K = keys): the stored layout serves both without a swizzle
    constexpr uint32_t IDESC_KV = umma_idesc(FMT, 128, D, 0, 1), IDESC_Q = umma_idesc(FMT, 128, D, 1, 1);

    extern __shared__ unsigned char smem_raw[];
    const uint32_t sbase = (smem_addr(smem_raw) + 1023u) & ~1023u;
    unsigned char* sgen = smem_raw + (sbase - smem_addr(smem_raw));
    const uint32_t bars = sbase + 2 * L::kStage;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + 2 * L::kStage + 8 * GB_COUNT);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sgen + 2 * L::kStage + 8 * GB_COUNT + 8);
    auto bar = [&](int i) { return bars + 8u * i; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int local = blockIdx.x;
    const Geometry geo(a, a.unit0 + local);
    const int b = geo.b, hk = geo.hk, sq = geo.sq, sk = geo.sk;
    const int G = a.hq / a.hkv;
    if (g_bwd_wide_error) return;

    // mode 0: dV, 1: dK, 2: dQ
    const bool is_q = (int)blockIdx.y >= 2 * a.grid.nkb;
    const int mode = is_q ? 2 : (int)(blockIdx.y & 1);
    int g_q = 0, blk, steps;
    BlockRange br;                                           // query blocks (dV, dK) or key blocks (dQ) that are summed over
    if (!is_q) {
        blk = blockIdx.y >> 1;
        if (blk * 128 >= sk) return;
        br = wide_query_blocks(a.grid, sq, sk, blk);
        steps = (br.hi - br.lo) * G;
    } else {
        const int y = blockIdx.y - 2 * a.grid.nkb;
        g_q = y % G;
        blk = a.grid.nqb - 1 - y / G;
        if (blk * 128 >= sq) return;
        br = wide_key_blocks(a.grid, sq, sk, blk);
        steps = max(0, br.hi - br.lo);
    }
    const int rows = min(128, (is_q ? sq : sk) - blk * 128);
    T* out;
    int64_t ss;
    if (mode == 0) { ss = a.dv_ss; out = reinterpret_cast<T*>(a.dv) + (a.cu_q ? 0 : (int64_t)b * a.dv_sb) + (int64_t)(geo.k_off + blk * 128) * ss + (int64_t)hk * a.dv_sh; }
    else if (mode == 1) { ss = a.dk_ss; out = reinterpret_cast<T*>(a.dk) + (a.cu_q ? 0 : (int64_t)b * a.dk_sb) + (int64_t)(geo.k_off + blk * 128) * ss + (int64_t)hk * a.dk_sh; }
    else { ss = a.dq_ss; out = reinterpret_cast<T*>(a.dq) + (a.cu_q ? 0 : (int64_t)b * a.dq_sb) + (int64_t)(geo.q_off + blk * 128) * ss + (int64_t)(hk * G + g_q) * a.dq_sh; }

    if (steps == 0) {                                        // nothing is visible from here: zero gradient
        if (tid < rows) {
            uint4* row = reinterpret_cast<uint4*>(out + (int64_t)tid * ss);
            for (int c = 0; c < a.d / 8; ++c) row[c] = make_uint4(0, 0, 0, 0);
        }
        return;
    }
    if (tid == 0) {
        for (int i = 0; i < GB_COUNT; ++i) mbar_init(bar(i), 1u);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) { tmem_alloc(smem_addr(tmem_slot), TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    int* err = &g_bwd_wide_error;
    const int bb = a.cu_q ? 0 : b;

    if (warp == 0) {
        if (lane == 0) {
            const CUtensorMap* map = mode == 0 ? &a.tdo : (mode == 1 ? &a.tq : &a.tk);
            const unsigned char* tiles = mode == 0 ? a.p_tiles : a.ds_tiles;
            const int row0 = a.cu_q ? (is_q ? geo.k_off : geo.q_off) : 0;
            tma_prefetch_desc(map);
            bool ok = true;
            for (int j = 0; j < steps && ok; ++j) {
                const int st = j & 1;
                const int g = is_q ? g_q : j / (br.hi - br.lo);
                const int other = br.lo + (is_q ? j : j % (br.hi - br.lo));
                const size_t tile = is_q ? wide_tile_at(a.grid, G, local, g, other, blk) : wide_tile_at(a.grid, G, local, g, blk, other);
                if (j >= 2) ok = mbar_wait(bar(GB_E0 + st), ((j >> 1) - 1) & 1, abort_flag, err, 71);
                if (!ok) break;
                const uint32_t s0 = sbase + st * L::kStage;
                mbar_expect_tx(bar(GB_F0 + st), L::kStage);
                bulk_load_1d(s0, tiles + tile, (uint32_t)kWideTileBytes, bar(GB_F0 + st));
#pragma unroll
                for (int c = 0; c < NSUB; ++c)
                    tma_load_4d(s0 + (uint32_t)kWideTileBytes + c * kSub, map, bar(GB_F0 + st), c * 64, is_q ? hk : hk * G + g, row0 + other * 128, bb);
            }
        }
    } else if (warp == 1) {
        // the block in which a packed sequence ends, if it ends inside one
        const int b_rows = is_q ? sk : sq, tail = a.cu_q && (b_rows & 127) ? b_rows >> 7 : -1;
        int other = br.lo;
        bool ok = true;
        for (int j = 0; j < steps && ok; ++j) {
            const int st = j & 1;
            ok = mbar_wait(bar(GB_F0 + st), (j >> 1) & 1, abort_flag, err, 72);
            if (!ok) break;
            tc_fence_after();
            const uint32_t s0 = sbase + st * L::kStage;
            const uint64_t dB = umma_desc(s0 + (uint32_t)kWideTileBytes, kSub, 1024);
            // Stored tile: element (key k, query q) at chunk (q / 8) x 2048 + k x 16 + (q % 8) x 2 bytes.
            // dV, dK: a K step is 16 queries = 2 chunks; along K the chunks lie 2048 bytes apart, along M eight keys are 128
            // bytes.  dQ: a K step is 16 keys = 256 bytes; along K eight keys are 128 bytes, along M the chunks lie 2048 apart.
            const uint64_t dA = is_q ? umma_desc_noswizzle(s0, 128, 2048) : umma_desc_noswizzle(s0, 2048, 128);
            const int block = other;                         // query block (dV, dK) or key block (dQ)
            if (++other == br.hi) other = br.lo;
            if (block == tail) {
                // Rows past the end of a packed sequence are the next one's and meet zeros of the tile, but 0 x NaN is NaN (past
                // the end of a dense batch entry the copy fills with zeros): only the K steps that hold own rows are multiplied,
                // and what is left of the last one is cleared.
                const int left = b_rows & 127, end = (left + 15) & ~15;
#pragma unroll
                for (int sub = 0; sub < NSUB; ++sub)
                    for (int idx = left * 8 + lane; idx < end * 8; idx += 32)       // 16-byte chunks of rows left .. end - 1
                        *reinterpret_cast<uint4*>(sgen + st * L::kStage + kWideTileBytes + sub * kSub + idx * 16) = make_uint4(0, 0, 0, 0);
                fence_proxy_async_smem();
                __syncwarp();
                for (int k = 0; k < end; k += 16) {
                    const uint64_t ak = umma_desc_at(dA, k * (is_q ? 16 : 256)), bk = umma_desc_at(dB, k * 128);
                    if (j == 0 && k == 0) umma_ss_w<0>(tmem, ak, bk, is_q ? IDESC_Q : IDESC_KV);
                    else umma_ss_w<1>(tmem, ak, bk, is_q ? IDESC_Q : IDESC_KV);
                }
            } else if (!is_q) {
                umma_ss_group4<0, 256, 512, 768, 0, 128, 256, 384>(tmem, dA, dB, IDESC_KV, j > 0);
                umma_ss_group4<1024, 1280, 1536, 1792, 512, 640, 768, 896>(tmem, dA, dB, IDESC_KV, 1);
            } else {
                umma_ss_group4<0, 16, 32, 48, 0, 128, 256, 384>(tmem, dA, dB, IDESC_Q, j > 0);
                umma_ss_group4<64, 80, 96, 112, 512, 640, 768, 896>(tmem, dA, dB, IDESC_Q, 1);
            }
            umma_commit_w(bar(GB_E0 + st));
        }
        if (ok) umma_commit_w(bar(GB_ACC));
    } else {
        const int r = (warp & 3) * 32 + lane;                // warps 2..5 cover the lane quarters 2, 3, 0, 1
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        if (mbar_wait(bar(GB_ACC), 0, abort_flag, err, 73)) {
            tc_fence_after();
            T* row = out + (int64_t)r * ss;
            const float sc = mode == 0 ? 1.f : a.scale;
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
                uint32_t acc[32];
                tmem_ld32(tmem + lane_base + c * 32, acc);
                tmem_wait_ld();
                if (r < rows) store_row_scaled<T>(row + c * 32, acc, sc, a.d - c * 32);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

// ------------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------------
// Tiles of the KV heads of one launch: what a launch writes should still be in the 126 MB L2 when the next launch reads
// it, and one launch should fill the GPU.  Under a causal mask about half of a head's tiles exist.  Measured at
// B2 S2048 H8/4 / B1 S8192 H8 / B4 S1024 H16 (causal) with 32, 64, 128 MiB: 223 / 151 / 133, 1147 / 1050 / 1002,
// 238 / 212 / 211 us.  A KV head whose tiles alone are more than L2 goes by itself, through HBM, at about the same rate: whole
// training steps at D256 causal B1 S8192, H8 on one KV head (2 GiB of tiles) 1150 us, on eight (256 MiB each) 1295; D192
// full B1 S12000 H8 on one, 3730 us = 830 TFLOP/s.
constexpr size_t kWideGroupBytes = (size_t)128 << 20;
constexpr size_t kWideWorkspaceLimit = (size_t)6 << 30;      // one KV head's tiles may take this much at most

size_t unit_bytes(const fa_bwd_params& p) {                  // P^T and dS^T tiles of one (batch entry, KV head) pair
    return (size_t)(p.hq / p.hkv) * ((p.sk + 127) / 128) * ((p.sq + 127) / 128) * 2 * kWideTileBytes;
}
int64_t units_per_launch(const fa_bwd_params& p) {
    const int64_t units = (int64_t)p.b * p.hkv;
    const size_t per = unit_bytes(p) / (p.causal ? 2 : 1);
    const int64_t n = (int64_t)(kWideGroupBytes / (per ? per : 1));
    return n < 1 ? 1 : (n < units ? n : units);
}
size_t delta_bytes(const fa_bwd_params& p) { return (bwd_generic_workspace(p) + 255) & ~(size_t)255; }

template <typename T, int D>
int launch_t(const fa_bwd_params& p, WideBwdArgs& a, cudaStream_t st) {
    auto k1 = (p.softcap > 0.f || p.alibi_slopes) ? bwd_wide_scores_kernel<T, D, true> : bwd_wide_scores_kernel<T, D, false>;
    auto k2 = bwd_wide_grads_kernel<T, D>;
    const int smem1 = ScoreSmem<D>::kBytes + 1024, smem2 = GradSmem<D>::kBytes + 1024;
    static_assert(ScoreSmem<D>::kBytes + 1024 <= 232448 && GradSmem<D>::kBytes + 1024 <= 232448, "shared memory limit of a CTA");
    if (int e = cuda_ok(cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1), "cudaFuncSetAttribute")) return e;
    if (int e = cuda_ok(cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2), "cudaFuncSetAttribute")) return e;
    const int G = p.hq / p.hkv;
    const int64_t units = (int64_t)p.b * p.hkv, per = units_per_launch(p);
    // Query blocks a score CTA walks: long walks amortise its K and V (128 KiB against 128 KiB a step), short ones fill the
    // GPU: sixteen while that leaves two CTAs for three SMs (sixteen against about two CTAs an SM: 1002 against 1050 us at
    // B1 S8192 H8, 133 against 142 at B2 S2048 H8/4), fewer below.
    const int64_t tiles = per * G * a.grid.nkb * a.grid.nqb / (p.causal ? 2 : 1);
    a.steps_per_cta = 16;
    while (a.steps_per_cta > 4 && tiles / a.steps_per_cta < sm_count() * 2 / 3) a.steps_per_cta /= 2;
    const unsigned nz = (unsigned)(((int64_t)a.grid.nqb * G + a.steps_per_cta - 1) / a.steps_per_cta);
    for (int64_t u = 0; u < units; u += per) {
        const unsigned n = (unsigned)(units - u < per ? units - u : per);
        a.unit0 = (int)u;
        k1<<<dim3(n, a.grid.nkb, nz), 608, smem1, st>>>(a);
        mark_kernel(st);
        k2<<<dim3(n, 2 * a.grid.nkb + G * a.grid.nqb), 192, smem2, st>>>(a);
        mark_kernel(st);
    }
    return cuda_ok(cudaGetLastError(), "bwd_wide launch");
}

}  // namespace

bool bwd_wide_sm100_supported(const fa_bwd_params& p) {
    if (p.d != p.dv_dim || p.d % 8 != 0 || p.d <= 128 || p.d > 256) return false;
    if (!(p.scale > 0.f) || p.sq <= 0 || p.sk <= 0 || p.hkv <= 0) return false;
    if ((p.cu_seqlens_q != nullptr) != (p.cu_seqlens_k != nullptr)) return false;
    if (p.cu_seqlens_q && (p.total_q <= 0 || p.total_k <= 0)) return false;
    if (unit_bytes(p) > kWideWorkspaceLimit) return false;
    const int64_t nkb = (p.sk + 127) / 128, nqb = (p.sq + 127) / 128, G = p.hq / p.hkv;
    if (2 * nkb + G * nqb > 65535 || (nqb * G + 3) / 4 > 65535) return false;            // blocks stay inside a grid dimension
    const fa_tensor* ts[4] = {&p.q, &p.k, &p.v, &p.dout};
    for (const fa_tensor* t : ts) {
        if (t->stride_h <= 0 || t->stride_s <= 0) return false;
        if (!p.cu_seqlens_q && p.b > 1 && t->stride_b <= 0) return false;
    }
    return tensor_map_encoder_available();
}

size_t bwd_wide_sm100_workspace(const fa_bwd_params& p) { return delta_bytes(p) + (size_t)units_per_launch(p) * unit_bytes(p); }

int launch_bwd_wide_sm100(const fa_bwd_params& p) {
    WideBwdArgs a;
    const bool packed = p.cu_seqlens_q != nullptr;
    const int64_t q_rows = packed ? p.total_q : p.sq, k_rows = packed ? p.total_k : p.sk;
    const int nb = packed ? 1 : p.b;
    auto map = [&](CUtensorMap* m, const fa_tensor& t, int heads, int64_t rows) {
        return make_tile_map(m, p.dtype, t.ptr, p.d, heads, rows, nb, t.stride_h, t.stride_s, packed || p.b == 1 ? rows * t.stride_s : t.stride_b, 128);
    };
    if (int e = map(&a.tq, p.q, p.hq, q_rows)) return e;
    if (int e = map(&a.tdo, p.dout, p.hq, q_rows)) return e;
    if (int e = map(&a.tk, p.k, p.hkv, k_rows)) return e;
    if (int e = map(&a.tv, p.v, p.hkv, k_rows)) return e;
    a.dq = p.dq.ptr; a.dk = p.dk.ptr; a.dv = p.dv.ptr;
    a.dq_sb = p.dq.stride_b; a.dq_ss = p.dq.stride_s; a.dq_sh = p.dq.stride_h;
    a.dk_sb = p.dk.stride_b; a.dk_ss = p.dk.stride_s; a.dk_sh = p.dk.stride_h;
    a.dv_sb = p.dv.stride_b; a.dv_ss = p.dv.stride_s; a.dv_sh = p.dv.stride_h;
    a.lse = p.lse; a.lse_sb = p.lse_stride_b; a.lse_sh = p.lse_stride_h; a.lse_ss = p.lse_stride_s;
    float* delta = reinterpret_cast<float*>(p.workspace);
    a.delta = delta;
    a.cu_q = p.cu_seqlens_q; a.cu_k = p.cu_seqlens_k;
    a.b = p.b; a.sq = p.sq; a.sk = p.sk; a.hq = p.hq; a.hkv = p.hkv; a.d = p.d;
    a.scale = p.scale; a.scale_log2 = p.scale * kLog2e;
    a.grid = {(p.sk + 127) / 128, (p.sq + 127) / 128, p.causal, p.window_left, p.window_right};
    a.softcap = p.softcap; a.cap_in = p.softcap > 0.f ? p.scale / p.softcap : 0.f; a.cap_out = p.softcap * kLog2e;
    a.alibi = p.alibi_slopes; a.alibi_sb = p.alibi_stride_b;
    a.p_tiles = reinterpret_cast<unsigned char*>(p.workspace) + delta_bytes(p);
    a.ds_tiles = a.p_tiles + (size_t)units_per_launch(p) * (unit_bytes(p) / 2);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(p.stream);
    note_kernel("sm100_wide_tcgen05_bwd");
    if (int e = launch_bwd_delta_sm100(p, delta)) return e;
    if (p.dtype == FA_F16) return p.d <= 192 ? launch_t<__half, 192>(p, a, st) : launch_t<__half, 256>(p, a, st);
    return p.d <= 192 ? launch_t<__nv_bfloat16, 192>(p, a, st) : launch_t<__nv_bfloat16, 256>(p, a, st);
}

}  // namespace fa
