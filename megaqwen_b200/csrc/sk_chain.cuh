// The linears of one layer for at most 64 rows, a decode step of a batch, each with the
// work around it: q|k|v with the norm before and QK-norm + RoPE + cache write behind, O and down with the
// residual add, gate|up with the norm before and SwiGLU behind.
//
// With so few rows a linear streams its weights (8 to 13 MB, 1.3 to 2 us of HBM) and its time is the chain of latencies
// around them, so what counts is the number of dependent kernels and what stands between the wait for the
// preceding one and the store.  The operands are swapped (128 weight rows are the M of tcgen05.mma, the rows of
// the activation its N) and K is split over the CTAs of a CLUSTER, so that a linear spreads over 64 to 144 SMs with all
// of a CTA's weights requested before the wait; the split's partial sums meet in distributed shared memory: rank r
// of the cluster gets the rows [r TPC, (r + 1) TPC) of all partial tiles, adds them in rank order and
// finishes those rows.  One layer used to be eight kernels with fp32 planes in global memory between them: step of
// batch 8 / 32 / 64 at contexts 400 / 384 / 1024 893 / 1107 / 2283 -> 747 / 967 / 2079 us.  The planes and the order in which they are
// added are those of the eight kernels.  Prompts of as many rows do not come here: their sums over K are not split.
//
// RMSNorm: the kernel that finishes a row of the residual stream leaves the row's sum of squares of its 128 columns
// in ssq[row][8]; the next linear adds the eight, first to last, normalises its K slice of the rows itself and writes it
// as the swizzled operand tile that TMA would have written.
#pragma once

#include "tc_core.cuh"

namespace mq {

enum { SK_QKV = 0, SK_O = 1, SK_GU = 2, SK_DOWN = 3 };
constexpr int SK_THREADS = 256, SK_BK = 64, SK_SSQ = H / 128, SK_MAX_ROWS = 64;

// Cluster sizes: 32 tiles x 4 = 128, 8 x 8 = 64 and 48 x 4 = 192 CTAs.  With one CTA to an SM the device holds 45 clusters of
// three, 33 of four, 15 of eight; gate|up therefore keeps to 110 KB, so that 71 clusters of four find room and its 48
// run in one round (one CTA an SM and three slices of K: two rounds, 12.0 against 4.9 us at 32 rows).
template <int MPAD, int MODE>
struct SkCfg {
    static constexpr int K = MODE == SK_O ? QSZ : MODE == SK_DOWN ? I : H;
    static constexpr int KS = MODE == SK_QKV || MODE == SK_GU ? 4 : 8;
    static constexpr int NKB = (K / SK_BK + KS - 1) / KS;                // k-blocks of one CTA, at most
    static constexpr int W_BYTES = 128 * SK_BK * 2, X_BYTES = MPAD * SK_BK * 2;
    static constexpr int TPC = (MPAD + KS - 1) / KS;                     // rows that one CTA of the cluster finishes
    static constexpr int RED_BYTES = KS * TPC * 128 * 4;
    static constexpr bool ALIAS = NKB * (W_BYTES + X_BYTES) + RED_BYTES > (MODE == SK_GU ? 110 : 220) * 1024;   // the sums take the operands' place, behind one more barrier
    static constexpr int RED_OFF = ALIAS ? 0 : NKB * (W_BYTES + X_BYTES);
    static constexpr int BAR_OFF = ALIAS ? NKB * (W_BYTES + X_BYTES) : RED_OFF + RED_BYTES;
    static constexpr size_t SMEM = (size_t)BAR_OFF + MPAD * 4 + 128 + 1024;
    static constexpr int TILES = MODE == SK_QKV ? QKV / 128 : MODE == SK_GU ? 2 * I / 128 : H / 128;
    static_assert((MODE != SK_QKV && MODE != SK_GU) || K == KS * 4 * SK_BK, "a K slice that is normed is 256 columns, eight a lane");
    static_assert(MPAD % 16 == 0 && MPAD <= SK_MAX_ROWS && (!ALIAS || RED_BYTES <= NKB * (W_BYTES + X_BYTES)) && SMEM <= 232448, "one CTA's shared memory");
};

struct SkArgs {
    int M;
    bf16* h;                       // residual stream [M, H]: normed on read (QKV, GU), added to (O, DOWN)
    float* ssq;                    // [M, 8] sums of squares of h by 128 columns: read (QKV, GU), written (O, DOWN)
    const bf16* gain;              // norm weight (QKV, GU)
    bf16* out;                     // QKV: [M, 4096], of which the rotated query heads are written; GU: [M, 3072]
    // QKV: row s is position pos_rows[s] of sequence s, whose caches begin s * seq_stride elements in
    const bf16 *q_norm, *k_norm, *cos, *sin;
    bf16 *k_cache, *v_cache;
    int layer, max_seq;
    const int* pos_rows;
    size_t seq_stride;
    unsigned int* status;
    int drop = -1;                 // test hook: block drop % 16 of rank drop / 16 of every cluster is never requested
};

// of the eight sums of a row, first to last
__device__ __forceinline__ float row_square_sum(const float4& a, const float4& b) { return ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w; }
// products of two pairs of bf16, each rounded once
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_map(uint32_t saddr, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

// one head's 128 values, lane l holding 2 l, 2 l + 1 (lo) and 64 + 2 l, 64 + 2 l + 1 (hi): RMSNorm, then split-half RoPE evaluated
// in bf16 (reference: prefill_qk_norm_rope_kernel, fused_prefill_kernels.inl:112-258)
__device__ __forceinline__ void head_norm_rope(const float (&xl)[2], const float (&xh)[2], uint32_t wl, uint32_t wh, uint32_t cl, uint32_t ch, uint32_t sl,
                                               uint32_t sh, uint32_t& plo, uint32_t& phi) {
    const float ss = warp_sum(xl[0] * xl[0] + xl[1] * xl[1] + xh[0] * xh[0] + xh[1] * xh[1]);
    const float r = 1.0f / sqrtf(ss * (1.0f / D) + RMS_EPS);
    const float wlo[2] = {bf_lo(wl), bf_hi(wl)}, whi[2] = {bf_lo(wh), bf_hi(wh)};
    const float clo[2] = {bf_lo(cl), bf_hi(cl)}, chi[2] = {bf_lo(ch), bf_hi(ch)};
    const float slo[2] = {bf_lo(sl), bf_hi(sl)}, shi[2] = {bf_lo(sh), bf_hi(sh)};
    float lo[2], hi[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float nl = rbf(wlo[e] * rbf(xl[e] * r)), nh = rbf(whi[e] * rbf(xh[e] * r));
        lo[e] = rbf(rbf(nl * clo[e]) + rbf(-nh * slo[e]));
        hi[e] = rbf(rbf(nh * chi[e]) + rbf(nl * shi[e]));
    }
    plo = pack_bf16x2(lo[0], lo[1]);
    phi = pack_bf16x2(hi[0], hi[1]);
}

// tm0, tm1, tm2: q, k, v (boxes of 128 rows), or gate, up (boxes of 64: a tile is 64 gate rows and the 64 up rows of the same columns),
// or the one matrix; tmX: the activation (O, DOWN).
template <int MPAD, int MODE>
__global__ void __launch_bounds__(SK_THREADS, 1)
k_sk(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, const __grid_constant__ CUtensorMap tm2,
     const __grid_constant__ CUtensorMap tmX, SkArgs a) {
    using Cfg = SkCfg<MPAD, MODE>;
    constexpr int KS = Cfg::KS, TPC = Cfg::TPC, KB = Cfg::K / SK_BK;
    constexpr bool NORM = MODE == SK_QKV || MODE == SK_GU;
    constexpr int TM_COLS = MPAD < 32 ? 32 : MPAD;
    pdl_trigger();
    extern __shared__ uint8_t sk_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sk_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* xs = smem + Cfg::NKB * Cfg::W_BYTES;
    float* red = reinterpret_cast<float*>(smem + Cfg::RED_OFF);           // [KS][TPC][128]
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);    // [NKB]
    uint64_t* accum = full + Cfg::NKB;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    volatile uint32_t* bad = tmem_slot + 1;                               // a bounded wait of some CTA of the cluster has run out: its sums are missing
    float* inv = reinterpret_cast<float*>(smem + Cfg::BAR_OFF + 128);     // [MPAD]
    static_assert((Cfg::NKB + 1) * 8 + 8 <= 128 && Cfg::NKB <= 16, "barriers");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x, rank = blockIdx.y;                       // the cluster runs along y
    const int kb0 = rank * KB / KS, nkb = (rank + 1) * KB / KS - kb0;

    if (tid == 0) {
        for (int i = 0; i < Cfg::NKB; ++i) mbar_init(&full[i], 1);
        mbar_init(accum, 1);
        mbar_fence_init();
        *bad = 0u;
    }
    if (warp == 1) tmem_alloc(tmem_slot, TM_COLS);
    uint4 gv = make_uint4(0u, 0u, 0u, 0u);                                // norm weights of this lane's eight columns
    if (NORM) gv = __ldg(reinterpret_cast<const uint4*>(a.gain + kb0 * SK_BK) + lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    cluster_arrive();          // the shared memory of a CTA may be accessed once it is known to run: waited for ahead of the first access
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

    if (tid == 0) {
        // the weights hang on nothing: all of them are requested before the wait
        for (int i = 0; i < nkb; ++i) {
            if (rank * 16 + i == a.drop) continue;
            uint8_t* w = smem + i * Cfg::W_BYTES;
            mbar_expect_tx(&full[i], (uint32_t)(Cfg::W_BYTES + (NORM ? 0 : Cfg::X_BYTES)));
            const int x = (kb0 + i) * SK_BK;
            if (MODE == SK_GU) {
                tma_load_2d(w, &tm0, x, tile * 64, &full[i]);
                tma_load_2d(w + Cfg::W_BYTES / 2, &tm1, x, tile * 64, &full[i]);
            } else if (MODE == SK_QKV) {
                constexpr int TQ = QSZ / 128, TK = KVSZ / 128;
                tma_load_2d(w, tile < TQ ? &tm0 : tile < TQ + TK ? &tm1 : &tm2, x, (tile < TQ ? tile : tile < TQ + TK ? tile - TQ : tile - TQ - TK) * 128, &full[i]);
            } else {
                tma_load_2d(w, &tm0, x, tile * 128, &full[i]);
            }
        }
    }
    const bool is_v = MODE == SK_QKV && tile >= (QSZ + KVSZ) / 128, is_q = MODE == SK_QKV && tile < QSZ / 128;
    uint32_t wl = 0u, wh = 0u;
    if (MODE == SK_QKV && !is_v) {
        const bf16* wn = is_q ? a.q_norm : a.k_norm;
        wl = __ldg(reinterpret_cast<const uint32_t*>(wn + 2 * lane));
        wh = __ldg(reinterpret_cast<const uint32_t*>(wn + 64 + 2 * lane));
    }
    pdl_wait();
    if (!NORM && tid == 0)
        for (int i = 0; i < nkb; ++i)
            if (rank * 16 + i != a.drop) tma_load_2d(xs + i * Cfg::X_BYTES, &tmX, (kb0 + i) * SK_BK, 0, &full[i]);
    // what the rows that this CTA finishes need besides the sums; a warp takes rows warp, warp + 8, .. of them
    constexpr int TW = (TPC + 7) / 8;
    uint2 hv[TW] = {};
    if (MODE == SK_O || MODE == SK_DOWN) {
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int n = rank * TPC + warp + i * 8;
            if (warp + i * 8 < TPC && n < a.M) hv[i] = ld_cg_u2(a.h + (size_t)n * H + tile * 128 + 4 * lane);
        }
    }
    int pos[TW] = {};
    if (MODE == SK_QKV) {
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int n = rank * TPC + warp + i * 8;
            if (warp + i * 8 < TPC && n < a.M) pos[i] = min(max(ld_cg_i32(a.pos_rows + n), 0), a.max_seq - 1);
        }
    }
    if (NORM) {
        static_assert(MPAD <= SK_THREADS, "a thread a row");
        float4 p[2] = {};
        if (tid < a.M) {
            p[0] = __ldcg(reinterpret_cast<const float4*>(a.ssq + tid * SK_SSQ));
            p[1] = __ldcg(reinterpret_cast<const float4*>(a.ssq + tid * SK_SSQ) + 1);
        }
        // this CTA's K slice of the rows: a warp takes a row at a time, a lane 16 bytes of it; all requested before the first is used
        constexpr int CI = MPAD / 8;
        uint4 v[CI];
#pragma unroll
        for (int i = 0; i < CI; ++i) {
            const int row = warp + 8 * i;
            v[i] = row < a.M ? ld_cg_u4(a.h + (size_t)row * H + kb0 * SK_BK + lane * 8) : make_uint4(0u, 0u, 0u, 0u);
        }
        if (tid < a.M) inv[tid] = 1.0f / sqrtf(row_square_sum(p[0], p[1]) * (1.0f / H) + RMS_EPS);
        __syncthreads();
        // 128-byte swizzle: 16-byte chunk j of row r of a k-block stands at chunk j ^ (r & 7), and r & 7 is this warp's number
        uint8_t* dst = xs + (lane >> 3) * Cfg::X_BYTES + warp * 128 + (((lane & 7) ^ warp) << 4);
#pragma unroll
        for (int i = 0; i < CI; ++i) {
            const int row = warp + 8 * i;
            if (row < a.M) {
                const float r = inv[row];
                *reinterpret_cast<uint4*>(dst + i * 1024) = make_uint4(mul_bf16x2(gv.x, pack_bf16x2(bf_lo(v[i].x) * r, bf_hi(v[i].x) * r)),
                                                                       mul_bf16x2(gv.y, pack_bf16x2(bf_lo(v[i].y) * r, bf_hi(v[i].y) * r)),
                                                                       mul_bf16x2(gv.z, pack_bf16x2(bf_lo(v[i].z) * r, bf_hi(v[i].z) * r)),
                                                                       mul_bf16x2(gv.w, pack_bf16x2(bf_lo(v[i].w) * r, bf_hi(v[i].w) * r)));
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic stores, read by the tensor core
        __syncthreads();
    }
    uint32_t cl[TW] = {}, ch[TW] = {}, sl[TW] = {}, sh[TW] = {};
    if (MODE == SK_QKV && !is_v) {
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const bf16 *c = a.cos + (size_t)pos[i] * D, *s = a.sin + (size_t)pos[i] * D;
            cl[i] = *reinterpret_cast<const uint32_t*>(c + 2 * lane);
            ch[i] = *reinterpret_cast<const uint32_t*>(c + 64 + 2 * lane);
            sl[i] = *reinterpret_cast<const uint32_t*>(s + 2 * lane);
            sh[i] = *reinterpret_cast<const uint32_t*>(s + 64 + 2 * lane);
        }
    }
    bool ok = true;            // after an expired wait nothing more is issued, and no CTA of the cluster stores a result
    if (tid == 32) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MPAD >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        for (int i = 0; i < nkb; ++i) {
            if (!mbar_wait(&full[i], 0, a.status)) { ok = false; break; }
            tc_fence_after();
            const uint64_t dw = smem_desc_sw128(smem + i * Cfg::W_BYTES), dx = smem_desc_sw128(xs + i * Cfg::X_BYTES);
#pragma unroll
            for (int k = 0; k < SK_BK / 16; ++k) umma_bf16(tmem, dw + 2 * k, dx + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(accum);
    }
    __syncwarp();
    if (!mbar_wait(accum, 0, a.status)) ok = false;
    tc_fence_after();
    __syncwarp();
    cluster_wait();            // every CTA of the cluster has started, microseconds ago
    if (!ok)
        for (int r = 0; r < KS; ++r) st_cluster_f32(cluster_map(smem_u32(tmem_slot + 1), r), 1u);
    if (Cfg::ALIAS) {          // every CTA of the cluster has read its operands: their place may be written
        cluster_arrive();
        cluster_wait();
    }
    if (__all_sync(0xffffffffu, ok)) {
        // warp w reads lanes 32 (w % 4) .. (weight rows) and half of the columns (activation rows)
        constexpr int HALF = MPAD / 2;
        const int quarter = warp & 3, c0 = (warp >> 2) * HALF;
        uint32_t v[HALF];
#pragma unroll
        for (int c = 0; c < HALF; c += 8) tmem_ld8_nowait(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c0 + c), v + c);
        tmem_ld_wait();
        const uint32_t mine = smem_u32(red) + (uint32_t)((rank * TPC * 128 + quarter * 32 + lane) * 4);
#pragma unroll
        for (int c = 0; c < HALF; ++c) {
            const int n = c0 + c, to = n / TPC;
            if (n < a.M) st_cluster_f32(cluster_map(mine, to) + (uint32_t)((n - to * TPC) * 512), v[c]);
        }
        tc_fence_before();
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    const bool store = *bad == 0u;                                        // the same for the whole cluster
#pragma unroll
    for (int i = 0; i < TW; ++i) {
        const int t = warp + i * 8, n = rank * TPC + t;
        if (t >= TPC || n >= a.M || !store) continue;
        const float* p = red + t * 128;
        if (MODE == SK_O || MODE == SK_DOWN) {
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                const float4 u = *reinterpret_cast<const float4*>(p + k * TPC * 128 + 4 * lane);
                s.x += u.x; s.y += u.y; s.z += u.z; s.w += u.w;
            }
            const float o[4] = {rbf(bf_lo(hv[i].x) + rbf(s.x)), rbf(bf_hi(hv[i].x) + rbf(s.y)), rbf(bf_lo(hv[i].y) + rbf(s.z)), rbf(bf_hi(hv[i].y) + rbf(s.w))};
            *reinterpret_cast<uint2*>(a.h + (size_t)n * H + tile * 128 + 4 * lane) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
            const float ss = warp_sum(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]);
            if (lane == 0) a.ssq[(size_t)n * SK_SSQ + tile] = ss;
        } else {
            float xl[2] = {0.f, 0.f}, xh[2] = {0.f, 0.f};
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                const float2 u = *reinterpret_cast<const float2*>(p + k * TPC * 128 + 2 * lane), w = *reinterpret_cast<const float2*>(p + k * TPC * 128 + 64 + 2 * lane);
                xl[0] += u.x; xl[1] += u.y; xh[0] += w.x; xh[1] += w.y;
            }
            if (MODE == SK_GU) {
                const float g0 = rbf(silu_f32(rbf(xl[0]))), g1 = rbf(silu_f32(rbf(xl[1])));
                *reinterpret_cast<uint32_t*>(a.out + (size_t)n * I + tile * 64 + 2 * lane) = pack_bf16x2(g0 * rbf(xh[0]), g1 * rbf(xh[1]));
            } else {
#pragma unroll
                for (int e = 0; e < 2; ++e) { xl[e] = rbf(xl[e]); xh[e] = rbf(xh[e]); }
                uint32_t lo = pack_bf16x2(xl[0], xl[1]), hi = pack_bf16x2(xh[0], xh[1]);
                if (!is_v) head_norm_rope(xl, xh, wl, wh, cl[i], ch[i], sl[i], sh[i], lo, hi);
                const int head = is_q ? tile : is_v ? tile - (QSZ + KVSZ) / 128 : tile - QSZ / 128;
                const size_t seq = (size_t)n * a.seq_stride;
                bf16* dst = is_q ? a.out + (size_t)n * QKV + tile * 128
                                 : (is_v ? a.v_cache : a.k_cache) + seq + ((size_t)(a.layer * NKV + head) * a.max_seq + pos[i]) * D;
                *reinterpret_cast<uint32_t*>(dst + 2 * lane) = lo;
                *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = hi;
            }
        }
    }
    __syncthreads();
    if (!store) {              // copies and products that were issued end before their memory is given back
        if (tid == 0)
            for (int i = 0; i < nkb; ++i)
                if (rank * 16 + i != a.drop) mbar_wait_drain(&full[i], 0);
        if (tid == 32) mbar_wait_drain(accum, 0);
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem, TM_COLS);
}

// h[s,:] = embed[ids[s],:], one warp per row.  The row's sum of squares stands in the first of its eight places, in the order in which
// rmsnorm_slice adds it.
__global__ void __launch_bounds__(32) k_sk_embed(const int* ids, const bf16* __restrict__ embed, bf16* __restrict__ h, float* __restrict__ ssq,
                                                 int vocab, unsigned int* status) {
    pdl_wait();
    pdl_trigger();   // only now: the kernels behind may read cache rows of earlier steps ahead of their own waits
    const int s = blockIdx.x, lane = threadIdx.x;
    int tok = ld_cg_i32(ids + s);
    if (tok < 0 || tok >= vocab) {
        if (lane == 0) atomicOr(status, MQ_STATUS_BAD_TOKEN);
        tok = min(max(tok, 0), vocab - 1);
    }
    float v[32];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(embed + (size_t)tok * H + j * 256) + lane);
        *(reinterpret_cast<uint4*>(h + (size_t)s * H + j * 256) + lane) = u;
        v[j * 8 + 0] = bf_lo(u.x); v[j * 8 + 1] = bf_hi(u.x); v[j * 8 + 2] = bf_lo(u.y); v[j * 8 + 3] = bf_hi(u.y);
        v[j * 8 + 4] = bf_lo(u.z); v[j * 8 + 5] = bf_hi(u.z); v[j * 8 + 6] = bf_lo(u.w); v[j * 8 + 7] = bf_hi(u.w);
    }
    const float ss = slice_square_sum(v);
    if (lane < SK_SSQ) ssq[(size_t)s * SK_SSQ + lane] = lane == 0 ? ss : 0.f;
}

// x[s,:] = norm of h[s,:] behind the last layer, one warp per row
__global__ void __launch_bounds__(256) k_sk_norm(const bf16* h, const float* ssq, const bf16* __restrict__ w, bf16* __restrict__ x, int rows) {
    pdl_trigger();
    const int lane = threadIdx.x & 31, s = blockIdx.x * 8 + (threadIdx.x >> 5);
    uint4 g[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) g[j] = __ldg(reinterpret_cast<const uint4*>(w + j * 256) + lane);
    pdl_wait();
    if (s >= rows) return;
    const float4 p0 = __ldcg(reinterpret_cast<const float4*>(ssq + (size_t)s * SK_SSQ)), p1 = __ldcg(reinterpret_cast<const float4*>(ssq + (size_t)s * SK_SSQ) + 1);
    const float r = 1.0f / sqrtf(row_square_sum(p0, p1) * (1.0f / H) + RMS_EPS);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 u = ld_cg_u4(h + (size_t)s * H + j * 256 + lane * 8);
        *(reinterpret_cast<uint4*>(x + (size_t)s * H + j * 256) + lane) =
            make_uint4(mul_bf16x2(g[j].x, pack_bf16x2(bf_lo(u.x) * r, bf_hi(u.x) * r)), mul_bf16x2(g[j].y, pack_bf16x2(bf_lo(u.y) * r, bf_hi(u.y) * r)),
                       mul_bf16x2(g[j].z, pack_bf16x2(bf_lo(u.z) * r, bf_hi(u.z) * r)), mul_bf16x2(g[j].w, pack_bf16x2(bf_lo(u.w) * r, bf_hi(u.w) * r)));
    }
}

// ---------------------------------------------------------------- host side
template <int MPAD, int MODE>
static int launch_sk(const CUtensorMap& m0, const CUtensorMap& m1, const CUtensorMap& m2, const CUtensorMap& mx, const SkArgs& a, cudaStream_t stream) {
    using Cfg = SkCfg<MPAD, MODE>;
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_sk<MPAD, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM);
        if (e != cudaSuccess) return (int)e;
        attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(Cfg::TILES, Cfg::KS);
    cfg.blockDim = dim3(SK_THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = Cfg::KS;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return (int)cudaLaunchKernelEx(&cfg, k_sk<MPAD, MODE>, m0, m1, m2, mx, a);
}

// One linear of a layer; `x` is the activation of O (attention output) and DOWN, else unused.
template <int MODE>
static int sk_linear(const MqLayerWeights& w, const bf16* x, SkArgs a, cudaStream_t stream) {
    CUtensorMap m0, m1, m2, mx;
    const int mpad = a.M <= 16 ? 16 : a.M <= 32 ? 32 : 64;
    constexpr int K = SkCfg<16, MODE>::K;
    int rc;
    if (MODE == SK_QKV) {
        rc = get_map(w.q_proj, QSZ, K, K, 128, &m0);
        if (rc == MQ_OK) rc = get_map(w.k_proj, KVSZ, K, K, 128, &m1);
        if (rc == MQ_OK) rc = get_map(w.v_proj, KVSZ, K, K, 128, &m2);
        mx = m0;
    } else if (MODE == SK_GU) {
        rc = get_map(w.gate_proj, I, K, K, 64, &m0);
        if (rc == MQ_OK) rc = get_map(w.up_proj, I, K, K, 64, &m1);
        m2 = mx = m0;
    } else {
        rc = get_map(MODE == SK_O ? w.o_proj : w.down_proj, H, K, K, 128, &m0);
        if (rc == MQ_OK) rc = get_map(x, (uint64_t)a.M, K, K, (uint32_t)mpad, &mx);
        m1 = m2 = m0;
    }
    if (rc != MQ_OK) return rc;
    switch (mpad) {
    case 16: return launch_sk<16, MODE>(m0, m1, m2, mx, a, stream);
    case 32: return launch_sk<32, MODE>(m0, m1, m2, mx, a, stream);
    default: return launch_sk<64, MODE>(m0, m1, m2, mx, a, stream);
    }
}

}  // namespace mq
