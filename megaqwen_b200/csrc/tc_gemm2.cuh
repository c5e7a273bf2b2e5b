// Tile GEMM on pairs of SMs: C[M, N] = A[M, K] B[N, K]^T with the epilogues of tc_gemm.cuh.
//
// A cluster of two CTAs computes a tile of 256 rows and BN columns with tcgen05.mma.cta_group::2: each CTA stages its 128 rows of
// A and its half of the BN rows of B, the leader (rank 0) issues the instructions, and each CTA's tensor memory
// receives its 128 rows of all BN columns.  An SM so takes in 32 KB for 4.2 MFLOP of a 256-column tile, as
// k_gemm's 256 x 256 tile on one SM does, but needs half of the tensor memory for it: TWO accumulators fit, the
// grid is persistent (pair p takes tiles p, p + pairs, ..) and a tile's epilogue runs while the next
// tile is multiplied.
#pragma once

#include "tc_gemm.cuh"

namespace mq {

constexpr int G2_THREADS = GM_TILE_THREADS;                   // warp 0 TMA, warp 1 MMA (leader only), warps 2-9 epilogue

template <int BN, int EPI>
struct Gemm2Cfg {
    static constexpr bool GLU = EPI == EPI_SWIGLU;            // a tile is BN / 2 gate columns (CTA 0's half of B) and the BN / 2 up columns of the same outputs (CTA 1's)
    static constexpr int OUT = GLU ? BN / 2 : BN;             // output columns of a tile
    static constexpr int A_BYTES = 128 * GM_BK * 2, B_BYTES = BN / 2 * GM_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = 184 * 1024 / STAGE_BYTES > 7 ? 7 : 184 * 1024 / STAGE_BYTES;
    static constexpr int OUT_BYTES = GM_EPI_WARPS * 2048;     // a warp's 32 rows of 32 columns on their way to whole sectors
    static constexpr int TMEM_COLS = BN > 128 ? 512 : 256;    // two accumulators, the second at half of them
    static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + OUT_BYTES + 1024 + 256;
    static_assert(BN % 64 == 0 && BN <= 256 && OUT % 32 == 0 && OUT >= 64 && B_BYTES % 1024 == 0 && SMEM <= 232448, "tile");
};

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t leader_addr(const void* p) {          // shared::cluster address of rank 0's copy of a shared variable
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
    return a;
}
// a copy into this CTA's shared memory that reports to a barrier of the pair's leader
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(leader_bar)
        : "memory");
}
__device__ __forceinline__ void umma2_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on this barrier of both CTAs once every MMA issued so far by this thread has completed
__device__ __forceinline__ void umma2_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}

// EPI_HEADS: the 256 columns of a tile are two heads of q | k | v, one for each of the two warps of a quarter.  A thread holds a
// whole row of a head: norm and rotation need nobody else, the row goes to C (q) or to the caches (k, v).  Row s is position pos0 + s
// of one sequence or, with row_pos, position row_pos[s] of sequence row_seq[s], whose caches begin that many times seq_stride in.
// On one SM per tile, with nothing to hide it, this epilogue was slower than a kernel of its own; here it runs under the next tile's
// products: 64 x 1024 packed rows 83.1 -> 76.7 ms, 32 prompts of 256 to 512 15.1 -> 14.1, 2048 rows 3.63 -> 3.58.
enum { EPI_HEADS = 6 };
struct Heads {
    const bf16 *q_norm, *k_norm, *cos, *sin;
    bf16 *k_cache, *v_cache;
    int layer, pos0, max_seq;
    const int *row_pos, *row_seq;
    size_t seq_stride;
};
// x: the head's 128 values, pairs 2 i, 2 i + 1; the same operations in the same order as head_norm_rope, whose lane i holds x[i] and x[32 + i]
__device__ __forceinline__ void row_norm_rope(uint32_t (&x)[64], const bf16* w, const bf16* cosr, const bf16* sinr) {
    float p[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const float a = bf_lo(x[i]), b = bf_hi(x[i]), c = bf_lo(x[32 + i]), d = bf_hi(x[32 + i]);
        p[i] = fmaf(d, d, fmaf(c, c, fmaf(b, b, a * a)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) p[i] += p[i + o];
    const float r = 1.0f / sqrtf(p[0] * (1.0f / D) + RMS_EPS);
#pragma unroll
    for (int q = 0; q < 8; ++q) {                                   // eight columns of either half
        auto words = [](const bf16* m, int at) { return __ldg(reinterpret_cast<const uint4*>(m + at)); };
        const uint4 w4[2] = {words(w, 8 * q), words(w, 64 + 8 * q)}, c4[2] = {words(cosr, 8 * q), words(cosr, 64 + 8 * q)}, s4[2] = {words(sinr, 8 * q), words(sinr, 64 + 8 * q)};
        auto pick = [](const uint4& v, int e) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; };
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = 4 * q + e;
            const uint32_t wl = pick(w4[0], e), wh = pick(w4[1], e), cl = pick(c4[0], e), ch = pick(c4[1], e), sl = pick(s4[0], e), sh = pick(s4[1], e);
            const float nl0 = rbf(bf_lo(wl) * rbf(bf_lo(x[i]) * r)), nl1 = rbf(bf_hi(wl) * rbf(bf_hi(x[i]) * r));
            const float nh0 = rbf(bf_lo(wh) * rbf(bf_lo(x[32 + i]) * r)), nh1 = rbf(bf_hi(wh) * rbf(bf_hi(x[32 + i]) * r));
            x[i] = pack_bf16x2(rbf(nl0 * bf_lo(cl)) + rbf(-nh0 * bf_lo(sl)), rbf(nl1 * bf_hi(cl)) + rbf(-nh1 * bf_hi(sl)));
            x[32 + i] = pack_bf16x2(rbf(nh0 * bf_lo(ch)) + rbf(nl0 * bf_lo(sh)), rbf(nh1 * bf_hi(ch)) + rbf(nl1 * bf_hi(sh)));
        }
    }
}

struct Gemm2Args {
    int M, N, K, ldc;              // N: output columns
    int tiles0, tiles1;            // B is up to three matrices along N (GLU: gate and up): tiles [0, tiles0) the first, the next tiles1 the second
    int tiles_m, tiles_n, ksplit;  // PARTIAL: tiles of plane z = 0, then of z = 1, ..
    bf16* C;
    const bf16* R;
    unsigned int* status;
    int early_b;                   // B is written by nothing on the stream
    int drop_kb;                   // test hook: the k-block, counted over a pair's tiles, that is never requested; -1 in every production launch
};

template <int BN, int EPI, class Sink = NoSink>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G2_THREADS, 1)
k_gemm2(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmB2,
        const __grid_constant__ CUtensorMap tmB3, Gemm2Args a, Sink sink) {
    using Cfg = Gemm2Cfg<BN, EPI>;
    constexpr int ST = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);   // the same offset in both CTAs
    uint8_t* outbuf = smem + (size_t)ST * Cfg::STAGE_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(outbuf + Cfg::OUT_BYTES);   // the leader's: both CTAs' copies of a stage have landed
    uint64_t* empty = full + ST;                                            // both: the stage has been multiplied
    uint64_t* acc_full = empty + ST;                                        // [2] both: an accumulator is complete
    uint64_t* acc_free = acc_full + 2;                                      // [2] the leader's: sixteen warps have read it
    uint64_t* drained = acc_free + 2;                                       // after an expired wait: the products issued so far
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile uint32_t* aborted = tmem_slot + 1;                             // a bounded wait of this CTA has run out
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool leader = cluster_rank() == 0;
    const int side = leader ? 0 : 1;
    const int kblocks = (a.K + GM_BK - 1) / GM_BK, plane_tiles = a.tiles_m * a.tiles_n, tiles = plane_tiles * a.ksplit;
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (tid == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_free[s], 2 * GM_EPI_WARPS); }
        mbar_init(drained, 1);
        mbar_fence_init();
        *aborted = 0u;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)Cfg::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                       // barriers of both CTAs stand before either's copies and commits reach them
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    pdl_trigger();                            // behind the allocation: nothing that is launched early can take the columns from this grid

    // tile t: rows 256 tm, column tile tn, k-blocks [kb0, kb0 + nk) of plane z
    auto place = [&](int t, int& tm, int& tn, int& z, int& kb0, int& nk) {
        z = t / plane_tiles;
        const int u = t - z * plane_tiles;
        tm = u / a.tiles_n; tn = u - tm * a.tiles_n;
        kb0 = (int)(((long long)z * kblocks) / a.ksplit);
        nk = (int)(((long long)(z + 1) * kblocks) / a.ksplit) - kb0;
    };
    auto load_b = [&](uint8_t* st, uint32_t bar, int tn, int kb) {
        if (Cfg::GLU) {
            tma_load_2d_pair(st + Cfg::A_BYTES, leader ? &tmB : &tmB2, kb * GM_BK, tn * (BN / 2), bar);
        } else {
            const CUtensorMap* m = tn < a.tiles0 ? &tmB : tn < a.tiles0 + a.tiles1 ? &tmB2 : &tmB3;
            const int tt = tn < a.tiles0 ? tn : tn < a.tiles0 + a.tiles1 ? tn - a.tiles0 : tn - a.tiles0 - a.tiles1;
            tma_load_2d_pair(st + Cfg::A_BYTES, m, kb * GM_BK, tt * BN + side * (BN / 2), bar);
        }
    };

    int c = 0, npre = 0;                      // k-blocks requested so far, over all tiles, and those whose B tile is requested early (producer)
    if (warp == 0) {
        if (lane == 0) {
            if (a.early_b && first < tiles) { // the first tile's weights, ring permitting, before the preceding grid has finished
                int tm, tn, z, kb0, nk;
                place(first, tm, tn, z, kb0, nk);
                npre = nk < ST ? nk : ST;
                for (int i = 0; i < npre; ++i) {
                    if (i == a.drop_kb) continue;
                    if (leader) mbar_expect_tx(&full[i], 2 * Cfg::STAGE_BYTES);
                    load_b(smem + (size_t)i * Cfg::STAGE_BYTES, leader_addr(&full[i]), tn, kb0 + i);
                }
            }
            pdl_wait();
            for (int t = first; t < tiles && !*aborted; t += step) {
                int tm, tn, z, kb0, nk;
                place(t, tm, tn, z, kb0, nk);
                for (int i = 0; i < nk; ++i, ++c) {
                    const int s = c % ST;
                    if (c >= ST && !mbar_wait(&empty[s], (uint32_t)(c / ST - 1) & 1u, a.status)) { *aborted = 1u; break; }
                    if (c == a.drop_kb) continue;
                    uint8_t* st = smem + (size_t)s * Cfg::STAGE_BYTES;
                    const uint32_t bar = leader_addr(&full[s]);
                    if (c >= npre && leader) mbar_expect_tx(&full[s], 2 * Cfg::STAGE_BYTES);
                    tma_load_2d_pair(st, &tmA, (kb0 + i) * GM_BK, tm * 256 + side * 128, bar);
                    if (c >= npre) load_b(st, bar, tn, kb0 + i);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (leader && lane == 0) {
            // D = f32, A = B = bf16, both K-major, N >> 3, M = 256 >> 4
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            int it = 0;
            for (int t = first; t < tiles && !*aborted; t += step, ++it) {
                int tm, tn, z, kb0, nk;
                place(t, tm, tn, z, kb0, nk);
                const int as = it & 1;
                if (it >= 2 && !mbar_wait(&acc_free[as], (uint32_t)((it >> 1) - 1) & 1u, a.status)) { *aborted = 1u; break; }
                tc_fence_after();
                const uint32_t d = tmem + as * (Cfg::TMEM_COLS / 2);
                for (int i = 0; i < nk; ++i, ++c) {
                    const int s = c % ST;
                    if (!mbar_wait(&full[s], (uint32_t)(c / ST) & 1u, a.status)) { *aborted = 1u; break; }
                    tc_fence_after();
                    const uint64_t da = smem_desc_sw128(smem + (size_t)s * Cfg::STAGE_BYTES), db = smem_desc_sw128(smem + (size_t)s * Cfg::STAGE_BYTES + Cfg::A_BYTES);
#pragma unroll
                    for (int k = 0; k < GM_BK / 16; ++k) umma2_bf16(d, da + 2 * k, db + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma2_commit(&empty[s]);
                }
                if (!*aborted) umma2_commit(&acc_full[as]);
            }
            if (*aborted) {                   // tensor memory is freed below: nothing may still be writing it
                umma2_commit(drained);
                mbar_wait_drain(drained, 0);
            }
        }
        __syncwarp();
    } else {
        pdl_wait();
        // warp w reads lanes 32 (w % 4) .. of tensor memory; the two warps of a quarter take 32-column pieces in turn
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        uint8_t* buf = outbuf + (warp - 2) * 2048;
        int it = 0;
        for (int t = first; t < tiles; t += step, ++it) {
            int tm, tn, z, kb0, nk;
            place(t, tm, tn, z, kb0, nk);
            const int as = it & 1;
            const bool ok = mbar_wait(&acc_full[as], (uint32_t)(it >> 1) & 1u, a.status);
            if (!__all_sync(0xffffffffu, ok && !*aborted)) { *aborted = 1u; break; }
            tc_fence_after();
            const int row0 = tm * 256 + side * 128 + quarter * 32, row = row0 + lane;
            const uint32_t trow = tmem + as * (Cfg::TMEM_COLS / 2) + ((uint32_t)(quarter * 32) << 16);
            constexpr int PIECES = Cfg::OUT / 32;
            if constexpr (EPI == EPI_HEADS) {
                static_assert(BN == 256, "two heads");
                uint32_t x[64];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t v[32];
                    tmem_ld32(trow + half * 128 + c * 32, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) x[c * 16 + j] = pack_bf16x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_addr(&acc_free[as])) : "memory");
                const int head = tn * 2 + half, rr = min(row, a.M - 1);
                const bool is_q = head < NQ, is_v = head >= NQ + NKV;
                const int pos = sink.row_pos ? min(max(sink.row_pos[rr], 0), sink.max_seq - 1) : sink.pos0 + rr;
                if (!is_v) row_norm_rope(x, is_q ? sink.q_norm : sink.k_norm, sink.cos + (size_t)pos * D, sink.sin + (size_t)pos * D);
                const size_t seq = sink.row_pos ? (size_t)sink.row_seq[rr] * sink.seq_stride : 0;
                bf16* mine = is_q ? a.C + (size_t)rr * a.ldc + head * D
                                  : (is_v ? sink.v_cache : sink.k_cache) + seq + ((size_t)(sink.layer * NKV + head - (is_v ? NQ + NKV : NQ)) * sink.max_seq + pos) * D;
#pragma unroll
                for (int c = 0; c < 4; ++c) {             // through shared memory as below
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        *reinterpret_cast<uint4*>(buf + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) =
                            make_uint4(x[c * 16 + 4 * q], x[c * 16 + 4 * q + 1], x[c * 16 + 4 * q + 2], x[c * 16 + 4 * q + 3]);
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const int r = g * 8 + (lane >> 2), q = lane & 3;
                        bf16* to = reinterpret_cast<bf16*>(__shfl_sync(0xffffffffu, (unsigned long long)mine, r));
                        const uint4 w = *reinterpret_cast<const uint4*>(buf + r * 64 + ((q ^ ((r >> 1) & 3)) << 4));
                        if (row0 + r < a.M) *reinterpret_cast<uint4*>(to + c * 32 + q * 8) = w;
                    }
                    __syncwarp();
                }
            } else
#pragma unroll 1
            for (int p = half; p < PIECES; p += 2) {
                uint32_t v[32], out[16];
                tmem_ld32_nowait(trow + p * 32, v);
                if constexpr (Cfg::GLU) {
                    uint32_t u[32];
                    tmem_ld32_nowait(trow + Cfg::OUT + p * 32, u);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float g0 = rbf(__uint_as_float(v[2 * j])), g1 = rbf(__uint_as_float(v[2 * j + 1]));
                        const float u0 = rbf(__uint_as_float(u[2 * j])), u1 = rbf(__uint_as_float(u[2 * j + 1]));
                        out[j] = pack_bf16x2(rbf(silu_fast(g0)) * u0, rbf(silu_fast(g1)) * u1);
                    }
                } else {
                    tmem_ld_wait();
                }
                if (p + 2 >= PIECES) {        // this warp has read its part of the accumulator
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_addr(&acc_free[as])) : "memory");
                }
                const int n0 = tn * Cfg::OUT + p * 32;
                if constexpr (EPI == EPI_PARTIAL) {
                    if (row < a.M) {
                        float4* fp = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.C) + ((size_t)z * a.M + row) * a.ldc + n0);
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            fp[q] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
                    }
                } else if constexpr (EPI == EPI_SINK) {
                    if (row < a.M) sink(row, n0, v);
                } else {
                    if constexpr (!Cfg::GLU) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) out[j] = pack_bf16x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                    }
                    // a lane holds 64 bytes of one row; through shared memory four lanes store them side by side, eight rows at once.
                    // 16-byte piece q of row r stands at q ^ (r / 2 % 4): no bank twice in either direction.
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        *reinterpret_cast<uint4*>(buf + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) = make_uint4(out[4 * q], out[4 * q + 1], out[4 * q + 2], out[4 * q + 3]);
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const int r = g * 8 + (lane >> 2), q = lane & 3;
                        uint4 w = *reinterpret_cast<const uint4*>(buf + r * 64 + ((q ^ ((r >> 1) & 3)) << 4));
                        if (row0 + r < a.M) {
                            const size_t at = (size_t)(row0 + r) * a.ldc + n0 + q * 8;
                            if constexpr (EPI == EPI_RESID) {
                                const uint4 h = *reinterpret_cast<const uint4*>(a.R + at);
                                w = make_uint4(pack_bf16x2(bf_lo(h.x) + bf_lo(w.x), bf_hi(h.x) + bf_hi(w.x)), pack_bf16x2(bf_lo(h.y) + bf_lo(w.y), bf_hi(h.y) + bf_hi(w.y)),
                                               pack_bf16x2(bf_lo(h.z) + bf_lo(w.z), bf_hi(h.z) + bf_hi(w.z)), pack_bf16x2(bf_lo(h.w) + bf_lo(w.w), bf_hi(h.w) + bf_hi(w.w)));
                            }
                            *reinterpret_cast<uint4*>(a.C + at) = w;
                        }
                    }
                    __syncwarp();
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    // After an expired wait (which the other CTA of the pair then runs into as well): copies that were requested still land.  The leader
    // waits for the last of every stage, with a limit; the other CTA, whose copies report to the leader's barriers, for as long as that limit.
    if (*aborted && tid == 0) {
        if (leader)
            for (int s = 0; s < ST && s < max(c, npre); ++s) mbar_wait_drain(&full[s], c > s ? (uint32_t)((c - 1 - s) / ST) & 1u : 0u);
        else
            for (const long long t0 = clock64(); clock64() - t0 < DRAIN_LIMIT_CYCLES;) {}
    }
    __syncwarp();
    cluster_sync_all();                       // both CTAs' copies, products and remote arrivals are done
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)Cfg::TMEM_COLS) : "memory");
}

// Arguments as launch_gemm's.  N is a multiple of the tile's width, except for a sink (which looks at the column) and
// for planes at least as wide as the tiles.
template <int BN, int EPI, class Sink = NoSink>
static int launch_gemm2(const bf16* A, int lda, const bf16* B, const bf16* B2, bf16* C, const bf16* R, int M, int N, int K, int ldc, unsigned int* status,
                        cudaStream_t stream, const bf16* B3 = nullptr, int rows0 = 0, int rows1 = 0, int ksplit = 1, bool early_b = true, Sink sink = Sink(), int drop_kb = -1) {
    using Cfg = Gemm2Cfg<BN, EPI>;
    static int sms[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return MQ_ERR_UNSUPPORTED;
    if (!sms[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_gemm2<BN, EPI, Sink>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM);
        int n = 0;
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        sms[dev] = n;
    }
    Gemm2Args a = {};
    const bool concat = rows0 > 0;
    a.tiles_n = (N + Cfg::OUT - 1) / Cfg::OUT; a.tiles_m = (M + 255) / 256; a.ksplit = ksplit;
    const int kblocks = (K + GM_BK - 1) / GM_BK;
    if (EPI != EPI_SINK && N % Cfg::OUT != 0 && !(EPI == EPI_PARTIAL && ldc >= a.tiles_n * Cfg::OUT)) return MQ_ERR_BAD_ARG;
    if (K % 8 != 0 || (EPI != EPI_SINK && EPI != EPI_PARTIAL && K % GM_BK != 0)) return MQ_ERR_BAD_ARG;
    if (concat && (rows0 % BN || rows1 % BN || Cfg::GLU)) return MQ_ERR_BAD_ARG;
    if (ksplit < 1 || (ksplit > 1 && EPI != EPI_PARTIAL) || kblocks < ksplit) return MQ_ERR_BAD_ARG;
    CUtensorMap ma, mb, mb2, mb3;
    int rc = get_map(A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 128, &ma);
    if (rc == MQ_OK) rc = get_map(B, (uint64_t)(concat ? rows0 : N), (uint64_t)K, (uint64_t)K, BN / 2, &mb);
    if (rc != MQ_OK) return rc;
    mb2 = mb3 = mb;
    if (Cfg::GLU) {
        rc = get_map(B2, (uint64_t)N, (uint64_t)K, (uint64_t)K, BN / 2, &mb2);
    } else if (concat) {
        rc = get_map(B2, (uint64_t)rows1, (uint64_t)K, (uint64_t)K, BN / 2, &mb2);
        if (rc == MQ_OK) rc = get_map(B3, (uint64_t)(N - rows0 - rows1), (uint64_t)K, (uint64_t)K, BN / 2, &mb3);
    }
    if (rc != MQ_OK) return rc;
    a.M = M; a.N = N; a.K = K; a.ldc = ldc; a.C = C; a.R = R; a.status = status; a.early_b = early_b ? 1 : 0; a.drop_kb = drop_kb;
    a.tiles0 = concat ? rows0 / BN : (1 << 30);
    a.tiles1 = concat ? rows1 / BN : 0;
    const int tiles = a.tiles_m * a.tiles_n * ksplit, pairs = sms[dev] / 2;
    launch_pdl(k_gemm2<BN, EPI, Sink>, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(G2_THREADS), Cfg::SMEM, stream, ma, mb, mb2, mb3, a, sink);
    return (int)cudaGetLastError();
}

}  // namespace mq
