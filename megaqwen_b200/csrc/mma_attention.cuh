// Causal attention of prompts, and portions of prompts, of fewer than 128 rows: tiles of 64 queries on mma.sync.
#pragma once

#include "tc_core.cuh"

namespace mq {

// QK^T and PV run on mma.sync m16n8k16 (bf16 in, fp32 accumulate) with an online softmax in
// registers; probabilities are rounded to bf16 before the PV product and the row sum uses the
// unrounded values.
// Causal attention of the prompt.  One CTA per (query head, 64-query tile).  Under the causal
// mask the last query tile of a prompt has sixteen times the work of the first, and the pass
// is as long as its longest CTA, so the key tiles of a query tile are dealt out to FA_NG
// groups of four warps that walk them in parallel (group g takes key tiles g, g + FA_NG, ..)
// and are merged through shared memory at the end; the grid is ordered longest query tile
// first.  Each group streams its K/V tiles through its own two-stage ring of padded rows
// (16-byte cp.async, the next tile in flight while this one is multiplied).
constexpr int FA_BQ = 64, FA_BK = 64, FA_LD = D + 8, FA_NG = 2, FA_THREADS = FA_NG * 128;
constexpr int FA_TILE_ELEMS = FA_BK * FA_LD;                                  // one K or V tile
constexpr size_t FA_SMEM = (size_t)(FA_BQ * FA_LD + FA_NG * 2 * 2 * FA_TILE_ELEMS) * 2;

__device__ __forceinline__ void group_barrier(int group) {
    asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const bf16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const bf16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One query tile, rows q0 .. q0 + 63 of S queries at positions pos0 .., of query head `head`, by the first FA_THREADS threads of a CTA (the
// others have left).  qkv: the row of query 0; kbase, vbase: the head's cached rows; out: row 0 of the result.
__device__ __forceinline__ void fa_tile(uint8_t* fa_smem, const bf16* qkv, const bf16* kbase, const bf16* vbase, bf16* out, int S, int pos0, int q0, int head) {
    bf16* sq = reinterpret_cast<bf16*>(fa_smem);                    // [64][FA_LD]
    bf16* ring = sq + FA_BQ * FA_LD;                                // [FA_NG][2 stages][K tile | V tile]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = warp >> 2, wq = warp & 3, gtid = tid & 127;
    bf16* gring = ring + (size_t)grp * 4 * FA_TILE_ELEMS;

    const int kv_end = min(pos0 + S, pos0 + q0 + FA_BQ);     // exclusive bound of keys any row of the tile may see
    const int ntiles = (kv_end + FA_BK - 1) / FA_BK;
    auto load_tile = [&](int t, int stage) {
        bf16* sk = gring + (size_t)stage * 2 * FA_TILE_ELEMS;
        bf16* sv = sk + FA_TILE_ELEMS;
        const int p0 = t * FA_BK;
        for (int c = gtid; c < FA_BK * (D / 8); c += 128) {
            const int r = c / (D / 8), cc = c % (D / 8);
            const bool ok = p0 + r < kv_end;
            const size_t off = (size_t)(ok ? p0 + r : 0) * D + cc * 8;
            cp_async16_zfill(sk + r * FA_LD + cc * 8, kbase + off, ok);
            cp_async16_zfill(sv + r * FA_LD + cc * 8, vbase + off, ok);
        }
    };
    if (grp < ntiles) load_tile(grp, 0);
    cp_async_commit();

    // Q tile -> shared (rows past S are zero)
    for (int c = tid; c < FA_BQ * (D / 8); c += FA_THREADS) {
        const int r = c / (D / 8), cc = c % (D / 8);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (q0 + r < S) v = ld_cg_u4(qkv + (size_t)(q0 + r) * QKV + head * D + cc * 8);
        *reinterpret_cast<uint4*>(sq + r * FA_LD + cc * 8) = v;
    }
    __syncthreads();
    uint32_t qf[8][4];
#pragma unroll
    for (int kk = 0; kk < 8; ++kk)
        ldsm_x4(qf[kk], sq + (wq * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * FA_LD + kk * 16 + (lane >> 4) * 8);

    float o[16][4];
#pragma unroll
    for (int i = 0; i < 16; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m_run[2] = {-1e30f, -1e30f}, l_run[2] = {0.f, 0.f};
    // scores are kept in the log2 domain (scale * log2(e) folded in) so that the softmax uses
    // the single-instruction exp2 instead of expf; the probabilities are the same numbers
    const float scale = 0.08838834764831845f * 1.4426950408889634f;
    const int row_a = pos0 + q0 + wq * 16 + (lane >> 2);   // absolute position of this thread's first row; second is +8

    int it = 0;
    for (int t = grp; t < ntiles; t += FA_NG, ++it) {
        // the other stage was consumed in the previous iteration (barrier at its end): request the next tile
        if (t + FA_NG < ntiles) load_tile(t + FA_NG, (it + 1) & 1);
        cp_async_commit();
        cp_async_wait<1>();          // this thread's copies of tile t have landed
        group_barrier(grp);          // .. and everybody's in the group
        const bf16* sk = gring + (size_t)(it & 1) * 2 * FA_TILE_ELEMS;
        const bf16* sv = sk + FA_TILE_ELEMS;
        const int p0 = t * FA_BK;

        float sacc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) { sacc[i][0] = sacc[i][1] = sacc[i][2] = sacc[i][3] = 0.f; }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
#pragma unroll
            for (int np = 0; np < 4; ++np) {   // pairs of 8-key tiles
                uint32_t kf[4];
                ldsm_x4(kf, sk + (np * 16 + (lane & 7) + (lane >> 4) * 8) * FA_LD + kk * 16 + ((lane >> 3) & 1) * 8);
                mma_bf16_16816(sacc[2 * np], qf[kk], kf[0], kf[1]);
                mma_bf16_16816(sacc[2 * np + 1], qf[kk], kf[2], kf[3]);
            }
        }
        // scale, causal mask, online softmax
        float mx[2] = {-1e30f, -1e30f};
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = p0 + nt * 8 + (lane & 3) * 2 + (e & 1);
                const int rowp = row_a + (e >> 1) * 8;
                const float sv_ = (key <= rowp) ? sacc[nt][e] * scale : -1e30f;
                sacc[nt][e] = sv_;
                mx[e >> 1] = fmaxf(mx[e >> 1], sv_);
            }
        }
        float corr[2];
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            mx[h2] = fmaxf(mx[h2], __shfl_xor_sync(0xffffffffu, mx[h2], 1));
            mx[h2] = fmaxf(mx[h2], __shfl_xor_sync(0xffffffffu, mx[h2], 2));
            const float m_new = fmaxf(m_run[h2], mx[h2]);
            corr[h2] = fast_exp2(m_run[h2] - m_new);
            m_run[h2] = m_new;
        }
        float rs[2] = {0.f, 0.f};
        uint32_t pf[4][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            float pe[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                pe[e] = (sacc[nt][e] <= -1e29f) ? 0.f : fast_exp2(sacc[nt][e] - m_run[e >> 1]);
                rs[e >> 1] += pe[e];
            }
            pf[nt >> 1][(nt & 1) * 2 + 0] = pack_bf16x2(pe[0], pe[1]);
            pf[nt >> 1][(nt & 1) * 2 + 1] = pack_bf16x2(pe[2], pe[3]);
        }
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            rs[h2] += __shfl_xor_sync(0xffffffffu, rs[h2], 1);
            rs[h2] += __shfl_xor_sync(0xffffffffu, rs[h2], 2);
            l_run[h2] = l_run[h2] * corr[h2] + rs[h2];
        }
#pragma unroll
        for (int dt = 0; dt < 16; ++dt) { o[dt][0] *= corr[0]; o[dt][1] *= corr[0]; o[dt][2] *= corr[1]; o[dt][3] *= corr[1]; }
        // O += P V
#pragma unroll
        for (int j = 0; j < 4; ++j) {          // 16 keys per step
#pragma unroll
            for (int dp = 0; dp < 8; ++dp) {   // pairs of 8-wide output tiles
                uint32_t vf[4];
                ldsm_x4_t(vf, sv + (j * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * FA_LD + dp * 16 + (lane >> 4) * 8);
                mma_bf16_16816(o[2 * dp], pf[j], vf[0], vf[1]);
                mma_bf16_16816(o[2 * dp + 1], pf[j], vf[2], vf[3]);
            }
        }
        group_barrier(grp);          // the stage may be overwritten by the next iteration's request
    }
    cp_async_wait_all();
    __syncthreads();
    // merge the groups: groups 1.. leave (m, l, O) of every thread in the ring, group 0 combines
    float* xch = reinterpret_cast<float*>(ring);        // [FA_NG - 1][128 threads][68]
    if (grp > 0) {
        float* mine = xch + ((size_t)(grp - 1) * 128 + gtid) * 68;
        mine[0] = m_run[0]; mine[1] = m_run[1]; mine[2] = l_run[0]; mine[3] = l_run[1];
#pragma unroll
        for (int dt = 0; dt < 16; ++dt) *reinterpret_cast<float4*>(mine + 4 + dt * 4) = make_float4(o[dt][0], o[dt][1], o[dt][2], o[dt][3]);
    }
    __syncthreads();
    if (grp > 0) return;
#pragma unroll
    for (int og = 1; og < FA_NG; ++og) {
        const float* oth = xch + ((size_t)(og - 1) * 128 + gtid) * 68;
        float f_me[2], f_ot[2];
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            const float mo = oth[h2], mn = fmaxf(m_run[h2], mo);
            f_me[h2] = fast_exp2(m_run[h2] - mn);
            f_ot[h2] = fast_exp2(mo - mn);
            l_run[h2] = l_run[h2] * f_me[h2] + oth[2 + h2] * f_ot[h2];
            m_run[h2] = mn;
        }
#pragma unroll
        for (int dt = 0; dt < 16; ++dt) {
            const float4 ov = *reinterpret_cast<const float4*>(oth + 4 + dt * 4);
            o[dt][0] = o[dt][0] * f_me[0] + ov.x * f_ot[0];
            o[dt][1] = o[dt][1] * f_me[0] + ov.y * f_ot[0];
            o[dt][2] = o[dt][2] * f_me[1] + ov.z * f_ot[1];
            o[dt][3] = o[dt][3] * f_me[1] + ov.w * f_ot[1];
        }
    }
    // normalise and store
    const int r_lo = q0 + wq * 16 + (lane >> 2), r_hi = r_lo + 8;
    const float inv0 = 1.0f / l_run[0], inv1 = 1.0f / l_run[1];
#pragma unroll
    for (int dt = 0; dt < 16; ++dt) {
        const int col = head * D + dt * 8 + (lane & 3) * 2;
        if (r_lo < S) *reinterpret_cast<uint32_t*>(out + (size_t)r_lo * QSZ + col) = pack_bf16x2(o[dt][0] * inv0, o[dt][1] * inv0);
        if (r_hi < S) *reinterpret_cast<uint32_t*>(out + (size_t)r_hi * QSZ + col) = pack_bf16x2(o[dt][2] * inv1, o[dt][3] * inv1);
    }
}

}  // namespace mq
