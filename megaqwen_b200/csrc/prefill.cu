// Prefill (full-sequence forward) for sm_100a.
//
// The reference runs prefill as 7 cuBLAS GEMMs per layer plus ~14 small kernels
// and a serial-per-warp O(S^2) attention (csrc/megakernel/fused_prefill_launch.inl:71-731,
// fused_prefill_kernels.inl:3-824).  Here the dense contractions run on the
// 5th-generation tensor cores directly: one kernel per GEMM that stages both
// operands with TMA (128-byte swizzle) into a multi-stage shared-memory ring,
// issues tcgen05.mma from a single elected thread into a TMEM accumulator and
// drains it with tcgen05.ld in four epilogue warps, with the residual add and
// the SwiGLU product fused into the epilogue.  Activations are bf16 between
// all ops (the rounding points of the HF bf16 model, as in the reference's
// launch_prefill_float).
//
// Every mbarrier wait is bounded (mq_device.cuh) and TMEM is always freed.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mma_attention.cuh"
#include "sk_chain.cuh"
#include "tc_attention.cuh"
#include "tc_gemm2.cuh"

namespace mq {

// h = bf16(h + bf16(sum of the two fp32 planes of a K split));  x = rmsnorm(h) * w      one CTA per row (N = 1024), 4 columns per thread
__global__ void __launch_bounds__(256) k_sk_resid_norm(const float* part, int M, bf16* __restrict__ h,
                                                       const bf16* __restrict__ w, bf16* __restrict__ x) {
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    __shared__ float s_red[8];
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t base = (size_t)row * H + 4 * tid, plane = (size_t)M * H;
    const uint2 hu = ld_cg_u2(h + base);
    const uint2 wu = w ? *reinterpret_cast<const uint2*>(w + 4 * tid) : make_uint2(0u, 0u);   // requested with the planes, used after the row sum
    const float4 p0 = __ldcg(reinterpret_cast<const float4*>(part + base)), p1 = __ldcg(reinterpret_cast<const float4*>(part + plane + base));
    const float4 acc = make_float4(p0.x + p1.x, p0.y + p1.y, p0.z + p1.z, p0.w + p1.w);
    float v[4] = {rbf(bf_lo(hu.x) + rbf(acc.x)), rbf(bf_hi(hu.x) + rbf(acc.y)), rbf(bf_lo(hu.y) + rbf(acc.z)), rbf(bf_hi(hu.y) + rbf(acc.w))};
    *reinterpret_cast<uint2*>(h + base) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    if (!w) return;   // residual stream only (after the last layer nothing is normalised here)
    float ss = warp_sum(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3]);
    if (lane == 0) s_red[warp] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += s_red[i];
    const float r = 1.0f / sqrtf(tot * (1.0f / H) + RMS_EPS);
    const uint2 o = make_uint2(pack_bf16x2(rbf(bf_lo(wu.x) * rbf(v[0] * r)), rbf(bf_hi(wu.x) * rbf(v[1] * r))),
                               pack_bf16x2(rbf(bf_lo(wu.y) * rbf(v[2] * r)), rbf(bf_hi(wu.y) * rbf(v[3] * r))));
    *reinterpret_cast<uint2*>(x + base) = o;
}

// ---------------------------------------------------------------- row-wise kernels
// h[s,:] = embed[ids[s],:]      (reference: prefill_embed_kernel, fused_prefill_kernels.inl:3-20)
// Rows audio_start .. audio_start + audio_len - 1 take externally computed embeddings instead
// (reference: prefill_patch_audio_kernel, fused_prefill_kernels.inl:28-45, a separate launch there).
__global__ void __launch_bounds__(128) k_pf_embed(const int* ids, const bf16* __restrict__ embed, bf16* __restrict__ h,
                                                  int vocab, unsigned int* status, const bf16* __restrict__ audio = nullptr,
                                                  int audio_start = 0, int audio_len = 0) {
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    pdl_trigger();   // only now: the kernels behind may read cache rows of earlier passes ahead of their own waits
    const int s = blockIdx.x;
    if (audio != nullptr && s >= audio_start && s < audio_start + audio_len) {
        reinterpret_cast<uint4*>(h + (size_t)s * H)[threadIdx.x] =
            __ldg(reinterpret_cast<const uint4*>(audio + (size_t)(s - audio_start) * H) + threadIdx.x);
        return;
    }
    int tok = ld_cg_i32(ids + s);
    if (tok < 0 || tok >= vocab) {
        if (threadIdx.x == 0) atomicOr(status, MQ_STATUS_BAD_TOKEN);
        tok = min(max(tok, 0), vocab - 1);
    }
    reinterpret_cast<uint4*>(h + (size_t)s * H)[threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(embed + (size_t)tok * H) + threadIdx.x);
}

// x[s,:] = bf16( w * bf16( h[s,:] * rsqrt(mean(h^2) + eps) ) )   one warp per row
// (reference: prefill_rmsnorm_kernel, fused_prefill_kernels.inl:52-105)
__global__ void __launch_bounds__(256) k_pf_rmsnorm(const bf16* h, const bf16* __restrict__ w, bf16* __restrict__ x, int rows) {
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    float v[32];
    const bf16* src = h + (size_t)row * H;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 u = ld_cg_u4(src + j * 256 + lane * 8);
        v[j * 8 + 0] = bf_lo(u.x); v[j * 8 + 1] = bf_hi(u.x); v[j * 8 + 2] = bf_lo(u.y); v[j * 8 + 3] = bf_hi(u.y);
        v[j * 8 + 4] = bf_lo(u.z); v[j * 8 + 5] = bf_hi(u.z); v[j * 8 + 6] = bf_lo(u.w); v[j * 8 + 7] = bf_hi(u.w);
    }
    rmsnorm_slice(v, w, lane);
    bf16* dst = x + (size_t)row * H;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint4 o;
        o.x = pack_bf16x2(v[j * 8 + 0], v[j * 8 + 1]); o.y = pack_bf16x2(v[j * 8 + 2], v[j * 8 + 3]);
        o.z = pack_bf16x2(v[j * 8 + 4], v[j * 8 + 5]); o.w = pack_bf16x2(v[j * 8 + 6], v[j * 8 + 7]);
        *reinterpret_cast<uint4*>(dst + j * 256 + lane * 8) = o;
    }
}

// Per (position, head): q/k heads get RMSNorm(128) * w and split-half RoPE evaluated in
// bf16; q stays in the qkv buffer, k and v go to the cache at position pos0 + s
// (reference: prefill_qk_norm_rope_kernel, fused_prefill_kernels.inl:112-258).
// One warp per head: 16 q + 8 k + 8 v = 32 warps per position.
__global__ void __launch_bounds__(256) k_pf_qknorm_rope(bf16* __restrict__ qkv, const bf16* __restrict__ wq, const bf16* __restrict__ wk,
                                                        const bf16* __restrict__ cos, const bf16* __restrict__ sin, bf16* __restrict__ k_cache,
                                                        bf16* __restrict__ v_cache, int layer, int pos0, int max_seq,
                                                        const int* pos_rows, size_t seq_stride, const int* row_seq) {
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    // pos_rows == nullptr: one sequence, row s sits at position pos0 + s.
    // pos_rows != nullptr: row s is at position pos_rows[s] of sequence row_seq[s] (sequence s if row_seq is
    // null), whose cache starts that many times seq_stride elements in.
    // A warp handles units (q heads 0..15, k heads 16..23, v heads 24..31) blockIdx.y * 8 + warp,
    // then every gridDim.y * 8 further: one CTA per row with gridDim.y = 1, four with 4.
    const int lane = threadIdx.x & 31;
    const int s = blockIdx.x;
    const int pos = pos_rows ? min(max(ld_cg_i32(pos_rows + s), 0), max_seq - 1) : pos0 + s;
    if (pos_rows) {
        const size_t seq = row_seq ? (size_t)ld_cg_i32(row_seq + s) : (size_t)s;
        k_cache += seq * seq_stride;
        v_cache += seq * seq_stride;
    }
    bf16* row = qkv + (size_t)s * QKV;
    const bf16* cosr = cos + (size_t)pos * D;
    const bf16* sinr = sin + (size_t)pos * D;
    const uint32_t cl = *reinterpret_cast<const uint32_t*>(cosr + 2 * lane), ch = *reinterpret_cast<const uint32_t*>(cosr + 64 + 2 * lane);
    const uint32_t sl = *reinterpret_cast<const uint32_t*>(sinr + 2 * lane), sh = *reinterpret_cast<const uint32_t*>(sinr + 64 + 2 * lane);
    for (int unit = blockIdx.y * 8 + (threadIdx.x >> 5); unit < NQ + 2 * NKV; unit += gridDim.y * 8) {
        if (unit >= NQ + NKV) {   // V head: raw copy into the cache
            const int g = unit - NQ - NKV;
            *reinterpret_cast<uint2*>(v_cache + ((size_t)(layer * NKV + g) * max_seq + pos) * D + 4 * lane) =
                ld_cg_u2(row + QSZ + KVSZ + g * D + 4 * lane);
            continue;
        }
        const bool is_q = unit < NQ;
        bf16* head = is_q ? row + unit * D : row + QSZ + (unit - NQ) * D;
        const bf16* wn = is_q ? wq : wk;
        const uint32_t ulo = ld_cg_u32(head + 2 * lane), uhi = ld_cg_u32(head + 64 + 2 * lane);
        const float xl[2] = {bf_lo(ulo), bf_hi(ulo)}, xh[2] = {bf_lo(uhi), bf_hi(uhi)};
        uint32_t plo, phi;
        head_norm_rope(xl, xh, *reinterpret_cast<const uint32_t*>(wn + 2 * lane), *reinterpret_cast<const uint32_t*>(wn + 64 + 2 * lane), cl, ch, sl, sh, plo, phi);
        bf16* dst = is_q ? head : k_cache + ((size_t)(layer * NKV + (unit - NQ)) * max_seq + pos) * D;
        *reinterpret_cast<uint32_t*>(dst + 2 * lane) = plo;
        *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = phi;
    }
}

// ---------------------------------------------------------------- causal GQA attention of a prompt below 128 rows
__global__ void __launch_bounds__(FA_THREADS, 1) k_pf_attention(const bf16* qkv, const bf16* k_cache, const bf16* v_cache, bf16* out, int S, int pos0,
                                                               int layer, int max_seq) {
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    extern __shared__ __align__(16) uint8_t fa_smem[];
    const int head = blockIdx.x;
    const size_t plane = (size_t)(layer * NKV + head / (NQ / NKV)) * max_seq * D;
    const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * FA_BQ;  // longest query tiles are dispatched first
    fa_tile(fa_smem, qkv, k_cache + plane, v_cache + plane, out, S, pos0, q0, head);
}

// ---------------------------------------------------------------- host side
// defined in decode.cu: final RMSNorm + LM head + arg-max on buf->hidden
int launch_lmhead_only(const MqModel* model, const MqDecodeBuffers* buf, int* out_token, float* logits, cudaStream_t stream);

__global__ void k_pf_copy_row(const bf16* src, bf16* __restrict__ dst) {
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    reinterpret_cast<uint4*>(dst)[threadIdx.x] = ld_cg_u4(src + threadIdx.x * 8);
}

// dst[b] = src[last packed row of sequence b]
__global__ void k_pf_gather_last(const bf16* src, const int* seq_row0, const int* seq_len, bf16* __restrict__ dst) {
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    const int b = blockIdx.x;
    const size_t row = (size_t)ld_cg_i32(seq_row0 + b) + (size_t)ld_cg_i32(seq_len + b) - 1;
    reinterpret_cast<uint4*>(dst + (size_t)b * H)[threadIdx.x] = ld_cg_u4(src + row * H + threadIdx.x * 8);
}

}  // namespace mq

namespace mq {

// ---------------------------------------------------------------- batched decode (one new token per sequence)
// One CTA per (sequence, kv head); the two query heads share the K/V stream.  Each warp owns
// the 16-position tiles warp, warp + 12, .. of the sequence and streams them through its own
// two-stage ring of padded rows in shared memory (16-byte cp.async, the next tile in flight
// while this one is multiplied, no block barrier inside the loop; twelve warps per SM rather
// than eight with deeper rings, because the per-tile chain of dependent instructions, not
// the bytes in flight, bounds a warp; one 256-byte bulk copy per row instead of sixteen
// cp.async was measured slower: 3.07 vs 2.81 ms per step at batch 64).  Per tile: scores = K_tile . q on mma.sync (positions
// are M, the two heads two of the eight N columns), softmax of the tile, P rounded to bf16,
// out += P . V_tile (ldmatrix.trans on V).  About a sixth of the instructions of an fp32-FMA
// loop over the same bytes, which is what bounded the FMA version at 2.7 TB/s.
constexpr int BD_STAGES = 2, BD_LD = D + 8;                                     // per warp: 2 stages x 8.5 KB
constexpr int BD_STAGE_ELEMS = 2 * 16 * BD_LD;                                  // K tile then V tile
// Two shapes: twelve warps, one CTA per SM (209 KB), or six warps, two CTAs per SM (105 KB each).  The
// SM streams with twelve warps either way; bd_shape() below says which is used when.
constexpr size_t bd_smem_bytes(int warps) { return (size_t)warps * BD_STAGES * BD_STAGE_ELEMS * 2 + 2 * D * 2 + warps * 32 * 2; }
constexpr int BD_MAX_PARTS = 4;                                                 // CTAs that may share one item's keys
constexpr int BD_PART = D + 2;                                                  // m, l, acc[128] of one head of one part
// FP8 cache: a warp's ring holds the raw e4m3 rows (K 16 x 128 bytes, then V), two stages, followed
// by ONE padded f16 tile pair the current stage is expanded into before it is multiplied
constexpr int BD8_RAW = 2 * 16 * D;                                             // bytes per raw stage
constexpr int BD8_WARP_BYTES = BD_STAGES * BD8_RAW + BD_STAGE_ELEMS * 2;
static_assert(BD8_WARP_BYTES <= BD_STAGES * BD_STAGE_ELEMS * 2, "the fp8 ring fits the bf16 ring");

__device__ __forceinline__ void bd_load_tile(bf16* stage, const bf16* kb, const bf16* vb, int tile, int len, int lane) {
    // 16 rows x 16 chunks of 16 bytes for K and the same for V: 16 copies per lane.  Rows past
    // the end of the sequence re-read the last row (their probabilities are zero).
    // copy i of a lane is chunk (lane & 15) of row 2 * i + (lane >> 4)
    const int c8 = (lane & 15) * 8, r0 = lane >> 4;
    bf16* sdst = stage + r0 * BD_LD + c8;
    const int last = len - 1 - tile * 16 - r0;            // copies with 2 * i > last re-read the last row
    const size_t gbase = (size_t)(tile * 16 + r0) * D + c8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const size_t goff = gbase + (size_t)min(2 * i, last) * D;
        cp_async16(sdst + 2 * i * BD_LD, kb + goff);
        cp_async16(sdst + (16 + 2 * i) * BD_LD, vb + goff);
    }
}
// e4m3 rows: 16 rows x 8 chunks of 16 bytes for K and for V, 8 copies per lane; copy i of a lane
// is chunk (lane & 7) of row 4 * (i & 3) + (lane >> 3) of K (i < 4) or V
__device__ __forceinline__ void bd_load_tile_fp8(uint8_t* raw, const uint8_t* kb, const uint8_t* vb, int tile, int len, int lane) {
    const int c16 = (lane & 7) * 16, r0 = lane >> 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * i + r0;
        const size_t goff = (size_t)min(tile * 16 + r, len - 1) * D + c16;
        cp_async16(raw + r * D + c16, kb + goff);
        cp_async16(raw + 16 * D + r * D + c16, vb + goff);
    }
}
// the raw stage -> padded f16 tiles (same chunk assignment as the copies)
__device__ __forceinline__ void bd_expand_tile_fp8(const uint8_t* raw, bf16* tile16, int lane) {
    const int c16 = (lane & 7) * 16, r0 = lane >> 3;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 4 * (i & 3) + r0 + (i >> 2) * 16;      // rows 16..31 are V
        const uint4 w = *reinterpret_cast<const uint4*>(raw + r * D + c16);
        uint4 a, b;
        fp8x16_to_f16x16(w, a, b);
        uint4* dst = reinterpret_cast<uint4*>(tile16 + r * BD_LD + c16);
        dst[0] = a;
        dst[1] = b;
    }
}

// FP8 = true: K and V are read from the e4m3 shadow cache (k8 / v8, one scale per sequence, layer
// and kv head: scores are multiplied by the K scale, the output by the V scale; reference:
// decode attention with KV_FP8, csrc/megakernel/split_decode_gemm.cu:950-1310).  The row of
// the new position was written to the bf16 cache by the preceding kernel; this CTA quantises
// it into the shadow cache first (split_decode_gemm.cu:487-493).
// One-dimensional grid: CTAs 0 .. n_full - 1 take one (sequence, kv head) item each; the remaining items
// are split over p_tail CTAs each (CTA n_full + r: item n_full + r / p_tail, part r % p_tail).  The CTAs
// of a split item write their (m, l, acc) to `parts` and take a ticket, and the one that takes the last
// merges them (no CTA waits for another).  tickets: one zero-initialised counter per item, reset by the merger.
template <bool FP8, int WARPS>
__device__ __forceinline__ void bd_attention_body(const bf16* qkv, const bf16* k_cache, const bf16* v_cache,
                                                  bf16* out, const int* positions, int layer, int max_seq,
                                                  size_t seq_stride, uint8_t* __restrict__ k8, uint8_t* __restrict__ v8,
                                                  const float* k_scale, const float* v_scale, int scale_stride,
                                                  float* __restrict__ parts, unsigned int* __restrict__ tickets, int n_full, int p_tail) {
    constexpr int BD_THREADS = WARPS * 32;
    const int cta = (int)blockIdx.x;
    const int item_i = cta < n_full ? cta : n_full + (cta - n_full) / p_tail;
    const int part = cta < n_full ? 0 : (cta - n_full) % p_tail;
    const int nparts = cta < n_full ? 1 : p_tail;
    const int b = item_i / NKV, g = item_i % NKV;
    // the scales are set by the quantise kernel before the first step and constant afterwards
    float ks = 1.f, vs = 1.f;
    if constexpr (FP8) {
        ks = kv_fp8_scale_guard(ld_cg_f32(k_scale + (size_t)b * scale_stride + layer * NKV + g));
        vs = kv_fp8_scale_guard(ld_cg_f32(v_scale + (size_t)b * scale_stride + layer * NKV + g));
    }
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    extern __shared__ __align__(128) uint8_t bd_smem[];
    bf16* ring = reinterpret_cast<bf16*>(bd_smem);                                    // [12 warps][2 stages][K 16 rows | V 16 rows][BD_LD]
    bf16* qs = ring + (size_t)(BD_THREADS / 32) * BD_STAGES * BD_STAGE_ELEMS;         // [2][D]
    bf16* ps = qs + 2 * D;                                                            // [12 warps][2][16]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pos = min(max(ld_cg_i32(positions + b), 0), max_seq - 1);
    const int len = pos + 1;
    const int ntiles_all = (len + 15) >> 4;
    // this CTA's share of the item's key tiles: [tile_lo, ntiles)
    const int tile_lo = (int)(((long long)part * ntiles_all) / nparts);
    const int ntiles = (int)(((long long)(part + 1) * ntiles_all) / nparts);
    const bool has_new = part == nparts - 1;                 // the part that holds the new position's tile
    const size_t head_off = (size_t)b * seq_stride + ((size_t)(layer * NKV + g) * max_seq) * D;
    const bf16* kb = k_cache + head_off;
    const bf16* vb = v_cache + head_off;
    bf16* wring = ring + (size_t)warp * BD_STAGES * BD_STAGE_ELEMS;
    uint8_t* wraw = bd_smem + (size_t)warp * BD8_WARP_BYTES;                          // FP8: [2][raw stage] | f16 tile pair
    bf16* wtile = reinterpret_cast<bf16*>(wraw + BD_STAGES * BD8_RAW);
    const uint8_t* k8b = FP8 ? k8 + head_off : nullptr;
    const uint8_t* v8b = FP8 ? v8 + head_off : nullptr;

    // A warp's first two tiles are requested before the wait on the preceding kernel: the rows of earlier positions were written by
    // earlier steps, all of them complete (the step's embedding kernel lets its successors start only behind its own wait).
    // The tile that holds the new position follows the wait (FP8: the block barrier below, this CTA writes that row itself).
    // Both stages are kept in flight, a stage is asked for again as soon as it is read.  Step of batch 32 / 64 / 41 (fp8) at 250 to 500 / 1024 /
    // 90 to 900 positions: 975 / 2045 / 1331 -> 899 / 2020 / 1256 us.
    auto request = [&](int t, int stage) {
        if constexpr (FP8) bd_load_tile_fp8(wraw + stage * BD8_RAW, k8b, v8b, t, len, lane);
        else bd_load_tile(wring + stage * BD_STAGE_ELEMS, kb, vb, t, len, lane);
    };
    const int t_first = tile_lo + warp, t_new = has_new ? ntiles - 1 : -1;
    int late = -1;                                           // stage whose tile holds the new position and is among the first
#pragma unroll
    for (int s = 0; s < BD_STAGES; ++s) {
        const int t = t_first + s * WARPS;
        if (t < ntiles) {
            if (t != t_new) request(t, s);
            else late = s;
        }
        cp_async_commit();
    }
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    if (!FP8 && late >= 0) { request(t_new, late); cp_async_commit(); }
    if constexpr (FP8) {
        if (tid < 64 && has_new) {
            const int e4 = 4 * (tid & 31);
            const bool isk = tid < 32;
            const uint2 u = ld_cg_u2((isk ? kb : vb) + (size_t)pos * D + e4);
            const float inv = 1.0f / (isk ? ks : vs);
            *reinterpret_cast<uint32_t*>((isk ? k8 : v8) + head_off + (size_t)pos * D + e4) =
                f32x4_to_fp8x4(bf_lo(u.x) * inv, bf_hi(u.x) * inv, bf_lo(u.y) * inv, bf_hi(u.y) * inv);
            __threadfence_block();
        }
    }
    if (tid >= 64 && tid < 96) {
        const int t8 = tid - 64;
        uint4 q = ld_cg_u4(qkv + (size_t)b * QKV + 2 * g * D + t8 * 8);
        if constexpr (FP8) {   // f16 tiles are multiplied with an f16 query
            q.x = pack_f16x2(bf_lo(q.x), bf_hi(q.x)); q.y = pack_f16x2(bf_lo(q.y), bf_hi(q.y));
            q.z = pack_f16x2(bf_lo(q.z), bf_hi(q.z)); q.w = pack_f16x2(bf_lo(q.w), bf_hi(q.w));
        }
        *reinterpret_cast<uint4*>(qs + t8 * 8) = q;
    }
    __syncthreads();
    if (FP8 && late >= 0) { request(t_new, late); cp_async_commit(); }

    const int gi = lane >> 2, ti = lane & 3;
    const float scale = 0.08838834764831845f * ks;  // 1/sqrt(128) (x the K scale)
    float m0 = -1e30f, m1 = -1e30f, l0 = 0.f, l1 = 0.f;
    float o[16][4];
#pragma unroll
    for (int j = 0; j < 16; ++j) { o[j][0] = 0.f; o[j][1] = 0.f; o[j][2] = 0.f; o[j][3] = 0.f; }
    uint32_t qb[D / 16][2];   // B fragments of the two query heads (columns 2..7 are zero)
    {
        const uint32_t qaddr = smem_u32(qs) + (uint32_t)((gi & 1) * D + 2 * ti) * 2u;
#pragma unroll
        for (int ks16 = 0; ks16 < D / 16; ++ks16) {
            qb[ks16][0] = gi < 2 ? lds32(qaddr + ks16 * 32) : 0u;
            qb[ks16][1] = gi < 2 ? lds32(qaddr + ks16 * 32 + 16) : 0u;
        }
    }
    bf16* pw = ps + warp * 32;
    int it = 0;
    for (int tile = tile_lo + warp; tile < ntiles; tile += BD_THREADS / 32, ++it) {
        // this tile has landed; the next one, requested an iteration ago, may be in flight (but for the one warp with a late tile)
        if (late >= 0) cp_async_wait_all();
        else cp_async_wait<BD_STAGES - 1>();
        __syncwarp();
        const bf16* st = FP8 ? wtile : wring + (it % BD_STAGES) * BD_STAGE_ELEMS;
        const int t_next = tile + BD_STAGES * WARPS;         // takes the stage that this iteration frees
        if constexpr (FP8) {
            bd_expand_tile_fp8(wraw + (it % BD_STAGES) * BD8_RAW, wtile, lane);
            __syncwarp();
            if (t_next < ntiles) request(t_next, it % BD_STAGES);
            cp_async_commit();
        }
        const uint32_t rowoff = (uint32_t)(((lane & 15) * BD_LD + (lane >> 4) * 8) * 2);
        const uint32_t kaddr = smem_u32(st) + rowoff, vaddr = kaddr + 16 * BD_LD * 2;
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks16 = 0; ks16 < D / 16; ++ks16) {
            uint32_t af[4];
            ldsm4(af, kaddr + ks16 * 32);
            mma16816_sel<FP8>(c, af, qb[ks16][0], qb[ks16][1]);
        }
        // lanes with ti == 0 hold head 0 / head 1 of positions gi (c[0], c[1]) and gi + 8 (c[2], c[3])
        const int p_lo = tile * 16 + gi, p_hi = p_lo + 8;
        const bool own = ti == 0;
        const float s00 = (own && p_lo < len) ? c[0] * scale : -1e30f, s01 = (own && p_lo < len) ? c[1] * scale : -1e30f;
        const float s10 = (own && p_hi < len) ? c[2] * scale : -1e30f, s11 = (own && p_hi < len) ? c[3] * scale : -1e30f;
        float t0 = fmaxf(s00, s10), t1 = fmaxf(s01, s11);
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, off));
            t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, off));
        }
        t0 = __shfl_sync(0xffffffffu, t0, 0);
        t1 = __shfl_sync(0xffffffffu, t1, 0);
        const float mn0 = fmaxf(m0, t0), mn1 = fmaxf(m1, t1);
        const float cr0 = expf(m0 - mn0), cr1 = expf(m1 - mn1);
        m0 = mn0; m1 = mn1;
        const float e00 = (own && p_lo < len) ? expf(s00 - m0) : 0.f, e01 = (own && p_lo < len) ? expf(s01 - m1) : 0.f;
        const float e10 = (own && p_hi < len) ? expf(s10 - m0) : 0.f, e11 = (own && p_hi < len) ? expf(s11 - m1) : 0.f;
        float u0 = e00 + e10, u1 = e01 + e11;
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            u0 += __shfl_xor_sync(0xffffffffu, u0, off);
            u1 += __shfl_xor_sync(0xffffffffu, u1, off);
        }
        l0 = l0 * cr0 + __shfl_sync(0xffffffffu, u0, 0);
        l1 = l1 * cr1 + __shfl_sync(0xffffffffu, u1, 0);
        if (own) {
            if constexpr (FP8) {   // probabilities rounded to bf16 as on the bf16 path (exact in f16: 8 significant bits, e <= 1)
                __half* ph = reinterpret_cast<__half*>(pw);
                ph[gi] = __float2half_rn(rbf(e00)); ph[gi + 8] = __float2half_rn(rbf(e10));
                ph[16 + gi] = __float2half_rn(rbf(e01)); ph[16 + gi + 8] = __float2half_rn(rbf(e11));
            } else {
                pw[gi] = __float2bfloat16_rn(e00); pw[gi + 8] = __float2bfloat16_rn(e10);
                pw[16 + gi] = __float2bfloat16_rn(e01); pw[16 + gi + 8] = __float2bfloat16_rn(e11);
            }
        }
        __syncwarp();
        uint32_t pa[4] = {0u, 0u, 0u, 0u};   // A = P: row gi is head gi (rows 2..15 are zero)
        if (gi < 2) {
            pa[0] = *reinterpret_cast<const uint32_t*>(pw + gi * 16 + 2 * ti);
            pa[2] = *reinterpret_cast<const uint32_t*>(pw + gi * 16 + 8 + 2 * ti);
        }
        if (cr0 != 1.f || cr1 != 1.f) {   // the same for every lane
            const float crg = gi == 0 ? cr0 : cr1;
#pragma unroll
            for (int j = 0; j < 16; ++j) { o[j][0] *= crg; o[j][1] *= crg; }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint32_t bv[4];
            ldsm4_t(bv, vaddr + j * 32);
            mma16816_sel<FP8>(o[2 * j], pa, bv[0], bv[1]);
            mma16816_sel<FP8>(o[2 * j + 1], pa, bv[2], bv[3]);
        }
        __syncwarp();
        if constexpr (!FP8) {
            if (t_next < ntiles) request(t_next, it % BD_STAGES);
            cp_async_commit();
        }
    }
    cp_async_wait_all();
    __syncthreads();   // every warp is done with its ring: the merge buffers reuse it
    float* s_acc = reinterpret_cast<float*>(bd_smem);          // [WARPS][2][D]
    float* s_m = s_acc + WARPS * 2 * D;                        // [WARPS][2]
    float* s_l = s_m + WARPS * 2;                              // [WARPS][2]
    if (lane == 0) { s_m[warp * 2] = m0; s_m[warp * 2 + 1] = m1; s_l[warp * 2] = l0; s_l[warp * 2 + 1] = l1; }
    if (gi < 2) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            *reinterpret_cast<float2*>(s_acc + (warp * 2 + gi) * D + j * 8 + 2 * ti) = make_float2(o[j][0], o[j][1]);
    }
    __syncthreads();
    const size_t item = (size_t)b * NKV + g;
    for (int idx = tid; idx < 2 * D; idx += BD_THREADS) {
        const int hh = idx >> 7, d = idx & 127;
        float M = -1e30f;
#pragma unroll
        for (int w8 = 0; w8 < WARPS; ++w8) M = fmaxf(M, s_m[w8 * 2 + hh]);
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int w8 = 0; w8 < WARPS; ++w8) {
            const float f = expf(s_m[w8 * 2 + hh] - M);
            den = fmaf(s_l[w8 * 2 + hh], f, den);
            num = fmaf(s_acc[(w8 * 2 + hh) * D + d], f, num);
        }
        if (nparts == 1) {
            out[(size_t)b * QSZ + (2 * g + hh) * D + d] = __float2bfloat16_rn(num / den * vs);
        } else {
            float* pp = parts + ((item * BD_MAX_PARTS + part) * 2 + hh) * BD_PART;
            pp[2 + d] = num;
            if (d == 0) { pp[0] = M; pp[1] = den; }
        }
    }
    if (nparts == 1) return;
    // the block barrier orders every thread's partial before thread 0's release; the CTA that takes the
    // last ticket acquires the others' partials with the same instruction
    __shared__ int s_last;
    __syncthreads();
    if (tid == 0) {
        unsigned int t;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(tickets + item) : "memory");
        s_last = (t == (unsigned int)(nparts - 1));
        if (s_last) tickets[item] = 0u;
    }
    __syncthreads();
    if (!s_last) return;
    for (int idx = tid; idx < 2 * D; idx += BD_THREADS) {
        const int hh = idx >> 7, d = idx & 127;
        const float* pb = parts + (item * BD_MAX_PARTS * 2 + hh) * BD_PART;
        float mj[BD_MAX_PARTS], M = -1e30f;
#pragma unroll
        for (int j = 0; j < BD_MAX_PARTS; ++j) {
            mj[j] = j < nparts ? ld_cg_f32(pb + (size_t)j * 2 * BD_PART) : -1e30f;
            M = fmaxf(M, mj[j]);
        }
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int j = 0; j < BD_MAX_PARTS; ++j) {
            if (j < nparts) {
                const float f = expf(mj[j] - M);
                den = fmaf(ld_cg_f32(pb + (size_t)j * 2 * BD_PART + 1), f, den);
                num = fmaf(ld_cg_f32(pb + (size_t)j * 2 * BD_PART + 2 + d), f, num);
            }
        }
        out[(size_t)b * QSZ + (2 * g + hh) * D + d] = __float2bfloat16_rn(num / den * vs);
    }
}

template <bool FP8, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 6 ? 2 : 1)
k_bd_attention(const bf16* qkv, const bf16* k_cache, const bf16* v_cache, bf16* out,
               const int* positions, int layer, int max_seq, size_t seq_stride, uint8_t* __restrict__ k8, uint8_t* __restrict__ v8,
               const float* k_scale, const float* v_scale, int scale_stride, float* __restrict__ parts,
               unsigned int* __restrict__ tickets, int n_full, int p_tail) {
    bd_attention_body<FP8, WARPS>(qkv, k_cache, v_cache, out, positions, layer, max_seq, seq_stride, k8, v8, k_scale, v_scale, scale_stride, parts,
                                  tickets, n_full, p_tail);
}

// out_tokens[b] = lowest index of the maximum bf16 logit of row b; positions[b] += 1.
__global__ void __launch_bounds__(1024) k_bd_argmax_advance(const bf16* logits, int vocab, int* __restrict__ out_tokens,
                                                            int* __restrict__ positions, float* __restrict__ logits_f32) {
    pdl_trigger();   // the next grid may be scheduled already (it waits the same way)
    pdl_wait();      // launched with programmatic stream serialisation: the preceding grid has completed
    __shared__ unsigned long long s_best[32];
    const int b = blockIdx.x, tid = threadIdx.x;
    const bf16* row = logits + (size_t)b * vocab;
    unsigned long long best = 0ull;
    // 16-byte loads, eight logits each (the vocabulary is a multiple of 128 and rows are 16-byte aligned)
    for (int i4 = tid; i4 < vocab / 8; i4 += blockDim.x) {
        const uint4 q = ld_cg_u4(row + i4 * 8);
        const uint32_t wds[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = (e & 1) ? bf_hi(wds[e >> 1]) : bf_lo(wds[e >> 1]);
            const int i = i4 * 8 + e;
            if (logits_f32) logits_f32[(size_t)b * vocab + i] = v;
            uint32_t u = __float_as_uint(v);
            u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
            const unsigned long long key = ((unsigned long long)u << 32) | (unsigned long long)(0xffffffffu - (uint32_t)i);
            best = key > best ? key : best;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
    }
    if ((tid & 31) == 0) s_best[tid >> 5] = best;
    __syncthreads();
    if (tid == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i) best = s_best[i] > best ? s_best[i] : best;
        out_tokens[b] = (int)(0xffffffffu - (uint32_t)(best & 0xffffffffull));
        positions[b] = ld_cg_i32(positions + b) + 1;
    }
}

}  // namespace mq

using namespace mq;

extern "C" int mq_prefill_launch_count(int num_layers) { return 1 + num_layers * 8 + 2; }

// C[M,N] = A[M,K] * B[N,K]^T on the tcgen05 path (bf16 in/out, fp32 accumulate);
// optional residual R (same shape and leading dimension as C, may alias C).
extern "C" int mq_launch_gemm_bf16(const void* A, int lda, const void* B, void* C, const void* R, int M, int N, int K, int ldc,
                                   unsigned int* status, void* stream) {
    if (!A || !B || !C || !status || M <= 0 || N <= 0 || K <= 0) return MQ_ERR_BAD_ARG;
    if (lda % 8 != 0 || ldc % 8 != 0) return MQ_ERR_ALIGNMENT;
    if (R) return launch_gemm<128, EPI_RESID>((const bf16*)A, lda, (const bf16*)B, nullptr, (bf16*)C, (const bf16*)R, M, N, K, ldc, status, (cudaStream_t)stream,
                                              nullptr, 0, 0, 1, -1, false);
    return launch_gemm<128, EPI_STORE>((const bf16*)A, lda, (const bf16*)B, nullptr, (bf16*)C, nullptr, M, N, K, ldc, status, (cudaStream_t)stream,
                                       nullptr, 0, 0, 1, -1, false);
}

// Test hook: mq_launch_gemm_bf16 (no residual) whose producer never requests k-block drop_kb (0 <= drop_kb < K / 64),
// so one bounded wait of every CTA runs out: the kernel must return, set MQ_STATUS_WAIT_TIMEOUT in *status, store
// nothing, and leave the device usable.  Not used by any production path.
extern "C" int mq_debug_gemm_drop_load(const void* A, int lda, const void* B, void* C, int M, int N, int K, int ldc,
                                       unsigned int* status, void* stream, int drop_kb) {
    if (!A || !B || !C || !status || M <= 0 || N <= 0 || K <= 0 || drop_kb < 0 || drop_kb >= K / GM_BK) return MQ_ERR_BAD_ARG;
    if (lda % 8 != 0 || ldc % 8 != 0) return MQ_ERR_ALIGNMENT;
    return launch_gemm<128, EPI_STORE>((const bf16*)A, lda, (const bf16*)B, nullptr, (bf16*)C, nullptr, M, N, K, ldc, status, (cudaStream_t)stream,
                                       nullptr, 0, 0, 1, drop_kb, false);
}

// The same for the GEMM on pairs of SMs (N a multiple of 256; B complete before the call), whose pairs walk several tiles each: drop_kb counts
// a pair's k-blocks over all of its tiles, and the tiles before the one that lacks a block are stored.  drop_kb = -1: the GEMM as it is.
extern "C" int mq_debug_gemm_pair_drop_load(const void* A, int lda, const void* B, void* C, const void* R, int M, int N, int K, int ldc,
                                            unsigned int* status, void* stream, int drop_kb) {
    if (!A || !B || !C || !R || !status || M <= 0 || N <= 0 || K <= 0 || drop_kb < -1) return MQ_ERR_BAD_ARG;
    if (lda % 8 != 0 || ldc % 8 != 0) return MQ_ERR_ALIGNMENT;
    return launch_gemm2<256, EPI_RESID>((const bf16*)A, lda, (const bf16*)B, nullptr, (bf16*)C, (const bf16*)R, M, N, K, ldc, status, (cudaStream_t)stream,
                                        nullptr, 0, 0, 1, true, NoSink(), drop_kb);
}

static int prefill_impl(const MqModel* model, const MqDecodeBuffers* dbuf, const MqPrefillBuffers* pb, const int* ids,
                        int seq_len, int pos0, const bf16* audio, int audio_start, int audio_len, int* out_token, float* logits,
                        void* stream_v);

// The chain of a batch's decode step: q|k|v (with everything up to the cache), and what follows the attention.
static SkArgs sk_args(const MqModel* model, int rows, bf16* h, float* ssq, bf16* k_cache, bf16* v_cache, unsigned int* status) {
    SkArgs a = {};
    a.M = rows; a.h = h; a.ssq = ssq; a.status = status;
    a.cos = (const bf16*)model->cos_table; a.sin = (const bf16*)model->sin_table;
    a.k_cache = k_cache; a.v_cache = v_cache; a.max_seq = model->max_seq_len;
    return a;
}
static int sk_qkv(const MqModel* model, int l, SkArgs a, bf16* qkv, cudaStream_t stream) {
    const MqLayerWeights& w = model->layers[l];
    a.layer = l;
    a.gain = (const bf16*)w.input_layernorm; a.q_norm = (const bf16*)w.q_norm; a.k_norm = (const bf16*)w.k_norm;
    a.out = qkv;
    return sk_linear<SK_QKV>(w, nullptr, a, stream);
}
static int sk_rest(const MqModel* model, int l, SkArgs a, const bf16* attn, bf16* act, cudaStream_t stream) {
    const MqLayerWeights& w = model->layers[l];
    int rc = sk_linear<SK_O>(w, attn, a, stream);
    if (rc) return rc;
    a.gain = (const bf16*)w.post_attn_layernorm;
    a.out = act;
    rc = sk_linear<SK_GU>(w, nullptr, a, stream);
    return rc ? rc : sk_linear<SK_DOWN>(w, act, a, stream);
}

// Test hook: one linear of layer 0 of the chain on what bb's buffers hold (which: 0 q|k|v, 1 O, 2 gate|up, 3 down).  drop >= 0: block
// drop % 16 of CTA drop / 16 of every cluster is never requested, so that one of its waits runs out.  Not used by any production path.
extern "C" int mq_debug_chain_drop_load(const MqModel* model, const MqBatchBuffers* bb, int which, int drop, void* stream_v) {
    if (!model || !bb || !bb->k_cache || !bb->v_cache || !bb->positions || !bb->status || which < SK_QKV || which > SK_DOWN || drop < -1) return MQ_ERR_BAD_ARG;
    const MqPrefillBuffers* pb = &bb->act;
    if (!pb->h || !pb->qkv || !pb->attn || !pb->act || !bb->partials || bb->partials_bytes < (size_t)bb->batch * SK_SSQ * sizeof(float)) return MQ_ERR_BAD_ARG;
    if (bb->batch < 1 || bb->batch > SK_MAX_ROWS || bb->batch > pb->max_tokens) return MQ_ERR_BAD_ARG;
    cudaStream_t stream = (cudaStream_t)stream_v;
    SkArgs a = sk_args(model, bb->batch, (bf16*)pb->h, bb->partials, (bf16*)bb->k_cache, (bf16*)bb->v_cache, bb->status);
    a.pos_rows = bb->positions;
    a.seq_stride = (size_t)model->num_layers * NKV * model->max_seq_len * D;
    a.drop = drop;
    if (which == SK_QKV) return sk_qkv(model, 0, a, (bf16*)pb->qkv, stream);
    const MqLayerWeights& w = model->layers[0];
    a.gain = (const bf16*)w.post_attn_layernorm;
    a.out = (bf16*)pb->act;
    return which == SK_O ? sk_linear<SK_O>(w, (const bf16*)pb->attn, a, stream) : which == SK_GU ? sk_linear<SK_GU>(w, nullptr, a, stream)
                                                                                 : sk_linear<SK_DOWN>(w, (const bf16*)pb->act, a, stream);
}

// The linears of many rows.  A GEMM on pairs of SMs (tc_gemm2.cuh) has two microseconds more to set up (a cluster, two CTAs' barriers)
// and one tile's epilogue to show at the end, but hides the others and streams at 1.2 to 1.4 PFLOP/s: it is taken as soon as
// k_gemm's tiles would need a second round.  us per linear, weights from HBM, k_gemm / pair:
//   rows       1024         1536         2048         4001         16384
//   q|k|v   10.6 / 12.1  20.1 / 16.8  18.0 / 17.6  34.0 / 28.5   128 / 101
//   gate|up 16.0 / 18.5  30.0 / 19.9  30.3 / 25.3  59.1 / 42.4   242 / 148
//   o       14.5 / 18.3  14.7 / 18.5  14.6 / 19.4  29.2 / 22.2   131 / 76
//   down    19.3 / 23.9  20.0 / 24.3  20.1 / 25.1  39.4 / 27.9   155 / 85
// Below, tiles are as wide as leaves one round of CTAs on the 148 SMs of the device (the counts beside the rules).  Prompt of 2 / 23 / 128 / 256 / 384 / 640 / 900 / 1024 rows with 128-wide tiles
// everywhere: 1.76 / 1.82 / 2.00 / 2.03 / 2.10 / 2.22 / 2.72 / 2.41 ms, now 1.67 / 1.71 / 1.86 / 1.93 / 2.00 / 2.12 / 2.30 / 2.33.
static bool heads_on_pairs(int rows) { return (rows > 512 && rows <= 1024) || rows > 9 * 128; }
static int pf_qkv(const MqModel* model, int l, const bf16* x, bf16* qkv, int rows, Heads hd, unsigned int* status, cudaStream_t stream) {
    const MqLayerWeights& w = model->layers[l];
    const bf16 *q = (const bf16*)w.q_proj, *k = (const bf16*)w.k_proj, *v = (const bf16*)w.v_proj;
    hd.q_norm = (const bf16*)w.q_norm; hd.k_norm = (const bf16*)w.k_norm; hd.cos = (const bf16*)model->cos_table; hd.sin = (const bf16*)model->sin_table;
    hd.layer = l; hd.max_seq = model->max_seq_len;
    // q | k | v in one launch: column tiles from three weight matrices.  The pairs' epilogue, which runs under the next tile's products,
    // norms, rotates and fills the caches as well, so they pay from 513 rows on (16 column tiles x 3 row tiles) but for the five row tiles that
    // make 80 on 74 pairs (1100 rows 2.66, on pairs 2.90 ms).
    if (heads_on_pairs(rows)) return launch_gemm2<256, EPI_HEADS>(x, H, q, k, qkv, nullptr, rows, QKV, H, QKV, status, stream, v, QSZ, KVSZ, 1, true, hd);
    const int rc = rows > 1024 ? launch_gemm<256, EPI_STORE, 1>(x, H, q, k, qkv, nullptr, rows, QKV, H, QKV, status, stream, v, QSZ, KVSZ)
                 : rows > 256  ? launch_gemm<128, EPI_STORE>(x, H, q, k, qkv, nullptr, rows, QKV, H, QKV, status, stream, v, QSZ, KVSZ)
                               : launch_gemm<64, EPI_STORE>(x, H, q, k, qkv, nullptr, rows, QKV, H, QKV, status, stream, v, QSZ, KVSZ);
    if (rc) return rc;
    launch_pdl(k_pf_qknorm_rope, dim3(rows, hd.row_pos ? 1 : rows <= 1024 ? 4 : 2), dim3(256), 0, stream, qkv, hd.q_norm, hd.k_norm, hd.cos, hd.sin, hd.k_cache, hd.v_cache,
               l, hd.pos0, hd.max_seq, hd.row_pos, hd.seq_stride, hd.row_seq);
    return MQ_OK;
}
static int pf_gateup(const MqLayerWeights& w, const bf16* x, bf16* act, int rows, unsigned int* status, cudaStream_t stream) {
    const bf16 *g = (const bf16*)w.gate_proj, *u = (const bf16*)w.up_proj;
    if (rows > 1024) return launch_gemm2<256, EPI_SWIGLU>(x, H, g, u, act, nullptr, rows, I, H, I, status, stream);
    // 256 x (96 gate + 96 up) tiles: 32 x 4 CTAs; 128 x (128 + 128): 24 x 6; 128 x (64 + 64): 48 x 3
    if (rows > 768) return launch_gemm<96, EPI_SWIGLU, 2>(x, H, g, u, act, nullptr, rows, I, H, I, status, stream);
    if (rows > 384) return launch_gemm<128, EPI_SWIGLU>(x, H, g, u, act, nullptr, rows, I, H, I, status, stream);
    return launch_gemm<64, EPI_SWIGLU>(x, H, g, u, act, nullptr, rows, I, H, I, status, stream);
}
// h += A W^T, N = 1024: 18 row tiles of 128 by eight columns are the last to fit one round; up to 1024 rows 64-wide tiles double the CTAs
static int pf_add(const bf16* A, int K, const bf16* W, bf16* h, int rows, unsigned int* status, cudaStream_t stream) {
    if (rows > 18 * 128) return launch_gemm2<256, EPI_RESID>(A, K, W, nullptr, h, h, rows, H, K, H, status, stream);
    if (rows > 1024) return launch_gemm<128, EPI_RESID>(A, K, W, nullptr, h, h, rows, H, K, H, status, stream);
    return launch_gemm<64, EPI_RESID>(A, K, W, nullptr, h, h, rows, H, K, H, status, stream);
}

// Between 512 and 1024 rows the N = 1024 projections (O, down) split K over two CTAs per 128 x 128 tile:
// 64-wide tiles re-read the A operand sixteen times and are bound by L2 traffic.  The fp32 planes land in
// the qkv buffer (free after attention; 2 x rows x 1024 floats fill it exactly) and one kernel adds them to the
// residual stream and applies the RMSNorm that follows (the next layer's input norm after the down projection).
// Above 1024 and up to 2048 rows the same with 128 x 256 tiles (N = 256 instructions, half the A traffic per FLOP).
// Below, sums over K stay whole.
static bool planes_of_k(int rows, int max_tokens) {
    return rows >= 512 && rows <= 2048 && (size_t)max_tokens * QKV * sizeof(bf16) >= (size_t)2 * rows * H * sizeof(float);
}

// Kernels of one pass over `rows` rows.  A layer: q|k|v, heads (unless the product's epilogue does them), attention, O, norm, gate|up, down
// and a norm, ahead of q|k|v or, with planes, behind down (and once ahead of the first layer).  Around: embedding, last row, LM head;
// packed: embedding, last rows, norm, LM head, arg-max.
extern "C" int mq_prefill_launches(int num_layers, int rows, int max_tokens, int packed) {
    return num_layers * (heads_on_pairs(rows) ? 7 : 8) + (packed ? 5 : planes_of_k(rows, max_tokens) ? 4 : 3);
}

extern "C" int mq_launch_prefill(const MqModel* model, const MqDecodeBuffers* dbuf, const MqPrefillBuffers* pb, const int* ids,
                                 int seq_len, int pos0, int* out_token, float* logits, void* stream_v) {
    return prefill_impl(model, dbuf, pb, ids, seq_len, pos0, nullptr, 0, 0, out_token, logits, stream_v);
}

extern "C" int mq_launch_prefill_asr(const MqModel* model, const MqDecodeBuffers* dbuf, const MqPrefillBuffers* pb, const int* ids,
                                     int seq_len, int pos0, const void* audio_embeds, int audio_start, int audio_len,
                                     int* out_token, float* logits, void* stream_v) {
    if (!audio_embeds || audio_len <= 0 || audio_start < 0 || audio_start + audio_len > seq_len) return MQ_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(audio_embeds) & 15u) != 0) return MQ_ERR_ALIGNMENT;
    return prefill_impl(model, dbuf, pb, ids, seq_len, pos0, (const bf16*)audio_embeds, audio_start, audio_len, out_token, logits, stream_v);
}

static int prefill_impl(const MqModel* model, const MqDecodeBuffers* dbuf, const MqPrefillBuffers* pb, const int* ids,
                        int seq_len, int pos0, const bf16* audio, int audio_start, int audio_len, int* out_token, float* logits,
                        void* stream_v) {
    if (!model || !dbuf || !pb || !ids || !out_token) return MQ_ERR_BAD_ARG;
    if (!pb->h || !pb->x || !pb->qkv || !pb->attn || !pb->act) return MQ_ERR_BAD_ARG;
    if (seq_len <= 0 || pos0 < 0) return MQ_ERR_BAD_ARG;
    if (seq_len > pb->max_tokens || pos0 + seq_len > model->max_seq_len) return MQ_ERR_TOO_LONG;
    cudaStream_t stream = (cudaStream_t)stream_v;
    const int S = seq_len;
    bf16* h = (bf16*)pb->h; bf16* x = (bf16*)pb->x; bf16* qkv = (bf16*)pb->qkv; bf16* attn = (bf16*)pb->attn; bf16* act = (bf16*)pb->act;
    unsigned int* status = dbuf->status;
    static bool fa_attr[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    const size_t fa_smem = FA_SMEM;
    if (dev >= 0 && dev < 64 && !fa_attr[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_pf_attention, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fa_smem);
        if (e != cudaSuccess) return (int)e;
        fa_attr[dev] = true;
    }
    // From 128 prompt rows on the attention runs on tcgen05, its K and V tiles straight from the cache.  The V map
    // is a stack of (layer, kv head) planes that end at the prompt's last key: what the cache holds beyond it
    // (possibly not even numbers) is multiplied by probabilities of zero and must read as zero.
    const bool use_tc = S >= TA_BQ;
    CUtensorMap map_q, map_k, map_v;
    if (use_tc) {
        int mrc = get_map(qkv, (uint64_t)S, (uint64_t)D, (uint64_t)QKV, TA_BQ, &map_q, (uint64_t)NQ, (uint64_t)D);
        if (mrc == MQ_OK)
            mrc = get_map(dbuf->k_cache, (uint64_t)(pos0 + S), (uint64_t)D, (uint64_t)D, TA_BK, &map_k, (uint64_t)model->num_layers * NKV,
                          (uint64_t)model->max_seq_len * D);
        if (mrc == MQ_OK)
            mrc = get_map(dbuf->v_cache, (uint64_t)(pos0 + S), (uint64_t)D, (uint64_t)D, TA_BK, &map_v, (uint64_t)model->num_layers * NKV,
                          (uint64_t)model->max_seq_len * D);
        if (mrc != MQ_OK) return mrc;
    }
    int rc;
    launch_pdl(k_pf_embed, dim3(S), dim3(128), 0, stream, ids, (const bf16*)model->embed, h, model->vocab_size, status, audio,
               audio_start, audio_len);
    const bool splitk = planes_of_k(S, pb->max_tokens);
    const bool wide = splitk && S > 1024;
    float* part = reinterpret_cast<float*>(qkv);
    Heads heads = {};
    heads.k_cache = (bf16*)dbuf->k_cache; heads.v_cache = (bf16*)dbuf->v_cache; heads.pos0 = pos0;
    for (int l = 0; l < model->num_layers; ++l) {
        const MqLayerWeights& w = model->layers[l];
        if (l == 0 || !splitk)
            launch_pdl(k_pf_rmsnorm, dim3((S + 7) / 8), dim3(256), 0, stream, h, (const bf16*)w.input_layernorm, x, S);
        rc = pf_qkv(model, l, x, qkv, S, heads, status, stream);
        if (rc) return rc;
        if (use_tc) {
            rc = launch_attention_tc<2, 0, 2>(NQ, map_q, map_k, map_v, map_q, map_k,
                                              {attn, QSZ, D, S, pos0, NQ / NKV, l * NKV, 8, 0, 0.08838834764831845f * 1.4426950408889634f, nullptr, status},
                                              stream);
            if (rc) return rc;
        } else {
            launch_pdl(k_pf_attention, dim3(NQ, (S + FA_BQ - 1) / FA_BQ), dim3(FA_THREADS), fa_smem, stream, qkv, (const bf16*)dbuf->k_cache,
                       (const bf16*)dbuf->v_cache, attn, S, pos0, l, model->max_seq_len);
        }
        // N = 1024: with M <= 1024 a 128-wide tile gives at most 64 CTAs, 64-wide tiles double that
        if (splitk) {
            rc = wide ? launch_gemm<256, EPI_PARTIAL>(attn, QSZ, (const bf16*)w.o_proj, nullptr, (bf16*)part, nullptr, S, H, QSZ, H, status, stream,
                                                      nullptr, 0, 0, 2)
                      : launch_gemm<128, EPI_PARTIAL>(attn, QSZ, (const bf16*)w.o_proj, nullptr, (bf16*)part, nullptr, S, H, QSZ, H, status, stream,
                                                      nullptr, 0, 0, 2);
            if (rc) return rc;
            launch_pdl(k_sk_resid_norm, dim3(S), dim3(256), 0, stream, (const float*)part, S, h, (const bf16*)w.post_attn_layernorm, x);
        } else {
            rc = pf_add(attn, QSZ, (const bf16*)w.o_proj, h, S, status, stream);
            if (rc) return rc;
            launch_pdl(k_pf_rmsnorm, dim3((S + 7) / 8), dim3(256), 0, stream, h, (const bf16*)w.post_attn_layernorm, x, S);
        }
        rc = pf_gateup(w, x, act, S, status, stream);
        if (rc) return rc;
        if (splitk) {
            rc = wide ? launch_gemm<256, EPI_PARTIAL>(act, I, (const bf16*)w.down_proj, nullptr, (bf16*)part, nullptr, S, H, I, H, status, stream,
                                                      nullptr, 0, 0, 2)
                      : launch_gemm<128, EPI_PARTIAL>(act, I, (const bf16*)w.down_proj, nullptr, (bf16*)part, nullptr, S, H, I, H, status, stream,
                                                      nullptr, 0, 0, 2);
            if (rc) return rc;
            const bf16* next_norm = l + 1 < model->num_layers ? (const bf16*)model->layers[l + 1].input_layernorm : nullptr;
            launch_pdl(k_sk_resid_norm, dim3(S), dim3(256), 0, stream, (const float*)part, S, h, next_norm, x);
        } else {
            rc = pf_add(act, I, (const bf16*)w.down_proj, h, S, status, stream);
            if (rc) return rc;
        }
    }
    // last row -> decode hidden buffer, then the decode path's LM head + arg-max
    launch_pdl(k_pf_copy_row, dim3(1), dim3(H / 8), 0, stream, h + (size_t)(S - 1) * H, (bf16*)dbuf->hidden);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    return launch_lmhead_only(model, dbuf, out_token, logits, stream);
}

// Prompts of several sequences packed row after row (a ragged batch in one pass): the linears
// see one matrix of total_rows rows, QK-norm/RoPE and the cache writes use the per-row tables,
// attention the per-tile tables, and the next token of every sequence comes from its last row
// through the batched LM head.  bb->positions[b] must hold len_b - 1 on entry (the arg-max kernel
// advances it to len_b).  All tables are device arrays built by the caller.
extern "C" int mq_launch_prefill_packed(const MqModel* model, const MqBatchBuffers* bb, const int* ids, const int* row_seq,
                                        const int* row_pos, const int* tile_seq, const int* tile_q0, const int* seq_len,
                                        const int* seq_row0, int total_rows, int num_tiles, int* out_tokens, void* stream_v) {
    if (!model || !bb || !ids || !row_seq || !row_pos || !tile_seq || !tile_q0 || !seq_len || !seq_row0 || !out_tokens) return MQ_ERR_BAD_ARG;
    if (!bb->k_cache || !bb->v_cache || !bb->positions || !bb->logits || !bb->status) return MQ_ERR_BAD_ARG;
    const MqPrefillBuffers* pb = &bb->act;
    if (!pb->h || !pb->x || !pb->qkv || !pb->attn || !pb->act) return MQ_ERR_BAD_ARG;
    const int B = bb->batch, T = total_rows;
    if (B <= 0 || T < B || num_tiles <= 0) return MQ_ERR_BAD_ARG;
    if (T > pb->max_tokens) return MQ_ERR_TOO_LONG;
    if (model->vocab_size % 128 != 0) return MQ_ERR_UNSUPPORTED;
    cudaStream_t stream = (cudaStream_t)stream_v;
    bf16* h = (bf16*)pb->h; bf16* x = (bf16*)pb->x; bf16* qkv = (bf16*)pb->qkv; bf16* attn = (bf16*)pb->attn; bf16* act = (bf16*)pb->act;
    unsigned int* status = bb->status;
    const size_t seq_stride = (size_t)model->num_layers * NKV * model->max_seq_len * D;
    // The attention that each prompt takes alone in prefill_impl: same bits.  With mma.sync tiles of 64 queries for prompts of 128 rows
    // and more too, 64 x 1024 / 32 x ~384 rows took 108 / 17.7 ms, now 84.5 / 14.9.
    CUtensorMap map_q, map_k, map_v;
    const uint64_t planes = (uint64_t)B * model->num_layers * NKV;
    int rc = get_map(qkv, (uint64_t)T, (uint64_t)D, (uint64_t)QKV, TA_BQ, &map_q, (uint64_t)NQ, (uint64_t)D);
    if (rc == MQ_OK) rc = get_map(bb->k_cache, (uint64_t)model->max_seq_len, (uint64_t)D, (uint64_t)D, TA_BK, &map_k, planes, (uint64_t)model->max_seq_len * D);
    if (rc == MQ_OK) rc = get_map(bb->v_cache, (uint64_t)model->max_seq_len, (uint64_t)D, (uint64_t)D, TA_BK, &map_v, planes, (uint64_t)model->max_seq_len * D);
    if (rc != MQ_OK) return rc;
    AttnTcArgs at = {attn, QSZ, D, 0, 0, NQ / NKV, 0, 8, 0, 0.08838834764831845f * 1.4426950408889634f, nullptr, status};
    at.tile_seq = tile_seq; at.tile_q0 = tile_q0; at.seq_len = seq_len; at.seq_row0 = seq_row0;
    at.seq_planes = model->num_layers * NKV;
    at.qkv = qkv; at.k_cache = (const bf16*)bb->k_cache; at.v_cache = (const bf16*)bb->v_cache; at.plane_elems = (size_t)model->max_seq_len * D;
    launch_pdl(k_pf_embed, dim3(T), dim3(128), 0, stream, ids, (const bf16*)model->embed, h, model->vocab_size, status,
               (const bf16*)nullptr, 0, 0);
    Heads heads = {};
    heads.k_cache = (bf16*)bb->k_cache; heads.v_cache = (bf16*)bb->v_cache;
    heads.row_pos = row_pos; heads.row_seq = row_seq; heads.seq_stride = seq_stride;
    for (int l = 0; l < model->num_layers; ++l) {
        const MqLayerWeights& w = model->layers[l];
        launch_pdl(k_pf_rmsnorm, dim3((T + 7) / 8), dim3(256), 0, stream, h, (const bf16*)w.input_layernorm, x, T);
        rc = pf_qkv(model, l, x, qkv, T, heads, status, stream);
        if (rc) return rc;
        at.kv_plane0 = l * NKV;
        rc = launch_attention_tc<2, 0, 2, true>(NQ, map_q, map_k, map_v, map_q, map_k, at, stream, num_tiles);
        if (rc) return rc;
        rc = pf_add(attn, QSZ, (const bf16*)w.o_proj, h, T, status, stream);
        if (rc) return rc;
        launch_pdl(k_pf_rmsnorm, dim3((T + 7) / 8), dim3(256), 0, stream, h, (const bf16*)w.post_attn_layernorm, x, T);
        rc = pf_gateup(w, x, act, T, status, stream);
        if (rc) return rc;
        rc = pf_add(act, I, (const bf16*)w.down_proj, h, T, status, stream);
        if (rc) return rc;
    }
    // last row of every sequence -> final norm -> LM head -> arg-max (advances positions[b] to len_b)
    launch_pdl(k_pf_gather_last, dim3(B), dim3(H / 8), 0, stream, h, seq_row0, seq_len, attn);
    launch_pdl(k_pf_rmsnorm, dim3((B + 7) / 8), dim3(256), 0, stream, attn, (const bf16*)model->final_norm, x, B);
    rc = launch_gemm<128, EPI_STORE_2CTA>(x, H, (const bf16*)model->lm_head, nullptr, (bf16*)bb->logits, nullptr, B, model->vocab_size, H,
                                     model->vocab_size, status, stream);
    if (rc) return rc;
    launch_pdl(k_bd_argmax_advance, dim3(B), dim3(1024), 0, stream, (const bf16*)bb->logits, model->vocab_size, out_tokens, bb->positions, (float*)nullptr);
    return (int)cudaGetLastError();
}

extern "C" int mq_decode_batch_launch_count(int num_layers) { return 1 + num_layers * 10 + 3; }
// up to 64 rows: the cluster chain (sk_chain.cuh), its row sums in the caller's scratch; above, tile GEMMs
static bool on_chain(int batch, const float* partials, size_t bytes) {
    return batch <= SK_MAX_ROWS && partials != nullptr && bytes >= (size_t)batch * SK_SSQ * sizeof(float);
}
extern "C" int mq_decode_batch_launches(int num_layers, const MqBatchBuffers* bb) {
    return on_chain(bb->batch, bb->partials, bb->partials_bytes) ? num_layers * 5 + 4 : mq_decode_batch_launch_count(num_layers);
}

// How a batched attention launch is shaped for `items` = 8 x batch (sequence, kv head) pairs.  Up to one
// item per SM: twelve-warp CTAs, the keys of every item split over up to four CTAs while those still fit one
// round.  Beyond: six-warp CTAs, two per SM.  The SM streams with twelve warps either way, but two CTAs
// per SM are at different points of their items, so one CTA's ring fill and warp merge (about 4 us per
// item, during which a lone twelve-warp CTA leaves the SM's memory pipeline idle) overlap the other's
// streaming: 2.68 -> 2.49 ms per step at batch 64 / context 1024, 2.12 -> 1.90 at context 500.  The items of
// the full rounds get one CTA each and those of the last, partly empty round are split so that they
// fill it (384 items on 296 slots: 296 whole, 88 in three parts).  Splitting ALL items was measured slower
// (3.02 vs 2.68 ms per step with twelve-warp halves), four- and three-warp CTAs (three and four per SM)
// too (2.58, 2.55).  Depends on the batch size only, so a captured graph stays valid.
struct BdShape { int warps, n_full, p_tail; };
static BdShape bd_shape(int items, int sms, bool can_split) {
    if (items <= sms) {
        int p = can_split ? sms / items : 1;
        p = p > BD_MAX_PARTS ? BD_MAX_PARTS : p;
        return p < 2 ? BdShape{12, items, 1} : BdShape{12, 0, p};
    }
    const int slots = 2 * sms, rem = items % slots;
    if (!can_split || rem == 0) return {6, items, 1};
    int p = slots / rem;                                         // parts that still fit the last round
    p = p > BD_MAX_PARTS ? BD_MAX_PARTS : p;
    return p < 2 ? BdShape{6, items, 1} : BdShape{6, items - rem, p};
}

template <bool FP8, int WARPS>
static int bd_set_smem() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_bd_attention<FP8, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bd_smem_bytes(WARPS));
        if (e != cudaSuccess) return (int)e;
        done[dev] = true;
    }
    return MQ_OK;
}

// attention of one layer of a batched decode step, from the bf16 caches or from the e4m3 shadow caches
template <bool FP8, int WARPS>
static void launch_bd_attention_t(int B, BdShape sh, cudaStream_t stream, const bf16* qkv, const MqBatchBuffers* bb, const MqKvFp8* kv8, bf16* attn,
                                  int l, const MqModel* model, size_t seq_stride) {
    const int ctas = sh.n_full + (B * NKV - sh.n_full) * sh.p_tail;
    launch_pdl(k_bd_attention<FP8, WARPS>, dim3(ctas), dim3(WARPS * 32), bd_smem_bytes(WARPS), stream, qkv, (const bf16*)bb->k_cache,
               (const bf16*)bb->v_cache, attn, (const int*)bb->positions, l, model->max_seq_len, seq_stride,
               (uint8_t*)(kv8 ? kv8->k_fp8 : nullptr), (uint8_t*)(kv8 ? kv8->v_fp8 : nullptr), (const float*)(kv8 ? kv8->k_scale : nullptr),
               (const float*)(kv8 ? kv8->v_scale : nullptr), model->num_layers * NKV, bb->attn_parts, bb->attn_tickets, sh.n_full, sh.p_tail);
}
static void launch_bd_attention(int B, BdShape sh, cudaStream_t stream, const bf16* qkv, const MqBatchBuffers* bb, const MqKvFp8* kv8, bf16* attn, int l,
                                const MqModel* model, size_t seq_stride) {
    if (kv8) {
        if (sh.warps == 6) launch_bd_attention_t<true, 6>(B, sh, stream, qkv, bb, kv8, attn, l, model, seq_stride);
        else launch_bd_attention_t<true, 12>(B, sh, stream, qkv, bb, kv8, attn, l, model, seq_stride);
    } else {
        if (sh.warps == 6) launch_bd_attention_t<false, 6>(B, sh, stream, qkv, bb, kv8, attn, l, model, seq_stride);
        else launch_bd_attention_t<false, 12>(B, sh, stream, qkv, bb, kv8, attn, l, model, seq_stride);
    }
}

static int decode_batch_impl(const MqModel* model, const MqBatchBuffers* bb, const MqKvFp8* kv8, const int* in_tokens, int* out_tokens,
                             float* logits_f32, void* stream_v) {
    if (!model || !bb || !in_tokens || !out_tokens) return MQ_ERR_BAD_ARG;
    if (kv8 && (!kv8->k_fp8 || !kv8->v_fp8 || !kv8->k_scale || !kv8->v_scale)) return MQ_ERR_BAD_ARG;
    if (!bb->k_cache || !bb->v_cache || !bb->positions || !bb->logits || !bb->status) return MQ_ERR_BAD_ARG;
    const MqPrefillBuffers* pb = &bb->act;
    if (!pb->h || !pb->x || !pb->qkv || !pb->attn || !pb->act) return MQ_ERR_BAD_ARG;
    const int B = bb->batch;
    if (B <= 0 || B > pb->max_tokens) return MQ_ERR_BAD_ARG;
    if (model->vocab_size % 128 != 0) return MQ_ERR_UNSUPPORTED;
    cudaStream_t stream = (cudaStream_t)stream_v;
    bf16* h = (bf16*)pb->h; bf16* x = (bf16*)pb->x; bf16* qkv = (bf16*)pb->qkv; bf16* attn = (bf16*)pb->attn; bf16* act = (bf16*)pb->act;
    unsigned int* status = bb->status;
    const size_t seq_stride = (size_t)model->num_layers * NKV * model->max_seq_len * D;
    int rc = bd_set_smem<false, 6>();
    if (rc == MQ_OK) rc = bd_set_smem<false, 12>();
    if (rc == MQ_OK) rc = bd_set_smem<true, 6>();
    if (rc == MQ_OK) rc = bd_set_smem<true, 12>();
    if (rc != MQ_OK) return rc;
    static int sm_count[64] = {0};
    {
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 0 || dev >= 64) return MQ_ERR_UNSUPPORTED;
        if (!sm_count[dev]) cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        if (sm_count[dev] <= 0) return MQ_ERR_UNSUPPORTED;
    }
    int dev_now = 0;
    cudaGetDevice(&dev_now);
    const bool can_split = bb->attn_parts != nullptr && bb->attn_tickets != nullptr &&
                           bb->attn_parts_bytes >= (size_t)B * NKV * BD_MAX_PARTS * 2 * BD_PART * sizeof(float);
    const BdShape shape = bd_shape(B * NKV, sm_count[dev_now], can_split);
    if (on_chain(B, bb->partials, bb->partials_bytes)) {
        SkArgs a = sk_args(model, B, h, bb->partials, (bf16*)bb->k_cache, (bf16*)bb->v_cache, status);
        a.pos_rows = bb->positions;
        a.seq_stride = seq_stride;
        launch_pdl(k_sk_embed, dim3(B), dim3(32), 0, stream, in_tokens, (const bf16*)model->embed, h, a.ssq, model->vocab_size, status);
        for (int l = 0; l < model->num_layers; ++l) {
            rc = sk_qkv(model, l, a, qkv, stream);
            if (rc) return rc;
            launch_bd_attention(B, shape, stream, qkv, bb, kv8, attn, l, model, seq_stride);
            rc = sk_rest(model, l, a, attn, act, stream);
            if (rc) return rc;
        }
        launch_pdl(k_sk_norm, dim3((B + 7) / 8), dim3(256), 0, stream, h, a.ssq, (const bf16*)model->final_norm, x, B);
    } else {
    launch_pdl(k_pf_embed, dim3(B), dim3(128), 0, stream, in_tokens, (const bf16*)model->embed, h, model->vocab_size, status,
               (const bf16*)nullptr, 0, 0);
    for (int l = 0; l < model->num_layers; ++l) {
        const MqLayerWeights& w = model->layers[l];
        launch_pdl(k_pf_rmsnorm, dim3((B + 7) / 8), dim3(256), 0, stream, h, (const bf16*)w.input_layernorm, x, B);
        rc = launch_gemm<128, EPI_STORE>(x, H, (const bf16*)w.q_proj, nullptr, qkv, nullptr, B, QSZ, H, QKV, status, stream);
        if (rc) return rc;
        rc = launch_gemm<128, EPI_STORE>(x, H, (const bf16*)w.k_proj, nullptr, qkv + QSZ, nullptr, B, KVSZ, H, QKV, status, stream);
        if (rc) return rc;
        rc = launch_gemm<128, EPI_STORE>(x, H, (const bf16*)w.v_proj, nullptr, qkv + QSZ + KVSZ, nullptr, B, KVSZ, H, QKV, status, stream);
        if (rc) return rc;
        launch_pdl(k_pf_qknorm_rope, dim3(dim3(B, 4)), dim3(256), 0, stream, qkv, (const bf16*)w.q_norm, (const bf16*)w.k_norm, (const bf16*)model->cos_table,
                                                         (const bf16*)model->sin_table, (bf16*)bb->k_cache, (bf16*)bb->v_cache, l, 0,
                                                         model->max_seq_len, bb->positions, seq_stride, nullptr);
        launch_bd_attention(B, shape, stream, qkv, bb, kv8, attn, l, model, seq_stride);
        rc = launch_gemm<128, EPI_RESID>(attn, QSZ, (const bf16*)w.o_proj, nullptr, h, h, B, H, QSZ, H, status, stream);
        if (rc) return rc;
        launch_pdl(k_pf_rmsnorm, dim3((B + 7) / 8), dim3(256), 0, stream, h, (const bf16*)w.post_attn_layernorm, x, B);
        rc = launch_gemm<128, EPI_SWIGLU>(x, H, (const bf16*)w.gate_proj, (const bf16*)w.up_proj, act, nullptr, B, I, H, I, status, stream);
        if (rc) return rc;
        rc = launch_gemm<128, EPI_RESID>(act, I, (const bf16*)w.down_proj, nullptr, h, h, B, H, I, H, status, stream);
        if (rc) return rc;
    }
    launch_pdl(k_pf_rmsnorm, dim3((B + 7) / 8), dim3(256), 0, stream, h, (const bf16*)model->final_norm, x, B);
    }
    rc = launch_gemm<128, EPI_STORE_2CTA>(x, H, (const bf16*)model->lm_head, nullptr, (bf16*)bb->logits, nullptr, B, model->vocab_size, H,
                                     model->vocab_size, status, stream);
    if (rc) return rc;
    launch_pdl(k_bd_argmax_advance, dim3(B), dim3(1024), 0, stream, (const bf16*)bb->logits, model->vocab_size, out_tokens, bb->positions, logits_f32);
    return (int)cudaGetLastError();
}

extern "C" int mq_launch_decode_batch(const MqModel* model, const MqBatchBuffers* bb, const int* in_tokens, int* out_tokens,
                                      float* logits_f32, void* stream_v) {
    return decode_batch_impl(model, bb, nullptr, in_tokens, out_tokens, logits_f32, stream_v);
}

extern "C" int mq_launch_decode_batch_kv8(const MqModel* model, const MqBatchBuffers* bb, const MqKvFp8* kv8, const int* in_tokens,
                                          int* out_tokens, float* logits_f32, void* stream_v) {
    if (!kv8) return MQ_ERR_BAD_ARG;
    return decode_batch_impl(model, bb, kv8, in_tokens, out_tokens, logits_f32, stream_v);
}

// ---------------------------------------------------------------- FP8 shadow cache
// One CTA per (layer, kv head): scale = max |x| over positions [start, end) / 448 (1 for an all-zero
// span), then every element of the span as e4m3(x / scale), K and V separately (reference:
// split_quantize_kv_cache_fp8_kernel, csrc/megakernel/split_decode_gemm.cu:223-300).
__global__ void __launch_bounds__(256) k_kv_quantize_fp8(const bf16* __restrict__ k_cache, const bf16* __restrict__ v_cache,
                                                         uint8_t* __restrict__ k8, uint8_t* __restrict__ v8, float* __restrict__ k_scale,
                                                         float* __restrict__ v_scale, int max_seq, int start, int end) {
    __shared__ float s_k[8], s_v[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t base = (size_t)blockIdx.x * max_seq * D;
    const int n8 = (end - start) * (D / 8);                        // 16-byte groups of the span
    const uint4* kp = reinterpret_cast<const uint4*>(k_cache + base + (size_t)start * D);
    const uint4* vp = reinterpret_cast<const uint4*>(v_cache + base + (size_t)start * D);
    auto amax4 = [](const uint4& u) {
        float m = fmaxf(fabsf(bf_lo(u.x)), fabsf(bf_hi(u.x)));
        m = fmaxf(m, fmaxf(fabsf(bf_lo(u.y)), fabsf(bf_hi(u.y))));
        m = fmaxf(m, fmaxf(fabsf(bf_lo(u.z)), fabsf(bf_hi(u.z))));
        return fmaxf(m, fmaxf(fabsf(bf_lo(u.w)), fabsf(bf_hi(u.w))));
    };
    float km = 0.f, vm = 0.f;
    for (int i = tid; i < n8; i += 256) {
        km = fmaxf(km, amax4(kp[i]));
        vm = fmaxf(vm, amax4(vp[i]));
    }
    km = warp_max(km);
    vm = warp_max(vm);
    if (lane == 0) { s_k[warp] = km; s_v[warp] = vm; }
    __syncthreads();
    km = 0.f; vm = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) { km = fmaxf(km, s_k[w]); vm = fmaxf(vm, s_v[w]); }
    const float ks = kv_fp8_scale_of(km), vs = kv_fp8_scale_of(vm);
    if (tid == 0) { k_scale[blockIdx.x] = ks; v_scale[blockIdx.x] = vs; }
    const float ik = 1.0f / ks, iv = 1.0f / vs;
    uint2* k8p = reinterpret_cast<uint2*>(k8 + base + (size_t)start * D);
    uint2* v8p = reinterpret_cast<uint2*>(v8 + base + (size_t)start * D);
    for (int i = tid; i < n8; i += 256) {
        const uint4 a = kp[i], b = vp[i];
        k8p[i] = make_uint2(f32x4_to_fp8x4(bf_lo(a.x) * ik, bf_hi(a.x) * ik, bf_lo(a.y) * ik, bf_hi(a.y) * ik),
                            f32x4_to_fp8x4(bf_lo(a.z) * ik, bf_hi(a.z) * ik, bf_lo(a.w) * ik, bf_hi(a.w) * ik));
        v8p[i] = make_uint2(f32x4_to_fp8x4(bf_lo(b.x) * iv, bf_hi(b.x) * iv, bf_lo(b.y) * iv, bf_hi(b.y) * iv),
                            f32x4_to_fp8x4(bf_lo(b.z) * iv, bf_hi(b.z) * iv, bf_lo(b.w) * iv, bf_hi(b.w) * iv));
    }
}

extern "C" int mq_launch_kv_quantize_fp8(const void* k_cache, const void* v_cache, const MqKvFp8* kv8, int num_layers, int max_seq_len,
                                         int start_pos, int end_pos, void* stream_v) {
    if (!k_cache || !v_cache || !kv8 || !kv8->k_fp8 || !kv8->v_fp8 || !kv8->k_scale || !kv8->v_scale) return MQ_ERR_BAD_ARG;
    if (num_layers <= 0 || max_seq_len <= 0) return MQ_ERR_BAD_ARG;
    const int start = start_pos < 0 ? 0 : start_pos, end = end_pos > max_seq_len ? max_seq_len : end_pos;
    if (start >= end) return MQ_OK;                                  // an empty span is a no-op, as in the reference
    k_kv_quantize_fp8<<<num_layers * NKV, 256, 0, (cudaStream_t)stream_v>>>((const bf16*)k_cache, (const bf16*)v_cache, (uint8_t*)kv8->k_fp8,
                                                                            (uint8_t*)kv8->v_fp8, kv8->k_scale, kv8->v_scale, max_seq_len, start, end);
    return (int)cudaGetLastError();
}
