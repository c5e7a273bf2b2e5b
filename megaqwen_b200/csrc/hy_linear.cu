// Matrix products of the layer-listed decoder for more than one token: bf16 on the tcgen05
// tile GEMM (tc_gemm.cuh), 32-bit on plain FMA tiles (no reduced-precision tensor mode).
#include "hy_common.cuh"
#include "tc_gemm2.cuh"

namespace mq {
namespace hy {

int sm_count() {
    static int n[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
    return n[dev];
}

// ---------------------------------------------------------------- 32-bit
// Every output is one chain of FMAs over k, first to last, whatever the tile: K is split neither over CTAs nor over warps nor over
// even and odd k.  (The 32-bit mode is what other implementations are compared with, and where a head's output nearly cancels
// before its norm the order of a sum is what one sees: split sums took the logits of some prompts 7e-5 from where they were.)
// Bound by the FMA pipes from some hundred rows on (128 a clock and SM) and below by the weights' bytes that few CTAs have in flight.
// A CTA of four warps, two by two, makes 8 TI x 16 TJ outputs; a thread TI x TJ of them at a distance of 4 rows and 8 columns, so that
// a warp's 16-byte loads of four k take one wavefront each: TI + TJ loads for 4 TI TJ FMAs.  Steps of FK k by cp.async into a ring
// as deep as the tile is small, one block barrier each; the finished tile goes through shared memory so that the sink sees 32
// columns of a row.  Prompt of 150 rows, 28 layers of width 1024: 27.9 -> 11.5 ms (64 x 64 tiles of one 16-step buffer before).
constexpr int F_THREADS = 128;
template <int TI_, int TJ_, int FK_, int STAGES_>
struct F32Tile {
    static constexpr int TI = TI_, TJ = TJ_, FK = FK_, STAGES = STAGES_;
    static constexpr int M = 8 * TI, N = 16 * TJ, LD = FK + 4, STAGE = (M + N) * LD, CLD = N + 4, PASS = F_THREADS / (FK / 4);   // rows copied side by side
    static constexpr size_t SMEM = (size_t)STAGES * STAGE * 4;
    static_assert(N % 32 == 0 && N % PASS == 0 && M % PASS == 0 && FK % 16 == 0 && M * (N / 32) <= F_THREADS && M * CLD <= STAGES * STAGE,
                  "a thread takes 32 columns of a row; the finished tile takes the place of the ring");
};
template <class Tile, bool PLANES>
__global__ void __launch_bounds__(F_THREADS) k_gemm_f32(const float* __restrict__ A, int lda, const float* __restrict__ W, int M, int N, int K,
                                                        SegmentSink<float> sink, float* __restrict__ plane, int ldp) {
    constexpr int TI = Tile::TI, TJ = Tile::TJ, FK = Tile::FK, STAGES = Tile::STAGES, LD = Tile::LD;
    extern __shared__ __align__(16) float f32_ring[];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * Tile::M, n0 = blockIdx.x * Tile::N;
    const int row = (warp & 1) * 4 * TI + (lane >> 3), col = (warp >> 1) * 8 * TJ + (lane & 7);       // of this thread's first output
    const int steps = (K + FK - 1) / FK;        // K is a multiple of 16: the last step may be part of one
    const int lr = tid / (FK / 4), lk = tid % (FK / 4) * 4;
    auto load_w = [&](int s) {
        float* dst = f32_ring + (s % STAGES) * Tile::STAGE + (Tile::M + lr) * LD + lk;
        const int k = s * FK + lk;
#pragma unroll
        for (int i = 0; i < Tile::N; i += Tile::PASS) {
            const bool ok = k < K && n0 + lr + i < N;
            cp_async16_zfill(dst + i * LD, ok ? W + (size_t)(n0 + lr + i) * K + k : W, ok);
        }
    };
    auto load_a = [&](int s) {
        float* dst = f32_ring + (s % STAGES) * Tile::STAGE + lr * LD + lk;
        const int k = s * FK + lk;
#pragma unroll
        for (int i = 0; i < Tile::M; i += Tile::PASS) {
            const bool ok = k < K && m0 + lr + i < M;
            cp_async16_zfill(dst + i * LD, ok ? A + (size_t)(m0 + lr + i) * lda + k : A, ok);
        }
    };
    // the weights do not hang on the kernel before this one
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < steps) load_w(s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load_a(s);
        cp_async_commit();
    }
    float acc[TI][TJ] = {};
    for (int s = 0; s < steps; ++s) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                        // step s has landed, for everybody, and the stage of step s - 1 has been read
        if (s + STAGES - 1 < steps) { load_w(s + STAGES - 1); load_a(s + STAGES - 1); }
        cp_async_commit();
        const float* sa = f32_ring + (s % STAGES) * Tile::STAGE + row * LD;
        const float* sb = f32_ring + (s % STAGES) * Tile::STAGE + (Tile::M + col) * LD;
#pragma unroll
        for (int k0 = 0; k0 < FK; k0 += 16) {
            if (k0 > 0 && s * FK + k0 >= K) break;
#pragma unroll
            for (int k = k0; k < k0 + 16; k += 4) {
                float4 av[TI], bv[TJ];
#pragma unroll
                for (int i = 0; i < TI; ++i) av[i] = load4(sa + 4 * i * LD + k);
#pragma unroll
                for (int j = 0; j < TJ; ++j) bv[j] = load4(sb + 8 * j * LD + k);
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int i = 0; i < TI; ++i)
#pragma unroll
                        for (int j = 0; j < TJ; ++j) acc[i][j] = fmaf((&av[i].x)[e], (&bv[j].x)[e], acc[i][j]);
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) f32_ring[(row + 4 * i) * Tile::CLD + col + 8 * j] = acc[i][j];
    __syncthreads();
    constexpr int PIECES = Tile::N / 32;
    if (tid < Tile::M * PIECES) {
        const int r = tid / PIECES, c = tid % PIECES * 32;
        if (m0 + r >= M || n0 + c >= N) return;
        const float* p = f32_ring + r * Tile::CLD + c;
        if (PLANES) {                            // the plane is at least as wide as the tiles
            float* out = plane + (size_t)(m0 + r) * ldp + n0 + c;
#pragma unroll
            for (int q = 0; q < 8; ++q) store4(out + 4 * q, load4(p + 4 * q));
        } else {
            uint32_t u[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) u[j] = __float_as_uint(p[j]);
            sink(m0 + r, n0 + c, u);
        }
    }
}

// ---------------------------------------------------------------- tile shape
// Estimated cycles of one CTA round: a k-block costs the larger of its tensor time (256 cycles per 128 x 128) and its
// operand traffic (64 bytes per clock into an SM); a tile costs its start-up and epilogue on top.  Pairs of SMs (mt = 0, 256 x 256
// tiles) are persistent: start-up and one epilogue are paid once, and 10 000 cycles is what those of a one-round product
// were measured above its k-blocks (q|k|v of 1024 x 1024 rows by 4096: 12.1 us, one SM 10.6).
struct TileShape { int bn, mt; };
static long long tile_cost(TileShape s, int M, int N, int kblocks, int split, int sms) {
    if (s.mt == 0) {
        const long long tiles = (long long)((N + 255) / 256) * ((M + 255) / 256) * split;
        return ((tiles + sms / 2 - 1) / (sms / 2)) * ((kblocks + split - 1) / split) * 512 + 10000;
    }
    const long long tiles = (long long)((N + s.bn - 1) / s.bn) * ((M + 128 * s.mt - 1) / (128 * s.mt)) * split;
    const long long mma = 2LL * s.bn * s.mt, load = (16384LL * s.mt + 128LL * s.bn) / 64;
    const long long per_tile = ((kblocks + split - 1) / split) * (mma > load ? mma : load) + 3000 + 6LL * s.bn * s.mt;
    return ((tiles + sms - 1) / sms) * per_tile;
}
static TileShape pick_tile(int M, int N, int kblocks, int max_split, int* split) {
    static const TileShape shapes[] = {{256, 2}, {128, 2}, {256, 1}, {128, 1}, {64, 1}, {256, 0}};
    TileShape best = shapes[3];
    const int sms = sm_count();
    long long cost = -1;
    for (const TileShape& s : shapes)
        for (int z = 1; z <= max_split && z * 4 <= kblocks + 3; z *= 2) {
            // every plane is written and read back once: 8 bytes per element over the memory of the whole device
            const long long c = tile_cost(s, M, N, kblocks, z, sms) + (long long)(z - 1) * ((long long)M * N / 500 + 1500);
            if (cost < 0 || c < cost) { cost = c; best = s; *split = z; }
        }
    return best;
}

template <class Tile, bool PLANES>
static int go_f32(Stream& st, const float* A, int lda, const float* W, int M, int N, int K, const SegmentSink<float>& sink, float* plane, int ldp) {
    const int rc = allow_smem(k_gemm_f32<Tile, PLANES>, Tile::SMEM);
    if (rc) return rc;
    return launch(st, k_gemm_f32<Tile, PLANES>, dim3((N + Tile::N - 1) / Tile::N, (M + Tile::M - 1) / Tile::M), dim3(F_THREADS), Tile::SMEM, A, lda, W, M, N, K,
                  sink, plane, ldp);
}
template <bool PLANES>
static int gemm_f32(Stream& st, const float* A, int lda, const float* W, int M, int N, int K, const SegmentSink<float>& sink, float* plane, int ldp) {
    // The narrower a tile, the more CTAs stream the weights of a product with N = 1024, and the deeper the rings; the wider, the more often
    // a load serves.  Prompt of 8 / 64 / 100 / 150 / 300 rows, 28 layers of width 1024, with the first of these everywhere: 4.0 / 8.8 / 13.8 / 19.5 / 36.0 ms,
    // the second: 4.9 / 7.6 / 10.0 / 15.3 / 24.8, the third: 6.3 / 9.2 / 10.2 / 11.5 / 19.6; 4 x 4 outputs a thread: 8.1 / 11.2 / 13.3 / 15.3 / 21.6.
    if (M <= 8) return go_f32<F32Tile<1, 2, 64, 8>, PLANES>(st, A, lda, W, M, N, K, sink, plane, ldp);
    if (M <= 96) return go_f32<F32Tile<2, 2, 64, 6>, PLANES>(st, A, lda, W, M, N, K, sink, plane, ldp);
    return go_f32<F32Tile<4, 2, 32, 6>, PLANES>(st, A, lda, W, M, N, K, sink, plane, ldp);
}
template <>
int linear_segments<float>(Stream& st, const float* A, int lda, const float* W, int M, int N, int K, const Segments& g, unsigned int*) {
    return gemm_f32<false>(st, A, lda, W, M, N, K, SegmentSink<float>{g}, nullptr, 0);
}
template <>
int linear_planes<float>(Stream& st, const float* A, int lda, const float* W, float* planes, int M, int N, int K, int ldp, int* nplanes, unsigned int*) {
    *nplanes = 1;
    return gemm_f32<true>(st, A, lda, W, M, N, K, SegmentSink<float>{}, planes, ldp);
}

template <>
int linear_segments<bf16>(Stream& st, const bf16* A, int lda, const bf16* W, int M, int N, int K, const Segments& g, unsigned int* status) {
    int z = 1;
    const TileShape s = pick_tile(M, N, (K + 63) / 64, 1, &z);
    const SegmentSink<bf16> sink{g};
    ++st.launches;
#define MQH_GO(BN, MT) \
    if (s.bn == BN && s.mt == MT) \
        return launch_gemm<BN, EPI_SINK, MT>(A, lda, W, nullptr, nullptr, nullptr, M, N, K, 0, status, st.s, nullptr, 0, 0, 1, -1, true, sink);
    if (s.mt == 0) return launch_gemm2<256, EPI_SINK>(A, lda, W, nullptr, nullptr, nullptr, M, N, K, 0, status, st.s, nullptr, 0, 0, 1, true, sink);
    MQH_GO(256, 2) MQH_GO(128, 2) MQH_GO(256, 1) MQH_GO(128, 1) MQH_GO(64, 1)
#undef MQH_GO
    return MQ_ERR_UNSUPPORTED;
}
template <>
int linear_planes<bf16>(Stream& st, const bf16* A, int lda, const bf16* W, float* planes, int M, int N, int K, int ldp, int* nplanes, unsigned int* status) {
    int z = 1;
    const TileShape s = pick_tile(M, N, (K + 63) / 64, *nplanes, &z);
    *nplanes = z;
    ++st.launches;
#define MQH_GO(BN, MT) \
    if (s.bn == BN && s.mt == MT) \
        return launch_gemm<BN, EPI_PARTIAL, MT>(A, lda, W, nullptr, (bf16*)planes, nullptr, M, N, K, ldp, status, st.s, nullptr, 0, 0, z);
    if (s.mt == 0) return launch_gemm2<256, EPI_PARTIAL>(A, lda, W, nullptr, (bf16*)planes, nullptr, M, N, K, ldp, status, st.s, nullptr, 0, 0, z);
    MQH_GO(256, 2) MQH_GO(128, 2) MQH_GO(256, 1) MQH_GO(128, 1) MQH_GO(64, 1)
#undef MQH_GO
    return MQ_ERR_UNSUPPORTED;
}

}  // namespace hy
}  // namespace mq
