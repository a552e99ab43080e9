// True 32-bit matrix product for the float32 path on the FMA units: C[n, m] = sum_k A[n, k] * W[m, k], no tensor cores, no
// TF32.  It takes the matrices that do not go to gemm_f32_tc5.cu (ops.f32_split_supports: fewer than 64 rows, a short K, rows off
// 16-byte boundaries), whatever the number of rows of A.
// Every output element is one float accumulator fed by fused multiply-adds in ascending k, so its value depends on neither
// the number of rows in the call nor on the tile it falls into: the 32-bit path gives the same logits however the tokens
// are cut into steps.
//
// Bound by the FMA pipes for prompts (some 74 TFLOP/s: 148 SMs x 128 lanes; 50 reached on 509 x 16384 x 2048 with aligned rows, which
// go to the tensor cores now, 45 with K 2,050), by memory and the latency of a stage for a handful of rows.  A thread owns
// TM x TN outputs and works on pairs of neighbouring columns (fma.rn.f32x2: one issue slot, two results, each rounded as
// the single one is), so that half of the issue slots are left for the reads of shared memory that feed them.  The operands
// lie k by k in shared memory, two stages of BK; the next stage is in registers while the current one is worked through.
#include "common.cuh"

__device__ __forceinline__ uint64_t gf_pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void gf_unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ void gf_fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(d) : "l"(a), "l"(b));
}

// BM tokens x BN output columns a block, TM x TN a thread: its columns are TN / 4 groups of four, BN / (TN / 4) apart, its
// rows likewise, so that a warp's 16-byte reads of a stage lie side by side.  VEC: rows of A and W start on
// 16-byte boundaries and K is a multiple of 4.
template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 512 / ((BM / TM) * (BN / TN)))
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int N, int M, int K, int ldc) {
    constexpr int BK = 16, TX = BN / TN, TY = BM / TM, THREADS = TX * TY, PAD = 4;
    constexpr int QA = BM * BK / 4, QW = BN * BK / 4;                                  // quads of a stage
    constexpr int LA = (QA + THREADS - 1) / THREADS, LW = (QW + THREADS - 1) / THREADS;
    constexpr int CG = TN / 4, RG = TM / 4;                                        // groups of columns and of rows
    static_assert(TN % 4 == 0 && TM % 4 == 0 && TX % 8 == 0 && TY % 4 == 0, "groups of four, warps of 4 x 8 threads");
    __shared__ __align__(16) float As[2][BK][BM + PAD];
    __shared__ __align__(16) float Ws[2][BK][BN + PAD];
    // a warp is 4 x 8 threads: its reads of either operand are one pass of shared memory
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx = warp % (TX / 8) * 8 + (lane & 7), ty = warp / (TX / 8) * 4 + (lane >> 3);
    const int n0 = blockIdx.y * BM, m0 = blockIdx.x * BN;
    float4 ra[LA], rw[LW];
    auto quad = [&](const float* __restrict__ src, int row, int rows, int k) {
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row < rows) {
            const float* p = src + (size_t)row * K + k;
            if (VEC) {
                if (k < K) x = *reinterpret_cast<const float4*>(p);
            } else {
                if (k < K) x.x = p[0];
                if (k + 1 < K) x.y = p[1];
                if (k + 2 < K) x.z = p[2];
                if (k + 3 < K) x.w = p[3];
            }
        }
        return x;
    };
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; i++) {
            const int e = threadIdx.x + i * THREADS;
            if (QA % THREADS == 0 || e < QA) ra[i] = quad(A, n0 + e / (BK / 4), N, k0 + e % (BK / 4) * 4);
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            const int e = threadIdx.x + i * THREADS;
            if (QW % THREADS == 0 || e < QW) rw[i] = quad(W, m0 + e / (BK / 4), M, k0 + e % (BK / 4) * 4);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < LA; i++) {
            const int e = threadIdx.x + i * THREADS, r = e / (BK / 4), k = e % (BK / 4) * 4;
            if (QA % THREADS == 0 || e < QA) {
                As[buf][k][r] = ra[i].x; As[buf][k + 1][r] = ra[i].y; As[buf][k + 2][r] = ra[i].z; As[buf][k + 3][r] = ra[i].w;
            }
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            const int e = threadIdx.x + i * THREADS, r = e / (BK / 4), k = e % (BK / 4) * 4;
            if (QW % THREADS == 0 || e < QW) {
                Ws[buf][k][r] = rw[i].x; Ws[buf][k + 1][r] = rw[i].y; Ws[buf][k + 2][r] = rw[i].z; Ws[buf][k + 3][r] = rw[i].w;
            }
        }
    };
    uint64_t acc[TM][TN / 2];
    const uint64_t zero2 = gf_pack2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = zero2;
    load(0);
    store(0);
    __syncthreads();
    for (int k0 = 0, buf = 0; k0 < K; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < K;
        if (more) load(k0 + BK);
        // values beyond K are zeros in both operands: they add a product of zeros, which changes no sum but the sign of an
        // exact -0, so the last, partial stage stops at K
        const int depth = min(BK, K - k0);
        auto work = [&](int kk) {
            float a[TM];
            uint64_t w2[TN / 2];
#pragma unroll
            for (int g = 0; g < RG; g++) {
                const float4 x = *reinterpret_cast<const float4*>(&As[buf][kk][g * (BM / RG) + ty * 4]);
                a[g * 4] = x.x; a[g * 4 + 1] = x.y; a[g * 4 + 2] = x.z; a[g * 4 + 3] = x.w;
            }
#pragma unroll
            for (int g = 0; g < CG; g++) {
                const float4 x = *reinterpret_cast<const float4*>(&Ws[buf][kk][g * (BN / CG) + tx * 4]);
                w2[g * 2] = gf_pack2(x.x, x.y);
                w2[g * 2 + 1] = gf_pack2(x.z, x.w);
            }
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const uint64_t a2 = gf_pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; j++) gf_fma2(acc[i][j], a2, w2[j]);
            }
        };
        if (depth == BK) {
#pragma unroll
            for (int kk = 0; kk < BK; kk++) work(kk);
        } else {
            for (int kk = 0; kk < depth; kk++) work(kk);
        }
        if (more) store(buf ^ 1);
        __syncthreads();
    }
    const bool vec = (ldc & 3) == 0 && ((uintptr_t)C & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int n = n0 + i / 4 * (BM / RG) + ty * 4 + i % 4;
        if (n >= N) continue;
#pragma unroll
        for (int g = 0; g < CG; g++) {
            const int m = m0 + g * (BN / CG) + tx * 4;
            float x[4];
            gf_unpack2(acc[i][g * 2], x[0], x[1]);
            gf_unpack2(acc[i][g * 2 + 1], x[2], x[3]);
            float* p = C + (size_t)n * ldc + m;
            if (vec && m + 3 < M) {
                *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (m + j < M) p[j] = x[j];
            }
        }
    }
}

// rows of C are ldc floats apart
MB_API int mb_gemm_f32(const float* A, const float* W, float* C, int N, int M, int K, int ldc, cudaStream_t st) {
    if (N == 0 || M == 0) return 0;
    if (ldc < M) return -2;
    const bool vec = K % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    auto padded = [&](int bm) { return ((long long)N + bm - 1) / bm * bm; };
    auto tiles = [&](int bm, int bn) { return padded(bm) / bm * ((M + bn - 1) / bn); };
    // The largest tile that still gives every SM its four blocks, since it reads the operands least (64 rows of the first cost
    // what 56 of the second do), unless its padding costs more than that; measured at sizes that come here (us, 128 x 64 / 64 x 64 /
    // 32 x 64 / 16 x 64): a short K: 2,048 x 2,048 x 128 29 / 28 / 34 / 45, 2,048 x 8,192 x 192 131 / 149 / 185 / 252, 509 x 1,024 x 192
    // 16 / 9.6 / 11 / 11, 64 x 2,048 x 128 11 / 6.9 / 6.7 / 4.8; few rows of W: 509 x 48 x 8,192 552 / 287 / 280 / 177; K no multiple of 4,
    // in single loads: 509 x 16,384 x 2,050 755 / 985 / 1437 / 1884, 509 x 2,048 x 2,050 145 / 149 / 191 / 244, 160 x 32,000 x 2,050 731 /
    // 759 / 927 / 1342, 64 rows 408 / 295 / 331 / 543, 33 rows 399 / 277 / 335 / 522, 17 rows 394 / 264 / 180 / 235, one 391 / 253 / 171 /
    // 138.  (It costs up to 15 % where the first tile has nearly enough blocks: 128 x 32,000 x 2,050 444 / 509 / 742 / 1077.)
    const int t = N <= 16                                                        ? 3
                  : tiles(128, 64) >= 592 && 7 * padded(128) <= 8 * padded(64) ? 0
                  : N > 32 && tiles(64, 64) >= 148                             ? 1
                  : N <= 32 && tiles(32, 64) >= 148                            ? 2
                                                                               : 3;
    const int rows[4] = {128, 64, 32, 16};
    if (padded(rows[t]) / rows[t] > 65535) return -2;
#define GF_CASE(ID, BM, BN, TM, TN)                                                                                        \
    if (t == ID) {                                                                                                         \
        const dim3 grid((M + BN - 1) / BN, (N + BM - 1) / BM);                                                             \
        if (vec) gemm_f32_kernel<BM, BN, TM, TN, true><<<grid, (BM / TM) * (BN / TN), 0, st>>>(A, W, C, N, M, K, ldc);     \
        else gemm_f32_kernel<BM, BN, TM, TN, false><<<grid, (BM / TM) * (BN / TN), 0, st>>>(A, W, C, N, M, K, ldc);        \
        MB_LAUNCH_CHECK();                                                                                                 \
        return 0;                                                                                                          \
    }
    GF_CASE(0, 128, 64, 8, 8) GF_CASE(1, 64, 64, 8, 4) GF_CASE(2, 32, 64, 4, 8) GF_CASE(3, 16, 64, 4, 4)
#undef GF_CASE
    return -2;
}
