// The routed experts' products of steps of 128 tokens and more (bf16), on the 5th-generation tensor cores with the WEIGHTS on
// the M side of the instructions and an expert's tokens, whatever their number, on the N side.
//
// The rows of act are sorted by expert, an expert's rows starting at a multiple of 128 (moe.cu: moe_sort_gather).  groups[t]
// says of the tile of rows 128 t: -1, nothing starts here; else the low 12 bits are the expert, the 12 bits above them how
// many rows from 128 t on are its own, 1 to 256, and the bit above those whether the tile is an odd one of its expert.
//
// Bound by what the blocks bring in from the L2 and, behind it, by the weights, which a step reads once: 2,000 tokens of 6 of
// 64 experts are some 190 rows an expert, so a tile of 256 rows of W x all the rows of an expert reads 256 + 192 rows of
// each k where two tiles of 128 rows of act x 256 of W read 2 x (128 + 256), and only 16 columns at a time are padding.
// A tile takes up to 256 rows of an expert or up to 128, which the caller says (ops.moe_tc5_rows has the times of both): tiles of
// 128 fill tensor memory with two pairs of accumulators, and one is written out under the products of the next.  2,000 tokens,
// K 2,048, 2 x 1,408 features: 223 us with act on the M side in rows padded to 128, 162 now; down (K 1,408, 2,048 features): 134 and
// 89.  128 tokens: 148 and 115, 89 and 61; twice the width, 8 experts a token: 722 and 555, 408 and 288; 2,048 tokens of 2 of 8
// experts (512 rows each; tiles of 256 alone: 65 and 41): 51 and 50, 32 and 27; 2,000 tokens of 2 of 4, K 512, 2 x 72 features 9.6 and 10.
//
// One persistent block per SM, warp-specialised: warp 0 brings stages of 64 k in by TMA (128-byte swizzle; 2 x 128 rows of
// W, the rows of act by boxes of 64; a ring of 3, or 4 with tiles of 128), warp 1 issues the products, all lanes walking together
// (from a branch of one lane 123 us for 119 and 67 for 64 at 300 tokens of 6 of 64), into two accumulators of up to 256 float columns
// (gate and up, or the two halves of 256 features: all of tensor memory), or two pairs of up to 128; warps 4-11 write them out, while
// the next tile's stages come in.
// Sizes: K and M multiples of 8.  Every wait is bounded; on a timeout the roles fall through to the common exit.
#include "tcgen05.cuh"

#define GE_BK 64
#define GE_W_BYTES (128 * GE_BK * 2)
#define GE_BOX 64                                             // rows of act in one copy
#define GE_BOX_BYTES (GE_BOX * GE_BK * 2)
#define GE_THREADS 384
#define GE_LIST 2048                                          // tiles of rows whose list is kept in shared memory

// GATED: W has 2 M rows an expert, gate rows then up rows; out (rows, M) bf16 = g sigmoid(alpha g) (u + shift) with g = min(gate,
// limit), u = clamp(up, -limit, limit), both first times the row's row_scale when that is given.  Else W has M rows an expert, out
// (rows, M) float32.
// ROWS: how many rows a tile takes at most, 256 or 128.
template <bool GATED, int ROWS>
__global__ void __launch_bounds__(GE_THREADS, 1)
gemm_experts_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap wmap, void* __restrict__ out, int tiles,
                    int M, int K, const int* __restrict__ groups, float limit, float alpha, float shift,
                    const float* __restrict__ row_scale, int* err) {
    constexpr int FEATS = GATED ? 128 : 256;                  // output features of one tile
    constexpr int STAGES = ROWS == 256 ? 3 : 4, STAGE_BYTES = 2 * GE_W_BYTES + ROWS * GE_BK * 2, BUFS = 256 / ROWS;
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)STAGES * STAGE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 5);
    const uint32_t stage0 = smem_u32(smem), full0 = smem_u32(bars), empty0 = full0 + 8 * STAGES, tfull = empty0 + 8 * STAGES,
                   tempty = tfull + 16, done = tempty + 16;
    const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
    __shared__ int list[GE_LIST];
    __shared__ int listed;

    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < BUFS; b++) { mbar_init(tfull + 8 * b, 1); mbar_init(tempty + 8 * b, 8); }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    // a tile of ROWS rows starts there: tiles of 128 everywhere, tiles of 256 on every other one of an expert
    auto starts = [](int v) { return v >= 0 && (ROWS == 128 || !(v >> 24)); };
    // the tiles where rows start, side by side, so that the blocks get equal shares (beyond GE_LIST tiles: as they come)
    const bool short_list = tiles <= GE_LIST;
    if (warp == 2) {
        int n = 0;
        for (int t = 0; short_list && t < tiles; t += 32) {
            const bool has = t + lane < tiles && starts(groups[t + lane]);
            const unsigned vote = __ballot_sync(0xffffffffu, has);
            if (has) list[n + __popc(vote & ((1u << lane) - 1))] = t + lane;
            n += __popc(vote);
        }
        if (lane == 0) listed = short_list ? n : tiles;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = warp_uniform(*tmem_slot);
    const int m_tiles = (M + FEATS - 1) / FEATS, kblocks = (K + GE_BK - 1) / GE_BK;
    const long long units = (long long)listed * m_tiles;
    // a unit: a tile of W's rows for the rows that start at a tile; neighbours share the rows
    struct Unit { int row0, rows, expert, m0; };
    auto unit_at = [&](long long u) {
        const int i = (int)(u / m_tiles), t = short_list ? list[i] : i, v = groups[t];
        return Unit{t * 128, starts(v) ? min(ROWS, v >> 12 & 4095) : 0, v & 4095, (int)(u % m_tiles) * FEATS};
    };

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;                                       // stages issued so far
            bool ok = true;
            for (long long u = blockIdx.x; u < units && ok; u += gridDim.x) {
                const Unit x = unit_at(u);
                if (x.rows <= 0) continue;
                const int boxes = (x.rows + GE_BOX - 1) / GE_BOX, w0 = x.expert * (GATED ? 2 * M : M) + x.m0, w1 = w0 + (GATED ? M : 128);
                for (int kb = 0; kb < kblocks; kb++, it++) {
                    const int s = it % STAGES, round = it / STAGES;
                    if (round > 0 && !mbar_wait(empty0 + 8 * s, (round - 1) & 1, err)) { ok = false; break; }
                    const uint32_t fb = full0 + 8 * s, dst = stage0 + s * STAGE_BYTES;
                    mbar_expect_tx(fb, 2 * GE_W_BYTES + boxes * GE_BOX_BYTES);
                    tma_load_2d(dst, &wmap, kb * GE_BK, w0, fb);
                    tma_load_2d(dst + GE_W_BYTES, &wmap, kb * GE_BK, w1, fb);
                    for (int b = 0; b < boxes; b++)
                        tma_load_2d(dst + 2 * GE_W_BYTES + b * GE_BOX_BYTES, &amap, kb * GE_BK, x.row0 + b * GE_BOX, fb);
                }
            }
            copies_landed(full0, STAGES, it, err);
        }
        __syncwarp();
    } else if (warp == 1) {
        // the whole warp walks, one lane issues (umma_f16_warp)
        auto wait = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)); };
        int s = 0, round = 0, j = 0;                          // stage, rounds of the ring, units done by this block
        bool ok = true;
        for (long long u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const int rows = warp_uniform(unit_at(u).rows);
            if (rows <= 0) continue;
            const int buf = j % BUFS, use = j / BUFS;
            if (use > 0 && !wait(tempty + 8 * buf, (use - 1) & 1)) break;
            tc_fence_after();
            const uint32_t idesc = umma_idesc(128, (rows + 15) / 16 * 16), d = tmem_base + buf * 256;
            for (int kb = 0; kb < kblocks; kb++) {
                if (!wait(full0 + 8 * s, round & 1)) { ok = false; break; }
                tc_fence_after();
                const uint32_t at = stage0 + s * STAGE_BYTES;
                const uint64_t w0 = umma_desc(at), w1 = umma_desc(at + GE_W_BYTES), a = umma_desc(at + 2 * GE_W_BYTES);
#pragma unroll
                for (int k = 0; k < GE_BK / 16; k++) {
                    umma_f16_warp(d, w0 + 2 * k, a + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_f16_warp(d + ROWS, w1 + 2 * k, a + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit_warp(empty0 + 8 * s);
                if (++s == STAGES) { s = 0; round++; }
            }
            if (!ok) break;
            umma_commit_warp(tfull + 8 * buf);
            j++;
        }
        products_landed<true>(done, err);
        __syncwarp();
    } else if (warp >= 4) {
        const int q = warp & 3, half = (warp - 4) >> 2;       // the 32 rows of W this warp may read; which groups of 16 columns
        int j = 0;
        for (long long u = blockIdx.x; u < units; u += gridDim.x) {
            const Unit x = unit_at(u);
            if (x.rows <= 0) continue;
            const int buf = j % BUFS, use = j / BUFS;
            const bool got = mbar_wait(tfull + 8 * buf, use & 1, err);
            if (!__all_sync(0xffffffffu, got)) break;
            j++;
            const uint32_t taddr = tmem_base + buf * 256 + ((uint32_t)(q * 32) << 16);
            tc_fence_after();
            const int m = x.m0 + q * 32 + lane;
            for (int c = half * 16; c < x.rows; c += 32) {
                uint32_t r[16], v[16];
                tmem_ld16(taddr + c, r);
                tmem_ld16(taddr + ROWS + c, v);
                tmem_ld_wait();
                const int n = min(16, x.rows - c);
                if (GATED) {
                    // all sixteen side by side, the stores alone depend on how many rows there are
                    bf16 o[16];
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const float rs = row_scale ? row_scale[x.row0 + c + min(i, n - 1)] : 1.0f;
                        // gate and up pass through bf16 as they do when the products are separate kernels
                        const float g = fminf(__bfloat162float(__float2bfloat16_rn(__uint_as_float(r[i]) * rs)), limit);
                        const float up = fminf(fmaxf(__bfloat162float(__float2bfloat16_rn(__uint_as_float(v[i]) * rs)), -limit), limit) + shift;
                        o[i] = __float2bfloat16_rn(__fdividef(g, 1.0f + __expf(-alpha * g)) * up);
                    }
                    bf16* dst = reinterpret_cast<bf16*>(out) + (size_t)(x.row0 + c) * M + m;
#pragma unroll
                    for (int i = 0; i < 16; i++, dst += M)
                        if (i < n && m < M) *dst = o[i];
                } else {
                    float* dst = reinterpret_cast<float*>(out) + (size_t)(x.row0 + c) * M + m;
#pragma unroll
                    for (int i = 0; i < 16; i++, dst += M) {
                        if (i < n && m < M) *dst = __uint_as_float(r[i]);
                        if (i < n && m + 128 < M) dst[128] = __uint_as_float(v[i]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty + 8 * buf);
        }
    }
    // common exit: every role comes here, also after a wait that ran out; then the tensor memory is given back
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <bool GATED, int ROWS>
static int experts_launch(const void* act, const void* W, void* out, int N, int M, int K, const int* groups, int experts, float limit,
                          float alpha, float shift, const float* row_scale, int* err, cudaStream_t st) {
    if (N == 0 || M == 0) return 0;
    if (!groups || experts < 1 || experts > 4096 || N % 128 || K % 8 || M % 8 || K < 8 || (reinterpret_cast<uintptr_t>(W) & 15) ||
        (reinterpret_cast<uintptr_t>(act) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) ||
        (long long)experts * (GATED ? 2 : 1) * M + 256 > 0x7fffffffLL)
        return -2;
    CUtensorMap amap, wmap;
    int rc = matrix_map(act, N, K, GE_BOX, &amap);
    if (rc) return rc;
    rc = matrix_map(W, (long long)(GATED ? 2 : 1) * M * experts, K, 128, &wmap);
    if (rc) return rc;
    constexpr int STAGES = ROWS == 256 ? 3 : 4;
    constexpr size_t smem = 1024 + (size_t)STAGES * (2 * GE_W_BYTES + ROWS * GE_BK * 2) + (2 * STAGES + 5) * 8 + 16;
    static bool configured = false;
    static int sms = 0;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_experts_kernel<GATED, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
        configured = true;
    }
    gemm_experts_kernel<GATED, ROWS><<<sms, GE_THREADS, smem, st>>>(amap, wmap, out, N / 128, M, K, groups, limit, alpha, shift, row_scale, err);
    MB_LAUNCH_CHECK();
    return 0;
}

// act (N, K) with N a multiple of 128, laid out and described by groups (N / 128) as above.  W (experts, 2 M, K), gate rows then up
// rows of each expert; out (N, M) bf16; rows that are no expert's are left as they are.
MB_API int mb_gemm_experts_gated_bf16(const void* act, const void* W, void* out, int N, int M, int K, const int* groups, int experts,
                                      int most, float limit, float alpha, float shift, const float* row_scale, int* err,
                                      cudaStream_t st) {
    return most == 128 ? experts_launch<true, 128>(act, W, out, N, M, K, groups, experts, limit, alpha, shift, row_scale, err, st)
                       : experts_launch<true, 256>(act, W, out, N, M, K, groups, experts, limit, alpha, shift, row_scale, err, st);
}
// W (experts, M, K); out (N, M) float32
MB_API int mb_gemm_experts_f32out(const void* act, const void* W, void* out, int N, int M, int K, const int* groups, int experts, int most,
                                  int* err, cudaStream_t st) {
    return most == 128 ? experts_launch<false, 128>(act, W, out, N, M, K, groups, experts, 0.0f, 0.0f, 0.0f, nullptr, err, st)
                       : experts_launch<false, 256>(act, W, out, N, M, K, groups, experts, 0.0f, 0.0f, 0.0f, nullptr, err, st);
}
