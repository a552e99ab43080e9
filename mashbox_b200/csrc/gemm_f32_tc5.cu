// True 32-bit matrix product on the tensor cores: C[n, m] = sum_k A[n, k] * W[m, k], float32 operands and results.
//
// Every float32 operand, times 2^24, is cut into three bf16 numbers that add up to it exactly, x = h + m + l (h its upper 8
// significant bits, m the rest rounded to 8, l what is left; the factor keeps the last bit of the smallest subnormal above
// what a bf16 can hold), so a product is a sum of exact bf16 products.  Eight of the nine run as tcgen05.mma (kind::f16, float
// accumulator); l l, left out, is at most 2^-32 of the product.  The tensor cores cut off the low bits of what they add to an
// accumulator instead of rounding it, so h h, which carries the result, has an accumulator of its own that takes ONE block of
// 32 k (a single product of 16 bits lies in it exactly) and is then added, rounded to nearest, to a sum in registers.  The
// other seven, together at most 2^-6 of the product, share two accumulators over up to 512 k and are added to that sum, rounded
// to nearest.  So a result that one product decides is that product rounded once, as a fused multiply-add rounds it,
// and sums of many are nearer to 64 bits than one chain of fused multiply-adds over k (gemm_f32.cu): relative error 0.8e-7 /
// 1.0e-7 / 1.6e-7 at K 512 / 2,048 / 8,192 on normal values, the chain's 4e-7 / 8e-7 / 16e-7; measured by the sum of the products'
// magnitudes the worst element is nearer too, but where two to a few products of one block of 32 decide a result, what h h is cut
// off by (up to 2^-23) beside the last rounding is some 1.6 times the chain's few roundings (tests/test_float32_split_gpu.py).
// (With h h in one accumulator with the rest and m l, l m left out, up to 2^-22 of a product was missing; a block was 12 instructions
// then, not 10, but 256 rows of A fitted: 509 x 2048 x 2048 37 us, now 48.)  Bound by the chain of a stage: 0.73 us with 128 rows of A,
// tensor pipes busy 0.59 of it; before the products waited on one barrier alone 0.77, 0.58 with 2 of the 10 instructions, 0.51 without
// the cutting besides; more stages of either ring bring nothing.  W's planes in tensor memory, so that the instructions read half
// as much shared memory, 0.97 (16 instructions, two waits).  The FMA units' product at the same size and this one, us: 509 x 16384 x
// 2048 684 and 247, 509 x 2048 x 8192 491 and 119, 509 x 2048 x 2048 123 and 48, one row x 2048 x 2048 97 and 18.
//
// An output is the same operations in the same order however many rows a call has: blocks of 32 k in ascending order
// within a quarter of K, the quarters' sums in ascending order.  Tiles, and whether one block or a cluster of four goes
// through the quarters, change no bit.
//
// One block: 128 rows of W (the M side of the instructions) x TN rows of A, warp-specialised:
//   warp 0      TMA: 128 x 32 floats of W per stage into a ring of 4
//   warp 2      TMA: the three bf16 planes of TN x 32 values of A (64-byte swizzle), cut by split_rows_kernel beforehand:
//               they are read once per tile of W, W once per tile of A
//   warps 4-7   cut a stage of W into its three planes in shared memory, as the instructions want them
//   warp 3      tells the products' barrier that planes of A have come
//   warp 1      one lane issues the products; accumulators of TN columns, two in turn for h h, two side by side for the rest
//   warps 8-15  add the accumulators to the sums in registers (thread = a row of W, half of the columns)
// A cluster of four blocks takes a quarter of K each where the tiles alone leave the device idle: the sums meet in
// shared memory.  A single block puts the sum of a quarter down in C and adds the next to it.
//
// A result that is not finite is computed again as one chain of fused multiply-adds (fs_chains), so infinities and NaN come out as
// the plain product has them: an infinite operand has no such parts, and sums from 2^80 on overflow with the factors of 2^24.
// The cut into three parts is that of Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for
// higher-precision computations" (2019).
#include "tcgen05.cuh"

MB_PDL_SWITCH(mb_gemm_f32_tc5_set_pdl)              // the product starts, and brings W in, while the planes are cut

#define FS_BK 32                                   // k of a stage and of an accumulator
#define FS_RAW 4                                   // stages of W as it comes
#define FS_RAW_BYTES (128 * FS_BK * 4)
#define FS_W_PLANE (128 * FS_BK * 2)
#define FS_THREADS 512
#define FS_PERIOD 16                               // blocks of 32 k that the accumulators of the small parts take at most
#define FS_UP 16777216.0f                          // 2^24: what operands are multiplied by before they are cut
#define FS_DOWN 3.5527136788005009e-15f            // 2^-48: what sums are multiplied by

template <int TN> struct FsShape {
    static constexpr int X_PLANE = TN * FS_BK * 2;
    static constexpr int STAGE = 3 * FS_W_PLANE + 3 * X_PLANE;
    static constexpr int STAGES = TN == 128 ? 3 : 4;
    static constexpr int TMEM = 4 * TN;                        // two accumulators of h h in turn, two side by side of the rest
    static constexpr int SMEM = 1024 + STAGES * STAGE + FS_RAW * FS_RAW_BYTES + 320;
};

// four floats -> the three bf16 parts of 2^24 times each, two to a word.  h is cut off, m is rounded, l is exact.
__device__ __forceinline__ void fs_split4(const float4 v, uint2& h, uint2& m, uint2& l) {
    const float4 x = make_float4(v.x * FS_UP, v.y * FS_UP, v.z * FS_UP, v.w * FS_UP);
    const uint32_t a = __float_as_uint(x.x), b = __float_as_uint(x.y), c = __float_as_uint(x.z), d = __float_as_uint(x.w);
    h.x = __byte_perm(a, b, 0x7632);
    h.y = __byte_perm(c, d, 0x7632);
    const float ra = x.x - __uint_as_float(a & 0xffff0000u), rb = x.y - __uint_as_float(b & 0xffff0000u);
    const float rc = x.z - __uint_as_float(c & 0xffff0000u), rd = x.w - __uint_as_float(d & 0xffff0000u);
    m.x = pack_bf16(ra, rb);
    m.y = pack_bf16(rc, rd);
    l.x = pack_bf16(ra - __uint_as_float(m.x << 16), rb - __uint_as_float(m.x & 0xffff0000u));
    l.y = pack_bf16(rc - __uint_as_float(m.y << 16), rd - __uint_as_float(m.y & 0xffff0000u));
}

// A (N, K) -> planes (3, N, Kp) bf16, Kp = K rounded up to 8, zeros behind K.  A thread cuts four values.
template <bool VEC>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ A, bf16* __restrict__ planes, int N, int K, int Kp) {
    const int quads = Kp / 4;
    const size_t total = (size_t)N * quads, plane = (size_t)N * Kp;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (size_t)gridDim.x * 256) {
        const int n = (int)(i / quads), k = (int)(i % quads) * 4;
        const float* p = A + (size_t)n * K + k;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (k < K) x = VEC ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
        uint2 h, m, l;
        fs_split4(x, h, m, l);
        uint2* o = reinterpret_cast<uint2*>(planes + (size_t)n * Kp + k);
        o[0] = h;
        o[plane / 4] = m;
        o[plane / 2] = l;
    }
    pdl_launch_dependents();
}

// the shared-memory descriptor of a K-major tile of 64-byte rows with the 64-byte swizzle (8 rows 512 bytes apart, version 1, layout
// type 4): only its low word, the address in units of 16 bytes, differs from product to product
__device__ __forceinline__ uint64_t fs_desc(uint32_t lo) {
    constexpr uint32_t HI = (512u >> 4) | (1u << 14) | (4u << 29);
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(d) : "r"(lo), "r"(HI));
    return d;
}

__device__ __forceinline__ void fs_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}

// sum += (first: =) the HALF columns of an accumulator from taddr on
template <int HALF> __device__ __forceinline__ void fs_add(uint32_t taddr, bool first, float (&sum)[HALF]) {
    constexpr int B = HALF < 32 ? HALF : 32;
#pragma unroll
    for (int c = 0; c < HALF; c += B) {
        uint32_t r[32];
        if (B == 32) tmem_ld32(taddr + c, r);
        else {
#pragma unroll
            for (int j = 0; j < B; j += 8) fs_ld8(taddr + c + j, r + j);
        }
        tmem_ld_wait();
        if (first) {
#pragma unroll
            for (int j = 0; j < B; j++) sum[c + j] = __uint_as_float(r[j]);
        } else {
#pragma unroll
            for (int j = 0; j < B; j++) sum[c + j] += __uint_as_float(r[j]);
        }
    }
}

// sum += the two accumulators of the small parts, TN columns apart
template <int HALF, int TN> __device__ __forceinline__ void fs_add_small(uint32_t taddr, float (&sum)[HALF]) {
    constexpr int B = HALF < 16 ? HALF : 16;
#pragma unroll
    for (int c = 0; c < HALF; c += B) {
        uint32_t r[B], t[B];
#pragma unroll
        for (int j = 0; j < B; j += 8) {
            fs_ld8(taddr + c + j, r + j);
            fs_ld8(taddr + TN + c + j, t + j);
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < B; j++) sum[c + j] += __uint_as_float(r[j]) + __uint_as_float(t[j]);
    }
}

__device__ __forceinline__ bool fs_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }

// The results of a block's tile that are not finite, as chains of fused multiply-adds in ascending k: `odd` has a bit for every column
// that holds one.  The whole block goes through them, 32 columns at a time, operands staged in shared memory (buf); a thread has a row of
// W and eight columns.  (A thread by itself for each such result made 509 rows of NaN x 16384 x 2048 take 71 ms, now 4.1; one such row 0.62.)
__device__ __noinline__ void fs_chains(float* buf, const uint32_t* odd, int words, const float* __restrict__ A, const float* __restrict__ W,
                                       float* C, int M, int K, int ldc, int tok0, int m0) {
    constexpr int PITCH = 36;                                  // floats of a staged row of 32: 16-byte reads of 8 rows side by side
    float *ws = buf, *as = buf + 128 * PITCH;
    int *list = reinterpret_cast<int*>(as + 32 * PITCH), count = 0;
    for (int i = 0; i < words; i++)
        for (uint32_t left = odd[i]; left; left &= left - 1, count++)
            if (threadIdx.x == 0) list[count] = i * 32 + __ffs(left) - 1;
    const int r = threadIdx.x & 127, g = threadIdx.x >> 7;
    for (int base = 0; base < count; base += 32) {
        float acc[8] = {};
        for (int k0 = 0; k0 < K; k0 += 32) {
            __syncthreads();
            for (int e = threadIdx.x; e < 128 * 8; e += FS_THREADS) {
                const int row = e >> 3, k = (e & 7) * 4;
                if (m0 + row < M && k0 + k < K)
                    *reinterpret_cast<float4*>(ws + row * PITCH + k) = *reinterpret_cast<const float4*>(W + (size_t)(m0 + row) * K + k0 + k);
            }
            for (int e = threadIdx.x; e < 32 * 32; e += FS_THREADS) {
                const int col = e >> 5, k = e & 31;
                if (base + col < count && k0 + k < K) as[col * PITCH + k] = A[(size_t)(tok0 + list[base + col]) * K + k0 + k];
            }
            __syncthreads();
            const int depth = min(32, K - k0);                  // a multiple of 4
            for (int k = 0; k < depth; k += 4) {
                const float4 w = *reinterpret_cast<const float4*>(ws + r * PITCH + k);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float4 a = *reinterpret_cast<const float4*>(as + (g * 8 + j) * PITCH + k);
                    acc[j] = fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, acc[j]))));
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (m0 + r < M && base + g * 8 + j < count) {
                float* p = C + (size_t)(tok0 + list[base + g * 8 + j]) * ldc + m0 + r;
                if (!fs_finite(*p)) *p = acc[j];
            }
    }
}

__device__ __forceinline__ float fs_ld_cluster(uint32_t addr, int rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void fs_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// CL blocks of a cluster: 1 (the block goes through all of K) or 4 (block r through the r-th quarter)
template <int TN, int CL>
__global__ void __launch_bounds__(FS_THREADS, 1)
gemm_f32_tc5_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const float* __restrict__ A,
                    const float* __restrict__ W, float* C, int N, int M, int K, int ldc, int* err) {
    using S = FsShape<TN>;
    constexpr int HALF = TN / 2;                               // columns of a warp of the last two groups
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
    const uint32_t stage0 = smem_u32(smem), raw0 = stage0 + S::STAGES * S::STAGE;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::STAGES * S::STAGE + FS_RAW * FS_RAW_BYTES);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t*>(bars + 32), *odd = tmem_slot + 1;
    constexpr int ODD = (TN + 31) / 32;                        // a bit for every column of the tile with a result that is not finite
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * S::STAGES, rfull0 = empty0 + 8 * S::STAGES,
                   rempty0 = rfull0 + 8 * FS_RAW, tfull0 = rempty0 + 8 * FS_RAW, sfull = tfull0 + 16, sempty = sfull + 8,
                   xfull0 = sempty + 8, done = xfull0 + 8 * S::STAGES;
    const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;

    if (tid == 0) {
        // a stage: four warps that cut W, the planes of A, eight warps that have read the accumulator it goes to
        for (int s = 0; s < S::STAGES; s++) { mbar_init(full0 + 8 * s, 13); mbar_init(xfull0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int s = 0; s < FS_RAW; s++) { mbar_init(rfull0 + 8 * s, 1); mbar_init(rempty0 + 8 * s, 4); }
        for (int a = 0; a < 2; a++) mbar_init(tfull0 + 8 * a, 1);
        mbar_init(sfull, 1);
        mbar_init(done, 1);
        for (int i = 0; i < ODD; i++) odd[i] = 0;
        mbar_init(sempty, 8);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), S::TMEM);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = warp_uniform(*tmem_slot);

    // neighbours share a tile of W: it is read from memory once
    const int tile = blockIdx.x / CL, rank = CL == 1 ? 0 : blockIdx.x % CL, tok_tiles = (N + TN - 1) / TN;
    const int tok0 = tile % tok_tiles * TN, m0 = tile / tok_tiles * 128;
    const int blocks = (K + FS_BK - 1) / FS_BK, quarter = (blocks + 3) / 4, quarters = (blocks + quarter - 1) / quarter;
    const int kb0 = CL == 1 ? 0 : min(rank * quarter, blocks), nb = CL == 1 ? blocks : min(quarter, blocks - kb0);

    if (warp < 4) {
        if (warp == 0 && lane == 0) {
            int i = 0;
            for (; i < nb; i++) {
                const int s = i % FS_RAW, round = i / FS_RAW;
                if (round > 0 && !mbar_wait(rempty0 + 8 * s, (round - 1) & 1, err)) break;
                mbar_expect_tx(rfull0 + 8 * s, FS_RAW_BYTES);
                tma_load_2d(raw0 + s * FS_RAW_BYTES, &wmap, (kb0 + i) * FS_BK, m0, rfull0 + 8 * s);
            }
            copies_landed(rfull0, FS_RAW, i, err);
        } else if (warp == 2 && lane == 0) {
            pdl_wait();                                        // the planes are the kernel before's
            int i = 0;
            for (; i < nb; i++) {
                const int s = i % S::STAGES, round = i / S::STAGES;
                if (round > 0 && !mbar_wait(empty0 + 8 * s, (round - 1) & 1, err)) break;
                const uint32_t fb = xfull0 + 8 * s, dst = stage0 + s * S::STAGE + 3 * FS_W_PLANE;
                mbar_expect_tx(fb, 3 * S::X_PLANE);
#pragma unroll
                for (int p = 0; p < 3; p++) tma_load_2d(dst + p * S::X_PLANE, &xmap, (kb0 + i) * FS_BK, p * N + tok0, fb);
            }
            copies_landed(xfull0, S::STAGES, i, err);
        } else if (warp == 3 && lane == 0) {
            // the planes of A have a barrier of their own, so that their copies can be waited for by themselves; the products wait on one
            // barrier a stage, which hears of them from here (with two waits a stage of 16 rows took 0.84 us, not 0.6)
            for (int i = 0; i < nb; i++) {
                if (!mbar_wait(xfull0 + 8 * (i % S::STAGES), (i / S::STAGES) & 1, err)) break;
                mbar_arrive(full0 + 8 * (i % S::STAGES));
            }
        } else if (warp == 1) {
            // the whole warp walks, one lane issues (umma_f16_warp)
            constexpr uint32_t one = umma_idesc(128, TN), two = umma_idesc(128, 2 * TN);
            auto wait = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)); };
            int s = 0, round = 0, at = 0, periods = 0;          // at: blocks into the quarter; periods of the small parts begun
            const uint32_t small = tmem_base + 2 * TN;
            for (int i = 0; i < nb; i++) {
                const int acc = i & 1;
                if (!wait(full0 + 8 * s, round & 1)) break;
                tc_fence_after();
                // planes of 128 rows of W; planes of TN rows of A, one below the other: h m and m l are tiles of 2 TN rows
                const uint32_t w = (stage0 + s * S::STAGE) >> 4, x = w + (3 * FS_W_PLANE >> 4);
                constexpr uint32_t WP = FS_W_PLANE >> 4, XP = S::X_PLANE >> 4;
#pragma unroll
                for (int k = 0; k < 4; k += 2) umma_f16_warp(tmem_base + acc * TN, fs_desc(w + k), fs_desc(x + k), one, k > 0);
                umma_commit_warp(tfull0 + 8 * acc);
                const bool fresh = at % FS_PERIOD == 0;
                if (fresh) {
                    if (periods > 0 && !wait(sempty, (periods - 1) & 1)) break;
                    tc_fence_after();
                    periods++;
                }
#pragma unroll
                for (int k = 0; k < 4; k += 2) {
                    umma_f16_warp(small, fs_desc(w + WP + k), fs_desc(x + k), two, k > 0 || !fresh);            // m h, m m
                    umma_f16_warp(small, fs_desc(w + k), fs_desc(x + XP + k), two, 1u);                         // h m, h l
                    umma_f16_warp(small, fs_desc(w + 2 * WP + k), fs_desc(x + k), two, 1u);                     // l h, l m
                    umma_f16_warp(small, fs_desc(w + WP + k), fs_desc(x + 2 * XP + k), one, 1u);                // m l
                }
                umma_commit_warp(empty0 + 8 * s);
                at++;
                if (at % FS_PERIOD == 0 || at == quarter || i + 1 == nb) umma_commit_warp(sfull);
                if (at == quarter) at = 0;
                if (++s == S::STAGES) { s = 0; round++; }
            }
            products_landed<true>(done, err);
        }
        __syncwarp();
    } else if (warp < 8) {
        const int t = tid - 128;
        for (int i = 0; i < nb; i++) {
            const int rs = i % FS_RAW, s = i % S::STAGES, round = i / S::STAGES;
            const bool got = mbar_wait(rfull0 + 8 * rs, (i / FS_RAW) & 1, err);
            if (!__all_sync(0xffffffffu, got)) break;
            uint2 h[8], m[8], l[8];                             // cut before the stage they go to is waited for
            const unsigned char* raw = smem + S::STAGES * S::STAGE + rs * FS_RAW_BYTES;
#pragma unroll
            for (int j = 0; j < 8; j++) fs_split4(*reinterpret_cast<const float4*>(raw + (t + j * 128) * 16), h[j], m[j], l[j]);
            const bool free_ = round == 0 || mbar_wait(empty0 + 8 * s, (round - 1) & 1, err);
            if (!__all_sync(0xffffffffu, free_)) break;
            unsigned char* dst = smem + s * S::STAGE;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int row = (t >> 3) + j * 16, c = t & 7;           // four values: half of the row's 16-byte piece c / 2
                unsigned char* p = dst + row * 64 + (((c >> 1) ^ ((row >> 1) & 3)) << 4) + (c & 1) * 8;
                *reinterpret_cast<uint2*>(p) = h[j];
                *reinterpret_cast<uint2*>(p + FS_W_PLANE) = m[j];
                *reinterpret_cast<uint2*>(p + 2 * FS_W_PLANE) = l[j];
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(full0 + 8 * s);
                mbar_arrive(rempty0 + 8 * rs);
            }
        }
    } else {
        const int q = warp & 3, half = (warp - 8) >> 2, m = m0 + q * 32 + lane;
        const uint32_t taddr = tmem_base + half * HALF + ((uint32_t)(q * 32) << 16);
        float sum[HALF];
#pragma unroll
        for (int j = 0; j < HALF; j++) sum[j] = 0.0f;
        float* out = C + (size_t)(tok0 + half * HALF) * ldc + m;
        const int cols = m < M ? min(HALF, N - tok0 - half * HALF) : 0;        // columns this thread has (0 or less: none)
        bool some = false;
        int at = 0, periods = 0;                                // as the products count them
        // an accumulator that has been read is among the arrivals that the products of the block after the next wait for
        if (lane == 0) {
            mbar_arrive(full0);
            if (nb > 1) mbar_arrive(full0 + 8);
        }
        pdl_wait();
        for (int i = 0; i < nb; i++) {
            const int acc = i & 1;
            bool got = mbar_wait(tfull0 + 8 * acc, (i >> 1) & 1, err);
            if (!__all_sync(0xffffffffu, got)) break;
            tc_fence_after();
            fs_add<HALF>(taddr + acc * TN, at == 0, sum);
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && i + 2 < nb) mbar_arrive(full0 + 8 * ((i + 2) % S::STAGES));
            at++;
            const bool ends = at == quarter || i + 1 == nb;
            if (ends || at % FS_PERIOD == 0) {
                got = mbar_wait(sfull, periods & 1, err);
                if (!__all_sync(0xffffffffu, got)) break;
                periods++;
                tc_fence_after();
                fs_add_small<HALF, TN>(taddr + 2 * TN, sum);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(sempty);
            }
            if (ends) {
#pragma unroll
                for (int j = 0; j < HALF; j++) sum[j] *= FS_DOWN;
            }
            if (CL == 1 && ends) {
                const bool start = i < quarter, last = i + 1 == nb;
                constexpr int B = 8;
                int step = ldc;
                asm volatile("" : "+r"(step));                  // the addresses are made here, not kept over the loop
                float* p = out;
#pragma unroll
                for (int c = 0; c < HALF; c += B, p += (size_t)B * step) {
                    float before[B];
#pragma unroll
                    for (int j = 0; j < B; j++) before[j] = !start && c + j < cols ? p[(size_t)j * step] : 0.0f;
#pragma unroll
                    for (int j = 0; j < B; j++) {
                        const float v = start ? sum[c + j] : before[j] + sum[c + j];
                        if (c + j < cols) {
                            p[(size_t)j * step] = v;
                            if (last) some |= !fs_finite(v);
                        }
                    }
                }
            }
            if (at == quarter) at = 0;
        }
        if (CL == 1 && some) {
            for (int c = 0; c < cols; c++)
                if (!fs_finite(out[(size_t)c * ldc])) atomicOr(odd + (half * HALF + c) / 32, 1u << ((half * HALF + c) % 32));
        }
        if (CL > 1) {
            // every product and copy of this block is done: its sums go where the stages lay, a row of 128 for every column
            float* ex = reinterpret_cast<float*>(smem);
#pragma unroll
            for (int j = 0; j < HALF; j++) ex[(half * HALF + j) * 128 + q * 32 + lane] = sum[j];
        }
    }
    if (CL > 1) {
        __syncwarp();
        fs_cluster_sync();
        if (warp >= 8) {
            constexpr int MINE = TN / CL;                       // columns this block adds up
            const int r = tid & 127, m = m0 + r, c0 = rank * MINE;
            bool some = false;
            for (int c = (tid - 256) >> 7; c < MINE; c += 2) {
                const int n = tok0 + c0 + c;
                float v = 0.0f;
                for (int b = 0; b < quarters; b++) {
                    const float x = fs_ld_cluster(stage0 + ((c0 + c) * 128 + r) * 4, b);
                    v = b == 0 ? x : v + x;
                }
                if (n < N && m < M) {
                    some |= !fs_finite(v);
                    C[(size_t)n * ldc + m] = v;
                }
            }
            if (some)
                for (int c = (tid - 256) >> 7; c < MINE; c += 2)
                    if (tok0 + c0 + c < N && m < M && !fs_finite(C[(size_t)(tok0 + c0 + c) * ldc + m]))
                        atomicOr(odd + (c0 + c) / 32, 1u << ((c0 + c) % 32));
        }
        __syncwarp();
        fs_cluster_sync();                                      // nobody leaves while its sums are read
    }
    // common exit: every role comes here, also after a wait that ran out; then the tensor memory is given back
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, S::TMEM);
    }
    uint32_t any = 0;
#pragma unroll
    for (int i = 0; i < ODD; i++) any |= odd[i];
    if (any) fs_chains(reinterpret_cast<float*>(smem), odd, ODD, A, W, C, M, K, ldc, tok0, m0);
}

// ------------------------------------------------------------------------------------------------ host side
static int fs_map(const void* base, CUtensorMapDataType type, int item, long long rows, int cols, int box_cols, int box_rows,
                  CUtensorMapSwizzle swizzle, CUtensorMap* out) {
    EncodeTiled enc = encode_fn();
    if (!enc) return -6;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * item};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, estr[2] = {1u, 1u};
    return enc(out, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -6;
}

template <int TN, int CL>
static int fs_launch(const CUtensorMap& wmap, const float* A, const float* W, float* C, const bf16* planes, int N, int M, int K, int Kp,
                     int ldc, int* err, cudaStream_t st) {
    CUtensorMap xmap;
    int rc = fs_map(planes, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 3LL * N, Kp, FS_BK, TN, CU_TENSOR_MAP_SWIZZLE_64B, &xmap);
    if (rc) return rc;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc5_kernel<TN, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, FsShape<TN>::SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const long long grid = (long long)((N + TN - 1) / TN) * ((M + 127) / 128) * CL;
    if (grid > 0x7fffffffLL) return -2;
    cudaError_t e = mb_launch_cluster(mb_pdl, CL, gemm_f32_tc5_kernel<TN, CL>, dim3((unsigned)grid), dim3(FS_THREADS), FsShape<TN>::SMEM,
                                      st, wmap, xmap, A, W, C, N, M, K, ldc, err);
    if (e != cudaSuccess) return (int)e;
    MB_LAUNCH_CHECK();
    return 0;
}

// blocks the device holds at once, and clusters of four of them (a block fills an SM): asked for once, on the device of the first call
struct FsSlots { int blocks, clusters; };
static FsSlots fs_ask() {
    FsSlots s = {148, 35};
    int dev = 0, sms = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        return s;
    s = {sms, sms / 4 > 2 ? sms / 4 - 2 : 1};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 4;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(4);
    cfg.blockDim = dim3(FS_THREADS);
    cfg.dynamicSmemBytes = FsShape<128>::SMEM;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(gemm_f32_tc5_kernel<128, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, FsShape<128>::SMEM) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, gemm_f32_tc5_kernel<128, 4>, &cfg) == cudaSuccess && n > 0)
        s.clusters = n;
    else
        cudaGetLastError();
    return s;
}

// The tile: rows of A a block, and whether a cluster shares K.  Cost of a choice = rounds of blocks x (stages x time of a stage +
// what a block costs beside them), both as measured (one tile size alone on 2,048 and 8,192 k; the sums of the quarters through C
// are in it).  us, 64 alone / 128 alone / 128 in fours: 509 x 16384 x 2048 340 / 247 / 338, 509 x 2048 x 2048 54 / 64 / 48, 509 x 2048 x
// 8192 183 / 202 / 119, 509 x 3072 x 2048 99 / 65 / 69, 300 x 16384 x 2048 237 / 188 / 257, 64 x 2048 x 256 14 / 20 / 13 (32 in fours
// 8.6); one row x 2048 x 2048: 16 alone 47, in fours 18.
static void fs_choose(int N, int M, int K, int* tn, int* cl) {
    static const int TNS[4] = {16, 32, 64, 128};
    static const int STAGE_NS[4][2] = {{575, 575}, {630, 600}, {680, 650}, {740, 760}};
    static const int BLOCK_NS[4][2] = {{4000, 6000}, {5000, 6000}, {9000, 7000}, {16000, 10000}};
    static const FsSlots held = fs_ask();
    const long long blocks = (K + FS_BK - 1) / FS_BK, quarter = (blocks + 3) / 4, rows = (M + 127) / 128;
    long long best = -1;
    for (int i = 0; i < 4; i++)
        for (int c = 0; c < 2; c++) {
            const long long units = rows * ((N + TNS[i] - 1) / TNS[i]), slots = c ? held.clusters : held.blocks;
            const long long cost = (units + slots - 1) / slots * ((c ? quarter : blocks) * STAGE_NS[i][c] + BLOCK_NS[i][c]);
            if (best < 0 || cost < best) { best = cost; *tn = TNS[i]; *cl = c ? 4 : 1; }
        }
}

MB_API int mb_gemm_f32_tc5_supports(const void* W, int M, int K) {
    return K % 4 == 0 && K >= 128 && M >= 64 && (reinterpret_cast<uintptr_t>(W) & 15) == 0;
}

// planes: 3 x N x (K rounded up to 8) bf16, working memory.  rows of C are ldc floats apart.  tile (16, 32, 64 or 128 rows of A
// a block; more: 128) and cluster (1 or 4 blocks share K): 0 leaves the choice to the sizes; the result is the same.
MB_API int mb_gemm_f32_tc5(const float* A, const float* W, float* C, bf16* planes, int N, int M, int K, int ldc, int tile, int cluster,
                           int* err, cudaStream_t st) {
    if (N == 0 || M == 0) return 0;
    if (ldc < M || !mb_gemm_f32_tc5_supports(W, M, K) || (reinterpret_cast<uintptr_t>(planes) & 15)) return -2;
    const int Kp = (K + 7) / 8 * 8;
    int tn, cl;
    fs_choose(N, M, K, &tn, &cl);
    if (tile) tn = tile < 128 ? tile : 128;
    if (cluster) cl = cluster;
    CUtensorMap wmap;
    int rc = fs_map(W, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, M, K, FS_BK, 128, CU_TENSOR_MAP_SWIZZLE_NONE, &wmap);
    if (rc) return rc;
    const size_t quads = (size_t)N * (Kp / 4);
    const unsigned grid = (unsigned)((quads + 255) / 256 < 2368 ? (quads + 255) / 256 : 2368);
    if ((reinterpret_cast<uintptr_t>(A) & 15) == 0) split_rows_kernel<true><<<grid, 256, 0, st>>>(A, planes, N, K, Kp);
    else split_rows_kernel<false><<<grid, 256, 0, st>>>(A, planes, N, K, Kp);
    MB_LAUNCH_CHECK();
#define FS_CASE(TN)                                                                                      \
    if (tn == TN) return cl == 1 ? fs_launch<TN, 1>(wmap, A, W, C, planes, N, M, K, Kp, ldc, err, st)   \
                                 : fs_launch<TN, 4>(wmap, A, W, C, planes, N, M, K, Kp, ldc, err, st);
    FS_CASE(16) FS_CASE(32) FS_CASE(64) FS_CASE(128)
#undef FS_CASE
    return -2;
}
