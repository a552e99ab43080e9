// Paged attention, plain form: one warp per (token, query head), keys in ascending position through the block table.
// It serves the whole float32 path and, on the bf16 path, every head size the tensor-core kernel does not take.
// Runs of tokens of one sequence go to a tiled form of the same arithmetic (float32, no window).
// Scores, softmax and the weighted sum are float.  The order of every sum depends only on the query's position and
// the window, never on how tokens were cut into steps or which pages hold the keys.
//
// Keys and values may differ in width (HD values of a key row enter the score, HDV values of a value row the sum) and a
// row of either pool may be wider than what is read of it (k_row, v_row: the distance between two positions' rows; a
// pool whose rows are key and value at once is handed in twice).  Optional: a cap on the scores, s <- cap tanh(s / cap);
// a sink per query head, one more term exp(sink_h) in the softmax's denominator that has no value; a gate per token and
// query head, the head's result times sigmoid(gate); behind a window, the first `keep` positions stay visible.
#include "common.cuh"

#define SIMPLE_MAX_HD 1024         // the widest rows (three instantiations: up to 256, up to 512, and up to this)
#define WARPS 4

// Which tokens the tiled form (below) takes: the step's tokens are looked at in tiles of `tile` neighbours; a run of at least
// SIMPLE_RUN neighbours inside a tile that are tokens of one sequence in order is the tiled form's, the others -- decoded tokens,
// the ends of short portions, tokens in any other order -- are the plain form's.  Both forms compute the same bits.
#define SIMPLE_RUN 4
__device__ __forceinline__ bool simple_same(const int* __restrict__ tok_seq, const int* __restrict__ positions, int j, int n) {
    return tok_seq[j] == tok_seq[n] && positions[j] - positions[n] == j - n;
}

template <typename T, int MAXHD>
__global__ void __launch_bounds__(WARPS * 32) attn_simple_kernel(
    const T* __restrict__ q, int q_stride, T* __restrict__ out, const int* __restrict__ positions,
    const int* __restrict__ tok_seq, const int* __restrict__ table, int max_blocks, const T* __restrict__ kpool,
    const T* __restrict__ vpool, int N, int H, int KV, int HD, int page, int num_pages, int window, float scale,
    int* err, int HDV, int k_row, int v_row, float softcap, const float* __restrict__ sinks,
    const T* __restrict__ gate, int gate_stride, int keep, int tile) {
    __shared__ float qs[WARPS][MAXHD];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * WARPS + warp;
    if (item >= (long long)N * H) return;
    const int n = (int)(item / H), h = (int)(item % H);
    if (tile) {
        // the run around n: its tokens stand side by side (a tile has at most 64)
        const int t0 = n - n % tile, t1 = min(t0 + tile, N), i = n - t0;
        const bool lo = t0 + lane < t1 && simple_same(tok_seq, positions, t0 + lane, n);
        const bool hi = t0 + 32 + lane < t1 && simple_same(tok_seq, positions, t0 + 32 + lane, n);
        const unsigned long long same = __ballot_sync(0xffffffffu, lo) | (unsigned long long)__ballot_sync(0xffffffffu, hi) << 32;
        const unsigned long long after = ~(same >> i), before = i ? ~(same << (64 - i)) : ~0ull;       // zeros: the run's
        if ((after ? __ffsll(after) - 1 : 64) + __clzll(before) >= SIMPLE_RUN) return;
    }
    const int kvh = h / (H / KV);
    const int pos = positions[n];
    const int* tb = table + (size_t)tok_seq[n] * max_blocks;
    const T* qr = q + (size_t)n * q_stride + (size_t)h * HD;
    for (int d = lane; d < HD; d += 32) qs[warp][d] = mb_load(qr + d);
    __syncwarp();
    const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    float m = -INFINITY, l = 0.0f;
    float acc[MAXHD / 32];
#pragma unroll
    for (int i = 0; i < MAXHD / 32; i++) acc[i] = 0.0f;
    // the keys that are seen, numbered in ascending order: `front` kept ones, then the window's
    const int front = min(keep, lo), seen = front + pos - lo + 1;
    for (int base = 0; base < seen; base += 32) {
        const int kp = base + lane < front ? base + lane : lo + base + lane - front;
        const bool valid = base + lane < seen;
        long long off = -1;        // the position's row among the rows of its kv head's pages (times k_row or v_row)
        float s = -INFINITY;
        if (valid) {
            const int pg = tb[kp / page];
            if (pg < 0 || pg >= num_pages) {
                mb_set_error(err, pg < 0 ? MB_ERR_PAGE_MISSING : MB_ERR_PAGE_RANGE);
            } else {
                off = ((long long)pg * KV + kvh) * page + (kp % page);
                const T* kr = kpool + off * k_row;
                float a = 0.0f;
                for (int d = 0; d < HD; d++) a = fmaf(qs[warp][d], mb_load(kr + d), a);
                s = a * scale;
                if (softcap > 0.0f) s = softcap * tanhf(s / softcap);
            }
        }
        const float tmax = mb_warp_max(s);
        const float m_new = fmaxf(m, tmax);
        if (m_new == -INFINITY) continue;                      // only after a table error: nothing to add
        const float p = (off >= 0) ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);
        l = l * corr + mb_warp_sum(p);
#pragma unroll
        for (int i = 0; i < MAXHD / 32; i++) acc[i] *= corr;
        const int cnt = min(32, seen - base);
        for (int j = 0; j < cnt; j++) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const long long oj = __shfl_sync(0xffffffffu, off, j);
            if (oj < 0) continue;
            const T* vr = vpool + oj * v_row;
#pragma unroll
            for (int i = 0; i < MAXHD / 32; i++) {
                const int d = lane + 32 * i;
                if (d < HDV) acc[i] = fmaf(pj, mb_load(vr + d), acc[i]);
            }
        }
        m = m_new;
    }
    if (sinks) {                                                // one more term in the denominator, after every key
        const float sk = sinks[h], m_new = fmaxf(m, sk), corr = expf(m - m_new);
        l = l * corr + expf(sk - m_new);
#pragma unroll
        for (int i = 0; i < MAXHD / 32; i++) acc[i] *= corr;
    }
    float inv = l > 0.0f ? 1.0f / l : 0.0f;
    if (gate) inv /= 1.0f + expf(-mb_load(gate + (size_t)n * gate_stride + h));
    T* o = out + (size_t)n * H * HDV + (size_t)h * HDV;
#pragma unroll
    for (int i = 0; i < MAXHD / 32; i++) {
        const int d = lane + 32 * i;
        if (d < HDV) mb_store(o + d, acc[i] * inv);
    }
}

// The tiled form, float32, every key from position 0 on: a block is a run of tokens of one sequence (up to 64 / HB of them)
// times HB query heads of one kv head, 64 rows that read the same keys.  The plain form reads every key once for every
// row, one float at a time; here a tile of 32 keys and values is brought to shared memory once for the 64 rows, and the two
// products are register-tiled (4 rows x 4 keys, 4 rows x HDV / 8 values a thread), the next tile on its way meanwhile.
// The arithmetic of a row is the plain form's, operation by operation and in its order -- scores by fused multiply-adds in
// ascending channel, 32 keys to a step of the softmax counted from position 0, the weights met by the same tree, values added
// in ascending key --, so the two forms give the same bits and a prompt's logits do not depend on how it was cut.
// 509 tokens of 32 heads of 64 (8 kv heads): 1,338 us in the plain form, 123 here; 24 heads of 128: 1,824 and 190.
#define ST_ROWS 64
#define ST_KEYS 32
#define ST_THREADS 128
__device__ __forceinline__ void st_cp16(float* smem, const float* gmem, int size) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem), "r"(size));
}

// DG groups of 32 value channels: HDV <= 32 DG.  HD, HDV, k_row, v_row and q_stride multiples of 4, rows on 16-byte
// boundaries.  Thread (ty, tx): rows 4 ty .. 4 ty + 3, keys tx + 8 j, channels 4 tx .. of every group of 32: a row's eight
// threads are in one warp, so its softmax needs shuffles alone and its weights cross the warp through shared memory.
template <int DG>
__global__ void __launch_bounds__(ST_THREADS) attn_simple_tiled_kernel(
    const float* __restrict__ q, int q_stride, float* __restrict__ out, const int* __restrict__ positions,
    const int* __restrict__ tok_seq, const int* __restrict__ table, int max_blocks, const float* __restrict__ kpool,
    const float* __restrict__ vpool, int N, int H, int KV, int HD, int page, int num_pages, float scale, int* err, int HDV,
    int k_row, int v_row, float softcap, const float* __restrict__ sinks, const float* __restrict__ gate, int gate_stride,
    int HB, int tile) {
    constexpr int RS = ST_ROWS + 4, VS = 32 * DG;
    const int KS = HD + 4 + (HD & 4 ? 4 : 0);       // an odd number of quads at HD = 64, 128, ..: eight keys on eight banks of quads
    extern __shared__ __align__(16) float st_smem[];
    float* Qs = st_smem;                    // [HD][RS]
    float* Ps = Qs + HD * RS;               // [ST_KEYS][RS]: weights, key by key
    float* Ks = Ps + ST_KEYS * RS;          // [2][ST_KEYS][KS]
    float* Vs = Ks + 2 * ST_KEYS * KS;      // [2][ST_KEYS][VS]
    __shared__ long long s_off[2][ST_KEYS];         // where the rows of a tile's keys are, -1: nowhere
    const int G = H / KV, parts = (G + HB - 1) / HB;
    const int kvh = blockIdx.y / parts, h0 = kvh * G + blockIdx.y % parts * HB, nh = min(HB, (kvh + 1) * G - h0);
    // the tiles with the most keys (the last ones of a prompt) start first
    const int t0 = (gridDim.x - 1 - blockIdx.x) * tile, t1 = min(t0 + tile, N);
    const int lane = threadIdx.x & 31, tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    for (int first = t0, next; first < t1; first = next) {
        next = first + 1;
        while (next < t1 && simple_same(tok_seq, positions, next, first)) next++;
        const int count = next - first;
        if (count < SIMPLE_RUN) continue;                       // the plain form's
        const int pos0 = positions[first], rows = count * nh;   // row r: token first + r / nh, head h0 + r % nh
        const int seen_most = pos0 + count, tiles = (seen_most + ST_KEYS - 1) / ST_KEYS;
        const int* tb = table + (size_t)tok_seq[first] * max_blocks;
        auto place = [&](int t) {                               // by the first warp: the rows of tile t's keys
            const int kp = t * ST_KEYS + lane;
            long long off = -1;
            if (kp < seen_most) {
                const int pg = tb[kp / page];
                if (pg < 0 || pg >= num_pages) mb_set_error(err, pg < 0 ? MB_ERR_PAGE_MISSING : MB_ERR_PAGE_RANGE);
                else off = ((long long)pg * KV + kvh) * page + (kp % page);
            }
            s_off[t & 1][lane] = off;
        };
        auto fetch = [&](int t) {                               // sends for tile t; keys that are nowhere are zeros
            float* kd = Ks + (t & 1) * ST_KEYS * KS;
            float* vd = Vs + (t & 1) * ST_KEYS * VS;
            const int kq = HD / 4, vq = HDV / 4;
            for (int i = threadIdx.x; i < ST_KEYS * kq; i += ST_THREADS) {
                const int j = i / kq, d = (i - j * kq) * 4;
                const long long off = s_off[t & 1][j];
                st_cp16(kd + j * KS + d, kpool + (off < 0 ? 0 : off * k_row + d), off < 0 ? 0 : 16);
            }
            for (int i = threadIdx.x; i < ST_KEYS * vq; i += ST_THREADS) {
                const int j = i / vq, d = (i - j * vq) * 4;
                const long long off = s_off[t & 1][j];
                st_cp16(vd + j * VS + d, vpool + (off < 0 ? 0 : off * v_row + d), off < 0 ? 0 : 16);
            }
            asm volatile("cp.async.commit_group;\n" ::);
        };
        __syncthreads();                                        // the run before is done with everything
        if (threadIdx.x < 32) {
            place(0);
            if (tiles > 1) place(1);
        }
        for (int i = threadIdx.x; i < ST_ROWS * (HD / 4); i += ST_THREADS) {
            const int r = i % ST_ROWS, d = i / ST_ROWS * 4;
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r < rows) x = *reinterpret_cast<const float4*>(q + (size_t)(first + r / nh) * q_stride + (size_t)(h0 + r % nh) * HD + d);
            Qs[d * RS + r] = x.x; Qs[(d + 1) * RS + r] = x.y; Qs[(d + 2) * RS + r] = x.z; Qs[(d + 3) * RS + r] = x.w;
        }
        __syncthreads();
        fetch(0);
        float acc[4][4 * DG], m[4], l[4];
        int seen_row[4];                                        // keys that a row sees, from position 0 on
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = ty * 4 + i;
            seen_row[i] = r < rows ? pos0 + r / nh + 1 : 0;
            m[i] = -INFINITY;
            l[i] = 0.0f;
#pragma unroll
            for (int j = 0; j < 4 * DG; j++) acc[i][j] = 0.0f;
        }
        for (int t = 0; t < tiles; t++) {
            const float* kb = Ks + (t & 1) * ST_KEYS * KS;
            const float* vb = Vs + (t & 1) * ST_KEYS * VS;
            if (t + 1 < tiles) {
                fetch(t + 1);
                asm volatile("cp.async.wait_group 1;\n" ::);
            } else {
                asm volatile("cp.async.wait_group 0;\n" ::);
            }
            __syncthreads();
            const unsigned there = __ballot_sync(0xffffffffu, s_off[t & 1][lane] >= 0);        // keys whose page was found
            float s[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) s[i][j] = 0.0f;
#pragma unroll 2
            for (int d = 0; d < HD; d += 4) {
                float4 a[4], b[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    a[e] = *reinterpret_cast<const float4*>(Qs + (d + e) * RS + ty * 4);
                    b[e] = *reinterpret_cast<const float4*>(kb + (tx + 8 * e) * KS + d);
                }
#pragma unroll
                for (int e = 0; e < 4; e++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float k = e == 0 ? b[j].x : e == 1 ? b[j].y : e == 2 ? b[j].z : b[j].w;
                        s[0][j] = fmaf(a[e].x, k, s[0][j]);
                        s[1][j] = fmaf(a[e].y, k, s[1][j]);
                        s[2][j] = fmaf(a[e].z, k, s[2][j]);
                        s[3][j] = fmaf(a[e].w, k, s[3][j]);
                    }
            }
            unsigned mask[4];
            bool all = true;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int seen = seen_row[i] - t * ST_KEYS;     // keys of the tile that the row sees
                mask[i] = seen >= ST_KEYS ? there : seen > 0 ? there & ((1u << seen) - 1u) : 0u;
                float best = -INFINITY;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float x = s[i][j] * scale;
                    if (softcap > 0.0f) x = softcap * tanhf(x / softcap);
                    s[i][j] = (mask[i] >> (tx + 8 * j)) & 1 ? x : -INFINITY;
                    best = fmaxf(best, s[i][j]);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
                const float m_new = fmaxf(m[i], best);
                const bool add = m_new != -INFINITY && seen > 0;
                const float corr = add ? expf(m[i] - m_new) : 1.0f;
                float p[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    p[j] = add && ((mask[i] >> (tx + 8 * j)) & 1) ? expf(s[i][j] - m_new) : 0.0f;
                    s[i][j] = p[j];
                }
                // the tree of the plain form: keys 16 apart, 8 apart, then 4, 2 and 1
                float sum = (p[0] + p[2]) + (p[1] + p[3]);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (add) {
                    l[i] = l[i] * corr + sum;
                    m[i] = m_new;
                }
#pragma unroll
                for (int j = 0; j < 4 * DG; j++) acc[i][j] *= corr;
                if (ty * 4 + i < rows) all = all && mask[i] == 0xffffffffu;
            }
#pragma unroll
            for (int j = 0; j < 4; j++)
                *reinterpret_cast<float4*>(Ps + (tx + 8 * j) * RS + ty * 4) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
            __syncwarp();
            const bool whole = __all_sync(0xffffffffu, all);
#pragma unroll 4
            for (int j = 0; j < ST_KEYS; j++) {
                const float4 p4 = *reinterpret_cast<const float4*>(Ps + j * RS + ty * 4);
                const float pv[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                for (int g = 0; g < DG; g++) {
                    const float4 v4 = *reinterpret_cast<const float4*>(vb + j * VS + g * 32 + tx * 4);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (!whole && !((mask[i] >> j) & 1)) continue;      // a key the row does not see adds nothing, whatever it holds
                        acc[i][g * 4] = fmaf(pv[i], v4.x, acc[i][g * 4]);
                        acc[i][g * 4 + 1] = fmaf(pv[i], v4.y, acc[i][g * 4 + 1]);
                        acc[i][g * 4 + 2] = fmaf(pv[i], v4.z, acc[i][g * 4 + 2]);
                        acc[i][g * 4 + 3] = fmaf(pv[i], v4.w, acc[i][g * 4 + 3]);
                    }
                }
            }
            __syncthreads();                                    // this tile's buffers and places are free
            if (t + 2 < tiles) {
                if (threadIdx.x < 32) place(t + 2);
                __syncthreads();
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = ty * 4 + i;
            if (r >= rows) continue;
            const int n = first + r / nh, h = h0 + r % nh;
            float sum = l[i], corr = 1.0f;
            if (sinks) {
                const float sk = sinks[h], m_new = fmaxf(m[i], sk);
                corr = expf(m[i] - m_new);
                sum = sum * corr + expf(sk - m_new);
            }
            float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
            if (gate) inv /= 1.0f + expf(-gate[(size_t)n * gate_stride + h]);
            float* o = out + (size_t)n * H * HDV + (size_t)h * HDV;
#pragma unroll
            for (int g = 0; g < DG; g++) {
                const int d = g * 32 + tx * 4;
                float x[4] = {acc[i][g * 4], acc[i][g * 4 + 1], acc[i][g * 4 + 2], acc[i][g * 4 + 3]};
                if (d < HDV) {
                    if (sinks) { x[0] *= corr; x[1] *= corr; x[2] *= corr; x[3] *= corr; }
                    *reinterpret_cast<float4*>(o + d) = make_float4(x[0] * inv, x[1] * inv, x[2] * inv, x[3] * inv);
                }
            }
        }
    }
}

// -> the tile the tiled form cuts the step's tokens into, once it is launched; 0 when it does not take the call
static int attn_simple_tiled_launch(const float* q, int q_stride, float* out, const int* positions, const int* tok_seq,
                                    const int* table, int max_blocks, const float* kpool, const float* vpool, int N, int H, int KV,
                                    int HD, int page, int num_pages, int window, float scale, int* err, cudaStream_t st, int HDV,
                                    int k_row, int v_row, float softcap, const float* sinks, const float* gate, int gate_stride,
                                    int* status) {
    // Windows are the plain form's: its steps of 32 keys are counted from a row's own first key there.  Seven tiles of rows
    // are the least that pays: 70 tokens of 7 heads 152 us plain, 76 tiled; 65 of 4 heads 76 and 119; 16 of 32 heads 19 and 22.
    const uintptr_t ptrs = (uintptr_t)q | (uintptr_t)out | (uintptr_t)kpool | (uintptr_t)vpool;
    if (window > 0 || N < 32 || (long long)N * H < 7 * ST_ROWS || HD > 256 || HDV > 256 || ((HD | HDV | k_row | v_row | q_stride) & 3) ||
        (ptrs & 15))
        return 0;
    const int G = H / KV, HB = G < 4 ? G : 4, tile = ST_ROWS / HB, parts = (G + HB - 1) / HB;
    if ((long long)KV * parts > 65535) return 0;
    const int DG = HDV <= 64 ? 2 : HDV <= 128 ? 4 : 8;
    const size_t smem = ((size_t)HD * (ST_ROWS + 4) + ST_KEYS * (ST_ROWS + 4) + 2 * ST_KEYS * (HD + 4 + (HD & 4 ? 4 : 0)) +
                         2 * ST_KEYS * 32 * DG) * sizeof(float);
    const dim3 grid((N + tile - 1) / tile, KV * parts);
#define ST_CASE(D)                                                                                                         \
    if (DG == D) {                                                                                                         \
        static bool configured = false;                                                                                    \
        if (!configured) {                                                                                                 \
            cudaError_t e = cudaFuncSetAttribute(attn_simple_tiled_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                 224 * 1024);                                                              \
            if (e != cudaSuccess) { *status = (int)e; return 0; }                                                          \
            configured = true;                                                                                             \
        }                                                                                                                  \
        attn_simple_tiled_kernel<D><<<grid, ST_THREADS, smem, st>>>(q, q_stride, out, positions, tok_seq, table, max_blocks, \
            kpool, vpool, N, H, KV, HD, page, num_pages, scale, err, HDV, k_row, v_row, softcap, sinks, gate, gate_stride, \
            HB, tile);                                                                                                     \
    }
    ST_CASE(2) ST_CASE(4) ST_CASE(8)
#undef ST_CASE
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { *status = (int)e; return 0; }
    return tile;
}

template <typename T>
static int attn_simple_launch(const void* q, int q_stride, void* out, const int* positions, const int* tok_seq,
                              const int* table, int max_blocks, const void* kpool, const void* vpool, int N, int H,
                              int KV, int HD, int page, int num_pages, int window, float scale, int* err,
                              cudaStream_t st, int HDV = 0, int k_row = 0, int v_row = 0, float softcap = 0.0f,
                              const float* sinks = nullptr, const void* gate_ = nullptr, int gate_stride = 0,
                              int keep = 0) {
    if (N == 0) return 0;
    if (HDV == 0) HDV = HD;
    if (k_row == 0) k_row = HD;
    if (v_row == 0) v_row = HDV;
    const T* gate = (const T*)gate_;
    const int widest = HD > HDV ? HD : HDV;
    if (widest > SIMPLE_MAX_HD || keep < 0 || HD < 1 || HDV < 1 || KV < 1 || H % KV || k_row < HD || v_row < HDV) return -2;
    const long long items = (long long)N * H;
    int tile = 0, status = 0;
    if (sizeof(T) == 4 && keep == 0)
        tile = attn_simple_tiled_launch((const float*)q, q_stride, (float*)out, positions, tok_seq, table, max_blocks,
                                        (const float*)kpool, (const float*)vpool, N, H, KV, HD, page, num_pages, window, scale,
                                        err, st, HDV, k_row, v_row, softcap, sinks, (const float*)gate_, gate_stride, &status);
    if (status) return status;
    if (widest <= 256)
        attn_simple_kernel<T, 256><<<(unsigned)((items + WARPS - 1) / WARPS), WARPS * 32, 0, st>>>(
            (const T*)q, q_stride, (T*)out, positions, tok_seq, table, max_blocks, (const T*)kpool, (const T*)vpool, N, H,
            KV, HD, page, num_pages, window, scale, err, HDV, k_row, v_row, softcap, sinks, gate, gate_stride, keep, tile);
    else if (widest <= 512)
        attn_simple_kernel<T, 512><<<(unsigned)((items + WARPS - 1) / WARPS), WARPS * 32, 0, st>>>(
            (const T*)q, q_stride, (T*)out, positions, tok_seq, table, max_blocks, (const T*)kpool, (const T*)vpool, N, H,
            KV, HD, page, num_pages, window, scale, err, HDV, k_row, v_row, softcap, sinks, gate, gate_stride, keep, tile);
    else
        attn_simple_kernel<T, SIMPLE_MAX_HD><<<(unsigned)((items + WARPS - 1) / WARPS), WARPS * 32, 0, st>>>(
            (const T*)q, q_stride, (T*)out, positions, tok_seq, table, max_blocks, (const T*)kpool, (const T*)vpool, N, H,
            KV, HD, page, num_pages, window, scale, err, HDV, k_row, v_row, softcap, sinks, gate, gate_stride, keep, tile);
    MB_LAUNCH_CHECK();
    return 0;
}

MB_API int mb_attn_simple_f32(const void* q, int q_stride, void* out, const int* positions, const int* tok_seq,
                              const int* table, int max_blocks, const void* kpool, const void* vpool, int N, int H,
                              int KV, int HD, int page, int num_pages, int window, float scale, int* err,
                              cudaStream_t st) {
    return attn_simple_launch<float>(q, q_stride, out, positions, tok_seq, table, max_blocks, kpool, vpool, N, H, KV,
                                     HD, page, num_pages, window, scale, err, st);
}
MB_API int mb_attn_simple_bf16(const void* q, int q_stride, void* out, const int* positions, const int* tok_seq,
                               const int* table, int max_blocks, const void* kpool, const void* vpool, int N, int H,
                               int KV, int HD, int page, int num_pages, int window, float scale, int* err,
                               cudaStream_t st) {
    return attn_simple_launch<__nv_bfloat16>(q, q_stride, out, positions, tok_seq, table, max_blocks, kpool, vpool, N,
                                             H, KV, HD, page, num_pages, window, scale, err, st);
}

// the general form: keys of HD and values of HDV, rows k_row and v_row apart, capped scores, sinks, a gate per head
MB_API int mb_attn_simple_ext_f32(const void* q, int q_stride, void* out, const int* positions, const int* tok_seq,
                                  const int* table, int max_blocks, const void* kpool, const void* vpool, int N, int H,
                                  int KV, int HD, int HDV, int k_row, int v_row, int page, int num_pages, int window,
                                  float scale, float softcap, const float* sinks, const void* gate, int gate_stride, int keep,
                                  int* err, cudaStream_t st) {
    return attn_simple_launch<float>(q, q_stride, out, positions, tok_seq, table, max_blocks, kpool, vpool, N, H, KV,
                                     HD, page, num_pages, window, scale, err, st, HDV, k_row, v_row, softcap, sinks, gate,
                                     gate_stride, keep);
}
MB_API int mb_attn_simple_ext_bf16(const void* q, int q_stride, void* out, const int* positions, const int* tok_seq,
                                   const int* table, int max_blocks, const void* kpool, const void* vpool, int N, int H,
                                   int KV, int HD, int HDV, int k_row, int v_row, int page, int num_pages, int window,
                                   float scale, float softcap, const float* sinks, const void* gate, int gate_stride, int keep,
                                   int* err, cudaStream_t st) {
    return attn_simple_launch<__nv_bfloat16>(q, q_stride, out, positions, tok_seq, table, max_blocks, kpool, vpool, N,
                                             H, KV, HD, page, num_pages, window, scale, err, st, HDV, k_row, v_row, softcap,
                                             sinks, gate, gate_stride, keep);
}
