// The recurrences of the linear-attention layers over long stretches of tokens, 32 tokens (a chunk) at a time:
//
//     MODE 0 (delta rule)       S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q     g (N, H, dim)
//     MODE 1 (gated, channels)  S <- diag(g) S + k v^T;  o = S^T q                                     g (N, H, dim)
//     MODE 2 (gated, heads)     S <- g S + k v^T;  o = S^T q                                           g (N, H)
//     MODE 3 (wkv)              o = S^T q + b v;  S <- diag(g) S + k v^T                               g as in 1, b (N, H)
//     MODE 4 (fixed decay)      S <- g S + k v^T;  o = S^T q                                           g (H)
//
// With S0 the state before a chunk, P_t the product of the chunk's decays up to token t, and D_ts = the product of those
// after s up to t, the chunk is four small matrix products (elementwise products with decays are per key channel):
//
//     O = (q_t P_t) S0 + A U,   A_ts = sum_i q_ti k_si D_ts,i (s <= t)      S = P_32 S0 + sum_s (k_s D_32,s) u_s^T
//     U = V, and for the delta rule U = (I + B)^-1 diag(beta) (V - (k_t P_t) S0),  B_ts = beta_t sum_i k_ti k_si D_ts,i (s < t)
//
// (wkv reads S before the token joins: its P and D stop one token earlier and A_tt = b_t.)  Every D is a running product
// of decays, never a quotient, so a decay near zero costs no accuracy; all of it is float32.
//
//   chunk_prep   a block per chunk and head, all of them side by side: what does not depend on the state -- the scaled
//                rows, A, and for the delta rule T = (I + B)^-1 diag(beta) -- goes to a record in scratch.
//   chunk_walk   a block per sequence, head and 16 value columns walks the sequence's records in order with its part of
//                S in registers.  Records come by bulk copy into two buffers of shared memory.
//
// A sequence of fewer than `shortest` tokens (32 at least) is passed over by both and left to the scan, which follows: a
// record of one token costs as much as one of 32 (16 sequences of one token beside one of 64: 103 us against 46 by the scan).
//
// What bounds the walk is the shared-memory pipe: a lane takes one float a cycle, a thread's 4 x 4 tile needs eight for 16
// multiply-adds, and the pipe is busy for 80 % of the cycles (delta rule, 16 heads of 128 x 128, 2,048 tokens: prep 46, walk
// 182 us).  The token-by-token scan, which reads every q, k, g for every column pair and pays shuffles for every token,
// takes 646 us there; with decays per channel (24 heads) 577 against 231, per head (48 of 128 x 64) 507 against 247, wkv 506
// against 157, fixed decays (two passes over segments) 413 against 153.
#include <type_traits>
#include "tcgen05.cuh"

#define LC_C 32                 // tokens of a chunk
#define LC_COLS 16              // value columns of a walking block
#define LC_STAGES 2             // records in shared memory (3 measured the same where one block has an SM to itself, and cost
                                // the second block of an SM where it has not: 172 against 240 us on 24 heads)
#define LC_MIN 32               // the least a sequence can be asked to have
#define LC_RED 20               // floats a row of the partial sums takes (16 used; the padding keeps banks apart)

// ---- pairs of floats: one issue slot, two results, each rounded as the single one is
__device__ __forceinline__ uint64_t lc_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void lc_unpack(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t lc_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t lc_mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The record of a chunk and head, in floats: rows that meet the state, channel by channel ([i][q 0..31 | k 0..31], without
// the k half unless MODE is 0); then keys [t][i], A transposed [s][t], T transposed [s][t] (MODE 0), and P_32 [i].
template <int DP, int MODE>
struct Rec {
    static constexpr int ROWS = MODE == 0 ? 2 * LC_C : LC_C;
    static constexpr int FIRST = DP * ROWS;
    static constexpr int KEYS = 0, A = LC_C * DP, T = A + LC_C * LC_C, P = T + (MODE == 0 ? LC_C * LC_C : 0);
    static constexpr int SECOND = P + DP;
    static constexpr int ALL = FIRST + SECOND;
};

// chunks of a sequence
__device__ __forceinline__ int lc_chunks(int len, int shortest) { return len < shortest ? 0 : (len + LC_C - 1) / LC_C; }

// the sequence a slot (number of a chunk through all sequences in order) belongs to -> false beyond the last one
__device__ __forceinline__ bool lc_find(int slot, int S, const int* __restrict__ q_len, int shortest, int& s, int& c) {
    int base = 0;
    for (s = 0; s < S; s++) {
        const int n = lc_chunks(q_len[s], shortest);
        if (slot < base + n) { c = slot - base; return true; }
        base += n;
    }
    return false;
}

// grid (slots, H), 128 threads.
template <int DP, int MODE>
__global__ void __launch_bounds__(128) chunk_prep_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                         const float* __restrict__ g, const float* __restrict__ beta,
                                                         float* __restrict__ scratch, const int* __restrict__ q_start,
                                                         const int* __restrict__ q_len, int S, int H, int G, int dim,
                                                         int shortest) {
    typedef Rec<DP, MODE> R;
    constexpr bool HEAD = MODE == 2 || MODE == 4;                // one decay per head
    constexpr int VEC = DP / 32;                                 // channels of a lane
    extern __shared__ __align__(16) float sm[];
    float* sq = sm;                                              // [32][DP]
    float* sk = sq + LC_C * DP;
    float* sg = sk + LC_C * DP;                                  // [32][DP]; HEAD: [s][t] products of decays after s up to t
    float* sA = sg + (HEAD ? LC_C * LC_C : LC_C * DP);           // [s][t]
    float* sB = sA + LC_C * LC_C;                                // [t][s], MODE 0
    float* sb = sB + (MODE == 0 ? LC_C * LC_C : 0);              // [32] beta, b, or a head's decays
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, j = h / (H / G);
    int s_, c_;
    if (!lc_find(blockIdx.x, S, q_len, shortest, s_, c_)) return;
    const int n0 = q_start[s_] + c_ * LC_C, nb = min(LC_C, q_len[s_] - c_ * LC_C);
    float* rec = scratch + ((size_t)blockIdx.x * H + h) * R::ALL;
    auto fetch = [](float* d, const float* x) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(d)), "l"(x));
    };
#pragma unroll 4
    for (int idx = tid; idx < LC_C * (DP / 4); idx += 128) {
        const int t = idx / (DP / 4), i = (idx - t * (DP / 4)) * 4;
        if (t < nb && i < dim) {
            const size_t n = (size_t)(n0 + t);
            fetch(sq + t * DP + i, q + (n * G + j) * dim + i);
            fetch(sk + t * DP + i, k + (n * G + j) * dim + i);
            if (!HEAD) fetch(sg + t * DP + i, g + (n * H + h) * dim + i);
        } else {
            *reinterpret_cast<float4*>(sq + t * DP + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            *reinterpret_cast<float4*>(sk + t * DP + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (!HEAD) *reinterpret_cast<float4*>(sg + t * DP + i) = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        }
    }
    if (MODE != 1 && tid < LC_C) {
        float x = HEAD ? 1.0f : 0.0f;
        if (tid < nb) x = MODE == 4 ? g[h] : MODE == 2 ? g[(size_t)(n0 + tid) * H + h] : beta[(size_t)(n0 + tid) * H + h];
        sb[tid] = x;
    }
    for (int idx = tid; idx < LC_C * LC_C; idx += 128) { sA[idx] = 0.0f; if (MODE == 0) sB[idx] = 0.0f; }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if (HEAD) {
        if (tid < LC_C) {                                        // thread s: its products, token by token
            float p = 1.0f;
            for (int t = 0; t < LC_C; t++) {
                if (t > tid) p *= sb[t];
                sg[tid * LC_C + t] = p;
            }
        }
        __syncthreads();
    }

    // A and B: a warp takes four keys at a time (groups w and 7 - w: equal work) and walks the tokens from them on, the
    // keys decaying as it goes; a lane sums its channels, in pairs, and eight tokens' sums are met across the lanes at once
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        const int s0 = 4 * (half ? 7 - warp : warp);
        uint64_t kp[4][VEC / 2];
#pragma unroll
        for (int x = 0; x < 4; x++)
#pragma unroll
            for (int e = 0; e < VEC / 2; e++)
                kp[x][e] = *reinterpret_cast<const uint64_t*>(sk + (s0 + x) * DP + lane * VEC + 2 * e);
#pragma unroll 1
        for (int tb = s0 & ~7; tb < nb; tb += 8) {
            float va[32], vb[MODE == 0 ? 32 : 1];
            auto tokens = [&](auto diagonal) {
                constexpr bool DIAG = decltype(diagonal)::value;                // the keys' own tokens are among the eight
#pragma unroll
                for (int jj = 0; jj < 8; jj++) {
                    const int t = tb + jj;
                    uint64_t qv[VEC / 2], kv[VEC / 2], gv[VEC / 2];
#pragma unroll
                    for (int e = 0; e < VEC / 2; e++) {
                        qv[e] = *reinterpret_cast<const uint64_t*>(sq + t * DP + lane * VEC + 2 * e);
                        if (MODE == 0) kv[e] = *reinterpret_cast<const uint64_t*>(sk + t * DP + lane * VEC + 2 * e);
                        if (!HEAD) gv[e] = *reinterpret_cast<const uint64_t*>(sg + t * DP + lane * VEC + 2 * e);
                    }
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        const bool later = !DIAG || t > s0 + x;
                        if (!HEAD && MODE != 3 && later)
#pragma unroll
                            for (int e = 0; e < VEC / 2; e++) kp[x][e] = lc_mul(kp[x][e], gv[e]);
                        uint64_t a = lc_mul(qv[0], kp[x][0]), b = MODE == 0 ? lc_mul(kv[0], kp[x][0]) : 0;
#pragma unroll
                        for (int e = 1; e < VEC / 2; e++) {
                            a = lc_fma(qv[e], kp[x][e], a);
                            if (MODE == 0) b = lc_fma(kv[e], kp[x][e], b);
                        }
                        if (MODE == 3 && later)
#pragma unroll
                            for (int e = 0; e < VEC / 2; e++) kp[x][e] = lc_mul(kp[x][e], gv[e]);
                        float lo, hi;
                        lc_unpack(a, lo, hi);
                        va[jj * 4 + x] = !DIAG || (MODE == 3 ? later : t >= s0 + x) ? lo + hi : 0.0f;
                        if (MODE == 0) {
                            lc_unpack(b, lo, hi);
                            vb[jj * 4 + x] = later ? lo + hi : 0.0f;
                        }
                    }
                }
            };
            if (tb < s0 + 4) tokens(std::true_type());
            else tokens(std::false_type());
            // sums over the lanes, 32 values at once: lane L ends with value L
#pragma unroll
            for (int m = 16; m > 0; m >>= 1)
#pragma unroll
                for (int i = 0; i < m; i++) {
                    const bool up = lane & m;
                    const float keep = up ? va[i + m] : va[i], send = up ? va[i] : va[i + m];
                    va[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                    if (MODE == 0) {
                        const float keep2 = up ? vb[i + m] : vb[i], send2 = up ? vb[i] : vb[i + m];
                        vb[i] = keep2 + __shfl_xor_sync(0xffffffffu, send2, m);
                    }
                }
            const int t = tb + (lane >> 2), s = s0 + (lane & 3);
            float a = va[0];
            if (HEAD) a *= sg[s * LC_C + t];
            if (MODE == 3 && t == s) a = sb[t];
            sA[s * LC_C + t] = a;
            if (MODE == 0) sB[t * LC_C + s] = vb[0] * sb[t];
        }
    }

    // the rows that meet the state, the keys as the chunk's end sees them, and the decay of the whole chunk: a thread per channel
    if (tid < DP) {
        float p = 1.0f;
        float4* dst = reinterpret_cast<float4*>(rec + (size_t)tid * R::ROWS);
#pragma unroll
        for (int t4 = 0; t4 < LC_C / 4; t4++) {
            float a[4], b[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = t4 * 4 + e;
                const float d = HEAD ? sb[t] : sg[t * DP + tid];
                if (MODE == 3) { a[e] = sq[t * DP + tid] * p; p *= d; }
                else { p *= d; a[e] = sq[t * DP + tid] * p; }
                if (MODE == 0) b[e] = sk[t * DP + tid] * p;
            }
            dst[t4] = make_float4(a[0], a[1], a[2], a[3]);
            if (MODE == 0) dst[LC_C / 4 + t4] = make_float4(b[0], b[1], b[2], b[3]);
        }
        rec[R::FIRST + R::P + tid] = p;
        float r = 1.0f;
#pragma unroll 8
        for (int t = LC_C - 1; t >= 0; t--) {
            rec[R::FIRST + R::KEYS + t * DP + tid] = sk[t * DP + tid] * r;
            r *= HEAD ? sb[t] : sg[t * DP + tid];
        }
    }
    __syncthreads();
    for (int idx = tid; idx < LC_C * LC_C / 4; idx += 128)
        reinterpret_cast<float4*>(rec + R::FIRST + R::A)[idx] = reinterpret_cast<const float4*>(sA)[idx];
    if (MODE == 0 && warp == 0) {
        // (I + B)^-1 by forward substitution, a lane per column; then times beta of the column's token
        float m[LC_C];
#pragma unroll
        for (int t = 0; t < LC_C; t++) {
            float acc[4] = {t == lane ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int s = 0; s < t; s++) acc[s & 3] = fmaf(-sB[t * LC_C + s], m[s], acc[s & 3]);
            m[t] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        }
        const float bt = sb[lane];
        float4* dst = reinterpret_cast<float4*>(rec + R::FIRST + R::T + lane * LC_C);
#pragma unroll
        for (int t = 0; t < LC_C; t += 4) dst[t / 4] = make_float4(m[t] * bt, m[t + 1] * bt, m[t + 2] * bt, m[t + 3] * bt);
    }
}

__device__ __forceinline__ void lc_fetch(float* dst, const float* src, uint32_t bytes, uint32_t bar) {
    mbar_expect_tx(bar, bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// barriers between the two halves of a walking block: one half arrives, the other waits
// (their numbers are constants of the code, so that the block holds nine barriers and not all sixteen)
enum { LC_BAR_A = 1, LC_BAR_B = 2, LC_S_READY = 3, LC_U_READY = 5, LC_S_READ = 7 };      // the last three: + parity of the chunk
template <int ID> __device__ __forceinline__ void lc_half() { asm volatile("bar.sync %0, 128;\n" ::"n"(ID) : "memory"); }
template <int ID> __device__ __forceinline__ void lc_wait(int parity) {
    if (parity) asm volatile("bar.sync %0, 256;\n" ::"n"(ID + 1) : "memory");
    else asm volatile("bar.sync %0, 256;\n" ::"n"(ID) : "memory");
}
template <int ID> __device__ __forceinline__ void lc_arrive(int parity) {
    if (parity) asm volatile("bar.arrive %0, 256;\n" ::"n"(ID + 1) : "memory");
    else asm volatile("bar.arrive %0, 256;\n" ::"n"(ID) : "memory");
}

// 32 rows of a record (channel by channel, `rows` floats a channel) times S over a warp's channels: 4 rows, in pairs, and 4
// columns a thread; the partial sums go to red (32, LC_RED)
template <int SLAB>
__device__ __forceinline__ void lc_rows(const float* fa, int rows, const float* fs, float* red, int rg, int cg) {
    uint64_t acc[2][4];
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
        for (int x = 0; x < 4; x++) acc[p][x] = lc_pack(0.0f, 0.0f);
#pragma unroll 16
    for (int kk = 0; kk < SLAB; kk++) {
        const float4 s = *reinterpret_cast<const float4*>(fs + kk * LC_COLS + cg * 4);
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(fa + kk * rows + rg * 4);
        const uint64_t s0 = lc_pack(s.x, s.x), s1 = lc_pack(s.y, s.y), s2 = lc_pack(s.z, s.z), s3 = lc_pack(s.w, s.w);
        acc[0][0] = lc_fma(a.x, s0, acc[0][0]);
        acc[0][1] = lc_fma(a.x, s1, acc[0][1]);
        acc[0][2] = lc_fma(a.x, s2, acc[0][2]);
        acc[0][3] = lc_fma(a.x, s3, acc[0][3]);
        acc[1][0] = lc_fma(a.y, s0, acc[1][0]);
        acc[1][1] = lc_fma(a.y, s1, acc[1][1]);
        acc[1][2] = lc_fma(a.y, s2, acc[1][2]);
        acc[1][3] = lc_fma(a.y, s3, acc[1][3]);
    }
#pragma unroll
    for (int p = 0; p < 2; p++) {
        float x[4], y[4];
#pragma unroll
        for (int e = 0; e < 4; e++) lc_unpack(acc[p][e], x[e], y[e]);
        float* d = red + (rg * 4 + 2 * p) * LC_RED + cg * 4;
        *reinterpret_cast<float4*>(d) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4*>(d + LC_RED) = make_float4(y[0], y[1], y[2], y[3]);
    }
}
__device__ __forceinline__ float4 lc_sum(const float* red, int row, int cg) {
    float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int w = 0; w < 4; w++) {
        const float4 x = *reinterpret_cast<const float4*>(red + (w * LC_C + row) * LC_RED + cg * 4);
        y.x += x.x; y.y += x.y; y.z += x.z; y.w += x.w;
    }
    return y;
}
// out += sum over tokens s <= t of m[s][t] r[s] (m lower triangular; nothing of a later token is touched: no 0 * inf)
__device__ __forceinline__ void lc_lower(float4& out, const float* m, const float* r, int t, int last, int cg) {
#pragma unroll 8
    for (int s = 0; s < last; s++) {
        const float w = m[s * LC_C + t];
        const float4 x = *reinterpret_cast<const float4*>(r + s * LC_COLS + cg * 4);
        if (s <= t) {
            out.x = fmaf(w, x.x, out.x); out.y = fmaf(w, x.y, out.y); out.z = fmaf(w, x.z, out.z); out.w = fmaf(w, x.w, out.w);
        }
    }
}

// grid (column tiles, H, S), 256 threads in two halves.  Half A keeps S (warp w: channels w DP/4 ..+DP/4, all 16 columns),
// makes U and takes it in; half B makes the outputs from the S that A left in shared memory, so that what is not on the
// chain from one state to the next runs beside it.  Records go through two buffers.  TRANS: a head's state is stored
// (vdim, dim).
template <int DP, int MODE, bool TRANS>
__global__ void __launch_bounds__(256) chunk_walk_kernel(const float* __restrict__ v, float* __restrict__ o,
                                                         float* __restrict__ state, long long state_stride,
                                                         const float* __restrict__ scratch, const int* __restrict__ q_start,
                                                         const int* __restrict__ q_len, const int* __restrict__ state_slot,
                                                         int H, int dim, int vdim, int shortest, int* err) {
    typedef Rec<DP, MODE> R;
    constexpr int SLAB = DP / 4, CH = DP / 32;
    extern __shared__ __align__(128) float sm[];
    float* sS = sm + LC_STAGES * R::ALL;                                // [2][DP][16]
    float* sU = sS + 2 * DP * LC_COLS;                           // [2][32][16]
    float* redB = sU + 2 * LC_C * LC_COLS;                       // [4][32][LC_RED]
    float* redA = redB + 4 * LC_C * LC_RED;                      // MODE 0
    float* sR = redA + 4 * LC_C * LC_RED;                        // [32][16], MODE 0
    __shared__ __align__(8) uint64_t bars[LC_STAGES];
    const int tid = threadIdx.x & 127, warp = tid >> 5, lane = tid & 31, rg = lane >> 2, cg = lane & 3;
    const int col0 = blockIdx.x * LC_COLS, h = blockIdx.y, sq = blockIdx.z;
    const int a0 = q_start[sq], len = q_len[sq], chunks = lc_chunks(len, shortest);
    if (chunks == 0) return;
    int slot = 0;
    for (int r = 0; r < sq; r++) slot += lc_chunks(q_len[r], shortest);
    const float* rec = scratch + ((size_t)slot * H + h) * R::ALL;
    const size_t next = (size_t)H * R::ALL;
    const uint32_t bar0 = smem_u32(bars);
    if (threadIdx.x == 0) {
        for (int c = 0; c < LC_STAGES; c++) mbar_init(bar0 + 8 * c, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 128)
        for (int c = 0; c < min(LC_STAGES, chunks); c++) lc_fetch(sm + c * R::ALL, rec + c * next, R::ALL * 4, bar0 + 8 * c);
    // token (of a chunk) and columns this thread reads v for, or writes o for
    const int tt = tid >> 2, c0 = col0 + cg * 4, last = warp * 8 + 8;
    const bool colin = c0 < vdim;                                // vdim is a multiple of 4
    const size_t vat = ((size_t)(a0 + tt) * H + h) * vdim + c0, vnext = (size_t)LC_C * H * vdim;
    bool bad = false;
    if (threadIdx.x < 128) {
        // the state: CH channels from i0 on, four columns, channels in pairs
        float* Sg = state + (size_t)state_slot[sq] * state_stride + (size_t)h * dim * vdim;
        const int i0 = warp * SLAB + rg * CH;
        auto at = [&](int i, int c) { return TRANS ? (size_t)c * dim + i : (size_t)i * vdim + c; };
        uint64_t st[CH / 2][4];
#pragma unroll
        for (int p = 0; p < CH / 2; p++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const bool in = c0 + c < vdim && i0 + 2 * p < dim;   // dim is a multiple of 4: both channels are in, or neither
                st[p][c] = in ? lc_pack(Sg[at(i0 + 2 * p, c0 + c)], Sg[at(i0 + 2 * p + 1, c0 + c)]) : lc_pack(0.0f, 0.0f);
            }
        auto leave = [&](int buf) {
#pragma unroll
            for (int p = 0; p < CH / 2; p++) {
                float x[4], y[4];
#pragma unroll
                for (int c = 0; c < 4; c++) lc_unpack(st[p][c], x[c], y[c]);
                float* d = sS + (size_t)(buf * DP + i0 + 2 * p) * LC_COLS + cg * 4;
                *reinterpret_cast<float4*>(d) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4*>(d + LC_COLS) = make_float4(y[0], y[1], y[2], y[3]);
            }
        };
        leave(0);
        lc_arrive<LC_S_READY>(0);
        float4 vv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (colin && tt < len) vv = *reinterpret_cast<const float4*>(v + vat);
        for (int c = 0; c < chunks; c++) {
            const int buf = c & 1, at_stage = c % LC_STAGES;
            const float* record = sm + at_stage * R::ALL;
            const float* second = record + R::FIRST;
            const float4 vnow = vv;
            vv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (colin && (c + 1) * LC_C + tt < len) vv = *reinterpret_cast<const float4*>(v + vat + (size_t)(c + 1) * vnext);
            if (!bad) bad = !mbar_wait(bar0 + 8 * at_stage, (c / LC_STAGES) & 1, err);
            float4 u = vnow;
            if (MODE == 0) {
                __syncwarp();                                    // this warp's channels of S are this warp's own stores
                lc_rows<SLAB>(record + warp * SLAB * R::ROWS + LC_C, R::ROWS,
                              sS + (size_t)(buf * DP + warp * SLAB) * LC_COLS, redA + warp * LC_C * LC_RED, rg, cg);
                lc_half<LC_BAR_A>();
                const float4 ks = lc_sum(redA, tt, cg);
                *reinterpret_cast<float4*>(sR + tt * LC_COLS + cg * 4) =
                    make_float4(vnow.x - ks.x, vnow.y - ks.y, vnow.z - ks.z, vnow.w - ks.w);
                lc_half<LC_BAR_A>();
                u = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                lc_lower(u, second + R::T, sR, tt, last, cg);
            }
            // B has read the state before last and finished with the U of two chunks ago
            if (c > 0) lc_wait<LC_S_READ>(buf ^ 1);
            *reinterpret_cast<float4*>(sU + (buf * LC_C + tt) * LC_COLS + cg * 4) = u;
            lc_half<LC_BAR_A>();
            lc_arrive<LC_U_READY>(buf);
            // the state takes the chunk in
#pragma unroll
            for (int p = 0; p < CH / 2; p++) {
                const uint64_t d = *reinterpret_cast<const uint64_t*>(second + R::P + i0 + 2 * p);
#pragma unroll
                for (int x = 0; x < 4; x++) st[p][x] = lc_mul(st[p][x], d);
            }
            const float* keys = second + R::KEYS + i0;
            const float* us = sU + buf * LC_C * LC_COLS + cg * 4;
#pragma unroll 16
            for (int t = 0; t < LC_C; t++) {
                const float4 x = *reinterpret_cast<const float4*>(us + t * LC_COLS);
                const uint64_t u0 = lc_pack(x.x, x.x), u1 = lc_pack(x.y, x.y), u2 = lc_pack(x.z, x.z), u3 = lc_pack(x.w, x.w);
                uint64_t a[CH / 2];
                if (CH == 4) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(keys + t * DP);
                    a[0] = w.x;
                    a[CH / 2 - 1] = w.y;
                } else {
                    a[0] = *reinterpret_cast<const uint64_t*>(keys + t * DP);
                }
#pragma unroll
                for (int p = 0; p < CH / 2; p++) {
                    st[p][0] = lc_fma(a[p], u0, st[p][0]);
                    st[p][1] = lc_fma(a[p], u1, st[p][1]);
                    st[p][2] = lc_fma(a[p], u2, st[p][2]);
                    st[p][3] = lc_fma(a[p], u3, st[p][3]);
                }
            }
            if (c + 1 < chunks) {
                leave(buf ^ 1);
                lc_arrive<LC_S_READY>(buf ^ 1);
            }
        }
        lc_wait<LC_S_READ>((chunks - 1) & 1);             // takes up B's last arrival
#pragma unroll
        for (int p = 0; p < CH / 2; p++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                float lo, hi;
                lc_unpack(st[p][x], lo, hi);
                if (c0 + x < vdim && i0 + 2 * p < dim) {
                    Sg[at(i0 + 2 * p, c0 + x)] = lo;
                    Sg[at(i0 + 2 * p + 1, c0 + x)] = hi;
                }
            }
    } else {
        int sent = min(LC_STAGES, chunks);                       // records sent for (thread 128)
        for (int c = 0; c < chunks; c++) {
            const int buf = c & 1, at_stage = c % LC_STAGES;
            const float* record = sm + at_stage * R::ALL;
            const float* second = record + R::FIRST;
            // A has taken the chunk before this one in, and all of B is done with it: its record's buffer is free
            lc_wait<LC_S_READY>(buf);
            if (threadIdx.x == 128 && c > 0 && c - 1 + LC_STAGES < chunks && !bad) {
                const int free = (c - 1) % LC_STAGES;
                lc_fetch(sm + free * R::ALL, rec + (size_t)(c - 1 + LC_STAGES) * next, R::ALL * 4, bar0 + 8 * free);
                sent = c + LC_STAGES;
            }
            if (!bad) bad = !mbar_wait(bar0 + 8 * at_stage, (c / LC_STAGES) & 1, err);
            lc_rows<SLAB>(record + warp * SLAB * R::ROWS, R::ROWS, sS + (size_t)(buf * DP + warp * SLAB) * LC_COLS,
                          redB + warp * LC_C * LC_RED, rg, cg);
            lc_arrive<LC_S_READ>(buf);
            lc_half<LC_BAR_B>();
            float4 out = lc_sum(redB, tt, cg);
            lc_wait<LC_U_READY>(buf);
            lc_lower(out, second + R::A, sU + buf * LC_C * LC_COLS, tt, last, cg);
            if (colin && c * LC_C + tt < len) *reinterpret_cast<float4*>(o + vat + (size_t)c * vnext) = out;
        }
        // a wait ran out: the block does not leave while copies into its shared memory may still be on their way
        if (threadIdx.x == 128 && bad)
            for (int r = max(0, sent - LC_STAGES); r < sent; r++) mbar_wait(bar0 + 8 * (r % LC_STAGES), (r / LC_STAGES) & 1, err);
    }
}

template <int DP, int MODE>
static int lc_launch(const float* q, const float* k, const float* v, const float* g, const float* beta, float* o, float* state,
                     long long state_stride, const int* q_start, const int* q_len, const int* state_slot, int S, int N, int H,
                     int G, int dim, int vdim, int shortest, float* scratch, long long scratch_floats, int* err, cudaStream_t st) {
    typedef Rec<DP, MODE> R;
    constexpr bool HEAD = MODE == 2 || MODE == 4;
    // at least the sum of ceil(len / 32) over the sequences of `shortest` tokens and more, of which there are at most N / shortest
    const int slots = N / LC_C + (S < N / shortest ? S : N / shortest);
    if (slots == 0) return 0;
    if ((long long)slots * H * R::ALL > scratch_floats) return -2;
    const size_t smem1 = (size_t)(2 * LC_C * DP + (HEAD ? LC_C * LC_C : LC_C * DP) + (MODE == 0 ? 2 : 1) * LC_C * LC_C + LC_C) * 4;
    const size_t smem2 = (size_t)(LC_STAGES * R::ALL + 2 * DP * LC_COLS + 2 * LC_C * LC_COLS + 4 * R::ROWS * LC_RED +
                                  (MODE == 0 ? LC_C * LC_COLS : 0)) * 4;
    constexpr bool TRANS = MODE == 4;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(chunk_prep_kernel<DP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(chunk_walk_kernel<DP, MODE, TRANS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    chunk_prep_kernel<DP, MODE><<<dim3(slots, H), 128, smem1, st>>>(q, k, g, beta, scratch, q_start, q_len, S, H, G, dim, shortest);
    MB_LAUNCH_CHECK();
    const dim3 grid((vdim + LC_COLS - 1) / LC_COLS, H, S);
    chunk_walk_kernel<DP, MODE, TRANS><<<grid, 256, smem2, st>>>(v, o, state, state_stride, scratch, q_start, q_len, state_slot, H,
                                                                 dim, vdim, shortest, err);
    MB_LAUNCH_CHECK();
    return 0;
}

// floats of a chunk's record for one head; 0: sizes the kernels do not take
MB_API int mb_linear_chunks_record(int dim, int vdim, int mode) {
    if (dim < 4 || dim > 128 || dim % 4 || vdim < 4 || vdim % 4 || mode < 0 || mode > 4) return 0;
    return dim <= 64 ? (mode == 0 ? Rec<64, 0>::ALL : Rec<64, 1>::ALL) : (mode == 0 ? Rec<128, 0>::ALL : Rec<128, 1>::ALL);
}

// q, k (N, G, dim), v, o (N, H, vdim), all of them and g on 16-byte boundaries; state: a head's matrix at h dim vdim,
// (dim, vdim), with mode 4 (vdim, dim).  scratch: (N / 32 + min(S, N / shortest)) H records.  Sequences of fewer than
// `shortest` tokens (32 or more) are left as they are.
MB_API int mb_linear_chunks(const float* q, const float* k, const float* v, const float* g, const float* beta, float* o,
                            float* state, long long state_stride, const int* q_start, const int* q_len,
                            const int* state_slot, int S, int N, int H, int G, int dim, int vdim, int mode, int shortest, float* scratch,
                            long long scratch_floats, int* err, cudaStream_t st) {
    if (S == 0 || N == 0) return 0;
    if (G < 1 || H % G || H > 65535 || S > 65535 || shortest < LC_MIN || !mb_linear_chunks_record(dim, vdim, mode)) return -2;
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o | (uintptr_t)scratch) & 15) return -2;
    if ((mode == 0 || mode == 1 || mode == 3) && ((uintptr_t)g & 15)) return -2;
    if ((mode == 0 || mode == 3) && !beta) return -2;
#define LC_CASE(MODE)                                                                                                       \
    if (mode == MODE)                                                                                                       \
        return dim <= 64 ? lc_launch<64, MODE>(q, k, v, g, beta, o, state, state_stride, q_start, q_len, state_slot, S, N, H, G, \
                                               dim, vdim, shortest, scratch, scratch_floats, err, st)                                 \
                         : lc_launch<128, MODE>(q, k, v, g, beta, o, state, state_stride, q_start, q_len, state_slot, S, N, H, \
                                                G, dim, vdim, shortest, scratch, scratch_floats, err, st);
    LC_CASE(0) LC_CASE(1) LC_CASE(2) LC_CASE(3) LC_CASE(4)
#undef LC_CASE
    return -2;
}
