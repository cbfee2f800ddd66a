// The scan of recurrent mixers whose matrix state decays by one number per head and token, for prompts, on tensor cores: per head
// S_t = a_t S_(t-1) + b_t k_t v_t^T and o_t = S_t^T q_t, with bfloat16 q, k and v.  Over a chunk of CHUNK tokens this is
//     o_t = exp(c_t) q_t^T S_in + sum over s <= t of (q_t . k_s) exp(c_t - c_s) b_s v_s,     c_t = log a_1 + .. + log a_t,
//     S_out = exp(c_end) S_in + sum over s of k_s (exp(c_end - c_s) b_s v_s)^T,
// matrix products instead of a chain over the tokens (the chunked form of state-space duality, Dao and Gu 2024).  Three launches: chunk_states_kernel leaves every chunk's own share of
// S_out (from S_in = 0), chunk_chain_kernel turns the shares into the chunks' S_in in order and updates the slot, and
// chunk_outputs_kernel writes o.
//
// Exactness: the products of stored bfloat16 values are exact in float32; what is float32 (S_in, the weighted v, the
// weighted scores) enters as the sum of three bfloat16 numbers, which holds all 24 bits, so every product is the float32
// one and every sum is float32.  A tensor-core sum drops what lies below its largest term's last bits: long sums are
// therefore taken in short runs that are added up by rounded float32 additions.  The logs are summed in float64 and kept as
// two float32 numbers, so a difference of two of them is as good as a float32 number near zero.  Measured against float64
// (relative, 2-norm; one prompt of 2,048 tokens, 64 heads of 128 x 64): outputs 1.4e-7, last state 6.4e-8; token by token in
// float32 1.5e-7 and 7.0e-8, and with slow decays 1.4e-7 and 2.4e-7 against 5.2e-7 and 9.2e-7.
//
// Values that are not finite, and columns whose results are not, are taken token by token (chunk_in_order).
//
// What bounds it: the phases of a block (loads, logs, conversion, products) follow one another and two blocks share a
// multiprocessor; the tensor pipe is 33 to 37 % busy, issue slots 40 %.  The state shares (N * P floats a chunk and head,
// written, chained and read) stay in L2.  CHUNK = 128: 64 would double the shares' traffic for a tenth fewer products, 256
// would not fit its operands into half of a multiprocessor's shared memory.  Measured, one prompt of 2,048 tokens, 64 heads of
// 128 x 64: 471 us token by token in chunks of time, 101 us here (states 33, chain 9, outputs 60; 67 while a block asked for S_in
// only after its logs and rows).
#pragma once
#include "common.cuh"

#define CHUNK 128
#define CHUNK_PB 64        // columns of v a block
#define CHUNK_SSM 0        // k = B, q = C of the head's group, v = x; b and a from step sizes; o gets d v on top
#define CHUNK_MEMORY 1     // b and log a from `gates` and `log_a`; beside S runs n (a column of v that is always 1)

struct ChunkArgs {
    const __nv_bfloat16 *q, *k, *v;             // first element of head 0's values in row 0
    long long q_stride, k_stride, v_stride;     // elements from row to row
    int share;                                  // heads that share a q and a k (a group)
    const __nv_bfloat16* dt;                    // CHUNK_SSM: raw step sizes, one per head
    long long dt_stride;
    const float *dt_bias, *a_log, *d_skip;
    const float *gates, *log_a;                 // CHUNK_MEMORY: [T, heads, 2] (its second number is b), [T, heads]
    float q_scale;
    float* state;                               // [slots][heads][N][P]
    float* n_state;                             // CHUNK_MEMORY: [slots][heads][N]
    long long slot_stride;
    float *o, *nq;                              // [T, heads * P], [T, heads]
    const int *meta, *cu_tokens, *slots;
    int slot_pairs;                             // slots start on 8 bytes
    int S, heads, N, P, max_chunks;             // max_chunks: at least the chunks of all entries together
    float *scratch, *decay;                     // [max_chunks][heads][N * P (+ N)], [max_chunks][heads]; the entries' chunks one behind the other
};

__device__ __forceinline__ uint32_t smem_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldmatrix4_t(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory"); }

// Two float32 numbers as three pairs of bfloat16 numbers whose sum they are (low half: the first number).
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(b), "f"(a));
    a -= __uint_as_float(h << 16), b -= __uint_as_float(h & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(m) : "f"(b), "f"(a));
    a -= __uint_as_float(m << 16), b -= __uint_as_float(m & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(b), "f"(a));
}

// Byte offset of 16-byte piece `c` of row `r` in a tile whose rows are ROW bytes: pieces are exchanged within a row by the
// row's last three bits, so that ldmatrix reads eight rows' pieces from eight different bank groups.
template <int ROW>
__device__ __forceinline__ uint32_t piece(int r, int c) {
    static_assert(ROW % 64 == 0, "rows of 64 bytes or more");
    if (ROW == 64) return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
    return (uint32_t)(r * ROW + ((c ^ (r & 7)) << 4));
}

// The logs of a chunk's decays, summed in order, as two float32 numbers each (hi + lo), and every token's weight b.  All 256
// threads call it; the first CHUNK have a token each (tokens behind the chunk's end: log 0, weight 0).
struct ChunkLogs {
    float hi[CHUNK], lo[CHUNK], b[CHUNK];
    double warp_sums[CHUNK / 32];
};
template <int KIND>
__device__ __forceinline__ void chunk_logs(ChunkLogs& L, const ChunkArgs& A, int h, int t0, int nt) {
    const int tid = threadIdx.x, lane = tid & 31;
    double s = 0.0;
    if (tid < CHUNK) {
        float b = 0.f, la = 0.f;
        if (tid < nt) {
            const size_t t = (size_t)(t0 + tid);
            if (KIND == CHUNK_SSM) {
                const float raw = __bfloat162float(A.dt[t * A.dt_stride + h]) + A.dt_bias[h];
                b = raw > 20.f ? raw : log1pf(expf(raw));  // softplus; beyond 20 the difference is below rounding
                la = -expf(A.a_log[h]) * b;
            } else {
                b = A.gates[(t * A.heads + h) * 2 + 1];
                la = A.log_a[t * A.heads + h];
            }
            la = la < -1e4f ? -1e4f : la;  // (a factor of zero either way, and no difference of infinities)
        }
        L.b[tid] = b;
        s = (double)la;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double below = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += below;
        }
        if (lane == 31) L.warp_sums[tid >> 5] = s;
    }
    __syncthreads();
    if (tid < CHUNK) {
        for (int w = 0; w < (tid >> 5); ++w) s += L.warp_sums[w];
        const float hi = (float)s;
        L.hi[tid] = hi;
        L.lo[tid] = (float)(s - (double)hi);
    }
    __syncthreads();
}
// exp(c_t - c_s) for c_t <= c_s
__device__ __forceinline__ float decay_between(float hi_t, float lo_t, float hi_s, float lo_s) {
    const float d = (hi_t - hi_s) + (lo_t - lo_s);
    return expf(d > 0.f ? 0.f : d);  // (what is no number stays none)
}

// Rows t0 .. t0 + nt of `src` (n of `ROW / 2` values wanted, zeros behind them and behind the rows) into a tile.
template <int ROW>
__device__ __forceinline__ void stage_rows(char* tile, const __nv_bfloat16* src, long long stride, int t0, int nt, int rows, int n) {
    constexpr int PIECES = ROW / 16;
    for (int i = threadIdx.x; i < rows * PIECES; i += 256) {
        const int r = i / PIECES, c = i % PIECES;
        char* dst = tile + piece<ROW>(r, c);
        if (r < nt && c * 8 < n) copy16_async(smem_address(dst), src + (size_t)(t0 + r) * stride + c * 8);
        else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
    }
}

// Which chunk (of LEN tokens) the step's `index`-th one is: its entry, its first token and its tokens, and whether it is the entry's only one.
// Every warp finds out by itself: a lane an entry, chunks counted up over the lanes.
struct ChunkPlace {
    int e, t0, nt, only;
};
template <int LEN>
__device__ __forceinline__ bool chunk_of(const int* __restrict__ meta, const int* __restrict__ cu_tokens, int index, ChunkPlace& p) {
    const int entries = meta[META_NUM_ENTRIES], lane = threadIdx.x & 31;
    int before = 0;
    for (int e0 = 0; e0 < entries; e0 += 32) {
        const int e = e0 + lane, first = e < entries ? cu_tokens[e] : 0, count = e < entries ? cu_tokens[e + 1] - first : 0;
        const int own = (count + LEN - 1) / LEN;
        int upto = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= d) upto += below;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, index < before + upto);
        if (hit) {
            const int from = __ffs(hit) - 1, c = index - before - __shfl_sync(0xffffffffu, upto - own, from);
            p.e = e0 + from;
            p.t0 = __shfl_sync(0xffffffffu, first, from) + c * LEN;
            p.nt = min(__shfl_sync(0xffffffffu, count, from) - c * LEN, LEN);
            p.only = __shfl_sync(0xffffffffu, own, from) == 1;
            return true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// ----------------------------------------------------------------------------- token by token
// A block's columns of its chunk in order and in float32, for what the products cannot carry: a weight of 0 times a later token's
// infinity is no number, and an infinity is no sum of three bfloat16 numbers.  A kernel whose results are not all finite ends with
// it, so that only the tokens behind such a value see it, as a scan in order gives it.  `outputs`: o (and n . q) from the chunk's S_in;
// else the chunk's share of S_out, or for an entry's only chunk the slot, what it held staying as S_in.  All 256 threads: a
// column of the block each, the rows dealt out over four of them.  (It finds its chunk by itself: nothing has to be kept for it.)
template <int NB, int KIND>
__device__ __noinline__ void chunk_in_order(const ChunkArgs& A, int col_blocks, bool outputs) {
    const int h = blockIdx.x / col_blocks, p0 = blockIdx.x % col_blocks * CHUNK_PB;
    ChunkPlace at;
    if (!chunk_of<CHUNK>(A.meta, A.cu_tokens, blockIdx.y, at)) return;
    const size_t HS = (size_t)A.N * A.P, CS = HS + (KIND == CHUNK_MEMORY ? A.N : 0);
    float* kept = A.scratch + ((size_t)blockIdx.y * A.heads + h) * CS;
    float* slot = A.state + (size_t)A.slots[at.e] * A.slot_stride + (size_t)h * HS;
    const float* from = outputs ? kept : (at.only ? slot : nullptr);
    float *first = !outputs && at.only ? kept : nullptr, *last = outputs ? nullptr : (at.only ? slot : kept);
    constexpr int ROWS = NB / 4;
    __shared__ float part[4][CHUNK_PB];
    const int col = threadIdx.x % CHUNK_PB, p = p0 + col, n0 = threadIdx.x / CHUNK_PB * ROWS;
    const bool real = p < A.P;
    float S[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        S[i] = from && real && n0 + i < A.N ? from[(size_t)(n0 + i) * A.P + p] : 0.f;
        if (first && real && n0 + i < A.N) first[(size_t)(n0 + i) * A.P + p] = S[i];
    }
    for (int t = at.t0; t < at.t0 + at.nt; ++t) {
        const __nv_bfloat16 *q = A.q + (size_t)t * A.q_stride + (size_t)(h / A.share) * A.N, *k = A.k + (size_t)t * A.k_stride + (size_t)(h / A.share) * A.N;
        const float v = real ? __bfloat162float(A.v[(size_t)t * A.v_stride + (size_t)h * A.P + p]) : 0.f;
        float a, b;
        if (KIND == CHUNK_SSM) {
            const float raw = __bfloat162float(A.dt[(size_t)t * A.dt_stride + h]) + A.dt_bias[h];
            b = raw > 20.f ? raw : log1pf(expf(raw));
            a = expf(-expf(A.a_log[h]) * b);
        } else {
            a = A.gates[((size_t)t * A.heads + h) * 2], b = A.gates[((size_t)t * A.heads + h) * 2 + 1];
        }
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            if (n0 + i >= A.N) break;
            const float kv = __bfloat162float(k[n0 + i]);
            S[i] = fmaf(a, S[i], KIND == CHUNK_SSM ? kv * (b * v) : kv * b * v);
            sum = fmaf(S[i], __bfloat162float(q[n0 + i]) * A.q_scale, sum);
        }
        if (!outputs) continue;
        __syncthreads();
        part[threadIdx.x / CHUNK_PB][col] = sum;
        __syncthreads();
        if (threadIdx.x < CHUNK_PB && real) {
            const float y = (part[0][col] + part[1][col]) + (part[2][col] + part[3][col]);
            A.o[((size_t)t * A.heads + h) * A.P + p] = KIND == CHUNK_SSM ? fmaf(A.d_skip[h], v, y) : y;
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
        if (last && real && n0 + i < A.N) last[(size_t)(n0 + i) * A.P + p] = S[i];
    if (KIND == CHUNK_MEMORY && outputs && p0 == 0 && threadIdx.x < 32) {  // n . q
        float n[NB / 32];
#pragma unroll
        for (int i = 0; i < NB / 32; ++i) n[i] = threadIdx.x + i * 32 < A.N ? kept[HS + threadIdx.x + i * 32] : 0.f;
        for (int t = at.t0; t < at.t0 + at.nt; ++t) {
            const __nv_bfloat16 *q = A.q + (size_t)t * A.q_stride + (size_t)h * A.N, *k = A.k + (size_t)t * A.k_stride + (size_t)h * A.N;
            const float a = A.gates[((size_t)t * A.heads + h) * 2], b = A.gates[((size_t)t * A.heads + h) * 2 + 1];
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < NB / 32; ++i) {
                const int row = threadIdx.x + i * 32;
                if (row >= A.N) break;
                n[i] = fmaf(a, n[i], __bfloat162float(k[row]) * b);
                sum = fmaf(n[i], __bfloat162float(q[row]) * A.q_scale, sum);
            }
            sum = warp_sum(sum);
            if (threadIdx.x == 0) A.nq[(size_t)t * A.heads + h] = sum;
        }
    }
}

// ----------------------------------------------------------------------------- every chunk's share of the state
// One block per (head x column block, chunk): NB (N rounded up) rows x CHUNK_PB columns, the eight warps a grid of WM x WN.
// The k values are the A operand, read transposed; the weighted v the B operand, as three pairs.
template <int NB, int KIND>
__global__ void __launch_bounds__(256, 2) chunk_states_kernel(const __grid_constant__ ChunkArgs A, int col_blocks) {
    constexpr int WM = NB >= 64 ? 4 : 2, WN = 8 / WM, MT = NB / 16 / WM, NT = CHUNK_PB / 8 / WN, KROW = NB * 2, VROW = CHUNK_PB * 2;
    extern __shared__ __align__(128) char chunk_smem[];
    char *ks = chunk_smem, *vs = chunk_smem + CHUNK * KROW;  // [CHUNK][NB]; three tiles [CHUNK][CHUNK_PB]
    __shared__ ChunkLogs L;
    __shared__ float wt[CHUNK];
    const int h = blockIdx.x / col_blocks, p0 = blockIdx.x % col_blocks * CHUNK_PB, c = blockIdx.y, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    ChunkPlace at;
    if (!chunk_of<CHUNK>(A.meta, A.cu_tokens, c, at)) return;
    const int t0 = at.t0, nt = at.nt;
    const int rows = (nt + 15) / 16 * 16;
    stage_rows<KROW>(ks, A.k + (size_t)(h / A.share) * A.N, A.k_stride, t0, nt, rows, A.N);
    uint4 vr[CHUNK * CHUNK_PB / 8 / 256];
#pragma unroll
    for (int u = 0; u < CHUNK * CHUNK_PB / 8 / 256; ++u) {
        const int i = tid + u * 256, r = i / (CHUNK_PB / 8), p = p0 + i % (CHUNK_PB / 8) * 8;
        vr[u] = make_uint4(0u, 0u, 0u, 0u);
        if (r < nt && p < A.P) vr[u] = *reinterpret_cast<const uint4*>(A.v + (size_t)(t0 + r) * A.v_stride + (size_t)h * A.P + p);
    }
    chunk_logs<KIND>(L, A, h, t0, nt);
    if (tid < CHUNK) wt[tid] = decay_between(L.hi[CHUNK - 1], L.lo[CHUNK - 1], L.hi[tid], L.lo[tid]) * L.b[tid];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < CHUNK * CHUNK_PB / 8 / 256; ++u) {
        const int i = tid + u * 256, r = i / (CHUNK_PB / 8);
        if (r >= rows) continue;
        const float w = wt[r];
        const uint32_t x[4] = {vr[u].x, vr[u].y, vr[u].z, vr[u].w};
        uint32_t s[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split_pair(__uint_as_float(x[j] << 16) * w, __uint_as_float(x[j] & 0xffff0000u) * w, s[0][j], s[1][j], s[2][j]);
#pragma unroll
        for (int j = 0; j < 3; ++j)
            *reinterpret_cast<uint4*>(vs + j * CHUNK * VROW + piece<VROW>(r, i % (CHUNK_PB / 8))) = make_uint4(s[j][0], s[j][1], s[j][2], s[j][3]);
    }
    copies_done();
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5, m0 = warp / WN * (MT * 16), n0 = warp % WN * (NT * 8);
    float acc[MT][NT][4] = {};
    for (int kt = 0; kt < rows; kt += 16) {
        float run[MT][NT][4] = {};
        uint32_t a[MT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i)
            ldmatrix4_t(a[i], smem_address(ks) + piece<KROW>(kt + (lane & 7) + ((lane >> 4) & 1) * 8, (m0 + i * 16) / 8 + ((lane >> 3) & 1)));
#pragma unroll
        for (int j = 2; j >= 0; --j)
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b[4];
                ldmatrix4_t(b, smem_address(vs) + j * CHUNK * VROW + piece<VROW>(kt + (lane & 7) + ((lane >> 3) & 1) * 8, n0 / 8 + n + (lane >> 4)));
#pragma unroll
                for (int i = 0; i < MT; ++i) mma16816(run[i][n], a[i], b[0], b[1]), mma16816(run[i][n + 1], a[i], b[2], b[3]);
            }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][n][j] += run[i][n][j];
    }
    const size_t HS = (size_t)A.N * A.P, CS = HS + (KIND == CHUNK_MEMORY ? A.N : 0), ch = (size_t)c * A.heads + h;
    float* dst = A.scratch + ch * CS;
    const float decay = expf(L.hi[CHUNK - 1] + L.lo[CHUNK - 1]);
    // an entry's only chunk needs no chain: what the slot holds is its S_in, and the slot is updated here
    float* slot = A.state + (size_t)A.slots[at.e] * A.slot_stride + (size_t)h * HS;
    float odd = 0.f;  // no number as soon as one result is not finite
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) odd = fmaf(acc[i][n][j], 0.f, odd);
    if (__syncthreads_or(odd != 0.f)) {
        chunk_in_order<NB, KIND>(A, col_blocks, false);
    } else {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const int row = m0 + i * 16 + (lane >> 2) + z * 8, p = p0 + n0 + n * 8 + (lane & 3) * 2;
                    if (p >= A.P || row >= A.N) continue;
                    float2 x = make_float2(acc[i][n][2 * z], acc[i][n][2 * z + 1]);
                    if (at.only) {
                        float* s = slot + (size_t)row * A.P + p;
                        const float2 in = A.slot_pairs ? *reinterpret_cast<const float2*>(s) : make_float2(s[0], s[1]);
                        const float2 out = make_float2(fmaf(decay, in.x, x.x), fmaf(decay, in.y, x.y));
                        if (A.slot_pairs) *reinterpret_cast<float2*>(s) = out;
                        else s[0] = out.x, s[1] = out.y;
                        x = in;
                    }
                    *reinterpret_cast<float2*>(dst + (size_t)row * A.P + p) = x;
                }
    }
    if (p0 == 0) {
        if (KIND == CHUNK_MEMORY && tid < A.N) {
            float s = 0.f;
            for (int t = 0; t < nt; ++t)
                s = fmaf(wt[t], __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(ks + piece<KROW>(t, tid / 8) + tid % 8 * 2)), s);
            if (at.only) {
                float* n = A.n_state + (size_t)A.slots[at.e] * A.slot_stride + (size_t)h * A.N + tid;
                const float in = *n;
                *n = fmaf(decay, in, s);
                s = in;
            }
            dst[HS + tid] = s;
        }
        if (tid == 0) A.decay[ch] = decay;
    }
}

// ----------------------------------------------------------------------------- the chunks' start states
// In place: share -> S_in of the chunk, S_out = decay * S_in + share; the last one goes to the slot.  A thread walks four neighbouring
// elements over the chunks, four to eight chunks loaded ahead (one element a thread: four times the blocks, each a chain of dependent
// loads before its first useful one: 42 against 35 us for 96 heads of 128 x 64 and three prompts of 17 chunks together).
template <int KIND>
__global__ void __launch_bounds__(256) chunk_chain_kernel(const ChunkArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.x, e = blockIdx.y;
    if (e >= A.meta[META_NUM_ENTRIES]) return;
    const int chunks = (A.cu_tokens[e + 1] - A.cu_tokens[e] + CHUNK - 1) / CHUNK;
    if (chunks < 2) return;  // (an only chunk has updated its slot itself)
    const size_t HS = (size_t)A.N * A.P, CS = HS + (KIND == CHUNK_MEMORY ? A.N : 0), i = ((size_t)blockIdx.z * 256 + threadIdx.x) * 4;
    if (i >= CS) return;
    float* slot = (i < HS ? A.state + (size_t)h * HS + i : A.n_state + (size_t)h * A.N + (i - HS)) + (size_t)A.slots[e] * A.slot_stride;
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = slot[j];  // (a slot may start on any float)
    int before = 0;
    for (int k = 0; k < e; ++k) before += (A.cu_tokens[k + 1] - A.cu_tokens[k] + CHUNK - 1) / CHUNK;
    float* at = A.scratch + ((size_t)before * A.heads + h) * CS + i;
    const float* dec = A.decay + (size_t)before * A.heads + h;
    const size_t step = (size_t)A.heads * CS;
    float own[4][4], d[4], own_next[4][4], d_next[4];
    auto fetch = [&](int c0, float (&x)[4][4], float (&f)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c0 + u < chunks) load4(at + (c0 + u) * step, x[u]), f[u] = dec[(size_t)(c0 + u) * A.heads];
    };
    fetch(0, own, d);
    for (int c0 = 0; c0 < chunks; c0 += 4) {
        fetch(c0 + 4, own_next, d_next);  // ahead of the stores
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c0 + u < chunks) {
                store4(at + (c0 + u) * step, s);
#pragma unroll
                for (int j = 0; j < 4; ++j) s[j] = fmaf(d[u], s[j], own[u][j]);
            }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            d[u] = d_next[u];
#pragma unroll
            for (int j = 0; j < 4; ++j) own[u][j] = own_next[u][j];
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) slot[j] = s[j];
}

// ----------------------------------------------------------------------------- the outputs
// One block per (head x column block, chunk); a warp has 16 tokens (warps of one scheduler get rows whose causal work adds up
// to the same).  q waits in registers; its tile's place then holds S_in as three pairs.
template <int NB, int KIND>
__global__ void __launch_bounds__(256, 2) chunk_outputs_kernel(const __grid_constant__ ChunkArgs A, int col_blocks) {
    constexpr int KROW = NB * 2, VROW = CHUNK_PB * 2, KT = NB / 16, NT = CHUNK_PB / 8;
    constexpr int SHARED0 = CHUNK * KROW > 3 * NB * VROW ? CHUNK * KROW : 3 * NB * VROW;
    extern __shared__ __align__(128) char chunk_smem[];
    char *qs = chunk_smem, *ss = chunk_smem, *ks = chunk_smem + SHARED0, *vs = ks + CHUNK * KROW;  // q, then S_in; k; v
    __shared__ ChunkLogs L;
    __shared__ float n_in[NB];
    const int h = blockIdx.x / col_blocks, p0 = blockIdx.x % col_blocks * CHUNK_PB, c = blockIdx.y, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    ChunkPlace at;
    if (!chunk_of<CHUNK>(A.meta, A.cu_tokens, c, at)) return;
    const int t0 = at.t0, nt = at.nt;
    const int rows = (nt + 15) / 16 * 16;
    stage_rows<KROW>(qs, A.q + (size_t)(h / A.share) * A.N, A.q_stride, t0, nt, rows, A.N);
    stage_rows<KROW>(ks, A.k + (size_t)(h / A.share) * A.N, A.k_stride, t0, nt, rows, A.N);
    stage_rows<VROW>(vs, A.v + (size_t)h * A.P + p0, A.v_stride, t0, nt, rows, A.P - p0);
    const size_t HS = (size_t)A.N * A.P, CS = HS + (KIND == CHUNK_MEMORY ? A.N : 0);
    const float* s_in = A.scratch + ((size_t)c * A.heads + h) * CS;
    if (KIND == CHUNK_MEMORY && tid < NB) n_in[tid] = tid < A.N ? s_in[HS + tid] : 0.f;
    constexpr int S_ITEMS = NB * (CHUNK_PB / 8) / 256;
    float4 sx[S_ITEMS][2];
    auto fetch_s = [&]() {
#pragma unroll
        for (int u = 0; u < S_ITEMS; ++u) {
            const int i = tid + u * 256, n = i / (CHUNK_PB / 8), p = p0 + i % (CHUNK_PB / 8) * 8;
            sx[u][0] = sx[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (n < A.N && p < A.P) {
                sx[u][0] = *reinterpret_cast<const float4*>(s_in + (size_t)n * A.P + p);
                sx[u][1] = *reinterpret_cast<const float4*>(s_in + (size_t)n * A.P + p + 4);
            }
        }
    };
    // S_in sets out with the rows and waits in registers until q's tile is read (67 -> 60 us; the memory's logs are loads, not
    // arithmetic, and there it cost 1 of 51)
    if (KIND == CHUNK_SSM) fetch_s();
    chunk_logs<KIND>(L, A, h, t0, nt);
    copies_done();
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5, rb = warp < 4 ? warp : 11 - warp, g = lane >> 2, q2 = (lane & 3) * 2;
    const bool busy = rb * 16 < nt;
    uint32_t qa[KT][4];
    if (busy) {
#pragma unroll
        for (int k = 0; k < KT; ++k) ldmatrix4(qa[k], smem_address(qs) + piece<KROW>(rb * 16 + (lane & 15), k * 2 + (lane >> 4)));
    }
    if (KIND != CHUNK_SSM) fetch_s();
    __syncthreads();  // q's tile is read: S_in takes its place
#pragma unroll
    for (int u = 0; u < S_ITEMS; ++u) {
        const int i = tid + u * 256, n = i / (CHUNK_PB / 8), pc = i % (CHUNK_PB / 8);
        const float4 x = sx[u][0], y = sx[u][1];
        uint32_t s[3][4];
        split_pair(x.x, x.y, s[0][0], s[1][0], s[2][0]);
        split_pair(x.z, x.w, s[0][1], s[1][1], s[2][1]);
        split_pair(y.x, y.y, s[0][2], s[1][2], s[2][2]);
        split_pair(y.z, y.w, s[0][3], s[1][3], s[2][3]);
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(ss + j * NB * VROW + piece<VROW>(n, pc)) = make_uint4(s[j][0], s[j][1], s[j][2], s[j][3]);
    }
    __syncthreads();
    float odd = 0.f;  // no number as soon as one result is not finite
    if (busy) {
        float acc[NT][4] = {};
#pragma unroll
        for (int k2 = 0; k2 < KT; k2 += 2) {  // q^T S_in: two steps of k a run
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                float run[2][4] = {};
#pragma unroll
                for (int k = k2; k < k2 + 2; ++k)
#pragma unroll
                    for (int j = 2; j >= 0; --j) {
                        uint32_t b[4];
                        ldmatrix4_t(b, smem_address(ss) + j * NB * VROW + piece<VROW>(k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, n + (lane >> 4)));
                        mma16816(run[0], qa[k], b[0], b[1]);
                        mma16816(run[1], qa[k], b[2], b[3]);
                    }
#pragma unroll
                for (int z = 0; z < 2; ++z)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[n + z][j] += run[z][j];
            }
        }
        const int ta = rb * 16 + g, tb = ta + 8;
        const float hi_a = L.hi[ta], lo_a = L.lo[ta], hi_b = L.hi[tb], lo_b = L.lo[tb], ea = expf(hi_a + lo_a), eb = expf(hi_b + lo_b);
        float na = 0.f, nb = 0.f;  // CHUNK_MEMORY: n . q
        if (KIND == CHUNK_MEMORY) {
#pragma unroll
            for (int k = 0; k < KT; ++k)
#pragma unroll
                for (int z = 0; z < 4; ++z) {  // registers 0 and 2: row g, 1 and 3: row g + 8; 0 and 1: k, 2 and 3: k + 8
                    const int n = k * 16 + q2 + (z >> 1) * 8;
                    float& s = z & 1 ? nb : na;
                    s = fmaf(__uint_as_float(qa[k][z] << 16), n_in[n], s);
                    s = fmaf(__uint_as_float(qa[k][z] & 0xffff0000u), n_in[n + 1], s);
                }
            na *= ea, nb *= eb;
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[n][0] *= ea, acc[n][1] *= ea, acc[n][2] *= eb, acc[n][3] *= eb;
#pragma unroll 1
        for (int sb = 0; sb <= rb; ++sb) {
            float sc[2][4] = {};
#pragma unroll
            for (int k = 0; k < KT; ++k) {
                uint32_t b[4];
                ldmatrix4(b, smem_address(ks) + piece<KROW>(sb * 16 + (lane & 7) + (lane >> 4) * 8, k * 2 + ((lane >> 3) & 1)));
                mma16816(sc[0], qa[k], b[0], b[1]);
                mma16816(sc[1], qa[k], b[2], b[3]);
            }
            uint32_t w[3][4];
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                const int s0 = sb * 16 + z * 8 + q2;
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int s = s0 + (j & 1), t = j < 2 ? ta : tb;
                    const float f = decay_between(j < 2 ? hi_a : hi_b, j < 2 ? lo_a : lo_b, L.hi[s], L.lo[s]) * L.b[s];
                    v[j] = s <= t ? sc[z][j] * f : 0.f;
                }
                if (KIND == CHUNK_MEMORY) na += v[0] + v[1], nb += v[2] + v[3];
                split_pair(v[0], v[1], w[0][z * 2], w[1][z * 2], w[2][z * 2]);
                split_pair(v[2], v[3], w[0][z * 2 + 1], w[1][z * 2 + 1], w[2][z * 2 + 1]);
            }
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b[4];
                ldmatrix4_t(b, smem_address(vs) + piece<VROW>(sb * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, n + (lane >> 4)));
                float run[2][4] = {};
#pragma unroll
                for (int j = 2; j >= 0; --j) mma16816(run[0], w[j], b[0], b[1]), mma16816(run[1], w[j], b[2], b[3]);
#pragma unroll
                for (int z = 0; z < 2; ++z)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[n + z][j] += run[z][j];
            }
        }
        const size_t out_stride = (size_t)A.heads * A.P;
        float* oa = A.o + (size_t)(t0 + ta) * out_stride + (size_t)h * A.P + p0 + q2;
        const float dskip = KIND == CHUNK_SSM ? A.d_skip[h] : 0.f;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            if (p0 + n * 8 >= A.P) break;
            float* x = acc[n];
            if (KIND == CHUNK_SSM) {
                const uint32_t va = *reinterpret_cast<const uint32_t*>(vs + piece<VROW>(ta, n) + q2 * 2), vb = *reinterpret_cast<const uint32_t*>(vs + piece<VROW>(tb, n) + q2 * 2);
                x[0] = fmaf(dskip, __uint_as_float(va << 16), x[0]), x[1] = fmaf(dskip, __uint_as_float(va & 0xffff0000u), x[1]);
                x[2] = fmaf(dskip, __uint_as_float(vb << 16), x[2]), x[3] = fmaf(dskip, __uint_as_float(vb & 0xffff0000u), x[3]);
            } else {
                x[0] *= A.q_scale, x[1] *= A.q_scale, x[2] *= A.q_scale, x[3] *= A.q_scale;
            }
            odd = fmaf(x[0], 0.f, fmaf(x[1], 0.f, fmaf(x[2], 0.f, fmaf(x[3], 0.f, odd))));
            if (ta < nt) *reinterpret_cast<float2*>(oa + n * 8) = make_float2(x[0], x[1]);
            if (tb < nt) *reinterpret_cast<float2*>(oa + 8 * out_stride + n * 8) = make_float2(x[2], x[3]);
        }
        if (KIND == CHUNK_MEMORY && p0 == 0) {
#pragma unroll
            for (int d = 1; d < 4; d <<= 1) na += __shfl_xor_sync(0xffffffffu, na, d), nb += __shfl_xor_sync(0xffffffffu, nb, d);
            odd = fmaf(na, 0.f, fmaf(nb, 0.f, odd));
            if ((lane & 3) == 0) {
                if (ta < nt) A.nq[(size_t)(t0 + ta) * A.heads + h] = na * A.q_scale;
                if (tb < nt) A.nq[(size_t)(t0 + tb) * A.heads + h] = nb * A.q_scale;
            }
        }
    }
    if (__syncthreads_or(odd != 0.f)) chunk_in_order<NB, KIND>(A, col_blocks, true);
}

// ----------------------------------------------------------------------------- launches
template <int KIND>
static size_t chunk_scratch_floats(int heads, int N, int P, int max_chunks) {
    return (size_t)max_chunks * heads * ((size_t)N * P + (KIND == CHUNK_MEMORY ? N : 0) + 1);
}

// Whether these sizes and addresses are served: rows in 16-byte pieces, at most 128 rows of state.
static bool chunk_scan_takes(const void* q, const void* k, const void* v, long long q_stride, long long k_stride, long long v_stride,
                             const void* o, int N, int P) {
    return N > 0 && N <= 128 && N % 8 == 0 && P > 0 && P % 8 == 0 && q_stride % 8 == 0 && k_stride % 8 == 0 && v_stride % 8 == 0 &&
           (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) == 0 && ((uintptr_t)o & 7) == 0;
}

template <int NB, int KIND>
static int chunk_scan_run(const ChunkArgs& a, cudaStream_t stream) {
    const int col_blocks = (a.P + CHUNK_PB - 1) / CHUNK_PB;
    constexpr size_t krow = NB * 2, vrow = CHUNK_PB * 2;
    constexpr size_t smem_s = CHUNK * krow + 3 * CHUNK * vrow, first = CHUNK * krow > 3 * NB * vrow ? CHUNK * krow : 3 * NB * vrow;
    constexpr size_t smem_o = first + CHUNK * krow + CHUNK * vrow;
    static bool configured = false;
    cudaError_t err = cudaSuccess;
    if (!configured) {
        err = cudaFuncSetAttribute(chunk_states_kernel<NB, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_s);
        if (err == cudaSuccess) err = cudaFuncSetAttribute(chunk_outputs_kernel<NB, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_o);
        if (err != cudaSuccess) return (int)err;
        configured = true;
    }
    const dim3 grid(a.heads * col_blocks, a.max_chunks);
    err = launch_kernel(chunk_states_kernel<NB, KIND>, grid, 256, smem_s, stream, a, col_blocks);
    if (err != cudaSuccess) return (int)err;
    const size_t CS = (size_t)a.N * a.P + (KIND == CHUNK_MEMORY ? a.N : 0);
    err = launch_kernel(chunk_chain_kernel<KIND>, dim3(a.heads, a.S, (unsigned)((CS + 1023) / 1024)), 256, 0, stream, a);
    if (err != cudaSuccess) return (int)err;
    return (int)launch_kernel(chunk_outputs_kernel<NB, KIND>, grid, 256, smem_o, stream, a, col_blocks);
}

// `a.scratch` of chunk_scratch_floats(..) floats, on 16 bytes.
template <int KIND>
static int chunk_scan(ChunkArgs a, cudaStream_t stream) {
    if (a.S <= 0 || a.max_chunks <= 0) return 0;
    if (a.max_chunks > 65535) return (int)cudaErrorInvalidValue;
    if (!chunk_scan_takes(a.q, a.k, a.v, a.q_stride, a.k_stride, a.v_stride, a.o, a.N, a.P) || ((uintptr_t)a.scratch & 15)) return (int)cudaErrorInvalidValue;
    a.slot_pairs = a.slot_stride % 2 == 0 && ((uintptr_t)a.state & 7) == 0;
    a.decay = a.scratch + chunk_scratch_floats<KIND>(a.heads, a.N, a.P, a.max_chunks) - (size_t)a.max_chunks * a.heads;
    if (a.N <= 32) return chunk_scan_run<32, KIND>(a, stream);
    if (a.N <= 64) return chunk_scan_run<64, KIND>(a, stream);
    return chunk_scan_run<128, KIND>(a, stream);
}
