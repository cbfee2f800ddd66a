// The scan of recurrent mixers whose matrix state decays by a number per ROW (key channel), head and token, for bfloat16 prompts, on
// tensor cores: S_t = diag(a_t) S_(t-1) + k_t v_t^T, and
//  * ROW_DECAY: o_t = S_t^T q_t, a_t = sigmoid(z_t)^(1/tau);
//  * ROW_BONUS: o_t = (S_(t-1) + diag(u) k_t v_t^T)^T q_t, a_t = exp(-exp(z_t)).
// Over a chunk of RCHUNK tokens, c_t the sum of the logs of a_1 .. a_t (per channel; ROW_BONUS: queries use c_(t-1)):
//     o_t = (q_t exp(c_t))^T S_in + sum over s <= t of W[t, s] v_s,   W[t, s] = sum over n of q_t[n] k_s[n] exp(c_t[n] - c_s[n]),
//     S_out = diag(exp(c_end)) S_in + sum over s of (k_s exp(c_end - c_s)) v_s^T.
// Four launches.  row_prepare_kernel does everything with exponentials once per head and chunk and leaves the three factors
// q exp(c), k exp(c_end - c) and W as operands of the matrix instructions, in the order in which a lane loads them;
// row_states_kernel every chunk's own share of S_out; row_chain_kernel the chunks' S_in in order, and the slot;
// row_outputs_kernel o.
//
// W (the two-level chunking of gated linear attention, Yang et al. 2023, with a third level below): between two sub-blocks of 16
// tokens both factors are taken relative to the earlier one's last token, q exp(c_t - c_e) and
// k exp(c_e - c_s), so no exponent is above zero; the half of a diagonal sub-block below its corner likewise with 8 tokens;
// the triangles of 8 that remain are summed over the channels directly.
//
// Exactness as in chunk_scan.cuh: stored bfloat16 values enter as they are, float32 factors as sums of three bfloat16 numbers; a
// product of two such factors leaves out the three of its nine partial products that lie below float32's last place.  Logs are
// summed in float64 and kept as two float32 numbers.  Measured against float64 (relative, 2-norm, three prompts of 2,048 tokens
// together, 8 heads of 128 x 256): outputs 1.3e-7, last states 7.9e-8; token by token in float32 2.5e-7 and 2.6e-7.
//
// What bounds it: the chain of phases of a block that prepares (40 us; a block a head and chunk is few blocks, hence 16 warps), then
// mma.sync (shares of the state 21 us, outputs 35, 37 before all of S_in
// was on its way at once) and the chunks' states through L2 (11).  105 us for the prompts above; token by
// token in chunks of time 283.  Heads of 64 x 64 (32 of them, 2,048 tokens): 131 against 184.
#pragma once
#include "chunk_scan.cuh"

#define RCHUNK 64
#define ROW_DECAY 0
#define ROW_BONUS 1
#define PREPARE_THREADS 512

struct RowScanArgs {
    const __nv_bfloat16 *q, *k, *v;
    long long q_stride, k_stride, v_stride;
    const float *z, *z_bias, *bonus;
    long long z_stride;
    float inv_tau, q_scale;
    float* state;                    // [slots][heads][N][P]
    long long slot_stride;
    float* o;                        // [T, heads * P]
    const int *meta, *cu_tokens, *slots;
    int slot_pairs, S, heads, N, P, max_chunks;
    int h0, hn;                      // the heads of this round of launches
    uint4 *qf, *kf, *wf;             // per (chunk, head): operands, see above
    float *share, *decay;            // [chunk][hn][N * P], [chunk][hn][N]
};

// exp(c_a - c_b) for c_a <= c_b, both as (hi, lo)
__device__ __forceinline__ float row_decay(float2 a, float2 b) { return decay_between(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float2 wide2(uint32_t x) { return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }
// c += the product of two factors given as three terms each: six of the nine products, the small ones first
__device__ __forceinline__ void mma_split6(float (&c)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
    mma16816(c, a[2], b[0][0], b[0][1]);
    mma16816(c, a[0], b[2][0], b[2][1]);
    mma16816(c, a[1], b[1][0], b[1][1]);
    mma16816(c, a[1], b[0][0], b[0][1]);
    mma16816(c, a[0], b[1][0], b[1][1]);
    mma16816(c, a[0], b[0][0], b[0][1]);
}

// ----------------------------------------------------------------------------- logs, factors, W
template <int NB>
struct RowTile {
    static constexpr int LOG_LD = NB * 2 + 4;           // floats of a row of logs: (hi, lo) per channel; rows four banks apart
    static constexpr int ROW_LD = NB + 8;               // values of a row of q or k, likewise
    static constexpr size_t LOGS = (size_t)(RCHUNK + 1) * LOG_LD * 4, ROWS = (size_t)RCHUNK * ROW_LD * 2;
    static constexpr size_t SMEM = LOGS + 2 * ROWS + 4 * 16 * 17 * 4;
};

template <int NB, int KIND>
__global__ void __launch_bounds__(PREPARE_THREADS, 2) row_prepare_kernel(const RowScanArgs A) {
    using L = RowTile<NB>;
    constexpr int KT = NB / 16, PARTS = PREPARE_THREADS / NB, SPAN = RCHUNK / PARTS, PL = NB / 32;
    extern __shared__ __align__(16) char row_smem[];
    float* logs = reinterpret_cast<float*>(row_smem);    // row 0: zeros; row t + 1: c_t
    __nv_bfloat16 *qs = reinterpret_cast<__nv_bfloat16*>(row_smem + L::LOGS), *ks = reinterpret_cast<__nv_bfloat16*>(row_smem + L::LOGS + L::ROWS);
    float* diag = reinterpret_cast<float*>(row_smem + L::LOGS + 2 * L::ROWS);  // [4][16][17]
    __shared__ double totals[PARTS][NB];
    const int hl = blockIdx.x, h = A.h0 + hl, c = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q2 = (lane & 3) * 2;
    pdl_launch_dependents();
    pdl_wait();
    ChunkPlace at;
    if (!chunk_of<RCHUNK>(A.meta, A.cu_tokens, c, at)) return;
    const int t0 = at.t0, nt = at.nt;
    for (int i = tid; i < RCHUNK * (NB / 8) * 2; i += PREPARE_THREADS) {
        const int which = i / (RCHUNK * (NB / 8)), r = i / (NB / 8) % RCHUNK, n = i % (NB / 8) * 8;
        __nv_bfloat16* dst = (which ? ks : qs) + r * L::ROW_LD + n;
        const __nv_bfloat16* src = (which ? A.k + (size_t)(t0 + r) * A.k_stride : A.q + (size_t)(t0 + r) * A.q_stride) + (size_t)h * A.N + n;
        if (r < nt && n < A.N) copy16_async(smem_address(dst), src);
        else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
    }
    for (int i = tid; i < 4 * 16 * 17; i += PREPARE_THREADS) diag[i] = 0.f;
    for (int i = tid; i < L::LOG_LD; i += PREPARE_THREADS) logs[i] = 0.f;
    {   // a thread a channel and stretch of tokens
        const int n = tid % NB, part = tid / NB;
        const bool real = n < A.N;
        const float bias = real && A.z_bias ? A.z_bias[(size_t)h * A.N + n] : 0.f;
        const float* zp = A.z + (size_t)(t0 + part * SPAN) * A.z_stride + (size_t)h * A.N + n;
        double s = 0.0;
        for (int i0 = 0; i0 < SPAN; i0 += 8) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = real && part * SPAN + i0 + i < nt ? zp[(size_t)(i0 + i) * A.z_stride] + bias : 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int t = part * SPAN + i0 + i;
                float la = 0.f;
                if (real && t < nt) la = KIND == ROW_BONUS ? -expf(x[i]) : -(-x[i] > 20.f ? -x[i] : log1pf(expf(-x[i]))) * A.inv_tau;
                s += (double)(la < -1e4f ? -1e4f : la);  // (a factor of zero either way, and no difference of infinities)
                const float hi = (float)s;
                *reinterpret_cast<float2*>(logs + (t + 1) * L::LOG_LD + n * 2) = make_float2(hi, (float)(s - (double)hi));
            }
        }
        totals[part][n] = s;
        __syncthreads();
        double before = 0.0;
        for (int p = 0; p < part; ++p) before += totals[p][n];
        if (part > 0)
            for (int i = 0; i < SPAN; ++i) {
                float2* e = reinterpret_cast<float2*>(logs + (part * SPAN + i + 1) * L::LOG_LD + n * 2);
                const double x = ((double)e->x + (double)e->y) + before;
                const float hi = (float)x;
                *e = make_float2(hi, (float)(x - (double)hi));
            }
    }
    copies_done();
    __syncthreads();
    // (hi, lo) of the channels n and n + 1 at a key's token; at a query's (KEY 0)
    auto log_at = [&](int row, int n) { return *reinterpret_cast<const float2*>(logs + row * L::LOG_LD + n * 2); };
    constexpr int QROW = KIND == ROW_BONUS ? 0 : 1;  // the row of logs that the query of token t uses is t + QROW
    const size_t ch = (size_t)c * A.hn + hl;
    const float2 zero = make_float2(0.f, 0.f);

    // ---- q exp(c): tiles of 16 tokens x 16 channels
    for (int tile = warp; tile < 4 * KT; tile += PREPARE_THREADS / 32) {
        const int rb = tile / KT, kt = tile % KT;
        if (rb * 16 >= nt) continue;
        uint32_t f[3][4];
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const int t = rb * 16 + g + (z & 1) * 8, n = kt * 16 + q2 + (z >> 1) * 8;
            const float2 x = wide2(*reinterpret_cast<const uint32_t*>(qs + t * L::ROW_LD + n));
            const float4 l = *reinterpret_cast<const float4*>(logs + (t + QROW) * L::LOG_LD + n * 2);
            split_pair(x.x * row_decay(make_float2(l.x, l.y), zero), x.y * row_decay(make_float2(l.z, l.w), zero), f[0][z], f[1][z], f[2][z]);
        }
        uint4* dst = A.qf + ((ch * 4 + rb) * KT + kt) * 96 + lane;
#pragma unroll
        for (int j = 0; j < 3; ++j) dst[j * 32] = make_uint4(f[j][0], f[j][1], f[j][2], f[j][3]);
    }
    // ---- k exp(c_end - c): tiles of 16 channels x 16 tokens
    for (int tile = warp; tile < KT * 4; tile += PREPARE_THREADS / 32) {
        const int mt = tile / 4, kt = tile % 4;
        uint32_t f[3][4];
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const int n = mt * 16 + g + (z & 1) * 8, t = kt * 16 + q2 + (z >> 1) * 8;
            const float2 end = log_at(RCHUNK, n);
            const float a = __bfloat162float(ks[t * L::ROW_LD + n]) * row_decay(end, log_at(t + 1, n));
            const float b = __bfloat162float(ks[(t + 1) * L::ROW_LD + n]) * row_decay(end, log_at(t + 2, n));
            split_pair(a, b, f[0][z], f[1][z], f[2][z]);
        }
        uint4* dst = A.kf + ((ch * KT + mt) * 4 + kt) * 96 + lane;
#pragma unroll
        for (int j = 0; j < 3; ++j) dst[j * 32] = make_uint4(f[j][0], f[j][1], f[j][2], f[j][3]);
    }
    if (tid < A.N) {
        const float2 end = log_at(RCHUNK, tid);
        A.decay[ch * A.N + tid] = expf(end.x + end.y);
    }

    // ---- W.  A tile: the scores of 16 queries (HALF: the upper eight only) and 16 (8) keys relative to key `e`
    auto tile_scores = [&](int tq, int ts, int e, bool half, float (&acc)[2][4]) {
        for (int kt = 0; kt < KT; ++kt) {
            uint32_t a[3][4], b[2][3][2];
#pragma unroll
            for (int z = 0; z < 2; ++z) {  // channels q2 and q2 + 8
                const int n = kt * 16 + q2 + z * 8;
                const float4 r = *reinterpret_cast<const float4*>(logs + (e + 1) * L::LOG_LD + n * 2);
                const float2 r0 = make_float2(r.x, r.y), r1 = make_float2(r.z, r.w);
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const int t = tq + g + y * 8, s = ts + g + y * 8;
                    const float2 x = wide2(*reinterpret_cast<const uint32_t*>(qs + t * L::ROW_LD + n));
                    const float4 l = *reinterpret_cast<const float4*>(logs + (t + QROW) * L::LOG_LD + n * 2);
                    float x0 = x.x * row_decay(make_float2(l.x, l.y), r0), x1 = x.y * row_decay(make_float2(l.z, l.w), r1);
                    if (half && y == 0) x0 = x1 = 0.f;
                    split_pair(x0, x1, a[0][z * 2 + y], a[1][z * 2 + y], a[2][z * 2 + y]);
                    if (half && y == 1) continue;
                    const float2 u = wide2(*reinterpret_cast<const uint32_t*>(ks + s * L::ROW_LD + n));
                    const float4 m = *reinterpret_cast<const float4*>(logs + (s + 1) * L::LOG_LD + n * 2);
                    split_pair(u.x * row_decay(r0, make_float2(m.x, m.y)), u.y * row_decay(r1, make_float2(m.z, m.w)), b[y][0][z], b[y][1][z], b[y][2][z]);
                }
            }
            float run[2][4] = {};
            mma_split6(run[0], a, b[0]);
            if (!half) mma_split6(run[1], a, b[1]);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[0][j] += run[0][j], acc[1][j] += run[1][j];
        }
    };
    if (warp < 6) {  // sub-blocks (1, 0), (2, 0), (2, 1), (3, 0), (3, 1), (3, 2)
        const int tb = warp < 1 ? 1 : (warp < 3 ? 2 : 3), sb = warp - (tb == 1 ? 0 : (tb == 2 ? 1 : 3));
        if (tb * 16 < nt) {
            float w[2][4] = {};
            tile_scores(tb * 16, sb * 16, sb * 16 + 15, false, w);
            uint32_t f[3][4];
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                split_pair(w[z][0], w[z][1], f[0][z * 2], f[1][z * 2], f[2][z * 2]);
                split_pair(w[z][2], w[z][3], f[0][z * 2 + 1], f[1][z * 2 + 1], f[2][z * 2 + 1]);
            }
            uint4* dst = A.wf + ((ch * 4 + tb) * 4 + sb) * 96 + lane;
#pragma unroll
            for (int j = 0; j < 3; ++j) dst[j * 32] = make_uint4(f[j][0], f[j][1], f[j][2], f[j][3]);
        }
    } else if (warp < 10) {
        const int b = warp - 6;
        if (b * 16 + 8 < nt) {
            float w[2][4] = {};
            tile_scores(b * 16, b * 16, b * 16 + 7, true, w);
            float* d = diag + (b * 16 + 8 + g) * 17 + q2;
            d[0] = w[0][2], d[1] = w[0][3];
        }
    }
    // triangles of eight: a warp one of them (the six warps without a tile, and two with half a one), a lane PL neighbouring channels
    if (warp >= 8) {
        const int base = (warp - 8) * 8, n = lane * PL;
        float u[PL];
#pragma unroll
        for (int j = 0; j < PL; ++j) u[j] = KIND == ROW_BONUS && n + j < A.N ? A.bonus[(size_t)h * A.N + n + j] : 1.f;
        for (int i = 0; i < 8 && base + i < nt; ++i) {
            float qv[PL];
            float2 lq[PL];
#pragma unroll
            for (int j = 0; j < PL; ++j) qv[j] = __bfloat162float(qs[(base + i) * L::ROW_LD + n + j]), lq[j] = log_at(base + i + QROW, n + j);
            for (int s = 0; s <= i; ++s) {
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < PL; ++j) {
                    const float kv = __bfloat162float(ks[(base + s) * L::ROW_LD + n + j]);
                    const float f = s == i ? u[j] : row_decay(lq[j], log_at(base + s + 1, n + j));
                    sum = fmaf(qv[j] * kv, f, sum);
                }
                sum = warp_sum(sum);
                if (lane == 0) diag[((base / 16) * 16 + (base & 8) + i) * 17 + (base & 8) + s] = sum;
            }
        }
    }
    __syncthreads();
    if (warp < 4 && warp * 16 < nt) {
        uint32_t f[3][4];
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const float* d = diag + (warp * 16 + g + (z & 1) * 8) * 17 + q2 + (z >> 1) * 8;
            split_pair(d[0], d[1], f[0][z], f[1][z], f[2][z]);
        }
        uint4* dst = A.wf + ((ch * 4 + warp) * 4 + warp) * 96 + lane;
#pragma unroll
        for (int j = 0; j < 3; ++j) dst[j * 32] = make_uint4(f[j][0], f[j][1], f[j][2], f[j][3]);
    }
}

__device__ __forceinline__ void load_split(uint32_t (&f)[3][4], const uint4* src) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const uint4 x = src[j * 32];
        f[j][0] = x.x, f[j][1] = x.y, f[j][2] = x.z, f[j][3] = x.w;
    }
}

// ----------------------------------------------------------------------------- token by token
// As chunk_in_order (chunk_scan.cuh), for the same reasons; the decays from the logits again.
template <int NB, int KIND>
__device__ __noinline__ void row_in_order(const RowScanArgs& A, int col_blocks, bool outputs) {
    const int hl = blockIdx.x / col_blocks, h = A.h0 + hl, p0 = blockIdx.x % col_blocks * CHUNK_PB;
    ChunkPlace at;
    if (!chunk_of<RCHUNK>(A.meta, A.cu_tokens, blockIdx.y, at)) return;
    const size_t HS = (size_t)A.N * A.P;
    float* kept = A.share + ((size_t)blockIdx.y * A.hn + hl) * HS;
    float* slot = A.state + (size_t)A.slots[at.e] * A.slot_stride + (size_t)h * HS;
    const float* from = outputs ? kept : (at.only ? slot : nullptr);
    float *first = !outputs && at.only ? kept : nullptr, *last = outputs ? nullptr : (at.only ? slot : kept);
    constexpr int ROWS = NB / 4;
    __shared__ float part[2][4][CHUNK_PB];
    const int col = threadIdx.x % CHUNK_PB, p = p0 + col, g = threadIdx.x / CHUNK_PB, n0 = g * ROWS;
    const bool real = p < A.P;
    float S[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        S[i] = from && real && n0 + i < A.N ? from[(size_t)(n0 + i) * A.P + p] : 0.f;
        if (first && real && n0 + i < A.N) first[(size_t)(n0 + i) * A.P + p] = S[i];
    }
    for (int t = at.t0; t < at.t0 + at.nt; ++t) {
        const __nv_bfloat16 *q = A.q + (size_t)t * A.q_stride + (size_t)h * A.N, *k = A.k + (size_t)t * A.k_stride + (size_t)h * A.N;
        const float* z = A.z + (size_t)t * A.z_stride + (size_t)h * A.N;
        const float v = real ? __bfloat162float(A.v[(size_t)t * A.v_stride + (size_t)h * A.P + p]) : 0.f;
        float sum = 0.f, own = 0.f;  // ROW_BONUS: `own`, the current token's weight on its own v
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const int n = n0 + i;
            if (n >= A.N) break;
            const float x = z[n] + (A.z_bias ? A.z_bias[(size_t)h * A.N + n] : 0.f), kv = __bfloat162float(k[n]);
            const float a = KIND == ROW_BONUS ? expf(-expf(x)) : expf(-(-x > 20.f ? -x : log1pf(expf(-x))) * A.inv_tau);
            const float qv = __bfloat162float(q[n]) * A.q_scale, before = S[i];
            S[i] = fmaf(a, before, kv * v);
            sum = fmaf(KIND == ROW_BONUS ? before : S[i], qv, sum);
            if (KIND == ROW_BONUS) own = fmaf(qv * A.bonus[(size_t)h * A.N + n], kv, own);
        }
        if (!outputs) continue;
        __syncthreads();
        part[0][g][col] = sum, part[1][g][col] = own;
        __syncthreads();
        if (g == 0 && real) {
            float y = (part[0][0][col] + part[0][1][col]) + (part[0][2][col] + part[0][3][col]);
            if (KIND == ROW_BONUS) y = fmaf((part[1][0][col] + part[1][1][col]) + (part[1][2][col] + part[1][3][col]), v, y);
            A.o[((size_t)t * A.heads + h) * A.P + p] = y;
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
        if (last && real && n0 + i < A.N) last[(size_t)(n0 + i) * A.P + p] = S[i];
}

// ----------------------------------------------------------------------------- every chunk's share of the state
template <int NB, int KIND>
__global__ void __launch_bounds__(256, 2) row_states_kernel(const __grid_constant__ RowScanArgs A, int col_blocks) {
    constexpr int MT = NB / 16, WN = 8 / MT, NT = CHUNK_PB / 8 / WN, VROW = CHUNK_PB * 2;
    __shared__ __align__(128) char vs[RCHUNK * VROW];
    const int hl = blockIdx.x / col_blocks, h = A.h0 + hl, p0 = blockIdx.x % col_blocks * CHUNK_PB, c = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_launch_dependents();
    pdl_wait();
    ChunkPlace at;
    if (!chunk_of<RCHUNK>(A.meta, A.cu_tokens, c, at)) return;
    const int rows = (at.nt + 15) / 16 * 16, mt = warp / WN, n0 = warp % WN * NT * 8;
    stage_rows<VROW>(vs, A.v + (size_t)h * A.P + p0, A.v_stride, at.t0, at.nt, rows, A.P - p0);
    const size_t ch = (size_t)c * A.hn + hl;
    const uint4* src = A.kf + (ch * MT + mt) * 4 * 96 + lane;
    uint32_t a[3][4];
    load_split(a, src);
    copies_done();
    __syncthreads();
    float acc[NT][4] = {};
    for (int kt = 0; kt * 16 < rows; ++kt) {
        uint32_t next[3][4];
        load_split(next, src + min(kt + 1, 3) * 96);
        float run[NT][4] = {};
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
            uint32_t b[4];
            ldmatrix4_t(b, smem_address(vs) + piece<VROW>(kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, n0 / 8 + n + (lane >> 4)));
#pragma unroll
            for (int j = 2; j >= 0; --j) mma16816(run[n], a[j], b[0], b[1]), mma16816(run[n + 1], a[j], b[2], b[3]);
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[n][j] += run[n][j];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int z = 0; z < 4; ++z) a[j][z] = next[j][z];
    }
    const size_t HS = (size_t)A.N * A.P;
    float* dst = A.share + ch * HS;
    float* slot = A.state + (size_t)A.slots[at.e] * A.slot_stride + (size_t)h * HS;
    float odd = 0.f;  // no number as soon as one result is not finite
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) odd = fmaf(acc[n][j], 0.f, odd);
    if (__syncthreads_or(odd != 0.f)) {
        row_in_order<NB, KIND>(A, col_blocks, false);
        return;
    }
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        const int row = mt * 16 + (lane >> 2) + z * 8;
        if (row >= A.N) continue;
        const float decay = at.only ? A.decay[ch * A.N + row] : 0.f;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int p = p0 + n0 + n * 8 + (lane & 3) * 2;
            if (p >= A.P) continue;
            float2 x = make_float2(acc[n][2 * z], acc[n][2 * z + 1]);
            if (at.only) {  // an entry's only chunk: what the slot holds is its S_in, and the slot is updated here
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
}

// ----------------------------------------------------------------------------- the chunks' start states
// In place: share -> S_in of the chunk, S_out = decay * S_in + share; the last one goes to the slot.  Four neighbouring elements (of
// one row: P is a multiple of 8) a thread, four to eight chunks loaded ahead.
static __global__ void __launch_bounds__(256) row_chain_kernel(const RowScanArgs A) {
    pdl_launch_dependents();
    pdl_wait();
    const int hl = blockIdx.x, e = blockIdx.y;
    if (e >= A.meta[META_NUM_ENTRIES]) return;
    const int chunks = (A.cu_tokens[e + 1] - A.cu_tokens[e] + RCHUNK - 1) / RCHUNK;
    if (chunks < 2) return;
    const size_t HS = (size_t)A.N * A.P, i = ((size_t)blockIdx.z * 256 + threadIdx.x) * 4;
    if (i >= HS) return;
    float* slot = A.state + (size_t)A.slots[e] * A.slot_stride + (size_t)(A.h0 + hl) * HS + i;
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = slot[j];  // (a slot may start on any float)
    int before = 0;
    for (int k = 0; k < e; ++k) before += (A.cu_tokens[k + 1] - A.cu_tokens[k] + RCHUNK - 1) / RCHUNK;
    float* at = A.share + ((size_t)before * A.hn + hl) * HS + i;
    const float* dec = A.decay + ((size_t)before * A.hn + hl) * A.N + i / A.P;
    const size_t step = (size_t)A.hn * HS;
    float own[4][4], d[4], own_next[4][4], d_next[4];
    auto fetch = [&](int c0, float (&x)[4][4], float (&f)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c0 + u < chunks) load4(at + (c0 + u) * step, x[u]), f[u] = dec[(size_t)(c0 + u) * A.hn * A.N];
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
// One block per (head x column block, chunk): four rows of 16 tokens x two halves of the columns, a warp each.
template <int NB, int KIND>
__global__ void __launch_bounds__(256, 2) row_outputs_kernel(const __grid_constant__ RowScanArgs A, int col_blocks) {
    constexpr int KT = NB / 16, NT = CHUNK_PB / 16, VROW = CHUNK_PB * 2;
    extern __shared__ __align__(128) char row_out_smem[];
    char *ss = row_out_smem, *vs = row_out_smem + 3 * NB * VROW;  // S_in as three tiles [NB][CHUNK_PB]; v
    const int hl = blockIdx.x / col_blocks, h = A.h0 + hl, p0 = blockIdx.x % col_blocks * CHUNK_PB, c = blockIdx.y, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    ChunkPlace at;
    if (!chunk_of<RCHUNK>(A.meta, A.cu_tokens, c, at)) return;
    const int t0 = at.t0, nt = at.nt, rows = (nt + 15) / 16 * 16;
    stage_rows<VROW>(vs, A.v + (size_t)h * A.P + p0, A.v_stride, t0, nt, rows, A.P - p0);
    const size_t ch = (size_t)c * A.hn + hl, HS = (size_t)A.N * A.P;
    const float* s_in = A.share + ch * HS;
    const int lane = tid & 31, warp = tid >> 5, rb = warp >> 1, n0 = (warp & 1) * NT, g = lane >> 2, q2 = (lane & 3) * 2;
    const uint4* qsrc = A.qf + (ch * 4 + rb) * KT * 96 + lane;
    constexpr int S_ITEMS = NB * (CHUNK_PB / 8) / 256;
    float4 sx[S_ITEMS][2];  // all of S_in on its way before the first of it is split
#pragma unroll
    for (int u = 0; u < S_ITEMS; ++u) {
        const int i = tid + u * 256, n = i / (CHUNK_PB / 8), p = p0 + i % (CHUNK_PB / 8) * 8;
        sx[u][0] = sx[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < A.N && p < A.P) {
            sx[u][0] = *reinterpret_cast<const float4*>(s_in + (size_t)n * A.P + p);
            sx[u][1] = *reinterpret_cast<const float4*>(s_in + (size_t)n * A.P + p + 4);
        }
    }
    uint32_t a[3][4];
    if (rb * 16 < nt) load_split(a, qsrc);
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
    copies_done();
    __syncthreads();
    float odd = 0.f;  // no number as soon as one result is not finite
    if (rb * 16 < nt) {
        float acc[NT][4] = {};
#pragma unroll 2
        for (int kt = 0; kt < KT; ++kt) {
            uint32_t next[3][4];
            load_split(next, qsrc + min(kt + 1, KT - 1) * 96);
            float run[NT][4] = {};
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b0[3][2], b1[3][2];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    uint32_t b[4];
                    ldmatrix4_t(b, smem_address(ss) + j * NB * VROW + piece<VROW>(kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, n0 + n + (lane >> 4)));
                    b0[j][0] = b[0], b0[j][1] = b[1], b1[j][0] = b[2], b1[j][1] = b[3];
                }
                mma_split6(run[n], a, b0);
                mma_split6(run[n + 1], a, b1);
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[n][j] += run[n][j];
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int z = 0; z < 4; ++z) a[j][z] = next[j][z];
        }
        const uint4* wsrc = A.wf + (ch * 4 + rb) * 4 * 96 + lane;
        for (int sb = 0; sb <= rb; ++sb) {
            load_split(a, wsrc + sb * 96);
            float run[NT][4] = {};
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b[4];
                ldmatrix4_t(b, smem_address(vs) + piece<VROW>(sb * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, n0 + n + (lane >> 4)));
#pragma unroll
                for (int j = 2; j >= 0; --j) mma16816(run[n], a[j], b[0], b[1]), mma16816(run[n + 1], a[j], b[2], b[3]);
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[n][j] += run[n][j];
        }
        const int ta = rb * 16 + g;
        const size_t stride = (size_t)A.heads * A.P;
        float* oa = A.o + (size_t)(t0 + ta) * stride + (size_t)h * A.P + p0 + q2;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            if (p0 + (n0 + n) * 8 >= A.P) break;
            odd = fmaf(acc[n][0], 0.f, fmaf(acc[n][1], 0.f, fmaf(acc[n][2], 0.f, fmaf(acc[n][3], 0.f, odd))));
            if (ta < nt) *reinterpret_cast<float2*>(oa + (n0 + n) * 8) = make_float2(acc[n][0] * A.q_scale, acc[n][1] * A.q_scale);
            if (ta + 8 < nt) *reinterpret_cast<float2*>(oa + 8 * stride + (n0 + n) * 8) = make_float2(acc[n][2] * A.q_scale, acc[n][3] * A.q_scale);
        }
    }
    if (__syncthreads_or(odd != 0.f)) row_in_order<NB, KIND>(A, col_blocks, true);
}

// ----------------------------------------------------------------------------- launches
// Floats of scratch a head takes for that many chunks (a multiple of four).
static size_t row_scan_head_floats(int N, int P, int max_chunks) {
    const size_t nb = N <= 64 ? 64 : 128;
    const size_t per = (2 * 4 * (nb / 16) + 16) * 96 * 4 + (size_t)N * P + N;
    return (size_t)max_chunks * per;
}

template <int NB, int KIND>
static int row_scan_run(RowScanArgs a, float* scratch, size_t scratch_floats, cudaStream_t stream) {
    const int col_blocks = (a.P + CHUNK_PB - 1) / CHUNK_PB;
    constexpr size_t smem_p = RowTile<NB>::SMEM, smem_o = (size_t)3 * NB * CHUNK_PB * 2 + RCHUNK * CHUNK_PB * 2;
    static bool configured = false;
    cudaError_t err = cudaSuccess;
    if (!configured) {
        err = cudaFuncSetAttribute(row_prepare_kernel<NB, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_p);
        if (err == cudaSuccess) err = cudaFuncSetAttribute(row_outputs_kernel<NB, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_o);
        if (err != cudaSuccess) return (int)err;
        configured = true;
    }
    const size_t head = row_scan_head_floats(a.N, a.P, a.max_chunks);
    const int at_once = (int)(scratch_floats / head < (size_t)a.heads ? scratch_floats / head : (size_t)a.heads);
    if (at_once < 1) return (int)cudaErrorInvalidValue;
    const int rounds = (a.heads + at_once - 1) / at_once, per_round = (a.heads + rounds - 1) / rounds;
    for (a.h0 = 0; a.h0 < a.heads; a.h0 += per_round) {
        a.hn = a.heads - a.h0 < per_round ? a.heads - a.h0 : per_round;
        const size_t units = (size_t)a.max_chunks * a.hn;
        a.qf = reinterpret_cast<uint4*>(scratch);
        a.kf = a.qf + units * 4 * (NB / 16) * 96;
        a.wf = a.kf + units * 4 * (NB / 16) * 96;
        a.share = reinterpret_cast<float*>(a.wf + units * 16 * 96);
        a.decay = a.share + units * a.N * a.P;
        err = launch_kernel(row_prepare_kernel<NB, KIND>, dim3(a.hn, a.max_chunks), PREPARE_THREADS, smem_p, stream, a);
        if (err == cudaSuccess) err = launch_kernel(row_states_kernel<NB, KIND>, dim3(a.hn * col_blocks, a.max_chunks), 256, 0, stream, a, col_blocks);
        if (err == cudaSuccess)
            err = launch_kernel(row_chain_kernel, dim3(a.hn, a.S, (unsigned)(((size_t)a.N * a.P + 1023) / 1024)), 256, 0, stream, a);
        if (err == cudaSuccess) err = launch_kernel(row_outputs_kernel<NB, KIND>, dim3(a.hn * col_blocks, a.max_chunks), 256, smem_o, stream, a, col_blocks);
        if (err != cudaSuccess) return (int)err;
    }
    return 0;
}

// `scratch` on 16 bytes, of at least one head's floats; with fewer than all heads' the heads run in rounds.
template <int KIND>
static int row_scan(RowScanArgs a, float* scratch, size_t scratch_floats, cudaStream_t stream) {
    if (a.S <= 0 || a.max_chunks <= 0) return 0;
    if (a.max_chunks > 65535 || ((uintptr_t)scratch & 15) || !chunk_scan_takes(a.q, a.k, a.v, a.q_stride, a.k_stride, a.v_stride, a.o, a.N, a.P))
        return (int)cudaErrorInvalidValue;
    a.slot_pairs = a.slot_stride % 2 == 0 && ((uintptr_t)a.state & 7) == 0;
    return a.N <= 64 ? row_scan_run<64, KIND>(a, scratch, scratch_floats, stream) : row_scan_run<128, KIND>(a, scratch, scratch_floats, stream);
}
