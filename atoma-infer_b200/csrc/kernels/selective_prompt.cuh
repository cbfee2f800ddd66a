// The selective scan of prompts in one pass, in order, with many channels side by side instead of chunks of time.
//
// The work that cannot be left out is an ex2 per state and token; taken once, 2,048 tokens of 4,096 channels x 16 states are
// 30 us of the special-function pipe.  A scan cut into chunks of time takes them twice (for the chunks' own states and again
// for the outputs) and chains the states in between.  Here a block keeps 32 channels from the first token to the last: warps 0..3
// run the recurrence, a lane four states of a channel (512 warps for 4,096 channels: about one for each of the chip's 592
// schedulers), and sixteen warps do everything else, a tile of 32 tokens ahead or behind: the copies, the step sizes
// (softplus, once a token and channel) and B and C as float32 before, the sum over the four warps' states, the skip, the gate and the
// stores after.  One block-wide barrier a tile.  A warp holds 32 channels rather than all states of eight: B and C then come by loads of
// one address (with four or eight lanes a channel, shared memory and shuffles took 96 to 113 clocks a token, now 66).
//
// The sums are those of selective_scan_kernel up to the order of a token's sum over the states: a warp's even and odd states, then the
// warps' sums in pairs.
//
// Bound by the issue slots, shared memory and the special-function pipe together: 66 clocks a token, of which ex2 takes 38, the
// recurrence's warp 25 issue slots and the others' share 28.  Measured (B200, us; in brackets the scan in chunks): 2,048 tokens x 4,096
// channels 86 (163), 8,192 channels 165 (296), 300 tokens x 4,096 18 (56), 64 tokens 10 (32).  With 8 or 2 tokens ahead 89 and 90.
#pragma once
#include "matrix_scan.cuh"

#define LOG2E_F 1.4426950408889634f

#define SP_TT 32   // tokens of a tile
#define SP_CH 32   // channels of a block
#define SP_N 16    // states a channel, padded with zeros
#define SP_R 4                  // warps that share the channels' states, SP_N / SP_R of them each
#define SP_SCAN (SP_CH * SP_R)  // threads that run the recurrence
#define SP_HELP 512             // threads that do everything else
#define SP_AHEAD 4              // tokens whose decays and inputs are taken ahead of the states
#define SP_W (SP_TT * SP_CH / SP_HELP)  // channels of a token that one of the SP_HELP threads prepares and finishes
#define SP_SLOTS 5 // tiles of inputs: one whose gates are still to be taken, one that is scanned, one prepared, two on their way

// 2^x for x <= 0 by one approximate PTX instruction (a result below the smallest normal number is zero, which a decay of
// that size is for every state that float32 holds).
__device__ __forceinline__ float ex2_nonpositive(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void sp_copy16(uint32_t dst, const void* src, bool real) {  // (zeros where there is nothing)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(real ? 16 : 0) : "memory");
}
// SP_W neighbouring values of shared memory.
__device__ __forceinline__ void sp_load(const float* p, float (&v)[SP_W]) {
#pragma unroll
    for (int i = 0; i < SP_W; i += 2) {
        const float2 q = *reinterpret_cast<const float2*>(p + i);
        v[i] = q.x, v[i + 1] = q.y;
    }
}
__device__ __forceinline__ void sp_load(const __nv_bfloat16* p, float (&v)[SP_W]) {
#pragma unroll
    for (int i = 0; i < SP_W; i += 2) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + i));
        v[i] = f.x, v[i + 1] = f.y;
    }
}
__device__ __forceinline__ void sp_store(float* p, const float (&v)[SP_W]) {
#pragma unroll
    for (int i = 0; i < SP_W; i += 2) *reinterpret_cast<float2*>(p + i) = make_float2(v[i], v[i + 1]);
}
__device__ __forceinline__ void sp_store(__nv_bfloat16* p, const float (&v)[SP_W]) {
#pragma unroll
    for (int i = 0; i < SP_W; i += 2) *reinterpret_cast<__nv_bfloat162*>(p + i) = __floats2bfloat162_rn(v[i], v[i + 1]);
}

template <typename T>
struct SelPromptShared {
    float dt[SP_SLOTS][SP_TT][SP_CH];
    T u[SP_SLOTS][SP_TT][SP_CH], z[SP_SLOTS][SP_TT][SP_CH], bc[SP_SLOTS][SP_TT][2 * SP_N];  // (bc: 2 N values a token, contiguous)
    float2 step[2][SP_TT][SP_CH];            // the step size, and it times u
    float b[2][SP_TT][SP_N], c[2][SP_TT][SP_N];
    float y[2][SP_R][SP_TT][SP_CH];          // a warp's share of the sum over the states
};

struct SelPromptToken {
    float2 decay[2], in[2], c[2];
};

template <typename T>
__global__ void __launch_bounds__(SP_SCAN + SP_HELP, 1)
selective_prompt_kernel(const T* __restrict__ u, long long u_stride, const float* __restrict__ dt_raw, const float* __restrict__ dt_bias,
                        const T* __restrict__ bc, long long bc_stride, const T* __restrict__ zg, long long z_stride,
                        const float* __restrict__ a_log, const float* __restrict__ d_skip, float* __restrict__ state, long long slot_stride,
                        T* __restrict__ out, const int* __restrict__ meta, const int* __restrict__ cu_tokens, const int* __restrict__ slots,
                        int inner, int N) {
    extern __shared__ __align__(16) unsigned char sp_raw[];
    SelPromptShared<T>& sm = *reinterpret_cast<SelPromptShared<T>*>(sp_raw);
    constexpr int PER16 = 16 / sizeof(T);  // values of a 16-byte copy
    const int tid = threadIdx.x, e = blockIdx.y, c0 = blockIdx.x * SP_CH;
    const bool scans = tid < SP_SCAN;
    pdl_launch_dependents();
    pdl_wait();
    if (e >= meta[META_NUM_ENTRIES]) return;
    const int first = cu_tokens[e], count = cu_tokens[e + 1] - first, tiles = (count + SP_TT - 1) / SP_TT;
    if (count <= 0) return;
    float* slot_state = state + (size_t)slots[e] * slot_stride;

    // ---- what the other sixteen warps do (ht: thread of them)
    const int ht = scans ? 0 : tid - SP_SCAN;
    // This thread's 16-byte copies of a tile: what from, to where in the first tile's place, how far on the next tile and place are.
    constexpr int DT = SP_TT * SP_CH / 4, ROWS = SP_TT * SP_CH / PER16, COPIES = (DT + 2 * ROWS + SP_TT * 2 * SP_N / PER16 + SP_HELP - 1) / SP_HELP;
    const unsigned char* from[COPIES];
    long long tile_step[COPIES];
    uint32_t to[COPIES], slot_step[COPIES];
    int token[COPIES];  // (beyond every count where there is nothing to copy)
#pragma unroll
    for (int j = 0; j < COPIES; ++j) {
        int i = ht + j * SP_HELP;
        const T* src = u;
        long long stride = 0;
        token[j] = 1 << 30, to[j] = 0, slot_step[j] = 0, tile_step[j] = 0, from[j] = (const unsigned char*)u;
        if (scans) continue;
        if (i < DT) {
            const int t = i / (SP_CH / 4), c = i % (SP_CH / 4) * 4;
            to[j] = (uint32_t)__cvta_generic_to_shared(&sm.dt[0][t][c]), slot_step[j] = sizeof(sm.dt[0]);
            if (c0 + c < inner)
                token[j] = t, from[j] = (const unsigned char*)(dt_raw + (size_t)(first + t) * inner + c0 + c), tile_step[j] = (long long)SP_TT * inner * 4;
        } else if ((i -= DT) < 2 * ROWS) {
            const bool gate = i >= ROWS;
            const int t = i % ROWS / (SP_CH / PER16), c = i % (SP_CH / PER16) * PER16;
            src = gate ? zg : u, stride = gate ? z_stride : u_stride;
            to[j] = (uint32_t)__cvta_generic_to_shared(gate ? &sm.z[0][t][c] : &sm.u[0][t][c]), slot_step[j] = sizeof(sm.u[0]);
            if (c0 + c < inner) token[j] = t, from[j] = (const unsigned char*)(src + (first + t) * stride + c0 + c), tile_step[j] = SP_TT * stride * sizeof(T);
        } else {
            i -= 2 * ROWS;
            const int per = 2 * N / PER16, t = i / per, k = i % per * PER16;
            if (t >= SP_TT) continue;
            to[j] = (uint32_t)__cvta_generic_to_shared(&sm.bc[0][t][k]), slot_step[j] = sizeof(sm.bc[0]);
            token[j] = t, from[j] = (const unsigned char*)(bc + (first + t) * bc_stride + k), tile_step[j] = SP_TT * bc_stride * sizeof(T);
        }
    }
    auto copy = [&](int tile) {  // the inputs of a tile (zeros beyond the last token and channel); always one group of copies
        const uint32_t slot = tile % SP_SLOTS;
#pragma unroll
        for (int j = 0; j < COPIES; ++j)
            if (slot_step[j]) {
                const bool real = tile * SP_TT + token[j] < count;
                sp_copy16(to[j] + slot * slot_step[j], real ? from[j] + tile * tile_step[j] : (const unsigned char*)u, real);
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int pt = ht / (SP_CH / SP_W), pc = ht % (SP_CH / SP_W) * SP_W;  // a token of the tile and SP_W channels: this thread's share of the two below
    float bias[SP_W], skip[SP_W];
    auto prepare = [&](int tile) {  // step sizes; B and C as float32
        if (tile >= tiles) return;
        const int slot = tile % SP_SLOTS, buf = tile & 1;
        float d[SP_W], uv[SP_W];
        sp_load(&sm.dt[slot][pt][pc], d);
        sp_load(&sm.u[slot][pt][pc], uv);
#pragma unroll
        for (int i = 0; i < SP_W; i += 2) {
            const float s0 = softplus_f(d[i] + bias[i]), s1 = softplus_f(d[i + 1] + bias[i + 1]);
            *reinterpret_cast<float4*>(&sm.step[buf][pt][pc + i]) = make_float4(s0, s0 * uv[i], s1, s1 * uv[i + 1]);
        }
        for (int i = ht; i < SP_TT * SP_N; i += SP_HELP) {
            const int t = i / SP_N, n = i % SP_N;
            sm.b[buf][t][n] = n < N ? to_float(sm.bc[slot][t][n]) : 0.f;
            sm.c[buf][t][n] = n < N ? to_float(sm.bc[slot][t][N + n]) : 0.f;
        }
    };
    auto finish = [&](int tile) {  // skip, gate, store
        if (tile < 0) return;
        const int slot = tile % SP_SLOTS, buf = tile & 1, t = tile * SP_TT + pt;
        if (t >= count || c0 + pc >= inner) return;
        float y[SP_W], uv[SP_W], zv[SP_W];
        float y1[SP_W], y2[SP_W], y3[SP_W];
        sp_load(&sm.y[buf][0][pt][pc], y), sp_load(&sm.y[buf][1][pt][pc], y1);
        sp_load(&sm.y[buf][2][pt][pc], y2), sp_load(&sm.y[buf][3][pt][pc], y3);
        sp_load(&sm.u[slot][pt][pc], uv);
        sp_load(&sm.z[slot][pt][pc], zv);
#pragma unroll
        for (int i = 0; i < SP_W; ++i) y[i] = fmaf(skip[i], uv[i], (y[i] + y1[i]) + (y2[i] + y3[i])) * silu_as<T>(zv[i]);
        T* dst = out + (size_t)(first + t) * inner + c0 + pc;
        sp_store(dst, y);
    };
    auto copies_done = [&]() {  // this thread's copies but the last two groups, then those of the other threads that copy
        asm volatile("cp.async.wait_group 2;" ::: "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(SP_HELP) : "memory");
    };

    // ---- what the recurrence's threads keep: states n0 .. n0 + 3 of channel c
    const int r = tid >> 5, cl = tid & 31, c = c0 + cl, n0 = 4 * r;
    const bool real = scans && c < inner;
    float2 A2[2], S[2];  // A log2(e)
    if (scans) {
        float a[4], s[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool in = real && n0 + i < N;
            a[i] = in ? -expf(a_log[(size_t)c * N + n0 + i]) * LOG2E_F : 0.f;
            s[i] = in ? slot_state[(size_t)c * N + n0 + i] : 0.f;
        }
        A2[0] = make_float2(a[0], a[1]), A2[1] = make_float2(a[2], a[3]);
        S[0] = make_float2(s[0], s[1]), S[1] = make_float2(s[2], s[3]);
        // states beyond N take no part (an infinite input would make a NaN of their zeros): their share of the sum is 0
        if (n0 >= N)
            for (int i = cl; i < 2 * SP_TT * SP_CH; i += 32) sm.y[i / (SP_TT * SP_CH)][r][i / SP_CH % SP_TT][i % SP_CH] = 0.f;
    } else {
#pragma unroll
        for (int i = 0; i < SP_W; ++i) {
            const bool in = c0 + pc + i < inner;
            bias[i] = in ? dt_bias[c0 + pc + i] : 0.f;
            skip[i] = in ? d_skip[c0 + pc + i] : 0.f;
        }
        copy(0), copy(1), copy(2);
        copies_done();
        prepare(0);
    }
    __syncthreads();

    for (int tile = 0; tile < tiles; ++tile) {
        const int buf = tile & 1;
        if (scans && n0 < N) {
            const int nt = min(SP_TT, count - tile * SP_TT);
            const float2* steps = &sm.step[buf][0][cl];
            const float* bs = &sm.b[buf][0][n0];
            const float* cs = &sm.c[buf][0][n0];
            float* ys = &sm.y[buf][r][0][cl];
            // What a token brings that does not wait for the state: decays, inputs, C.
            auto bring = [&](SelPromptToken& k, int t) {
                const float2 st = steps[t * SP_CH], st2 = make_float2(st.x, st.x), dx2 = make_float2(st.y, st.y);
                const float4 b4 = *reinterpret_cast<const float4*>(bs + t * SP_N), c4 = *reinterpret_cast<const float4*>(cs + t * SP_N);
                const float2 ea = mul2(st2, A2[0]), eb = mul2(st2, A2[1]);
                k.decay[0] = make_float2(ex2_nonpositive(ea.x), ex2_nonpositive(ea.y));
                k.decay[1] = make_float2(ex2_nonpositive(eb.x), ex2_nonpositive(eb.y));
                k.in[0] = mul2(dx2, make_float2(b4.x, b4.y)), k.in[1] = mul2(dx2, make_float2(b4.z, b4.w));
                k.c[0] = make_float2(c4.x, c4.y), k.c[1] = make_float2(c4.z, c4.w);
            };
            auto take = [&](const SelPromptToken& k, int t) {
                S[0] = fma2(k.decay[0], S[0], k.in[0]);
                S[1] = fma2(k.decay[1], S[1], k.in[1]);
                const float2 acc = fma2(S[1], k.c[1], mul2(S[0], k.c[0]));
                ys[t * SP_CH] = acc.x + acc.y;
            };
            if (nt == SP_TT) {
                // SP_AHEAD tokens are brought while as many before them are taken: a warp has its scheduler nearly to itself, and what
                // it waits for (shared memory, ex2) it must overlap with its own next tokens.
                SelPromptToken k[2][SP_AHEAD];
#pragma unroll
                for (int j = 0; j < SP_AHEAD; ++j) bring(k[0][j], j);
#pragma unroll
                for (int g = 0; g < SP_TT / SP_AHEAD; ++g) {
                    if (g + 1 < SP_TT / SP_AHEAD)
#pragma unroll
                        for (int j = 0; j < SP_AHEAD; ++j) bring(k[(g + 1) & 1][j], (g + 1) * SP_AHEAD + j);
#pragma unroll
                    for (int j = 0; j < SP_AHEAD; ++j) take(k[g & 1][j], g * SP_AHEAD + j);
                }
            } else {
                for (int t = 0; t < nt; ++t) {
                    SelPromptToken k;
                    bring(k, t);
                    take(k, t);
                }
            }
        } else if (!scans) {
            finish(tile - 1);
            copy(tile + 3);
            copies_done();
            prepare(tile + 1);
        }
        __syncthreads();
    }
    if (!scans) {
        finish(tiles - 1);
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (real) {
        const float s[4] = {S[0].x, S[0].y, S[1].x, S[1].y};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (n0 + i < N) slot_state[(size_t)c * N + n0 + i] = s[i];
    }
}

// Whether the kernel above takes these inputs: eight or sixteen states, rows that start on 16 bytes.
static bool selective_prompt_takes(const void* u, long long u_stride, const float* dt_raw, const void* bc, long long bc_stride, const void* zg,
                                   long long z_stride, int dtype, const void* out, int inner, int N) {
    const int per16 = dtype == DT_F32 ? 4 : 8;
    return (N == 8 || N == 16) && inner % 8 == 0 && u_stride % per16 == 0 && z_stride % per16 == 0 && bc_stride % per16 == 0 &&
           (((uintptr_t)u | (uintptr_t)dt_raw | (uintptr_t)bc | (uintptr_t)zg | (uintptr_t)out) & 15) == 0;
}

template <typename T>
static int selective_prompt(const void* u, long long u_stride, const float* dt_raw, const float* dt_bias, const void* bc, long long bc_stride,
                            const void* zg, long long z_stride, const float* a_log, const float* d_skip, float* state, long long slot_stride,
                            void* out, const int* meta, const int* cu_tokens, const int* slots, int S, int inner, int N, cudaStream_t stream) {
    constexpr size_t smem = sizeof(SelPromptShared<T>);
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(selective_prompt_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    return (int)launch_kernel(selective_prompt_kernel<T>, dim3((inner + SP_CH - 1) / SP_CH, S), SP_SCAN + SP_HELP, smem, stream, (const T*)u, u_stride, dt_raw,
                              dt_bias, (const T*)bc, bc_stride, (const T*)zg, z_stride, a_log, d_skip, state, slot_stride, (T*)out, meta,
                              cu_tokens, slots, inner, N);
}
