// Recurrent mixers whose state is a matrix per head or per channel and whose decay differs from row to row:
//  * gated linear attention: per head S_t = diag(a_t) S_(t-1) + k_t v_t^T, o_t = S_t^T q_t, a_t = sigmoid(z_t)^(1/tau);
//  * the selective scan of the Mamba kind: per channel c and state n, S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c u_c B_n,
//    y_c = sum_n S[c, n] C_n + D_c u_c, times silu(z_c);
//  * the norm per head with a weight shared by the heads, times silu(gate), behind the first.
// Storage of projections is float32 or bfloat16; states, decays, step sizes, gates and norms are float32 always.  A
// request's tokens run in order from its state slot (pass 0), or, for long portions, cut into chunks of time that run
// side by side: pass 1 runs every chunk but the last from a zero state and leaves its end state and what its decays
// amount to, a small kernel chains the chunks' start states in order, pass 3 runs every chunk again from its start
// state and writes the outputs, the last chunk the slot.  Every sum runs in an order that depends on the sizes only; the norm of
// bfloat16 rows takes one of two orders by the number of rows.
#include "matrix_scan.cuh"
#include "row_scan.cuh"
#include "selective_prompt.cuh"

int g_use_pdl = 1;
extern "C" void kernels_set_pdl(int mode) { g_use_pdl = mode; }

// ----------------------------------------------------------------------------- gated linear attention
// q, k [T, heads * N], v [T, heads * P]: slices of wider rows (strides in elements); z float32 [T, heads * N], the decay's
// logits before their bias.  state [slots][heads][N][P]; o float32 [T, heads * P].

extern "C" size_t gla_scan_scratch_floats(int S, int heads, int N, int P, int max_chunks) {
    return scan_scratch_floats<SCAN_DECAY>(S, heads, N, P, max_chunks);
}

// mode bit 0: the decay is a constant per head, z_bias[h] (float32 [heads]; z is not read); bit 1: q, k and v pass through
// SiLU as they are loaded.
extern "C" int gla_scan_mode(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                             int dtype, const float* z, long long z_stride, const float* z_bias, float tau, float q_scale,
                             float* state, long long slot_stride, float* o, const int* meta, const int* cu_tokens, const int* slots,
                             int S, int heads, int N, int P, int chunk_len, int max_chunks, float* scratch, int mode,
                             cudaStream_t stream) {
    if (S > 0 && ((mode & 1) ? !z_bias : !z)) return (int)cudaErrorInvalidValue;
    const ScanArgs a = {q, k, v, q_stride, k_stride, v_stride, dtype, z, z_bias, z_stride, tau, q_scale, state, slot_stride, o, meta,
                        cu_tokens, slots, S, heads, N, P, chunk_len, max_chunks, scratch, mode, {}};
    return run_matrix_scan<SCAN_DECAY>(a, stream);
}

extern "C" int gla_scan(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                        int dtype, const float* z, long long z_stride, const float* z_bias, float tau, float q_scale,
                        float* state, long long slot_stride, float* o, const int* meta, const int* cu_tokens, const int* slots,
                        int S, int heads, int N, int P, int chunk_len, int max_chunks, float* scratch, cudaStream_t stream) {
    return gla_scan_mode(q, q_stride, k, k_stride, v, v_stride, dtype, z, z_stride, z_bias, tau, q_scale, state, slot_stride, o, meta,
                         cu_tokens, slots, S, heads, N, P, chunk_len, max_chunks, scratch, 0, stream);
}

// The same for bfloat16 prompts with decay logits, as matrix products over chunks of RCHUNK tokens (row_scan.cuh).  max_chunks: at least
// the chunks of all entries together.  gla_row_scan_head_floats: scratch of one head, 0 where the sizes or addresses are not served;
// with scratch for fewer than all heads they run in rounds.
extern "C" size_t gla_row_scan_head_floats(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                                           const float* o, int N, int P, int max_chunks) {
    return chunk_scan_takes(q, k, v, q_stride, k_stride, v_stride, o, N, P) && max_chunks <= 65535 ? row_scan_head_floats(N, P, max_chunks) : 0;
}

extern "C" int gla_row_scan(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                            const float* z, long long z_stride, const float* z_bias, float tau, float q_scale, float* state,
                            long long slot_stride, float* o, const int* meta, const int* cu_tokens, const int* slots, int S, int heads,
                            int N, int P, int max_chunks, float* scratch, size_t scratch_floats, cudaStream_t stream) {
    if (S > 0 && (!z || tau <= 0.f)) return (int)cudaErrorInvalidValue;
    RowScanArgs a = {};
    a.q = (const __nv_bfloat16*)q, a.k = (const __nv_bfloat16*)k, a.v = (const __nv_bfloat16*)v;
    a.q_stride = q_stride, a.k_stride = k_stride, a.v_stride = v_stride;
    a.z = z, a.z_stride = z_stride, a.z_bias = z_bias, a.inv_tau = 1.f / tau, a.q_scale = q_scale;
    a.state = state, a.slot_stride = slot_stride, a.o = o;
    a.meta = meta, a.cu_tokens = cu_tokens, a.slots = slots;
    a.S = S, a.heads = heads, a.N = N, a.P = P, a.max_chunks = max_chunks;
    return row_scan<ROW_DECAY>(a, scratch, scratch_floats, stream);
}

// ----------------------------------------------------------------------------- norm per head, shared weight, gate
// out[t, h, :] = o[t, h, :] / sqrt(mean(o[t, h, :]^2) + eps) * w * silu(g[t, h, :]); o float32 [T, heads * P], g a slice of
// wider rows, w float32 [P].  A warp a (token, head).
template <typename T>
__global__ void __launch_bounds__(128)
head_norm_gate_kernel(const float* __restrict__ o, const T* __restrict__ g, long long g_stride, const float* __restrict__ w,
                      float eps, T* __restrict__ out, const int* __restrict__ meta, int heads, int P) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, lane = threadIdx.x & 31, h = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= meta[META_NUM_TOKENS] || h >= heads) return;
    const float* row = o + ((size_t)t * heads + h) * P;
    const T* gate = g + (size_t)t * g_stride + (size_t)h * P;
    float ss = 0.f;
    for (int i = lane; i < P; i += 32) ss = fmaf(row[i], row[i], ss);
    ss = warp_sum(ss);
    const float inv = rsqrtf(ss / (float)P + eps);
    T* dst = out + ((size_t)t * heads + h) * P;
    for (int i = lane; i < P; i += 32) dst[i] = from_float<T>(row[i] * inv * w[i] * silu_f(to_float(gate[i])));
}

// The same with at most 128 K values a head, four consecutive ones a lane and 16-byte accesses, all loads ahead of the sum.
template <typename T, int K>
__global__ void __launch_bounds__(256)
head_norm_gate_vec_kernel(const float* __restrict__ o, const T* __restrict__ g, long long g_stride, const float* __restrict__ w,
                          float eps, T* __restrict__ out, const int* __restrict__ meta, int heads, int P) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), t = item / heads, h = item % heads;
    if (t >= meta[META_NUM_TOKENS]) return;
    const float* row = o + (size_t)item * P;
    const T* gate = g + (size_t)t * g_stride + (size_t)h * P;
    float v[K][4], gv[K][4], ss = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = (lane + 32 * k) * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[k][j] = gv[k][j] = 0.f;
        if (i < P) load4(row + i, v[k]), load4(gate + i, gv[k]);
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) ss = fmaf(v[k][j], v[k][j], ss);
    const float inv = rsqrtf(warp_sum(ss) / (float)P + eps);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = (lane + 32 * k) * 4;
        if (i >= P) continue;
        float wv[4];
        load4(w + i, wv);
#pragma unroll
        for (int j = 0; j < 4; ++j) wv[j] = v[k][j] * inv * wv[j] * silu_as<T>(gv[k][j]);
        store4(out + (size_t)item * P + i, wv);
    }
}

template <typename T>
static int launch_head_norm_vec(const float* o, const T* g, long long g_stride, const float* w, float eps, T* out, const int* meta, int rows,
                                int heads, int P, cudaStream_t stream) {
    const int blocks = (rows * heads + 7) / 8;
    if (P <= 128) return (int)launch_kernel(head_norm_gate_vec_kernel<T, 1>, blocks, 256, 0, stream, o, g, g_stride, w, eps, out, meta, heads, P);
    if (P <= 256) return (int)launch_kernel(head_norm_gate_vec_kernel<T, 2>, blocks, 256, 0, stream, o, g, g_stride, w, eps, out, meta, heads, P);
    return (int)launch_kernel(head_norm_gate_vec_kernel<T, 4>, blocks, 256, 0, stream, o, g, g_stride, w, eps, out, meta, heads, P);
}

extern "C" int head_norm_gate(const float* o, const void* g, int dtype, long long g_stride, const float* w, float eps, void* out,
                              const int* meta, int T, int heads, int P, cudaStream_t stream) {
    if (T <= 0) return 0;
    // (float32 keeps one order of a row's sum, however many rows there are)
    if (dtype != DT_F32 && (long)T * heads >= 8 * multiprocessors() && P % 4 == 0 && P <= 512 && g_stride % 4 == 0 &&
        (((uintptr_t)o | (uintptr_t)w) & 15) == 0 && (((uintptr_t)g | (uintptr_t)out) & 7) == 0)
        return launch_head_norm_vec(o, (const __nv_bfloat16*)g, g_stride, w, eps, (__nv_bfloat16*)out, meta, T, heads, P, stream);
    const dim3 grid(T, (heads + 3) / 4);
    if (dtype == DT_F32)
        return (int)launch_kernel(head_norm_gate_kernel<float>, grid, 128, 0, stream, o, (const float*)g, g_stride, w, eps,
                                  (float*)out, meta, heads, P);
    return (int)launch_kernel(head_norm_gate_kernel<__nv_bfloat16>, grid, 128, 0, stream, o, (const __nv_bfloat16*)g, g_stride, w,
                              eps, (__nv_bfloat16*)out, meta, heads, P);
}

// ----------------------------------------------------------------------------- selective scan
// u [T, inner] (after convolution and activation), zg [T, inner] (the gate's input): slices of wider rows; dt_raw float32
// [T, inner] (softplus(dt_raw + dt_bias) is taken here); B at bc, C at bc + N of a row of bc_stride elements; a_log [inner, N];
// state [slots][inner][N]; out [T, inner] = (sum_n S[c, n] C_n + D_c u_c) * silu(zg_c).
// One block per (channel block, entry[, chunk]).  Thread (c, r) keeps NPT states n = r * NPT .. of channel c, as pairs of
// neighbouring states that one two-wide instruction updates.  y is the even states' sum plus the odd states', each in
// ascending order, then the R threads' sums by halving.  B and C of SEL_TT tokens are staged in shared memory; the channel's
// own u, step size and gate input of those tokens go straight into the thread's registers.  Pass 1 leaves the
// step sizes of its chunks for pass 3, which computes those of an entry's last chunk itself.
// Bound by the special-function pipe (an ex2 per state, token and pass: 60 of the us below) and the issue slots beside it:
// tiles of 8 tokens (128 registers, four blocks a multiprocessor; tiles of 16 took 236, two blocks) and then the softplus
// once instead of in both passes and bfloat16 gates by the reciprocal instruction took the scan of 2,048 tokens of 4,096
// channels x 16 states from 175 over 156 to 147 us, of 8,192 channels from 324 over 292 to 272, and 200 tokens of 4,096
// from 53 over 49 to 44.  Loading the next tile ahead (4 to 8 tokens, B and C of 64 at a time) gave 147 to 163 us.
#define SEL_TT 8

template <typename T, int NPT, int PASS>
__global__ void __launch_bounds__(128, NPT <= 16 ? 4 : 1)
selective_scan_kernel(const T* __restrict__ u, long long u_stride, const float* __restrict__ dt_raw,
                      const float* __restrict__ dt_bias, const T* __restrict__ bc, long long bc_stride,
                      const T* __restrict__ zg, long long z_stride, const float* __restrict__ a_log,
                      const float* __restrict__ d_skip, float* __restrict__ state, long long slot_stride, T* __restrict__ out,
                      const int* __restrict__ meta, const int* __restrict__ cu_tokens, const int* __restrict__ slots,
                      int inner, int N, int R, int CPB, int chunk_len, int max_chunks, float* __restrict__ scratch,
                      float* __restrict__ dt_sums, float* __restrict__ steps) {
    constexpr bool WRITE_Y = PASS != 1;
    extern __shared__ __align__(16) float sm[];
    const int SL = R > 1 ? NPT + 4 : NPT, NL = R * NPT, NP = R * SL;
    float* Bs = sm;                      // [SEL_TT][NP]
    float* Cs = Bs + SEL_TT * NP;        // [SEL_TT][NP]
    const int e = blockIdx.y, ch = blockIdx.z;
    const int tid = threadIdx.x, cl = tid / R, r = tid % R, c = blockIdx.x * CPB + cl;
    const bool real = cl < CPB && c < inner;
    // the weights come before the wait: no kernel writes them
    float2 A2[NPT / 2];  // A log2(e), pairs of neighbouring states
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
        const int n = r * NPT + i;
        const float a = (real && n < N) ? -expf(a_log[(size_t)c * N + n]) * LOG2E_F : 0.f;
        if (i & 1) A2[i / 2].y = a; else A2[i / 2].x = a;
    }
    const float dskip = real ? d_skip[c] : 0.f, dtb = real ? dt_bias[c] : 0.f;
    pdl_launch_dependents();
    pdl_wait();
    if (e >= meta[META_NUM_ENTRIES]) return;
    const int first = cu_tokens[e], count = cu_tokens[e + 1] - first;
    const int nchunks = PASS == 0 ? 1 : (count + chunk_len - 1) / chunk_len;
    if (ch >= nchunks || (PASS == 1 && ch == nchunks - 1)) return;
    const bool kept = PASS == 3 && ch < nchunks - 1;  // whether pass 1 has left this chunk's step sizes
    const int t0 = first + (PASS == 0 ? 0 : ch * chunk_len), t1 = PASS == 0 ? first + count : min(first + count, t0 + chunk_len);
    const size_t HS = (size_t)inner * N;
    float* slot_state = state + (size_t)slots[e] * slot_stride;
    float* chunk_state = scratch ? scratch + ((size_t)e * max_chunks + ch) * HS : nullptr;
    const float* init = PASS == 0 ? slot_state : (PASS == 3 ? chunk_state : nullptr);
    float2 S[NPT / 2];
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
        const int n = r * NPT + i;
        const float s0 = (init && real && n < N) ? init[(size_t)c * N + n] : 0.f;
        if (i & 1) S[i / 2].y = s0; else S[i / 2].x = s0;
    }
    float dt_sum = 0.f;
    for (int tb = t0; tb < t1; tb += SEL_TT) {
        const int nt = min(SEL_TT, t1 - tb);
        // this thread's channel of the tile's tokens, straight into registers: every load is on its way before the
        // first is used (the R threads of a channel read the same addresses)
        T ur[SEL_TT], zr[SEL_TT];
        float dr[SEL_TT];
#pragma unroll
        for (int tt = 0; tt < SEL_TT; ++tt) {
            const bool in = real && tt < nt;
            const size_t t = (size_t)(tb + tt);
            ur[tt] = in ? u[t * u_stride + c] : from_float<T>(0.f);
            dr[tt] = in ? (kept ? steps : dt_raw)[t * inner + c] : 0.f;
            if (WRITE_Y) zr[tt] = in ? zg[t * z_stride + c] : from_float<T>(0.f);
        }
        __syncthreads();
        for (int idx = tid; idx < nt * NL; idx += blockDim.x) {
            const int tt = idx / NL, n = idx % NL, at = tt * NP + (n / NPT) * SL + n % NPT;
            const T* row = bc + (size_t)(tb + tt) * bc_stride;
            Bs[at] = n < N ? to_float(row[n]) : 0.f;
            Cs[at] = n < N ? to_float(row[N + n]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int tt = 0; tt < SEL_TT; ++tt) {
            if (tt >= nt) break;
            const float uv = to_float(ur[tt]), step = kept ? dr[tt] : (real ? softplus_f(dr[tt] + dtb) : 0.f);
            if (PASS == 1 && real && r == 0) steps[(size_t)(tb + tt) * inner + c] = step;
            const float dx = step * uv;
            const float* Bt = Bs + tt * NP + r * SL;
            const float* Ct = Cs + tt * NP + r * SL;
            const float2 st2 = make_float2(step, step), dx2 = make_float2(dx, dx);
            float2 acc2 = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < NPT / 2; i += 2) {  // two pairs of neighbouring states a round
                const float4 b4 = *reinterpret_cast<const float4*>(Bt + 2 * i);
                float2 ea = mul2(st2, A2[i]), eb = mul2(st2, A2[i + 1]);
                ea = make_float2(ex2_nonpositive(ea.x), ex2_nonpositive(ea.y));
                eb = make_float2(ex2_nonpositive(eb.x), ex2_nonpositive(eb.y));
                S[i] = fma2(ea, S[i], mul2(dx2, make_float2(b4.x, b4.y)));
                S[i + 1] = fma2(eb, S[i + 1], mul2(dx2, make_float2(b4.z, b4.w)));
                if (WRITE_Y) {
                    const float4 c4 = *reinterpret_cast<const float4*>(Ct + 2 * i);
                    acc2 = fma2(S[i], make_float2(c4.x, c4.y), acc2);
                    acc2 = fma2(S[i + 1], make_float2(c4.z, c4.w), acc2);
                }
            }
            float acc = acc2.x + acc2.y;  // the even states' sum plus the odd states'
            if (WRITE_Y) {
                for (int s = R >> 1; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
                if (real && r == 0) {
                    const float y = fmaf(dskip, uv, acc);
                    out[(size_t)(tb + tt) * inner + c] = from_float<T>(y * silu_as<T>(to_float(zr[tt])));
                }
            }
            dt_sum += step;
        }
    }
    float* fin = PASS == 1 ? chunk_state + HS : ((PASS == 0 || ch == nchunks - 1) ? slot_state : nullptr);
    if (fin && real) {
#pragma unroll
        for (int i = 0; i < NPT; ++i) {
            const int n = r * NPT + i;
            if (n < N) fin[(size_t)c * N + n] = (i & 1) ? S[i / 2].y : S[i / 2].x;
        }
    }
    if (PASS == 1 && real && r == 0) dt_sums[((size_t)e * max_chunks + ch) * inner + c] = dt_sum;
}

// scratch[e, 0] = the slot's state; scratch[e, c] = exp(A * (sum of the steps of chunk c - 1)) * scratch[e, c - 1] + scratch[e, c].
__global__ void __launch_bounds__(256)
selective_chunk_states_kernel(const float* __restrict__ state, long long slot_stride, float* __restrict__ scratch,
                              const float* __restrict__ dt_sums, const float* __restrict__ a_log, const int* __restrict__ meta,
                              const int* __restrict__ cu_tokens, const int* __restrict__ slots, int inner, int N, int chunk_len,
                              int max_chunks) {
    pdl_launch_dependents();
    pdl_wait();
    const int e = blockIdx.y;
    if (e >= meta[META_NUM_ENTRIES]) return;
    const int count = cu_tokens[e + 1] - cu_tokens[e], nchunks = (count + chunk_len - 1) / chunk_len;
    const long long HS = (long long)inner * N, i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= HS) return;
    const int c = (int)(i / N);
    const float a2 = -expf(a_log[i]) * LOG2E_F;
    float s = state[(size_t)slots[e] * slot_stride + i];
    scratch[((size_t)e * max_chunks) * HS + i] = s;
    for (int k = 1; k < nchunks; ++k) {
        float* at = scratch + ((size_t)e * max_chunks + k) * HS + i;
        s = fmaf(exp2f(a2 * dt_sums[((size_t)e * max_chunks + k - 1) * inner + c]), s, *at);
        *at = s;
    }
}

extern "C" size_t selective_scan_scratch_floats(int T, int S, int inner, int N, int max_chunks) {
    return (size_t)S * max_chunks * ((size_t)inner * N + inner) + (size_t)T * inner;
}

// The same in one pass, in order, for prompts (selective_prompt.cuh), and whether it takes these inputs.
extern "C" int selective_scan_prompt_takes(const void* u, long long u_stride, const float* dt_raw, const void* bc, long long bc_stride,
                                           const void* zg, long long z_stride, int dtype, const void* out, int inner, int N) {
    return selective_prompt_takes(u, u_stride, dt_raw, bc, bc_stride, zg, z_stride, dtype, out, inner, N);
}
extern "C" int selective_scan_prompt(const void* u, long long u_stride, const float* dt_raw, const float* dt_bias, const void* bc,
                                     long long bc_stride, const void* zg, long long z_stride, int dtype, const float* a_log,
                                     const float* d_skip, float* state, long long slot_stride, void* out, const int* meta,
                                     const int* cu_tokens, const int* slots, int S, int inner, int N, cudaStream_t stream) {
    if (S <= 0) return 0;
    if (!selective_prompt_takes(u, u_stride, dt_raw, bc, bc_stride, zg, z_stride, dtype, out, inner, N)) return (int)cudaErrorInvalidValue;
    if (dtype == DT_F32)
        return selective_prompt<float>(u, u_stride, dt_raw, dt_bias, bc, bc_stride, zg, z_stride, a_log, d_skip, state, slot_stride, out, meta,
                                       cu_tokens, slots, S, inner, N, stream);
    return selective_prompt<__nv_bfloat16>(u, u_stride, dt_raw, dt_bias, bc, bc_stride, zg, z_stride, a_log, d_skip, state, slot_stride, out,
                                           meta, cu_tokens, slots, S, inner, N, stream);
}

extern "C" int selective_scan(const void* u, long long u_stride, const float* dt_raw, const float* dt_bias, const void* bc,
                              long long bc_stride, const void* zg, long long z_stride, int dtype, const float* a_log,
                              const float* d_skip, float* state, long long slot_stride, void* out, const int* meta,
                              const int* cu_tokens, const int* slots, int S, int inner, int N, int chunk_len, int max_chunks,
                              float* scratch, cudaStream_t stream) {
    if (S <= 0) return 0;
    int NPT = 0, R = 0, CPB = 0;
    if (!rec_geometry(N, inner, &NPT, &R, &CPB)) return (int)cudaErrorInvalidValue;
    if (CPB * R > 128) CPB = 128 / R > 0 ? 128 / R : 1;  // 128 threads a block: more blocks for few requests
    const int blocks = (inner + CPB - 1) / CPB, threads = ((CPB * R + 31) / 32) * 32;
    const size_t smem = (size_t)(2 * SEL_TT * R * (R > 1 ? NPT + 4 : NPT)) * sizeof(float);
    if (smem > 96 * 1024) return (int)cudaErrorInvalidValue;
    float* dt_sums = scratch ? scratch + (size_t)S * max_chunks * (size_t)inner * N : nullptr;
    float* steps = dt_sums ? dt_sums + (size_t)S * max_chunks * inner : nullptr;  // [T, inner]
#define SEL_CASE(TT, K, pass, chunks)                                                                                    \
    case K: {                                                                                                              \
        static size_t configured = 0;                                                                                      \
        if (smem > 48 * 1024 && smem > configured) {                                                                       \
            cudaError_t ce = cudaFuncSetAttribute(selective_scan_kernel<TT, K, pass>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            if (ce != cudaSuccess) return (int)ce;                                                                         \
            configured = smem;                                                                                             \
        }                                                                                                                  \
        err = (int)launch_kernel(selective_scan_kernel<TT, K, pass>, dim3(blocks, S, chunks), threads, smem, stream, (const TT*)u, u_stride, \
                                 dt_raw, dt_bias, (const TT*)bc, bc_stride, (const TT*)zg, z_stride, a_log, d_skip, state,       \
                                 slot_stride, (TT*)out, meta, cu_tokens, slots, inner, N, R, CPB, chunk_len, max_chunks,   \
                                 scratch, dt_sums, steps);                                                                        \
        break;                                                                                                             \
    }
#define SEL_PASS(TT, pass, chunks)                                                                                       \
    switch (NPT) { SEL_CASE(TT, 8, pass, chunks) SEL_CASE(TT, 16, pass, chunks) SEL_CASE(TT, 32, pass, chunks) SEL_CASE(TT, 64, pass, chunks) }
    int err = 0;
    if (chunk_len <= 0 || max_chunks <= 1 || !scratch) {
        if (dtype == DT_F32) { SEL_PASS(float, 0, 1) } else { SEL_PASS(__nv_bfloat16, 0, 1) }
        return err;
    }
    if (dtype == DT_F32) { SEL_PASS(float, 1, max_chunks) } else { SEL_PASS(__nv_bfloat16, 1, max_chunks) }
    if (err) return err;
    const long long HS = (long long)inner * N;
    err = (int)launch_kernel(selective_chunk_states_kernel, dim3((unsigned)((HS + 255) / 256), S), 256, 0, stream,
                             (const float*)state, slot_stride, scratch, (const float*)dt_sums, a_log, meta, cu_tokens, slots,
                             inner, N, chunk_len, max_chunks);
    if (err) return err;
    if (dtype == DT_F32) { SEL_PASS(float, 3, max_chunks) } else { SEL_PASS(__nv_bfloat16, 3, max_chunks) }
    return err;
#undef SEL_PASS
#undef SEL_CASE
}
