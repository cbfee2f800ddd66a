// A state-space mixer's decode step: one token of every entry through the convolution and the recurrence in one launch (as kernels of their
// own, ssm.cu, each starts, waits for a round trip to memory and hands over some hundred KB).  A block is a head of an entry: it keeps
// the head's matrix in registers, four neighbouring columns of every RG-th row a thread, and takes the head's columns of x and the group's B
// and C through the convolution itself.  The heads of a group share B and C, so nobody may change the ring while another block may still
// read it: the gated norm's launch, the next one, writes the new row (ring_row).
// In float32 the sum over a column's rows is taken in the scan's own order (ssm_scan_kernel: R shares of NPT rows, each in order, then by
// halving) from a copy of the new matrix in shared memory: a request's bits do not depend on how many others bring a token, which is
// what chooses this kernel.  In bfloat16 a thread sums the rows that it keeps.
// Bound by fixed cost for few entries and by the state's bytes for many.  The state is asked into the L2 before the wait for the
// linear ahead: a hint, so it may run before that state's last writer has finished.
// Measured, a whole layer (both linears too) of width 2,048 (64 heads of 128 x 64), us, in brackets the three kernels: 1 request 22.7 (26.8), 4
// 24.6 (27.0), 16 34.9 (39.0), 40 67.6 (68.5), 64 89.5 (85.9); width 4,096 (128 heads) 1 47.5 (53.1), 16 73.7 (77.9), 40 136 (130).  With many
// blocks the convolution of B and C, which every head repeats, costs more than the launch; how many are worth it is the caller's rule.
#pragma once
#include "common.cuh"

#define TOKEN_ROWS 8     // rows of the state a thread keeps

template <typename T>
struct SsmToken {
    const T *u, *dt;                             // slices of wider rows
    long long u_stride, dt_stride;
    const float *conv_w, *conv_b;                // [taps, channels], [channels] (or null)
    const float* ring;                           // [slots][taps - 1][channels]
    long long ring_stride;
    const float *dt_bias, *a_log, *d_skip;
    float* state;                                // [slots][heads][N][P]
    long long slot_stride;
    float* y;                                    // [T, heads * P]
    const int *meta, *positions, *cu_tokens, *slots;
    int heads, N, groups, taps;
    int R, NPT;                                  // float32: the scan's shares of a column (R * P at most 512)
};

template <typename T, int PQ>
__global__ void __launch_bounds__(256)
ssm_token_kernel(const __grid_constant__ SsmToken<T> A) {
    constexpr int P = PQ * 4, RG = 256 / PQ, MAX_N = RG * TOKEN_ROWS, ITEMS = (P + 2 * MAX_N + 255) / 256;
    constexpr bool IN_ORDER = sizeof(T) == 4;
    __shared__ __align__(16) float xs[P], part[IN_ORDER ? 512 / P : 8][P], bc[2 * MAX_N], mat[IN_ORDER ? MAX_N * P : 4];
    const int h = blockIdx.x, e = blockIdx.y, g = h / (A.heads / A.groups), tid = threadIdx.x, N = A.N;
    const int inner = A.heads * P, channels = inner + 2 * A.groups * N, R = A.taps - 1;
    if (e >= A.meta[META_NUM_ENTRIES]) {  // (padding; it waits all the same, so that no block is done before the linear ahead)
        pdl_wait();
        return;
    }
    const int t = A.cu_tokens[e], p = A.positions[t], slot = A.slots[e];
    float* S = A.state + (size_t)slot * A.slot_stride + (size_t)h * N * P;
    for (int i = tid * 32; i < N * P; i += 256 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(S + i));
    // my channels: item i < P is a column of x, the others the group's B and C
    int c[ITEMS];
    float w[ITEMS][4], acc[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int i = tid + k * 256, b = i - P;
        c[k] = i < P ? h * P + i : (b < 2 * N ? inner + (b < N ? g * N + b : A.groups * N + g * N + b - N) : -1);
        acc[k] = c[k] >= 0 && A.conv_b ? A.conv_b[c[k]] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) w[k][j] = c[k] >= 0 && j < A.taps ? A.conv_w[(size_t)j * channels + c[k]] : 0.f;
    }
    const float dt_bias = A.dt_bias[h], rate = expf(A.a_log[h]), dskip = A.d_skip[h];
    pdl_wait();
    pdl_launch_dependents();
    const int q = tid % PQ, rg = tid / PQ;
    const float raw = to_float(A.dt[(size_t)t * A.dt_stride + h]) + dt_bias;
    float u[ITEMS][4];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int back = R - j, src = p - back;
            u[k][j] = 0.f;
            if (c[k] >= 0 && back == 0) u[k][j] = to_float(A.u[(size_t)t * A.u_stride + c[k]]);
            else if (c[k] >= 0 && back > 0 && src >= 0) u[k][j] = A.ring[(size_t)slot * A.ring_stride + (size_t)(src % R) * channels + c[k]];
        }
    }
    float4 s[TOKEN_ROWS];
#pragma unroll
    for (int i = 0; i < TOKEN_ROWS; ++i) {
        const int n = rg + RG * i;
        s[i] = n < N ? *reinterpret_cast<const float4*>(S + (size_t)n * P + q * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (c[k] < 0) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)  // the arithmetic and its order are those of the convolution's own kernels
            if (j < A.taps && p - (R - j) >= 0) acc[k] = fmaf(w[k][j], u[k][j], acc[k]);
        const float v = to_float(from_float<T>(acc[k] / (1.f + expf(-acc[k]))));
        const int i = tid + k * 256;
        if (i < P) xs[i] = v;
        else bc[i - P] = v;
    }
    const float step = raw > 20.f ? raw : log1pf(expf(raw));  // softplus; beyond 20 the difference is below rounding
    const float dec = expf(-rate * step);
    __syncthreads();
    const float4 x = *reinterpret_cast<const float4*>(xs + q * 4), dx = make_float4(step * x.x, step * x.y, step * x.z, step * x.w);
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < TOKEN_ROWS; ++i) {
        const int n = rg + RG * i;
        if (n >= N) break;
        const float bn = bc[n], cn = bc[N + n];
        s[i].x = fmaf(dec, s[i].x, bn * dx.x), s[i].y = fmaf(dec, s[i].y, bn * dx.y);
        s[i].z = fmaf(dec, s[i].z, bn * dx.z), s[i].w = fmaf(dec, s[i].w, bn * dx.w);
        *reinterpret_cast<float4*>(S + (size_t)n * P + q * 4) = s[i];
        if (IN_ORDER) {
            *reinterpret_cast<float4*>(mat + n * P + q * 4) = s[i];
            continue;
        }
        y.x = fmaf(s[i].x, cn, y.x), y.y = fmaf(s[i].y, cn, y.y), y.z = fmaf(s[i].z, cn, y.z), y.w = fmaf(s[i].w, cn, y.w);
    }
    if (IN_ORDER) {
        __syncthreads();
        for (int i = tid; i < A.R * P; i += 256) {
            const int col = i % P, r = i / P;
            float v = 0.f;
#pragma unroll 8
            for (int j = 0; j < A.NPT; ++j) {
                const int n = r * A.NPT + j;
                if (n < N) v = fmaf(mat[n * P + col], bc[N + n], v);
            }
            part[r][col] = v;
        }
        __syncthreads();
        if (tid < P) {
            for (int o = A.R >> 1; o > 0; o >>= 1)
                for (int r = 0; r < o; ++r) part[r][tid] += part[r + o][tid];
            A.y[(size_t)t * inner + h * P + tid] = fmaf(dskip, xs[tid], part[0][tid]);
        }
        return;
    }
#pragma unroll
    for (int o = PQ; o < 32; o <<= 1) {
        y.x += __shfl_xor_sync(0xffffffffu, y.x, o), y.y += __shfl_xor_sync(0xffffffffu, y.y, o);
        y.z += __shfl_xor_sync(0xffffffffu, y.z, o), y.w += __shfl_xor_sync(0xffffffffu, y.w, o);
    }
    const int lane = tid & 31, warp = tid >> 5;
    if (lane < PQ) *reinterpret_cast<float4*>(&part[warp][q * 4]) = y;
    __syncthreads();
    if (tid < P) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) v += part[k][tid];
        A.y[(size_t)t * inner + h * P + tid] = fmaf(dskip, xs[tid], v);
    }
}

// The convolution's new ring rows: place p mod R of an entry's slot gets its token's row of u.
template <typename T>
struct RingRow {
    const T* u;
    long long u_stride;
    float* ring;  // null: nothing to do
    long long ring_stride;
    const int *positions, *cu_tokens, *slots;
    int channels, R;
};
template <typename T>
__device__ __forceinline__ void ring_row(const RingRow<T>& A, int e, int block, const int* meta) {
    const int c = block * blockDim.x + threadIdx.x;
    if (e >= meta[META_NUM_ENTRIES] || c >= A.channels) return;
    const int t = A.cu_tokens[e];
    A.ring[(size_t)A.slots[e] * A.ring_stride + (size_t)(A.positions[t] % A.R) * A.channels + c] = to_float(A.u[(size_t)t * A.u_stride + c]);
}

// Heads of 32, 64 or 128 columns whose state fits a block's registers, at most four taps.
static bool ssm_token_takes(int heads, int P, int N, int groups, int taps) {
    return (P == 32 || P == 64 || P == 128) && groups > 0 && heads % groups == 0 && taps >= 1 && taps <= 4 && N > 0 && N <= 8192 / P;
}
