// The float32 matrix product: y[M, N] = x[M, K] * w[N, K]^T in plain float32 multiply-adds, no tensor cores, no TF32.  Every
// output element is one accumulator that runs over k = 0..K-1 in order, so its value depends neither on M nor on the tile
// it falls in, and every tile size below gives the same bits.
//
// Bound by the FP32 pipe (148 multiprocessors x 128 multiply-adds a clock: 74 TFLOP/s at 1,965 MHz) for prompts, by the
// weights' bytes and a block's chain of loads for a few rows.  A thread keeps TM x TN accumulators as pairs of neighbouring
// columns and updates a pair with one two-wide instruction (sm_100; each half the plain IEEE operation), which leaves half
// of the issue slots for the operands: x and w are staged as [k][row] in two shared-memory buffers, the next stage's 16-byte
// loads are in flight while the current one is multiplied.
#include "common.cuh"

namespace {

__device__ __forceinline__ unsigned long long pair_of(float a, float b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// A stage of one operand: ROWS rows of GK values, kept as [GK][ROWS + 4].  Value (row, k) lies in line k at row ^ (k / 8 * RW),
// RW rows being what a warp stores at once: the stores of a warp's 32 float4 then fall into 32 different banks, and four
// neighbouring rows stay neighbours for the 16-byte reads (RW is 4 or 8).
template <int ROWS, int GK>
struct Stage {
    static constexpr int LD = ROWS + 4, C4 = GK / 4, RW = 32 / C4;
    static __device__ __forceinline__ int at(int row, int k) { return k * LD + (row ^ ((k >> 3) * RW)); }
};

__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// What a launch that takes again what is not finite looks at: a flag without which there is nothing to do, and where the number of
// rows that count stands (null: all M do).
struct Repair {
    const int *odd, *limit;
};

// BM x BN outputs a block, TM x TN (in groups of four rows and four columns) a thread.  VEC: rows of x and w start on 16
// bytes and K is a multiple of 4.  REPAIR: only the elements of y that are not finite, in the tiles that have one.
template <int BM, int BN, int TM, int TN, int GK, bool VEC, bool REPAIR>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, int vec_out, Repair repair) {
    constexpr int NT = (BM / TM) * (BN / TN), C4 = GK / 4, QA = BM * C4, QB = BN * C4;
    constexpr int LA = (QA + NT - 1) / NT, LB = (QB + NT - 1) / NT;
    using SA = Stage<BM, GK>;
    using SB = Stage<BN, GK>;
    __shared__ __align__(16) float xs[2][GK * SA::LD], ws[2][GK * SB::LD];
    const int tid = threadIdx.x, m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    int rows = M;  // that are stored
    if (REPAIR) {
        pdl_wait();
        if (!*repair.odd) return;
        if (repair.limit) rows = min(M, *repair.limit);
        int any = 0;
        for (int i = tid; i < BM * BN && !any; i += NT) {
            const int m = m0 + i / BN, n = n0 + i % BN;
            any = m < rows && n < N && !finite(y[(size_t)m * N + n]);
        }
        if (!__syncthreads_or(any)) return;
    }
    float4 ra[LA], rb[LB];

    auto quad = [&](const float* __restrict__ src, int row, int rows, int k) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < rows && k < K) {
            const float* p = src + (size_t)row * K + k;
            if (VEC) return *reinterpret_cast<const float4*>(p);
            v.x = p[0];
            if (k + 1 < K) v.y = p[1];
            if (k + 2 < K) v.z = p[2];
            if (k + 3 < K) v.w = p[3];
        }
        return v;
    };
    auto load_x = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int q = tid + i * NT;
            if (QA % NT == 0 || q < QA) ra[i] = quad(x, m0 + q / C4, M, k0 + q % C4 * 4);
        }
    };
    auto load_w = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int q = tid + i * NT;
            if (QB % NT == 0 || q < QB) rb[i] = quad(w, n0 + q / C4, N, k0 + q % C4 * 4);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int q = tid + i * NT, r = q / C4, k = q % C4 * 4;
            if (QA % NT == 0 || q < QA) {
                float* d = xs[buf] + SA::at(r, k);
                d[0] = ra[i].x, d[SA::LD] = ra[i].y, d[2 * SA::LD] = ra[i].z, d[3 * SA::LD] = ra[i].w;
            }
        }
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int q = tid + i * NT, r = q / C4, k = q % C4 * 4;
            if (QB % NT == 0 || q < QB) {
                float* d = ws[buf] + SB::at(r, k);
                d[0] = rb[i].x, d[SB::LD] = rb[i].y, d[2 * SB::LD] = rb[i].z, d[3 * SB::LD] = rb[i].w;
            }
        }
    };

    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    load_w(0);  // weights depend on no kernel of the step
    pdl_launch_dependents();
    pdl_wait();
    load_x(0);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += GK, buf ^= 1) {
        const bool more = k0 + GK < K;
        if (more) load_x(k0 + GK), load_w(k0 + GK);
        const float *xb = xs[buf], *wb = ws[buf];
#pragma unroll
        for (int kk = 0; kk < GK; ++kk) {
            float a[TM];
            unsigned long long b[TN / 2];
#pragma unroll
            for (int i = 0; i < TM; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(xb + SA::at(i / 4 * (BM / TM * 4) + ty * 4, kk));
                a[i] = v.x, a[i + 1] = v.y, a[i + 2] = v.z, a[i + 3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(wb + SB::at(j / 4 * (BN / TN * 4) + tx * 4, kk));
                b[j / 2] = v.x, b[j / 2 + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const unsigned long long aa = pair_of(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma_pair(acc[i][j], aa, b[j]);
            }
        }
        if (more) {
            store(buf ^ 1);  // (that buffer was last read before the barrier that ended the stage before this one)
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + i / 4 * (BM / TM * 4) + ty * 4 + i % 4;
        if (m >= rows) continue;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int n = n0 + j / 4 * (BN / TN * 4) + tx * 4;
            float* dst = y + (size_t)m * N + n;
            float v[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][j / 2]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[i][j / 2 + 1]));
            if (REPAIR) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (n + c < N && !finite(dst[c])) dst[c] = v[c];
            } else if (vec_out && n + 3 < N) {
                store4(dst, v);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (n + c < N) dst[c] = v[c];
            }
        }
    }
}

template <int BM, int BN, int TM, int TN, int GK>
int launch(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    const int vec = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0, vec_out = N % 4 == 0 && ((uintptr_t)y & 15) == 0;
    constexpr int threads = (BM / TM) * (BN / TN);
    if (vec) return (int)launch_kernel(gemm_f32_kernel<BM, BN, TM, TN, GK, true, false>, grid, threads, 0, stream, x, w, y, M, N, K, vec_out, Repair{});
    return (int)launch_kernel(gemm_f32_kernel<BM, BN, TM, TN, GK, false, false>, grid, threads, 0, stream, x, w, y, M, N, K, vec_out, Repair{});
}

}  // namespace

// A test and measurement lever: which tile (0: by the rule below).
static int g_tile = 0;
extern "C" void gemm_f32_set_tile(int n) { g_tile = n; }

extern "C" int gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    // The tile with the least estimated time.  Measured, ns for one step of k: a tile alone on its multiprocessor (`alone`: its
    // chain of loads, barrier and products) and what every further tile there adds (`more`: the FP32 pipe's share, with the
    // chip full).  The busiest multiprocessor has ceil(tiles / multiprocessors) of them, the others up to one fewer, and it
    // runs the faster for that: the mean of the two counts is taken.  Measured with this rule against one 64 x 64 tile for
    // all sizes (x rows, w rows, K; us): 2048 x 16384 x 2048 2,590 / 5,890 (53 TFLOP/s), 333 x 16384 x 2048 613 / 1,178, 333 x 2048
    // x 8192 422 / 1,036, 8 x 2048 x 8192 275 / 1,023, 1 x 16384 x 2048 74 / 302, 8 x 128256 x 2048 275 / 1,513.
    static const struct { int bm, bn; float alone, more; } tiles[] = {
        {128, 128, 113.f, 91.f}, {64, 128, 77.f, 51.5f}, {64, 64, 47.f, 25.4f}, {32, 64, 36.f, 16.1f}, {16, 128, 34.f, 18.3f}};
    const int sms = multiprocessors();
    int best = 0;
    float least = 0.f;
    for (int i = 0; i < 5; ++i) {
        const long count = (long)((M + tiles[i].bm - 1) / tiles[i].bm) * ((N + tiles[i].bn - 1) / tiles[i].bn);
        const float mean = fmaxf((float)count / sms, 1.f), n = ((float)((count + sms - 1) / sms) + mean) * .5f;
        const float cost = tiles[i].alone + (n - 1.f) * tiles[i].more;
        if (i == 0 || cost < least) least = cost, best = i;
    }
    switch (g_tile ? g_tile - 1 : best) {
        case 0: return launch<128, 128, 8, 8, 16>(x, w, y, M, N, K, stream);
        case 1: return launch<64, 128, 8, 4, 16>(x, w, y, M, N, K, stream);
        case 2: return launch<64, 64, 8, 4, 16>(x, w, y, M, N, K, stream);
        case 3: return launch<32, 64, 4, 4, 32>(x, w, y, M, N, K, stream);
        default: return launch<16, 128, 4, 4, 32>(x, w, y, M, N, K, stream);
    }
}

// The elements of y that are not finite again, by the product above (with its bits); the others stay.  odd: a device word without which nothing
// is done (the launch then ends at once); limit: a device word that says how many rows count (or null).  x and w on 16 bytes, K a
// multiple of 4.
extern "C" int gemm_f32_repair(const float* x, const float* w, float* y, const int* odd, const int* limit, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K % 4 || (((uintptr_t)x | (uintptr_t)w) & 15)) return (int)cudaErrorInvalidValue;
    if (M <= 32)
        return (int)launch_kernel(gemm_f32_kernel<32, 64, 4, 4, 32, true, true>, dim3((N + 63) / 64, 1), 128, 0, stream, x, w, y, M, N, K, 0,
                                  Repair{odd, limit});
    return (int)launch_kernel(gemm_f32_kernel<128, 128, 8, 8, 16, true, true>, dim3((N + 127) / 128, (M + 127) / 128), 256, 0, stream, x, w, y, M, N, K,
                              0, Repair{odd, limit});
}
