// The float32 matrix product of large weights on the 5th-generation tensor cores: y[M, N] = x[M, K] * w[N, K]^T.
//
// Every float32 operand is taken as the sum of two TF32 numbers, hi (the nearest one) and lo (the nearest one to what is left):
// 22 to 23 of its 24 bits.  A product is hi hi + hi lo + lo hi, three tcgen05.mma of kind::tf32 (the products of TF32 numbers
// are exact in float32).  The tensor core drops the last bits of what it adds to a larger sum, so it only sums runs of 32 along
// K, the small terms first, and the runs are added up by rounded float32 additions in registers.  Measured against float64
// (relative, 2-norm, normal operands; in brackets one float32 accumulator over k in order, gemm_f32.cu): 333 x 16384 x 2048 2.0e-7
// (8.1e-7), 333 x 2048 x 8192 1.8e-7 (1.6e-6).
//
// The order of an element's sum depends on N and K only: neither on M, nor on the tile it falls in.  An element that does not
// come out finite is taken again by plain multiply-adds over k in order (an infinity has no TF32 rest, and a number beyond the largest
// TF32 one rounds to infinity).
//
// A block makes 128 columns of y (rows of w, the MMA's 128-row side) for `bn` of its rows.  Warp 0 copies, warp 1 issues the
// MMAs, warps 4..7 split the weights (shared memory -> tensor memory, where the MMA takes its A operand from), warps 8..15 add
// up the runs and store.  x comes split (split_tf32_kernel).  Bound, for prompts, by shared memory: with A in tensor memory an MMA reads
// 64 of the 128 bytes a clock, the copies write 42 and splitting reads 14; with x split in the block it would be 42 more.  For a few
// rows: by the weights' bytes.  Few-tile weights are cut along K over a cluster, whose blocks add up their parts in order.
//
// Measured (B200, us, cold weights; in brackets gemm_f32.cu): 333 x 16384 x 2048 128 (613), 333 x 2048 x 8192 73 (426), 2048 x 16384 x
// 2048 601 (2,580; 686 TFLOP/s of TF32), 8 x 16384 x 2048 54 (87), 8 x 2048 x 8192 52 (279), 1 x 1024 x 1024 34 (40).  An
// accumulator's run takes 1,250 clocks at 176 rows for 1,056 of MMAs: the issuing warp waits once a run.
#include <cuda.h>

#include "common.cuh"

namespace {

constexpr int BN_W = 128;            // rows of w in a tile
constexpr int KSTEP = 32;            // values of k in a stage: 128 bytes of a row, one swizzle atom
constexpr int W_BYTES = BN_W * 128;  // a stage's weights
constexpr int MAX_BN = 192;          // rows of x in a tile: two accumulators and two stages of split weights fill tensor memory
constexpr int TMEM_COLS = 512, A_COLS = 64;  // a stage's split weights: 32 columns hi, 32 lo
constexpr int RING_BYTES = 224 * 1024, MAX_STAGES = 8;  // both rings: tiles of x first, then of w
constexpr uint32_t WAIT_LIMIT = 1u << 22;
#define STATUS_GEMM_TIMEOUT 2

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Whether the phase is over, without the time that try_wait may sleep.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded: false (and the status word raised) when the barrier did not flip in time.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, volatile int* abort_flag) {
    if (mbar_test(bar, parity)) return true;
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    atomicExch(&status[STATUS_GEMM_TIMEOUT], 1 + (int)blockIdx.z);
    return false;
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// D (tensor memory) (+)= A (tensor memory: row = lane, a value of K a column) * B (shared memory, K-major)
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
// The registers of the loads before it may be read from here on (they pass through, so that no read moves ahead of the wait).
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                   "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27])
                 :: "memory");
    asm volatile("" : "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
}
// Up to 32 columns of this thread's lane (a multiple of 8); their sum into acc.
__device__ __forceinline__ void load_run(uint32_t from, int cols, uint32_t (&r)[32]) {
#pragma unroll
    for (int j = 0; j < 32; j += 8)
        if (j < cols) tmem_ld8(from + j, r + j);
}
__device__ __forceinline__ void add_run(float* acc, const uint32_t (&r)[32], int cols) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
        if ((j & ~7) < cols) acc[j] += __uint_as_float(r[j]);
}
template <int N> __device__ __forceinline__ void regs_release() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
// v as hi + lo: hi rounded to TF32's 10 fraction bits (by an integer addition: the conversion instruction has a quarter of its rate),
// lo the rest, exact, cut to as many.  A NaN stays one in lo, an infinity leaves one there.
__device__ __forceinline__ void split_tf32(float v, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u);
    lo = __uint_as_float(__float_as_uint(v - hi) & 0xffffe000u);
}
// true in one lane of a whole warp
__device__ __forceinline__ bool elect_one() {
    uint32_t mine;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(mine));
    return mine != 0;
}
// Rows of 128 bytes with the 128-byte swizzle, eight rows to a 1,024-byte atom, K-major.
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// kind::tf32: float32 accumulator, TF32 A and B, both K-major.
__device__ __forceinline__ uint32_t make_idesc(int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BN_W >> 4) << 24);
}

// hi and lo of the rows of x, n values each (n a multiple of 4).
__global__ void __launch_bounds__(256) split_tf32_kernel(const float4* __restrict__ x, float4* __restrict__ hi, float4* __restrict__ lo, long long n4) {
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n4; i += (long long)gridDim.x * 256) {
        const float4 v = x[i];
        float4 h, l;
        split_tf32(v.x, h.x, l.x), split_tf32(v.y, h.y, l.y), split_tf32(v.z, h.z, l.z), split_tf32(v.w, h.w, l.w);
        hi[i] = h, lo[i] = l;
    }
}

// The element by plain multiply-adds, for one that is not finite.
__device__ __forceinline__ float in_order(const float* __restrict__ x, const float* __restrict__ w, int K) {
    float s = 0.f;
#pragma unroll 1
    for (int k = 0; k < K; ++k) s = fmaf(x[k], w[k], s);
    return s;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Four floats of another block of the cluster, at the address that they have in this one's shared memory.
__device__ __forceinline__ float4 load_from_block(uint32_t addr, int rank) {
    float4 v;
    uint32_t far;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(far) : "memory");
    return v;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// grid (parts of K = blocks of a cluster, tiles of x, tiles of w); bn: a multiple of 16, at most MAX_BN.
__global__ void __launch_bounds__(512, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                   const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, int bn, int x_stages,
                   int w_stages, int* __restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t x_full[MAX_STAGES], x_empty[MAX_STAGES], w_full[MAX_STAGES], w_empty[MAX_STAGES], a_full[2], a_empty[2], run_full[2], run_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int x_bytes = bn * 128, stage_bytes = 2 * x_bytes;  // hi, then lo
    unsigned char* w_ring = ring + x_stages * stage_bytes;
    const int parts = gridDim.x, part = blockIdx.x, m0 = blockIdx.y * bn, n0 = blockIdx.z * BN_W;
    const int all = (K + KSTEP - 1) / KSTEP, per = (all + parts - 1) / parts, first = part * per;
    const int runs = max(0, min(all, first + per) - first);  // stages of this block, each one run of the sums

    if (tid == 0) {
        for (int s = 0; s < x_stages; ++s) mbar_init(&x_full[s], 1), mbar_init(&x_empty[s], 1);
        for (int s = 0; s < w_stages; ++s) mbar_init(&w_full[s], 1), mbar_init(&w_empty[s], 4);  // (the splitting warps)
        for (int i = 0; i < 2; ++i) mbar_init(&a_full[i], 4), mbar_init(&a_empty[i], 1), mbar_init(&run_full[i], 1), mbar_init(&run_empty[i], 8);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, tmem_a = tmem + 2 * MAX_BN;

    // Registers: 64, 96, 176 and 176 a thread of the four warpgroups, the launch's 128 on average.
    if (warp < 4) {
        regs_release<64>();
        if (warp == 0 || warp == 2) {  // copies of w, copies of x
            const bool of_w = warp == 0;
            const int stages = of_w ? w_stages : x_stages;
            uint64_t *full = of_w ? w_full : x_full, *empty = of_w ? w_empty : x_empty;
            int armed = 0, s = 0;
            for (int i = 0, turn = 1; i < runs; ++i) {
                if (!mbar_wait(&empty[s], turn, status, abort_flag)) break;
                const int k = (first + i) * KSTEP;
                if (elect_one()) {
                    mbar_expect_tx(&full[s], of_w ? W_BYTES : stage_bytes);
                    if (of_w) {
                        tma_load_2d(w_ring + s * W_BYTES, &map_w, k, n0, &full[s]);
                    } else {
                        tma_load_2d(ring + s * stage_bytes, &map_hi, k, m0, &full[s]);
                        tma_load_2d(ring + s * stage_bytes + x_bytes, &map_lo, k, m0, &full[s]);
                    }
                }
                __syncwarp();
                armed = i + 1;
                if (++s == stages) s = 0, turn ^= 1;
            }
            if (*abort_flag)  // gave up: the copies in flight land (bounded) before the block goes away
                for (int i = max(0, armed - stages); i < armed; ++i)
                    for (uint32_t j = 0; j < WAIT_LIMIT && !mbar_try_wait(&full[i % stages], (i / stages) & 1); ++j) {}
        } else if (warp == 1) {
            // (whole-warp loop, one elected lane issues: under a branch on the lane the operands are no uniform values to the
            // compiler, and issuing a run took 2,200 clocks)
            const uint32_t idesc = make_idesc(bn);
            const uint64_t desc0 = make_desc(smem_u32(ring));
            const uint32_t to_lo = (uint32_t)x_bytes >> 4, to_stage = (uint32_t)stage_bytes >> 4;
            int s = 0;
            for (int i = 0; i < runs; ++i) {
                const int buf = i & 1;
                if (!mbar_wait(&a_full[buf], (i >> 1) & 1, status, abort_flag)) break;
                tc_fence_after();
                const uint32_t d = tmem + buf * MAX_BN, a_hi = tmem_a + buf * A_COLS, a_lo = a_hi + 32;
                const uint64_t b_hi = desc0 + s * to_stage, b_lo = b_hi + to_lo;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < KSTEP / 8; ++k) umma_tf32(d, a_hi + k * 8, b_lo + k * 2, idesc, k > 0);
#pragma unroll
                    for (int k = 0; k < KSTEP / 8; ++k) umma_tf32(d, a_lo + k * 8, b_hi + k * 2, idesc, 1);
#pragma unroll
                    for (int k = 0; k < KSTEP / 8; ++k) umma_tf32(d, a_hi + k * 8, b_hi + k * 2, idesc, 1);
                    umma_commit(&x_empty[s]);
                    umma_commit(&a_empty[buf]);
                    umma_commit(&run_full[buf]);
                }
                __syncwarp();
                if (++s == x_stages) s = 0;
            }
        }
        __syncwarp();
    } else if (warp < 8) {
        regs_release<96>();
        const int row = (warp & 3) * 32 + lane;
        // (These warps also wait for the tile of x and for the accumulator, so that the issuing warp has one barrier to wait for a run.)
        int s = 0, xs = 0, x_turn = 0;
        for (int i = 0, turn = 0; i < runs; ++i) {
            const int buf = i & 1;
            if (!mbar_wait(&w_full[s], turn, status, abort_flag)) break;
            const unsigned char* src = w_ring + s * W_BYTES + row * 128;
            float v[32];
            uint32_t r[32];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 q = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
                v[4 * c] = q.x, v[4 * c + 1] = q.y, v[4 * c + 2] = q.z, v[4 * c + 3] = q.w;
            }
            if (!mbar_wait(&a_empty[buf], ((i >> 1) & 1) ^ 1, status, abort_flag)) break;
            __syncwarp();
            tc_fence_after();
            const uint32_t at = tmem_a + buf * A_COLS + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                float h, l;
                split_tf32(v[j], h, l);
                r[j] = __float_as_uint(h), v[j] = l;
            }
            tmem_st32(at, r);
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(v[j]);
            tmem_st32(at + 32, r);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_empty[s]);
            if (!mbar_wait(&x_full[xs], x_turn, status, abort_flag)) break;
            if (!mbar_wait(&run_empty[buf], ((i >> 1) & 1) ^ 1, status, abort_flag)) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[buf]);
            if (++xs == x_stages) xs = 0, x_turn ^= 1;
            if (++s == w_stages) s = 0, turn ^= 1;
        }
        __syncwarp();
    } else {
        regs_take<176>();
        // ---- sums of the runs: this thread's row of w, half of the tile's rows of x (a multiple of 8)
        const int quarter = warp & 3, half = (warp - 8) >> 2, cols = bn / 2, c_first = half * cols;
        float acc[MAX_BN / 2];
#pragma unroll
        for (int j = 0; j < MAX_BN / 2; ++j) acc[j] = 0.f;
        bool ok = true;
        for (int i = 0; i < runs && ok; ++i) {
            const int buf = i & 1;
            ok = mbar_wait(&run_full[buf], (i >> 1) & 1, status, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t from = tmem + buf * MAX_BN + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c_first;
            // 32 columns are added while the next 32 are on their way
            uint32_t r[2][32];
            load_run(from, cols, r[0]);
            tmem_ld_wait(r[0]);
            if (cols > 32) load_run(from + 32, cols - 32, r[1]);
            add_run(acc, r[0], cols);
            if (cols > 32) {
                tmem_ld_wait(r[1]);
                if (cols > 64) load_run(from + 64, cols - 64, r[0]);
                add_run(acc + 32, r[1], cols - 32);
                if (cols > 64) {
                    tmem_ld_wait(r[0]);
                    add_run(acc + 64, r[0], cols - 64);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&run_empty[buf]);
        }
        const int n = n0 + quarter * 32 + lane;
        if (parts == 1) {
            if (ok && !*abort_flag && n < N) {
#pragma unroll
                for (int j = 0; j < MAX_BN / 2; ++j) {
                    const int m = m0 + c_first + j;
                    if (j < cols && m < M) {
                        float v = acc[j];
                        if (!finite(v)) v = in_order(x + (size_t)m * K, w + (size_t)n * K, K);
                        y[(size_t)m * N + n] = v;
                    }
                }
            }
        } else if (ok && !*abort_flag) {
            // this block's part of the sums, [rows of x][128], where the stages were (every copy has landed and been read)
            float* sums = reinterpret_cast<float*>(ring);
#pragma unroll
            for (int j = 0; j < MAX_BN / 2; ++j)
                if (j < cols) sums[(c_first + j) * BN_W + quarter * 32 + lane] = acc[j];
        }
        if (parts > 1) {
            cluster_sync();
            if (!*abort_flag) {
                // a band of the tile's rows of x, over all parts in order
                const int band = (bn + parts - 1) / parts, lo = part * band, count = max(0, min(bn, lo + band) - lo) * (BN_W / 4);
                const uint32_t sums = smem_u32(ring);
                for (int i = tid - 256; i < count; i += 256) {
                    const int j = lo + i / (BN_W / 4), c = i % (BN_W / 4) * 4, m = m0 + j, col = n0 + c;
                    if (m >= M || col >= N) continue;
                    float v[4] = {0.f, 0.f, 0.f, 0.f};
                    for (int p = 0; p < parts; ++p) {
                        const float4 q = load_from_block(sums + (uint32_t)(j * BN_W + c) * 4, p);
                        v[0] += q.x, v[1] += q.y, v[2] += q.z, v[3] += q.w;
                    }
                    float* dst = y + (size_t)m * N + col;
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (col + e < N && !finite(v[e])) v[e] = in_order(x + (size_t)m * K, w + (size_t)(col + e) * K, K);
                    if (N % 4 == 0) {
                        store4(dst, v);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (col + e < N) dst[e] = v[e];
                    }
                }
            }
            cluster_sync();  // no block leaves while its part may still be read
        }
    }
    if (warp < 8 && parts > 1) {
        cluster_sync();
        cluster_sync();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A [rows, K] float32 matrix as tiles of box_rows x 32 with the 128-byte swizzle.
bool make_map(EncodeTiledFn fn, CUtensorMap* map, const void* base, int rows, int K, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 4};
    cuuint32_t box[2] = {(cuuint32_t)KSTEP, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// x [M, K], w [N, K], y [M, N], split: 2 * M * K floats of scratch; K a multiple of 4, x, w, y and split 16-byte aligned.
extern "C" int gemm_f32_tcgen05(const float* x, const float* w, float* y, float* split, int M, int N, int K, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)split) & 15)) return (int)cudaErrorInvalidValue;
    static EncodeTiledFn encode = nullptr;
    if (!encode) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            return (int)cudaErrorNotSupported;
        encode = reinterpret_cast<EncodeTiledFn>(p);
    }
    const int sms = multiprocessors();
    const int tiles_w = (N + BN_W - 1) / BN_W;
    // K is cut where the weight has too few tiles to fill the chip, into parts of 1,024 values or more; by N and K alone, so that a
    // row's sums do not depend on M.  At most 4: blocks of a cluster of 8 find fewer places, 333 x 2048 x 8192 took 110 us for 73.
    int parts = 1;
    while (parts < 4 && tiles_w * parts * 2 <= sms && K / (parts * 2) >= 1024) parts *= 2;
    // Rows of x a tile: the count with the shortest rounds of blocks; a round costs its rows' products and what a block spends
    // on its start and end (as much as 24 rows).
    int bn = 0;
    long best = 0;
    for (int t = (M + MAX_BN - 1) / MAX_BN, last = t + 3; t <= last; ++t) {
        const int rows = ((M + t - 1) / t + 15) / 16 * 16, tiles = (M + rows - 1) / rows;
        const long rounds = ((long)tiles_w * tiles * parts + sms - 1) / sms, cost = rounds * (rows + 24);
        if (!bn || cost < best) best = cost, bn = rows;
    }
    // Three tiles of x or more, and what is left for the weights' tiles, four or more.
    const int stage_bytes = 2 * bn * 128;
    const int fit = (RING_BYTES - 4 * W_BYTES) / stage_bytes, x_stages = fit < MAX_STAGES ? fit : MAX_STAGES;
    const int left = (RING_BYTES - x_stages * stage_bytes) / W_BYTES, w_stages = left < MAX_STAGES ? left : MAX_STAGES;
    CUtensorMap mw, mh, ml;
    float *hi = split, *lo = split + (size_t)M * K;
    if (!make_map(encode, &mw, w, N, K, BN_W) || !make_map(encode, &mh, hi, M, K, bn) || !make_map(encode, &ml, lo, M, K, bn))
        return (int)cudaErrorInvalidValue;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES + 1024);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const long long n4 = (long long)M * K / 4, want = (n4 + 255) / 256;
    split_tf32_kernel<<<(unsigned)(want < sms * 8 ? want : sms * 8), 256, 0, stream>>>((const float4*)x, (float4*)hi, (float4*)lo, n4);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(parts, (M + bn - 1) / bn, tiles_w);
    cfg.blockDim = dim3(512, 1, 1);
    cfg.dynamicSmemBytes = RING_BYTES + 1024;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = parts, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = parts > 1 ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel, mw, mh, ml, x, w, y, M, N, K, bn, x_stages, w_stages, status);
}
