// The float32 matrix product of large weights on the 5th-generation tensor cores: y[M, N] = x[M, K] * w[N, K]^T.
//
// Every float32 operand is the sum of three bfloat16 numbers, hi + mid + lo, exactly: each is the nearest to what the ones before it
// leave.  Operands are taken times 2^24 for it, so that the rest of the smallest subnormal number is a normal one, and y times 2^-48.
// A product is the eight tcgen05.mma of kind::f16 of all pairs but lo lo (at most 2^-32 of it).  The tensor core drops the last bits of
// what it adds to a larger sum: it sums hi hi (16 bits a product) in runs of 32 along K only, which registers add up by rounded
// float32 additions, and the small terms, 2^-7 of a product together, in an accumulator of their own to the end; there the two meet.  One
// term's product is thus rounded once, as by a multiply-add.
//
// The order of an element's sum depends on N and K only: neither on M, nor on the tile it falls in.  An element that does not
// come out finite (an infinity has no rest; from 2^80 on the scaled sum overflows) raises a flag, after which gemm_f32.cu's repair takes all such
// elements again by plain multiply-adds over k in order.
//
// A block makes 128 columns of y (rows of w, the MMA's 128-row side) for `bn` of its rows.  Warp 0 copies w, warp 2 x, warp 1 issues the
// MMAs, warps 4..7 split the weights (shared memory -> tensor memory, where the MMA takes its A operand from), warps 8..15 add
// up the runs and store.  x comes split (split_bf16_kernel).  Bound, for prompts, by shared memory and the tensor pipe alike: of 128 bytes a
// clock the MMAs read 64, the copies write 35 and splitting reads 12.  For a few rows: by the weights' bytes.  Few-tile weights are cut
// along K over a cluster, whose blocks add up their parts in order.
//
// Measured against float64 (relative, 2-norm, normal operands; in brackets one float32 accumulator over k in order, gemm_f32.cu): 333 x 16384 x
// 2048 1.6e-7 (8.1e-7), 333 x 2048 x 8192 1.7e-7 (1.6e-6); rows of x with one number that is not zero 2.5e-8 (2.5e-8), two 2.6e-8 (3.1e-8),
// eight 2.9e-8 (5.4e-8), eight of one run 3.0e-8.  (Two TF32 numbers an operand and three products: 0.75 of the time below, but an
// operand lost up to 2^-23 and a product up to 2^-21, more where a rest fell below 2^-126.)
//
// Measured (B200, us, cold weights; in brackets gemm_f32.cu): 333 x 16384 x 2048 162 (608), 333 x 2048 x 8192 96 (420), 2048 x 16384 x 2048 785
// (2,600; 1.40 PFLOP/s of bfloat16, the library's sustained rate), 8 x 16384 x 2048 52 (72), 8 x 2048 x 8192 51 (274), 1 x 1024 x 1024 25 (34);
// of that the repair, when there is nothing to do, 1.0 to 2.8.  A whole batch of NaN, 333 x 4096 x 2048: 268 (176).
#include <cuda.h>

#include "common.cuh"
#include "gemm_tcgen05.cuh"

namespace {

constexpr int RUN = 32;               // values of k that the tensor core sums: a copy of w is 128 bytes of a row, one swizzle atom
constexpr int W_BYTES = BM * RUN * 4;  // a run's weights
// Rows of x in a tile: tensor memory holds their small terms' sum, a run's hi hi behind it, and two runs of split weights.
constexpr int MAX_BN = 192, TMEM_COLS = 512, HI_AT = MAX_BN, A_AT = 2 * MAX_BN, A_COLS = 48;  // (16 columns each of hi, mid and lo)
constexpr int RING_BYTES = 224 * 1024, MAX_STAGES = 8;  // both rings: tiles of x first, then of w
constexpr float SCALE = 16777216.f, UNSCALE = 3.5527136788005009e-15f;  // 2^24, 2^-48

// Whether the phase is over, without the time that try_wait may sleep.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, int* status, volatile int* abort_flag) {
    return mbar_test(bar, parity) || mbar_wait(bar, parity, status, abort_flag);
}
// D (tensor memory) (+)= A (tensor memory: row = lane, two values of K a column) * B (shared memory, K-major)
__device__ __forceinline__ void umma_from_tmem(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
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
// Two neighbouring values as hi + mid + lo, exactly; what is not finite, or rounds to an infinity, leaves a NaN in mid or lo.
__device__ __forceinline__ void split_two(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(b), "f"(a));
    a -= __uint_as_float(h << 16), b -= __uint_as_float(h & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(m) : "f"(b), "f"(a));
    a -= __uint_as_float(m << 16), b -= __uint_as_float(m & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(b), "f"(a));
}
// true in one lane of a whole warp
__device__ __forceinline__ bool elect_one() {
    uint32_t mine;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(mine));
    return mine != 0;
}

// hi, mid and lo of the rows of x, scaled: three matrices of M rows of `ld` numbers (K up to the next multiple of 8).  Clears the flag.
__global__ void __launch_bounds__(256) split_bf16_kernel(const float* __restrict__ x, uint4* __restrict__ out, int* __restrict__ odd, long long pieces,
                                                         int K, int per_row) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *odd = 0;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < pieces; i += (long long)gridDim.x * 256) {
        const long long row = i / per_row;
        const int k = (int)(i - row * per_row) * 8;
        const float4* src = reinterpret_cast<const float4*>(x + row * K + k);
        const float4 a = src[0], b = k + 4 < K ? src[1] : make_float4(0.f, 0.f, 0.f, 0.f);
        uint4 h, m, l;
        split_two(a.x * SCALE, a.y * SCALE, h.x, m.x, l.x);
        split_two(a.z * SCALE, a.w * SCALE, h.y, m.y, l.y);
        split_two(b.x * SCALE, b.y * SCALE, h.z, m.z, l.z);
        split_two(b.z * SCALE, b.w * SCALE, h.w, m.w, l.w);
        out[i] = h, out[i + pieces] = m, out[i + 2 * pieces] = l;
    }
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

// grid (parts of K = blocks of a cluster, tiles of x, tiles of w); bn: a multiple of 16, at most MAX_BN.  limit: where the number of rows
// that count stands (null: all M do).
__global__ void __launch_bounds__(512, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_mid,
                   const __grid_constant__ CUtensorMap map_lo, float* __restrict__ y, int* __restrict__ odd, const int* __restrict__ limit, int M, int N,
                   int K, int bn, int x_stages, int w_stages, int* __restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t x_full[MAX_STAGES], x_empty[MAX_STAGES], w_full[MAX_STAGES], w_empty[MAX_STAGES], a_full[2], a_empty[2], run_full, run_empty, rest_full;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int x_bytes = bn * 128, stage_bytes = 3 * x_bytes;  // two runs of hi, of mid, of lo
    unsigned char* w_ring = ring + x_stages * stage_bytes;
    const int parts = gridDim.x, part = blockIdx.x, m0 = blockIdx.y * bn, n0 = blockIdx.z * BM;
    const int all = (K + RUN - 1) / RUN, per = (all + parts - 1) / parts, first = part * per;
    const int runs = max(0, min(all, first + per) - first);  // of this block

    if (tid == 0) {
        for (int s = 0; s < x_stages; ++s) mbar_init(&x_full[s], 1), mbar_init(&x_empty[s], 1);
        for (int s = 0; s < w_stages; ++s) mbar_init(&w_full[s], 1), mbar_init(&w_empty[s], 4);  // (the splitting warps)
        for (int i = 0; i < 2; ++i) mbar_init(&a_full[i], 4), mbar_init(&a_empty[i], 1);
        mbar_init(&run_full, 1), mbar_init(&run_empty, 8), mbar_init(&rest_full, 1);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(&tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, tmem_a = tmem + A_AT;

    // Registers: 64, 96, 176 and 176 a thread of the four warpgroups, the launch's 128 on average.
    if (warp < 4) {
        regs_release<64>();
        if (warp == 0 || warp == 2) {  // copies of w (a run each), copies of x (two runs each)
            const bool of_w = warp == 0;
            const int stages = of_w ? w_stages : x_stages, copies = of_w ? runs : (runs + 1) / 2;
            uint64_t *full = of_w ? w_full : x_full, *empty = of_w ? w_empty : x_empty;
            int armed = 0, s = 0;
            for (int i = 0, turn = 1; i < copies; ++i) {
                if (!wait_for(&empty[s], turn, status, abort_flag)) break;
                if (elect_one()) {
                    mbar_expect_tx(&full[s], of_w ? W_BYTES : stage_bytes);
                    if (of_w) {
                        tma_load_2d(w_ring + s * W_BYTES, &map_w, (first + i) * RUN, n0, &full[s]);
                    } else {
                        unsigned char* dst = ring + s * stage_bytes;
                        const int k = (first + 2 * i) * RUN;
                        tma_load_2d(dst, &map_hi, k, m0, &full[s]);
                        tma_load_2d(dst + x_bytes, &map_mid, k, m0, &full[s]);
                        tma_load_2d(dst + 2 * x_bytes, &map_lo, k, m0, &full[s]);
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
            // compiler, and issuing a run's twelve MMAs took 2,200 clocks)
            const uint32_t idesc = make_idesc(BM, bn);
            const uint64_t desc0 = make_desc(smem_u32(ring));
            const uint32_t to_piece = (uint32_t)x_bytes >> 4, to_stage = (uint32_t)stage_bytes >> 4;
            int s = 0;
            for (int i = 0; i < runs; ++i) {
                const int buf = i & 1;
                if (!wait_for(&a_full[buf], (i >> 1) & 1, status, abort_flag)) break;
                tc_fence_after();
                const uint32_t d_hi = tmem + HI_AT, d_rest = tmem;
                const uint32_t a_hi = tmem_a + buf * A_COLS, a_mid = a_hi + 16, a_lo = a_hi + 32;
                const uint64_t b_hi = desc0 + s * to_stage + (i & 1) * (RUN * 2 >> 4), b_mid = b_hi + to_piece, b_lo = b_mid + to_piece;
                if (elect_one()) {
                    auto product = [&](uint32_t d, uint32_t a, uint64_t b, bool fresh) {
#pragma unroll
                        for (int k = 0; k < RUN / UMMA_K; ++k) umma_from_tmem(d, a + k * UMMA_K / 2, b + k * (UMMA_K * 2 >> 4), idesc, !fresh || k > 0);
                    };
                    // hi hi first: it is added up while the seven others run
                    product(d_hi, a_hi, b_hi, true);
                    umma_commit(&run_full);
                    product(d_rest, a_mid, b_lo, i == 0), product(d_rest, a_lo, b_mid, false);
                    product(d_rest, a_hi, b_lo, false), product(d_rest, a_lo, b_hi, false), product(d_rest, a_mid, b_mid, false);
                    product(d_rest, a_hi, b_mid, false), product(d_rest, a_mid, b_hi, false);
                    if ((i & 1) || i + 1 == runs) umma_commit(&x_empty[s]);
                    umma_commit(&a_empty[buf]);
                    if (i + 1 == runs) umma_commit(&rest_full);
                }
                __syncwarp();
                if ((i & 1) && ++s == x_stages) s = 0;
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
            if (!wait_for(&w_full[s], turn, status, abort_flag)) break;
            const unsigned char* src = w_ring + s * W_BYTES + row * 128;
            uint32_t h[2][8], m[2][8], l[2][8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 q = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
                const int g = c >> 2, j = c % 4 * 2;
                split_two(q.x * SCALE, q.y * SCALE, h[g][j], m[g][j], l[g][j]);
                split_two(q.z * SCALE, q.w * SCALE, h[g][j + 1], m[g][j + 1], l[g][j + 1]);
            }
            if (!wait_for(&a_empty[buf], ((i >> 1) & 1) ^ 1, status, abort_flag)) break;
            __syncwarp();
            tc_fence_after();
            const uint32_t at = tmem_a + buf * A_COLS + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
            for (int g = 0; g < 2; ++g) tmem_st8(at + g * 8, h[g]), tmem_st8(at + 16 + g * 8, m[g]), tmem_st8(at + 32 + g * 8, l[g]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_empty[s]);
            if (!(i & 1) && !wait_for(&x_full[xs], x_turn, status, abort_flag)) break;
            if (!wait_for(&run_empty, (i & 1) ^ 1, status, abort_flag)) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[buf]);
            if ((i & 1) && ++xs == x_stages) xs = 0, x_turn ^= 1;
            if (++s == w_stages) s = 0, turn ^= 1;
        }
        __syncwarp();
    } else {
        regs_take<176>();
        // ---- sums of the runs: this thread's row of w, half of the tile's rows of x (a multiple of 8)
        const int quarter = warp & 3, half = (warp - 8) >> 2, cols = bn / 2, c_first = half * cols;
        float hi[MAX_BN / 2];
#pragma unroll
        for (int j = 0; j < MAX_BN / 2; ++j) hi[j] = 0.f;
        const uint32_t mine = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c_first, from = mine + HI_AT;
        bool ok = true;
        for (int i = 0; i < runs && ok; ++i) {
            ok = wait_for(&run_full, i & 1, status, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            // 32 columns are added while the next 32 are on their way
            uint32_t r[2][32];
            load_run(from, cols, r[0]);
            tmem_ld_wait(r[0]);
            if (cols > 32) load_run(from + 32, cols - 32, r[1]);
            add_run(hi, r[0], cols);
            if (cols > 32) {
                tmem_ld_wait(r[1]);
                if (cols > 64) load_run(from + 64, cols - 64, r[0]);
                add_run(hi + 32, r[1], cols - 32);
                if (cols > 64) {
                    tmem_ld_wait(r[0]);
                    add_run(hi + 64, r[0], cols - 64);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&run_empty);
        }
        if (ok && runs > 0) ok = __all_sync(0xffffffffu, wait_for(&rest_full, 0, status, abort_flag));
        tc_fence_after();
        const int n = n0 + quarter * 32 + lane, real = limit ? min(M, *limit) : M;
        bool any_odd = false;
        // (with several parts: this block's sums, [hi hi, rest][rows of x][128], where the stages were: every copy has landed and been read)
        float* sums = reinterpret_cast<float*>(ring);
        if (ok && !*abort_flag) {
#pragma unroll
            for (int c = 0; c < MAX_BN / 2; c += 32) {
                if (c >= cols) break;
                uint32_t rest[32];
                load_run(mine + c, cols - c, rest);
                tmem_ld_wait(rest);
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const int row = c_first + c + j, m = m0 + row;
                    const float small = runs > 0 ? __uint_as_float(rest[j]) : 0.f;
                    if (c + j >= cols) break;
                    if (parts > 1) {
                        sums[row * BM + quarter * 32 + lane] = hi[c + j];
                        sums[(bn + row) * BM + quarter * 32 + lane] = small;
                    } else if (m < M && n < N) {
                        const float v = (hi[c + j] + small) * UNSCALE;
                        y[(size_t)m * N + n] = v;
                        any_odd = any_odd || (m < real && !finite(v));
                    }
                }
            }
        }
        if (parts > 1) {
            cluster_sync();
            if (!*abort_flag) {
                // a band of the tile's rows of x, over all parts in order
                const int band = (bn + parts - 1) / parts, lo = part * band, count = max(0, min(bn, lo + band) - lo) * (BM / 4);
                const uint32_t at = smem_u32(ring);
                for (int i = tid - 256; i < count; i += 256) {
                    const int j = lo + i / (BM / 4), c = i % (BM / 4) * 4, m = m0 + j, col = n0 + c;
                    if (m >= M || col >= N) continue;
                    float v[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
                    for (int p = 0; p < parts; ++p) {
                        const float4 q = load_from_block(at + (uint32_t)(j * BM + c) * 4, p);
                        const float4 s = load_from_block(at + (uint32_t)((bn + j) * BM + c) * 4, p);
                        v[0] += q.x, v[1] += q.y, v[2] += q.z, v[3] += q.w;
                        u[0] += s.x, u[1] += s.y, u[2] += s.z, u[3] += s.w;
                    }
                    float* dst = y + (size_t)m * N + col;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        v[e] = (v[e] + u[e]) * UNSCALE;
                        any_odd = any_odd || (m < real && col + e < N && !finite(v[e]));
                    }
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
        if (any_odd) *odd = 1;
    }
    if (warp < 8 && parts > 1) {
        cluster_sync();
        cluster_sync();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, TMEM_COLS);
}

// A matrix [rows, K] of `bytes`-byte numbers, rows `ld` numbers apart, as tiles of box_rows x 128 bytes with the 128-byte swizzle.
bool make_tile_map(CUtensorMap* map, const void* base, int rows, int K, int ld, int bytes, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * bytes};
    cuuint32_t box[2] = {(cuuint32_t)(128 / bytes), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Bytes of scratch: x in three pieces, and the flag behind them.
extern "C" size_t gemm_f32_tcgen05_scratch(int M, int K) { return (size_t)3 * M * ((K + 7) / 8 * 8) * 2 + 16; }

// x [M, K], w [N, K], y [M, N], scratch as above; K a multiple of 4, x, w, y and scratch 16-byte aligned.  limit: a device word that says how
// many of the rows count (or null).  The flag is left in the scratch's last 16 bytes: 1 if an element of theirs is not finite.
extern "C" int gemm_f32_tcgen05(const float* x, const float* w, float* y, unsigned char* scratch, const int* limit, int M, int N, int K, int* status,
                                cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)scratch) & 15)) return (int)cudaErrorInvalidValue;
    const int sms = multiprocessors(), ld = (K + 7) / 8 * 8;
    const int tiles_w = (N + BM - 1) / BM;
    // K is cut where the weight has too few tiles to fill the chip, into parts of 1,024 values or more; by N and K alone, so that a
    // row's sums do not depend on M.  At most 4: blocks of a cluster of 8 find fewer places (half as slow again).
    int parts = 1;
    while (parts < 4 && tiles_w * parts * 2 <= sms && K / (parts * 2) >= 1024) parts *= 2;
    // Rows of x a tile: the count with the shortest rounds of blocks; a round costs its rows' products and what a block spends
    // on its start and end (as much as 24 rows).
    int bn = 0;
    long best = 0;
    for (int t = (M + MAX_BN - 1) / MAX_BN, last = 2 * t + 4; t <= last; ++t) {
        const int rows = ((M + t - 1) / t + 15) / 16 * 16, tiles = (M + rows - 1) / rows;
        const long rounds = ((long)tiles_w * tiles * parts + sms - 1) / sms, cost = rounds * (rows + 24);
        if (!bn || cost < best) best = cost, bn = rows;
    }
    // As many tiles of x (two runs each) as fit beside four of the weights (a run each), and what is left for the weights.
    const int stage_bytes = 3 * bn * 128;
    const int fit = (RING_BYTES - 4 * W_BYTES) / stage_bytes, x_stages = fit < MAX_STAGES ? fit : MAX_STAGES;
    const int left = (RING_BYTES - x_stages * stage_bytes) / W_BYTES, w_stages = left < MAX_STAGES ? left : MAX_STAGES;
    CUtensorMap mw, mx[3];
    const size_t piece = (size_t)M * ld * 2;
    int* odd = reinterpret_cast<int*>(scratch + 3 * piece);
    if (!make_tile_map(&mw, w, N, K, K, 4, BM)) return (int)cudaErrorInvalidValue;
    for (int i = 0; i < 3; ++i)
        if (!make_tile_map(&mx[i], scratch + i * piece, M, K, ld, 2, bn)) return (int)cudaErrorInvalidValue;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES + 1024);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const long long pieces = (long long)M * (ld / 8), want = (pieces + 255) / 256;
    split_bf16_kernel<<<(unsigned)(want < sms * 8 ? want : sms * 8), 256, 0, stream>>>(x, (uint4*)scratch, odd, pieces, K, ld / 8);
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
    return (int)cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel, mw, mx[0], mx[1], mx[2], y, odd, limit, M, N, K, bn, x_stages, w_stages, status);
}
