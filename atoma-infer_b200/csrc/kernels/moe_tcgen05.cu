// The linears of routed experts for many bfloat16 rows, on the 5th-generation tensor cores: rows sorted by expert, every expert's
// stretch of them times that expert's weights, and the shared expert's product in the same launch.
//
//   mode 1: a[i, f] = silu(w[e, f] . x[i]) * (w[e, F + f] . x[i])   (w [E, 2F, K], f < F)
//   mode 0: y[i, n] = w[e, n] . a[i]                                (w [E, N, K]); mode 2: the same, stored as float32
//
// The weights are the MMA's row side and the tokens its columns: a stretch of n rows is cut into equal chunks of at most 256,
// rounded up to 32, so that an expert of 260 rows does the work of 320 and not of 384, as it does where 128 rows are the tile's least; and
// an expert with few rows costs its weights' bytes and little else.  In mode 1 a block's 128 rows are 64 of the gate and the same 64
// of up; two warps that hold the two halves of a result swap them through shared memory.
//
// Two blocks (cta_group::2) make a tile of 256 rows of the weights: each brings 128 of them and half of the chunk's rows of x.  With a
// block a tile, every 64 columns of k were 48 KB through the second-level cache for 512 clocks of MMAs, chunks of 144 rows 36 KB
// for 288: bound by those bytes.
//
// A pair of blocks walks tiles p, p + pairs, ... (a group's chunks fastest: they share its weights): warp 0 copies (a lane a box),
// warp 1 of the pair's first block issues the MMAs into one of two accumulators in tensor memory, warps 2..9 store the other one, a
// block its own rows.  How many tiles there are is known on the device only (`offsets`); nothing is read back.
//
// Measured (B200, experts and shared expert of 2,048 x 2,048, two of sixteen experts a row; both linears with the shared expert's in the
// same launches, beside the library's grouped products and its own for the shared expert): 2,048 rows 165 us (188 with the two
// activation kernels), 130 rows 86 (128); 33 to 127 rows 85 (the tile kernel for few rows 720).  With few rows the weights' bytes
// bound it (0.8 of the copy bandwidth), with many the rate of a tile (the library's) and seven tiles a pair of blocks, which do not come out even.
//
// Every element's sum runs over k in one accumulator in order: it does not depend on the rows beside it.
#include <cuda.h>

#include "common.cuh"
#include "gemm_tcgen05.cuh"

namespace {

constexpr int MAX_CHUNK = 256;  // rows of x in a tile at most
constexpr int W_BYTES = BM * BK * 2, X_BYTES = MAX_CHUNK / 2 * BK * 2, STAGE_BYTES = W_BYTES + X_BYTES;
constexpr int STORE_WARPS = 8, THREADS = 64 + 32 * STORE_WARPS;  // (four: the last tiles' stores took 3 us more of a launch)
constexpr int SWAP_FLOATS = STORE_WARPS * 16 * 32;  // 16 columns of a warp's lanes
// Six stages, or four where a count for every expert would not fit beside them (three cost 8 % of a launch's time); MAX_EXPERTS is what
// the sort by expert takes, too.
constexpr int STAGES_FEW = 6, STAGES_MANY = 4, FEW_EXPERTS = 1024, MAX_EXPERTS = 12287;

// ---- pairs of blocks
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of the same variable in the pair's first block.
__device__ __forceinline__ uint32_t of_first(const void* p) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void pair_arrive(uint32_t remote_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
// A copy into this block's shared memory whose bytes count at a barrier of the pair's first block.
__device__ __forceinline__ void pair_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_load_3d(void* smem_dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives at the barrier of this place in both blocks when the MMAs issued so far are complete.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

__device__ __forceinline__ void store_two(bf16* p, float2 v) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(v.x, v.y); }
__device__ __forceinline__ void store_two(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }

// A meeting of the two warps that hold the halves of a result.
__device__ __forceinline__ void pair_barrier(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

struct GroupedArgs {
    const int* offsets;  // [experts + 1]: an expert's stretch of the sorted rows
    const int* meta;     // the step's tokens: the shared expert's rows
    int experts, rows, depth;                              // an expert's results a row (mode 1: F) and its K
    int shared_tokens, shared_rows, shared_depth;          // (0 tokens: no shared expert)
    void* out;                                             // [sorted rows, rows], bfloat16 (mode 2: float32)
    bf16* shared_out;                                      // [tokens, shared_rows]
};

// A tile: `count` rows of x from `first` on, results from `w0` on, of expert `e` (or the shared one: -1).
struct Tile { int e, w0, first, count; };

// Which tile is which: the shared expert's first (they are the largest), then expert by expert.  (Shares of the shared expert between
// the experts, so that its arithmetic runs beside their weights' way from memory: no faster.)
struct Tiles {
    const GroupedArgs& a;
    const int* before;  // [segments + 1], in shared memory: tiles ahead of each segment
    int span;           // results of a tile
    __device__ static int chunk(int n) { const int c = (n + MAX_CHUNK - 1) / MAX_CHUNK; return ((n + c - 1) / c + 31) & ~31; }
    __device__ int segments() const { return a.experts + (a.shared_tokens > 0); }
    // A segment's expert, rows, the first of them, and its blocks of results.
    __device__ int segment(int s, int& n, int& from, int& blocks) const {
        const int e = s - (a.shared_tokens > 0);
        if (e < 0) {
            n = min(a.shared_tokens, a.meta[META_NUM_TOKENS]), from = 0;
            blocks = (a.shared_rows + span - 1) / span;
        } else {
            from = a.offsets[e], n = a.offsets[e + 1] - from;
            blocks = (a.rows + span - 1) / span;
        }
        return e;
    }
    __device__ int count(int s) const {
        int n, from, blocks;
        segment(s, n, from, blocks);
        return n > 0 ? blocks * ((n + chunk(n) - 1) / chunk(n)) : 0;
    }
    // `s` is where the last tile was found: tiles come in ascending order
    __device__ Tile find(int tile, int& s) const {
        while (tile >= before[s + 1]) ++s;
        int n, from, blocks;
        const int e = segment(s, n, from, blocks), size = chunk(n), chunks = (n + size - 1) / size, at = tile - before[s], c = at % chunks;
        return {e, at / chunks * span, from + c * size, min(size, n - c * size)};
    }
};

}  // namespace

struct RowMaps { CUtensorMap box[4]; };  // 16, 32, 64 and 128 rows in a copy

template <int MODE, int STAGES>
__global__ void __launch_bounds__(THREADS, 1)
moe_grouped_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ RowMaps map_x, const __grid_constant__ CUtensorMap map_sw,
                      const __grid_constant__ RowMaps map_sx, const GroupedArgs a, int* __restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int SPAN = MODE == 1 ? BM / 2 : BM;  // results a block makes of a row, half of the tile's
    unsigned char* ring = smem;
    float* swap = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES);
    // full_bar and acc_empty are used in the pair's first block, the others in both
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(swap + SWAP_FLOATS);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;   // [2]: an accumulator is complete
    uint64_t* acc_empty = acc_full + 2;        // [2]: both blocks' storing warps have read it
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* before = reinterpret_cast<int*>(tmem_slot + 2);
    const Tiles T{a, before, 2 * SPAN};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 2 * STORE_WARPS); }  // one arrival per storing warp
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    pdl_launch_dependents();  // (these launches start when the one ahead has drained; the weighted sum behind them starts early: 1 us)
    if (warp == 2) {
        int upto = 0;
        for (int s0 = 0; s0 < T.segments(); s0 += 32) {
            int tiles = s0 + lane < T.segments() ? T.count(s0 + lane) : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, tiles, d);
                if (lane >= d) tiles += below;
            }
            if (s0 + lane < T.segments()) before[s0 + lane + 1] = upto + tiles;
            upto += __shfl_sync(0xffffffffu, tiles, 31);
        }
        if (lane == 0) before[0] = 0;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other block's barriers are ready too
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int num_tiles = before[T.segments()];

    if (warp == 0) {
        // ---- copies: lane i < 4 a box of 16 << i rows of x where the block's half of the chunk has that bit, lane 4 the weights
        int it = 0, armed = 0, seg = 0;  // k blocks over all my tiles; those whose copies were started
        bool ok = true;
        for (int tile = pair; tile < num_tiles && ok; tile += pairs) {
            const Tile at = T.find(tile, seg);
            const bool own = at.e < 0;
            const int num_kb = ((own ? a.shared_depth : a.depth) + BK - 1) / BK, units = (at.count + 31) / 32;  // 16 rows each
            const int w_row = at.w0 + rank * SPAN, w_z = own ? 0 : at.e * (MODE == 1 ? 2 : 1);
            const int skip = (units & ~((2 << lane) - 1)) * 16;  // the boxes of the higher bits go before mine
            const bool mine = lane < 4 && (units >> lane & 1);
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const int s = it % STAGES;
                if (lane == 0) {
                    ok = mbar_wait(&empty_bar[s], ((it / STAGES) & 1) ^ 1, status, abort_flag);  // a fresh barrier passes a wait on parity 1
                    if (ok && rank == 0) mbar_expect_tx(&full_bar[s], 2 * (W_BYTES + units * 16 * BK * 2));  // what both blocks bring
                }
                ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                if (!ok) break;
                unsigned char* w_dst = ring + s * STAGE_BYTES;
                const uint32_t bar = of_first(&full_bar[s]);
                if (lane == 4)
                    pair_load_3d(w_dst, own ? &map_sw : &map_w, kb * BK, w_row, w_z, bar);
                else if (mine)
                    pair_load_2d(w_dst + W_BYTES + skip * BK * 2, own ? &map_sx.box[lane] : &map_x.box[lane], kb * BK, at.first + rank * units * 16 + skip, bar);
                armed = it + 1;
            }
        }
        if (*abort_flag && lane == 0 && rank == 0) {
            // gave up: let both blocks' copies in flight land (bounded) before the blocks go away
            for (int j = max(0, armed - STAGES); j < armed; ++j)
                for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try_wait(&full_bar[j % STAGES], (j / STAGES) & 1); ++i) {}
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // ---- MMAs
            int it = 0, n = 0, seg = 0;
            bool ok = true;
            for (int tile = pair; tile < num_tiles && ok; tile += pairs, ++n) {
                const Tile at = T.find(tile, seg);
                const int num_kb = ((at.e < 0 ? a.shared_depth : a.depth) + BK - 1) / BK;
                const uint32_t idesc = make_idesc(2 * BM, (at.count + 31) & ~31);
                const int buf = n & 1;
                ok = mbar_wait(&acc_empty[buf], (((uint32_t)n >> 1) & 1u) ^ 1u, status, abort_flag);  // its last tile is stored
                if (!ok) break;
                tc_fence_after();
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(&full_bar[s], (it / STAGES) & 1, status, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t w_addr = smem_u32(ring + s * STAGE_BYTES), x_addr = w_addr + W_BYTES;
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        pair_umma(tmem_base + buf * MAX_CHUNK, make_desc(w_addr + k * UMMA_K * 2), make_desc(x_addr + k * UMMA_K * 2), idesc,
                                  (kb > 0 || k > 0) ? 1u : 0u);
                    pair_commit(&empty_bar[s]);  // the stage is free again when these MMAs have read it
                }
                if (ok) pair_commit(&acc_full[buf]);  // arrives when every MMA issued so far is complete
            }
        }
        __syncwarp();
    } else {
        // ---- results: a warp reaches the 32 lanes of its quarter, a lane a row of the weights, a column a row of x
        const int quarter = warp & 3, part = (warp - 2) >> 2;  // the two warps of a quarter take every other step
        int n = 0, seg = 0;
        bool ok = true;
        // Two neighbouring lanes swap half of their results, so that each stores two neighbouring results of every other row of x
        // (half the stores, 64 bytes a row of x).
        auto store16 = [&](auto* dst, int ld, int row, int rows, int first_col, int cols, const float (&v)[16]) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float got = __shfl_xor_sync(0xffffffffu, lane & 1 ? v[2 * i] : v[2 * i + 1], 1);
                const int col = first_col + 2 * i + (lane & 1);
                const float2 two = lane & 1 ? make_float2(got, v[2 * i + 1]) : make_float2(v[2 * i], got);
                if (ok && col < cols && row < rows) store_two(dst + (size_t)col * ld + (row & ~1), two);
            }
        };
        // (after a timeout every wait returns at once and nothing is stored, but the pairs of warps still meet at their barriers)
        for (int tile = pair; tile < num_tiles; tile += pairs, ++n) {
            const Tile at = T.find(tile, seg);
            const bool own = at.e < 0;
            const int rows = own ? a.shared_rows : a.rows;
            bf16* dst = (own ? a.shared_out : (bf16*)a.out) + (size_t)at.first * rows;
            const int buf = n & 1;
            if (!mbar_wait(&acc_full[buf], ((uint32_t)n >> 1) & 1u, status, abort_flag)) ok = false;
            tc_fence_after();
            const uint32_t acc = tmem_base + buf * MAX_CHUNK + ((uint32_t)(quarter * 32) << 16);
            if (MODE != 1) {
#pragma unroll 1
                for (int c0 = part * 16; c0 < at.count; c0 += 32) {
                    float v[16];
                    tmem_ld16(acc + c0, v);
                    const int row = at.w0 + rank * SPAN + quarter * 32 + lane;
                    if (MODE == 2 && !own) store16((float*)a.out + (size_t)at.first * rows, rows, row, rows, c0, at.count, v);
                    else store16(dst, rows, row, rows, c0, at.count, v);
                }
            } else {
                const int up = quarter >> 1;  // quarters 0 and 1 hold the gate, 2 and 3 up; each finishes every other 16 columns
#pragma unroll 1
                for (int c0 = part * 32; c0 < at.count; c0 += 64) {
                    float give[16], v[16];
                    tmem_ld16(acc + c0 + (up ? 0 : 16), give);
                    float* slot = swap + (part * 4 + quarter) * 512 + lane;
                    pair_barrier(1 + part * 2 + (quarter & 1));  // the other warp has read what I gave it last
#pragma unroll
                    for (int i = 0; i < 16; ++i) slot[i * 32] = give[i];
                    tmem_ld16(acc + c0 + (up ? 16 : 0), v);
                    pair_barrier(1 + part * 2 + (quarter & 1));
                    const float* other = swap + (part * 4 + (quarter ^ 2)) * 512 + lane;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float o = other[i * 32];
                        v[i] = up ? silu_as<bf16>(o) * v[i] : silu_as<bf16>(v[i]) * o;
                    }
                    store16(dst, rows, at.w0 + rank * SPAN + (quarter & 1) * 32 + lane, rows, c0 + (up ? 16 : 0), at.count, v);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) pair_arrive(of_first(&acc_empty[buf]));  // this warp has read its lanes of the accumulator
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // nobody leaves while the other block's copies, MMAs or arrivals may still reach it
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
}

namespace {

// Weights [groups, rows, K] seen as tiles of `each` rows x 64 columns of `groups_box` neighbouring groups.
bool make_weight_map(CUtensorMap* map, const void* base, long long groups, int rows, int K, int each, int groups_box) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)groups};
    cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)K * 2 * rows};
    cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)each, (cuuint32_t)groups_box};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_row_maps(RowMaps* maps, const void* x, int rows, int K) {
    for (int i = 0; i < 4; ++i)
        if (!make_map(&maps->box[i], x, rows, K, 16 << i)) return false;
    return true;
}

template <int MODE, int STAGES>
int launch_grouped(const void* x, const void* w, int pairs, const void* sx, const void* sw, const GroupedArgs& a, int* status, cudaStream_t stream) {
    CUtensorMap mw, msw;
    RowMaps mx, msx;
    constexpr int BOTH = MODE == 1 ? 2 : 1;
    if (!make_weight_map(&mw, w, (long long)a.experts * BOTH, a.rows, a.depth, BM / BOTH, BOTH) || !make_row_maps(&mx, x, pairs, a.depth))
        return (int)cudaErrorInvalidValue;
    msw = mw, msx = mx;
    if (a.shared_tokens > 0 && (!make_weight_map(&msw, sw, BOTH, a.shared_rows, a.shared_depth, BM / BOTH, BOTH) ||
                                !make_row_maps(&msx, sx, a.shared_tokens, a.shared_depth)))
        return (int)cudaErrorInvalidValue;
    const size_t smem = STAGES * STAGE_BYTES + SWAP_FLOATS * 4 + (2 * STAGES + 4) * 8 + 8 + (a.experts + 2) * 4 + 1024;
    static size_t configured = 0;
    if (smem > configured) {
        const cudaError_t e = cudaFuncSetAttribute(moe_grouped_tc_kernel<MODE, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = smem;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(multiprocessors() & ~1);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, moe_grouped_tc_kernel<MODE, STAGES>, mw, mx, msw, msx, a, status);
}

}  // namespace

// act [pairs, F] = SwiGLU of the sorted rows xs [pairs, H] under w_gate_up [E, 2F, H], y [pairs, H] (float32 if `wide`) = act times
// w_down [E, H, F]; with
// T > 0 rows h also act_s [T, Fs] and y_s [T, H] of the shared expert (ws_gate_up [2 Fs, H], ws_down [H, Fs]).  H, F and Fs multiples
// of 8, matrices on 16 bytes, E <= moe_tc_most_experts().  Rows beyond the experts' stretches stay as they are.
extern "C" int moe_tc_most_experts() { return MAX_EXPERTS; }
extern "C" int moe_tc_ff(const void* xs, const void* w_gate_up, void* act, const void* w_down, void* y, const int* offsets, int pairs, int E, int H,
                         int F, const void* h, const void* ws_gate_up, void* act_s, const void* ws_down, void* y_s, int T, int Fs, int wide,
                         const int* meta, int* status, cudaStream_t stream) {
    if (pairs <= 0) return 0;
    if (E < 1 || E > MAX_EXPERTS || H <= 0 || F <= 0 || (H | F | Fs) % 8 || (T > 0 && Fs <= 0)) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)xs | (uintptr_t)w_gate_up | (uintptr_t)act | (uintptr_t)w_down | (uintptr_t)y | (uintptr_t)h | (uintptr_t)ws_gate_up |
         (uintptr_t)act_s | (uintptr_t)ws_down | (uintptr_t)y_s) & 15)
        return (int)cudaErrorInvalidValue;
    const GroupedArgs first{offsets, meta, E, F, H, T, Fs, H, act, (bf16*)act_s}, second{offsets, meta, E, H, F, T, H, Fs, y, (bf16*)y_s};
    const bool few = E <= FEW_EXPERTS;
    const int rc = few ? launch_grouped<1, STAGES_FEW>(xs, w_gate_up, pairs, h, ws_gate_up, first, status, stream)
                       : launch_grouped<1, STAGES_MANY>(xs, w_gate_up, pairs, h, ws_gate_up, first, status, stream);
    if (rc) return rc;
    if (wide)
        return few ? launch_grouped<2, STAGES_FEW>(act, w_down, pairs, act_s, ws_down, second, status, stream)
                   : launch_grouped<2, STAGES_MANY>(act, w_down, pairs, act_s, ws_down, second, status, stream);
    return few ? launch_grouped<0, STAGES_FEW>(act, w_down, pairs, act_s, ws_down, second, status, stream)
               : launch_grouped<0, STAGES_MANY>(act, w_down, pairs, act_s, ws_down, second, status, stream);
}
