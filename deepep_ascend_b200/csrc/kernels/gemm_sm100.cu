// Persistent tcgen05 GEMM for sm_100a: C[M, N] (bf16) = A[M, K] * B[g][N, K]^T.
//
//   warp 0   : TMA producer - tiled loads of A (128 rows) and B (kBlockN rows) x 128 bytes (128B swizzle) into a ring of
//              shared-memory stages, completion counted on mbarriers; optionally waits for an "A rows are ready"
//              flag per M tile (all-gather fused into the loads)
//   warp 1   : MMA issuer   - one elected thread issues tcgen05.mma (kind::f16 for bf16, kind::f8f6f4 for e4m3)
//              with fp32 accumulators in tensor memory; tcgen05.commit releases stages and publishes accumulators
//   warps 2-5 (2-9 for e4m3): epilogue - tcgen05.ld the accumulator (each warp its 32 TMEM lanes), scale / convert, store bf16
//
// bf16 operands: one accumulator per output tile, two TMEM buffers so the epilogue of tile i overlaps the MMAs of
// tile i+1.  e4m3 operands with fp32 block scales (A: per row x 128 channels, B: per 128 x 128 block): every
// 128-channel block is accumulated into its own TMEM buffer and promoted into fp32 registers with its scale by
// EIGHT epilogue warps, two per TMEM lane quadrant: 64 columns each of 128-column tiles, with four TMEM buffers, so that the MMAs
// run up to three blocks ahead of the promotion; 128 columns each of 256-column tiles, with two.
// In the 256-column kernel the loop of a K block (MMAs, commit, promotion, hand-over) is what takes the time: 783 cycles for 512 of
// MMAs at 36864 rows x 4096 x 7168 (65 % of the tensor cycles), at 1.3 to 1.45 GHz under the power cap: 1020 us in short runs, 1204 in
// long ones (1097 / 1275 before its producer and MMA threads were elected ones, the stage was awaited before the accumulator and
// the accumulator committed before the stage); 36864 x 7168 x 2048: 577 / 684 us (608 / 721).
// MN-major bf16 operands (`mn_operands`): the backward pass of a layer reads weights, activations and gradients row-major as the
// forward pass left them (64 x 64 TMA boxes, transposing descriptors), at the rate of the K-major kernel: 2.3 ms for the two data
// gradients and 2.6 ms for the two weight gradients of 34816 rows x (7168, 2 x 2048) bf16.  Transposed copies of the weights
// cost 5.6 ms per training step, those of the activations 0.3 ms.
// Grouped (MoE) use: `tile_group[m_tile]` selects the expert whose weights multiply that 128-row tile.
// Every pipeline wait is bounded; on expiry the kernel raises `*error`, leaves its loops and frees its TMEM.
#include <cuda.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "gemm_sm100.cuh"

namespace ep {

namespace {

constexpr int kBlockM = 128, kTileBytes = 128 * 128;   // A tile: 128 rows x 128 bytes; B tile: kBlockN rows x 128 bytes
constexpr int kMaxStages = 7;
constexpr int kEpiRowBytes = 128 * 2 + 16;              // one staged bf16 output row (128 columns), padded against bank conflicts
constexpr int kEpiStageBytes = 4 * 32 * kEpiRowBytes;   // four epilogue warps x 32 rows
constexpr int kOutStageBytes = 32 * 128;                // per epilogue warp: 32 output rows x 64 bf16 columns on their way out
// shared memory: [A stages | B stages | barriers (1 KB) | epilogue staging]
__host__ __device__ constexpr int stage_bytes(int block_n) { return kTileBytes + block_n * 128; }
// e4m3 tiles carry half the math per byte of bf16 tiles, so that kernel keeps as many bytes in flight as fit (7 stages)
__host__ __device__ constexpr int num_stages(int block_n, bool fp8) { return block_n == 256 ? 4 : (fp8 ? 7 : 5); }
__host__ __device__ constexpr int gemm_smem_bytes(int block_n, bool fp8) {
    return num_stages(block_n, fp8) * stage_bytes(block_n) + 1024 +
           (block_n == 256 ? (fp8 ? 8 : 4) * kOutStageBytes : (block_n == 128 && !fp8 ? kEpiStageBytes : 0));
}
constexpr int kMaxCopyWarps = 6;
// copy warps of a copier CTA (all-gather fusion): each owns two 16 KB staging buffers in the shared memory that the tensor-core
// CTAs use for their operand stages: 160 KB with 128-column tiles (five warps), at least 192 KB with wider tiles (all six warps)
__host__ __device__ constexpr int copy_warps(int block_n) { return block_n == 128 ? 5 : 6; }
constexpr int kGemmThreads = 192;        // bf16: TMA warp, MMA warp, 4 epilogue warps
constexpr int kGemmThreadsFp8 = 320;     // e4m3, 128-column tiles: TMA warp, MMA warp, 8 epilogue warps
constexpr int kGemmThreadsFp8Wide = 384; // e4m3, 256-column tiles: one producer warpgroup (TMA, MMA, two idle warps) that gives its
                                         // registers to the two epilogue warpgroups (128 fp32 sums + 64 loaded values per thread)
__host__ __device__ constexpr int gemm_threads(bool fp8, int block_n) {
    return fp8 ? (block_n == 256 ? kGemmThreadsFp8Wide : kGemmThreadsFp8) : kGemmThreads;
}
template <int kRegs>
__device__ __forceinline__ void reg_alloc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void reg_dealloc() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}
constexpr int kMaxAccBufs = 4;
constexpr uint64_t kDefaultWaitLimitNs = 4ull * 1000 * 1000 * 1000;   // when the caller gives no limit

struct GemmSmem {
    uint64_t full[kMaxStages], empty[kMaxStages], tmem_full[kMaxAccBufs], tmem_empty[kMaxAccBufs];
    uint64_t copy_bar[kMaxCopyWarps][2];
    uint32_t tmem_base;
    int failed;
};

__device__ __forceinline__ uint64_t gemm_timer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint64_t wait_limit_ns(const GemmArgs& g) { return g.timeout_ns != 0 ? g.timeout_ns : kDefaultWaitLimitNs; }

// A pipeline wait ran out: stop this CTA's loops, raise the per-device flag and, when the caller gave the status block of
// a communication buffer, record the failure there too, so that the buffer's check_status() reports it and poisons the
// buffer like any other failed device wait.  `code`: 1 = empty stage, 2 = free accumulator, 3 = rows-ready flag,
// 4 = full stage, 5 = finished accumulator, 6 = scales of the streaming kernel (a slot, or its values), 7 = all-gather copy.
__device__ __forceinline__ void gemm_fail_values(int* error, uint64_t* status, int status_rank, int* failed, int code) {
    *failed = code;
    if (error != nullptr && atomicCAS(error, 0, code) == 0 && status != nullptr) {
        volatile uint64_t* st = status;
        st[EP_STATUS_PHASE] = EP_PH_GEMM_PIPE;
        st[EP_STATUS_PEER] = static_cast<uint64_t>(-1ll);
        st[EP_STATUS_EXPECTED] = static_cast<uint64_t>(code);
        st[EP_STATUS_OBSERVED] = blockIdx.x;
        st[EP_STATUS_RANK] = static_cast<uint64_t>(status_rank);
        __threadfence_system();
        st[EP_STATUS_CODE] = EP_ERR_TIMEOUT;
        __threadfence_system();
    }
}
// Two ways to the same report.  By value: the arguments stay in the kernel's parameter bank.  By reference: the compiler keeps a copy of
// all arguments in local memory, made by every thread at kernel entry, which only the wide e4m3 kernel is better off with (its
// promotion loop spills without it: 0.98 -> 1.18 ms).
__device__ __noinline__ void gemm_fail_by_value(int* error, uint64_t* status, int status_rank, int* failed, int code) {
    gemm_fail_values(error, status, status_rank, failed, code);
}
__device__ __noinline__ void gemm_fail_by_reference(const GemmArgs& g, int* failed, int code) {
    gemm_fail_values(g.error, g.status, g.status_rank, failed, code);
}
template <bool kByReference, class Smem>
__device__ __forceinline__ void gemm_fail(const GemmArgs& g, Smem* sm, int code) {
    if constexpr (kByReference) gemm_fail_by_reference(g, &sm->failed, code);
    else gemm_fail_by_value(g.error, g.status, g.status_rank, &sm->failed, code);
}

// bounded mbarrier wait; returns false (and raises the failure flags) when the limit runs out
template <bool kByReference, class Smem>
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, Smem* sm, const GemmArgs& g, int code) {
    if (ptx::mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = gemm_timer();
    uint32_t spins = 0;
    while (!ptx::mbar_try_wait(bar, parity)) {
        if ((++spins & 63u) == 0u) {
            if (*reinterpret_cast<volatile int*>(&sm->failed)) return false;
            if (gemm_timer() - t0 > wait_limit_ns(g)) {
                gemm_fail<kByReference>(g, sm, code);
                return false;
            }
        }
    }
    return true;
}

// Tile order: M tiles are walked in groups of `group_m`; inside a group consecutive tiles step through M first, so
// the tiles that run at the same time share few distinct A and B tiles and stay in L2.
struct TileCoord {
    int m, n;
};
__device__ __forceinline__ TileCoord tile_coord(int tile, int num_m, int num_n, int group_m, int m_offset) {
    const int per_group = group_m * num_n;
    const int grp = tile / per_group, in_grp = tile - grp * per_group;
    const int first_m = grp * group_m;
    const int gm = min(group_m, num_m - first_m);
    TileCoord c;
    c.m = (first_m + in_grp % gm + m_offset) % num_m;
    c.n = in_grp / gm;
    return c;
}

// What one tile index means: output tile (m, n), weights group of B, K blocks [kb0, kb1), first output row of its group.
struct TileWork {
    int m, n, grp, kb0, kb1;
    int half;          // -1: the whole tile; 0 / 1: its first / second 128 columns (see the kernel)
    int64_t c_row0;
};
__device__ __forceinline__ TileWork tile_work(const GemmArgs& g, int tile, int num_m, int num_n, int num_k, int group_m, int block_k) {
    TileWork w;
    w.half = -1;
    int e = 0;
    if (g.k_group_off != nullptr) {
        e = tile / (num_m * num_n);
        tile -= e * num_m * num_n;
    }
    const TileCoord tc = tile_coord(tile, num_m, num_n, group_m, g.m_tile_offset);
    w.m = tc.m;
    w.n = tc.n;
    if (g.k_group_off != nullptr) {
        w.grp = 0;
        w.kb0 = *(g.k_group_off + e) / block_k;
        w.kb1 = *(g.k_group_off + e + 1) / block_k;
        w.c_row0 = static_cast<int64_t>(e) * g.M;
    } else {
        w.grp = g.tile_group != nullptr ? *(g.tile_group + tc.m) : 0;
        w.kb0 = 0;
        w.kb1 = num_k;
        w.c_row0 = 0;
    }
    return w;
}

// 32 rows x 64 columns of the output, one row per lane (packed bf16 pairs), leave as whole 128-byte lines: through shared memory
// (16-byte pieces, xor-swizzled: no bank conflicts) so that eight lanes write one row together.  Stored straight from the
// registers, every instruction touches 32 rows with 16 bytes each, and the 64 KB of a 128 x 256 tile take 4.8 us; this way
// 0.6 us.  That time is exposed in the e4m3 kernel (its epilogue warps promote) and in bf16 products with few K blocks: 32 experts x
// 1024 rows, e4m3 K = 7168 / N = 4096: 1.00 -> 0.96 ms, K = 2048 / N = 7168: 0.66 -> 0.55 ms; bf16 K = 2048: 0.76 -> 0.70 ms.
__device__ __forceinline__ void store_rows_64(uint8_t* stage, const uint32_t (&w)[32], uint8_t* c, int64_t ldc, int row0, int rows, int col0, int cols) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int v = 0; v < 8; ++v)
        *reinterpret_cast<int4*>(stage + lane * 128 + ((v ^ (lane & 7)) * 16)) = make_int4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
    __syncwarp();
    const int v = lane & 7, col = col0 + v * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + (lane >> 3);
        const int4 out = *reinterpret_cast<const int4*>(stage + r * 128 + ((v ^ (r & 7)) * 16));
        if (row0 + r < rows && col + 8 <= cols) *reinterpret_cast<int4*>(c + (static_cast<int64_t>(row0 + r) * ldc + col) * 2) = out;
    }
    __syncwarp();
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

template <int kStages>
struct PipeState {
    int stage = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void advance() {
        if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
        }
    }
};

// Products of few waves overlap their launch with the kernel before, and let the next one start when their last operands have been
// requested: barriers, tensor memory and the launch itself, about 2 us per kernel, are ready when the inputs are.  Not earlier: CTAs of
// the next kernel would wait on SMs that a product of fewer CTAs leaves to an exchange beside it, until the product ends.
// Where the line lies: product -> SwiGLU -> product -> reduction (e4m3, 7168 x 2 x 2048), in turn / overlapped, by waves of the
// products: 0.9 and 1.5: 95.0 / 91.0 us, 3.5 and 6.1: 320 / 315; 5 to 9 waves: the same within 1 %; (2048 x 2 x 1024) 10.4: 280 / 288.
// Layer of 64 tokens 370 / 364, of 4096 tokens (29 and 51 waves) 2187 / 2232; 8192 x 7168 x 7168 in bf16 (14 waves) 683 / 695.
// Launches that wait for others (fused ones, products whose rows are announced by flags) never let another one start beside them: it
// could hold the SMs that they are waiting for.
__host__ __device__ constexpr bool few_waves(int num_tiles, int ctas) { return num_tiles <= 8 * ctas; }

// kMnOperands: how many operands are MN-major (bf16 only).  0: A [M, K], B [N, K].  1: B is [K, N] (data gradients read the forward
// weights as they are).  2: A is [K, M] too (weight gradients read row-major activations and gradients as they are).
// kSplits: a tile's K blocks are shared out over CTAs (g.k_splits), and the sums leave in 32 bits (an instance of its own: the
// branches would cost small products 2 to 4 %)
template <bool kFp8, int kBlockN, int kMnOperands, bool kSplits = false>
__global__ void __launch_bounds__(gemm_threads(kFp8, kBlockN), 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
            const __grid_constant__ std::conditional_t<kFp8 && kBlockN == 256, CUtensorMap, int> map_a32,
            const __grid_constant__ std::conditional_t<kFp8 && kBlockN == 256, CUtensorMap, int> map_b128, const GemmArgs g) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int kStages = num_stages(kBlockN, kFp8);
    constexpr int kTileBytesB = kBlockN * 128;
    constexpr int kAccBufs = (kFp8 && kBlockN == 128) ? 4 : 2;   // accumulator buffers of kBlockN fp32 columns in tensor memory
    constexpr int kEpiWarps = kFp8 ? 8 : 4;
    constexpr bool kWide = kFp8 && kBlockN == 256;   // register re-allocation between warpgroups
    static_assert(!kSplits || (!kFp8 && kBlockN == 128 && kMnOperands == 0), "plain bf16 products of few tiles");
    constexpr int kEpiWarp0 = kWide ? 4 : 2;         // first epilogue warp
    constexpr int kTmemColumns = kAccBufs * kBlockN <= 256 ? 256 : 512;   // allocations are powers of two
    static_assert(kBlockN % 32 == 0 && kBlockN >= 32 && kBlockN <= 256 && kAccBufs * kBlockN <= 512, "tile width");
    uint8_t* s_a = smem;
    uint8_t* s_b = smem + kStages * kTileBytes;
    GemmSmem* sm = reinterpret_cast<GemmSmem*>(smem + kStages * (kTileBytes + kTileBytesB));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kBlockK = kFp8 ? 128 : 64;          // elements per 128-byte row
    constexpr int kUmmaK = kFp8 ? 32 : 16;            // elements per tcgen05.mma (32 bytes of K)
    static_assert(kMnOperands == 0 || (!kFp8 && kBlockN % 64 == 0), "MN-major operands: bf16, whole 64-element chunks");
    constexpr uint32_t kIdesc =
        umma::make_instr_desc(kBlockM, kBlockN, kFp8 ? umma::kFormatE4M3 : umma::kFormatBF16, kMnOperands >= 2, kMnOperands >= 1);
    constexpr uint32_t kIdescHalf = umma::make_instr_desc(kBlockM, 128, umma::kFormatE4M3);
    const int num_m = (g.M + kBlockM - 1) / kBlockM, num_n = (g.N + kBlockN - 1) / kBlockN;
    const int num_k = (g.K + kBlockK - 1) / kBlockK;
    const int num_tiles = num_m * num_n * (g.k_group_off != nullptr ? g.num_groups : 1);
    const int gemm_ctas = static_cast<int>(gridDim.x) - g.num_copy_ctas;
    const bool is_copier = static_cast<int>(blockIdx.x) >= gemm_ctas;
    // The last wave of the wide e4m3 kernel: if it would leave at least half of the CTAs idle, its tiles are cut into halves of 128
    // columns.  This is for products that are bound by reading the weights (one M tile per expert), where the CTAs of a
    // thin last wave cannot pull the bandwidth that is free.
    const int rem = num_tiles % gemm_ctas;
    const bool cut_last = kWide && 2 * rem <= gemm_ctas;
    const int whole_items = cut_last ? num_tiles - rem : num_tiles;
    const int num_items = kSplits ? num_tiles * g.k_splits : cut_last ? num_tiles + rem : num_tiles;
    // output staging: of the 256-column variants, and of the reduce-scatter in the bf16 128-column one (narrow products, mostly of one
    // wave: 64 x 128 x 128 takes 5.0 us with direct stores, 5.3 us staged)
    uint8_t* s_epi = smem + kStages * (kTileBytes + kTileBytesB) + 1024;
    Workspace* ws = g.fuse != EP_GEMM_FUSE_NONE ? local_ws(g.ctx) : nullptr;
    const uint64_t epoch = ws != nullptr ? ws->epoch[EP_CH_GEMM] + 1 : 0;
    const int tiles_per_shard = g.fuse != EP_GEMM_FUSE_NONE ? num_m / g.ctx.num_ranks : num_m;
    // all-gather fusion wants the M tiles in arrival order, so its groups never span two shards
    const int group_m = g.fuse == EP_GEMM_FUSE_ALL_GATHER ? min(8, tiles_per_shard) : 16;

    auto item_work = [&](int item) {
        if constexpr (kSplits) {
            // a part of the K blocks; its sums go to rows of their own in the workspace
            const int part = item / num_tiles;
            TileWork w = tile_work(g, item - part * num_tiles, num_m, num_n, num_k, group_m, kBlockK);
            w.kb0 = num_k * part / g.k_splits;
            w.kb1 = num_k * (part + 1) / g.k_splits;
            w.c_row0 = static_cast<int64_t>(part) * g.M;
            return w;
        }
        if (!kWide || item < whole_items) return tile_work(g, item, num_m, num_n, num_k, group_m, kBlockK);
        TileWork w = tile_work(g, whole_items + (item - whole_items) / 2, num_m, num_n, num_k, group_m, kBlockK);
        w.half = (item - whole_items) & 1;
        return w;
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            ptx::mbar_init(&sm->full[i], 1);
            ptx::mbar_init(&sm->empty[i], 1);
        }
        for (int i = 0; i < kAccBufs; ++i) {
            ptx::mbar_init(&sm->tmem_full[i], 1);
            ptx::mbar_init(&sm->tmem_empty[i], kEpiWarps);
        }
        sm->failed = 0;
        ptx::mbar_fence_init();
        umma::prefetch_tensormap(&map_a);
        umma::prefetch_tensormap(&map_b);
    }
    if (warp == 1) {
        umma::tmem_alloc(&sm->tmem_base, kTmemColumns);
        umma::tmem_relinquish();
    }
    umma::fence_before_thread_sync();
    __syncthreads();
    umma::fence_after_thread_sync();
    const uint32_t tmem_base = sm->tmem_base;
    ptx::wait_for_previous_kernel();
    const bool lets_next_start = g.fuse == EP_GEMM_FUSE_NONE && g.a_ready_flags == nullptr && few_waves(num_items, gemm_ctas);

    if (warp < kEpiWarp0) {
        // ---------------------------------------------------------------------- producer warps
        // wide e4m3 kernel: warps 0-3 (TMA, MMA, two idle) keep 40 registers each so that the epilogue warps can take 232
        if (kWide) reg_dealloc<40>();
        if (warp == 0) {
            // ------------------------------------------------------------------ TMA producer
            // One elected thread, here and in the MMA warp: with `lane == 0` the compiler does not know that a single thread runs the loop,
            // and a stage of three boxes took the producer 336 ns instead of 260 (six boxes 480 / 280), more than its MMAs.
            if (ptx::elect_one()) {
                PipeState<kStages> p;
                bool ok = true;
                for (int tile = blockIdx.x; !is_copier && tile < num_items && ok; tile += gemm_ctas) {
                    const TileWork tw = item_work(tile);
                    const int m_blk = tw.m, n_blk = tw.n, grp = tw.grp;
                    if (grp < 0 || tw.kb1 <= tw.kb0) continue;
                    if (g.fuse == EP_GEMM_FUSE_ALL_GATHER && m_blk / tiles_per_shard != g.ctx.rank) {
                        // rows of a remote shard: wait until a copier CTA of this kernel has landed the tile locally
                        const uint64_t* flag = &ws->tile_flags[m_blk];
                        const uint64_t t0 = gemm_timer();
                        while (ptx::ld_acquire_sys(flag) < epoch) {
                            if (gemm_timer() - t0 > wait_limit_ns(g) || *reinterpret_cast<volatile int*>(&sm->failed)) {
                                gemm_fail<kWide>(g, sm, 3);
                                ok = false;
                                break;
                            }
                        }
                        if (!ok) break;
                        ptx::fence_proxy_async_all();   // the tile was written through the async proxy of another SM
                    }
                    if (g.a_ready_flags != nullptr) {
                        // rows of this M tile arrive from another rank: wait (bounded) for their flag
                        const uint64_t* flag = g.a_ready_flags + (g.a_flag_of_tile != nullptr ? g.a_flag_of_tile[m_blk] : m_blk);
                        const uint64_t t0 = gemm_timer();
                        while (ptx::ld_acquire_sys(flag) < g.a_ready_value) {
                            if (gemm_timer() - t0 > wait_limit_ns(g) || *reinterpret_cast<volatile int*>(&sm->failed)) {
                                gemm_fail<kWide>(g, sm, 3);
                                ok = false;
                                break;
                            }
                        }
                        if (!ok) break;
                    }
                    // A thin tile (few tokens of an expert) is loaded in boxes of 32 rows: the SM's loads in flight are what bounds a
                    // product that streams the weights, and a full box takes a third of them.  The other rows of the stage keep
                    // what they held; their products are not stored.
                    const int a_boxes = kWide && g.tile_rows != nullptr ? min(4, max(1, (*(g.tile_rows + m_blk) + 31) / 32)) : 4;
                    for (int kb = tw.kb0; kb < tw.kb1 && ok; ++kb) {
                        ok = wait_bar<kWide>(&sm->empty[p.stage], p.phase ^ 1, sm, g, 1);
                        if (!ok) break;
                        ptx::mbar_arrive_expect_tx(&sm->full[p.stage], a_boxes * (kTileBytes / 4) + (tw.half >= 0 ? kTileBytesB / 2 : kTileBytesB));
                        if constexpr (kMnOperands >= 2) {
#pragma unroll
                            for (int i = 0; i < kBlockM / 64; ++i)
                                umma::tma_load_3d(s_a + p.stage * kTileBytes + i * umma::kMnChunkBytes, &map_a, m_blk * kBlockM + i * 64, kb * kBlockK, 0,
                                                  &sm->full[p.stage]);
                        } else {
                            if (a_boxes == 4) umma::tma_load_2d(s_a + p.stage * kTileBytes, &map_a, kb * kBlockK, m_blk * kBlockM, &sm->full[p.stage]);
                            if constexpr (kWide) {
                                for (int i = 0; i < (a_boxes & 3); ++i)
                                    umma::tma_load_2d(s_a + p.stage * kTileBytes + i * (kTileBytes / 4), &map_a32, kb * kBlockK, m_blk * kBlockM + i * 32,
                                                      &sm->full[p.stage]);
                            }
                        }
                        if constexpr (kMnOperands >= 1) {
#pragma unroll
                            for (int i = 0; i < kBlockN / 64; ++i)
                                umma::tma_load_3d(s_b + p.stage * kTileBytesB + i * umma::kMnChunkBytes, &map_b, n_blk * kBlockN + i * 64, kb * kBlockK, grp,
                                                  &sm->full[p.stage]);
                        } else if constexpr (kWide) {
                            // the whole tile in one box (128 rows x 4096 x 7168 x 32: 212 us, in two boxes 216), or one half of it
                            const int b_row = grp * g.N + n_blk * kBlockN + (tw.half > 0 ? 128 : 0);
                            umma::tma_load_2d(s_b + p.stage * kTileBytesB, tw.half < 0 ? &map_b : &map_b128, kb * kBlockK, b_row, &sm->full[p.stage]);
                        } else {
                            umma::tma_load_2d(s_b + p.stage * kTileBytesB, &map_b, kb * kBlockK, grp * g.N + n_blk * kBlockN, &sm->full[p.stage]);
                        }
                        p.advance();
                    }
                }
                if (lets_next_start) ptx::let_next_kernel_start();
            }
        } else if (warp == 1) {
            // ------------------------------------------------------------------ MMA issuer
            if (ptx::elect_one()) {
                PipeState<kStages> p;
                int acc = 0;
                uint32_t acc_phase = 0;
                bool ok = true;
                for (int tile = blockIdx.x; !is_copier && tile < num_items && ok; tile += gemm_ctas) {
                    const TileWork tw = item_work(tile);
                    if (tw.grp < 0 || tw.kb1 <= tw.kb0) continue;
                    if (!kFp8) {
                        ok = wait_bar<kWide>(&sm->tmem_empty[acc], acc_phase ^ 1, sm, g, 2);
                        if (!ok) break;
                        umma::fence_after_thread_sync();
                    }
                    for (int kb = tw.kb0; kb < tw.kb1 && ok; ++kb) {
                        ok = wait_bar<kWide>(&sm->full[p.stage], p.phase, sm, g, 4);
                        if (!ok) break;
                        const uint64_t desc_a = kMnOperands >= 2 ? umma::make_smem_desc_mn_sw128(s_a + p.stage * kTileBytes)
                                                                 : umma::make_smem_desc_sw128(s_a + p.stage * kTileBytes);
                        const uint64_t desc_b = kMnOperands >= 1 ? umma::make_smem_desc_mn_sw128(s_b + p.stage * kTileBytesB)
                                                                 : umma::make_smem_desc_sw128(s_b + p.stage * kTileBytesB);
                        // 16 (bf16) / 32 (e4m3) elements of K: 32 bytes along a K-major row, 16 K rows of 128 bytes otherwise
                        constexpr int kStepA = kMnOperands >= 2 ? kUmmaK * 128 : 32, kStepB = kMnOperands >= 1 ? kUmmaK * 128 : 32;
                        if (kFp8) {
                            // e4m3: the accumulator is what everyone waits for, so nothing stands between its hand-over and the MMAs
                            ok = wait_bar<kWide>(&sm->tmem_empty[acc], acc_phase ^ 1, sm, g, 2);
                            if (!ok) break;
                        }
                        umma::fence_after_thread_sync();
#pragma unroll
                        for (int k = 0; k < kBlockK / kUmmaK; ++k) {
                            const uint32_t accumulate = kFp8 ? (k != 0) : (kb != tw.kb0 || k != 0);
                            umma::mma_ss<kFp8>(tmem_base + acc * kBlockN, umma::advance_desc_k(desc_a, k * kStepA),
                                               umma::advance_desc_k(desc_b, k * kStepB), kWide && tw.half >= 0 ? kIdescHalf : kIdesc, accumulate);
                        }
                        if (kFp8) umma::mma_commit(&sm->tmem_full[acc]);   // one 128-channel block is ready for promotion
                        umma::mma_commit(&sm->empty[p.stage]);       // the stage may be refilled once these MMAs are done
                        p.advance();
                        if (kFp8) {
                            if (++acc == kAccBufs) {
                                acc = 0;
                                acc_phase ^= 1;
                            }
                        }
                    }
                    if (!kFp8 && ok) {
                        umma::mma_commit(&sm->tmem_full[acc]);
                        if (++acc == kAccBufs) {
                            acc = 0;
                            acc_phase ^= 1;
                        }
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (32 TMEM lanes per warp)
        if (kWide) reg_alloc<232>();
        const int quad = warp & 3;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        uint8_t* cb = reinterpret_cast<uint8_t*>(g.c);
        for (int tile = blockIdx.x; !is_copier && tile < num_items && ok; tile += gemm_ctas) {
            const TileWork tw = item_work(tile);
            const int m_blk = tw.m, n_blk = tw.n, grp = tw.grp;
            if (grp < 0) continue;
            const int row = m_blk * kBlockM + quad * 32 + lane;
            const int n0 = n_blk * kBlockN;
            if (tw.kb1 <= tw.kb0) {
                // empty K range (an expert without tokens): the product is zero
                if (row < g.M)
                    for (int col = n0; col < min(n0 + kBlockN, g.N); col += 8)
                        *reinterpret_cast<int4*>(cb + ((tw.c_row0 + row) * g.ldc + col) * 2) = make_int4(0, 0, 0, 0);
                continue;
            }
            const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
            if (!kFp8) {
                ok = wait_bar<kWide>(&sm->tmem_full[acc], acc_phase, sm, g, 5);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                umma::fence_after_thread_sync();
                const bool to_peer = kBlockN == 128 && g.fuse == EP_GEMM_FUSE_REDUCE_SCATTER;
                uint8_t* my_stage = s_epi + (quad * 32 + lane) * kEpiRowBytes;
                if (to_peer) {
                    ptx::bulk_wait_read<0>();     // the staging rows were the source of the previous tile's stores
                    __syncwarp();
                }
                if (kBlockN == 256) {
#pragma unroll
                    for (int c = 0; c < kBlockN / 64; ++c) {
                        uint32_t r0[32], r1[32], w[32];
                        umma::tmem_ld_32x32(tmem_base + lane_addr + acc * kBlockN + c * 64, r0);
                        umma::tmem_ld_32x32(tmem_base + lane_addr + acc * kBlockN + c * 64 + 32, r1);
                        umma::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            w[j] = pack_bf16(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1]));
                            w[16 + j] = pack_bf16(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
                        }
                        store_rows_64(s_epi + quad * kOutStageBytes, w, cb + tw.c_row0 * g.ldc * 2, g.ldc, m_blk * kBlockM + quad * 32, g.M, n0 + c * 64, g.N);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < kBlockN / 32; ++c) {
                        uint32_t r[32];
                        umma::tmem_ld_32x32(tmem_base + lane_addr + acc * kBlockN + c * 32, r);
                        umma::tmem_ld_wait();
                        if constexpr (kSplits) {
                            if (row < g.M) {
                                float* sums = g.partial + (tw.c_row0 + row) * g.N + n0 + c * 32;
#pragma unroll
                                for (int v = 0; v < 8; ++v)
                                    if (n0 + c * 32 + v * 4 < g.N) *reinterpret_cast<uint4*>(sums + v * 4) = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
                            }
                        } else if (row < g.M) {
#pragma unroll
                            for (int v = 0; v < 4; ++v) {
                                const int col = n0 + c * 32 + v * 8;
                                if (col + 8 <= g.N) {
                                    int4 out;
                                    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
                                    for (int j = 0; j < 4; ++j)
                                        h[j] = __floats2bfloat162_rn(__uint_as_float(r[v * 8 + 2 * j]), __uint_as_float(r[v * 8 + 2 * j + 1]));
                                    if (to_peer) *reinterpret_cast<int4*>(my_stage + (c * 32 + v * 8) * 2) = out;
                                    else *reinterpret_cast<int4*>(cb + ((tw.c_row0 + row) * g.ldc + col) * 2) = out;
                                }
                            }
                        }
                    }
                }
                if (to_peer) {
                    // GEMM -> reduce-scatter: this row of the partial result goes to the rank that owns it, into the
                    // slot reserved for this source rank (one 256-byte bulk store per row over NVLink)
                    ptx::fence_proxy_async_smem();
                    __syncwarp();
                    const int rows_per_rank = g.M / g.ctx.num_ranks;
                    const int owner = row / rows_per_rank, local_row = row - owner * rows_per_rank;
                    uint8_t* dst = g.ctx.peer_base[owner] + g.off_slots + (epoch & 1) * g.slot_set_bytes +
                                   ((static_cast<int64_t>(g.ctx.rank) * rows_per_rank + local_row) * g.N + n0) * 2;
                    ptx::bulk_store(dst, my_stage, kBlockN * 2);
                    ptx::bulk_commit();
                }
                umma::fence_before_thread_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm->tmem_empty[acc]);
                if (++acc == kAccBufs) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            } else {
                if constexpr (kWide) {
                    // this warp promotes 128 of the 256 columns for its 32 rows; little is kept alive across the K blocks (128 sums and 32
                    // loaded values per thread: with 64, or with the scales of four blocks held ahead, the loop spills)
                    constexpr int kCols = 128;
                    const int col_half = (warp - kEpiWarp0) >> 2;
                    if (tw.half >= 0 && col_half == 1) {
                        // half a tile: the first four warps have all of its columns, these only take part in the hand-over
                        for (int kb = 0; kb < num_k; ++kb) {
                            ok = wait_bar<kWide>(&sm->tmem_full[acc], acc_phase, sm, g, 5);
                            ok = __all_sync(0xffffffffu, ok);
                            if (!ok) break;
                            if (lane == 0) ptx::mbar_arrive(&sm->tmem_empty[acc]);
                            if (++acc == kAccBufs) {
                                acc = 0;
                                acc_phase ^= 1;
                            }
                        }
                        continue;
                    }
                    uint64_t sum2[kCols / 2];   // fp32 pairs (columns 2i, 2i + 1)
#pragma unroll
                    for (int i = 0; i < kCols / 2; ++i) sum2[i] = 0ull;
                    const int num_kb_sf = (g.K + 127) / 128, num_nb_sf = (g.N + 127) / 128;
                    const int nb_sf = min(n0 / 128 + (tw.half > 0 ? 1 : col_half), num_nb_sf - 1);
                    const float* sfb = g.sfb + (static_cast<int64_t>(grp) * num_nb_sf + nb_sf) * num_kb_sf;
                    const float* sfa = g.sfa + min(row, g.M - 1) * g.sfa_stride_row;     // rows past the end are not stored
                    const uint32_t taddr0 = tmem_base + lane_addr + col_half * kCols;
                    // The scales of the next block are requested a whole block ahead and multiplied only when they are used: a product formed
                    // at the load waits for it, and with 230 KB of shared memory taken, L1 keeps few of the scale lines.
                    float sa = *sfa, sb = *sfb;
#pragma unroll 1
                    for (int kb = 0; kb < num_k; ++kb) {
                        const float scale = sa * sb;
                        const uint64_t scale2 = umma::pack_f32x2(__float_as_uint(scale), __float_as_uint(scale));
                        if (kb + 1 < num_k) {
                            sfa += g.sfa_stride_kb;
                            sa = *sfa;
                            sb = *++sfb;
                        }
                        if (!__all_sync(0xffffffffu, ptx::mbar_try_wait(&sm->tmem_full[acc], acc_phase))) {
                            ok = wait_bar<kWide>(&sm->tmem_full[acc], acc_phase, sm, g, 5);
                            ok = __all_sync(0xffffffffu, ok);
                            if (!ok) break;
                        }
                        umma::fence_after_thread_sync();
                        const uint32_t taddr = taddr0 + acc * kBlockN;
#pragma unroll
                        for (int c = 0; c < kCols / 32; ++c) {
                            uint32_t r[32];
                            umma::tmem_ld_32x32(taddr + c * 32, r);
                            umma::tmem_ld_wait();
                            if (c == kCols / 32 - 1) {   // the values are in registers: hand the accumulator back before the arithmetic
                                umma::fence_before_thread_sync();
                                __syncwarp();
                                if (lane == 0) ptx::mbar_arrive(&sm->tmem_empty[acc]);
                            }
#pragma unroll
                            for (int i = 0; i < 16; ++i) umma::fma_f32x2(sum2[c * 16 + i], umma::pack_f32x2(r[2 * i], r[2 * i + 1]), scale2);
                        }
                        if (++acc == kAccBufs) {
                            acc = 0;
                            acc_phase ^= 1;
                        }
                    }
                    if (ok) {
                        const TileWork out = item_work(tile);
                        const int rows_end = g.tile_rows != nullptr ? min(g.M, out.m * kBlockM + *(g.tile_rows + out.m)) : g.M;
#pragma unroll
                        for (int c = 0; c < kCols / 64; ++c) {
                            uint32_t w[32];
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                float lo, hi;
                                umma::unpack_f32x2(sum2[c * 32 + j], lo, hi);
                                w[j] = pack_bf16(lo, hi);
                            }
                            store_rows_64(s_epi + (warp - kEpiWarp0) * kOutStageBytes, w, cb, g.ldc, out.m * kBlockM + quad * 32, rows_end,
                                          out.n * kBlockN + (out.half > 0 ? 1 : col_half) * kCols + c * 64, g.N);
                        }
                    }
                } else {
                    // this warp promotes one half of the tile's columns for its 32 rows
                    constexpr int kCols = kBlockN / 2;
                    const int col_half = (warp - kEpiWarp0) >> 2;
                    uint64_t sum2[kCols / 2];   // fp32 pairs (columns 2i, 2i + 1)
#pragma unroll
                    for (int i = 0; i < kCols / 2; ++i) sum2[i] = 0ull;
                    const int num_kb_sf = (g.K + 127) / 128, num_nb_sf = (g.N + 127) / 128;
                    // the B scale block of this warp's columns (a half tile never straddles two 128-column blocks)
                    const int nb_sf = min((n0 + col_half * kCols) / 128, num_nb_sf - 1);
                    const float* sfb = g.sfb + (static_cast<int64_t>(grp) * num_nb_sf + nb_sf) * num_kb_sf;
                    float scale_next = (row < g.M ? *(g.sfa + row * g.sfa_stride_row) : 0.f) * *sfb;
                    for (int kb = 0; kb < num_k && ok; ++kb) {
                        const uint64_t scale2 = umma::pack_f32x2(__float_as_uint(scale_next), __float_as_uint(scale_next));
                        if (kb + 1 < num_k)
                            scale_next = (row < g.M ? *(g.sfa + row * g.sfa_stride_row + (kb + 1) * g.sfa_stride_kb) : 0.f) * *(sfb + kb + 1);
                        ok = wait_bar<kWide>(&sm->tmem_full[acc], acc_phase, sm, g, 5);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        umma::fence_after_thread_sync();
                        const uint32_t taddr = tmem_base + lane_addr + acc * kBlockN + col_half * kCols;
                        uint32_t r0[32], r1[32];
                        umma::tmem_ld_32x32(taddr, r0);
                        umma::tmem_ld_32x32(taddr + 32, r1);
                        umma::tmem_ld_wait();
                        // the values are in registers: hand the buffer back before the arithmetic
                        umma::fence_before_thread_sync();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(&sm->tmem_empty[acc]);
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            umma::fma_f32x2(sum2[i], umma::pack_f32x2(r0[2 * i], r0[2 * i + 1]), scale2);
                            umma::fma_f32x2(sum2[16 + i], umma::pack_f32x2(r1[2 * i], r1[2 * i + 1]), scale2);
                        }
                        if (++acc == kAccBufs) {
                            acc = 0;
                            acc_phase ^= 1;
                        }
                    }
                    if (ok && row < g.M) {
#pragma unroll
                        for (int v = 0; v < kCols / 8; ++v) {
                            const int col = n0 + col_half * kCols + v * 8;
                            if (col + 8 <= g.N) {
                                int4 out;
                                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    float lo, hi;
                                    umma::unpack_f32x2(sum2[v * 4 + j], lo, hi);
                                    h[j] = __floats2bfloat162_rn(lo, hi);
                                }
                                *reinterpret_cast<int4*>(cb + (static_cast<int64_t>(row) * g.ldc + col) * 2) = out;
                            }
                        }
                    }
                }
            }
        }
    }
    constexpr int kCopyWarps = copy_warps(kBlockN);
    static_assert(kFp8 || kCopyWarps * 2 * 16384 <= num_stages(kBlockN, false) * stage_bytes(kBlockN), "copy staging must fit in front of the barriers");
    if (!kFp8 && g.fuse == EP_GEMM_FUSE_ALL_GATHER && is_copier && warp < kCopyWarps) {
        // ------------------------------------------------------------------ all-gather fused into this kernel
        // Copier CTAs pull the remote shards of A, one 128-row tile at a time, from the owners' symmetric buffers
        // (TMA bulk loads over NVLink, no multicast) into the local copy and publish one flag per tile.
        const RankCtx& ctx = g.ctx;
        const int copier = static_cast<int>(blockIdx.x) - gemm_ctas;
        const int row_bytes = g.K * (kFp8 ? 1 : 2);
        uint8_t* stage = smem + static_cast<size_t>(warp) * 2 * 16384;
        uint64_t* bars = sm->copy_bar[warp];
        if (lane == 0) {
            ptx::mbar_init(&bars[0], 1);
            ptx::mbar_init(&bars[1], 1);
            ptx::mbar_fence_init();
        }
        __syncwarp();
        bool alive = !is_aborted(ws);
        // every rank's shard must be in place: the first copier runs the cross-GPU barrier, the others wait for it
        uint64_t* entry_word = &ws->tile_flags[EP_MAX_TILE_FLAGS - 1];
        if (copier == 0 && warp == 0) {
            if (lane < ctx.num_ranks) {
                Workspace* pws = reinterpret_cast<Workspace*>(ctx.peer_base[lane]);
                ptx::red_add_release_sys(&pws->xbar[EP_CH_GEMM][ctx.rank], 1ull);
                const uint64_t* mine = &ws->xbar[EP_CH_GEMM][lane];
                alive = bounded_wait(
                    ctx, ws, EP_PH_XGPU_BARRIER, lane, 2 * epoch - 1, [&] { return ptx::ld_acquire_sys(mine) >= 2 * epoch - 1; },
                    [&] { return ptx::ld_relaxed_sys(mine); });
            }
            alive = __all_sync(0xffffffffu, alive);
            if (lane == 0 && alive) ptx::st_release_sys(entry_word, epoch);
        }
        if (alive)
            alive = bounded_wait(
                ctx, ws, EP_PH_TILE_FLAG, -1, epoch, [&] { return ptx::ld_acquire_sys(entry_word) >= epoch; },
                [&] { return ptx::ld_relaxed_sys(entry_word); });
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) sm->failed = 7;
        asm volatile("bar.sync 1, %0;" ::"r"(kCopyWarps * 32) : "memory");
        if (*reinterpret_cast<volatile int*>(&sm->failed)) alive = false;
        // work item = one 128-row tile of a remote shard, visited in the order in which the tensor-core CTAs need
        // them (nearest rank first); each copy warp keeps two row loads in flight
        uint32_t n_loaded = 0;
        const int num_items = (ctx.num_ranks - 1) * tiles_per_shard;
        for (int item = copier; item < num_items && alive; item += g.num_copy_ctas) {
            const int src = (ctx.rank + 1 + item / tiles_per_shard) % ctx.num_ranks;
            const int m_blk = src * tiles_per_shard + item % tiles_per_shard;
            // this warp's rows of the tile, each moved in pieces of at most one 16 KB staging buffer
            constexpr int kPiece = 16384;
            const int pieces = (row_bytes + kPiece - 1) / kPiece;
            const int my_rows = (kBlockM - warp + kCopyWarps - 1) / kCopyWarps * pieces;   // (row, piece) pairs
            auto row_offset = [&](int i) {
                return g.off_full + (static_cast<int64_t>(m_blk) * kBlockM + warp + (i / pieces) * kCopyWarps) * row_bytes + static_cast<int64_t>(i % pieces) * kPiece;
            };
            auto piece_bytes = [&](int i) { return min(kPiece, row_bytes - (i % pieces) * kPiece); };
            auto issue_load = [&](int i) {
                const uint32_t l = n_loaded + i;
                if (lane == 0) {
                    ptx::mbar_arrive_expect_tx(&bars[l & 1], piece_bytes(i));
                    ptx::bulk_load(stage + (l & 1) * kPiece, ctx.peer_base[src] + row_offset(i), piece_bytes(i), &bars[l & 1]);
                }
            };
            ptx::bulk_wait_read<0>();
            __syncwarp();
            issue_load(0);
            for (int i = 0; i < my_rows && alive; ++i) {
                if (i + 1 < my_rows) {
                    ptx::bulk_wait_read<0>();   // the other stage was the source of the previous piece's store
                    __syncwarp();
                    issue_load(i + 1);
                }
                const uint32_t l = n_loaded + i;
                alive = mbar_wait_bounded(ctx, ws, &bars[l & 1], (l >> 1) & 1, EP_PH_COMBINE_LOAD);
                if (!alive) {
                    sm->failed = 7;
                    break;
                }
                if (lane == 0) ptx::bulk_store(ctx.peer_base[ctx.rank] + row_offset(i), stage + (l & 1) * kPiece, piece_bytes(i));
                ptx::bulk_commit();
            }
            n_loaded += my_rows;
            ptx::bulk_wait<0>();
            __threadfence();
            // all copy warps of this CTA have finished their rows of the tile -> publish it
            asm volatile("bar.sync 1, %0;" ::"r"(kCopyWarps * 32) : "memory");
            if (*reinterpret_cast<volatile int*>(&sm->failed)) alive = false;   // same decision in every copy warp
            if (warp == 0 && lane == 0 && alive) ptx::st_release_sys(&ws->tile_flags[m_blk], epoch);
        }
    }
    if (!kFp8 && g.fuse == EP_GEMM_FUSE_REDUCE_SCATTER) {
        ptx::bulk_commit();
        ptx::bulk_wait<0>();
        __threadfence_system();
    }
    umma::fence_before_thread_sync();
    __syncthreads();
    if (warp == 1) umma::tmem_dealloc(tmem_base, kTmemColumns);

    if (!kFp8 && g.fuse != EP_GEMM_FUSE_NONE) {
        // All partial rows have left this rank (RS) / all pulls from the peers are done (AG): cross-GPU barrier.
        const RankCtx& ctx = g.ctx;
        bool alive = grid_sync(ctx, ws, EP_CH_GEMM, EP_PH_GRID_SYNC);
        if (blockIdx.x == 0) {
            // arrival number 2 * epoch of this channel (the AG entry barrier used 2 * epoch - 1)
            int ok = alive ? 1 : 0;
            if (alive && threadIdx.x < ctx.num_ranks) {
                Workspace* pws = reinterpret_cast<Workspace*>(ctx.peer_base[threadIdx.x]);
                if (g.fuse == EP_GEMM_FUSE_REDUCE_SCATTER) ptx::red_add_release_sys(&pws->xbar[EP_CH_GEMM][ctx.rank], 1ull);   // stands in for the entry arrival
                ptx::red_add_release_sys(&pws->xbar[EP_CH_GEMM][ctx.rank], 1ull);
                const uint64_t* mine = &ws->xbar[EP_CH_GEMM][threadIdx.x];
                ok = bounded_wait(
                    ctx, ws, EP_PH_XGPU_BARRIER, threadIdx.x, 2 * epoch, [&] { return ptx::ld_acquire_sys(mine) >= 2 * epoch; },
                    [&] { return ptx::ld_relaxed_sys(mine); });
            }
            alive = __syncthreads_and(ok) != 0;
        }
        alive = grid_sync(ctx, ws, EP_CH_GEMM, EP_PH_GRID_SYNC) && alive;
        if (g.fuse == EP_GEMM_FUSE_REDUCE_SCATTER && alive) {
            // every rank's partial rows for this rank have arrived: sum the R slots in rank order in fp32
            const int rows_per_rank = g.M / ctx.num_ranks;
            const int64_t vecs = static_cast<int64_t>(rows_per_rank) * g.N / 8;
            const uint8_t* slots = ctx.peer_base[ctx.rank] + g.off_slots + (epoch & 1) * g.slot_set_bytes;
            const int64_t slot_bytes = static_cast<int64_t>(rows_per_rank) * g.N * 2;
            for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < vecs; v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
                float acc[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = 0.f;
                for (int r = 0; r < ctx.num_ranks; ++r) {
                    const int4 raw = __ldcg(reinterpret_cast<const int4*>(slots + r * slot_bytes + v * 16));
                    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = __bfloat1622float2(h[j]);
                        acc[2 * j] += f.x;
                        acc[2 * j + 1] += f.y;
                    }
                }
                int4 out;
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
                for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
                *reinterpret_cast<int4*>(reinterpret_cast<uint8_t*>(g.rs_out) + v * 16) = out;
            }
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) ws->epoch[EP_CH_GEMM] = epoch;
    }
}

// ------------------------------------------------------------------------------------------------ products that stream the weights
// e4m3 products with at most one M tile per group (decode layers, short prompts): every weight is read once and the tokens decide
// nothing, so this kernel is built around how the weights arrive.
//   * A stage is 128 weight rows x 256 bytes, two TMA boxes side by side.  What streams 32 x 4096 x 7168 and 32 x 7168 x 2048 bytes from
//     HBM, boxes alone (148 SMs): 256 rows x 128 bytes 154 / 82 us, 128 x 256 141 / 77, 64 x 512 138 / 74, boxes of 32 rows 173 / 95
//     (a box costs its issuer 35 to 60 ns whatever its size).
//   * Operands change places: the 128 weight rows are the M of the MMA and the tokens, as many as the tile has (in steps of 16), its
//     N, so nothing is multiplied, read from tensor memory or promoted for rows that do not exist.  Same sums, same bits.  Tiles of more
//     than 64 token rows keep the usual places: with one scale per value instead of one per thread, 128 rows of 7168 x 2048 take
//     137 us instead of 110.
//   * Tokens come from L2 through a ring and a producer of their own; scales are multiplied and put into shared memory by a
//     fourth warp (reading them four K blocks ahead changes nothing).  Two accumulators of a stage (two K blocks of 128 columns each).
//   * The tiles of a last wave that would use at most half (a quarter) of the CTAs are cut into pieces of 64 (32) weight rows.
// warp 0: weights, 1: MMA, 2: tokens, 3: scales, 4-11: epilogue (32 weight rows each; two warps share the tokens, 16 by 16).
// Bound by HBM where the weights do not fit L2: 32 experts of 16 token rows, 4096 x 7168 at 6.7 TB/s (5.6 in the 256-column kernel), 7168 x
// 2048 at 5.9 (5.0); a plain copy moves 6.5.  The second is short of it by its epilogues: one per 16 K blocks.
constexpr int kStreamStagesW = 4, kStreamStagesA = 3, kStreamKb = 2, kStreamAccs = 2, kStreamScaleSlots = 2;
constexpr int kStreamThreads = 384, kStreamEpiWarps = 8;
constexpr int kStreamStageBytes = kStreamKb * kTileBytes;
struct StreamSmem {
    uint64_t w_full[kStreamStagesW], w_empty[kStreamStagesW], a_full[kStreamStagesA], a_empty[kStreamStagesA];
    uint64_t acc_full[kStreamAccs], acc_empty[kStreamAccs], sc_full[kStreamScaleSlots], sc_empty[kStreamScaleSlots];
    uint32_t tmem_base;
    int failed;
};
static_assert(sizeof(StreamSmem) <= 512, "barrier block");
constexpr int kStreamSwapRows = 64;      // token rows up to which the operands change places
constexpr int kStreamScaleBytes = kStreamScaleSlots * kStreamKb * kBlockM * 4;
constexpr int kStreamSmemBytes = (kStreamStagesW + kStreamStagesA) * kStreamStageBytes + 512 + kStreamScaleBytes;
static_assert(kStreamSmemBytes <= 232448, "shared memory of a CTA");

// pieces that a tile of the last wave is cut into
__host__ __device__ constexpr int stream_cut(int num_tiles, int ctas) {
    const int rem = num_tiles % ctas;
    return rem == 0 ? 1 : rem * 4 <= ctas ? 4 : rem * 2 <= ctas ? 2 : 1;
}
struct StreamItem {
    int m, col0, out_rows;    // M tile, first weight row of the group, weight rows of this piece
    int grp, rows;            // group (-1: none), token rows
};

__global__ void __launch_bounds__(kStreamThreads, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_a32, const __grid_constant__ CUtensorMap map_w,
                   const __grid_constant__ CUtensorMap map_w32, const GemmArgs g) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* s_w = smem;
    uint8_t* s_a = smem + kStreamStagesW * kStreamStageBytes;
    StreamSmem* sm = reinterpret_cast<StreamSmem*>(s_a + kStreamStagesA * kStreamStageBytes);
    float* s_scale = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(sm) + 512);      // [slot][K block][token]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_m = (g.M + kBlockM - 1) / kBlockM, num_n = (g.N + 127) / 128, num_k = (g.K + 127) / 128;
    const int num_tiles = num_m * num_n, ctas = static_cast<int>(gridDim.x);
    const int cut = stream_cut(num_tiles, ctas), whole = cut > 1 ? num_tiles - num_tiles % ctas : num_tiles;
    const int num_items = whole + (num_tiles - whole) * cut;
    // item -> piece.  Every role looks an item up before it works on the one in front of it, and looks at what was loaded only
    // afterwards (`busy`): the two loads take a microsecond.
    auto get_item = [&](int item) {
        StreamItem it;
        item = min(item, num_items - 1);
        const int tile = item < whole ? item : whole + (item - whole) / cut, piece = item < whole ? 0 : (item - whole) % cut;
        it.out_rows = item < whole ? 128 : 128 / cut;
        it.m = tile / num_n;
        it.col0 = (tile - it.m * num_n) * 128 + piece * it.out_rows;
        it.rows = *(g.tile_rows + it.m);
        it.grp = g.tile_group != nullptr ? *(g.tile_group + it.m) : 0;
        return it;
    };
    auto weights_as_m = [](const StreamItem& it) { return it.rows <= kStreamSwapRows; };
    auto busy = [&](StreamItem& it) {
        it.rows = min(it.rows, min(kBlockM, g.M - it.m * kBlockM));
        return it.grp >= 0 && it.rows > 0 && it.col0 < g.N;
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStreamStagesW; ++i) {
            ptx::mbar_init(&sm->w_full[i], 1);
            ptx::mbar_init(&sm->w_empty[i], 1);
        }
        for (int i = 0; i < kStreamStagesA; ++i) {
            ptx::mbar_init(&sm->a_full[i], 1);
            ptx::mbar_init(&sm->a_empty[i], 1);
        }
        for (int i = 0; i < kStreamAccs; ++i) {
            ptx::mbar_init(&sm->acc_full[i], 1);
            ptx::mbar_init(&sm->acc_empty[i], kStreamEpiWarps);
        }
        for (int i = 0; i < kStreamScaleSlots; ++i) {
            ptx::mbar_init(&sm->sc_full[i], 1);
            ptx::mbar_init(&sm->sc_empty[i], kStreamEpiWarps);
        }
        sm->failed = 0;
        ptx::mbar_fence_init();
        umma::prefetch_tensormap(&map_a);
        umma::prefetch_tensormap(&map_w);
    }
    if (warp == 1) {
        umma::tmem_alloc(&sm->tmem_base, 512);
        umma::tmem_relinquish();
    }
    umma::fence_before_thread_sync();
    __syncthreads();
    umma::fence_after_thread_sync();
    const uint32_t tmem_base = sm->tmem_base;
    ptx::wait_for_previous_kernel();

    if (warp == 0) {
        // ---------------------------------------------------------------------- weights
        if (ptx::elect_one()) {
            PipeState<kStreamStagesW> p;
            bool ok = true;
            StreamItem next = get_item(blockIdx.x);
            for (int item = blockIdx.x; item < num_items && ok; item += ctas) {
                StreamItem it = next;
                next = get_item(item + ctas);
                if (!busy(it)) continue;
                const int row = it.grp * g.N + it.col0;
                for (int kb = 0; kb < num_k; kb += kStreamKb) {
                    ok = wait_bar<false>(&sm->w_empty[p.stage], p.phase ^ 1, sm, g, 1);
                    if (!ok) break;
                    uint8_t* dst = s_w + p.stage * kStreamStageBytes;
                    const int blocks = min(kStreamKb, num_k - kb);
                    ptx::mbar_arrive_expect_tx(&sm->w_full[p.stage], blocks * it.out_rows * 128);
                    if (it.out_rows == 128) {
                        umma::tma_load_2d(dst, &map_w, kb * 128, row, &sm->w_full[p.stage]);
                        if (blocks > 1) umma::tma_load_2d(dst + kTileBytes, &map_w, (kb + 1) * 128, row, &sm->w_full[p.stage]);
                    } else {
                        for (int j = 0; j < blocks; ++j)
                            for (int r = 0; r < it.out_rows; r += 32)
                                umma::tma_load_2d(dst + j * kTileBytes + r * 128, &map_w32, (kb + j) * 128, row + r, &sm->w_full[p.stage]);
                    }
                    p.advance();
                }
            }
            // by the thread that has requested the last weights: one thread speaks for its CTA, and the lanes that were not elected are here at once
            if (few_waves(num_tiles, ctas)) ptx::let_next_kernel_start();
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------------- MMA issuer
        if (ptx::elect_one()) {
            PipeState<kStreamStagesW> pw;
            PipeState<kStreamStagesA> pa;
            PipeState<kStreamAccs> acc;
            bool ok = true;
            StreamItem next = get_item(blockIdx.x);
            for (int item = blockIdx.x; item < num_items && ok; item += ctas) {
                StreamItem it = next;
                next = get_item(item + ctas);
                if (!busy(it)) continue;
                const bool swap = weights_as_m(it);
                const uint32_t idesc = umma::make_instr_desc(128, swap ? (it.rows + 15) / 16 * 16 : it.out_rows, umma::kFormatE4M3);
                for (int kb = 0; kb < num_k && ok; kb += kStreamKb) {
                    ok = wait_bar<false>(&sm->a_full[pa.stage], pa.phase, sm, g, 4) && wait_bar<false>(&sm->w_full[pw.stage], pw.phase, sm, g, 4) &&
                         wait_bar<false>(&sm->acc_empty[acc.stage], acc.phase ^ 1, sm, g, 2);
                    if (!ok) break;
                    umma::fence_after_thread_sync();
                    const uint64_t desc_w = umma::make_smem_desc_sw128(s_w + pw.stage * kStreamStageBytes);
                    const uint64_t desc_a = umma::make_smem_desc_sw128(s_a + pa.stage * kStreamStageBytes);
                    const uint64_t desc_m = swap ? desc_w : desc_a, desc_n = swap ? desc_a : desc_w;
#pragma unroll
                    for (int j = 0; j < kStreamKb; ++j) {
                        if (kb + j >= num_k) break;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma::mma_ss<true>(tmem_base + (acc.stage * kStreamKb + j) * 128, umma::advance_desc_k(desc_m, j * kTileBytes + k * 32),
                                               umma::advance_desc_k(desc_n, j * kTileBytes + k * 32), idesc, k != 0);
                    }
                    umma::mma_commit(&sm->acc_full[acc.stage]);
                    acc.advance();
                    umma::mma_commit(&sm->w_empty[pw.stage]);
                    umma::mma_commit(&sm->a_empty[pa.stage]);
                    pw.advance();
                    pa.advance();
                }
            }
        }
    } else if (warp == 2) {
        // ---------------------------------------------------------------------- tokens
        if (ptx::elect_one()) {
            PipeState<kStreamStagesA> p;
            bool ok = true;
            StreamItem next = get_item(blockIdx.x);
            for (int item = blockIdx.x; item < num_items && ok; item += ctas) {
                StreamItem it = next;
                next = get_item(item + ctas);
                if (!busy(it)) continue;
                const int boxes = (it.rows + 31) / 32, row = it.m * kBlockM;
                for (int kb = 0; kb < num_k; kb += kStreamKb) {
                    ok = wait_bar<false>(&sm->a_empty[p.stage], p.phase ^ 1, sm, g, 1);
                    if (!ok) break;
                    const int blocks = min(kStreamKb, num_k - kb);
                    ptx::mbar_arrive_expect_tx(&sm->a_full[p.stage], blocks * boxes * (kTileBytes / 4));
                    for (int j = 0; j < blocks; ++j) {
                        uint8_t* dst = s_a + p.stage * kStreamStageBytes + j * kTileBytes;
                        if (boxes == 4) umma::tma_load_2d(dst, &map_a, (kb + j) * 128, row, &sm->a_full[p.stage]);
                        else
                            for (int i = 0; i < boxes; ++i) umma::tma_load_2d(dst + i * (kTileBytes / 4), &map_a32, (kb + j) * 128, row + i * 32, &sm->a_full[p.stage]);
                    }
                    p.advance();
                }
            }
        }
    } else if (warp == 3) {
        // ---------------------------------------------------------------------- scales: (token's x weight block's) of a stage's K blocks
        PipeState<kStreamScaleSlots> p;
        bool ok = true;
        StreamItem next = get_item(blockIdx.x);
        for (int item = blockIdx.x; item < num_items && ok; item += ctas) {
            StreamItem it = next;
            next = get_item(item + ctas);
            if (!busy(it)) continue;
            const float* sfb = g.sfb + (static_cast<int64_t>(it.grp) * num_n + it.col0 / 128) * num_k;
            const float* sfa = g.sfa + (static_cast<int64_t>(it.m) * kBlockM + lane) * g.sfa_stride_row;
            for (int kb = 0; kb < num_k; kb += kStreamKb) {
                float v[kStreamKb][kBlockM / 32];
#pragma unroll
                for (int j = 0; j < kStreamKb; ++j) {
                    const int k = min(kb + j, num_k - 1);
                    const float b = sfb[k];
#pragma unroll
                    for (int i = 0; i < kBlockM / 32; ++i) v[j][i] = i * 32 + lane < it.rows ? sfa[i * 32 * g.sfa_stride_row + k * g.sfa_stride_kb] * b : 0.f;
                }
                ok = __all_sync(0xffffffffu, wait_bar<false>(&sm->sc_empty[p.stage], p.phase ^ 1, sm, g, 6));
                if (!ok) break;
#pragma unroll
                for (int j = 0; j < kStreamKb; ++j)
#pragma unroll
                    for (int i = 0; i < kBlockM / 32; ++i) s_scale[(p.stage * kStreamKb + j) * kBlockM + i * 32 + lane] = v[j][i];
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm->sc_full[p.stage]);
                p.advance();
            }
        }
    } else {
        // ---------------------------------------------------------------------- epilogue: thread = one weight row, tokens 16 by 16
        const int quad = warp & 3, half = (warp - 4) >> 2;
        const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * 16;
        constexpr int kChunks = 4;          // of 16 tokens per warp: tokens (2 i + half) * 16 ...
        PipeState<kStreamAccs> acc;
        PipeState<kStreamScaleSlots> sc;
        bool ok = true;
        StreamItem next = get_item(blockIdx.x);
        for (int item = blockIdx.x; item < num_items && ok; item += ctas) {
            StreamItem it = next;
            next = get_item(item + ctas);
            if (!busy(it)) continue;
            if (!weights_as_m(it)) {
                // thread = one token, this warp's 64 of the weight rows: one scale per K block instead of one per value
                const int pieces = max(0, min(2, (it.out_rows - half * 64 + 31) / 32));      // of 32 weight rows
                uint64_t sum2[2][16];
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum2[c][i] = 0ull;
#pragma unroll 1
                for (int kb = 0; kb < num_k; kb += kStreamKb) {
                    ok = __all_sync(0xffffffffu, wait_bar<false>(&sm->sc_full[sc.stage], sc.phase, sm, g, 6));
                    if (!ok) break;
                    ok = __all_sync(0xffffffffu, wait_bar<false>(&sm->acc_full[acc.stage], acc.phase, sm, g, 5));
                    if (!ok) break;
                    umma::fence_after_thread_sync();
#pragma unroll
                    for (int j = 0; j < kStreamKb; ++j) {
                        if (kb + j >= num_k) break;
                        const uint32_t scale = __float_as_uint(s_scale[(sc.stage * kStreamKb + j) * kBlockM + quad * 32 + lane]);
                        const uint64_t scale2 = umma::pack_f32x2(scale, scale);
                        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + (acc.stage * kStreamKb + j) * 128 + half * 64;
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            if (c >= pieces) break;
                            uint32_t r[32];
                            umma::tmem_ld_32x32(taddr + c * 32, r);
                            umma::tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; ++i) umma::fma_f32x2(sum2[c][i], umma::pack_f32x2(r[2 * i], r[2 * i + 1]), scale2);
                        }
                    }
                    umma::fence_before_thread_sync();
                    __syncwarp();
                    if (lane == 0) {
                        ptx::mbar_arrive(&sm->acc_empty[acc.stage]);
                        ptx::mbar_arrive(&sm->sc_empty[sc.stage]);
                    }
                    acc.advance();
                    sc.advance();
                }
                if (!ok) break;
                if (quad * 32 + lane < it.rows) {
                    uint8_t* c_row = reinterpret_cast<uint8_t*>(g.c) + ((static_cast<int64_t>(it.m) * kBlockM + quad * 32 + lane) * g.ldc + it.col0 + half * 64) * 2;
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            int4 out;
                            uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                float lo, hi;
                                umma::unpack_f32x2(sum2[c][4 * v + i], lo, hi);
                                o[i] = pack_bf16(lo, hi);
                            }
                            if (c < pieces && it.col0 + half * 64 + c * 32 + v * 8 < g.N) *reinterpret_cast<int4*>(c_row + (c * 32 + v * 8) * 2) = out;
                        }
                }
                continue;
            }
            const int chunks = max(0, (it.rows - half * 16 + 31) / 32);      // of this warp that hold tokens
            float sum[kChunks][16];
#pragma unroll
            for (int i = 0; i < kChunks; ++i)
#pragma unroll
                for (int t = 0; t < 16; ++t) sum[i][t] = 0.f;
#pragma unroll 1
            for (int kb = 0; kb < num_k; kb += kStreamKb) {
                ok = __all_sync(0xffffffffu, wait_bar<false>(&sm->sc_full[sc.stage], sc.phase, sm, g, 6));
                if (!ok) break;
                ok = __all_sync(0xffffffffu, wait_bar<false>(&sm->acc_full[acc.stage], acc.phase, sm, g, 5));
                if (!ok) break;
                umma::fence_after_thread_sync();
#pragma unroll
                for (int j = 0; j < kStreamKb; ++j) {
                    if (kb + j >= num_k) break;
                    const float4* scale = reinterpret_cast<const float4*>(s_scale + (sc.stage * kStreamKb + j) * kBlockM + half * 16);
                    const uint32_t taddr = taddr0 + (acc.stage * kStreamKb + j) * 128;
#pragma unroll
                    for (int i0 = 0; i0 < kChunks; i0 += 2) {        // 32 values in registers at a time
                        if (i0 >= chunks) break;
                        uint32_t r[2][16];
                        umma::tmem_ld_32x16(taddr + i0 * 32, r[0]);
                        if (i0 + 1 < chunks) umma::tmem_ld_32x16(taddr + (i0 + 1) * 32, r[1]);
                        umma::tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            if (i0 + i < chunks)
#pragma unroll
                                for (int v = 0; v < 4; ++v) {
                                    const float4 f = scale[(i0 + i) * 8 + v];
                                    float* d = &sum[i0 + i][4 * v];
                                    d[0] = fmaf(__uint_as_float(r[i][4 * v]), f.x, d[0]);
                                    d[1] = fmaf(__uint_as_float(r[i][4 * v + 1]), f.y, d[1]);
                                    d[2] = fmaf(__uint_as_float(r[i][4 * v + 2]), f.z, d[2]);
                                    d[3] = fmaf(__uint_as_float(r[i][4 * v + 3]), f.w, d[3]);
                                }
                    }
                }
                umma::fence_before_thread_sync();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive(&sm->acc_empty[acc.stage]);
                    ptx::mbar_arrive(&sm->sc_empty[sc.stage]);
                }
                acc.advance();
                sc.advance();
            }
            if (!ok) break;
            // Two lanes trade values so that each has two neighbouring columns of every other token: half the stores, 4 bytes each.
            const int odd = lane & 1, row = quad * 32 + lane, col = it.col0 + row - odd;
            const bool stored = row < it.out_rows && col < g.N;
            uint8_t* c = reinterpret_cast<uint8_t*>(g.c) + ((static_cast<int64_t>(it.m) * kBlockM + half * 16 + odd) * g.ldc + col) * 2;
#pragma unroll
            for (int i = 0; i < kChunks; ++i) {
                if (i >= chunks) break;
#pragma unroll
                for (int t = 0; t < 16; t += 2) {
                    const float got = __shfl_xor_sync(0xffffffffu, odd ? sum[i][t] : sum[i][t + 1], 1);
                    const uint32_t two = odd ? pack_bf16(got, sum[i][t + 1]) : pack_bf16(sum[i][t], got);
                    if (stored && i * 32 + half * 16 + t + odd < it.rows) *reinterpret_cast<uint32_t*>(c + (i * 32 + t) * g.ldc * 2) = two;
                }
            }
        }
    }
    umma::fence_before_thread_sync();
    __syncthreads();
    if (warp == 1) umma::tmem_dealloc(tmem_base, 512);
}

constexpr int kReduceMaxThreads = 1024;
// Adds the parts of a product whose K blocks were shared out, in their order, and rounds once.  Eight columns per thread.
__global__ void __launch_bounds__(kReduceMaxThreads) gemm_reduce_kernel(const GemmArgs g) {
    ptx::wait_for_previous_kernel();
    ptx::let_next_kernel_start();
    const int64_t vecs = static_cast<int64_t>(g.M) * (g.N / 8), part = static_cast<int64_t>(g.M) * g.N;
    for (int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < vecs; v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float* p = g.partial + v * 8;
        float acc[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 4
        for (int s = 0; s < g.k_splits; ++s) {
            const float4 a = *reinterpret_cast<const float4*>(p + s * part), b = *reinterpret_cast<const float4*>(p + s * part + 4);
            acc[0] += a.x;
            acc[1] += a.y;
            acc[2] += a.z;
            acc[3] += a.w;
            acc[4] += b.x;
            acc[5] += b.y;
            acc[6] += b.z;
            acc[7] += b.w;
        }
        const int64_t row = v / (g.N / 8), col = (v - row * (g.N / 8)) * 8;
        *reinterpret_cast<int4*>(reinterpret_cast<uint8_t*>(g.c) + (row * g.ldc + col) * 2) =
            make_int4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
    }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// K-major [rows, K] operand, box = box_rows (32, 128, 224 or 256) rows x 128 bytes, 128B swizzle, out-of-range elements read as zero
bool make_operand_map(CUtensorMap* map, const void* base, int64_t rows, int64_t k, int64_t ld_elems, bool fp8, int box_rows) {
    EncodeTiledFn encode = get_encode_fn();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld_elems * (fp8 ? 1 : 2))};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(fp8 ? 128 : 64), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem_strides[2] = {1, 1};
    return encode(map, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
                  elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// MN-major operand [groups, K, mn] bf16 with contiguous mn: box = 64 elements of mn x 64 K rows of one group, 128B swizzle.  The
// group is a dimension of its own so that K rows past the end of one group read as zero and not as the next group's.
bool make_mn_operand_map(CUtensorMap* map, const void* base, int64_t groups, int64_t k, int64_t mn, int64_t ld_elems) {
    EncodeTiledFn encode = get_encode_fn();
    if (encode == nullptr) return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(mn), static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(groups)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld_elems * 2), static_cast<cuuint64_t>(ld_elems * k * 2)};
    const cuuint32_t box[3] = {64, 64, 1};
    const cuuint32_t elem_strides[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Plain bf16 products of so few tiles that a tile's K blocks can be shared out over several CTAs: bound by one CTA's chain of K blocks (0.15
// to 0.4 us each) on a few SMs otherwise.  A second kernel adds the parts, in 32 bits and always in the same order.  The rule weighs the K
// blocks that a CTA is spared against the second launch and the parts' way through L2, both in K blocks.  In a CUDA graph, whole / split:
// 512 x 1024 x 5000 33.7 / 17.5 us, 74 x 832 x 5704 32.2 / 11.7, 64 x 4096 x 4096 13.0 / 10.3, 296 x 888 x 2184 16.9 / 11.2; not split by it: 128 x 7168 x
// 2048 9.7 / 12.5, 1024^3 6.5 / 9.6, 96 x 2000 x 1600 7.4 / 8.5.
constexpr int kMaxSplits = 16, kMinSplitBlocks = 4, kSplitCost = 16, kSplitBytesPerBlock = 512 * 1024;

// e4m3 products of thin tiles that read every weight once.  Where the lines lie (32 experts, us in runs of half a second, 256-column kernel /
// this one, by token rows of an expert; the first two in bursts of five: 166 / 147 and 92 / 82 at 16 rows, 182 / 183 and 103 / 109 at 128):
//     rows            16          48          64          72          96          128
//     4096 x 7168     197 / 149   205 / 175   205 / 187   210 / 224   210 / 228   219 / 238
//     7168 x 2048     105 / 83    109 / 96    110 / 103   112 / 124   113 / 127   118 / 136
//     2048 x 1024    15.5 / 13.2 16.7 / 15.8 17.2 / 16.7 17.8 / 17.8 18.4 / 18.6 20.0 / 20.4
//     512 x 2048     10.7 / 7.8  11.1 / 9.0  11.0 / 9.5  11.1 / 9.9  11.2 / 10.1 11.1 / 10.3     (weights in L2)
//   * no more M tiles than groups: a second tile of a group reads its weights from L2, and the operand traffic of 128-column tiles bounds the
//     product (which tiles share a group is known on the device only)
//   * at most 56 token rows per tile on average (with uneven routing some tiles have more than 64 then).  A caller who gives no count may have full
//     tiles: the 256-column kernel
constexpr int kStreamMaxRows = 56;

}  // namespace

bool gemm_streams_weights(const GemmArgs& g) {
    const int64_t num_m = (g.M + kBlockM - 1) / kBlockM;
    return g.is_fp8 && g.N >= 256 && g.tile_rows != nullptr && g.fuse == EP_GEMM_FUSE_NONE && g.a_ready_flags == nullptr && g.k_group_off == nullptr &&
           g.mn_operands == 0 && num_m <= g.num_groups && g.total_rows > 0 && g.total_rows <= kStreamMaxRows * num_m;
}

int gemm_k_splits(const GemmArgs& g, int num_sms) {
    if (g.is_fp8 || g.fuse != EP_GEMM_FUSE_NONE || g.mn_operands != 0 || g.k_group_off != nullptr || g.tile_group != nullptr || g.a_ready_flags != nullptr ||
        g.M <= 0 || g.N <= 0 || g.K <= 0)
        return 1;
    const int64_t tiles = static_cast<int64_t>((g.M + kBlockM - 1) / kBlockM) * ((g.N + 127) / 128), num_k = (g.K + 63) / 64;
    const int64_t most = std::min<int64_t>(std::min<int64_t>(num_sms / tiles, num_k / kMinSplitBlocks), kMaxSplits), part_bytes = static_cast<int64_t>(g.M) * g.N * 4;
    int64_t best = 1, best_gain = 0;
    for (int64_t s = 2; s <= most; ++s) {
        const int64_t gain = num_k - (num_k + s - 1) / s - kSplitCost - s * part_bytes / kSplitBytesPerBlock;      // in K blocks
        if (gain > best_gain) best = s, best_gain = gain;
    }
    return static_cast<int>(best);
}

// The kernel that adds the parts stays on the product's SMs: with fewer than the device has, as many CTAs as SMs, and launched when the
// product has ended, since CTAs that wait for its end would do so on the SMs that it leaves to others.
GemmReduceShape gemm_reduce_shape(const GemmArgs& g, int num_sms, int device_sms) {
    GemmReduceShape r;
    const int64_t vecs = static_cast<int64_t>(g.M) * (g.N / 8);
    r.beside_product = num_sms >= device_sms;
    r.threads = r.beside_product ? 256 : kReduceMaxThreads;
    r.ctas = static_cast<int>(std::min<int64_t>(r.beside_product ? 8 * static_cast<int64_t>(device_sms) : num_sms, (vecs + r.threads - 1) / r.threads));
    return r;
}

cudaError_t launch_gemm(const GemmArgs& g, int num_sms, cudaStream_t stream) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0) return cudaSuccess;
    const int elem = g.is_fp8 ? 1 : 2;
    if ((g.lda * elem) % 16 != 0 || (g.ldb * elem) % 16 != 0 || g.ldc % 8 != 0 || g.N % 8 != 0) return cudaErrorInvalidValue;
    if (reinterpret_cast<uintptr_t>(g.a) % 16 != 0 || reinterpret_cast<uintptr_t>(g.b) % 16 != 0 || reinterpret_cast<uintptr_t>(g.c) % 16 != 0)
        return cudaErrorInvalidValue;
    // MN-major operands come in whole 64-element chunks, so they have no 224-column variant.
    // 128 x 256 output tiles (fewer A re-reads, longer MMAs); the reduce-scatter epilogue (which stages 128-column rows)
    // and narrow outputs use 128 x 128 tiles.  The bf16 kernel also has 128 x 224 tiles and takes them when they need less
    // tensor-core time: fewer idle CTAs in the last wave (8192 x 7168: 1792 tiles of 256 columns are 12.1 waves of 148
    // CTAs, paid as 13; 2048 tiles of 224 columns are 13.8 waves of 7/8 the length), or no half-empty last column tile
    // (N = 896 = 4 x 224).
    int block_n = (g.fuse != EP_GEMM_FUSE_REDUCE_SCATTER && g.N >= 256) ? 256 : 128;
    if (block_n == 256 && !g.is_fp8 && g.mn_operands == 0) {
        const int64_t num_m_tiles = (g.M + kBlockM - 1) / kBlockM, groups = g.k_group_off != nullptr ? g.num_groups : 1;
        const int64_t workers = std::max(1, (num_sms < 1 ? 1 : num_sms) - (g.fuse == EP_GEMM_FUSE_ALL_GATHER ? g.num_copy_ctas : 0));
        auto cost = [&](int bn) {
            const int64_t tiles = num_m_tiles * ((g.N + bn - 1) / bn) * groups;
            return (tiles + workers - 1) / workers * (bn + 16);     // waves x (columns + per-tile overhead)
        };
        if (cost(224) < cost(256)) block_n = 224;
        // Few tiles: 128 columns, where that still makes one wave (a K block of half the columns takes about 0.65 of the time).  In a CUDA
        // graph, 256 / 128 columns: 1000 x 2048 x 7168 (64 / 128 tiles) 36.0 / 26.9 us, 64 x 4096 x 4096 (16 / 32) 19.5 / 12.9, 1024^3 (32 / 64)
        // 9.3 / 6.6; with more than a wave of them 1315 x 2536 x 3144 (110 / 220) 32.6 / 44.7.
        if (g.fuse == EP_GEMM_FUSE_NONE && num_m_tiles * ((g.N + 127) / 128) * groups <= workers) block_n = 128;
    }
    if (gemm_streams_weights(g)) {
        CUtensorMap map_a, map_a32, map_w, map_w32;
        const int64_t w_rows = static_cast<int64_t>(g.num_groups) * g.N;
        if (!make_operand_map(&map_a, g.a, g.M, g.K, g.lda, true, 128) || !make_operand_map(&map_a32, g.a, g.M, g.K, g.lda, true, 32) ||
            !make_operand_map(&map_w, g.b, w_rows, g.K, g.ldb, true, 128) || !make_operand_map(&map_w32, g.b, w_rows, g.K, g.ldb, true, 32))
            return cudaErrorInvalidValue;
        const void* fn = (const void*)gemm_stream_kernel;
        const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmemBytes);
        if (err != cudaSuccess) return err;
        const int num_tiles = ((g.M + kBlockM - 1) / kBlockM) * ((g.N + 127) / 128);
        // with fewer tiles than SMs: the pieces that they are cut into (the kernel cuts by the same rule)
        int ctas = num_sms < 1 ? 1 : num_sms;
        if (num_tiles < ctas) ctas = num_tiles * stream_cut(num_tiles, ctas);
        void* params[] = {&map_a, &map_a32, &map_w, &map_w32, const_cast<GemmArgs*>(&g)};
        const dim3 block(kStreamThreads, 1, 1);
        if (few_waves(num_tiles, ctas)) return launch_dependent(fn, dim3(ctas, 1, 1), block, params, kStreamSmemBytes, stream);
        return cudaLaunchKernel(fn, dim3(ctas, 1, 1), block, params, kStreamSmemBytes, stream);
    }
    if (g.mn_operands < 0 || g.mn_operands > 2 || (g.mn_operands != 0 && (g.is_fp8 || g.fuse != EP_GEMM_FUSE_NONE))) return cudaErrorInvalidValue;
    if ((g.mn_operands == 2) != (g.k_group_off != nullptr && g.mn_operands != 0)) return cudaErrorInvalidValue;
    CUtensorMap map_a, map_b, map_a32, map_b128;
    const int64_t b_groups = g.k_group_off != nullptr ? 1 : g.num_groups;
    const bool maps_ok = (g.mn_operands >= 2 ? make_mn_operand_map(&map_a, g.a, 1, g.K, g.M, g.lda)
                                             : make_operand_map(&map_a, g.a, g.M, g.K, g.lda, g.is_fp8, 128)) &&
                         (g.mn_operands >= 1 ? make_mn_operand_map(&map_b, g.b, b_groups, g.K, g.N, g.ldb)
                                             : make_operand_map(&map_b, g.b, b_groups * g.N, g.K, g.ldb, g.is_fp8, block_n));
    if (!maps_ok) return cudaErrorInvalidValue;
    map_a32 = map_a;
    map_b128 = map_b;
    // halves of a thin last wave: only the wide e4m3 kernel reads them
    if (g.is_fp8 && block_n == 256 && !make_operand_map(&map_b128, g.b, b_groups * g.N, g.K, g.ldb, true, 128)) return cudaErrorInvalidValue;
    // boxes of 32 rows for thin tiles: only the wide e4m3 kernel reads them
    if (g.is_fp8 && block_n == 256 && g.tile_rows != nullptr && !make_operand_map(&map_a32, g.a, g.M, g.K, g.lda, true, 32)) return cudaErrorInvalidValue;
    const void* fn;
    if (g.mn_operands == 2) fn = block_n == 256 ? (const void*)gemm_kernel<false, 256, 2> : (const void*)gemm_kernel<false, 128, 2>;
    else if (g.mn_operands == 1) fn = block_n == 256 ? (const void*)gemm_kernel<false, 256, 1> : (const void*)gemm_kernel<false, 128, 1>;
    else if (g.is_fp8) fn = block_n == 256 ? (const void*)gemm_kernel<true, 256, 0> : (const void*)gemm_kernel<true, 128, 0>;
    else fn = block_n == 256   ? (const void*)gemm_kernel<false, 256, 0>
              : block_n == 224 ? (const void*)gemm_kernel<false, 224, 0>
                               : (const void*)gemm_kernel<false, 128, 0>;
    const int kGemmSmemBytes = gemm_smem_bytes(block_n, g.is_fp8 != 0);
    cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmemBytes);
    if (err != cudaSuccess) return err;
    if (g.k_group_off != nullptr && (g.is_fp8 || g.fuse != EP_GEMM_FUSE_NONE || g.tile_group != nullptr || g.num_groups < 1)) return cudaErrorInvalidValue;
    const int num_tiles = ((g.M + kBlockM - 1) / kBlockM) * ((g.N + block_n - 1) / block_n) * (g.k_group_off != nullptr ? g.num_groups : 1);
    int ctas = num_sms < 1 ? 1 : num_sms;
    void* params[] = {&map_a, &map_b, &map_a32, &map_b128, const_cast<GemmArgs*>(&g)};
    if (g.fuse != EP_GEMM_FUSE_NONE) {
        // the CTAs of a fused launch wait on one another (grid barrier, copier -> producer flags): cooperative launch
        const int R = g.ctx.num_ranks;
        if (g.is_fp8 || g.M % (kBlockM * R) != 0 || g.N % 128 != 0 || g.tile_group != nullptr) return cudaErrorInvalidValue;
        if (g.fuse == EP_GEMM_FUSE_ALL_GATHER && (g.num_copy_ctas < 1 || g.num_copy_ctas >= ctas)) return cudaErrorInvalidValue;
        if (g.fuse == EP_GEMM_FUSE_REDUCE_SCATTER && g.num_copy_ctas != 0) return cudaErrorInvalidValue;
        if (g.M / kBlockM >= EP_MAX_TILE_FLAGS - 1) return cudaErrorInvalidValue;
        return cudaLaunchCooperativeKernel(fn, dim3(ctas, 1, 1), dim3(kGemmThreads, 1, 1), params, kGemmSmemBytes, stream);
    }
    if (g.k_splits > 1) {
        // (one wave of 128-column tiles: gemm_k_splits)
        if (fn != (const void*)gemm_kernel<false, 128, 0> || g.partial == nullptr || reinterpret_cast<uintptr_t>(g.partial) % 16 != 0 || g.tile_group != nullptr)
            return cudaErrorInvalidValue;
        fn = (const void*)gemm_kernel<false, 128, 0, true>;
        err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmemBytes);
        if (err != cudaSuccess) return err;
        ctas = std::min(ctas, num_tiles * g.k_splits);
        err = launch_dependent(fn, dim3(ctas, 1, 1), dim3(kGemmThreads, 1, 1), params, kGemmSmemBytes, stream);
        if (err != cudaSuccess) return err;
        int device = 0, device_sms = 0;
        if ((err = cudaGetDevice(&device)) != cudaSuccess || (err = cudaDeviceGetAttribute(&device_sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess)
            return err;
        const GemmReduceShape r = gemm_reduce_shape(g, num_sms, device_sms);
        void* reduce_params[] = {const_cast<GemmArgs*>(&g)};
        const void* reduce = (const void*)gemm_reduce_kernel;
        if (r.beside_product) return launch_dependent(reduce, dim3(r.ctas, 1, 1), dim3(r.threads, 1, 1), reduce_params, 0, stream);
        return cudaLaunchKernel(reduce, dim3(r.ctas, 1, 1), dim3(r.threads, 1, 1), reduce_params, 0, stream);
    }
    // whole tiles, or halves where all of them fit into one wave (the kernel cuts its last wave by the same rule)
    if (ctas > num_tiles) ctas = g.is_fp8 && block_n == 256 && 2 * num_tiles <= ctas ? 2 * num_tiles : num_tiles;
    const dim3 block(gemm_threads(g.is_fp8 != 0, block_n), 1, 1);
    if (few_waves(num_tiles, ctas)) return launch_dependent(fn, dim3(ctas, 1, 1), block, params, kGemmSmemBytes, stream);
    return cudaLaunchKernel(fn, dim3(ctas, 1, 1), block, params, kGemmSmemBytes, stream);
}

}  // namespace ep
