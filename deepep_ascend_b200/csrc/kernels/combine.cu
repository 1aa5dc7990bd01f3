// Expert-parallel combine for one NVLink domain, as ONE kernel per call: the token's home rank PULLS the rows
// that its experts produced straight out of the expert ranks' symmetric buffers (TMA bulk loads through the
// peer mappings, no multicast) and reduces them in fp32 registers, so the reduction is fused into the gather
// and no intermediate slab is written or re-read.  With one rank and at most one row per token a kernel without barrier, claims and
// staging moves the rows instead (combine_local_kernel).
//
// A row is pulled in column chunks of 32 lanes x 16 B x kUnroll; units of work are claimed dynamically by the warps of all CTAs,
// whole tokens first and single chunks at the end (see the body).  Each warp owns a ring of chunk buffers with one mbarrier
// each: while it reduces one chunk, the loads of the following ones are in flight.  The accumulation order is fixed (bias0 +
// bias1 first, then the plan entries in top-k lane order), so results are bitwise reproducible.
//
// What bounds it: a warp's own chain per chunk (wait, read, convert, store, refill), so SM count and warps matter until HBM or the
// link does.  With divisions, queue and claim work per chunk taken off that chain, the claims and plan entries requested ahead,
// and 16 instead of 12 warps, 8192 rows x 7168 (235 MB moved by one rank, before it had the other kernel) took 378 / 104 / 56 / 47 us on
// 8 / 32 / 64 / 148 SMs (before: 717 / 190 / 101 / 53); 24 warps with 2 KB chunks were slower (403 / 111 / 63 / 47).
//
// There is no grid-wide barrier and no exit barrier.  Entry: CTA 0 signals every peer, every CTA watches the peers'
// signals itself (all ranks' input rows are in place once all ranks have entered the call).  Exit: the caller
// alternates between two input regions, and a rank can only pass the entry barrier of call n + 1 after every rank has
// entered it, i.e. has finished pulling for call n; so the region of call n is free again when call n + 1 returns.
//
// Parity: does the work of combine_impl + combine_reduce_epilogue_impl
// (deep_ep/include/deep_ep/impls/combine.cuh:15-243, combine_reduce_epilogue.cuh:12-143) plus the weighted
// reduction of the legacy low-latency combine (csrc/kernels/legacy/internode_ll.cu:1033-1136).
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace ep {

namespace {

constexpr int kCombineMaxWarps = 16;
constexpr int kCombineMaxRing = 32;              // chunk buffers (and mbarriers) per warp
constexpr int kCombineSmemBudget = 208 * 1024;
constexpr int kCombineQueue = 32;                // queue of started units per warp (producer -> consumer)

template <int kUnroll>
struct CombineCfg {
    static constexpr int kChunkBytes = 32 * 16 * kUnroll;
};

// Shared-memory plan: [peer table | mbarriers W x ring | unit queues W | chunk buffers W x ring]
struct CombineSmemPlan {
    int num_warps, ring, off_bar, off_queue, off_data, total;
};
__host__ __device__ inline CombineSmemPlan combine_smem_plan(int chunk_bytes, int num_warps) {
    CombineSmemPlan p;
    p.num_warps = num_warps;
    p.off_bar = 128;
    p.off_queue = 128 + num_warps * kCombineMaxRing * 8;
    p.off_data = p.off_queue + num_warps * kCombineQueue * 16;   // int4 per unit: token, first chunk, end chunk, source lanes
    p.off_data = (p.off_data + 1023) / 1024 * 1024;
    int ring = (kCombineSmemBudget - p.off_data) / (num_warps * chunk_bytes);
    p.ring = ring > kCombineMaxRing ? kCombineMaxRing : ring;
    p.total = p.off_data + num_warps * p.ring * chunk_bytes;
    return p;
}

// kFull: the row is a whole number of chunks, so no lane of a chunk is idle
template <int kUnroll, bool kFull>
__device__ __forceinline__ void combine_body(const CombineArgs& a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int kChunk = CombineCfg<kUnroll>::kChunkBytes;
    const RankCtx& ctx = a.ctx;
    Workspace* ws = local_ws(ctx);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int num_warps = blockDim.x >> 5;
    const int K = a.num_topk, T = a.num_tokens;
    const int row_bytes = a.hidden * 2;
    const int num_chunks = (row_bytes + kChunk - 1) / kChunk;
    const CombineSmemPlan sp = combine_smem_plan(kChunk, num_warps);
    const int ring = sp.ring;

    uint8_t** s_peer = reinterpret_cast<uint8_t**>(smem);
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + sp.off_bar) + warp * kCombineMaxRing;
    uint8_t* s_data = smem + sp.off_data + static_cast<size_t>(warp) * ring * kChunk;
    int4* s_queue = reinterpret_cast<int4*>(smem + sp.off_queue) + warp * kCombineQueue;
    // every CTA reads the entry-barrier sequence before it arrives anywhere; the last CTA to finish writes the new one
    const uint64_t entry_seq = *reinterpret_cast<volatile uint64_t*>(&ws->comb_seq) + 1;

    if (tid < EP_MAX_RANKS) s_peer[tid] = tid < ctx.num_ranks ? ctx.peer_base[tid] : nullptr;
    if (lane == 0)
        for (int b = 0; b < ring; ++b) ptx::mbar_init(&s_bar[b], 1);
    ptx::mbar_fence_init();
    __syncthreads();
    ptx::fence_proxy_async_smem();

    auto stamp = [&](int i) {
        if (a.prof != nullptr && blockIdx.x == 0 && tid == 0) a.prof[i] = globaltimer_ns();
    };
    stamp(0);
    // every rank's input rows must be in place before anyone pulls: CTA 0 tells the peers that this rank has entered
    // the call (stream order puts its rows before the kernel), every CTA waits for all peers' words itself
    bool alive = !is_aborted(ws);
    {
        int ok = alive ? 1 : 0;
        if (alive && tid < ctx.num_ranks) {
            if (blockIdx.x == 0) ptx::red_add_release_sys(&reinterpret_cast<Workspace*>(s_peer[tid])->xbar[EP_CH_COMBINE][ctx.rank], 1ull);
            const uint64_t* mine = &ws->xbar[EP_CH_COMBINE][tid];
            ok = bounded_wait(
                ctx, ws, EP_PH_COMBINE_ENTRY, tid, entry_seq, [&] { return ptx::ld_acquire_sys(mine) >= entry_seq; },
                [&] { return ptx::ld_relaxed_sys(mine); });
        }
        alive = __syncthreads_and(ok) != 0;
    }
    stamp(1);

    // Units of work: the first `whole` tokens are one unit each, every later token is num_chunks units of one chunk (about one
    // token per warp, so that no warp is left with a long tail).  Every warp's first unit is fixed; later ones are claimed from a
    // counter shared by all CTAs of this rank (SMs that get a smaller share of the NVLink bandwidth claim fewer), which is zero
    // at entry: the last CTA of every call clears it.  The producer side of a warp keeps two claims ahead: while the loads of one
    // unit are issued, the plan entries of the next are on their way and the atomic of the one after has been sent, so neither
    // latency is paid per token.  Started units travel through a small queue to the consumer side, which follows in order.
    if (alive) {
        const int total_warps = static_cast<int>(gridDim.x) * num_warps;
        const int whole = max(0, T - total_warps);
        const int num_units = whole + (T - whole) * num_chunks;
        auto unit_token = [&](int u) { return u < whole ? u : whole + (u - whole) / num_chunks; };
        auto claim = [&]() -> int {      // lane 0 holds the result
            return lane == 0 ? total_warps + static_cast<int>(atomicAdd(&ws->dyn_counter[EP_CH_COMBINE], 1u)) : 0;
        };
        auto load_plan = [&](int u) -> int {
            return u < num_units && lane < K ? __ldg(a.plan + static_cast<int64_t>(unit_token(u)) * K + lane) : -1;
        };
        // producer state: unit whose loads are being issued / the next one / the claim after that
        int p_chunk = 0, p_end = 0, p_plan = -1, p_slot = 0;
        uint32_t p_sources = 0, p_pending = 0;
        int n_unit = warp * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);
        int n_plan = load_plan(n_unit);
        int n_claim = n_unit < num_units ? claim() : 0;
        uint32_t pushed = 0, popped = 0;
        int in_flight = 0;

        // issue loads in sequence order until the ring is full or the work is exhausted
        auto issue_ahead = [&]() {
            while (in_flight < ring) {
                if (p_pending == 0) {
                    if (p_sources != 0 && p_chunk + 1 < p_end) {
                        ++p_chunk;
                        p_pending = p_sources;
                    } else {
                        if (n_unit >= num_units || pushed - popped >= kCombineQueue) break;
                        const int tkn = unit_token(n_unit);
                        p_chunk = n_unit < whole ? 0 : (n_unit - whole) - (tkn - whole) * num_chunks;
                        p_end = n_unit < whole ? num_chunks : p_chunk + 1;
                        p_plan = n_plan;
                        p_sources = p_pending = __ballot_sync(0xffffffffu, p_plan >= 0);
                        if (lane == 0) s_queue[pushed % kCombineQueue] = make_int4(tkn, p_chunk, p_end, static_cast<int>(p_sources));
                        ++pushed;
                        n_unit = __shfl_sync(0xffffffffu, n_claim, 0);
                        n_plan = load_plan(n_unit);
                        if (n_unit < num_units) n_claim = claim();
                    }
                    continue;
                }
                const int k = __ffs(p_pending) - 1;
                p_pending &= p_pending - 1;
                const int p = __shfl_sync(0xffffffffu, p_plan, k);
                if (lane == 0) {
                    const int bytes = kFull ? kChunk : min(kChunk, row_bytes - p_chunk * kChunk);
                    const uint8_t* src = s_peer[p >> 24] + a.off_x + static_cast<int64_t>(p & 0xffffff) * row_bytes + p_chunk * kChunk;
                    ptx::mbar_arrive_expect_tx(&s_bar[p_slot], bytes);
                    ptx::bulk_load(s_data + p_slot * kChunk, src, bytes, &s_bar[p_slot]);
                }
                p_slot = p_slot + 1 == ring ? 0 : p_slot + 1;
                ++in_flight;
            }
            __syncwarp();     // queue entries are visible to all lanes
        };

        int c_slot = 0;
        uint32_t c_parity = 0;
        issue_ahead();
        while (popped != pushed && alive) {
            const int4 unit = s_queue[popped % kCombineQueue];
            __syncwarp();
            ++popped;
            const int t = unit.x;
            float mul_k = 1.f;
            if (a.mul_weights != nullptr && lane < K) mul_k = __ldg(a.mul_weights + static_cast<int64_t>(t) * K + lane);
            // weights that travel back with the rows (dispatch backward): one small peer load per lane, stored after the chunk
            const bool with_w = unit.y == 0 && a.out_w != nullptr && lane < K;
            const int w_src = with_w ? __ldg(a.lane_src + static_cast<int64_t>(t) * K + lane) : -1;
            for (int c = unit.y; c < unit.z && alive; ++c) {
                const int col0 = c * kChunk;   // byte offset inside the row
                const int bytes = kFull ? kChunk : min(kChunk, row_bytes - col0);
                float acc[kUnroll * 8];
                bool first = true;             // nothing accumulated yet
                if (a.bias0 != nullptr || a.bias1 != nullptr) {
                    // bias0 + bias1 in fp32 first
                    first = false;
#pragma unroll
                    for (int i = 0; i < kUnroll * 8; ++i) acc[i] = 0.f;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const uint8_t* bias = reinterpret_cast<const uint8_t*>(b == 0 ? a.bias0 : a.bias1);
                        if (bias == nullptr) continue;
#pragma unroll
                        for (int u = 0; u < kUnroll; ++u) {
                            const int off = (u * 32 + lane) * 16;
                            if (kFull || off < bytes) {
                                const int4 raw = ptx::ld_nc_v4(bias + static_cast<int64_t>(t) * row_bytes + col0 + off);
                                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const float2 f = __bfloat1622float2(h[j]);
                                    acc[u * 8 + 2 * j] += f.x;
                                    acc[u * 8 + 2 * j + 1] += f.y;
                                }
                            }
                        }
                    }
                }
                float w_val = 0.f;
                if (c == 0 && with_w && w_src >= 0) {
                    const float* wp = reinterpret_cast<const float*>(s_peer[w_src >> 24] + a.off_w);
                    const int64_t row = w_src & 0xffffff;
                    w_val = *reinterpret_cast<const volatile float*>(a.w_cols == 1 ? wp + row : wp + row * a.w_cols + lane);
                }

                // sources in top-k lane order; each one sits in the next ring buffer
                uint32_t srcs = static_cast<uint32_t>(unit.w);
                while (srcs != 0) {
                    const int k = __ffs(srcs) - 1;
                    srcs &= srcs - 1;
                    alive = mbar_wait_bounded(ctx, ws, &s_bar[c_slot], c_parity, EP_PH_COMBINE_LOAD);
                    if (!alive) break;
                    const float w = __shfl_sync(0xffffffffu, mul_k, k);
                    const uint8_t* buf = s_data + c_slot * kChunk;
                    auto add = [&](auto is_first) {
#pragma unroll
                        for (int u = 0; u < kUnroll; ++u) {
                            const int off = (u * 32 + lane) * 16;
                            const int4 raw = kFull || off < bytes ? *reinterpret_cast<const int4*>(buf + off) : make_int4(0, 0, 0, 0);
                            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 f = __bfloat1622float2(h[j]);
                                acc[u * 8 + 2 * j] = fmaf(w, f.x, decltype(is_first)::value ? 0.f : acc[u * 8 + 2 * j]);
                                acc[u * 8 + 2 * j + 1] = fmaf(w, f.y, decltype(is_first)::value ? 0.f : acc[u * 8 + 2 * j + 1]);
                            }
                        }
                    };
                    if (first) add(std::true_type{});
                    else add(std::false_type{});
                    first = false;
                    // the buffer may be refilled once every lane has read it
                    ptx::fence_proxy_async_smem();
                    __syncwarp();
                    --in_flight;
                    if (++c_slot == ring) {
                        c_slot = 0;
                        c_parity ^= 1;
                    }
                    issue_ahead();
                }
                if (!alive) break;
                if (first) {
#pragma unroll
                    for (int i = 0; i < kUnroll * 8; ++i) acc[i] = 0.f;      // a token without any row
                }
                uint8_t* out = reinterpret_cast<uint8_t*>(a.out) + static_cast<int64_t>(t) * row_bytes + col0;
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) {
                    const int off = (u * 32 + lane) * 16;
                    if (kFull || off < bytes) {
                        int4 raw;
                        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
                        for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(acc[u * 8 + 2 * j], acc[u * 8 + 2 * j + 1]);
                        ptx::st_na_v4(out + off, raw);
                    }
                }
                if (c == 0 && with_w) a.out_w[static_cast<int64_t>(t) * K + lane] = w_val;
            }
            issue_ahead();
        }
        // loads still in flight belong to nobody once the loop was left early: give them time to land so that no
        // copy arrives in shared memory after the CTA has exited
        for (; in_flight > 0; --in_flight) {
            mbar_drain(&s_bar[c_slot], c_parity, 1000ull * 1000 * 1000);
            if (++c_slot == ring) {
                c_slot = 0;
                c_parity ^= 1;
            }
        }
    }

    stamp(2);
    // the last CTA to finish closes the call: new entry-barrier sequence, claim counter back to zero
    if (!arrive_is_last(&ws->arrive[EP_CH_COMBINE][0])) return;
    if (tid == 0) {
        if (a.prof != nullptr) a.prof[3] = globaltimer_ns();
        atomicExch(&ws->dyn_counter[EP_CH_COMBINE], 0u);
        ws->comb_seq = entry_seq;
        ws->epoch[EP_CH_COMBINE] += 1;
    }
}

// ------------------------------------------------------------------------------------------------ one rank
// With one rank and the non-expand layout a token has at most one row, which lies in this GPU's own memory, and there is nobody to
// wait for: no entry barrier, no claims (all SMs see the same bandwidth), no staging.  Units of up to eight 512-byte steps of a
// token's row are dealt out to the warps in turn; a warp requests a whole unit at once, and the plan entries of its next unit with it.
// An SM moves at most 97 GB/s in and out together (plain copies, any number of warps), which is what this reaches: 5003 rows x 7168 on
// 24 SMs 63 us against 80 in the pulling kernel, 8192 rows on 64 SMs 39 against 48, and 5 us less at entry and end.
constexpr int kLocalWarps = 32, kLocalSteps = 8, kStepBytes = 32 * 16;

// fp32 sum of one bf16 row with weight 1, rounded to bf16: the value itself, with -0 as 0 and any NaN as the one NaN
__device__ __forceinline__ int4 single_sum(const int4& raw) {
    int4 out;
    const __nv_bfloat162 zero = __float2bfloat162_rn(0.f);
    const __nv_bfloat162* x = reinterpret_cast<const __nv_bfloat162*>(&raw);
    __nv_bfloat162* y = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = __hadd2_rn(x[j], zero);
    return out;
}

__global__ void __launch_bounds__(kLocalWarps * 32, 1) combine_local_kernel(const __grid_constant__ CombineArgs a) {
    const RankCtx& ctx = a.ctx;
    Workspace* ws = local_ws(ctx);
    const int tid = threadIdx.x, lane = tid & 31;
    const int K = a.num_topk, T = a.num_tokens, row_bytes = a.hidden * 2;
    const uint8_t* base = ctx.peer_base[ctx.rank];
    const uint8_t* xb = base + a.off_x;
    const bool first_thread = blockIdx.x == 0 && tid == 0;
    auto stamp = [&](int i) {
        if (a.prof != nullptr && first_thread) a.prof[i] = globaltimer_ns();
    };
    stamp(0);
    stamp(1);
    const int steps = (row_bytes + kStepBytes - 1) / kStepBytes, parts = (steps + kLocalSteps - 1) / kLocalSteps;
    const int part_bytes = (steps + parts - 1) / parts * kStepBytes;
    const int stride = gridDim.x * (blockDim.x >> 5), stride_t = stride / parts, stride_p = stride - stride_t * parts;
    const int first = (tid >> 5) * gridDim.x + blockIdx.x;
    int t = first / parts, part = first - t * parts;
    auto load_plan = [&](int token) -> int { return token < T && lane < K ? __ldg(a.plan + static_cast<int64_t>(token) * K + lane) : -1; };
    int next_plan = load_plan(t);
    const bool alive = __all_sync(0xffffffffu, !is_aborted(ws));      // the flag can rise at any time: one decision per warp
    while (alive && t < T) {
        const int token = t, col0 = part * part_bytes, end = min(row_bytes, col0 + part_bytes);
        const uint32_t srcs = __ballot_sync(0xffffffffu, next_plan >= 0);
        const int64_t row = __shfl_sync(0xffffffffu, next_plan, srcs != 0 ? __ffs(srcs) - 1 : 0) & 0xffffff;
        const bool with_w = part == 0 && a.out_w != nullptr && lane < K;
        t += stride_t;
        part += stride_p;
        if (part >= parts) {
            part -= parts;
            ++t;
        }
        next_plan = load_plan(t);
        const int off0 = col0 + lane * 16;
        int4 raw[kLocalSteps];
#pragma unroll
        for (int i = 0; i < kLocalSteps; ++i)
            raw[i] = srcs != 0 && off0 + i * kStepBytes < end ? ptx::ld_nc_v4(xb + row * row_bytes + off0 + i * kStepBytes) : make_int4(0, 0, 0, 0);
        if (with_w) {
            // weights that travel back with the rows (dispatch backward)
            const int w_src = __ldg(a.lane_src + static_cast<int64_t>(token) * K + lane);
            const float* wp = reinterpret_cast<const float*>(base + a.off_w) + static_cast<int64_t>(w_src & 0xffffff) * a.w_cols;
            a.out_w[static_cast<int64_t>(token) * K + lane] = w_src >= 0 ? __ldg(a.w_cols == 1 ? wp : wp + lane) : 0.f;
        }
        uint8_t* out = reinterpret_cast<uint8_t*>(a.out) + static_cast<int64_t>(token) * row_bytes;
#pragma unroll
        for (int i = 0; i < kLocalSteps; ++i)
            if (off0 + i * kStepBytes < end) ptx::st_na_v4(out + off0 + i * kStepBytes, single_sum(raw[i]));     // no row: zeros
    }
    stamp(2);
    stamp(3);
    if (first_thread) ws->epoch[EP_CH_COMBINE] += 1;
}

template <int kUnroll, bool kFull>
__global__ void __launch_bounds__(kCombineMaxWarps * 32, 1) combine_kernel(const __grid_constant__ CombineArgs args) {
    combine_body<kUnroll, kFull>(args);
}
template <int kUnroll, bool kFull>
__global__ void __launch_bounds__(kCombineMaxWarps * 32, 1) combine_kernel_multi(const CombineArgs* args) {
    combine_body<kUnroll, kFull>(args[blockIdx.y]);
}
template <int kUnroll>
const void* combine_fn(bool full, int n) {
    if (full) return n == 1 ? (const void*)combine_kernel<kUnroll, true> : (const void*)combine_kernel_multi<kUnroll, true>;
    return n == 1 ? (const void*)combine_kernel<kUnroll, false> : (const void*)combine_kernel_multi<kUnroll, false>;
}
const void* combine_fn(int unroll, bool full, int n) {
    switch (unroll) {
        case 8: return combine_fn<8>(full, n);
        case 7: return combine_fn<7>(full, n);
        case 6: return combine_fn<6>(full, n);
        case 5: return combine_fn<5>(full, n);
        case 4: return combine_fn<4>(full, n);
        case 2: return combine_fn<2>(full, n);
        default: return combine_fn<1>(full, n);
    }
}

// Column chunk = 512 B x unroll.  A warp's chain per chunk, which hardly grows with the chunk, is what bounds the kernel, so a row is cut into
// as few chunks of at most 4 KB as it takes, all alike: 3001 tokens x 4096, six rows each, 64 SMs: 60 us in chunks of 2 KB, 43 us in
// chunks of 4 KB, weighted or not (the sums of a 4 KB chunk take 64 of the 128 registers).
inline int pick_unroll(const CombineArgs& a) {
    const int steps = (a.hidden * 2 + 511) / 512, chunks = (steps + 7) / 8, unroll = (steps + chunks - 1) / chunks;
    return unroll == 3 ? 4 : unroll;
}

}  // namespace

LaunchShape combine_launch_shape(const CombineArgs& a, int num_sms) {
    LaunchShape s;
    s.num_ctas = num_sms < 1 ? 1 : (num_sms > EP_MAX_CTAS ? EP_MAX_CTAS : num_sms);
    const CombineSmemPlan p = combine_smem_plan(512 * pick_unroll(a), kCombineMaxWarps);
    s.num_warps = p.num_warps;
    s.smem_bytes = p.total;
    return s;
}

cudaError_t launch_combine(const CombineArgs* args, int n, int num_sms, cudaStream_t stream) {
    const CombineArgs& a0 = args[0];
    if (n == 1 && a0.one_row && a0.mul_weights == nullptr && a0.bias0 == nullptr && a0.bias1 == nullptr) {
        const int steps = (a0.hidden * 2 + kStepBytes - 1) / kStepBytes, parts = (steps + kLocalSteps - 1) / kLocalSteps;
        const int ctas = num_sms < 1 ? 1 : (num_sms > EP_MAX_CTAS ? EP_MAX_CTAS : num_sms);
        const int64_t units = static_cast<int64_t>(a0.num_tokens) * parts;
        const int warps = static_cast<int>(std::min<int64_t>(kLocalWarps, std::max<int64_t>(1, (units + ctas - 1) / ctas)));
        void* params[] = {const_cast<CombineArgs*>(&a0)};
        return cudaLaunchKernel((const void*)combine_local_kernel, dim3(ctas, 1, 1), dim3(warps * 32, 1, 1), params, 0, stream);
    }
    const LaunchShape shape = combine_launch_shape(a0, num_sms);
    if (shape.smem_bytes > 227 * 1024) return cudaErrorInvalidValue;
    const int unroll = pick_unroll(a0);
    const bool full = a0.hidden * 2 % (512 * unroll) == 0;
    const void* fn = combine_fn(unroll, full, n);
    cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, shape.smem_bytes);
    if (err != cudaSuccess) return err;
    dim3 grid(shape.num_ctas, n, 1), block(shape.num_warps * 32, 1, 1);
    if (n == 1) {
        // no CTA waits on another CTA of its own rank, so a plain launch is enough (and can share the GPU with a
        // compute kernel that is already running)
        void* params[] = {const_cast<CombineArgs*>(&a0)};
        return cudaLaunchKernel(fn, grid, block, params, shape.smem_bytes, stream);
    }
    CombineArgs* dev = nullptr;
    err = cudaMallocAsync(reinterpret_cast<void**>(&dev), sizeof(CombineArgs) * n, stream);
    if (err != cudaSuccess) return err;
    err = cudaMemcpyAsync(dev, args, sizeof(CombineArgs) * n, cudaMemcpyHostToDevice, stream);
    if (err == cudaSuccess) {
        void* params[] = {&dev};
        err = cudaLaunchCooperativeKernel(fn, grid, block, params, shape.smem_bytes, stream);
    }
    cudaFreeAsync(dev, stream);
    return err;
}

}  // namespace ep
