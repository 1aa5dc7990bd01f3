// Element-wise pieces of the MoE expert FFN that sit between the two grouped GEMMs: SwiGLU fused with the
// e4m3 (1x128 scales) cast of the second GEMM's input, so the activation is written once in FP8 instead of being
// written in bf16 and re-read by a separate quantisation kernel; the cast of the weights, the expansion of received rows to
// expert rows and its inverse; and the element-wise kernels of the backward pass.  The layer's backward pass uses the row-major
// ones; those that also write transposed results serve callers of the K-major weight-gradient product (`gemm_kgrouped`).
#include <cuda_fp8.h>

#include <algorithm>

#include "common.cuh"

namespace ep {

namespace {

// A row-per-warp kernel with fewer CTAs than this splits its rows over several warps by columns (grid.y).
constexpr int kWantedCtas = 2 * 148;
inline int column_splits(int ctas, int steps) { return max(1, min(steps, (kWantedCtas + ctas - 1) / max(ctas, 1))); }

// Operands of 16-byte (8-byte) accesses; a kernel that is given others takes a misaligned access, so its launcher refuses them
inline bool aligned(const void* p, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }

// one warp per row (or per part of a row); each step covers 256 channels (two 128-channel scale groups).  The loads of two steps are issued
// before the arithmetic of the first, the sigmoid uses the fast reciprocal (the activation is rounded to bf16 right
// after), and the correctly rounded amax / 448 of a group is computed once per 16 steps by the lane that kept that amax
// (all lanes divide at once) instead of by two lanes in every step.
struct SwigluStep {
    int4 gate, up;
};
__device__ __forceinline__ SwigluStep swiglu_load(const uint8_t* gate, const uint8_t* up, int elem, int I) {
    SwigluStep s;
    if (elem < I) {
        s.gate = ptx::ld_na_v4(gate + elem * 2);
        s.up = ptx::ld_na_v4(up + elem * 2);
    } else {
        s.gate = s.up = make_int4(0, 0, 0, 0);
    }
    return s;
}

__global__ void swiglu_quant_kernel(const SwigluQuantArgs a) {
    ptx::wait_for_previous_kernel();
    ptx::let_next_kernel_start();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= a.rows || (a.valid != nullptr && a.valid[row] == 0)) return;
    // this warp's columns: [first, first + I) of the row
    const int first = blockIdx.y * a.col_chunk, I = min(a.inter - first, a.col_chunk);
    const uint8_t* gate = reinterpret_cast<const uint8_t*>(a.h) + (static_cast<int64_t>(row) * a.ldh + first) * 2;
    const uint8_t* up = gate + static_cast<int64_t>(a.inter) * 2;
    uint8_t* q = reinterpret_cast<uint8_t*>(a.q) + static_cast<int64_t>(row) * a.inter + first;
    float* sf_row = a.sf + static_cast<int64_t>(row) * a.sf_stride_row + (first / 128) * a.sf_stride_col;
    const int iters = (I + 255) / 256, num_groups = (I + 127) / 128;
    float kept = 0.f;                 // amax of the group this lane will divide: step (lane & 15) of the current 16, half lane >> 4
    auto flush_scales = [&](int first_step) {
        const int group = (first_step + (lane & 15)) * 2 + (lane >> 4);
        if (group < num_groups && first_step + (lane & 15) < iters) sf_row[group * a.sf_stride_col] = __fdiv_rn(kept, 448.f);
    };
    SwigluStep cur = swiglu_load(gate, up, lane * 8, I);
    for (int i = 0; i < iters; ++i) {
        const int elem = (i * 32 + lane) * 8;
        const bool in_range = elem < I;
        const SwigluStep nxt = swiglu_load(gate, up, i + 1 < iters ? elem + 256 : I, I);
        float v[8];
        {
            const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&cur.gate);
            const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&cur.up);
            int4 act_raw;
            __nv_bfloat162* ah = reinterpret_cast<__nv_bfloat162*>(&act_raw);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 gf = __bfloat1622float2(gh[j]), uf = __bfloat1622float2(uh[j]);
                const float a0 = __fdividef(gf.x, 1.f + __expf(-gf.x)) * uf.x, a1 = __fdividef(gf.y, 1.f + __expf(-gf.y)) * uf.y;
                // the activation is rounded to bf16 first so that the FP8 cast sees the same values as a bf16 pipeline
                ah[j] = __floats2bfloat162_rn(a0, a1);
                const float2 r = __bfloat1622float2(ah[j]);
                v[2 * j] = r.x;
                v[2 * j + 1] = r.y;
            }
            if (in_range && a.act_bf16 != nullptr)
                *reinterpret_cast<int4*>(reinterpret_cast<uint8_t*>(a.act_bf16) + (static_cast<int64_t>(row) * a.inter + first + elem) * 2) = act_raw;
        }
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
        amax = fmaxf(ptx::warp_max_16(amax), 1e-4f);
        const float scale = __fmul_rn(448.f, __frcp_rn(amax));
        if ((lane & 15) == (i & 15)) kept = amax;
        if (in_range) {
            uint32_t packed[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j] * scale, v[4 * j + 1] * scale), __NV_SATFINITE, __NV_E4M3);
                const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j + 2] * scale, v[4 * j + 3] * scale), __NV_SATFINITE, __NV_E4M3);
                packed[j] = lo | (hi << 16);
            }
            *reinterpret_cast<uint2*>(q + elem) = make_uint2(packed[0], packed[1]);
        }
        if ((i & 15) == 15) flush_scales(i - 15);
        cur = nxt;
    }
    if ((iters & 15) != 0) flush_scales(iters & ~15);
}

// ---------------------------------------------------------------------------------------------- weight casts
// One CTA per 128 x 128 scale block: the whole block sits in the registers of its 256 threads (thread = (row mod 16, 8 columns),
// eight rows each), so the weights are read once and the e4m3 bytes written once; the only other traffic is one scale per block.
// Bound by HBM: the 32 x (4096 x 7168 + 7168 x 2048) bf16 weights of one layer take 0.61 ms (4.2 GB, 6.9 TB/s); the PyTorch passes
// that it replaces (fp32 copy, abs, amax, multiply, cast) took 14 ms.  The amax of bf16 weights is taken two at a time: with one
// compare and select per element the kernel was bound by instruction issue (1.15 ms).
// The arithmetic is that of the PyTorch statement (`quantize_weight_blocks_ref`): amax clamped to 1e-4 with NaN kept,
// q = w * (448 * rcp(amax)), scale = amax * (1 / 448), so the results have the same bits.
constexpr int kWqThreads = 256;
__device__ __forceinline__ float max_keep_nan(float a, float b) {   // a NaN on either side wins
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

template <bool kF32>
__global__ void __launch_bounds__(kWqThreads) weight_quant_kernel(const WeightQuantArgs a) {
    __shared__ float s_amax[kWqThreads / 32];
    const int kb_count = (a.k + 127) / 128, nb_count = (a.n + 127) / 128;
    const int64_t blk = blockIdx.x;
    const int kb = static_cast<int>(blk % kb_count);
    const int64_t gn = blk / kb_count;
    const int nb = static_cast<int>(gn % nb_count);
    const int64_t grp = gn / nb_count;
    const int col = kb * 128 + (threadIdx.x & 15) * 8, row0 = nb * 128 + (threadIdx.x >> 4);
    const int64_t base = (grp * a.n + row0) * a.k + col;
    const bool col_ok = col < a.k;                    // k % 8 == 0: all eight columns or none
    constexpr int kVecs = kF32 ? 2 : 1;
    int4 raw[8][kVecs];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int v = 0; v < kVecs; ++v) {
            const int64_t at = (base + static_cast<int64_t>(i) * 16 * a.k) * (kF32 ? 4 : 2) + v * 16;
            raw[i][v] = col_ok && row0 + i * 16 < a.n ? ptx::ld_nc_v4(reinterpret_cast<const uint8_t*>(a.w) + at) : make_int4(0, 0, 0, 0);
        }
    auto values = [&](int i, float (&f)[8]) {
        if constexpr (kF32) {
            const float* p = reinterpret_cast<const float*>(raw[i]);
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = p[j];
        } else {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[i][0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 v = __bfloat1622float2(h[j]);
                f[2 * j] = v.x;
                f[2 * j + 1] = v.y;
            }
        }
    };
    float amax;
    if constexpr (kF32) {
        amax = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float f[8];
            values(i, f);
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = max_keep_nan(amax, fabsf(f[j]));
        }
    } else {
        // the largest of bf16 magnitudes is one of them: two per instruction, no rounding
        __nv_bfloat162 m = __float2bfloat162_rn(0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[i][0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) m = __hmax2_nan(m, __habs2(h[j]));
        }
        amax = max_keep_nan(__low2float(m), __high2float(m));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = max_keep_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) s_amax[threadIdx.x >> 5] = amax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWqThreads / 32; ++w) amax = max_keep_nan(amax, s_amax[w]);
    amax = amax < 1e-4f ? 1e-4f : amax;               // a NaN stays
    if (threadIdx.x == 0) a.sf[blk] = __fmul_rn(amax, 1.f / 448.f);
    const float scale = __fmul_rn(448.f, __frcp_rn(amax));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (!col_ok || row0 + i * 16 >= a.n) continue;
        float f[8];
        values(i, f);
        uint32_t packed[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j] * scale, f[4 * j + 1] * scale), __NV_SATFINITE, __NV_E4M3);
            const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j + 2] * scale, f[4 * j + 3] * scale), __NV_SATFINITE, __NV_E4M3);
            packed[j] = lo | (hi << 16);
        }
        *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(a.q) + base + static_cast<int64_t>(i) * 16 * a.k) = make_uint2(packed[0], packed[1]);
    }
}

// ---------------------------------------------------------------------------------------------- backward pass
// 64 x 64 tiles, 256 threads: thread (pair = tid / 8, c8 = tid % 8) owns rows 2 * pair, 2 * pair + 1 and the eight
// columns c8 * 8 ...  Results are written row-major straight from registers and, through a transposed
// shared-memory tile, column-major in 128-byte runs.
constexpr int kTile = 64, kTileThreads = 256;
constexpr int kTStride = 66;   // bf16 elements per transposed tile row (132 bytes: 4-byte aligned, 2-way bank conflicts at most)

struct TileT {
    __nv_bfloat16 v[kTile][kTStride];
};

// stash the two rows' values of column `col` (rows 2 * pair and 2 * pair + 1 of the tile) as one 4-byte word
__device__ __forceinline__ void stash_pair(TileT& t, int col, int pair, float lo, float hi) {
    *reinterpret_cast<__nv_bfloat162*>(&t.v[col][2 * pair]) = __floats2bfloat162_rn(lo, hi);
}
// write the tile transposed: out_t[(col0 + c) * ld + row0 + 0..63], one 128-byte run per warp instruction
__device__ __forceinline__ void flush_transposed(const TileT& t, void* out_t, int64_t ld, int col0, int row0) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < kTile / (kTileThreads / 32); ++i) {
        const int c = warp * (kTile / (kTileThreads / 32)) + i;
        const uint32_t word = *reinterpret_cast<const uint32_t*>(&t.v[c][2 * lane]);
        *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(out_t) + ((col0 + c) * ld + row0 + 2 * lane) * 2) = word;
    }
}
__device__ __forceinline__ void unpack8(const int4& raw, float (&f)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 v = __bfloat1622float2(h[j]);
        f[2 * j] = v.x;
        f[2 * j + 1] = v.y;
    }
}
__device__ __forceinline__ int4 pack8(const float (&f)[8]) {
    int4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
    return raw;
}
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// grid (rows / 64, ceil(H / kPrepCols)): one CTA = 64 rows x kPrepCols columns; the per-row dot product of its columns goes
// to row_dot[blockIdx.y * rows + row] and the caller adds the column blocks up (fixed order, so the result is deterministic)
constexpr int kPrepCols = 512;

__global__ void __launch_bounds__(kTileThreads) moe_bwd_prep_kernel(const MoeBwdArgs a) {
    __shared__ TileT tile;
    const int pair = threadIdx.x >> 3, c8 = threadIdx.x & 7;
    const int row0 = blockIdx.x * kTile;
    const int H = a.cols;
    const int col_begin = blockIdx.y * kPrepCols, col_end = min(H, col_begin + kPrepCols);
    const uint8_t* gb = reinterpret_cast<const uint8_t*>(a.g);
    const uint8_t* yb = reinterpret_cast<const uint8_t*>(a.y);
    uint8_t* ob = reinterpret_cast<uint8_t*>(a.out);
    float dot[2] = {0.f, 0.f}, w[2];
    bool ok[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = row0 + 2 * pair + r;
        ok[r] = a.valid[row] != 0;
        w[r] = ok[r] ? a.w[row] : 0.f;
    }
    for (int col0 = col_begin; col0 < col_end; col0 += kTile) {
        float res[2][8];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t off = (static_cast<int64_t>(row0 + 2 * pair + r) * H + col0 + c8 * 8) * 2;
            float g[8], y[8];
            if (ok[r]) {
                unpack8(ptx::ld_nc_v4(gb + off), g);
                if (yb != nullptr) unpack8(ptx::ld_nc_v4(yb + off), y);
                else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) y[j] = 0.f;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) g[j] = y[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                dot[r] = fmaf(g[j], y[j], dot[r]);
                res[r][j] = round_bf16(g[j] * w[r]);
            }
            if (ob != nullptr) *reinterpret_cast<int4*>(ob + off) = pack8(res[r]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) stash_pair(tile, c8 * 8 + j, pair, res[0][j], res[1][j]);
        __syncthreads();
        flush_transposed(tile, a.out_t, a.rows, col0, row0);
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        float d = dot[r];
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        d += __shfl_xor_sync(0xffffffffu, d, 4);
        if (c8 == 0 && a.row_dot != nullptr) a.row_dot[static_cast<int64_t>(blockIdx.y) * a.rows + row0 + 2 * pair + r] = d;
    }
}

// grid (rows / 64, I / 64)
__global__ void __launch_bounds__(kTileThreads) moe_bwd_swiglu_kernel(const MoeBwdArgs a) {
    __shared__ TileT t_gate, t_up, t_act;
    const int pair = threadIdx.x >> 3, c8 = threadIdx.x & 7;
    const int row0 = blockIdx.x * kTile, col0 = blockIdx.y * kTile;
    const int I = a.cols;
    const uint8_t* db = reinterpret_cast<const uint8_t*>(a.g);
    const uint8_t* hb = reinterpret_cast<const uint8_t*>(a.y);
    uint8_t* ob = reinterpret_cast<uint8_t*>(a.out);
    float dg[2][8], du[2][8], act[2][8], dot[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = row0 + 2 * pair + r;
        const int col = col0 + c8 * 8;
        if (a.valid[row] != 0) {
            float d[8], gate[8], up[8];
            unpack8(ptx::ld_nc_v4(db + (static_cast<int64_t>(row) * I + col) * 2), d);
            const float wr = a.w != nullptr ? a.w[row] : 1.f;
            unpack8(ptx::ld_nc_v4(hb + (static_cast<int64_t>(row) * 2 * I + col) * 2), gate);
            unpack8(ptx::ld_nc_v4(hb + (static_cast<int64_t>(row) * 2 * I + I + col) * 2), up);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float sig = 1.f / (1.f + __expf(-gate[j]));
                act[r][j] = round_bf16(gate[j] * sig * up[j]);
                // d[j] is the gradient w.r.t. the UNWEIGHTED activation when a row weight is given: its product with the
                // activation is d loss / d weight, and the weight enters the gradients that flow on
                dot[r] = fmaf(d[j], act[r][j], dot[r]);
                const float dj = d[j] * wr;
                du[r][j] = round_bf16(dj * gate[j] * sig);
                dg[r][j] = round_bf16(dj * up[j] * sig * (1.f + gate[j] * (1.f - sig)));
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) act[r][j] = du[r][j] = dg[r][j] = 0.f;
        }
        *reinterpret_cast<int4*>(ob + (static_cast<int64_t>(row) * 2 * I + col) * 2) = pack8(dg[r]);
        *reinterpret_cast<int4*>(ob + (static_cast<int64_t>(row) * 2 * I + I + col) * 2) = pack8(du[r]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        stash_pair(t_gate, c8 * 8 + j, pair, dg[0][j], dg[1][j]);
        stash_pair(t_up, c8 * 8 + j, pair, du[0][j], du[1][j]);
        stash_pair(t_act, c8 * 8 + j, pair, act[0][j], act[1][j]);
    }
    __syncthreads();
    flush_transposed(t_gate, a.out_t, a.rows, col0, row0);
    flush_transposed(t_up, a.out_t, a.rows, I + col0, row0);
    flush_transposed(t_act, a.out2_t, a.rows, col0, row0);
    if (a.row_dot != nullptr) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float d = dot[r];
            d += __shfl_xor_sync(0xffffffffu, d, 1);
            d += __shfl_xor_sync(0xffffffffu, d, 2);
            d += __shfl_xor_sync(0xffffffffu, d, 4);
            if (c8 == 0) a.row_dot[static_cast<int64_t>(blockIdx.y) * a.rows + row0 + 2 * pair + r] = d;
        }
    }
}

// grid (rows / 64, H / 64)
__global__ void __launch_bounds__(kTileThreads) moe_bwd_dequant_t_kernel(const MoeBwdArgs a) {
    __shared__ TileT tile;
    const int pair = threadIdx.x >> 3, c8 = threadIdx.x & 7;
    const int row0 = blockIdx.x * kTile, col0 = blockIdx.y * kTile;
    const int H = a.cols;
    const uint8_t* qb = reinterpret_cast<const uint8_t*>(a.y);
    float x[2][8];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = row0 + 2 * pair + r;
        const int col = col0 + c8 * 8;
        if (a.valid[row] != 0) {
            const uint2 raw = *reinterpret_cast<const uint2*>(qb + static_cast<int64_t>(row) * H + col);
            const float sf = __ldg(a.w + row * a.sf_stride_row + (col / 128) * a.sf_stride_col);
            const __nv_fp8x2_storage_t* p = reinterpret_cast<const __nv_fp8x2_storage_t*>(&raw);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(p[j], __NV_E4M3);
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
                x[r][2 * j] = f.x * sf;
                x[r][2 * j + 1] = f.y * sf;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) x[r][j] = 0.f;
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) stash_pair(tile, c8 * 8 + j, pair, x[0][j], x[1][j]);
    __syncthreads();
    flush_transposed(tile, a.out_t, a.rows, col0, row0);
}

// Row-major results only, for weight-gradient GEMMs that read MN-major operands (`gemm_kgrouped_tn`): one warp per row, no shared
// memory, every byte read and written once, so the kernels are bound by HBM (0.15 ms each for 34816 rows of 7168 / 2 x 2048).
constexpr int kRowWarps = 8;

// e4m3 of eight channels of a lane whose 16 neighbours hold the rest of a 128-channel group: the arithmetic of the stand-alone cast
__device__ __forceinline__ uint2 cast_group(const float (&v)[8], float& amax) {
    amax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
    amax = fmaxf(ptx::warp_max_16(amax), 1e-4f);
    const float scale = __fmul_rn(448.f, __frcp_rn(amax));
    uint32_t packed[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j] * scale, v[4 * j + 1] * scale), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j + 2] * scale, v[4 * j + 3] * scale), __NV_SATFINITE, __NV_E4M3);
        packed[j] = lo | (hi << 16);
    }
    return make_uint2(packed[0], packed[1]);
}

// kQuant: d_h also leaves as e4m3 with 1 x 128 scales, for the data gradient on the e4m3 tensor cores (cols % 128 == 0).  A cast of its own
// reads d_h once more: 14336 rows x 2 x 1024 33 + 17 us apart, 41 together (196 MB, 4.8 TB/s), 34816 x 2 x 2048 144 + 83 / 177.
template <bool kQuant>
__global__ void __launch_bounds__(kRowWarps * 32) moe_bwd_swiglu_rows_kernel(const MoeBwdArgs a) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    if (row >= a.rows) return;
    const int I = a.cols;
    const uint8_t* db = reinterpret_cast<const uint8_t*>(a.g) + static_cast<int64_t>(row) * I * 2;
    const uint8_t* hb = reinterpret_cast<const uint8_t*>(a.y) + static_cast<int64_t>(row) * I * 4;
    uint8_t* ob = reinterpret_cast<uint8_t*>(a.out) + static_cast<int64_t>(row) * I * 4;
    uint8_t* ab = reinterpret_cast<uint8_t*>(a.out2) + static_cast<int64_t>(row) * I * 2;
    uint8_t* qb = kQuant ? reinterpret_cast<uint8_t*>(a.q) + static_cast<int64_t>(row) * 2 * I : nullptr;
    float* sf = kQuant ? a.q_sf + static_cast<int64_t>(row) * (2 * I / 128) : nullptr;
    if (a.valid[row] == 0) {
        const int4 zero = make_int4(0, 0, 0, 0);
        if constexpr (kQuant) {
            for (int col = lane * 16; col < 2 * I; col += 512) *reinterpret_cast<int4*>(qb + col) = zero;
            for (int grp = lane; grp < 2 * I / 128; grp += 32) sf[grp] = __fdiv_rn(1e-4f, 448.f);
        }
        for (int col = lane * 8; col < I; col += 256) {
            *reinterpret_cast<int4*>(ob + col * 2) = zero;
            *reinterpret_cast<int4*>(ob + (I + col) * 2) = zero;
            *reinterpret_cast<int4*>(ab + col * 2) = zero;
        }
        if (lane == 0) a.row_dot[row] = 0.f;
        return;
    }
    const float wr = __ldg(a.w + row);
    float dot = 0.f, kept_g = 0.f, kept_u = 0.f;
#pragma unroll 2
    for (int col0 = 0; col0 < I; col0 += 256) {
        const int col = col0 + lane * 8;
        if (!kQuant && col >= I) break;
        const bool in_range = !kQuant || col < I;        // the cast needs whole warps for its shuffles
        float d[8], gate[8], up[8], dg[8], du[8], act[8];
        const int4 none = make_int4(0, 0, 0, 0);
        unpack8(in_range ? ptx::ld_nc_v4(db + col * 2) : none, d);
        unpack8(in_range ? ptx::ld_nc_v4(hb + col * 2) : none, gate);
        unpack8(in_range ? ptx::ld_nc_v4(hb + (I + col) * 2) : none, up);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float sig = 1.f / (1.f + __expf(-gate[j]));
            act[j] = round_bf16(gate[j] * sig * up[j]);
            dot = fmaf(d[j], act[j], dot);              // d loss / d weight of the row
            const float dj = d[j] * wr;
            du[j] = dj * gate[j] * sig;
            dg[j] = dj * up[j] * sig * (1.f + gate[j] * (1.f - sig));
        }
        const int4 dg_raw = pack8(dg), du_raw = pack8(du);
        if (in_range) {
            *reinterpret_cast<int4*>(ob + col * 2) = dg_raw;
            *reinterpret_cast<int4*>(ob + (I + col) * 2) = du_raw;
            *reinterpret_cast<int4*>(ab + col * 2) = pack8(act);
        }
        if constexpr (kQuant) {
            // the cast sees the values that were rounded to bf16
            unpack8(dg_raw, dg);
            unpack8(du_raw, du);
            float amax_g, amax_u;
            const uint2 qg = cast_group(dg, amax_g), qu = cast_group(du, amax_u);
            if (in_range) {
                *reinterpret_cast<uint2*>(qb + col) = qg;
                *reinterpret_cast<uint2*>(qb + I + col) = qu;
            }
            // the divisions of 16 steps together, one group of each half per lane
            const int step = col0 / 256;
            if ((lane & 15) == (step & 15)) {
                kept_g = amax_g;
                kept_u = amax_u;
            }
            if ((step & 15) == 15 || col0 + 256 >= I) {
                const int grp = ((step & ~15) + (lane & 15)) * 2 + (lane >> 4);
                if ((lane & 15) <= (step & 15) && grp < I / 128) {
                    sf[grp] = __fdiv_rn(kept_g, 448.f);
                    sf[I / 128 + grp] = __fdiv_rn(kept_u, 448.f);
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) a.row_dot[row] = dot;
}

// 16 channels per lane: one 16-byte load, two 16-byte stores (cols % 16 == 0)
__global__ void __launch_bounds__(kRowWarps * 32) moe_bwd_dequant_rows_kernel(const MoeBwdArgs a) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    if (row >= a.rows) return;
    const int H = a.cols;
    const uint8_t* qb = reinterpret_cast<const uint8_t*>(a.y) + static_cast<int64_t>(row) * H;
    uint8_t* ob = reinterpret_cast<uint8_t*>(a.out) + static_cast<int64_t>(row) * H * 2;
    const bool ok = a.valid[row] != 0;
    const float rw = a.row_w != nullptr ? __ldg(a.row_w + row) : 1.f;
#pragma unroll 4
    for (int col = lane * 16; col < H; col += 512) {
        int4 out[2] = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
        if (ok) {
            const int4 raw = ptx::ld_nc_v4(qb + col);
            const float sf = __ldg(a.w + row * a.sf_stride_row + (col / 128) * a.sf_stride_col) * rw;
            const __nv_fp8x2_storage_t* p = reinterpret_cast<const __nv_fp8x2_storage_t*>(&raw);
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                float f[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(p[v * 4 + j], __NV_E4M3);
                    const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&hr));
                    f[2 * j] = x.x * sf;
                    f[2 * j + 1] = x.y * sf;
                }
                out[v] = pack8(f);
            }
        }
        *reinterpret_cast<int4*>(ob + col * 2) = out[0];
        *reinterpret_cast<int4*>(ob + col * 2 + 16) = out[1];
    }
}

// rows times their weights
__global__ void __launch_bounds__(kRowWarps * 32) moe_bwd_weight_rows_kernel(const MoeBwdArgs a) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
    if (row >= a.rows) return;
    const uint8_t* gb = reinterpret_cast<const uint8_t*>(a.g) + static_cast<int64_t>(row) * a.cols * 2;
    uint8_t* ob = reinterpret_cast<uint8_t*>(a.out) + static_cast<int64_t>(row) * a.cols * 2;
    const bool ok = a.valid[row] != 0;
    const float rw = __ldg(a.row_w + row);
#pragma unroll 4
    for (int col = lane * 8; col < a.cols; col += 256) {
        int4 out = make_int4(0, 0, 0, 0);
        if (ok) {
            float f[8];
            unpack8(ptx::ld_nc_v4(gb + col * 2), f);
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] *= rw;
            out = pack8(f);
        }
        *reinterpret_cast<int4*>(ob + col * 2) = out;
    }
}

// Expand-layout bookkeeping of a grouped GEMM in one launch: from the inclusive segment ends (segment e starts at
// align(end[e - 1], alignment) and holds end[e] - start rows) -> the weights group of every 128-row tile (-1: no token
// in the tile), one validity byte per row (0: alignment padding) and the aligned segment boundaries [G + 1].
constexpr int kSegThreads = 256;
// s_seg: aligned ends of all segments; `ends`: their unaligned ends (shared or global memory); threads / CTAs of the grid share the rows
__device__ __forceinline__ void write_segments(const ExpertSegmentsArgs& a, const int* s_seg, const int* ends) {
    if (blockIdx.x == 0 && a.seg_off != nullptr) {
        for (int e = threadIdx.x; e <= a.num_groups; e += kSegThreads) a.seg_off[e] = e == 0 ? 0 : s_seg[e - 1];
    }
    const int padded_rows = (a.num_rows + 127) / 128 * 128;
    for (int row = blockIdx.x * kSegThreads + threadIdx.x; row < padded_rows; row += gridDim.x * kSegThreads) {
        // first segment whose aligned end lies beyond the row
        int lo = 0, hi = a.num_groups;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s_seg[mid] > row) hi = mid;
            else lo = mid + 1;
        }
        const int end = lo < a.num_groups ? ends[lo] : 0;
        const bool in_segment = row < end;
        if (row < a.num_rows && a.valid_row != nullptr) a.valid_row[row] = in_segment ? 1 : 0;
        if ((row & 127) == 0 && a.tile_group != nullptr) a.tile_group[row >> 7] = in_segment ? lo : -1;
        if ((row & 127) == 0 && a.tile_rows != nullptr) a.tile_rows[row >> 7] = in_segment ? min(128, end - row) : 0;
    }
}
__global__ void __launch_bounds__(kSegThreads) expert_segments_kernel(const ExpertSegmentsArgs a) {
    extern __shared__ int s_seg[];                    // aligned ends [G]
    for (int e = threadIdx.x; e < a.num_groups; e += kSegThreads)
        s_seg[e] = (__ldg(a.psum_ends + e) + a.alignment - 1) / a.alignment * a.alignment;
    __syncthreads();
    write_segments(a, s_seg, a.psum_ends);
}

// ------------------------------------------------------------------------------------------------ local expansion
// PLAN, two launches that each read the ids once.  The (row, k) pairs are cut into one contiguous share per warp
// (kPlanWarps warps per CTA).  COUNT: every warp counts its pairs per expert.  ASSIGN: a warp's first number for expert e
// is the segment start plus the counts of all warps before it, and inside its share the warp numbers the pairs in
// order (match_any groups the lanes of a step by expert), so the rows of an expert segment are ordered by received
// row: the same result on every run.  Both are bound by latency, so a CTA takes 1024 pairs (one batch of four per lane) and the
// sums over lower CTAs are shared out over its warps: 32768 pairs take 4 + 4 us (4096 pairs per CTA and serial sums: 10 + 14 us).
constexpr int kPlanWarps = 8;
__device__ __forceinline__ int plan_id(const LocalExpandPlanArgs& a, int i, int total) {   // rows * K < 2^31
    if (i >= total) return -1;
    const int row = i / a.num_topk;
    const int64_t at = static_cast<int64_t>(row) * a.idx_pitch + (i - row * a.num_topk);
    const long long id = a.idx_is_64 ? __ldg(reinterpret_cast<const long long*>(a.recv_idx) + at)
                                     : static_cast<long long>(__ldg(reinterpret_cast<const int*>(a.recv_idx) + at));
    return id >= 0 && id < a.num_local_experts ? static_cast<int>(id) : -1;
}
// share of warp `w` of the grid: multiples of 32 pairs
__device__ __forceinline__ void plan_share(const LocalExpandPlanArgs& a, int w, int num_warps, int& lo, int& hi) {
    const int total = a.num_rows * a.num_topk;
    const int share = ((total + num_warps * 32 - 1) / (num_warps * 32)) * 32;
    lo = min(w * share, total);
    hi = min(lo + share, total);
}
constexpr int kPlanBatch = 4, kPlanPairsPerCta = kPlanWarps * 32 * kPlanBatch;
// this warp's counts per expert of the pairs [lo, hi), added to `mine`
__device__ __forceinline__ void plan_count(const LocalExpandPlanArgs& a, int lo, int hi, int* mine) {
    const int lane = threadIdx.x & 31;
    for (int first = lo; first < hi; first += 32 * kPlanBatch) {
        int id[kPlanBatch];
#pragma unroll
        for (int j = 0; j < kPlanBatch; ++j) id[j] = plan_id(a, first + j * 32 + lane, hi);
#pragma unroll
        for (int j = 0; j < kPlanBatch; ++j)
            if (id[j] >= 0) atomicAdd(mine + id[j], 1);
    }
}
// numbers the pairs [lo, hi) from next[expert] on
__device__ __forceinline__ void plan_assign(const LocalExpandPlanArgs& a, int lo, int hi, int* next) {
    const int lane = threadIdx.x & 31;
    for (int first = lo; first < hi; first += 32 * kPlanBatch) {
        int id[kPlanBatch];
#pragma unroll
        for (int j = 0; j < kPlanBatch; ++j) id[j] = plan_id(a, first + j * 32 + lane, hi);
#pragma unroll
        for (int j = 0; j < kPlanBatch; ++j) {
            // lanes with the same expert: the lowest takes the numbers for all of them
            const uint32_t peers = __match_any_sync(0xffffffffu, id[j]);
            if (id[j] >= 0) {
                const int leader = __ffs(peers) - 1;
                int base = 0;
                if (lane == leader) {
                    base = next[id[j]];
                    next[id[j]] = base + __popc(peers);
                }
                base = __shfl_sync(peers, base, leader);
                a.pos[first + j * 32 + lane] = base + __popc(peers & ptx::lanemask_lt());
            } else if (first + j * 32 + lane < hi) {
                a.pos[first + j * 32 + lane] = -1;
            }
            __syncwarp();
        }
    }
}
__global__ void __launch_bounds__(kPlanWarps * 32) local_expand_count_kernel(const LocalExpandPlanArgs a) {
    extern __shared__ int s_plan[];                    // [kPlanWarps][El]
    const int El = a.num_local_experts, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* mine = s_plan + warp * El;
    for (int e = lane; e < El; e += 32) mine[e] = 0;
    __syncwarp();
    int lo, hi;
    plan_share(a, blockIdx.x * kPlanWarps + warp, gridDim.x * kPlanWarps, lo, hi);
    plan_count(a, lo, hi, mine);
    __syncthreads();
    // per-warp counts and, for the prefix over CTAs, their sum
    int* out = a.warp_counts + static_cast<int64_t>(blockIdx.x * kPlanWarps + warp) * El;
    for (int e = lane; e < El; e += 32) out[e] = mine[e];
    for (int e = threadIdx.x; e < El; e += kPlanWarps * 32) {
        int sum = 0;
        for (int w = 0; w < kPlanWarps; ++w) sum += s_plan[w * El + e];
        a.cta_counts[static_cast<int64_t>(blockIdx.x) * El + e] = sum;
    }
}
__global__ void __launch_bounds__(kPlanWarps * 32) local_expand_assign_kernel(const LocalExpandPlanArgs a) {
    extern __shared__ int s_plan[];                    // [kPlanWarps][El] next number of every expert for each warp, [kPlanWarps][El] partial sums
    const int El = a.num_local_experts, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int me = blockIdx.x * kPlanWarps + warp, num_warps = gridDim.x * kPlanWarps;
    int* next = s_plan + warp * El;
    int* part = s_plan + kPlanWarps * El;
    // counts of the CTAs below this one, shared out over the warps (CTA 0 has none below it: it sums all CTAs for seg_end)
    const int ctas = blockIdx.x == 0 ? gridDim.x : blockIdx.x;
    for (int e = lane; e < El; e += 32) {
        int sum = 0;
#pragma unroll 4
        for (int b = warp; b < ctas; b += kPlanWarps) sum += __ldg(a.cta_counts + static_cast<int64_t>(b) * El + e);
        part[warp * El + e] = sum;
    }
    __syncthreads();
    for (int e = lane; e < El; e += 32) {
        const int start = e == 0 ? 0 : __ldg(a.seg_end_aligned + e - 1);
        int below = 0, own = 0;
#pragma unroll
        for (int w = 0; w < kPlanWarps; ++w) {
            below += part[w * El + e];
            if (w < warp) own += __ldg(a.warp_counts + static_cast<int64_t>(blockIdx.x * kPlanWarps + w) * El + e);
        }
        if (me == 0) a.seg_end[e] = start + below;
        next[e] = start + (blockIdx.x == 0 ? 0 : below) + own;
    }
    __syncwarp();
    int lo, hi;
    plan_share(a, me, num_warps, lo, hi);
    plan_assign(a, lo, hi, next);
}
// Few pairs (one CTA's worth): plan and segments in ONE launch.  A layer on a short prompt waits for the launches of these small
// kernels rather than for the kernels (64 tokens: three launches less to queue between the dispatch and the first GEMM).
__global__ void __launch_bounds__(kPlanWarps * 32) local_expand_layout_kernel(const LocalExpandPlanArgs a, const ExpertSegmentsArgs seg) {
    extern __shared__ int s_plan[];                    // [kPlanWarps][El] counts, then next numbers; [El] segment ends; [El] aligned ends
    static_assert(kPlanWarps * 32 == kSegThreads, "write_segments counts on the block size");
    const int El = a.num_local_experts, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* mine = s_plan + warp * El;
    int* s_end = s_plan + kPlanWarps * El;
    int* s_seg = s_end + El;
    for (int e = lane; e < El; e += 32) mine[e] = 0;
    __syncwarp();
    int lo, hi;
    plan_share(a, warp, kPlanWarps, lo, hi);
    plan_count(a, lo, hi, mine);
    __syncthreads();
    for (int e = threadIdx.x; e < El; e += kPlanWarps * 32) {
        int next = e == 0 ? 0 : __ldg(a.seg_end_aligned + e - 1);
        for (int w = 0; w < kPlanWarps; ++w) {
            const int n = s_plan[w * El + e];
            s_plan[w * El + e] = next;
            next += n;
        }
        a.seg_end[e] = s_end[e] = next;
        s_seg[e] = (next + seg.alignment - 1) / seg.alignment * seg.alignment;
    }
    __syncthreads();
    plan_assign(a, lo, hi, mine);
    write_segments(seg, s_seg, s_end);
}

// COPY: one warp per received row (or part of it); every 512-byte piece is read once and written to each expert row of the row.
// This kernel, the reduction and the forward activation stand between products, so all start early (see few_waves); they let the next
// one start when their own last CTAs have started.
constexpr int kExpandWarps = 8, kMaxExpandTopk = 32;
__global__ void __launch_bounds__(kExpandWarps * 32) local_expand_copy_kernel(const LocalExpandCopyArgs a) {
    ptx::wait_for_previous_kernel();
    ptx::let_next_kernel_start();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kExpandWarps + (threadIdx.x >> 5);
    if (a.out_valid != nullptr) {
        // weights of alignment rows; those of token rows are written below
        const int threads = gridDim.x * gridDim.y * kExpandWarps * 32;
        for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * kExpandWarps * 32 + threadIdx.x; i < a.num_out; i += threads)
            if (a.out_valid[i] == 0) a.w_dst[i] = 0.f;
    }
    if (row >= a.num_rows) return;
    const int my_pos = lane < a.num_topk ? *(a.pos + static_cast<int64_t>(row) * a.num_topk + lane) : -1;
    uint32_t dests = __ballot_sync(0xffffffffu, my_pos >= 0);
    if (dests == 0) return;
    if (a.w_src != nullptr && my_pos >= 0 && blockIdx.y == 0) a.w_dst[my_pos] = *(a.w_src + static_cast<int64_t>(row) * a.w_pitch + lane);
    const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src) + static_cast<int64_t>(row) * a.src_pitch;
    uint8_t* dst = reinterpret_cast<uint8_t*>(a.dst);
    const int pieces = a.row_bytes / 16;
    for (int p0 = blockIdx.y * 128; p0 < pieces; p0 += 128 * gridDim.y) {
        int4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = p0 + j * 32 + lane;
            v[j] = p < pieces ? ptx::ld_na_v4(src + p * 16) : make_int4(0, 0, 0, 0);
        }
        for (uint32_t m = dests; m != 0; m &= m - 1) {
            const int64_t to = __shfl_sync(0xffffffffu, my_pos, __ffs(m) - 1);
            uint8_t* out = dst + to * a.row_bytes;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int p = p0 + j * 32 + lane;
                if (p < pieces) *reinterpret_cast<int4*>(out + p * 16) = v[j];
            }
        }
    }
    if (a.sf_src != nullptr && blockIdx.y == 0) {
        // every lane takes part in the shuffles, also where the last columns leave some without work
        for (int c0 = 0; c0 < a.sf_cols; c0 += 32) {
            const int c = c0 + lane;
            const float f = c < a.sf_cols ? *(a.sf_src + static_cast<int64_t>(row) * a.sf_stride_row + c * a.sf_stride_col) : 0.f;
            for (uint32_t m = dests; m != 0; m &= m - 1) {
                const int64_t to = __shfl_sync(0xffffffffu, my_pos, __ffs(m) - 1);
                if (c < a.sf_cols) a.sf_dst[to * a.sf_cols + c] = f;
            }
        }
    }
}

// REDUCE: one warp per received row (or part of it); fp32 sum of its expert rows (in top-k order), optionally weighted, rounded once to bf16.
// kAhead: source rows whose loads are in flight together (their products are always added in top-k order).  Two, with the rows split
// by columns, when there are so few rows that latency counts (8 x 7168 channels each: 64 rows 62 -> 12 us, 512 rows 65 -> 20 us);
// one, with whole rows, otherwise: it leaves registers for more warps (4096 rows, 530 MB: 96 us against 109 us).
template <int kAhead>
__global__ void __launch_bounds__(kExpandWarps * 32) local_reduce_kernel(const LocalReduceArgs a) {
    ptx::wait_for_previous_kernel();
    ptx::let_next_kernel_start();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kExpandWarps + (threadIdx.x >> 5);
    if (row >= a.num_rows) return;
    const int my_pos = lane < a.num_topk ? *(a.pos + static_cast<int64_t>(row) * a.num_topk + lane) : -1;
    const float my_w = (a.w != nullptr && my_pos >= 0) ? *(a.w + my_pos) : 1.f;
    const uint32_t srcs = __ballot_sync(0xffffffffu, my_pos >= 0);
    const uint8_t* src = reinterpret_cast<const uint8_t*>(a.src);
    uint8_t* out = reinterpret_cast<uint8_t*>(a.dst) + static_cast<int64_t>(row) * a.cols * 2;
    const int pieces = a.cols / 8;            // 16-byte pieces of 8 bf16
    constexpr int kPer = 4;                   // pieces per lane and step: the loads of a step are issued together
    const int part = kAhead == 2 ? blockIdx.y : 0, parts = kAhead == 2 ? gridDim.y : 1;     // columns of a split row
    for (int p0 = part * 32 * kPer; p0 < pieces; p0 += 32 * kPer * parts) {
        float acc[kPer][8];
#pragma unroll
        for (int j = 0; j < kPer; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[j][i] = 0.f;
        auto load = [&](int4 (&v)[kPer], int64_t from) {
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int p = p0 + j * 32 + lane;
                v[j] = p < pieces ? ptx::ld_na_v4(src + from * a.cols * 2 + p * 16) : make_int4(0, 0, 0, 0);
            }
        };
        auto add = [&](const int4 (&v)[kPer], float w) {
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __bfloat1622float2(h[i]);
                    acc[j][2 * i] = fmaf(w, f.x, acc[j][2 * i]);
                    acc[j][2 * i + 1] = fmaf(w, f.y, acc[j][2 * i + 1]);
                }
            }
        };
        if constexpr (kAhead == 1) {
            for (uint32_t m = srcs; m != 0; m &= m - 1) {
                const int k = __ffs(m) - 1;
                int4 v[kPer];
                load(v, __shfl_sync(0xffffffffu, my_pos, k));
                add(v, __shfl_sync(0xffffffffu, my_w, k));
            }
        } else {
            for (uint32_t m = srcs; m != 0; m &= m - 1) {
                const int k0 = __ffs(m) - 1;
                int4 v0[kPer], v1[kPer];
                load(v0, __shfl_sync(0xffffffffu, my_pos, k0));
                m &= m - 1;
                const int k1 = __ffs(m) - 1;              // -1: no second row
                if (k1 >= 0) load(v1, __shfl_sync(0xffffffffu, my_pos, k1));
                add(v0, __shfl_sync(0xffffffffu, my_w, k0));
                if (k1 < 0) break;
                add(v1, __shfl_sync(0xffffffffu, my_w, k1));
            }
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int p = p0 + j * 32 + lane;
            if (p < pieces) {
                int4 o;
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(acc[j][2 * i], acc[j][2 * i + 1]);
                *reinterpret_cast<int4*>(out + p * 16) = o;
            }
        }
    }
}

// One value per (row, k) pair from its expert row.  Bound by its launch: in PyTorch operations it was six of them.
__global__ void __launch_bounds__(256) local_gather_kernel(const int32_t* pos, const float* v, float* out, int total) {
    for (int i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
        const int at = __ldg(pos + i);
        out[i] = at >= 0 ? __ldg(v + at) : 0.f;
    }
}
}  // namespace

cudaError_t launch_local_gather(const int32_t* pos, const float* v, float* out, int64_t total, cudaStream_t stream) {
    if (total == 0) return cudaSuccess;
    if (total < 0 || total > 0x7fffffff - 256 * 1024) return cudaErrorInvalidValue;
    local_gather_kernel<<<static_cast<int>(std::min<int64_t>(1024, (total + 255) / 256)), 256, 0, stream>>>(pos, v, out, static_cast<int>(total));
    return cudaGetLastError();
}

int moe_bwd_prep_col_blocks(int cols) { return (cols + kPrepCols - 1) / kPrepCols; }

cudaError_t launch_moe_bwd(const MoeBwdArgs& a, cudaStream_t stream) {
    if (a.rows == 0) return cudaSuccess;
    if (!aligned(a.g, 16) || !aligned(a.y, a.op == EP_MOE_BWD_DEQUANT_T ? 8 : 16) || !aligned(a.out, 16) || !aligned(a.out2, 16)) return cudaErrorInvalidValue;
    if (a.op == EP_MOE_BWD_SWIGLU_ROWS || a.op == EP_MOE_BWD_DEQUANT_ROWS || a.op == EP_MOE_BWD_WEIGHT_ROWS) {
        const int blocks = (a.rows + kRowWarps - 1) / kRowWarps;
        if (a.cols % (a.op == EP_MOE_BWD_DEQUANT_ROWS ? 16 : 8) != 0) return cudaErrorInvalidValue;
        if (a.op == EP_MOE_BWD_SWIGLU_ROWS && a.q != nullptr) {
            if (a.cols % 128 != 0 || !aligned(a.q, 16) || a.q_sf == nullptr) return cudaErrorInvalidValue;
            moe_bwd_swiglu_rows_kernel<true><<<blocks, kRowWarps * 32, 0, stream>>>(a);
        } else if (a.op == EP_MOE_BWD_SWIGLU_ROWS) moe_bwd_swiglu_rows_kernel<false><<<blocks, kRowWarps * 32, 0, stream>>>(a);
        else if (a.op == EP_MOE_BWD_DEQUANT_ROWS) moe_bwd_dequant_rows_kernel<<<blocks, kRowWarps * 32, 0, stream>>>(a);
        else moe_bwd_weight_rows_kernel<<<blocks, kRowWarps * 32, 0, stream>>>(a);
        return cudaGetLastError();
    }
    if (a.rows % kTile != 0 || a.cols % kTile != 0) return cudaErrorInvalidValue;
    if (a.op == EP_MOE_BWD_PREP) moe_bwd_prep_kernel<<<dim3(a.rows / kTile, (a.cols + kPrepCols - 1) / kPrepCols), kTileThreads, 0, stream>>>(a);
    else if (a.op == EP_MOE_BWD_SWIGLU) moe_bwd_swiglu_kernel<<<dim3(a.rows / kTile, a.cols / kTile), kTileThreads, 0, stream>>>(a);
    else if (a.op == EP_MOE_BWD_DEQUANT_T) moe_bwd_dequant_t_kernel<<<dim3(a.rows / kTile, a.cols / kTile), kTileThreads, 0, stream>>>(a);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_local_expand_plan(const LocalExpandPlanArgs& a, cudaStream_t stream) {
    if (a.num_local_experts < 1 || a.num_topk < 1 || a.num_topk > kMaxExpandTopk || a.num_rows < 0) return cudaErrorInvalidValue;
    if (a.num_ctas < 1 || a.num_local_experts > 1024 || a.warp_counts == nullptr || a.cta_counts == nullptr) return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(kPlanWarps) * a.num_local_experts * sizeof(int);
    if (2 * smem > 48 * 1024) {
        const cudaError_t err = cudaFuncSetAttribute(local_expand_assign_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(2 * smem));
        if (err != cudaSuccess) return err;
    }
    local_expand_count_kernel<<<a.num_ctas, kPlanWarps * 32, smem, stream>>>(a);
    local_expand_assign_kernel<<<a.num_ctas, kPlanWarps * 32, 2 * smem, stream>>>(a);
    return cudaGetLastError();
}

int local_expand_pairs_per_cta() { return kPlanPairsPerCta; }

cudaError_t launch_local_expand_layout(const LocalExpandPlanArgs& a, const ExpertSegmentsArgs& seg, cudaStream_t stream) {
    if (a.num_ctas > 1 || a.num_local_experts > 512) {
        const cudaError_t err = launch_local_expand_plan(a, stream);
        return err != cudaSuccess ? err : launch_expert_segments(seg, stream);
    }
    if (a.num_local_experts < 1 || a.num_topk < 1 || a.num_topk > kMaxExpandTopk || a.num_rows < 0) return cudaErrorInvalidValue;
    if (seg.num_groups != a.num_local_experts || seg.alignment < 128 || seg.alignment % 128 != 0 || seg.num_rows < 0) return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(kPlanWarps + 2) * a.num_local_experts * sizeof(int);       // at most 20 KB
    local_expand_layout_kernel<<<1, kPlanWarps * 32, smem, stream>>>(a, seg);
    return cudaGetLastError();
}

cudaError_t launch_local_expand_copy(const LocalExpandCopyArgs& a, cudaStream_t stream) {
    if (a.num_rows == 0) return cudaSuccess;
    if (a.num_topk < 1 || a.num_topk > kMaxExpandTopk || a.row_bytes % 16 != 0 || a.src_pitch % 16 != 0 ||
        reinterpret_cast<uintptr_t>(a.src) % 16 != 0 || reinterpret_cast<uintptr_t>(a.dst) % 16 != 0)
        return cudaErrorInvalidValue;
    const int ctas = (a.num_rows + kExpandWarps - 1) / kExpandWarps;
    void* params[] = {const_cast<LocalExpandCopyArgs*>(&a)};
    return launch_dependent((const void*)local_expand_copy_kernel, dim3(ctas, column_splits(ctas, (a.row_bytes + 2047) / 2048)),
                            dim3(kExpandWarps * 32), params, 0, stream);
}

cudaError_t launch_local_reduce(const LocalReduceArgs& a, cudaStream_t stream) {
    if (a.num_rows == 0) return cudaSuccess;
    if (a.num_topk < 1 || a.num_topk > kMaxExpandTopk || a.cols % 8 != 0 || reinterpret_cast<uintptr_t>(a.src) % 16 != 0 ||
        reinterpret_cast<uintptr_t>(a.dst) % 16 != 0)
        return cudaErrorInvalidValue;
    const int ctas = (a.num_rows + kExpandWarps - 1) / kExpandWarps;
    const dim3 grid(ctas, column_splits(ctas, (a.cols + 1023) / 1024));
    void* params[] = {const_cast<LocalReduceArgs*>(&a)};
    const void* fn = ctas < kWantedCtas ? (const void*)local_reduce_kernel<2> : (const void*)local_reduce_kernel<1>;
    return launch_dependent(fn, grid, dim3(kExpandWarps * 32), params, 0, stream);
}

cudaError_t launch_expert_segments(const ExpertSegmentsArgs& a, cudaStream_t stream) {
    if (a.num_groups < 1 || a.num_groups > 8192 || a.alignment < 128 || a.alignment % 128 != 0 || a.num_rows < 0) return cudaErrorInvalidValue;
    const int blocks = max(1, min(1024, (a.num_rows + kSegThreads - 1) / kSegThreads));
    expert_segments_kernel<<<blocks, kSegThreads, a.num_groups * sizeof(int), stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_weight_quant(const WeightQuantArgs& a, cudaStream_t stream) {
    const int64_t blocks = a.groups * ((a.n + 127) / 128) * ((a.k + 127) / 128);
    if (blocks <= 0) return cudaSuccess;
    if (blocks > 0x7fffffffll || a.k % 8 != 0 || reinterpret_cast<uintptr_t>(a.w) % 16 != 0 || reinterpret_cast<uintptr_t>(a.q) % 8 != 0)
        return cudaErrorInvalidValue;
    if (a.w_is_f32) weight_quant_kernel<true><<<static_cast<unsigned>(blocks), kWqThreads, 0, stream>>>(a);
    else weight_quant_kernel<false><<<static_cast<unsigned>(blocks), kWqThreads, 0, stream>>>(a);
    return cudaGetLastError();
}

// A warp's steps of 256 columns are a chain (load, exponential, amax, store), and with a row mask many CTAs have next to nothing to do, so
// rows are split further than in the other kernels.  Not into single steps in general: such a warp has nothing to load ahead.  us by the valid
// ones of every 128 rows (16 / 64 / 128), split for 296 CTAs and by this:
//     768 to 1152 CTAs of one step each      2048 x 1024    2.9 / 4.1 / 4.4    2.7 / 3.3 / 4.1      1024 x 2048    2.7 / 4.0 / 5.2    2.8 / 3.4 / 4.1
//     up to 1536 CTAs of two steps or more   4096 x 2048    6.8 / 10.9 / 11.5  4.6 / 6.4 / 9.6      6016 x 1024    4.4 / 6.8 / 7.9    4.0 / 5.8 / 8.0
//     chains of more than eight steps        8192 x 4096    15.8 / 23.0 / 30.9 10.8 / 18.9 / 30.6   9344 x 3072    12.8 / 17.9 / 26.8 9.2 / 16.4 / 26.9
// Beyond these lines full rows get slower: one step each on 512 CTAs 512 x 2048 2.2 / 2.9 / 2.7 becomes 2.2 / 3.0 / 3.2, on 2048 CTAs 8192 x 512 3.6 / 4.5 / 5.7
// becomes 3.7 / 5.0 / 6.8; two steps each on 2048 CTAs 8192 x 1024 5.3 / 7.0 / 9.0 becomes 4.6 / 7.0 / 9.9, on 384 CTAs 512 x 3072 2.6 / 3.7 / 3.3 becomes
// 2.3 / 3.4 / 4.3.
constexpr int kSwigluWarps = 8;
int swiglu_quant_col_chunk(int rows, int inter) {
    const int ctas = (rows + kSwigluWarps - 1) / kSwigluWarps, steps = (inter + 255) / 256;
    int splits = column_splits(ctas, steps);
    if (ctas >= 96 && ctas <= 1152 && ctas * steps >= 768 && ctas * steps <= 1152) splits = steps;
    else if (ctas >= 128) splits = max(splits, max(min((steps + 1) / 2, 1536 / ctas), (steps + 7) / 8));
    return (steps + splits - 1) / splits * 256;
}

cudaError_t launch_swiglu_quant(const SwigluQuantArgs& a, cudaStream_t stream) {
    if (a.rows == 0 || a.inter == 0) return cudaSuccess;
    if (!aligned(a.h, 16) || (a.rows > 1 && a.ldh % 8 != 0) || !aligned(a.q, 8) || !aligned(a.act_bf16, 16)) return cudaErrorInvalidValue;
    SwigluQuantArgs args = a;
    args.col_chunk = swiglu_quant_col_chunk(a.rows, a.inter);
    void* params[] = {&args};
    return launch_dependent((const void*)swiglu_quant_kernel, dim3((a.rows + kSwigluWarps - 1) / kSwigluWarps, (a.inter + args.col_chunk - 1) / args.col_chunk),
                            dim3(kSwigluWarps * 32), params, 0, stream);
}

}  // namespace ep
