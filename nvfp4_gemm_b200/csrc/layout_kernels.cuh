// Data-movement kernels beside the matmul path (HBM-bound, 16-byte vector accesses):
//   * interleave_column_blocks: [g][rows][n_local] fp16 (what an all-gather of per-rank column
//     blocks leaves in memory) -> row-major [rows][g * n_local];
//   * permute_scales: plain [rows][K/16] scale bytes -> the 512-byte atom layout the tensor-core
//     GEMM reads (ref.txt:31, s_128t.py:554-562 in the reference project); scales_from_permuted:
//     the way back, or a comparison of the two forms;
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"
#include "quantize.cuh"

namespace nvfp4 {

// One thread moves 16 bytes (8 fp16).  n_local is a multiple of 8.
__global__ void __launch_bounds__(256) interleave_column_blocks_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst,
                                                                      long long rows, int vec_per_block_row, int g,
                                                                      long long dst_row_stride_vec) {
    const long long per_row = static_cast<long long>(vec_per_block_row) * g;
    const long long total = rows * per_row;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long row = i / per_row;
        const int in_row = static_cast<int>(i - row * per_row);
        const int blk = in_row / vec_per_block_row;
        const int v = in_row - blk * vec_per_block_row;
        const uint4 val = __ldcs(src + (static_cast<long long>(blk) * rows + row) * vec_per_block_row + v);
        dst[row * dst_row_stride_vec + in_row] = val;
    }
}

// All-gather by a copy kernel: rows [row0, row0 + rows) of up to seven column blocks go from
// src[i] to dst[i] (same offsets inside row-major matrices of one row stride).  Either side may be
// peer-mapped memory of another GPU.  16 bytes per thread and access, a warp reads and writes 512
// contiguous bytes of one row.
__device__ __forceinline__ uint4 ld_nc_na_v4(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
struct BlockCopyParams {
    const uint4* src[7];   // source matrix base + the block's column offset
    uint4* dst[7];         // destination matrix base + the same offset
    int n_src;
};
__global__ void __launch_bounds__(256) copy_column_blocks_kernel(const BlockCopyParams pp, long long row0, unsigned rows, unsigned vec_per_row,
                                                                 long long row_stride_vec) {
    // Loads over NVLink have a round trip of microseconds: every thread keeps kInFlight of them
    // outstanding before its first store.
    constexpr int kInFlight = 8;
    const unsigned per_src = rows * vec_per_row;
    const unsigned total = per_src * static_cast<unsigned>(pp.n_src);
    const unsigned chunk = blockDim.x * kInFlight;
    for (unsigned base = blockIdx.x * chunk; base < total; base += gridDim.x * chunk) {
        uint4 v[kInFlight];
        long long off[kInFlight];
        int src[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
            const unsigned i = base + u * blockDim.x + threadIdx.x;
            src[u] = -1;
            if (i < total) {
                const unsigned s = i / per_src;
                const unsigned rem = i - s * per_src;
                const unsigned row = rem / vec_per_row;
                src[u] = static_cast<int>(s);
                off[u] = (row0 + row) * row_stride_vec + (rem - row * vec_per_row);
                v[u] = ld_nc_na_v4(pp.src[s] + off[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kInFlight; ++u)
            if (src[u] >= 0) pp.dst[src[u]][off[u]] = v[u];
    }
}

// One thread produces 16 bytes of an atom: the four scales of rows {r32 + 32*j, j = 0..3}... laid
// out as [r32][j][k4]; it reads four 4-byte words (one per 32-row group) from the plain layout.
__global__ void __launch_bounds__(256) permute_scales_kernel(const uint8_t* __restrict__ plain, uint8_t* __restrict__ perm,
                                                             int rows, int sf_cols, long long plain_row_stride,
                                                             long long plain_batch_stride, long long perm_batch_stride,
                                                             int batches) {
    const int atoms_k = sf_cols / 4;
    const int row_blocks = (rows + 127) / 128;
    const long long per_batch = static_cast<long long>(row_blocks) * atoms_k * 32;  // 16-byte pieces
    const long long total = per_batch * batches;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int l = static_cast<int>(i / per_batch);
        long long rem = i - l * per_batch;
        const int r32 = static_cast<int>(rem % 32);
        rem /= 32;
        const int kk = static_cast<int>(rem % atoms_k);
        const int rb = static_cast<int>(rem / atoms_k);
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int row = rb * 128 + j * 32 + r32;
            w[j] = (row < rows) ? *reinterpret_cast<const uint32_t*>(plain + l * plain_batch_stride + row * plain_row_stride + kk * 4)
                                : 0u;
        }
        *reinterpret_cast<uint4*>(perm + l * perm_batch_stride + (static_cast<long long>(rb) * atoms_k + kk) * 512 + r32 * 16) =
            make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// The way back, and the check that the two scale tensors an operator call carries say the same
// (the reference's kernels silently trust whichever form they read, template.py:11-14): one
// thread takes 16 bytes of an atom (four rows x four scales) and either writes the four words to
// the plain layout or compares them with it.  result[0] counts differing scale bytes, result[1]
// keeps the smallest (l, row, scale column) linear index of one; padding rows are not looked at.
template <bool COMPARE>
__global__ void __launch_bounds__(256) scales_from_permuted_kernel(const uint8_t* __restrict__ perm, uint8_t* __restrict__ plain,
                                                                   int rows, int sf_cols, long long plain_row_stride,
                                                                   long long plain_batch_stride, long long perm_batch_stride,
                                                                   int batches, unsigned long long* __restrict__ result) {
    const int atoms_k = sf_cols / 4;
    const int row_blocks = (rows + 127) / 128;
    const long long per_batch = static_cast<long long>(row_blocks) * atoms_k * 32;
    const long long total = per_batch * batches;
    unsigned long long bad = 0, first = ~0ull;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int l = static_cast<int>(i / per_batch);
        long long rem = i - l * per_batch;
        const int r32 = static_cast<int>(rem % 32);
        rem /= 32;
        const int kk = static_cast<int>(rem % atoms_k);
        const int rb = static_cast<int>(rem / atoms_k);
        const uint4 v = *reinterpret_cast<const uint4*>(perm + l * perm_batch_stride + (static_cast<long long>(rb) * atoms_k + kk) * 512 + r32 * 16);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int row = rb * 128 + j * 32 + r32;
            if (row >= rows) continue;
            uint32_t* word = reinterpret_cast<uint32_t*>(plain + l * plain_batch_stride + row * plain_row_stride + kk * 4);
            if (!COMPARE) {
                *word = w[j];
            } else {
                uint32_t diff = *word ^ w[j];
                if (diff) {
                    const unsigned long long base = (static_cast<unsigned long long>(l) * rows + row) * sf_cols + kk * 4;
                    const int first_byte = (__ffs(diff) - 1) / 8;
                    if (base + first_byte < first) first = base + first_byte;
                    for (int b = 0; b < 4; ++b, diff >>= 8) bad += (diff & 0xFFu) ? 1 : 0;
                }
            }
        }
    }
    if (COMPARE && bad) {
        atomicAdd(result, bad);
        atomicMin(result + 1, first);
    }
}

// NVFP4 quantiser (the step before the matmul): fp16 / bf16 [rows][K] -> packed e2m1 + one e4m3
// scale per 16 elements, scale = RN(max|x| / 6), element = RN(x / scale) saturated to +-6.
//
// Bound by memory traffic (2 bytes in, 0.5625 or 0.625 out per element).  A lane takes one scale
// block: 32 bytes in by one load, 8 bytes of codes and a scale byte out, and a warp 32 neighbouring
// blocks of a row, so that every access of a warp is one contiguous piece (1024, 256 and 32 bytes; a
// lane that takes 64 elements of a row touches 32 cache lines per load instead, 123 us on bf16
// 8192 x 28672).  Four lanes put their scales together into the 4-byte word that both scale layouts
// have.  A CTA of eight warps covers 8 * R rows x 512 columns; a warp asks for its R rows first of all.
// Measured (us, bf16, graph replay, inputs beyond L2), R = 1 / 2 / 4 / 8:
//   8192 x 28672   108.2 / 104.4 / 101.0 / 129.4   (R = 4: 6.1 TB/s)
//   8192 x 8192     32.5 /  31.7 /  31.5 /  39.8
//   4096 x 7168     15.2 /  15.1 /  15.8 /  21.7
//   2048 x 7168      8.6 /   8.8 /   9.9 /  13.6
//   128 x 7168       2.2 /   2.6 /   3.2 /   5.6
// More rows in flight per warp help as long as there are CTAs enough to even out the end of the
// launch; units of a whole 128-row block, with the scales collected in shared memory and written as
// 16-byte pieces, were slower than either (129.7 and 25.6 us on 8192 and 4096 rows).
// kWide: every address is aligned for the wide accesses (32 bytes for x, 4 for the scales); otherwise
// 16-byte loads, and single bytes of scales.
constexpr int kQuantCols = 512;    // columns per CTA: 32 scale blocks, 8 scale atoms
struct QuantizeParams {
    const uint8_t* x;
    uint8_t* packed;
    uint8_t* sf_plain;   // or null
    uint8_t* sf_perm;    // or null
    int rows, k;
    long long x_row_stride, packed_row_stride, sf_plain_row_stride;   // bytes
};
template <bool kWide>
__device__ __forceinline__ void load_block16(const uint8_t* src, uint32_t (&w)[8]) {
    if (kWide) {
        asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(src));
    } else {
        const uint4 a = __ldcs(reinterpret_cast<const uint4*>(src)), b = __ldcs(reinterpret_cast<const uint4*>(src) + 1);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
        w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    }
}
// Sixteen fp16 / bf16 values -> eight bytes of codes and the scale byte.
template <bool BF16>
__device__ __forceinline__ uint32_t quantize_words(const uint32_t (&w)[8], uint32_t (&codes)[2]) {
    float v[16], amax;
    if (BF16) {
        __nv_bfloat162 top = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
        for (int j = 1; j < 8; ++j) top = __hmax2_nan(top, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[j])));
        const uint32_t t = *reinterpret_cast<const uint32_t*>(&top);
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(amax) : "f"(__uint_as_float(t << 16)), "f"(__uint_as_float(t & 0xffff0000u)));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[2 * j] = __uint_as_float(w[j] << 16);
            v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
        }
    } else {
        __half2 top = __habs2(*reinterpret_cast<const __half2*>(&w[0]));
#pragma unroll
        for (int j = 1; j < 8; ++j) top = __hmax2_nan(top, __habs2(*reinterpret_cast<const __half2*>(&w[j])));
        const float2 t = __half22float2(top);
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(amax) : "f"(t.x), "f"(t.y));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
            v[2 * j] = f.x;
            v[2 * j + 1] = f.y;
        }
    }
    return quantize_block16(v, amax, codes);
}
template <bool kWide>
__device__ __forceinline__ void store_scale_word(uint8_t* at, uint32_t w) {
    if (kWide) {
        *reinterpret_cast<uint32_t*>(at) = w;
    } else {
#pragma unroll
        for (int b = 0; b < 4; ++b) at[b] = static_cast<uint8_t>(w >> (8 * b));
    }
}
template <bool BF16, bool kWide, int R>
__global__ void __launch_bounds__(256) quantize_nvfp4_kernel(const QuantizeParams p) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int blocks = p.k / 16;
    const unsigned col_units = (p.k + kQuantCols - 1) / kQuantCols;
    const int unit_row = blockIdx.x / col_units;
    const int row0 = unit_row * (8 * R) + warp * R;                                    // first row of this warp
    const int blk = (blockIdx.x - unit_row * col_units) * (kQuantCols / 16) + lane;   // this lane's scale block
    const bool in_row = blk < blocks;                                                  // (blocks is a multiple of four)
    // A short quantiser stands between short GEMMs: its launch overlaps the end of the kernel before it.
    ptx::grid_dependency_launch_dependents();
    ptx::grid_dependency_wait();
    const uint8_t* src = p.x + row0 * p.x_row_stride + blk * 32;
    uint32_t w[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (in_row && row0 + r < p.rows) load_block16<kWide>(src + r * p.x_row_stride, w[r]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = row0 + r;
        const bool exists = in_row && row < p.rows;
        uint32_t scales = 0u;
        if (exists) {
            uint32_t codes[2];
            scales = quantize_words<BF16>(w[r], codes) << (8 * (lane & 3));
            *reinterpret_cast<uint2*>(p.packed + row * p.packed_row_stride + blk * 8) = make_uint2(codes[0], codes[1]);
        }
        scales |= __shfl_xor_sync(0xffffffffu, scales, 1);
        scales |= __shfl_xor_sync(0xffffffffu, scales, 2);   // the scales of blocks blk & ~3 ... blk | 3
        if (in_row && (lane & 3) == 0) {
            if (p.sf_perm)   // rows of the last 128-row block that do not exist get zero scales
                store_scale_word<kWide>(p.sf_perm + (static_cast<long long>(row / 128) * (blocks / 4) + blk / 4) * 512 + (row % 32) * 16 + (row % 128) / 32 * 4,
                                        scales);
            if (exists && p.sf_plain) store_scale_word<kWide>(p.sf_plain + row * p.sf_plain_row_stride + blk, scales);
        }
    }
}

}  // namespace nvfp4
