// NVFP4 block-scaled GEMV for sm_100a (CUDA cores; the op is HBM-bound, not a dense contraction):
//   c[m, l] = sum_k  e2m1(a[m,k,l]) * sfa[m,k/16,l] * e2m1(b[k,l]) * sfb[k/16,l]
//
// gemv_nvfp4_kernel (the other K, or a launch shape the caller asks for): one warp streams R rows; a lane owns 32-byte chunks (64 elements = 4 scale blocks) at a
// stride of 1024 bytes, so every warp-wide 256-bit load covers 1 KiB of contiguous row.  Per
// 16-element block the products are summed in f16x2 (8 terms per half: exact), widened to fp32,
// scaled by sfa*sfb and accumulated in fp32.  The vector and its scales are re-read through L1
// (evict-last) by every row; the matrix streams past L1 with evict-first hints.
//
// Covers the reference's GEMV (old_files/1.py:499-607) but keeps every cross-block add in fp32.
#pragma once
#include "ptx.cuh"

namespace nvfp4 {

constexpr int kGemvThreads = 128;

struct GemvParams {
    const uint8_t* a;    // [L][M][K/2]
    const uint8_t* b;    // [L][1][K/2]
    const uint8_t* sfa;  // plain [L][M][K/16]
    const uint8_t* sfb;  // plain [L][1][K/16]
    __half* c;
    long long a_row_stride, a_batch_stride;      // bytes
    long long b_batch_stride;                    // bytes
    long long sfa_row_stride, sfa_batch_stride;  // bytes
    long long sfb_batch_stride;                  // bytes
    long long c_row_stride, c_batch_stride;      // elements
    int M, K, L;
};

struct Chunk32 {
    uint32_t w[8];
};

__device__ __forceinline__ Chunk32 ld_stream_32B(const uint8_t* ptr) {
    Chunk32 v;
    uint64_t q0, q1, q2, q3;
    asm volatile("ld.global.L1::no_allocate.L2::evict_first.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(q0), "=l"(q1), "=l"(q2), "=l"(q3) : "l"(ptr));
    v.w[0] = static_cast<uint32_t>(q0); v.w[1] = static_cast<uint32_t>(q0 >> 32);
    v.w[2] = static_cast<uint32_t>(q1); v.w[3] = static_cast<uint32_t>(q1 >> 32);
    v.w[4] = static_cast<uint32_t>(q2); v.w[5] = static_cast<uint32_t>(q2 >> 32);
    v.w[6] = static_cast<uint32_t>(q3); v.w[7] = static_cast<uint32_t>(q3 >> 32);
    return v;
}
__device__ __forceinline__ Chunk32 ld_keep_32B(const uint8_t* ptr) {
    Chunk32 v;
    uint64_t q0, q1, q2, q3;
    asm volatile("ld.global.L1::evict_last.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(q0), "=l"(q1), "=l"(q2), "=l"(q3) : "l"(ptr));
    v.w[0] = static_cast<uint32_t>(q0); v.w[1] = static_cast<uint32_t>(q0 >> 32);
    v.w[2] = static_cast<uint32_t>(q1); v.w[3] = static_cast<uint32_t>(q1 >> 32);
    v.w[4] = static_cast<uint32_t>(q2); v.w[5] = static_cast<uint32_t>(q2 >> 32);
    v.w[6] = static_cast<uint32_t>(q3); v.w[7] = static_cast<uint32_t>(q3 >> 32);
    return v;
}
__device__ __forceinline__ uint32_t ld_stream_u32(const uint8_t* ptr) {
    uint32_t v;
    asm volatile("ld.global.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(ptr));
    return v;
}
__device__ __forceinline__ uint32_t ld_keep_u32(const uint8_t* ptr) {
    uint32_t v;
    asm volatile("ld.global.L1::evict_last.u32 %0, [%1];" : "=r"(v) : "l"(ptr));
    return v;
}

// Four bytes = eight e2m1 values -> four f16x2 (low nibble in the low half).
__device__ __forceinline__ void cvt_e2m1x8(uint32_t packed, uint32_t (&h2)[4]) {
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
        "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
        "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
        : "=r"(h2[0]), "=r"(h2[1]), "=r"(h2[2]), "=r"(h2[3]) : "r"(packed));
}
// Four e4m3 scale bytes -> four fp32.
__device__ __forceinline__ void cvt_e4m3x4(uint32_t packed, float (&f)[4]) {
    uint32_t lo, hi;
    asm("{\n\t.reg .b16 s0, s1;\n\t"
        "mov.b32 {s0, s1}, %2;\n\t"
        "cvt.rn.f16x2.e4m3x2 %0, s0;\n\t"
        "cvt.rn.f16x2.e4m3x2 %1, s1;\n\t}"
        : "=r"(lo), "=r"(hi) : "r"(packed));
    const float2 a = __half22float2(*reinterpret_cast<__half2*>(&lo));
    const float2 b = __half22float2(*reinterpret_cast<__half2*>(&hi));
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}

// A warp's share of R rows: chunks [chunk_begin, chunk_end) of 64 elements, partial sums in fp32.
template <int R, int UNROLL>
__device__ __forceinline__ void gemv_accumulate(const uint8_t* const (&a_ptr)[R], const uint8_t* const (&sfa_ptr)[R], const uint8_t* b_ptr,
                                                const uint8_t* sfb_ptr, int chunk_begin, int chunk_end, int lane, float (&sum)[R]) {
    for (int base = chunk_begin; base < chunk_end; base += 32 * UNROLL) {
        Chunk32 av[UNROLL][R];
        uint32_t sav[UNROLL][R];
        Chunk32 bv[UNROLL];
        uint32_t sbv[UNROLL];
#pragma unroll
        for (int i = 0; i < UNROLL; ++i) {
            const int chunk = base + i * 32 + lane;
            if (chunk < chunk_end) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    av[i][r] = ld_stream_32B(a_ptr[r] + chunk * 32);
                    sav[i][r] = ld_stream_u32(sfa_ptr[r] + chunk * 4);
                }
                bv[i] = ld_keep_32B(b_ptr + chunk * 32);
                sbv[i] = ld_keep_u32(sfb_ptr + chunk * 4);
            }
        }
#pragma unroll
        for (int i = 0; i < UNROLL; ++i) {
            const int chunk = base + i * 32 + lane;
            if (chunk < chunk_end) {
                float sfb_f[4];
                cvt_e4m3x4(sbv[i], sfb_f);
                float sfa_f[R][4];
#pragma unroll
                for (int r = 0; r < R; ++r) cvt_e4m3x4(sav[i][r], sfa_f[r]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {  // one 16-element scale block = two 32-bit words
                    uint32_t b2[8];
                    {
                        uint32_t t[4];
                        cvt_e2m1x8(bv[i].w[2 * j], t);
                        b2[0] = t[0]; b2[1] = t[1]; b2[2] = t[2]; b2[3] = t[3];
                        cvt_e2m1x8(bv[i].w[2 * j + 1], t);
                        b2[4] = t[0]; b2[5] = t[1]; b2[6] = t[2]; b2[7] = t[3];
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        uint32_t a2[8];
                        {
                            uint32_t t[4];
                            cvt_e2m1x8(av[i][r].w[2 * j], t);
                            a2[0] = t[0]; a2[1] = t[1]; a2[2] = t[2]; a2[3] = t[3];
                            cvt_e2m1x8(av[i][r].w[2 * j + 1], t);
                            a2[4] = t[0]; a2[5] = t[1]; a2[6] = t[2]; a2[7] = t[3];
                        }
                        __half2 acc = __float2half2_rn(0.f);
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            acc = __hfma2(*reinterpret_cast<__half2*>(&a2[e]), *reinterpret_cast<__half2*>(&b2[e]), acc);
                        const float2 s = __half22float2(acc);
                        sum[r] = fmaf(s.x + s.y, sfa_f[r][j] * sfb_f[j], sum[r]);
                    }
                }
            }
        }
    }
}

template <int R, int UNROLL = (R == 1) ? 4 : (R == 2 ? 2 : 1)>
__global__ void __launch_bounds__(kGemvThreads) gemv_nvfp4_kernel(const GemvParams p) {
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int l = blockIdx.y;
    const int row0 = (blockIdx.x * (blockDim.x >> 5) + warp) * R;   // 1, 2 or 4 warps per CTA, each on its own rows
    if (row0 >= p.M) return;

    const uint8_t* b_ptr = p.b + l * p.b_batch_stride;
    const uint8_t* sfb_ptr = p.sfb + l * p.sfb_batch_stride;
    const uint8_t* a_ptr[R];
    const uint8_t* sfa_ptr[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = min(row0 + r, p.M - 1);  // clamp: surplus rows recompute the last one and are not stored
        a_ptr[r] = p.a + l * p.a_batch_stride + row * p.a_row_stride;
        sfa_ptr[r] = p.sfa + l * p.sfa_batch_stride + row * p.sfa_row_stride;
    }

    float sum[R];
#pragma unroll
    for (int r = 0; r < R; ++r) sum[r] = 0.f;
    gemv_accumulate<R, UNROLL>(a_ptr, sfa_ptr, b_ptr, sfb_ptr, 0, p.K / 64, lane, sum);

#pragma unroll
    for (int r = 0; r < R; ++r) {
        float v = sum[r];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0 && row0 + r < p.M)
            p.c[l * p.c_batch_stride + static_cast<long long>(row0 + r) * p.c_row_stride] = __float2half_rn(v);
    }
}

// The form for K up to 8192, and 14400 to 16384: the vector stays in registers.  A row worker is LANES lanes (or, for K
// beyond 2048, k_warps whole warps side by side), a 64-element chunk of K per lane: it converts its
// chunks of the vector once and walks rows of the matrix, four at a time with the next four in flight.
// The matrix is then all that is loaded and converted, where the form above converts the vector again for
// every R rows.  The partial sums of k_warps warps meet in shared memory.  The grid is resident at once
// and the rows are split evenly over it (plan_gemv_split), so short rows neither pay a CTA each nor end
// in a ragged wave, and the launch can overlap the end of the kernel before it in the stream: the first
// rows are asked into L2 ahead of the dependency wait.
// Bound by HBM.  Measured (us, graph replay over rotating inputs, the form above -> this one): 7168 x 2048 x 4
// 9.1 -> 7.6, 7168 x 16384 x 1 15.3 -> 13.2, 7168 x 16384 x 4 45.2 -> 43.9 (6.0 TB/s), 4096 x 7168 x 8
// 26.3 -> 25.1; without the overlap of launches 8.9, 14.5, 45.6 and 26.4.
constexpr int kGemvRowsPerStep = 4;
constexpr int kGemvSliceChunks = 32;
constexpr int kGemvMaxKWarps = 8;
constexpr int kGemvBatchRows = 512;    // rows of a worker between two meetings of its warps

// How the rows of all batches go to the row workers: every `sharers` workers in turn take sharers * rows_each + rows_left
// rows, the first rows_left of them one more than the others.
struct GemvSplit {
    int workers, sharers, rows_each, rows_left;
    __host__ __device__ void rows_of(int worker, int total, int* begin, int* end) const {   // none for a worker beyond the last
        int i = worker, first = 0;
        if (sharers < workers) {
            const int share = worker / sharers;
            i -= share * sharers;
            first = share * (sharers * rows_each + rows_left);
        }
        const int b = first + i * rows_each + (i < rows_left ? i : rows_left), e = b + rows_each + (i < rows_left ? 1 : 0);
        *begin = b < total ? b : total;
        *end = e < total ? e : total;
    }
};
// m rows of each of l batches, in steps of step_rows, over `resident` workers that run at once.  Evenly shared, a
// worker may cross into the next batch, loads another vector and begins a step anew.  Up to three steps that shows
// (1 x 8192, 8 batches: 2 workers with four batches each 5.6 us, 8 workers 2.2; 100 x 1024 x 8: 3.4 and 2.3; 1000 x 2112 x 8:
// 6.5 and 5.2), and where workers cross batch after batch; there each batch has workers of its own if that takes no more
// steps.  With more steps the few that cross are lost among them, and the even share is as fast or faster (7168 x 2048 x 4:
// 7.8 us, by batches 8.5).
inline GemvSplit plan_gemv_split(int m, int l, int step_rows, int resident) {
    auto ceil_div = [](long long a, long long b) { return (a + b - 1) / b; };
    const long long rows = static_cast<long long>(m) * l;
    const long long own = resident / l < 1 ? 1 : resident / l < ceil_div(m, step_rows) ? resident / l : ceil_div(m, step_rows);
    const long long own_steps = ceil_div(ceil_div(m, own), step_rows) * ceil_div(own * l, resident);
    const long long all = resident < ceil_div(rows, step_rows) ? resident : ceil_div(rows, step_rows);
    const long long all_rows = ceil_div(rows, all), all_steps = ceil_div(all_rows, step_rows), crossings = ceil_div(all_rows, m);
    if (l > 1 && own_steps <= all_steps + crossings && (all_steps <= 3 || crossings > 1))
        return GemvSplit{static_cast<int>(own * l), static_cast<int>(own), static_cast<int>(m / own), static_cast<int>(m % own)};
    return GemvSplit{static_cast<int>(all), static_cast<int>(all), static_cast<int>(rows / all), static_cast<int>(rows % all)};
}

// Sums of four values over LANES neighbouring lanes; lanes that are a multiple of LANES / 4 hold value
// (lane % LANES) / (LANES / 4).
template <int LANES>
__device__ __forceinline__ float lanes_sum4(const float (&v)[4], int lane) {
    const bool up = lane & (LANES / 2);
    float a = up ? v[2] : v[0], b = up ? v[3] : v[1];
    a += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], LANES / 2);
    b += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], LANES / 2);
    const bool up2 = lane & (LANES / 4);
    float s = up2 ? b : a;
    s += __shfl_xor_sync(0xffffffffu, up2 ? a : b, LANES / 4);
#pragma unroll
    for (int off = LANES / 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

template <int LANES>
__global__ void __launch_bounds__(kGemvMaxKWarps * 32, 2) gemv_resident_kernel(const GemvParams p, int k_warps, int row_workers, GemvSplit split) {
    __shared__ float part[kGemvMaxKWarps * kGemvBatchRows];   // [row worker][row][k warp]
    constexpr int R = kGemvRowsPerStep;
    constexpr int kSub = 32 / LANES;                          // groups of lanes that take R rows each in a step of their warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int worker_in_cta = warp / k_warps, k_warp = warp % k_warps;
    // rows [row_begin, row_end) of all batches' rows
    const int worker = static_cast<int>(blockIdx.x) * row_workers + worker_in_cta;
    int row_begin, row_end;
    split.rows_of(worker, p.M * p.L, &row_begin, &row_end);
    const int batch_rows = k_warps > 1 ? kGemvBatchRows : split.rows_each + 1;
    const int batches = (split.rows_each + batch_rows) / batch_rows;   // the same for every warp of the grid
    const int chunks = p.K / 64;
    const int chunk_begin = k_warp * chunks / k_warps, chunk_end = (k_warp + 1) * chunks / k_warps;
    const int chunk = chunk_begin + lane % LANES;
    const int sub_row = lane / LANES * R;
    const bool active = chunk < chunk_end;

    // The first rows are asked into L2 ahead of the dependency wait (a prefetch consumes nothing).
    if (active && row_begin < row_end) {
        const int l = row_begin / p.M, row0 = row_begin - l * p.M;
        const int n = min(min(sub_row + R, row_end - row_begin), p.M - row0);
        const uint8_t* ptr = p.a + l * p.a_batch_stride + static_cast<long long>(row0) * p.a_row_stride + chunk * 32;
        for (int r = sub_row; r < n; ++r) asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr + r * p.a_row_stride));
    }
    ptx::grid_dependency_launch_dependents();
    ptx::grid_dependency_wait();

    __half2 b2[32];
    float sfb[4];
    int loaded_l = -1;
    for (int batch = 0; batch < batches; ++batch) {
        const int batch_begin = min(row_begin + batch * batch_rows, row_end);
        const int batch_end = min(batch_begin + batch_rows, row_end);
        for (int seg = batch_begin; seg < batch_end;) {   // rows of one l
            const int l = seg / p.M;
            const int row0 = seg - l * p.M;
            const int n_rows = min(batch_end - seg, p.M - row0);
            const uint8_t* a_ptr = p.a + l * p.a_batch_stride + static_cast<long long>(row0 + sub_row) * p.a_row_stride + chunk * 32;
            const uint8_t* sfa_ptr = p.sfa + l * p.sfa_batch_stride + static_cast<long long>(row0 + sub_row) * p.sfa_row_stride + chunk * 4;
            Chunk32 next[R];
            uint32_t next_sf[R];
            auto fetch = [&](int row) {   // rows [row + sub_row, + R) of the segment; the pointers stand at the first
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (active && row + sub_row + r < n_rows) {
                        next[r] = ld_stream_32B(a_ptr);
                        next_sf[r] = ld_stream_u32(sfa_ptr);
                    }
                    a_ptr += p.a_row_stride;
                    sfa_ptr += p.sfa_row_stride;
                }
                if constexpr (kSub > 1) {
                    a_ptr += (kSub - 1) * R * p.a_row_stride;
                    sfa_ptr += (kSub - 1) * R * p.sfa_row_stride;
                }
            };
#pragma unroll
            for (int r = 0; r < R; ++r) { next[r] = Chunk32{}; next_sf[r] = 0u; }
            fetch(0);
            if (l != loaded_l) {
                loaded_l = l;
                Chunk32 bv{};
                uint32_t sbv = 0u;
                if (active) {
                    bv = ld_keep_32B(p.b + l * p.b_batch_stride + chunk * 32);
                    sbv = ld_keep_u32(p.sfb + l * p.sfb_batch_stride + chunk * 4);
                }
                cvt_e4m3x4(sbv, sfb);
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    uint32_t t[4];
                    cvt_e2m1x8(bv.w[w], t);
#pragma unroll
                    for (int e = 0; e < 4; ++e) b2[4 * w + e] = *reinterpret_cast<__half2*>(&t[e]);
                }
            }
            for (int row = 0; row < n_rows; row += R * kSub) {
                Chunk32 cur[R];
                uint32_t cur_sf[R];
#pragma unroll
                for (int r = 0; r < R; ++r) { cur[r] = next[r]; cur_sf[r] = next_sf[r]; }
                fetch(row + R * kSub);
                float sum[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float sfa[4];
                    cvt_e4m3x4(cur_sf[r], sfa);
                    sum[r] = 0.f;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {   // one scale block: eight exact products per half, then fp32
                        uint32_t t0[4], t1[4];
                        cvt_e2m1x8(cur[r].w[2 * j], t0);
                        cvt_e2m1x8(cur[r].w[2 * j + 1], t1);
                        __half2 acc = __float2half2_rn(0.f);
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc = __hfma2(*reinterpret_cast<__half2*>(&t0[e]), b2[8 * j + e], acc);
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc = __hfma2(*reinterpret_cast<__half2*>(&t1[e]), b2[8 * j + 4 + e], acc);
                        const float2 s = __half22float2(acc);
                        sum[r] = fmaf(s.x + s.y, sfa[j] * sfb[j], sum[r]);
                    }
                    if (!active) sum[r] = 0.f;      // (lanes past the slice: whatever they hold does not count)
                }
                const float s = lanes_sum4<LANES>(sum, lane);
                const int r = sub_row + lane % LANES / (LANES / 4);
                if (lane % (LANES / 4) == 0 && row + r < n_rows) {
                    if (k_warps == 1) p.c[l * p.c_batch_stride + static_cast<long long>(row0 + row + r) * p.c_row_stride] = __float2half_rn(s);
                    else part[(worker_in_cta * kGemvBatchRows + seg - batch_begin + row + r) * k_warps + k_warp] = s;
                }
            }
            seg += n_rows;
        }
        if (k_warps > 1) {
            __syncthreads();
            for (int i = k_warp * 32 + lane; i < batch_end - batch_begin; i += k_warps * 32) {
                const float* src = part + (worker_in_cta * kGemvBatchRows + i) * k_warps;
                float v = 0.f;
                for (int w = 0; w < k_warps; ++w) v += src[w];
                const int row = batch_begin + i;
                const int l = row / p.M;
                p.c[l * p.c_batch_stride + static_cast<long long>(row - l * p.M) * p.c_row_stride] = __float2half_rn(v);
            }
            __syncthreads();
        }
    }
}

}  // namespace nvfp4
