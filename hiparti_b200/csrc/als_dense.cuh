// als_dense.cuh -- the dense steps of an ALS iteration on the FP64 tensor
// cores (mma.sync m8n8k4, the only FP64 tensor instruction of sm_100a): the
// row solve A = M W and the Gram matrix A^T A.  Operands are FP32 in memory,
// products and sums FP64.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace pti {

// D += A B for one 8x8x4 tile: lane l holds A[l / 4][l % 4], B[l % 4][l / 4]
// and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// Columns of A per CTA of solve_rows_kernel (blockIdx.y): wider rows would need
// more accumulators per lane than the register file gives two CTAs.
constexpr uint32_t kSolvePanel = 64;

inline size_t solve_smem(uint32_t R, uint32_t nt) { return (size_t)(R + 15) / 16 * 4 * nt * 32 * 8; }

// A[i, :] = M[i, :] * W (W symmetric); pad columns zeroed.  Adds the column
// sums of squares (FP64) and maxima of the FP32 results into colsq and colmax.
// `vec`: rows of M and A start on 16 bytes.
//
// A warp takes 8 rows at a time and NT column tiles of 8.  The k index of a
// tile is permuted so that a lane's four A operands are one 16-byte load of
// its row; W sits in shared memory in the matching fragment order.  Bound by
// the latency of one pass (load, R/4 dependent products, store) up to R = 32
// and by FP64 arithmetic above.  One thread per element, its statistics added
// with shared-memory atomics, took 13 us for 20,000 rows at R = 32 and 38 for
// the 18,000 (mean) of R = 64; this takes 5.6 and 13.
template <int NT>
__global__ void __launch_bounds__(256, 2) solve_rows_kernel(const float *M, const double *W, uint32_t I, uint32_t R,
                                                            uint32_t stride, float *A, double *colsq, int *colmax,
                                                            bool vec)
{
    extern __shared__ double sB[];  // [k / 4][NT][32]
    __shared__ double s_sq[8][NT * 8];
    __shared__ int s_mx[8][NT * 8];
    const uint32_t K16 = (R + 15) / 16, c0 = blockIdx.y * kSolvePanel;
    for (uint32_t e = threadIdx.x; e < K16 * 4 * NT * 32; e += blockDim.x) {
        const uint32_t l = e & 31, nt = (e >> 5) % NT, kq = (e >> 5) / NT;
        const uint32_t k = 16 * (kq >> 2) + 4 * (l & 3) + (kq & 3), n = c0 + 8 * nt + (l >> 2);
        sB[e] = k < R && n < R ? W[(size_t)k * R + n] : 0.0;
    }
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, t = lane & 3;
    double sq[NT][2];
    float mx[NT][2];
#pragma unroll
    for (int n = 0; n < NT; ++n) sq[n][0] = sq[n][1] = 0.0, mx[n][0] = mx[n][1] = 0.f;
    const uint32_t tiles = I / 8 + (I % 8 != 0);
    for (uint32_t tile = blockIdx.x * 8 + warp; tile < tiles; tile += gridDim.x * 8) {
        const uint32_t row = tile * 8 + r;
        const bool ok = row < I;
        const float *m = M + (size_t)row * stride;
        auto fetch = [&](uint32_t q) {
            const uint32_t c = 16 * q + 4 * t;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ok && c < R) {
                if (vec) v = *reinterpret_cast<const float4 *>(m + c);
                else v = make_float4(m[c], c + 1 < R ? m[c + 1] : 0.f, c + 2 < R ? m[c + 2] : 0.f, c + 3 < R ? m[c + 3] : 0.f);
                // pad columns are not data
                if (c + 1 >= R) v.y = 0.f;
                if (c + 2 >= R) v.z = 0.f;
                if (c + 3 >= R) v.w = 0.f;
            }
            return v;
        };
        double d[NT][2];
#pragma unroll
        for (int n = 0; n < NT; ++n) d[n][0] = d[n][1] = 0.0;
        float4 next = fetch(0);
        for (uint32_t q = 0; q < K16; ++q) {
            const float4 v = next;
            if (q + 1 < K16) next = fetch(q + 1);
            const float av[4] = {v.x, v.y, v.z, v.w};
            const double *b = sB + (size_t)q * 4 * NT * 32 + lane;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int n = 0; n < NT; ++n) dmma884(d[n], (double)av[kk], b[(kk * NT + n) * 32]);
        }
        if (!ok) continue;
        float *a = A + (size_t)row * stride;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const uint32_t c = c0 + 8 * n + 2 * t;
            float o[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                o[j] = c + j < R ? (float)d[n][j] : 0.f;
                sq[n][j] += (double)o[j] * (double)o[j];
                if (o[j] > mx[n][j]) mx[n][j] = o[j];
            }
            if (vec) {
                if (c < stride) *reinterpret_cast<float2 *>(a + c) = make_float2(o[0], o[1]);
            } else {
                if (c < stride) a[c] = o[0];
                if (c + 1 < stride) a[c + 1] = o[1];
            }
        }
        if (blockIdx.y + 1 == gridDim.y)
            for (uint32_t c = c0 + 8 * NT + t; c < stride; c += 4) a[c] = 0.f;
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                sq[n][j] += __shfl_xor_sync(0xffffffffu, sq[n][j], o);
                mx[n][j] = fmaxf(mx[n][j], __shfl_xor_sync(0xffffffffu, mx[n][j], o));
            }
            if (r == 0) {
                s_sq[warp][8 * n + 2 * t + j] = sq[n][j];
                s_mx[warp][8 * n + 2 * t + j] = __float_as_int(mx[n][j]);
            }
        }
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < NT * 8 && c0 + c < R; c += blockDim.x) {
        double s = 0.0;
        int x = 0;  // bits of +0.0f
        for (int w = 0; w < 8; ++w) {
            s += s_sq[w][c];
            x = max(x, s_mx[w][c]);
        }
        atomicAdd(colsq + c0 + c, s);
        atomicMax(colmax + c0 + c, x);
    }
}

// What a Gram pass does to the rows on their way.
struct GramArgs {
    float *A;
    uint32_t I, R, stride;
    // 0: rows as they are.  1 or 2: columns are first divided by lambda, which
    // is their 2-norm (1) or max(largest entry, 1) (2) from solve_rows_kernel's
    // statistics (src/matrix/matrix.c:389-553); rows and lambda are written back
    int scale;
    const double *colsq;
    const int *colmax;
    float *lambda;
    __nv_bfloat16 *bf16;  // receives the (scaled) rows, or null
    int round_bf16;       // the Gram is of the BF16-rounded values
    double *G;            // R x R: the upper triangle (row <= column) is added to
};

__device__ __forceinline__ float gram_lambda(const GramArgs &g, uint32_t c)
{
    if (c >= g.R || g.scale == 0) return 1.f;
    if (g.scale == 1) return (float)sqrt(g.colsq[c]);
    const float v = __int_as_float(g.colmax[c]);
    return v < 1.f ? 1.f : v;
}

// Element (row, c) of the factor, scaled, written back and rounded as asked.
__device__ __forceinline__ double gram_value(const GramArgs &g, float v, uint64_t at, uint32_t c, float lam)
{
    if (c >= g.R) v = 0.f;
    else if (g.scale) v = v / lam;
    if (g.scale) g.A[at] = v;
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    if (g.bf16) g.bf16[at] = h;
    return g.round_bf16 ? (double)__bfloat162float(h) : (double)v;
}

// G += A^T A for R <= 8 NT <= 64.  Both operands of a tile product are the same
// fragment (A[4 rows][8 columns]), so each element is loaded by one lane of one
// warp, and a warp keeps the NT (NT + 1) / 2 upper tiles of its rows in
// registers; the CTA's warps are added in shared memory and go out as one
// atomic per element.  Bound by FP64 arithmetic and those atomics.  With the
// rows in shared memory and one thread per element of G, summed serially,
// a pass took 16 us for 20,000 rows at R = 32 and 42 for 18,000 (mean) at R = 64;
// this takes 7.6 and 19.
template <int NT>
__global__ void __launch_bounds__(256, NT > 4 ? 1 : 2) gram_kernel(GramArgs g)
{
    constexpr int NP = NT * (NT + 1) / 2, SG = NT * 8;
    __shared__ double sG[SG * SG];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cl = lane >> 2;
    float lam[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) lam[n] = gram_lambda(g, 8 * n + cl);
    if (g.scale && blockIdx.x == 0 && warp == 0 && (lane & 3) == 0)
#pragma unroll
        for (int n = 0; n < NT; ++n)
            if (8 * n + cl < g.R) g.lambda[8 * n + cl] = lam[n];
    double acc[NP][2];
#pragma unroll
    for (int i = 0; i < NP; ++i) acc[i][0] = acc[i][1] = 0.0;
    const uint32_t steps = g.I / 8 + (g.I % 8 != 0);  // 8 rows: two tile depths
    for (uint32_t st = blockIdx.x * 8 + warp; st < steps; st += gridDim.x * 8) {
        float raw[2][NT];
        const uint32_t row = st * 8 + (lane & 3);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const uint32_t c = 8 * n + cl;
                raw[h][n] = row + 4 * h < g.I && c < g.stride ? g.A[(size_t)(row + 4 * h) * g.stride + c] : 0.f;
            }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double fr[NT];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const uint32_t c = 8 * n + cl;
                fr[n] = row + 4 * h < g.I && c < g.stride
                            ? gram_value(g, raw[h][n], (size_t)(row + 4 * h) * g.stride + c, c, lam[n])
                            : 0.0;
            }
#pragma unroll
            for (int p = 0, i = 0; p < NT; ++p)
#pragma unroll
                for (int q = p; q < NT; ++q, ++i) dmma884(acc[i], fr[p], fr[q]);
            if (row + 4 * h < g.I)
                for (uint32_t c = SG + cl; c < g.stride; c += 8)
                    gram_value(g, g.A[(size_t)(row + 4 * h) * g.stride + c], (size_t)(row + 4 * h) * g.stride + c, c, 1.f);
        }
    }
    for (uint32_t w = 0; w < 8; ++w) {
        if (warp == w) {
#pragma unroll
            for (int p = 0, i = 0; p < NT; ++p)
#pragma unroll
                for (int q = p; q < NT; ++q, ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        double &x = sG[(8 * p + cl) * SG + 8 * q + 2 * (lane & 3) + j];
                        x = w ? x + acc[i][j] : acc[i][j];
                    }
        }
        __syncthreads();
    }
    for (uint32_t e = threadIdx.x; e < g.R * g.R; e += blockDim.x) {
        const uint32_t p = e / g.R, q = e % g.R;
        if (p <= q) atomicAdd(g.G + e, sG[p * SG + q]);
    }
}

// The same for 64 < R <= 128: a CTA stages 32 scaled rows in shared memory and
// warp w takes the tile rows w and 15 - w of G, 17 tiles in registers, so no
// warp holds all 136.  Rows are 4 doubles longer than the columns, which
// puts the 4 rows of a fragment on different banks.
constexpr int kGramRows = 32, kGramLd = 132;
constexpr size_t kGramWideSmem = (size_t)kGramRows * kGramLd * 8;

__global__ void __launch_bounds__(256) gram_wide_kernel(GramArgs g)
{
    extern __shared__ double tile[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cl = lane >> 2, t = lane & 3;
    const uint32_t NT = (g.R + 7) / 8, n0 = 16 - warp;
    const uint32_t C = threadIdx.x & 127;
    const float lam = gram_lambda(g, C);
    if (g.scale && blockIdx.x == 0 && threadIdx.x < g.R) g.lambda[C] = lam;
    double acc[17][2];
#pragma unroll
    for (int i = 0; i < 17; ++i) acc[i][0] = acc[i][1] = 0.0;
    for (uint64_t r0 = (uint64_t)blockIdx.x * kGramRows; r0 < g.I; r0 += (uint64_t)gridDim.x * kGramRows) {
        __syncthreads();
        for (uint32_t r = threadIdx.x >> 7; r < kGramRows; r += 2) {
            const uint64_t at = (r0 + r) * g.stride + C;
            const bool ok = r0 + r < g.I;
            tile[r * kGramLd + C] = ok && C < g.stride ? gram_value(g, g.A[at], at, C, lam) : 0.0;
            if (ok)
                for (uint32_t c = C + 128; c < g.stride; c += 128)
                    gram_value(g, g.A[at - C + c], at - C + c, c, 1.f);
        }
        __syncthreads();
        for (uint32_t k = 0; k < kGramRows; k += 4) {
            const double *fr = tile + (k + t) * kGramLd + cl;
            const double a0 = fr[8 * warp], a1 = fr[8 * (15 - warp)];
#pragma unroll
            for (uint32_t i = 0; i < 17; ++i) {
                const bool first = i < n0;
                const uint32_t q = first ? warp + i : i - 1;
                if (q < NT) dmma884(acc[i], first ? a0 : a1, fr[8 * q]);
            }
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < 17; ++i) {
        const uint32_t p = 8 * (i < n0 ? warp : 15 - warp) + cl, q = 8 * (i < n0 ? warp + i : i - 1) + 2 * t;
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
            if (p < g.R && q + j < g.R && p <= q + j) atomicAdd(g.G + (size_t)p * g.R + q + j, acc[i][j]);
    }
}

inline cudaError_t launch_gram(const GramArgs &g, cudaStream_t s)
{
    const unsigned sms = (unsigned)sm_count();
    if (g.R > 64) {
        cudaError_t e = cudaFuncSetAttribute(gram_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGramWideSmem);
        if (e != cudaSuccess) return e;
        const unsigned grid = std::max(1u, std::min(ceil_div(g.I, kGramRows), sms));
        gram_wide_kernel<<<grid, 256, kGramWideSmem, s>>>(g);
        return cudaGetLastError();
    }
    const unsigned grid = std::max(1u, std::min(ceil_div(g.I, 64), sms));
    switch ((g.R + 7) / 8) {
        case 1: gram_kernel<1><<<grid, 256, 0, s>>>(g); break;
        case 2: gram_kernel<2><<<grid, 256, 0, s>>>(g); break;
        case 3: gram_kernel<3><<<grid, 256, 0, s>>>(g); break;
        case 4: gram_kernel<4><<<grid, 256, 0, s>>>(g); break;
        case 5: gram_kernel<5><<<grid, 256, 0, s>>>(g); break;
        case 6: gram_kernel<6><<<grid, 256, 0, s>>>(g); break;
        case 7: gram_kernel<7><<<grid, 256, 0, s>>>(g); break;
        default: gram_kernel<8><<<grid, 256, 0, s>>>(g); break;
    }
    return cudaGetLastError();
}

inline cudaError_t launch_solve_rows(const float *M, const double *W, uint32_t I, uint32_t R, uint32_t stride, float *A,
                                     double *colsq, int *colmax, cudaStream_t s)
{
    const bool vec = stride % 4 == 0 && ((uintptr_t)M & 15) == 0 && ((uintptr_t)A & 15) == 0;
    const unsigned panels = (R + kSolvePanel - 1) / kSolvePanel;
    const dim3 grid(std::max(1u, std::min(ceil_div(I, 64), (unsigned)sm_count() * 2 / panels)), panels);
    const uint32_t nt = R > kSolvePanel ? 8 : (R + 7) / 8;
    auto go = [&](auto k, uint32_t NT) {
        const size_t smem = solve_smem(R, NT);
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        k<<<grid, 256, smem, s>>>(M, W, I, R, stride, A, colsq, colmax, vec);
        return cudaGetLastError();
    };
    if (nt <= 1) return go(solve_rows_kernel<1>, 1);
    if (nt <= 2) return go(solve_rows_kernel<2>, 2);
    if (nt <= 3) return go(solve_rows_kernel<3>, 3);
    if (nt <= 4) return go(solve_rows_kernel<4>, 4);
    if (nt <= 6) return go(solve_rows_kernel<6>, 6);
    return go(solve_rows_kernel<8>, 8);
}

}  // namespace pti
