// spd.cuh -- inverse of a small symmetric positive (semi)definite matrix in
// shared memory, by one CTA (the normal-equation solve of an ALS step).
#pragma once
#include <cstdint>

namespace pti {

// Inverse of a symmetric positive definite R x R matrix by symmetric sweeps
// (Gauss-Jordan without pivoting, the pivots being Cholesky's squared diagonal
// and the result the sum of the same R outer products that L^-T L^-1 is), by a
// CTA of 32 x NTY threads.  Thread (x, y) keeps elements (y + NTY a, x + 32 b)
// in registers, a < PA, b < PB, so R <= min(NTY * PA, 32 * PB); a step costs
// one barrier and one row of the matrix through shared memory, double-buffered
// (s_row[2 * 32 * PB], s_piv[2]).  load(i, j) gives the elements, store(i, j,
// v) takes the inverse.  Returns false, storing nothing, if a pivot is not
// positive: the matrix is not positive definite.
//
// The chain of R dependent steps bounds it.  One warp factoring and R threads
// substituting, each step a chain of dependent loads, took 109 us at R = 32
// and 214 at R = 64; this takes 15 and 44.
// Against an extended-precision inverse its error is 0.3 to 0.6 of theirs, on
// Grams of condition 1e2 to 1e12.
template <int NTY, int PA, int PB, class Load, class Store>
__device__ bool sweep_inverse(uint32_t R, Load load, Store store, double *s_row, double *s_piv)
{
    const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double x[PA][PB];
#pragma unroll
    for (int a = 0; a < PA; ++a)
#pragma unroll
        for (int b = 0; b < PB; ++b) {
            const uint32_t i = ty + NTY * a, j = tx + 32 * b;
            x[a][b] = i < R && j < R ? load(i, j) : 0.0;
        }
    // row k and the reciprocal of its pivot (0: not positive) for step k
    auto publish = [&](uint32_t k) {
        double *row = s_row + (k & 1) * 32 * PB;
#pragma unroll
        for (int a = 0; a < PA; ++a)
            if (ty + NTY * a == k) {
#pragma unroll
                for (int b = 0; b < PB; ++b) {
                    row[tx + 32 * b] = x[a][b];
                    if (tx + 32 * b == k) s_piv[k & 1] = x[a][b] > 0.0 ? 1.0 / x[a][b] : 0.0;
                }
            }
    };
    publish(0);
    __syncthreads();
    for (uint32_t k = 0; k < R; ++k) {
        const double *row = s_row + (k & 1) * 32 * PB;
        const double p = s_piv[k & 1];
        if (!(p > 0.0)) {
            __syncthreads();  // the buffers are free again
            return false;
        }
        double vj[PB], wj[PB];
#pragma unroll
        for (int b = 0; b < PB; ++b) {
            vj[b] = row[tx + 32 * b];
            wj[b] = vj[b] * p;
        }
#pragma unroll
        for (int a = 0; a < PA; ++a) {
            const uint32_t i = ty + NTY * a;
            const double vi = row[i];
            const bool pivot_row = i == k;
#pragma unroll
            for (int b = 0; b < PB; ++b) {
                double v = x[a][b] - vi * wj[b];
                if (tx + 32 * b == k) v = vi * p;
                if (pivot_row) v = tx + 32 * b == k ? -p : wj[b];
                x[a][b] = v;
            }
        }
        if (k + 1 < R) publish(k + 1);
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < PA; ++a)
#pragma unroll
        for (int b = 0; b < PB; ++b) {
            const uint32_t i = ty + NTY * a, j = tx + 32 * b;
            if (i < R && j < R) store(i, j, -x[a][b]);
        }
    return true;
}

// W = V^-1 for a symmetric R x R matrix (R <= 32) in FP64 shared memory, by a
// CTA of 256 threads.  Returns 0 (positive definite), 1 (not positive
// definite: Gauss-Jordan elimination with partial pivoting, the counterpart of
// the reference's sgesv fallback, src/matrix/matrix_solver.c:66-80) or 2
// (singular: W = identity, so the rows stay unsolved as when sgesv fails).
// L and Li are the fallback's scratch.
__device__ inline int spd_inverse(const double *V, double *L, double *Li, double *W, uint32_t R)
{
    __shared__ int s_sing;
    __shared__ uint32_t s_piv;
    __shared__ double s_rows[64], s_rcp[2];
    const uint32_t tid = threadIdx.x;
    const uint32_t RR = R * R;
    if (sweep_inverse<8, 4, 1>(
            R, [&](uint32_t i, uint32_t j) { return V[i * R + j]; },
            [&](uint32_t i, uint32_t j, double v) { W[i * R + j] = v; }, s_rows, s_rcp)) {
        __syncthreads();
        return 0;
    }
    // Gauss-Jordan on [V | I]: L holds V, Li holds I
    for (uint32_t e = tid; e < RR; e += blockDim.x) {
        L[e] = V[e];
        Li[e] = (e / R == e % R) ? 1.0 : 0.0;
    }
    if (tid == 0) s_sing = 0;
    __syncthreads();
    for (uint32_t j = 0; j < R; ++j) {
        if (tid == 0) {
            uint32_t p = j;
            for (uint32_t i = j + 1; i < R; ++i)
                if (fabs(L[i * R + j]) > fabs(L[p * R + j])) p = i;
            s_piv = p;
            if (L[p * R + j] == 0.0) s_sing = 1;
        }
        __syncthreads();
        if (s_sing) break;
        const uint32_t p = s_piv;
        if (p != j)
            for (uint32_t c = tid; c < R; c += blockDim.x) {
                double t = L[j * R + c];
                L[j * R + c] = L[p * R + c];
                L[p * R + c] = t;
                t = Li[j * R + c];
                Li[j * R + c] = Li[p * R + c];
                Li[p * R + c] = t;
            }
        __syncthreads();
        const double piv = L[j * R + j];
        __syncthreads();
        for (uint32_t c = tid; c < R; c += blockDim.x) {
            L[j * R + c] /= piv;
            Li[j * R + c] /= piv;
        }
        __syncthreads();
        for (uint32_t e = tid; e < RR; e += blockDim.x) {
            const uint32_t i = e / R, c = e % R;
            if (i == j) continue;
            const double f = L[i * R + j];
            if (c != j) L[i * R + c] -= f * L[j * R + c];
            Li[i * R + c] -= f * Li[j * R + c];
        }
        __syncthreads();
        for (uint32_t i = tid; i < R; i += blockDim.x)
            if (i != j) L[i * R + j] = 0.0;
        __syncthreads();
    }
    const int sing = s_sing;
    for (uint32_t e = tid; e < RR; e += blockDim.x) W[e] = sing ? ((e / R == e % R) ? 1.0 : 0.0) : Li[e];
    __syncthreads();
    return sing ? 2 : 1;
}

}  // namespace pti
