// batched.cu -- CPD-ALS of many small 3-D tensors at once (no counterpart in
// the reference, whose CPD drivers factor one tensor per call:
// src/sptensor/cpd.c:32-208, src/sptensor/hicoo/cpd.c).
//
// Every tensor of the batch is converted to HiCOO on the GPU and given the
// per-mode schedules of sched.cu (blocks ordered by output block row, cut into
// tiles of kPlanTile nonzeros).  One ALS iteration of the WHOLE batch is one
// launch of a persistent kernel whose CTAs pull tasks from a queue:
//
//   tile    (b, m, t)  MTTKRP of tile t of tensor b's mode-m schedule into
//                      M_bm: the tile's decoded records (in output-row order)
//                      are bulk-copied, one vector atomic per row run and
//                      thread group
//   inverse (b, m)     W = (G_a o G_b)^-1, FP64 (symmetric sweeps; Gauss-Jordan
//                      fallback); it needs only the other modes' Grams, so it
//                      precedes the tensor's tiles and runs beside them
//   solve   (b, m, c)  rows of chunk c: A_bm = M_bm W, FP64, with the columns'
//                      sums of squares and maxima
//   gram    (b, m, c)  rows of chunk c: A_bm /= lambda (2-norm in iteration 0,
//                      else max(column max, 1)), the BF16 copy, the chunk's part
//                      of G_bm = A_bm^T A_bm, and of <X, model> after the last
//                      mode; the chunk that ends last stores the Gram and after
//                      the last mode the fit (src/sptensor/cpd.c:90-147 for one
//                      tensor)
//
// A mode's dense step is 3.2 I R^2 FP64 operations, which one SM takes 70 us
// for at I = 5,000 and R = 32 and which lie on every tensor's critical path
// three times an iteration, so it is cut into row chunks for many SMs.  One CTA
// a step, with tiles decoded by the CTA that walks them: 1.75 ms an iteration
// of 128 tensors (10M nonzeros) and 0.99 of 20; this takes 0.72 and 0.15.
//
// The queue is ordered in waves -- all mode-0 inverses and tiles, all mode-0
// solves, all mode-0 Grams, all mode-1 inverses and tiles, ... -- and a task
// waits (bounded) on per-tensor counters for the tasks it depends on.  Tasks
// are handed out in queue order and only depend on earlier tasks.  A CTA holds
// two: the one it runs and the next, whose records (which never change) are
// copied meanwhile.  The earliest unfinished task has its inputs complete and
// is the first of the two in the CTA that holds it (the one before it would be
// unfinished too), so the queue makes progress whatever the number of
// co-resident CTAs.
//
// Data written inside the launch (factors, M, Grams) is read after an acquire
// on the counter, never through the read-only path; static data (the
// schedules) is bulk-copied.
//
// The iteration (counter reset, persistent kernel, iteration-counter bump) is
// captured once per call in a CUDA graph and replayed; the kernel reads the
// iteration number from device memory, so one graph serves the BF16 and the
// closing FP32 iterations alike.
//
// An autotuner picks the HiCOO block size (sb_bits) and the columns per lane
// of the BF16 iterations (4 or 8, i.e. R/4 or R/8 threads per nonzero) by
// timing whole iterations of the batch, and caches the choice per batch shape.
#include <cuda_bf16.h>

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>
#include <tuple>

#include "kutil.cuh"
#include "spd.cuh"
#include "tensor.cuh"
#include "tma.cuh"

namespace pti {

constexpr int kBThreads = 256;
constexpr int kBMaxRank = 32;
constexpr int kRowPad = 40;                     // row stride (doubles) of the dense passes' row tiles
constexpr int kBTile = kPlanTile;
constexpr uint64_t kWaitNs = 2000000000ull;     // bound of every dependency wait: 2 s

// error bits of the batch's error word
constexpr uint32_t kErrRange = 1u, kErrCopy = 2u, kErrWait = 4u;

struct BatchPlan {        // the mode-m schedule of tensor b
    uint64_t nnz;
    const uint4 *recs;                // {output row, operand rows, value}, tiles in output-row order
    float *M;                         // MTTKRP output, dims[m] x stride
    const float *A32[2];              // operand factors (modes k != m, increasing)
    const __nv_bfloat16 *A16[2];
    uint32_t ntiles, chunks, R, stride;  // tiles; chunks of the mode's rows
};

struct BatchTensor {
    float *A[3];                      // FP32 factors, dims[m] x stride
    __nv_bfloat16 *Ab[3];             // BF16 copies read by the MTTKRP in mixed mode
    float *M[3];
    double *G;                        // [3][R][R] Grams
    float *lambda;                    // [R]
    const double *normX2;             // ||X||^2
    uint32_t dims[3];
    uint32_t R, stride;
};

// What the chunks of a mode's dense step add into, zeroed before each iteration.
struct BatchAcc {
    double G[kBMaxRank * kBMaxRank];  // upper triangle, row stride kBMaxRank
    double colsq[kBMaxRank];
    double inner;                     // <X, model> (last mode)
    int colmax[kBMaxRank];            // bits of the FP32 maxima
    int pad[2];
};

enum TaskKind : uint32_t { kTile = 0, kInverse = 1, kSolve = 2, kGram = 3 };
constexpr uint32_t kMinChunkRows = 128;  // rows of a solve or gram task: two blocks of 8 for each warp

struct BatchArgs {
    const uint2 *tasks;               // x = (b*3 + m) << 2 | kind, y = tile or chunk
    const BatchPlan *plans;           // [B*3], plan = b*3 + m
    const BatchTensor *tens;          // [B]
    BatchAcc *acc;                    // [B*3]
    double *W;                        // [B*3][kBMaxRank^2]
    uint32_t *ctrl;                   // queue head, then counters (ctrl_words)
    const uint32_t *iter;             // iteration number (bumped after every launch)
    double *fits;                     // [B][niters]
    uint32_t *err;
    uint32_t ntasks, ntensors, niters, fp32_sweeps, cpl;
    uint32_t chunk_rows;              // of a solve or gram task
    int mixed;
    uint64_t wait_ns;                 // bound of every dependency wait
};

// ctrl: head, then per (b, m) tiles, inverses, solve chunks and gram chunks
// done, then per tensor the modes done
inline size_t ctrl_words(size_t B) { return 1 + 13 * B; }

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Waits until *p >= target.  Gives up (false) after wait_ns, after 2^28
// polls should the timer not advance, or as soon as another wait of the
// launch has given up (err holds kErrWait), so a failed launch ends within
// about one wait bound instead of one per task.
__device__ bool wait_at_least(const uint32_t *p, uint32_t target, const uint32_t *err, uint64_t wait_ns)
{
    if (ld_acquire(p) >= target) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t i = 0; i < (1u << 28); ++i) {
        __nanosleep(64);
        if (ld_acquire(p) >= target) return true;
        if ((i & 255u) == 255u &&
            (global_ns() - t0 > wait_ns || (*(volatile const uint32_t *)err & kErrWait))) return false;
    }
    return false;
}

// CPL consecutive columns of a factor row.  The factors change during the
// launch, so the read-only path is not used; the acquire that a task starts
// with keeps older lines of the L1 from being read.
template <int CPL, class FT>
struct Cols {
    static constexpr int kWords = CPL * (int)sizeof(FT) / 4;
    uint32_t w[kWords];
    __device__ __forceinline__ void load(const FT *row, uint32_t col)
    {
        const FT *p = row + col;
        if constexpr (kWords >= 4) {
#pragma unroll
            for (int q = 0; q < kWords / 4; ++q) {
                const uint4 x = *(reinterpret_cast<const uint4 *>(p) + q);
                w[4 * q] = x.x; w[4 * q + 1] = x.y; w[4 * q + 2] = x.z; w[4 * q + 3] = x.w;
            }
        } else {
            const uint2 x = *reinterpret_cast<const uint2 *>(p);
            w[0] = x.x; w[1] = x.y;
        }
    }
    __device__ __forceinline__ float at(int c) const
    {
        if constexpr (sizeof(FT) == 4) {
            return __uint_as_float(w[c]);
        } else {
            const uint32_t h = w[c >> 1];
            return __uint_as_float((c & 1) ? (h & 0xFFFF0000u) : (h << 16));
        }
    }
};

// Shared memory (bytes): two record buffers, the current and the next task's,
// with a part between them.  A task that is not a tile has the buffer of its
// turn and that part to itself, kTaskSmem bytes from task_base().
constexpr uint32_t kRecBytes = 16 * kBTile;
constexpr uint32_t kMidBytes = 9 * 1024;
constexpr uint32_t kTaskSmem = kRecBytes + kMidBytes;
constexpr uint32_t kBatchSmem = 2 * kRecBytes + kMidBytes;
__device__ __forceinline__ uint32_t rec_base(uint32_t buf) { return buf ? kRecBytes + kMidBytes : 0u; }
__device__ __forceinline__ uint32_t task_base(uint32_t buf) { return buf ? kRecBytes : 0u; }
constexpr uint32_t kRR = kBMaxRank * kBMaxRank;
constexpr uint32_t kWarps = kBThreads / 32;
static_assert(4 * kRR * 8 <= kTaskSmem, "inverse: four matrices");
static_assert(kRR * 8 + kWarps * kBMaxRank * 12 <= kTaskSmem, "solve: fragments of W, column partials");
static_assert((kWarps * 8 * kRowPad + 4 * 20 * 32) * 8 <= kTaskSmem, "gram: row tiles, partial tiles");

// D += A B for one 8x8x4 FP64 tensor-core tile (mma.sync m8n8k4): lane l holds
// A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4)], D[l/4][2(l%4)+1].
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// One tile of a mode-m schedule whose n records are in shared memory: a group
// of 2^glog lanes x CPL columns per nonzero (the group size is chosen from the
// tensor's rank at run time, so a kernel holds one tile variant).  The records
// are in output-row order, so a group walks a contiguous slice and adds a row
// into M once per run.  A record of a bad coordinate adds nothing and comes
// last (its output row is kNone).
constexpr uint32_t kNone = 0xFFFFFFFFu;

template <int CPL, class FT>
__device__ void tile_task(const BatchPlan *__restrict__ gp, const uint4 *s_rec, uint32_t n)
{
    constexpr int U = 4;  // nonzeros in flight per group
    const uint32_t tid = threadIdx.x;
    const uint32_t R = gp->R, stride = gp->stride;
    const FT *mat0, *mat1;
    if constexpr (sizeof(FT) == 4) {
        mat0 = reinterpret_cast<const FT *>(gp->A32[0]);
        mat1 = reinterpret_cast<const FT *>(gp->A32[1]);
    } else {
        mat0 = reinterpret_cast<const FT *>(gp->A16[0]);
        mat1 = reinterpret_cast<const FT *>(gp->A16[1]);
    }
    float *out = gp->M;
    const uint32_t need = (R + CPL - 1) / CPL;
    const uint32_t glog = need <= 1 ? 0u : 32u - __clz(need - 1);
    const uint32_t g = tid >> glog, lane = tid & ((1u << glog) - 1u);
    const uint32_t kGroups = (uint32_t)kBThreads >> glog;
    const uint32_t col = lane * CPL;
    const bool active = col < R;
    // lanes beyond the rank read column 0 and write nothing
    mat0 += active ? col : 0u;
    mat1 += active ? col : 0u;
    // an odd slice length puts the groups' first nonzeros on different banks
    const uint32_t per = ((n + kGroups - 1) >> (8u - glog)) | 1u;
    const uint32_t j0 = min(g * per, n), j1 = min(j0 + per, n);
    float acc[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) acc[c] = 0.f;
    uint32_t cur = j0 < j1 ? s_rec[j0].x : kNone;
    auto row_change = [&](uint32_t row) {
        if (cur != kNone && active) {
#pragma unroll
            for (int q = 0; q < CPL / 4; ++q)
                if (col + 4 * q < R)
                    red_add4(out + (size_t)cur * stride + col + 4 * q,
                             mask4(make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]),
                                   col + 4 * q, R));
        }
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[c] = 0.f;
        cur = row;
    };
    auto add = [&](const Cols<CPL, FT> &f0, const Cols<CPL, FT> &f1, float v) {
        const float2 vv = make_float2(v, v);
#pragma unroll
        for (int c = 0; c < CPL; c += 2) {
            float2 p;
            if constexpr (sizeof(FT) == 2) p = bf16x2_mul(f0.w[c >> 1], f1.w[c >> 1]);
            else p = __fmul2_rn(make_float2(f0.at(c), f0.at(c + 1)), make_float2(f1.at(c), f1.at(c + 1)));
            const float2 r = __ffma2_rn(p, vv, make_float2(acc[c], acc[c + 1]));
            acc[c] = r.x;
            acc[c + 1] = r.y;
        }
    };
    uint32_t j = j0;
    for (; j + U <= j1; j += U) {
        uint4 r[U];
        Cols<CPL, FT> f0[U], f1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            r[u] = s_rec[j + u];
            f0[u].load(mat0 + (size_t)r[u].y * stride, 0);
            f1[u].load(mat1 + (size_t)r[u].z * stride, 0);
        }
        // every group of the warp still in full batches continues its row
        // (the rows of a slice never decrease): no row bookkeeping
        if (__all_sync(__activemask(), r[U - 1].x == cur)) {
#pragma unroll
            for (int u = 0; u < U; ++u) add(f0[u], f1[u], __uint_as_float(r[u].w));
            continue;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (r[u].x != cur) row_change(r[u].x);
            add(f0[u], f1[u], __uint_as_float(r[u].w));
        }
    }
    for (; j < j1; ++j) {
        const uint4 r = s_rec[j];
        Cols<CPL, FT> f0, f1;
        f0.load(mat0 + (size_t)r.y * stride, 0);
        f1.load(mat1 + (size_t)r.z * stride, 0);
        if (r.x != cur) row_change(r.x);
        add(f0, f1, __uint_as_float(r.w));
    }
    row_change(kNone);
}

// Block-wide sum of one double per thread; the result is returned to every
// thread.  red holds kBThreads/32 + 1 doubles.
__device__ double block_sum(double x, double *red)
{
    const uint32_t tid = threadIdx.x;
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = x;
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int w = 0; w < kBThreads / 32; ++w) s += red[w];
        red[kBThreads / 32] = s;
    }
    __syncthreads();
    return red[kBThreads / 32];
}

// W of (b, m) from the other modes' Grams.
__device__ void inverse_task(const BatchTensor *__restrict__ gt, uint32_t m, double *Wout, unsigned char *sm)
{
    double *V = reinterpret_cast<double *>(sm), *L = V + kRR, *Li = L + kRR, *W = Li + kRR;
    const uint32_t R = gt->R, RR = R * R;
    const double *Ga = gt->G + (size_t)((m + 1) % 3) * RR, *Gb = gt->G + (size_t)((m + 2) % 3) * RR;
    for (uint32_t e = threadIdx.x; e < RR; e += kBThreads) V[e] = __ldcg(Ga + e) * __ldcg(Gb + e);
    __syncthreads();
    spd_inverse(V, L, Li, W, R);
    for (uint32_t e = threadIdx.x; e < RR; e += kBThreads) Wout[e] = W[e];
}

// A = M W for the rows of one chunk, on the FP64 tensor cores (mma.sync
// m8n8k4), one warp per block of 8 rows; lane l is (g, t) = (l/4, l%4).  The
// columns' sums of squares and maxima are added into the accumulators.
__device__ void solve_task(const BatchTensor *__restrict__ gt, uint32_t m, uint32_t chunk, uint32_t chunk_rows,
                           const double *W, BatchAcc *acc, unsigned char *sm)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g8 = lane >> 2, t4 = lane & 3;
    const uint32_t R = gt->R, stride = gt->stride;
    const uint32_t r0 = chunk * chunk_rows, r1 = min(gt->dims[m], r0 + chunk_rows);
    float *A = gt->A[m];
    const float *M = gt->M[m];
    // B operands in fragment order: Wf[kt][nt][lane] = W[4kt + lane%4][8nt + lane/4]
    double *Wf = reinterpret_cast<double *>(sm);
    for (uint32_t e = tid; e < 8 * 4 * 32; e += kBThreads) {
        const uint32_t l = e & 31, nt = (e >> 5) & 3, kt = e >> 7;
        const uint32_t k = 4 * kt + (l & 3), c = 8 * nt + (l >> 2);
        Wf[e] = (k < R && c < R) ? __ldcg(W + k * R + c) : 0.0;
    }
    __syncthreads();
    const uint32_t KT = (R + 3) / 4, NT = (R + 7) / 8;  // k-steps and 8-column tiles (NT * 8 == stride)
    double csq[8];
    float cmx[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        csq[j] = 0.0;
        cmx[j] = 0.f;
    }
    float anext[8];
    auto load_a = [&](uint32_t row0, float (&av)[8]) {
        const uint32_t row = row0 + g8;
#pragma unroll
        for (int kt = 0; kt < 8; ++kt) {
            const uint32_t k = 4 * kt + t4;
            av[kt] = (row < r1 && k < R) ? __ldcg(M + (size_t)row * stride + k) : 0.f;
        }
    };
    uint32_t row0 = r0 + warp * 8;
    load_a(row0, anext);
    for (; row0 < r1; row0 += kWarps * 8) {
        float av[8];
#pragma unroll
        for (int kt = 0; kt < 8; ++kt) av[kt] = anext[kt];
        load_a(row0 + kWarps * 8, anext);
        double c[4][2];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) c[nt][0] = c[nt][1] = 0.0;
#pragma unroll
        for (int kt = 0; kt < 8; ++kt) {
            if (kt < (int)KT) {
                const double a = (double)av[kt];
#pragma unroll
                for (int nt = 0; nt < 4; ++nt)
                    if (nt < (int)NT) dmma(c[nt][0], c[nt][1], a, Wf[(kt * 4 + nt) * 32 + lane]);
            }
        }
        const uint32_t row = row0 + g8;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            if (nt >= (int)NT) break;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t col = 8 * nt + 2 * t4 + i;
                const float v = col < R ? (float)c[nt][i] : 0.f;
                if (row < r1) {
                    A[(size_t)row * stride + col] = v;
                    csq[2 * nt + i] += (double)v * (double)v;
                    cmx[2 * nt + i] = fmaxf(cmx[2 * nt + i], v);
                }
            }
        }
    }
    // the lanes of a column, then the warps (an FP64 atomic in shared memory
    // is a compare-and-swap loop), then one atomic per column
    double *psq = Wf + kRR;
    float *pmx = reinterpret_cast<float *>(psq + kWarps * kBMaxRank);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            csq[j] += __shfl_xor_sync(0xffffffffu, csq[j], o);
            cmx[j] = fmaxf(cmx[j], __shfl_xor_sync(0xffffffffu, cmx[j], o));
        }
        if (g8 == 0) {
            psq[warp * kBMaxRank + 8 * (j >> 1) + 2 * t4 + (j & 1)] = csq[j];
            pmx[warp * kBMaxRank + 8 * (j >> 1) + 2 * t4 + (j & 1)] = cmx[j];
        }
    }
    __syncthreads();
    if (tid < R) {
        double sq = 0.0;
        float mx = 0.f;
        for (uint32_t w = 0; w < kWarps; ++w) {
            sq += psq[w * kBMaxRank + tid];
            mx = fmaxf(mx, pmx[w * kBMaxRank + tid]);
        }
        atomicAdd(&acc->colsq[tid], sq);
        atomicMax(&acc->colmax[tid], __float_as_int(mx));
    }
}

// v / d, given inv = 1 / d in FP64: rounded to FP32 once, from within 2^-51 of
// the quotient, which is the rounded quotient unless it lies that close to the
// middle of two FP32 numbers.
__device__ __forceinline__ float scaled(float v, double inv) { return (float)((double)v * inv); }

// A /= lambda, the BF16 copy and the Gram of one chunk's rows, and its slice of
// the next mode's MTTKRP output zeroed (whose tiles wait for this step).  With
// gram_bf16 (the iterations whose MTTKRPs gather BF16 factors) the Gram is
// formed from the BF16-rounded factor, the values those gathers read, so that
// the next steps' right-hand sides and normal matrices come from the same
// factors.  The warp's 8 scaled rows go through a shared-memory tile, each half
// (4 rows) is one k-step for the tiles (p, q), p <= q, of the symmetric Gram.
// A chunk of 462 rows (mean) took 23.8 us, 9 of them FP32 divisions by lambda
// and 3 loads of M after the last mode; with scaled() and M fetched a block
// ahead it takes 14, and an iteration of 128 tensors 0.72 ms instead of 0.81.
__device__ void gram_task(const BatchTensor *__restrict__ gt, uint32_t b, uint32_t m, uint32_t chunk, uint32_t it,
                          const BatchArgs &a, BatchAcc *acc, unsigned char *sm, bool gram_bf16, double *s_red)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g8 = lane >> 2, t4 = lane & 3;
    const uint32_t R = gt->R, stride = gt->stride, I = gt->dims[m];
    const uint32_t r0 = chunk * a.chunk_rows, r1 = min(I, r0 + a.chunk_rows);
    const uint32_t NT = (R + 7) / 8;
    float *A = gt->A[m];
    const float *M = gt->M[m];
    __nv_bfloat16 *Ab = gt->Ab[m];
    const bool colok = lane < R, last = m == 2;
    // lambda: 2-norm in the first iteration (src/matrix/matrix.c:389-469),
    // max(column max, 1) afterwards (:472-553)
    const float lam = colok ? (it == 0 ? (float)sqrt(__ldcg(&acc->colsq[lane]))
                                       : fmaxf(__int_as_float(__ldcg(&acc->colmax[lane])), 1.f))
                            : 1.f;
    if (chunk == 0 && warp == 0 && colok) gt->lambda[lane] = lam;
    const double inv_lam = 1.0 / (double)lam;
    double inner = 0.0;
    double *tile = reinterpret_cast<double *>(sm) + warp * (8 * kRowPad);
    double gacc[10][2];
#pragma unroll
    for (int j = 0; j < 10; ++j) gacc[j][0] = gacc[j][1] = 0.0;
    float next[8], nextm[8];  // the rows of A, and after the last mode of M, of the warp's next block
    auto fetch = [&](uint32_t row0) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            next[q] = colok && row0 + q < r1 ? __ldcg(A + (size_t)(row0 + q) * stride + lane) : 0.f;
        if (last)
#pragma unroll
            for (int q = 0; q < 8; ++q)
                nextm[q] = colok && row0 + q < r1 ? __ldcg(M + (size_t)(row0 + q) * stride + lane) : 0.f;
    };
    fetch(r0 + warp * 8);
    for (uint32_t row0 = r0 + warp * 8; row0 < r1; row0 += kWarps * 8) {
        float v[8], mm[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            v[q] = next[q];
            mm[q] = nextm[q];
        }
        fetch(row0 + kWarps * 8);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t row = row0 + q;
            if (colok) v[q] = scaled(v[q], inv_lam);
            const __nv_bfloat16 h = __float2bfloat16_rn(colok ? v[q] : 0.f);
            // the value the next MTTKRPs gather (and the fit's model uses)
            const double used = gram_bf16 ? (double)__bfloat162float(h) : (double)v[q];
            if (colok && row < r1) {
                A[(size_t)row * stride + lane] = v[q];
                if (last) inner += (double)lam * used * (double)mm[q];
            }
            if (a.mixed && lane < stride && row < r1) Ab[(size_t)row * stride + lane] = h;
            tile[q * kRowPad + lane] = used;
        }
        __syncwarp();
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            double fr[4];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) fr[nt] = tile[(4 * ks + t4) * kRowPad + 8 * nt + g8];
            int j = 0;
#pragma unroll
            for (int pt = 0; pt < 4; ++pt)
#pragma unroll
                for (int qt = pt; qt < 4; ++qt, ++j)
                    if (qt < (int)NT) dmma(gacc[j][0], gacc[j][1], fr[pt], fr[qt]);
        }
        __syncwarp();
    }
    {
        const uint32_t mn = (m + 1) % 3, chunks = __ldg(&a.plans[3 * b + m].chunks);
        float4 *Mn = reinterpret_cast<float4 *>(gt->M[mn]);
        const size_t n4 = (size_t)gt->dims[mn] * stride / 4;
        for (size_t e = (size_t)chunk * kBThreads + tid; e < n4; e += (size_t)chunks * kBThreads)
            Mn[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // the warps' tiles, half of the warps to the other half at a time
    double *part = reinterpret_cast<double *>(sm) + kWarps * 8 * kRowPad;
    for (uint32_t h = kWarps / 2; h > 0; h >>= 1) {
        double *slot = part + (size_t)(warp < h ? warp : warp - h) * 20 * 32 + lane;
        if (warp >= h && warp < 2 * h) {
#pragma unroll
            for (int j = 0; j < 20; ++j) slot[j * 32] = gacc[j / 2][j & 1];
        }
        __syncthreads();
        if (warp < h) {
#pragma unroll
            for (int j = 0; j < 20; ++j) gacc[j / 2][j & 1] += slot[j * 32];
        }
        __syncthreads();
    }
    // tile (p, q) holds G[8p + g][8q + 2t + i]
    if (warp == 0) {
        int j = 0;
#pragma unroll
        for (int pt = 0; pt < 4; ++pt)
#pragma unroll
            for (int qt = pt; qt < 4; ++qt, ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t r = 8 * pt + g8, c = 8 * qt + 2 * t4 + i;
                    if (r <= c && c < R) atomicAdd(&acc->G[r * kBMaxRank + c], gacc[j][i]);
                }
    }
    if (last) {
        const double all = block_sum(inner, s_red);
        if (tid == 0) atomicAdd(&acc->inner, all);
    }
}

// The end of (b, m)'s dense step, in the CTA whose gram chunk ended last: the
// Gram in full, and after the last mode
// fit = 1 - sqrt(||X||^2 + |lambda^T (G_0 o G_1 o G_2) lambda| - 2 <X, model>) / ||X||
// (src/ktensor/ktensor.c:77-99, with full symmetric Grams).
__device__ void finish_mode(const BatchTensor *__restrict__ gt, uint32_t b, uint32_t m, uint32_t it,
                            const BatchArgs &a, const BatchAcc *acc, double *s_red)
{
    const uint32_t R = gt->R, RR = R * R;
    double *G = gt->G;
    double s = 0.0;
    for (uint32_t e = threadIdx.x; e < RR; e += kBThreads) {
        const uint32_t i = e / R, j = e % R;
        const double g = __ldcg(&acc->G[min(i, j) * kBMaxRank + max(i, j)]);
        G[(size_t)m * RR + e] = g;
        if (m == 2)
            s += __ldcg(G + e) * __ldcg(G + RR + e) * g * (double)__ldcg(gt->lambda + i) * (double)__ldcg(gt->lambda + j);
    }
    if (m != 2) return;
    const double norm_mats = fabs(block_sum(s, s_red));
    if (threadIdx.x == 0) {
        const double nx = *gt->normX2;
        double residual = nx + norm_mats - 2.0 * __ldcg(&acc->inner);
        if (residual > 0.0) residual = sqrt(residual);
        a.fits[(size_t)b * a.niters + it] = 1.0 - residual / sqrt(nx);
    }
}

// One ALS iteration of the batch; CPL columns per lane and factor type FT for
// the MTTKRP gathers (BF16 iterations and FP32 iterations launch different
// instantiations).
template <int CPL, class FT>
__global__ void __launch_bounds__(kBThreads, 2) batch_als_kernel(BatchArgs a)
{
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint64_t mbar[2];
    __shared__ uint2 s_task[2];
    __shared__ uint32_t s_copy[2];  // records of the held task on their way: their count, else 0
    __shared__ bool s_ready[2];     // what the held task waits for was there when it was taken
    __shared__ int s_ok, s_last;
    __shared__ uint32_t *s_done;    // thread 32: the counter the CTA's last task goes into
    __shared__ int s_copies_ok;     // 0 once a tile's bulk copy missed its wait bound
    __shared__ double s_red[kBThreads / 32 + 1];
    const uint32_t tid = threadIdx.x;
    const uint32_t it = *a.iter, B = a.ntensors;
    uint32_t *head = a.ctrl, *tiles_done = a.ctrl + 1, *inv_done = tiles_done + 3 * B, *solve_done = inv_done + 3 * B,
             *gram_done = solve_done + 3 * B, *modes_done = gram_done + 3 * B;
    const uint2 none = make_uint2(kNone, 0u);
    const auto ready = [&](uint32_t pid, uint32_t kind) {
        if (ld_acquire(modes_done + pid / 3) < pid % 3) return false;
        if (kind == kSolve)
            return ld_acquire(inv_done + pid) >= 1u && ld_acquire(tiles_done + pid) >= __ldg(&a.plans[pid].ntiles);
        return kind != kGram || ld_acquire(solve_done + pid) >= __ldg(&a.plans[pid].chunks);
    };
    // thread 0: takes the next task of the queue into slot `buf`, starts the
    // copy of its records and looks whether it may run
    auto claim = [&](uint32_t buf) {
        const uint32_t q = atomicAdd(head, 1u);
        const uint2 task = q < a.ntasks ? __ldg(a.tasks + q) : none;
        s_task[buf] = task;
        s_copy[buf] = 0;
        if (task.x != kNone && (task.x & 3u) == kTile && s_copies_ok) {
            const BatchPlan *gp = a.plans + (task.x >> 2);
            const uint64_t z0 = (uint64_t)task.y * kBTile, left = gp->nnz - z0;
            const uint32_t n = left < (uint64_t)kBTile ? (uint32_t)left : (uint32_t)kBTile;
            s_copy[buf] = n;
            mbar_arrive_expect_tx(&mbar[buf], 16 * n);
            bulk_g2s_ef(sm + rec_base(buf), gp->recs + z0, 16 * n, &mbar[buf]);
        }
        s_ready[buf] = task.x != kNone && ready(task.x >> 2, task.x & 3u);
        __threadfence();
    };
    // thread 32, behind a barrier that ends a task: counts it as done
    auto publish = [&] {
        if (s_done) {
            __threadfence();
            atomicAdd(s_done, 1u);
            s_done = nullptr;
        }
    };
    if (tid == 0) {
        mbar_init(&mbar[0], 1);
        mbar_init(&mbar[1], 1);
        mbar_fence_init();
        s_copies_ok = 1;
        claim(0);
    }
    if (tid == 32) s_done = nullptr;
    uint32_t phase[2] = {0, 0};
    for (uint32_t buf = 0;; buf ^= 1u) {
        __syncthreads();
        const uint2 task = s_task[buf];
        // Beside the task itself one warp counts the last one as done and
        // another takes the next one and, where that is settled, sees that it
        // may run.  Between the tasks, by one thread before the others went
        // on, this took 3.7 us of a tile's 9.9 (128 tensors: 0.85 ms an
        // iteration; 0.81 so).
        if (tid == 32) publish();
        if (task.x == kNone) break;  // nothing follows the end of the queue: no copy is in flight
        const uint32_t pid = task.x >> 2, kind = task.x & 3u, b = pid / 3, m = pid % 3;
        bool ok = s_ready[buf];
        if (tid == 0) {
            claim(buf ^ 1u);
            if (!ok) {
                bool now = wait_at_least(modes_done + b, m, a.err, a.wait_ns);
                if (kind == kSolve) {
                    if (now) now = wait_at_least(inv_done + pid, 1u, a.err, a.wait_ns);
                    if (now) now = wait_at_least(tiles_done + pid, __ldg(&a.plans[pid].ntiles), a.err, a.wait_ns);
                }
                if (kind == kGram && now)
                    now = wait_at_least(solve_done + pid, __ldg(&a.plans[pid].chunks), a.err, a.wait_ns);
                __threadfence();
                if (!now) atomicOr(a.err, kErrWait);
                s_ok = now;
            }
        }
        if (!s_ready[buf]) {
            __syncthreads();
            ok = s_ok;
        }
        const uint32_t n = s_copy[buf];
        if (n) {
            // the records, even if the task is not run: the next task in this
            // buffer must not find them still on their way.  After a miss the
            // CTA waits once more and issues no further copy.
            const bool here = mbar_wait_bounded(&mbar[buf], phase[buf]);
            if (!__syncthreads_and(here)) {
                if (tid == 0) {
                    atomicOr(a.err, kErrCopy);
                    s_copies_ok = 0;
                    mbar_wait_bounded(&mbar[buf], phase[buf]);
                }
                ok = false;
            }
            phase[buf] ^= 1u;
        }
        BatchAcc *acc = a.acc + pid;
        double *W = a.W + (size_t)pid * kRR;
        unsigned char *mine = sm + task_base(buf);
        if (ok) {
            if (kind == kTile) {
                if (n) tile_task<CPL, FT>(a.plans + pid, reinterpret_cast<const uint4 *>(sm + rec_base(buf)), n);
            } else if (kind == kInverse) {
                inverse_task(a.tens + b, m, W, mine);
            } else if (kind == kSolve) {
                solve_task(a.tens + b, m, task.y, a.chunk_rows, W, acc, mine);
            } else {
                gram_task(a.tens + b, b, m, task.y, it, a, acc, mine, sizeof(FT) == 2, s_red);
            }
        }
        // shared memory written by this task may next be filled by bulk copies
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (kind != kGram) {
            if (tid == 32) s_done = (kind == kTile ? tiles_done : kind == kInverse ? inv_done : solve_done) + pid;
            continue;
        }
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            s_last = atomicAdd(gram_done + pid, 1u) + 1 == __ldg(&a.plans[pid].chunks);
            __threadfence();
        }
        __syncthreads();
        if (s_last) {
            if (ok) finish_mode(a.tens + b, b, m, it, a, acc, s_red);
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                atomicAdd(modes_done + b, 1u);
            }
        }
    }
}

__global__ void bump_kernel(uint32_t *iter) { *iter += 1; }

// Grams of the current factors and their BF16 copies; one CTA per (tensor,
// mode).  With round_bf16 the Grams are of the BF16-rounded factors (the
// values the BF16 iterations gather, see dense_task).  Tensor-core tiles as in
// dense_task: both operands of a tile product are the same fragment, so a lane
// loads each element it needs itself.  (Rows broadcast column by column
// through shuffles took 1.18 ms for 128 tensors of up to 5,000 rows a mode;
// this takes 0.08.)
__global__ void __launch_bounds__(kBThreads) batch_init_kernel(const BatchTensor *tens, int mixed, int round_bf16)
{
    __shared__ double part[kBThreads / 64][20][32];
    const BatchTensor *gt = tens + blockIdx.x / 3;
    const uint32_t m = blockIdx.x % 3;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g8 = lane >> 2, t4 = lane & 3;
    const uint32_t R = gt->R, stride = gt->stride, RR = R * R, I = gt->dims[m];
    const float *A = gt->A[m];
    __nv_bfloat16 *Ab = gt->Ab[m];
    double acc[10][2];
#pragma unroll
    for (int j = 0; j < 10; ++j) acc[j][0] = acc[j][1] = 0.0;
    for (uint32_t i0 = warp * 16; i0 < I; i0 += kBThreads / 32 * 16) {
        float v[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const uint32_t row = i0 + 4 * k + t4, col = 8 * n + g8;
                v[k][n] = row < I && col < R ? A[(size_t)row * stride + col] : 0.f;
            }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double fr[4];
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const uint32_t row = i0 + 4 * k + t4, col = 8 * n + g8;
                const __nv_bfloat16 h = __float2bfloat16_rn(v[k][n]);
                if (mixed && row < I && col < stride) Ab[(size_t)row * stride + col] = h;
                fr[n] = round_bf16 ? (double)__bfloat162float(h) : (double)v[k][n];
            }
            int j = 0;
#pragma unroll
            for (int pt = 0; pt < 4; ++pt)
#pragma unroll
                for (int qt = pt; qt < 4; ++qt, ++j) dmma(acc[j][0], acc[j][1], fr[pt], fr[qt]);
        }
    }
    for (uint32_t h = kBThreads / 64; h > 0; h >>= 1) {
        __syncthreads();
        if (warp >= h && warp < 2 * h) {
#pragma unroll
            for (int j = 0; j < 20; ++j) part[warp - h][j][lane] = acc[j / 2][j & 1];
        }
        __syncthreads();
        if (warp < h) {
#pragma unroll
            for (int j = 0; j < 20; ++j) acc[j / 2][j & 1] += part[warp][j][lane];
        }
    }
    if (warp == 0) {
        double *G = gt->G + (size_t)m * RR;
        int j = 0;
#pragma unroll
        for (int pt = 0; pt < 4; ++pt)
#pragma unroll
            for (int qt = pt; qt < 4; ++qt, ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t r = 8 * pt + g8, c = 8 * qt + 2 * t4 + i;
                    if (r < R && c < R) {
                        G[r * R + c] = acc[j][i];
                        if (pt != qt) G[c * R + r] = acc[j][i];
                    }
                }
    }
}

// ||X||^2 of every tensor; one CTA per tensor.
__global__ void batch_norm_kernel(const float *const *vals, const uint64_t *nnz, double *out)
{
    __shared__ double red[kBThreads / 32 + 1];
    const float *v = vals[blockIdx.x];
    const uint64_t n = nnz[blockIdx.x];
    double s = 0.0;
    for (uint64_t i = threadIdx.x; i < n; i += kBThreads) s += (double)v[i] * (double)v[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// Column sums of squares of the FP32 factors into the Grams' diagonals, for a
// last iteration whose Grams are of the BF16-rounded factors.
__global__ void __launch_bounds__(kBThreads) batch_colsq_kernel(const BatchTensor *tens)
{
    __shared__ double part[kBThreads / 32][kBMaxRank];
    const BatchTensor *gt = tens + blockIdx.x / 3;
    const uint32_t m = blockIdx.x % 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t R = gt->R, stride = gt->stride, I = gt->dims[m];
    const float *A = gt->A[m];
    double sq = 0.0;
#pragma unroll 8
    for (uint32_t i = warp; i < I; i += kBThreads / 32) {
        const double v = lane < R ? A[(size_t)i * stride + lane] : 0.f;
        sq += v * v;
    }
    part[warp][lane] = sq;
    __syncthreads();
    if (threadIdx.x < R) {
        double s = 0.0;
        for (int w = 0; w < kBThreads / 32; ++w) s += part[w][threadIdx.x];
        gt->G[((size_t)m * R + threadIdx.x) * R + threadIdx.x] = s;
    }
}

struct CopyItem {
    const float *src;
    float *dst;
    uint64_t n;  // floats
};

// The result (src/matrix/matrix.c:556-572): the columns of every factor divided
// by their norms -- the square roots of the Grams' diagonals -- on their way to
// the caller, and lambda multiplied by them.  items: the 3 factors of every
// tensor, then every lambda.  blockIdx.x: factor, blockIdx.y: part of its rows.
// (One CTA per tensor, its modes and the norms one after another, then a copy:
// 1.48 + 0.09 ms for 128 tensors; this takes 0.08.)
constexpr uint32_t kOutParts = 8;
__global__ void __launch_bounds__(kBThreads) batch_out_kernel(const BatchTensor *tens, const CopyItem *items,
                                                              uint32_t B)
{
    __shared__ float s_norm[kBMaxRank];
    const uint32_t b = blockIdx.x / 3, m = blockIdx.x % 3, tid = threadIdx.x;
    const BatchTensor *gt = tens + b;
    const uint32_t R = gt->R, stride = gt->stride;
    if (tid < kBMaxRank) s_norm[tid] = tid < R ? (float)sqrt(gt->G[((size_t)m * R + tid) * R + tid]) : 1.f;
    if (m == 0 && blockIdx.y == 0 && tid < R) {
        float l = gt->lambda[tid];
        for (uint32_t k = 0; k < 3; ++k) l *= (float)sqrt(gt->G[((size_t)k * R + tid) * R + tid]);
        items[3 * B + b].dst[tid] = l;
    }
    __syncthreads();
    const CopyItem c = items[blockIdx.x];  // rows of `stride` floats, 16-byte aligned at both ends
    const float4 *src = reinterpret_cast<const float4 *>(c.src);
    float4 *dst = reinterpret_cast<float4 *>(c.dst);
    const uint32_t q = stride / 4;
    for (uint64_t e = (uint64_t)blockIdx.y * kBThreads + tid; e < c.n / 4; e += (uint64_t)kOutParts * kBThreads) {
        const uint32_t col = (uint32_t)(e % q) * 4;
        float4 v = src[e];
        v.x /= s_norm[col];
        v.y /= s_norm[col + 1];
        v.z /= s_norm[col + 2];
        v.w /= s_norm[col + 3];
        dst[e] = v;
    }
}

// blockIdx.x: item, blockIdx.y: part of it.  The items are factors: multiples
// of 8 floats, 16-byte aligned at both ends.
__global__ void __launch_bounds__(kBThreads) batch_copy_kernel(const CopyItem *items)
{
    const CopyItem c = items[blockIdx.x];
    const float4 *s = reinterpret_cast<const float4 *>(c.src);
    float4 *d = reinterpret_cast<float4 *>(c.dst);
    for (uint64_t i = (uint64_t)blockIdx.y * kBThreads + threadIdx.x; i < c.n / 4; i += (uint64_t)kOutParts * kBThreads)
        d[i] = s[i];
}

// Fills the factor arena with values in [0.1, 1.1) from a hash (used to time
// autotuning candidates on a well-conditioned problem).
__global__ void batch_fill_kernel(float *A, uint64_t n)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t x = i * 0x9E3779B97F4A7C15ull;
        x ^= x >> 31;
        x *= 0xBF58476D1CE4E5B9ull;
        x ^= x >> 29;
        A[i] = 0.1f + (float)(x >> 40) * (1.0f / 16777216.0f);
    }
}

}  // namespace pti

struct ptiB200Batch {
    uint32_t B = 0;
    int device = 0;
    cudaStream_t s = nullptr;
    std::vector<uint32_t> dims, R, stride;  // dims: [B][3]
    std::vector<uint64_t> nnz;
    std::vector<std::unique_ptr<ptiB200Tensor>> coo;  // device COO copies (kept while tuning)
    std::vector<std::unique_ptr<ptiB200Tensor>> hic;  // HiCOO tensors with their per-mode schedules
    int sb = 7, cpl = 4;
    float tune_ms = 0.f, setup_ms = 0.f;
    std::vector<size_t> off;   // element offset of factor (b, m) in the arenas
    std::vector<size_t> goff;  // Gram offset (doubles) of tensor b
    std::vector<size_t> loff;  // lambda offset (floats) of tensor b
    size_t elems = 0;
    pti::DevBuf A, Ab, M, G, W, acc, lam, norm2, ctrl, misc, plans, tens, tasks, copies;
    uint32_t ntasks = 0, chunk_rows = pti::kMinChunkRows;
};

namespace pti {
namespace {

const char *kMod = "B200 Batched CPD-ALS";

int batch_build_plans(ptiB200Batch *bt, int sb)
{
    cudaStream_t s = bt->s;
    const uint32_t B = bt->B;
    for (uint32_t b = 0; b < B; ++b) {
        bt->hic[b].reset();
        ptiB200Tensor *h = nullptr;
        PTI_TRY(ptiB200ConvertToHiCOO(&h, bt->coo[b].get(), (ptiElementIndex)sb, (ptiElementIndex)sb,
                                      (ptiElementIndex)sb, nullptr, nullptr, s));
        bt->hic[b].reset(h);
        for (uint32_t m = 0; m < 3; ++m) PTI_TRY(prepare_mode(h, m, s));
    }
    // Chunks of the dense steps: about two and a half for each of the two CTAs
    // of an SM.  Fewer leave SMs idle in a small batch, more pay for their
    // fragments of W and their reductions: 20 tensors 0.209 / 0.176 / 0.155 ms
    // an iteration with chunks of 512 / 256 / 128 rows, 128 tensors 0.828 /
    // 0.871 / 0.990.
    {
        uint64_t rows = 0;
        for (uint32_t d : bt->dims) rows += d;
        bt->chunk_rows = kMinChunkRows;
        while (bt->chunk_rows < 1024 && rows / 3 > (uint64_t)bt->chunk_rows * 5 * sm_count()) bt->chunk_rows *= 2;
    }
    bt->sb = sb;
    std::vector<BatchPlan> hp(3 * (size_t)B);
    std::vector<uint32_t> ntiles(3 * (size_t)B);
    float *A = bt->A.as<float>();
    auto *Ab = bt->Ab.as<__nv_bfloat16>();
    float *M = bt->M.as<float>();
    for (uint32_t b = 0; b < B; ++b) {
        ptiB200Tensor *h = bt->hic[b].get();
        for (uint32_t m = 0; m < 3; ++m) {
            const HicooModePlan &P = h->hicoo_plan[m];
            BatchPlan p{};
            p.nnz = h->nnz;
            p.recs = P.recs.as<uint4>();
            for (uint32_t k = 0, i = 0; k < 3; ++k) {
                if (k == m) continue;
                p.A32[i] = A + bt->off[3 * b + k];
                p.A16[i] = Ab + bt->off[3 * b + k];
                ++i;
            }
            p.M = M + bt->off[3 * b + m];
            p.ntiles = P.ntiles;
            p.chunks = (bt->dims[3 * b + m] + bt->chunk_rows - 1) / bt->chunk_rows;
            p.R = bt->R[b];
            p.stride = bt->stride[b];
            hp[3 * b + m] = p;
            ntiles[3 * b + m] = P.ntiles;
        }
    }
    PTI_CUDA(bt->plans.alloc(padded(hp.size() * sizeof(BatchPlan)), s), kMod);
    PTI_CUDA(cudaMemcpyAsync(bt->plans.ptr, hp.data(), hp.size() * sizeof(BatchPlan), cudaMemcpyHostToDevice, s),
             kMod);

    // the queue, each wave with the largest tensors first: a tensor whose step
    // ends early starts its next mode early
    std::vector<uint32_t> order(B);
    std::vector<uint2> tasks;
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return bt->nnz[x] > bt->nnz[y]; });
    for (uint32_t m = 0; m < 3; ++m) {
        for (uint32_t b : order) {
            const uint32_t pid = 3 * b + m;
            tasks.push_back(make_uint2(pid << 2 | kInverse, 0u));
            for (uint32_t t = 0; t < ntiles[pid]; ++t) tasks.push_back(make_uint2(pid << 2 | kTile, t));
        }
        for (uint32_t kind : {kSolve, kGram})
            for (uint32_t b : order)
                for (uint32_t c = 0; c < hp[3 * b + m].chunks; ++c)
                    tasks.push_back(make_uint2((3 * b + m) << 2 | kind, c));
    }
    bt->ntasks = (uint32_t)tasks.size();
    PTI_CUDA(bt->tasks.alloc(padded(tasks.size() * sizeof(uint2)), s), kMod);
    PTI_CUDA(cudaMemcpyAsync(bt->tasks.ptr, tasks.data(), tasks.size() * sizeof(uint2), cudaMemcpyHostToDevice, s),
             kMod);
    PTI_CUDA(cudaStreamSynchronize(s), kMod);
    return 0;
}

using BatchKernel = void (*)(BatchArgs);

// 8 columns per lane is one 16-byte load of BF16; FP32 iterations always use
// 4 columns (one 16-byte load) per lane.
BatchKernel batch_kernel(int cpl, bool bf16)
{
    if (!bf16) return batch_als_kernel<4, float>;
    return cpl == 8 ? batch_als_kernel<8, __nv_bfloat16> : batch_als_kernel<4, __nv_bfloat16>;
}

// Grid of the persistent kernel: as many CTAs as fit on the GPU at once, at
// most one per task.
int batch_grid(const ptiB200Batch *bt, BatchKernel k, uint32_t *grid)
{
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        for (int cpl : {4, 8})
            for (bool bf16 : {false, true}) {
                const cudaError_t e = cudaFuncSetAttribute(batch_kernel(cpl, bf16),
                                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                           (int)kBatchSmem);
                if (e != cudaSuccess) attr_err = e;
            }
    });
    PTI_CUDA(attr_err, kMod);
    int per_sm = 0;
    PTI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kBThreads, kBatchSmem), kMod);
    PTI_CHECK(per_sm >= 1, PTIERR_CUDA_ERROR, kMod, "batched kernel does not fit on an SM");
    *grid = (uint32_t)std::min<uint64_t>((uint64_t)per_sm * sm_count(), bt->ntasks);
    return 0;
}

// Captures one iteration (counter and accumulator reset, persistent kernel,
// iteration bump).
int batch_capture(ptiB200Batch *bt, const BatchArgs &a, BatchKernel k, cudaGraphExec_t *exec)
{
    cudaStream_t s = bt->s;
    uint32_t grid = 0;
    PTI_TRY(batch_grid(bt, k, &grid));
    cudaGraph_t graph = nullptr;
    PTI_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), kMod);
    cudaMemsetAsync(bt->ctrl.ptr, 0, ctrl_words(bt->B) * 4, s);
    cudaMemsetAsync(bt->acc.ptr, 0, 3 * (size_t)bt->B * sizeof(BatchAcc), s);
    k<<<grid, kBThreads, kBatchSmem, s>>>(a);
    bump_kernel<<<1, 1, 0, s>>>(const_cast<uint32_t *>(a.iter));
    PTI_CUDA(cudaStreamEndCapture(s, &graph), kMod);
    const cudaError_t inst = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    PTI_CUDA(inst, kMod);
    return 0;
}

// Runs `niters` ALS iterations from the factors in the arena (Grams and BF16
// copies already initialised): the BF16 iterations, then the FP32 ones, each
// phase a replay of its own captured graph.  fits (device, B x niters)
// receives the fits.  *ms: device time per iteration.
int batch_iterate(ptiB200Batch *bt, uint32_t niters, int mixed, uint32_t fp32_sweeps, int cpl, double *fits,
                  float *ms)
{
    cudaStream_t s = bt->s;
    uint32_t *misc = bt->misc.as<uint32_t>();  // [0] iteration, [1] error word
    PTI_CUDA(cudaMemsetAsync(misc, 0, 8, s), kMod);
    BatchArgs a{};
    a.tasks = bt->tasks.as<uint2>();
    a.plans = bt->plans.as<BatchPlan>();
    a.tens = bt->tens.as<BatchTensor>();
    a.acc = bt->acc.as<BatchAcc>();
    a.W = bt->W.as<double>();
    a.ctrl = bt->ctrl.as<uint32_t>();
    a.iter = misc;
    a.fits = fits;
    a.err = misc + 1;
    a.ntasks = bt->ntasks;
    a.ntensors = bt->B;
    a.niters = niters;
    a.fp32_sweeps = fp32_sweeps;
    a.cpl = (uint32_t)cpl;
    a.chunk_rows = bt->chunk_rows;
    a.mixed = mixed;
    a.wait_ns = kWaitNs;
    const uint32_t n16 = mixed && niters > fp32_sweeps ? niters - fp32_sweeps : 0, n32 = niters - n16;
    cudaGraphExec_t g16 = nullptr, g32 = nullptr;
    int r = 0;
    if (n16) r = batch_capture(bt, a, batch_kernel(cpl, true), &g16);
    if (!r && n32) r = batch_capture(bt, a, batch_kernel(cpl, false), &g32);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t lerr = cudaSuccess;
    float t = 0.f;
    if (!r) {
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        cudaEventRecord(e0, s);
        for (uint32_t i = 0; i < n16 && lerr == cudaSuccess; ++i) lerr = cudaGraphLaunch(g16, s);
        if (n16 && n32 && lerr == cudaSuccess) {  // the FP32 sweeps start from Grams of the FP32 factors
            batch_init_kernel<<<3 * bt->B, kBThreads, 0, s>>>(bt->tens.as<BatchTensor>(), mixed, 0);
            lerr = cudaGetLastError();
        }
        for (uint32_t i = 0; i < n32 && lerr == cudaSuccess; ++i) lerr = cudaGraphLaunch(g32, s);
        cudaEventRecord(e1, s);
        const cudaError_t serr = cudaStreamSynchronize(s);
        if (lerr == cudaSuccess) lerr = serr;
        cudaEventElapsedTime(&t, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
    if (g16) cudaGraphExecDestroy(g16);
    if (g32) cudaGraphExecDestroy(g32);
    if (r) return r;
    PTI_CUDA(lerr, kMod);
    if (ms) *ms = t / (float)niters;
    uint32_t err = 0;
    PTI_CUDA(cudaMemcpy(&err, misc + 1, 4, cudaMemcpyDeviceToHost), kMod);
    PTI_CHECK(!(err & kErrRange), PTIERR_VALUE_ERROR, kMod, "tensor coordinate out of range");
    PTI_CHECK(err == 0, PTIERR_CUDA_ERROR, kMod, "a work-queue or copy wait timed out");
    return 0;
}

// round_bf16: the first iterations gather BF16 factors (their Grams are of
// the rounded values)
int batch_init_factors(ptiB200Batch *bt, int mixed, int round_bf16)
{
    cudaStream_t s = bt->s;
    PTI_CUDA(cudaMemsetAsync(bt->M.ptr, 0, bt->elems * 4, s), kMod);
    batch_init_kernel<<<3 * bt->B, kBThreads, 0, s>>>(bt->tens.as<BatchTensor>(), mixed, round_bf16);
    PTI_CUDA(cudaGetLastError(), kMod);
    return 0;
}

struct TuneKey {
    uint32_t B;
    uint64_t nnz_sum, dims_sum, rank_sum;
    int device;
    bool operator<(const TuneKey &o) const
    {
        return std::tie(B, nnz_sum, dims_sum, rank_sum, device) <
               std::tie(o.B, o.nnz_sum, o.dims_sum, o.rank_sum, o.device);
    }
};
std::mutex g_tune_mu;
std::map<TuneKey, std::pair<int, int>> g_tuned;

}  // namespace
}  // namespace pti

extern "C" {

int ptiB200BatchCreate(ptiB200Batch **out, ptiIndex ntensors, const ptiIndex *ndims, const ptiNnzIndex *nnz,
                       const ptiIndex *const *dev_inds, const ptiValue *const *dev_vals, const ptiIndex *ranks,
                       int tune, void *stream)
{
    using namespace pti;
    PTI_CHECK(out && ndims && nnz && dev_inds && dev_vals && ranks, PTIERR_VALUE_ERROR, kMod, "null argument");
    PTI_CHECK(ntensors >= 1 && ntensors <= (1u << 24), PTIERR_VALUE_ERROR, kMod, "ntensors must be in [1, 2^24]");
    for (uint32_t b = 0; b < ntensors; ++b) {
        PTI_CHECK(nnz[b] >= 1 && nnz[b] < 0xFFFFFFFFull, PTIERR_VALUE_ERROR, kMod,
                  "every tensor needs between 1 and 2^32-2 nonzeros");
        PTI_CHECK(ranks[b] >= 1 && ranks[b] <= (uint32_t)kBMaxRank, PTIERR_VALUE_ERROR, kMod,
                  "ranks must be in [1, 32]");
        for (uint32_t m = 0; m < 3; ++m)
            PTI_CHECK(ndims[3 * b + m] >= 1, PTIERR_VALUE_ERROR, kMod, "empty mode");
        PTI_CHECK(dev_vals[b] && dev_inds[3 * b] && dev_inds[3 * b + 1] && dev_inds[3 * b + 2], PTIERR_VALUE_ERROR,
                  kMod, "null tensor array");
    }
    configure_pool_once();
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    auto bt = std::make_unique<ptiB200Batch>();
    cudaGetDevice(&bt->device);
    bt->s = sync_stream();
    cudaStream_t s = bt->s;
    {   // order after the caller's stream
        cudaEvent_t ev;
        PTI_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), kMod);
        cudaEventRecord(ev, static_cast<cudaStream_t>(stream));
        cudaStreamWaitEvent(s, ev, 0);
        cudaEventDestroy(ev);
    }
    cudaEventRecord(t0, s);
    const uint32_t B = ntensors;
    bt->B = B;
    bt->dims.assign(ndims, ndims + 3 * (size_t)B);
    bt->nnz.assign(nnz, nnz + B);
    bt->R.resize(B);
    bt->stride.resize(B);
    bt->coo.resize(B);
    bt->hic.resize(B);
    bt->off.resize(3 * (size_t)B);
    bt->goff.resize(B);
    bt->loff.resize(B);
    size_t elems = 0, gel = 0, lel = 0;
    for (uint32_t b = 0; b < B; ++b) {
        bt->R[b] = ranks[b];
        bt->stride[b] = ((ranks[b] + 7) / 8) * 8;
        for (uint32_t m = 0; m < 3; ++m) {
            bt->off[3 * b + m] = elems;
            elems += (size_t)bt->dims[3 * b + m] * bt->stride[b];
        }
        bt->goff[b] = gel;
        gel += 3 * (size_t)ranks[b] * ranks[b];
        bt->loff[b] = lel;
        lel += ((ranks[b] + 3) / 4) * 4;
    }
    bt->elems = elems;
    for (uint32_t b = 0; b < B; ++b) {
        ptiB200Tensor *t = nullptr;
        PTI_TRY(ptiB200TensorFromDeviceCOO(&t, 3, ndims + 3 * (size_t)b, nnz[b], dev_inds + 3 * (size_t)b,
                                           dev_vals[b], s));
        bt->coo[b].reset(t);
    }
    PTI_CUDA(bt->A.alloc(padded(elems * 4), s), kMod);
    PTI_CUDA(bt->Ab.alloc(padded(elems * 2), s), kMod);
    PTI_CUDA(bt->M.alloc(padded(elems * 4), s), kMod);
    PTI_CUDA(bt->G.alloc(padded(gel * 8), s), kMod);
    PTI_CUDA(bt->lam.alloc(padded(lel * 4), s), kMod);
    PTI_CUDA(bt->norm2.alloc(padded((size_t)B * 8), s), kMod);
    PTI_CUDA(bt->W.alloc(padded(3 * (size_t)B * kRR * 8), s), kMod);
    PTI_CUDA(bt->acc.alloc(padded(3 * (size_t)B * sizeof(BatchAcc)), s), kMod);
    PTI_CUDA(bt->ctrl.alloc(padded(ctrl_words(B) * 4), s), kMod);
    PTI_CUDA(bt->misc.alloc(64, s), kMod);
    {
        std::vector<BatchTensor> ht(B);
        for (uint32_t b = 0; b < B; ++b) {
            BatchTensor &T = ht[b];
            for (uint32_t m = 0; m < 3; ++m) {
                T.A[m] = bt->A.as<float>() + bt->off[3 * b + m];
                T.Ab[m] = bt->Ab.as<__nv_bfloat16>() + bt->off[3 * b + m];
                T.M[m] = bt->M.as<float>() + bt->off[3 * b + m];
                T.dims[m] = bt->dims[3 * b + m];
            }
            T.G = bt->G.as<double>() + bt->goff[b];
            T.lambda = bt->lam.as<float>() + bt->loff[b];
            T.normX2 = bt->norm2.as<double>() + b;
            T.R = bt->R[b];
            T.stride = bt->stride[b];
        }
        PTI_CUDA(bt->tens.alloc(padded(B * sizeof(BatchTensor)), s), kMod);
        PTI_CUDA(cudaMemcpyAsync(bt->tens.ptr, ht.data(), B * sizeof(BatchTensor), cudaMemcpyHostToDevice, s), kMod);
        std::vector<const float *> vp(B);
        for (uint32_t b = 0; b < B; ++b) vp[b] = bt->coo[b]->vals.as<float>();
        DevBuf dvp, dnnz;
        PTI_CUDA(dvp.alloc(padded(B * sizeof(void *)), s), kMod);
        PTI_CUDA(dnnz.alloc(padded(B * 8), s), kMod);
        PTI_CUDA(cudaMemcpyAsync(dvp.ptr, vp.data(), B * sizeof(void *), cudaMemcpyHostToDevice, s), kMod);
        PTI_CUDA(cudaMemcpyAsync(dnnz.ptr, bt->nnz.data(), B * 8, cudaMemcpyHostToDevice, s), kMod);
        batch_norm_kernel<<<B, kBThreads, 0, s>>>(dvp.as<const float *>(), dnnz.as<uint64_t>(),
                                                  bt->norm2.as<double>());
        PTI_CUDA(cudaGetLastError(), kMod);
        PTI_CUDA(cudaStreamSynchronize(s), kMod);
    }

    TuneKey key{B, 0, 0, 0, bt->device};
    for (uint32_t b = 0; b < B; ++b) {
        key.nnz_sum += bt->nnz[b];
        key.rank_sum += (uint64_t)bt->R[b] * (b + 1);
        for (uint32_t m = 0; m < 3; ++m) key.dims_sum += (uint64_t)bt->dims[3 * b + m] * (3 * b + m + 1);
    }
    int best_sb = 7, best_cpl = 4;
    bool cached = false;
    // HIPARTI_B200_BATCH_CONFIG="sb_bits,cols_per_lane" fixes the choice
    // (sb_bits in [4, 8], cols_per_lane 4 or 8) and skips the tuner.
    if (const char *env = std::getenv("HIPARTI_B200_BATCH_CONFIG")) {
        int e_sb = 0, e_cpl = 0;
        PTI_CHECK(std::sscanf(env, "%d,%d", &e_sb, &e_cpl) == 2 && e_sb >= 4 && e_sb <= 8 &&
                      (e_cpl == 4 || e_cpl == 8),
                  PTIERR_VALUE_ERROR, kMod, "HIPARTI_B200_BATCH_CONFIG must be \"sb_bits,cols_per_lane\"");
        best_sb = e_sb;
        best_cpl = e_cpl;
        cached = true;
    }
    if (!cached) {
        std::lock_guard<std::mutex> g(g_tune_mu);
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) {
            best_sb = it->second.first;
            best_cpl = it->second.second;
            cached = true;
        }
    }
    if (tune && !cached) {
        // time one BF16 and one FP32 iteration of the whole batch per candidate
        cudaEvent_t u0, u1;
        cudaEventCreate(&u0);
        cudaEventCreate(&u1);
        cudaEventRecord(u0, s);
        DevBuf fits;
        PTI_CUDA(fits.alloc(padded((size_t)B * 2 * 8), s), kMod);
        float best = 3.4e38f;
        const int sbs[] = {7, 6, 5, 4};
        for (int sb : sbs) {
            PTI_TRY(batch_build_plans(bt.get(), sb));
            for (int cpl : {4, 8}) {
                batch_fill_kernel<<<sm_count() * 4, 256, 0, s>>>(bt->A.as<float>(), elems);
                PTI_TRY(batch_init_factors(bt.get(), 1, 1));
                float ms = 0.f;
                PTI_TRY(batch_iterate(bt.get(), 2, 1, 1, cpl, fits.as<double>(), &ms));  // warm-up
                PTI_TRY(batch_iterate(bt.get(), 2, 1, 1, cpl, fits.as<double>(), &ms));
                if (ms < best) {
                    best = ms;
                    best_sb = sb;
                    best_cpl = cpl;
                }
            }
        }
        cudaEventRecord(u1, s);
        cudaEventSynchronize(u1);
        cudaEventElapsedTime(&bt->tune_ms, u0, u1);
        cudaEventDestroy(u0);
        cudaEventDestroy(u1);
        std::lock_guard<std::mutex> g(g_tune_mu);
        g_tuned[key] = {best_sb, best_cpl};
    }
    if (bt->sb != best_sb || !bt->hic[0]) PTI_TRY(batch_build_plans(bt.get(), best_sb));
    bt->cpl = best_cpl;
    for (auto &c : bt->coo) c.reset();
    cudaEventRecord(t1, s);
    PTI_CUDA(cudaEventSynchronize(t1), kMod);
    cudaEventElapsedTime(&bt->setup_ms, t0, t1);
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    *out = bt.release();
    return 0;
}

int ptiB200BatchInfo(const ptiB200Batch *bt, int *sb_bits, int *cols_per_lane, float *tune_ms, float *setup_ms,
                     ptiNnzIndex *ntasks)
{
    PTI_CHECK(bt, PTIERR_VALUE_ERROR, pti::kMod, "null batch");
    if (sb_bits) *sb_bits = bt->sb;
    if (cols_per_lane) *cols_per_lane = bt->cpl;
    if (tune_ms) *tune_ms = bt->tune_ms;
    if (setup_ms) *setup_ms = bt->setup_ms;
    if (ntasks) *ntasks = bt->ntasks;
    return 0;
}

int ptiB200BatchWaitProbe(ptiB200Batch *bt, double wait_seconds)
{
    using namespace pti;
    PTI_CHECK(bt && bt->B >= 1, PTIERR_VALUE_ERROR, kMod, "empty batch");
    PTI_CHECK(wait_seconds > 0.0 && wait_seconds <= 2.0, PTIERR_VALUE_ERROR, kMod,
              "wait bound must be in (0, 2] seconds");
    cudaStream_t s = bt->s;
    // one task: the mode-1 inverse of tensor 0, which waits for the mode-0
    // dense step -- tasks this queue does not hold, so the counter it waits
    // on stays 0 and the wait must give up after its bound
    DevBuf task;
    PTI_CUDA(task.alloc(64, s), kMod);
    const uint2 t = make_uint2(1u << 2 | kInverse, 0u);
    PTI_CUDA(cudaMemcpyAsync(task.ptr, &t, sizeof t, cudaMemcpyHostToDevice, s), kMod);
    uint32_t *misc = bt->misc.as<uint32_t>();
    PTI_CUDA(cudaMemsetAsync(misc, 0, 8, s), kMod);
    PTI_CUDA(cudaMemsetAsync(bt->ctrl.ptr, 0, ctrl_words(bt->B) * 4, s), kMod);
    BatchArgs a{};
    a.tasks = task.as<uint2>();
    a.plans = bt->plans.as<BatchPlan>();
    a.tens = bt->tens.as<BatchTensor>();
    a.acc = bt->acc.as<BatchAcc>();
    a.W = bt->W.as<double>();
    a.ctrl = bt->ctrl.as<uint32_t>();
    a.iter = misc;
    a.fits = nullptr;
    a.err = misc + 1;
    a.ntasks = 1;
    a.ntensors = bt->B;
    a.niters = 1;
    a.cpl = 4;
    a.chunk_rows = bt->chunk_rows;
    a.wait_ns = (uint64_t)(wait_seconds * 1e9);
    uint32_t grid = 0;
    PTI_TRY(batch_grid(bt, batch_kernel(4, false), &grid));
    batch_kernel(4, false)<<<1, kBThreads, kBatchSmem, s>>>(a);
    PTI_CUDA(cudaGetLastError(), kMod);
    PTI_CUDA(cudaStreamSynchronize(s), kMod);
    uint32_t err = 0;
    PTI_CUDA(cudaMemcpy(&err, misc + 1, 4, cudaMemcpyDeviceToHost), kMod);
    PTI_CUDA(cudaMemsetAsync(misc, 0, 8, s), kMod);
    PTI_CHECK(err == 0, PTIERR_CUDA_ERROR, kMod, "a work-queue or copy wait timed out");
    return 0;
}

int ptiB200BatchCpdAls(ptiB200Batch *bt, ptiIndex niters, int precision, ptiIndex fp32_sweeps,
                       float *const *dev_factors, float *const *dev_lambda, double *fits, float *ms_per_iter,
                       void *stream)
{
    using namespace pti;
    PTI_CHECK(bt && dev_factors && dev_lambda, PTIERR_VALUE_ERROR, kMod, "null argument");
    PTI_CHECK(niters >= 1 && niters <= 1000000, PTIERR_VALUE_ERROR, kMod, "niters must be in [1, 10^6]");
    PTI_CHECK(precision == PTI_B200_F32 || precision == PTI_B200_BF16, PTIERR_VALUE_ERROR, kMod, "bad precision");
    const uint32_t B = bt->B;
    for (uint32_t i = 0; i < 3 * B; ++i)
        PTI_CHECK(dev_factors[i] && ((uintptr_t)dev_factors[i] & 15) == 0, PTIERR_VALUE_ERROR, kMod,
                  "factors must be non-null and 16-byte aligned");
    for (uint32_t b = 0; b < B; ++b) PTI_CHECK(dev_lambda[b], PTIERR_VALUE_ERROR, kMod, "null lambda");
    cudaStream_t s = bt->s;
    {
        cudaEvent_t ev;
        PTI_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), kMod);
        cudaEventRecord(ev, static_cast<cudaStream_t>(stream));
        cudaStreamWaitEvent(s, ev, 0);
        cudaEventDestroy(ev);
    }
    const int mixed = precision == PTI_B200_BF16;
    // factors in: caller's arrays -> arena
    std::vector<CopyItem> items(3 * (size_t)B);
    for (uint32_t b = 0; b < B; ++b)
        for (uint32_t m = 0; m < 3; ++m) {
            const size_t n = (size_t)bt->dims[3 * b + m] * bt->stride[b];
            items[3 * b + m] = CopyItem{dev_factors[3 * b + m], bt->A.as<float>() + bt->off[3 * b + m], n};
        }
    PTI_CUDA(bt->copies.alloc(padded(items.size() * sizeof(CopyItem)), s), kMod);
    PTI_CUDA(cudaMemcpyAsync(bt->copies.ptr, items.data(), 3 * (size_t)B * sizeof(CopyItem), cudaMemcpyHostToDevice,
                             s), kMod);
    batch_copy_kernel<<<dim3(3 * B, kOutParts), kBThreads, 0, s>>>(bt->copies.as<CopyItem>());
    PTI_TRY(batch_init_factors(bt, mixed, mixed && niters > fp32_sweeps));
    DevBuf dfits;
    PTI_CUDA(dfits.alloc(padded((size_t)B * niters * 8), s), kMod);
    float ms = 0.f;
    PTI_TRY(batch_iterate(bt, niters, mixed, fp32_sweeps, bt->cpl, dfits.as<double>(), &ms));
    // factors and lambda out, normalised: arena -> caller's arrays
    std::vector<CopyItem> outs(4 * (size_t)B);
    for (uint32_t b = 0; b < B; ++b) {
        for (uint32_t m = 0; m < 3; ++m)
            outs[3 * b + m] = CopyItem{bt->A.as<float>() + bt->off[3 * b + m], dev_factors[3 * b + m], items[3 * b + m].n};
        outs[3 * (size_t)B + b] = CopyItem{bt->lam.as<float>() + bt->loff[b], dev_lambda[b], bt->R[b]};
    }
    DevBuf out_items;
    PTI_CUDA(out_items.alloc(padded(outs.size() * sizeof(CopyItem)), s), kMod);
    PTI_CUDA(cudaMemcpyAsync(out_items.ptr, outs.data(), outs.size() * sizeof(CopyItem), cudaMemcpyHostToDevice, s),
             kMod);
    if (mixed && fp32_sweeps == 0)  // the last Grams are of the BF16-rounded factors
        batch_colsq_kernel<<<3 * B, kBThreads, 0, s>>>(bt->tens.as<BatchTensor>());
    batch_out_kernel<<<dim3(3 * B, kOutParts), kBThreads, 0, s>>>(bt->tens.as<BatchTensor>(), out_items.as<CopyItem>(), B);
    PTI_CUDA(cudaGetLastError(), kMod);
    if (fits) PTI_CUDA(cudaMemcpyAsync(fits, dfits.ptr, (size_t)B * niters * 8, cudaMemcpyDeviceToHost, s), kMod);
    PTI_CUDA(cudaStreamSynchronize(s), kMod);
    if (ms_per_iter) *ms_per_iter = ms;
    return 0;
}

void ptiB200BatchFree(ptiB200Batch *bt)
{
    if (!bt) return;
    cudaStreamSynchronize(bt->s);
    delete bt;
}

}  // extern "C"
