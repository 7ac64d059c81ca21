// sched.cu -- per-mode schedules and the output-privatised MTTKRP kernels.
//
// Problem.  With skewed (power-law) mode sizes a few output rows receive a
// large share of all nonzeros; adding every product straight into global
// memory serialises the atomics of such a row in one L2 slice.
//
// Schedule (built once per tensor and mode, kept in the device handle).
// HiCOO: the blocks are stably re-ordered by their block coordinate in the
// output mode -- the reference's per-mode kernel scheduler (kschr,
// src/sptensor/hicoo/convert.c:378-421) taken down to block granularity --
// and the nonzeros follow their blocks; the nonzeros are then cut into tiles
// of kPlanTile and re-ordered by output row inside each tile, each keeping its
// 8-bit element offsets and the index of its block among the tile's blocks.
// COO: the nonzeros are stably sorted by their output index and packed as
// records {output index, operand indices, value}.
//
// Kernels (one CTA per tile).  The tile is staged into shared memory with
// bulk (TMA) copies.  Its nonzeros are in output-row order, so each thread
// group walks a contiguous slice, gathers the operand rows with 16-byte
// loads, accumulates the rank-R Hadamard products in registers and adds a row
// into global memory once per run of equal rows (16-byte vector atomics); a
// row shared by neighbouring groups is merged in shared memory first, so a hot
// row costs one global add per tile instead of one per nonzero.
#include <mutex>
#include <type_traits>

#include "kutil.cuh"
#include "primitives.cuh"
#include "split.cuh"
#include "tensor.cuh"
#include "tma.cuh"

namespace pti {


// Nonzeros per CTA of the COO kernel: 2048, or what 32 KB hold of the records
// of 8 modes.  (1024 of 8 words fit a fourth CTA on an SM, 505 -> 485 us for the
// four modes of a uniform 4-D tensor of 5M nonzeros at R = 32, but add a hot
// row's parts to the output twice as often, see coo_sched_kernel.)
constexpr uint32_t coo_tile(int words) { return words <= 8 ? 2048u : 8192u / words & ~3u; }
constexpr int kHiTile = kPlanTile; // nonzeros per CTA (HiCOO kernel)
constexpr int kSchedThreads = 256;

uint32_t *err_word(ptiB200Tensor *t);
int ensure_err_word(ptiB200Tensor *t, cudaStream_t s);

struct SchedArgs {
    uint64_t nnz, nb;
    uint32_t R, stride, sb;
    const uint16_t *lblk;       // HiCOO: block of each nonzero within its tile
    const uint32_t *tile_block;
    const uint32_t *out_bind;   // HiCOO: block coords of the output mode; COO: output indices
    const uint8_t *out_eind;
    uint32_t out_dim;
    const uint32_t *in_bind[kMaxModes - 1];  // HiCOO block coords / COO indices of operand modes
    const uint8_t *in_eind[kMaxModes - 1];
    uint32_t in_dim[kMaxModes - 1];
    const void *in_mat[kMaxModes - 1];
    const float *vals;          // COO: substituted values, or null
    const uint32_t *perm;       // COO: where each record's is among them; null: in record order
    float *out;
    uint32_t *err;
    bool cut;                   // COO: CTAs may take less than a tile
    const uint4 *bquad;         // HiCOO 4-D: per block {output, operand 0, 1, 2} block coordinates
    const uint4 *recs;          // HiCOO: decoded records of the schedule (HicooModePlan::recs)
    const float *rvals;         // HiCOO 4-D: their values
};


__device__ __forceinline__ uint32_t round16(uint32_t x) { return (x + 15u) & ~15u; }

// Words per packed nonzero record {output row, operand rows..., value},
// rounded up to 16 bytes.
constexpr int rec_words(int nin) { return (nin + 2 + 3) / 4 * 4; }
template <int NIN>
struct Rec {
    static constexpr int words = rec_words(NIN);
};

// Columns of one operand row held by a lane: CPL consecutive columns, loaded
// with 8- or 16-byte loads (4 FP32 columns = one 16-byte load, 8 FP32 = two,
// 8 BF16 = one, 4 BF16 = one 8-byte load).
template <int CPL, class FT>
struct RowPart {
    static constexpr int kWords = CPL * (int)sizeof(FT) / 4;
    static_assert(kWords == 2 || kWords % 4 == 0, "8- or 16-byte loads");
    uint32_t w[kWords];
    __device__ __forceinline__ void load(const FT *row, uint32_t col)
    {
        const FT *p = row + col;
        if constexpr (kWords == 2) {
            const uint2 r = __ldg(reinterpret_cast<const uint2 *>(p));
            w[0] = r.x;
            w[1] = r.y;
        } else {
#pragma unroll
            for (int q = 0; q < kWords / 4; ++q) {
                const uint4 r = __ldg(reinterpret_cast<const uint4 *>(p) + q);
                w[4 * q] = r.x;
                w[4 * q + 1] = r.y;
                w[4 * q + 2] = r.z;
                w[4 * q + 3] = r.w;
            }
        }
    }
    // 32-bit word i of the loaded columns
    __device__ __forceinline__ uint32_t word(int i) const { return w[i]; }
    // column c (0 <= c < CPL) as FP32
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

// acc[c] += v * prod_k f[k][c] for the CPL columns of a lane, with packed
// FP32x2 arithmetic; BF16 rows multiply their first two factors exactly in
// FP32 without unpacking them.
template <int CPL, class FT, int NIN>
__device__ __forceinline__ void accumulate(float *acc, const RowPart<CPL, FT> (&f)[NIN], float v)
{
    const float2 vv = make_float2(v, v);
#pragma unroll
    for (int c = 0; c < CPL; c += 2) {
        float2 p;
        if constexpr (sizeof(FT) == 2 && NIN >= 2) {
            p = bf16x2_mul(f[0].word(c >> 1), f[1].word(c >> 1));
#pragma unroll
            for (int k = 2; k < NIN; ++k) p = __fmul2_rn(p, make_float2(f[k].at(c), f[k].at(c + 1)));
        } else {
            p = make_float2(f[0].at(c), f[0].at(c + 1));
#pragma unroll
            for (int k = 1; k < NIN; ++k) p = __fmul2_rn(p, make_float2(f[k].at(c), f[k].at(c + 1)));
        }
        const float2 r = __ffma2_rn(p, vv, make_float2(acc[c], acc[c + 1]));
        acc[c] = r.x;
        acc[c + 1] = r.y;
    }
}

constexpr uint32_t kNoRow = 0xFFFFFFFFu;

// Lane groups of G lanes, any G up to 32: 32 / G to a warp.  A warp's lanes
// that make up no group take an index past the groups', where slices are empty.
// Groups of 9, 10 and 6 lanes are used where rounding the lanes of a row up to a
// power of two leaves room for fewer: 3 instead of 2 groups of a warp, or 5
// instead of 4 (launch_r has the rule and what it measured).
template <int G>
struct Groups {
    static constexpr uint32_t per_warp = 32 / G;
    static constexpr uint32_t count = kSchedThreads / 32 * per_warp;
    uint32_t g, lane;
    __device__ __forceinline__ explicit Groups(uint32_t tid)
    {
        const uint32_t l = tid & 31;
        if constexpr ((G & (G - 1)) == 0) {
            g = tid / G;
            lane = tid % G;
        } else {
            const bool idle = l >= per_warp * G;
            g = idle ? kSchedThreads - 1 : (tid >> 5) * per_warp + l / G;
            lane = idle ? 0u : l % G;
        }
    }
};

// Row runs of one thread group.  Products arrive in output-row order; a run
// that ends is added into the output with one vector atomic per 4 columns,
// except the runs a group shares with its neighbours in the CTA: the run that
// continues the previous group's last row is parked in the group's merge slot
// (shared memory), and the run that continues into the next group stays in
// registers until merge(), where the group that started the row adds the
// parked parts and writes the row once.  A row that fills many slices of a
// tile (a hot row of a power-law mode) is so written once per tile instead of
// once per group.  (Writing it once per 8 groups shortens that chain and took
// 2.27 instead of 2.31 ms on 50M Zipf nonzeros, but adds more FP32 parts in
// global memory: 9.9e-7 instead of 5.7e-7 from FP64.)
template <int CPL>
struct RunWriter {
    float acc[CPL];
    uint32_t cur = kNoRow;
    bool in_first = true, first_shared, last_shared, active;
    uint32_t col;
    float *slot;  // this lane's CPL floats of the group's merge slot

    __device__ __forceinline__ RunWriter(bool fs, bool ls, uint32_t col_, bool active_, float *slot_)
        : first_shared(fs), last_shared(ls), active(active_), col(col_), slot(slot_)
    {
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[c] = 0.f;
    }
    __device__ __forceinline__ void flush(const SchedArgs &a)
    {
        if (!active) return;
#pragma unroll
        for (int q = 0; q < CPL / 4; ++q)
            if (col + 4 * q < a.R)
                red_add4(a.out + (size_t)cur * a.stride + col + 4 * q,
                         mask4(make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]),
                               col + 4 * q, a.R));
    }
    __device__ __forceinline__ void park()
    {
#pragma unroll
        for (int c = 0; c < CPL; ++c) slot[c] = acc[c];
    }
    // a product for `row` follows
    __device__ __forceinline__ void start(uint32_t row, const SchedArgs &a)
    {
        if (row == cur) return;
        if (cur != kNoRow) {
            if (in_first && first_shared) park();
            else flush(a);
            in_first = false;
        }
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[c] = 0.f;
        cur = row;
    }
    // after the slice: true if this group owns a row that continues into the
    // next group (merge() after a barrier)
    __device__ __forceinline__ bool finish(const SchedArgs &a)
    {
        if (cur == kNoRow) return false;
        if (in_first && first_shared) {
            park();
            return false;
        }
        if (last_shared) return true;
        flush(a);
        return false;
    }
    // adds the parked parts of the following groups that continue row `cur`
    // and writes the row
    template <int G>
    __device__ __forceinline__ void merge(const SchedArgs &a, const float *slots, const uint32_t *slot_row,
                                          const uint8_t *slot_whole, uint32_t g, uint32_t lane, uint32_t ngroups)
    {
        for (uint32_t h = g + 1; h < ngroups; ++h) {
            if (slot_row[h] != cur) break;
            const float *p = slots + ((size_t)h * G + lane) * CPL;
#pragma unroll
            for (int c = 0; c < CPL; ++c) acc[c] += p[c];
            if (!slot_whole[h]) break;
        }
        flush(a);
    }
};

// True when every record of the batch, in every group of the warp still
// walking, continues its group's current output row: the batch then needs no
// row bookkeeping (what RunWriter::start would do for each record is nothing).
// Deciding for the whole warp keeps its groups on one path.
template <int U>
__device__ __forceinline__ bool same_row_batch(const uint32_t (&orow)[U], uint32_t cur)
{
    bool same = cur != kNoRow;
#pragma unroll
    for (int u = 0; u < U; ++u) same = same && orow[u] == cur;
    return __all_sync(__activemask(), same);
}

// Walks records [j0, j1) (ordered by output row) of a tile whose records are
// s_rec[0, n): gathers the operand rows and accumulates v * prod_k A_k[row_k]
// in registers, one output row run at a time (RunWriter).
template <int G, int CPL, int U, int NIN, class FT>
__device__ __forceinline__ void process_records(const uint32_t *s_rec, uint32_t n, uint32_t j0, uint32_t j1,
                                                uint32_t g, uint32_t lane, const SchedArgs &a, float *s_slots,
                                                uint32_t *s_slot_row, uint8_t *s_slot_whole)
{
    constexpr int RW = Rec<NIN>::words;
    constexpr uint32_t kGroups = Groups<G>::count;
    const uint32_t col = lane * CPL;
    const bool active = col < a.R;
    bool first_shared = false, last_shared = false;
    if (j0 < j1) {
        const uint32_t rf = s_rec[(size_t)j0 * RW], rl = s_rec[(size_t)(j1 - 1) * RW];
        first_shared = j0 > 0 && s_rec[(size_t)(j0 - 1) * RW] == rf;
        last_shared = j1 < n && s_rec[(size_t)j1 * RW] == rl;
        if (lane == 0) {
            s_slot_row[g] = first_shared ? rf : kNoRow;
            s_slot_whole[g] = rf == rl;
        }
    } else if (lane == 0) {
        s_slot_row[g] = kNoRow;
        s_slot_whole[g] = 0;
    }
    RunWriter<CPL> w(first_shared, last_shared, col, active, s_slots + ((size_t)g * G + lane) * CPL);
    const FT *base[NIN];  // this lane's columns of each operand factor
#pragma unroll
    for (int k = 0; k < NIN; ++k) base[k] = static_cast<const FT *>(a.in_mat[k]) + col;
    // full batches of U records without per-record bounds tests, then one
    // partial batch
    auto batch = [&](uint32_t j, auto check) {
        constexpr bool CHECK = decltype(check)::value;
        uint32_t orow[U];
        float val[U];
        RowPart<CPL, FT> f[U][NIN];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            orow[u] = kNoRow;
            if (!CHECK || j + u < j1) {
                uint32_t wd[RW];
#pragma unroll
                for (int q = 0; q < RW; q += 4) {
                    const uint4 r = *reinterpret_cast<const uint4 *>(s_rec + (size_t)(j + u) * RW + q);
                    wd[q] = r.x; wd[q + 1] = r.y; wd[q + 2] = r.z; wd[q + 3] = r.w;
                }
                orow[u] = wd[0];
                val[u] = __uint_as_float(wd[1 + NIN]);
                if (orow[u] != kNoRow && active) {
#pragma unroll
                    for (int k = 0; k < NIN; ++k) f[u][k].load(base[k] + (size_t)wd[1 + k] * a.stride, 0);
                }
            }
        }
        if (same_row_batch<U>(orow, w.cur)) {  // no row bookkeeping
            if (active) {
#pragma unroll
                for (int u = 0; u < U; ++u) accumulate<CPL, FT, NIN>(w.acc, f[u], val[u]);
            }
            return;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (orow[u] == kNoRow) continue;
            w.start(orow[u], a);
            if (active) accumulate<CPL, FT, NIN>(w.acc, f[u], val[u]);
        }
    };
    uint32_t j = j0;
    for (; j + U <= j1; j += U) batch(j, std::false_type{});
    if (j < j1) batch(j, std::true_type{});
    const bool owner = w.finish(a);
    __syncthreads();
    if (owner) w.template merge<G>(a, s_slots, s_slot_row, s_slot_whole, g, lane, kGroups);
}

// Walks records [j0, j1) of a tile whose n records s_rec ({output row,
// operand rows, value or third operand row}) are in output-row order and
// accumulates v * prod_k A_k[row_k] one row run at a time.  Every
// record is walkable: the decode gave a record with a bad coordinate value 0
// and operand offsets 0, and an output row kNoRow only where its own row is
// out of range (such records sort after every valid row), so the rows of a
// slice never decrease and a batch whose last record continues the current
// row lies wholly in that row.  The batch loop is therefore one compare and
// one warp vote per U records; a row change falls to the per-record path.
// Runs shared with neighbouring groups are merged as RunWriter does.
template <int G, int CPL, int U, class FT, int NIN>
__device__ __forceinline__ void walk_rows(const uint4 *s_rec, const float *s_v3, uint32_t n, uint32_t j0,
                                          uint32_t j1, uint32_t g, uint32_t lane, const SchedArgs &a,
                                          float *s_slots, uint32_t *s_slot_row, uint8_t *s_slot_whole)
{
    constexpr uint32_t kGroups = Groups<G>::count;
    const uint32_t col = lane * CPL;
    const bool active = col < a.R;
    bool first_shared = false, last_shared = false;
    uint32_t cur = kNoRow;
    if (j0 < j1) {
        const uint32_t rl = s_rec[j1 - 1].x;
        cur = s_rec[j0].x;
        first_shared = j0 > 0 && s_rec[j0 - 1].x == cur;
        last_shared = j1 < n && s_rec[j1].x == rl;
        if (lane == 0) {
            s_slot_row[g] = first_shared ? cur : kNoRow;
            s_slot_whole[g] = cur == rl;
        }
    } else if (lane == 0) {
        s_slot_row[g] = kNoRow;
        s_slot_whole[g] = 0;
    }
    float *slot = s_slots + ((size_t)g * G + lane) * CPL;
    // inactive lanes (col >= R) read column 0 and never write
    const FT *base[NIN];
#pragma unroll
    for (int k = 0; k < NIN; ++k) base[k] = static_cast<const FT *>(a.in_mat[k]) + (active ? col : 0u);
    const uint32_t stride = a.stride;
    float acc[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) acc[c] = 0.f;
    bool in_first = true;
    auto flush = [&]() {
#pragma unroll
        for (int q = 0; q < CPL / 4; ++q)
            if (col + 4 * q < a.R)
                red_add4(a.out + (size_t)cur * a.stride + col + 4 * q,
                         mask4(make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]),
                               col + 4 * q, a.R));
    };
    // the run of `cur` ends before the slice does
    auto end_run = [&]() {
        if (in_first && first_shared) {
#pragma unroll
            for (int c = 0; c < CPL; ++c) slot[c] = acc[c];
        } else if (cur != kNoRow && active) {
            flush();
        }
        in_first = false;
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[c] = 0.f;
    };
    auto value = [&](const uint4 &r, uint32_t j) {
        return NIN == 3 ? s_v3[j] : __uint_as_float(NIN == 2 ? r.w : r.z);
    };
    uint32_t j = j0;
    for (; j + U <= j1; j += U) {
        uint4 r[U];
        RowPart<CPL, FT> f[U][NIN];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            r[u] = s_rec[j + u];
            const uint32_t rr[3] = {r[u].y, r[u].z, r[u].w};
#pragma unroll
            for (int k = 0; k < NIN; ++k) f[u][k].load(base[k] + (size_t)rr[k] * stride, 0);
        }
        if (__all_sync(__activemask(), r[U - 1].x == cur)) {
#pragma unroll
            for (int u = 0; u < U; ++u) accumulate<CPL, FT, NIN>(acc, f[u], value(r[u], j + u));
            continue;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (r[u].x != cur) {
                end_run();
                cur = r[u].x;
            }
            accumulate<CPL, FT, NIN>(acc, f[u], value(r[u], j + u));
        }
    }
    for (; j < j1; ++j) {
        const uint4 r = s_rec[j];
        const uint32_t rr[3] = {r.y, r.z, r.w};
        RowPart<CPL, FT> f[NIN];
#pragma unroll
        for (int k = 0; k < NIN; ++k) f[k].load(base[k] + (size_t)rr[k] * stride, 0);
        if (r.x != cur) {
            end_run();
            cur = r.x;
        }
        accumulate<CPL, FT, NIN>(acc, f, value(r, j));
    }
    // the slice's last run: parked if it is also the first and shared with the
    // previous group, kept for merging if it continues into the next group
    bool owner = false;
    if (cur != kNoRow) {
        if (in_first && first_shared) {
#pragma unroll
            for (int c = 0; c < CPL; ++c) slot[c] = acc[c];
        } else if (last_shared) {
            owner = true;
        } else if (active) {
            flush();
        }
    }
    __syncthreads();
    if (owner) {
        for (uint32_t h = g + 1; h < kGroups; ++h) {
            if (s_slot_row[h] != cur) break;
            const float *p = s_slots + ((size_t)h * G + lane) * CPL;
#pragma unroll
            for (int c = 0; c < CPL; ++c) acc[c] += p[c];
            if (!s_slot_whole[h]) break;
        }
        if (active) flush();
    }
}

template <int NIN, int CPL>
struct HiSmem {
    // byte offsets inside the dynamic shared memory of hicoo_sched_kernel
    static constexpr uint32_t val = 0;                                  // float[kHiTile]
    static constexpr uint32_t eout = val + 4 * kHiTile;                 // u8[kHiTile]
    static constexpr uint32_t ein = eout + kHiTile;                     // u8[NIN][kHiTile]
    static constexpr uint32_t blk = ein + NIN * kHiTile;                // u16[kHiTile]
    static constexpr uint32_t brow = blk + 2 * kHiTile;                 // u32[kHiTile + 4]
    static constexpr uint32_t bin = brow + 4 * (kHiTile + 4);           // u32[NIN][kHiTile + 4]
    static constexpr uint32_t staged = bin + 4 * NIN * (kHiTile + 4);   // end of the staged tile
    // decoded records, written over the staged arrays once they are read
    static constexpr uint32_t rec = 0;                                  // uint4[kHiTile]
    static constexpr uint32_t rval = rec + 16 * kHiTile;                // float[kHiTile] (4-D only)
    // FP32 rows (CPL 4): the groups' merge slots follow the records, over
    // the staged tile (they are first written during the walk, after the
    // decode), which lets one more CTA share an SM.  BF16 rows (CPL 8) keep
    // them after the tile: their walk is bound by L1 wavefronts, and the
    // extra CTA's shared memory comes out of the L1 that caches the rows.
    static constexpr uint32_t slots =
        CPL == 4 ? rval + (NIN == 3 ? 4 * kHiTile : 0) : staged;  // float[kSchedThreads * CPL]
    static constexpr uint32_t slots_end = slots + 4 * kSchedThreads * CPL;
    static constexpr uint32_t total = staged > slots_end ? staged : slots_end;
    static_assert(slots <= staged, "records must fit over the staged tile");
};

// HiCOO schedule, one CTA per tile of kHiTile nonzeros.  The tile's nonzeros
// (8-bit element offsets, values, block index within the tile) and its blocks'
// coordinates are staged into shared memory with bulk copies; the nonzeros
// are already in output-row order (the schedule sorted each tile), so every
// thread group walks a contiguous slice: a lane decodes one nonzero's output
// and operand rows from its block coordinates and offsets, the group shares
// them by shuffles, gathers the operand rows and accumulates row runs.
// Records in flight per thread group of the 3-D FP32 walk, and the CTAs per
// SM the compiler is asked to fit (0: no register cap): compile-time choices.
#ifndef PTI_HICOO_U
#define PTI_HICOO_U 2
#endif
#ifndef PTI_HICOO_MINB
#define PTI_HICOO_MINB 0
#endif

template <int G, int CPL, int U, class FT, int NIN>
__global__ void __launch_bounds__(kSchedThreads, PTI_HICOO_MINB) hicoo_sched_kernel(SchedArgs a)
{
    using L = HiSmem<NIN, CPL>;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t s_slot_row[kSchedThreads];
    __shared__ uint8_t s_slot_whole[kSchedThreads];
    float *s_val = reinterpret_cast<float *>(sm + L::val);
    uint8_t *s_eout = sm + L::eout;
    uint8_t *s_ein = sm + L::ein;
    uint16_t *s_blk = reinterpret_cast<uint16_t *>(sm + L::blk);
    uint32_t *s_brow = reinterpret_cast<uint32_t *>(sm + L::brow);
    uint32_t *s_bin = reinterpret_cast<uint32_t *>(sm + L::bin);
    float *s_slots = reinterpret_cast<float *>(sm + L::slots);
    const uint32_t tid = threadIdx.x;

    const uint64_t z0 = (uint64_t)blockIdx.x * kHiTile;
    const uint32_t n = (uint32_t)((a.nnz - z0) < (uint64_t)kHiTile ? (a.nnz - z0) : (uint64_t)kHiTile);
    const uint32_t b0 = a.tile_block[blockIdx.x];
    uint32_t nblk = a.tile_block[blockIdx.x + 1] - b0 + 1;
    if (nblk > kHiTile + 1) nblk = kHiTile + 1;
    if (b0 + (uint64_t)nblk > a.nb) nblk = (uint32_t)(a.nb - b0);

    // Stage the tile with bulk copies.  A bulk copy starts on 16 bytes, so the
    // block coordinates are copied from b0 rounded down to 4 entries.
    const uint32_t bo4 = b0 & 3u;
    if (tid == 0) {
        mbar_init(&mbar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    // 4-D: the blocks' four coordinates come as one 16-byte record each, so a
    // nonzero's decode reads them with one shared-memory load
    const uint4 *s_bq = reinterpret_cast<const uint4 *>(sm + L::brow);
    if (tid == 0) {
        const uint32_t be = round16(n), bv = round16(4 * n), bl = round16(2 * n);
        const uint32_t bb = 4 * ((nblk + bo4 + 3) & ~3u);
        const uint32_t bq = 16 * nblk;
        mbar_arrive_expect_tx(&mbar, bv + (NIN + 1) * be + bl + (NIN == 3 ? bq : (NIN + 1) * bb));
        bulk_g2s_ef(s_val, a.vals + z0, bv, &mbar);
        bulk_g2s_ef(s_eout, a.out_eind + z0, be, &mbar);
#pragma unroll
        for (int k = 0; k < NIN; ++k) bulk_g2s_ef(s_ein + k * kHiTile, a.in_eind[k] + z0, be, &mbar);
        bulk_g2s_ef(s_blk, a.lblk + z0, bl, &mbar);
        if constexpr (NIN == 3) {
            bulk_g2s_ef(sm + L::brow, a.bquad + b0, bq, &mbar);
        } else {
            bulk_g2s_ef(s_brow, a.out_bind + (b0 - bo4), bb, &mbar);
#pragma unroll
            for (int k = 0; k < NIN; ++k)
                bulk_g2s_ef(s_bin + k * (kHiTile + 4), a.in_bind[k] + (b0 - bo4), bb, &mbar);
        }
    }
    const bool ok = mbar_wait_bounded(&mbar, 0);
    if (!__syncthreads_and(ok)) {
        if (tid == 0) {
            atomicOr(a.err, 2u);
            mbar_wait_bounded(&mbar, 0);
        }
        return;
    }
    s_brow += bo4;  // block i of the tile is entry i + bo4 of the staged coordinates
    s_bin += bo4;

    // Decode every nonzero once into a 16-byte record {output row, operand
    // row offsets (row x stride)} (the value in the last free word, or beside
    // the records for 4-D), written over the staged arrays once they have all
    // been read.  A nonzero with a coordinate out of range sets the error
    // word and becomes a record that adds nothing (value 0, operand rows 0);
    // its output row is kept if that is valid, else it is kNoRow, which sorts
    // where the schedule put it (after every valid row of the tile).
    constexpr int PER = kHiTile / kSchedThreads;
    {
        uint4 rec[PER];
        float vv[PER];
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const uint32_t z = tid + p * kSchedThreads;
            rec[p] = make_uint4(kNoRow, 0u, 0u, 0u);
            vv[p] = 0.f;
            if (z < n) {
                const uint32_t i0 = s_blk[z];
                const bool ok_b = i0 < nblk;
                const uint32_t i = ok_b ? i0 : 0u;
                uint32_t bo, bi[3];
                if constexpr (NIN == 3) {
                    const uint4 q = s_bq[i];
                    bo = q.x;
                    bi[0] = q.y;
                    bi[1] = q.z;
                    bi[2] = q.w;
                } else {
                    bo = s_brow[i];
#pragma unroll
                    for (int k = 0; k < NIN; ++k) bi[k] = s_bin[k * (kHiTile + 4) + i];
                }
                const uint64_t o = ((uint64_t)bo << a.sb) + s_eout[z];
                const bool ok_o = ok_b && o < a.out_dim;
                uint32_t r[3] = {0u, 0u, 0u};
                bool ok_in = true;
#pragma unroll
                for (int k = 0; k < NIN; ++k) {
                    const uint64_t rk = ((uint64_t)bi[k] << a.sb) + s_ein[k * kHiTile + z];
                    ok_in = ok_in && rk < a.in_dim[k];
                    r[k] = (uint32_t)rk;
                }
#pragma unroll
                for (int k = 0; k < NIN; ++k) r[k] = ok_in ? r[k] : 0u;
                vv[p] = ok_o && ok_in ? s_val[z] : 0.f;
                if (NIN == 1) r[1] = __float_as_uint(vv[p]);
                if (NIN == 2) r[2] = __float_as_uint(vv[p]);
                rec[p] = make_uint4(ok_o ? (uint32_t)o : kNoRow, r[0], r[1], r[2]);
                if (!(ok_o && ok_in)) atomicOr(a.err, 1u);
            }
        }
        __syncthreads();
        uint4 *s_rec_w = reinterpret_cast<uint4 *>(sm + L::rec);
        float *s_v3_w = reinterpret_cast<float *>(sm + L::rval);
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const uint32_t z = tid + p * kSchedThreads;
            if (z < n) {
                s_rec_w[z] = rec[p];
                if (NIN == 3) s_v3_w[z] = vv[p];
            }
        }
    }
    __syncthreads();
    const uint4 *s_rec = reinterpret_cast<const uint4 *>(sm + L::rec);
    const float *s_v3 = reinterpret_cast<const float *>(sm + L::rval);

    const Groups<G> grp(tid);
    const uint32_t g = grp.g, lane = grp.lane;
    constexpr uint32_t kGroups = Groups<G>::count;
    // an odd slice length puts the groups' first records on different shared-memory banks
    const uint32_t per = ((n + kGroups - 1) / kGroups) | 1u;
    const uint32_t j0 = min(g * per, n), j1 = min(j0 + per, n);
    walk_rows<G, CPL, U, FT, NIN>(s_rec, s_v3, n, j0, j1, g, lane, a, s_slots, s_slot_row, s_slot_whole);
}

template <int NIN, int CPL>
struct RecSmem {
    // byte offsets inside the dynamic shared memory of hicoo_rec_kernel
    static constexpr uint32_t rec = 0;                                 // uint4[kHiTile]
    static constexpr uint32_t rval = rec + 16 * kHiTile;               // float[kHiTile] (4-D only)
    static constexpr uint32_t slots = rval + (NIN == 3 ? 4 * kHiTile : 0);  // float[kSchedThreads * CPL]
    static constexpr uint32_t total = slots + 4 * kSchedThreads * CPL;
};

// HiCOO schedule, one CTA per tile of kHiTile nonzeros whose records the
// schedule already holds decoded (HicooModePlan::recs, in output-row order
// within the tile): one bulk copy stages them (and the 4-D values), then the
// thread groups walk contiguous slices (walk_rows).
template <int G, int CPL, int U, class FT, int NIN>
__global__ void __launch_bounds__(kSchedThreads, PTI_HICOO_MINB) hicoo_rec_kernel(SchedArgs a)
{
    using L = RecSmem<NIN, CPL>;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t s_slot_row[kSchedThreads];
    __shared__ uint8_t s_slot_whole[kSchedThreads];
    uint4 *s_rec = reinterpret_cast<uint4 *>(sm + L::rec);
    float *s_v3 = reinterpret_cast<float *>(sm + L::rval);
    float *s_slots = reinterpret_cast<float *>(sm + L::slots);
    const uint32_t tid = threadIdx.x;
    const uint64_t z0 = (uint64_t)blockIdx.x * kHiTile;
    const uint32_t n = (uint32_t)min((uint64_t)kHiTile, a.nnz - z0);
    if (tid == 0) {
        mbar_init(&mbar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (tid == 0) {
        const uint32_t bv = NIN == 3 ? round16(4 * n) : 0u;
        mbar_arrive_expect_tx(&mbar, 16 * n + bv);
        bulk_g2s_ef(s_rec, a.recs + z0, 16 * n, &mbar);
        if constexpr (NIN == 3) bulk_g2s_ef(s_v3, a.rvals + z0, bv, &mbar);
    }
    const bool ok = mbar_wait_bounded(&mbar, 0);
    if (!__syncthreads_and(ok)) {
        if (tid == 0) {
            atomicOr(a.err, 2u);
            mbar_wait_bounded(&mbar, 0);
        }
        return;
    }
    const Groups<G> grp(tid);
    const uint32_t g = grp.g, lane = grp.lane;
    constexpr uint32_t kGroups = Groups<G>::count;
    // an odd slice length puts the groups' first records on different shared-memory banks
    const uint32_t per = ((n + kGroups - 1) / kGroups) | 1u;
    const uint32_t j0 = min(g * per, n), j1 = min(j0 + per, n);
    walk_rows<G, CPL, U, FT, NIN>(s_rec, s_v3, n, j0, j1, g, lane, a, s_slots, s_slot_row, s_slot_whole);
}

// COO schedule: packed records sorted by output index; no sorting in the
// kernel.  A CTA takes one tile, whatever their number: smaller ones are faster
// where tiles are few (100,000 Zipf nonzeros in HiCOO 50 -> 25 us, COO 1M 55 ->
// 49), but add the hot rows of a power-law mode to the output in more parts,
// and the error of those sums against 64 bits grows (mean over ten tensors of
// positive terms 8.6e-8 with whole tiles, 1.22e-7 with parts).  Calls whose other
// choice is the direct kernel, which adds every product by itself, are cut
// (a.cut; split.cuh): its error is 2e-4 where this has 3e-7.  Substituted values
// (the residual of a CP gradient) are fetched while the records are on their
// way and put into them, so the walk knows one kind of record: a load and a
// choice per record less, every mode and both sides cut into even turns, COO 3M Zipf R = 64 281 -> 264 us, 1M R =
// 16 51 -> 49.5, 4-D 5M R = 32 503 -> 489; 20M uniform R = 64 loss and gradient
// 3.10 -> 3.03 ms, Zipf 2.92 -> 2.78.
template <int G, int CPL, int U, int MINB, class FT, int NIN>
__global__ void __launch_bounds__(kSchedThreads, MINB) coo_sched_kernel(SchedArgs a, const uint32_t *recs, uint32_t tile)
{
    constexpr int RW = Rec<NIN>::words;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint64_t mbar;
    uint32_t *s_rec = reinterpret_cast<uint32_t *>(sm);
    const uint32_t tid = threadIdx.x;
    const uint64_t z0 = (uint64_t)blockIdx.x * tile;
    const uint32_t n = (uint32_t)((a.nnz - z0) < (uint64_t)tile ? (a.nnz - z0) : (uint64_t)tile);
    if (tid == 0) {
        mbar_init(&mbar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (tid == 0) {
        const uint32_t bytes = n * RW * 4;
        mbar_arrive_expect_tx(&mbar, bytes);
        bulk_g2s_ef(s_rec, recs + z0 * RW, bytes, &mbar);
    }
    constexpr uint32_t kPer = (coo_tile(RW) + kSchedThreads - 1) / kSchedThreads;
    float sub[kPer];
    if (a.vals) {
        uint32_t z[kPer];
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            const uint32_t j = tid + i * kSchedThreads;
            z[i] = j < n ? (a.perm ? __ldcs(a.perm + z0 + j) : (uint32_t)(z0 + j)) : 0;
        }
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) sub[i] = __ldcg(a.vals + z[i]);
    }
    const bool ok = mbar_wait_bounded(&mbar, 0);
    if (!__syncthreads_and(ok)) {
        if (tid == 0) {
            atomicOr(a.err, 2u);
            mbar_wait_bounded(&mbar, 0);
        }
        return;
    }
    if (a.vals) {
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            const uint32_t j = tid + i * kSchedThreads;
            if (j < n) s_rec[(size_t)j * RW + 1 + NIN] = __float_as_uint(sub[i]);
        }
        __syncthreads();
    }
    __shared__ uint32_t s_slot_row[kSchedThreads];
    __shared__ uint8_t s_slot_whole[kSchedThreads];
    float *s_slots = reinterpret_cast<float *>(sm + (size_t)tile * RW * 4);  // [groups][G][CPL]
    const Groups<G> grp(tid);
    const uint32_t g = grp.g, lane = grp.lane;
    constexpr uint32_t kGroups = Groups<G>::count;
    const uint32_t per = ((n + kGroups - 1) / kGroups) | 1u;  // odd: groups start on different banks
    const uint32_t j0 = min(g * per, n), j1 = min(j0 + per, n);
    process_records<G, CPL, U, NIN, FT>(s_rec, n, j0, j1, g, lane, a, s_slots, s_slot_row, s_slot_whole);
}

// ---------------------------------------------------------------------------
// Schedule construction
// ---------------------------------------------------------------------------
__global__ void iota_keys_kernel(const uint32_t *src, uint64_t n, uint32_t *keys, uint32_t *vals)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        keys[i] = src[i];
        vals[i] = (uint32_t)i;
    }
}

// COO packed records in sorted order: {out index, operand indices (modes in
// increasing order, skipping the output mode), value, 0...}.
struct PackArgs {
    uint32_t nin, rw;
    const uint32_t *out;
    const uint32_t *in[kMaxModes - 1];
    const float *vals;
};

__global__ void pack_records_kernel(PackArgs pa, const uint32_t *perm, uint64_t n, uint32_t *recs)
{
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t z = perm[j];
        uint32_t *r = recs + j * pa.rw;
        r[0] = pa.out[z];
        for (uint32_t k = 0; k < pa.nin; ++k) r[1 + k] = pa.in[k][z];
        r[1 + pa.nin] = __float_as_uint(pa.vals[z]);
        for (uint32_t k = pa.nin + 2; k < pa.rw; ++k) r[k] = 0;
    }
}

// The schedule order of one tile of kHiTile nonzeros, by one CTA: the blocks
// in their new order with their nonzeros behind one another, then
// stably by output row.  Writes for each position the nonzero there (order)
// and its block, counted from the tile's first (lblk).
//
// The blocks are ascending in their output coordinate, so a tile spans few
// rows: a stable radix sort by 8-bit digits of the row, counted from the tile's
// first, takes one pass for most tiles and at most four.  (A bitonic sort of
// 64-bit {row, position} pairs, fed by passes that spelt out every nonzero's
// block, took 0.63 ms a mode for 10M Zipf nonzeros; this takes 0.12.)
struct TileOrderArgs {
    uint64_t nnz, nb;
    uint32_t sb;
    const uint32_t *tile_block;
    const uint64_t *nbptr;     // first position of each block of the new order
    const uint32_t *first;     // its first nonzero where it is stored
    const uint32_t *out_bind;  // its output coordinate
    const uint8_t *out_eind;
    uint32_t *order;
    uint16_t *lblk;
};

__global__ void __launch_bounds__(kSortThreads) tile_order_kernel(TileOrderArgs t)
{
    constexpr uint32_t T = kHiTile, PER = T / kSortThreads;
    static_assert(T == 32 * PER * kSortWarps && T <= 2048, "shared memory");
    __shared__ uint32_t s_key[2][T], s_z[T], s_cnt[kSortWarps][256], s_warp[32], s_min, s_max;
    __shared__ uint16_t s_pos[2][T], s_l[T];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t z0 = (uint64_t)blockIdx.x * T;
    const uint32_t cnt = (uint32_t)((t.nnz - z0) < T ? (t.nnz - z0) : T);
    const uint32_t b0 = t.tile_block[blockIdx.x];
    const uint32_t nblk = (uint32_t)min((uint64_t)min(t.tile_block[blockIdx.x + 1] - b0 + 1, T + 1), t.nb - b0);
    // each position's block: the number of blocks that start up to it
    for (uint32_t i = tid; i < T; i += kSortThreads) s_key[1][i] = 0;
    if (tid == 0) {
        s_min = 0xFFFFFFFFu;
        s_max = 0;
    }
    __syncthreads();
    for (uint32_t i = tid; i < nblk; i += kSortThreads) {
        const uint64_t st = t.nbptr[b0 + i];
        if (st < z0 + cnt) s_key[1][st > z0 ? (uint32_t)(st - z0) : 0u] = 1u;
    }
    __syncthreads();
    uint32_t row[PER], sum = 0, total, lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
    for (uint32_t p = 0; p < PER; ++p) sum += s_key[1][tid * PER + p];
    uint32_t run = block_exclusive_scan<uint32_t>(sum, s_warp, total);
    // the loads of all PER positions together; only the element offsets are
    // read from where the nonzeros are stored
    uint32_t z[PER], ob[PER], eo[PER];
#pragma unroll
    for (uint32_t p = 0; p < PER; ++p) {
        const uint32_t pos = tid * PER + p;
        run += s_key[1][pos];
        row[p] = run - 1;
        z[p] = ob[p] = 0;
        if (pos < cnt) {
            const uint32_t j = b0 + row[p];
            z[p] = __ldg(t.first + j) + (uint32_t)(z0 + pos - __ldg(t.nbptr + j));
            ob[p] = __ldg(t.out_bind + j);
        }
    }
#pragma unroll
    for (uint32_t p = 0; p < PER; ++p) eo[p] = tid * PER + p < cnt ? __ldg(t.out_eind + z[p]) : 0u;
#pragma unroll
    for (uint32_t p = 0; p < PER; ++p) {
        const uint32_t pos = tid * PER + p;
        s_z[pos] = z[p];
        s_l[pos] = (uint16_t)row[p];
        // (a coordinate beyond 32 bits is out of range: behind every row)
        const uint64_t o = ((uint64_t)ob[p] << t.sb) + eo[p];
        row[p] = 0xFFFFFFFFu;
        if (pos < cnt) {
            row[p] = o < 0xFFFFFFFFull ? (uint32_t)o : 0xFFFFFFFFu;
            lo = min(lo, row[p]);
            hi = max(hi, row[p]);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
        atomicMin(&s_min, lo);
        atomicMax(&s_max, hi);
    }
    __syncthreads();
    const uint32_t first = s_min, range = s_max - first;
#pragma unroll
    for (uint32_t p = 0; p < PER; ++p) {
        const uint32_t pos = tid * PER + p;
        s_key[0][pos] = pos < cnt ? row[p] - first : 0xFFFFFFFFu;  // past the end: behind every nonzero
        s_pos[0][pos] = (uint16_t)pos;
    }
    uint32_t cur = 0;
    for (uint32_t shift = 0; shift < 32 && range >> shift; shift += 8, cur ^= 1) {
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) s_cnt[w][tid] = 0;
        __syncthreads();
        uint32_t key[PER], rank[PER];
#pragma unroll
        for (uint32_t r = 0; r < PER; ++r) {
            key[r] = s_key[cur][warp * (32 * PER) + 32 * r + lane];
            rank[r] = warp_digit_rank(key[r] >> shift & 0xFFu, s_cnt[warp]);
        }
        __syncthreads();
        digit_starts(s_cnt, s_warp);
        __syncthreads();
#pragma unroll
        for (uint32_t r = 0; r < PER; ++r) {
            const uint32_t to = s_cnt[warp][key[r] >> shift & 0xFFu] + rank[r];
            s_key[cur ^ 1][to] = key[r];
            s_pos[cur ^ 1][to] = s_pos[cur][warp * (32 * PER) + 32 * r + lane];
        }
        __syncthreads();
    }
    __syncthreads();
    for (uint32_t j = tid; j < cnt; j += kSortThreads) {
        const uint32_t pos = s_pos[cur][j];
        t.order[z0 + j] = s_z[pos];
        t.lblk[z0 + j] = s_l[pos];
    }
}

// The schedule's arrays, gathered in its order in two passes: the blocks'
// coordinates, then everything of a nonzero, its decoded record included
// (HicooModePlan::recs; the nonzero at position j lies in block
// tile_block[j / kHiTile] + lblk[j]).  Operands in increasing mode order.
struct PlanGatherArgs {
    uint64_t n, nb;
    uint32_t nmodes, mode, sb;
    uint32_t dims[kMaxModes];
    const uint32_t *bperm, *order, *tile_block;
    const uint16_t *lblk;
    const uint32_t *binds_in[kMaxModes];
    const uint8_t *einds_in[kMaxModes];
    const float *vals_in;
    uint32_t *binds[kMaxModes];
    uint8_t *einds[kMaxModes];
    float *vals;
    uint4 *bquad;   // 4-D: {output, operands}
    uint4 *recs;
    float *rvals;   // 4-D
    uint32_t *err;
};

__global__ void __launch_bounds__(256) plan_blocks_kernel(PlanGatherArgs g)
{
    for (uint64_t j = (uint64_t)blockIdx.x * 256 + threadIdx.x; j < g.nb; j += (uint64_t)gridDim.x * 256) {
        const uint32_t b = g.bperm[j];
        uint32_t c[kMaxModes], q[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int k = 0; k < kMaxModes; ++k)
            if (k < (int)g.nmodes) {
                if (k == (int)g.mode) c[k] = g.binds[k][j];  // in the new order already
                else g.binds[k][j] = c[k] = g.binds_in[k][b];
            }
        if (g.bquad) {
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k == (int)g.mode ? 0 : k < (int)g.mode ? k + 1 : k] = c[k];
            g.bquad[j] = make_uint4(q[0], q[1], q[2], q[3]);
        }
    }
}

template <int N>
__global__ void __launch_bounds__(256) plan_nonzeros_kernel(PlanGatherArgs g)
{
    for (uint64_t j = (uint64_t)blockIdx.x * 256 + threadIdx.x; j < g.n; j += (uint64_t)gridDim.x * 256) {
        const uint32_t z = g.order[j];
        const uint64_t b0 = (uint64_t)g.tile_block[j / kHiTile] + g.lblk[j];
        const float val = g.vals_in[z];
        const bool ok_b = b0 < g.nb;
        const uint64_t b = ok_b ? b0 : 0;
        uint32_t row[3] = {0u, 0u, 0u}, out = 0;
        bool ok_in = true, ok_o = ok_b;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint8_t e = g.einds_in[k][z];
            g.einds[k][j] = e;
            const uint64_t c = ((uint64_t)g.binds[k][b] << g.sb) + e;
            const bool ok = c < g.dims[k];
            if (k == (int)g.mode) {
                out = (uint32_t)c;
                ok_o = ok_o && ok;
            } else {
                ok_in = ok_in && ok;
                const int i = k < (int)g.mode ? k : k - 1;
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    if (x == i) row[x] = (uint32_t)c;
            }
        }
        g.vals[j] = val;
        if (!ok_in) row[0] = row[1] = row[2] = 0u;
        const float v = ok_o && ok_in ? val : 0.f;
        uint4 rec = make_uint4(ok_o ? out : kNoRow, row[0], row[1], row[2]);
        if (N == 2) rec.z = __float_as_uint(v);
        if (N == 3) rec.w = __float_as_uint(v);
        if (N == 4) g.rvals[j] = v;
        g.recs[j] = rec;
        if (!(ok_o && ok_in)) atomicOr(g.err, 1u);
    }
}

// (Bound by the random 32-byte sectors: four reads in flight a thread, from a
// 16-byte load of perm, took 143 us instead of 134 for 20M values.)
__global__ void gather_kernel(const float *src, const uint32_t *perm, uint64_t n, float *dst)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        dst[i] = src[perm[i]];
}

__global__ void tile_block_kernel_t(const uint64_t *bptr, uint64_t nb, uint32_t ntiles, uint32_t tile,
                                    uint32_t *tile_block)
{
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t zs = bptr[b], ze = bptr[b + 1];
        for (uint64_t t = (zs + tile - 1) / tile; t * tile < ze && t < ntiles; ++t) tile_block[t] = (uint32_t)b;
        if (b == nb - 1) tile_block[ntiles] = (uint32_t)b;
    }
}

// First nonzero and size of each block of the new order (nonzeros are indexed
// by 32 bits).
__global__ void __launch_bounds__(256) block_spans_kernel(const uint32_t *perm, uint64_t nb, const uint64_t *bptr,
                                                          uint32_t *first, uint32_t *size)
{
    for (uint64_t j = (uint64_t)blockIdx.x * 256 + threadIdx.x; j < nb; j += (uint64_t)gridDim.x * 256) {
        const uint32_t b = perm[j];
        const uint64_t z = bptr[b];
        first[j] = (uint32_t)z;
        size[j] = (uint32_t)(bptr[b + 1] - z);
    }
}

struct SizeIn {
    const uint32_t *p;
    __device__ uint64_t operator()(uint64_t i) const { return p[i]; }
};
struct BptrOut {
    uint64_t *p;
    __device__ void operator()(uint64_t i, uint64_t prefix, uint64_t) const { p[i] = prefix; }
};

static uint32_t bits_for_count(uint64_t count)
{
    uint32_t b = 0;
    while (b < 64 && ((uint64_t)1 << b) < count) ++b;
    return b;
}

static unsigned grid_n(uint64_t n)
{
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)sm_count() * 32));
}

static int build_plan(ptiB200Tensor *t, uint32_t mode, cudaStream_t s, const Arrivals *arr)
{
    const char *mod = "B200 Prepare";
    const uint32_t N = t->nmodes;
    const uint64_t n = t->nnz;
    PTI_CHECK(n < 0xFFFFFFFFull, PTIERR_VALUE_ERROR, mod, "too many nonzeros");
    if (n == 0) return 0;
    if (!t->hicoo) {
        CooModePlan &P = t->coo_plan[mode];
        if (P.ready) return 0;
        DevBuf keys, perm;
        RadixScratchT<uint32_t> rs;
        PTI_CUDA(keys.alloc(padded(n * 4), s), mod);
        PTI_CUDA(perm.alloc(padded(n * 4), s), mod);
        PTI_TRY(rs.alloc(n, s));
        iota_keys_kernel<<<grid_n(n), 256, 0, s>>>(t->inds[mode].as<uint32_t>(), n, keys.as<uint32_t>(),
                                                   perm.as<uint32_t>());
        PTI_TRY(radix_sort_pairs(keys, perm, n, (int)bits_for_count(t->ndims[mode]), rs, s));
        const int RW = rec_words((int)N - 1);
        PTI_CUDA(P.recs.alloc(padded(n * RW * 4), s), mod);
        PackArgs pa{};
        pa.nin = N - 1;
        pa.rw = RW;
        pa.out = t->inds[mode].as<uint32_t>();
        for (uint32_t k = 0, i = 0; k < N; ++k)
            if (k != mode) pa.in[i++] = t->inds[k].as<uint32_t>();
        pa.vals = t->vals.as<float>();
        pack_records_kernel<<<grid_n(n), 256, 0, s>>>(pa, perm.as<uint32_t>(), n, P.recs.as<uint32_t>());
        PTI_CUDA(cudaGetLastError(), mod);
        P.perm = std::move(perm);
        P.ready = true;
        return 0;
    }
    HicooModePlan &P = t->hicoo_plan[mode];
    if (P.ready || N > 4) return 0;  // a record holds three operand rows; other orders take the direct kernel
    const uint64_t nb = t->nb;
    PTI_CHECK(t->sb <= 8, PTIERR_VALUE_ERROR, mod, "sb_bits must be <= 8");
    // 1. blocks by output-mode block coordinate (stable)
    DevBuf bperm, nbptr, first, order;  // (the sorted coordinates stay as P.binds[mode])
    {
        RadixScratchT<uint32_t> rs;
        DevBuf &bkeys = P.binds[mode];
        PTI_CUDA(bkeys.alloc(padded(nb * 4), s), mod);
        PTI_CUDA(bperm.alloc(padded(nb * 4), s), mod);
        PTI_TRY(rs.alloc(nb, s));
        iota_keys_kernel<<<grid_n(nb), 256, 0, s>>>(t->binds[mode].as<uint32_t>(), nb, bkeys.as<uint32_t>(),
                                                    bperm.as<uint32_t>());
        const uint64_t brows = ((uint64_t)t->ndims[mode] + ((uint64_t)1 << t->sb) - 1) >> t->sb;
        PTI_TRY(radix_sort_pairs(bkeys, bperm, nb, (int)std::min(32u, bits_for_count(brows + 1)), rs, s));
    }
    PTI_CUDA(nbptr.alloc(padded((nb + 1) * 8), s), mod);
    PTI_CUDA(first.alloc(padded(nb * 4), s), mod);
    {
        DevBuf tmp, bsize;
        PTI_CUDA(bsize.alloc(padded(nb * 4), s), mod);
        block_spans_kernel<<<grid_n(nb), 256, 0, s>>>(bperm.as<uint32_t>(), nb, t->bptr.as<uint64_t>(),
                                                      first.as<uint32_t>(), bsize.as<uint32_t>());
        PTI_CUDA(tmp.alloc(padded(scan_tmp_elems<uint64_t>(nb) * 8), s), mod);
        PTI_TRY((exclusive_scan<uint64_t>(SizeIn{bsize.as<uint32_t>()}, BptrOut{nbptr.as<uint64_t>()}, nb,
                                          tmp.as<uint64_t>(), nullptr, s)));
        PTI_CUDA(cudaMemcpyAsync(nbptr.as<uint64_t>() + nb, tmp.as<uint64_t>() + (nb + kScanTile - 1) / kScanTile,
                                 8, cudaMemcpyDeviceToDevice, s), mod);
    }
    P.nb = nb;
    P.ntiles = (uint32_t)((n + kHiTile - 1) / kHiTile);
    PTI_CUDA(P.tile_block.alloc(padded(((size_t)P.ntiles + 1) * 4), s), mod);
    tile_block_kernel_t<<<grid_n(nb), 256, 0, s>>>(nbptr.as<uint64_t>(), nb, P.ntiles, kHiTile,
                                                   P.tile_block.as<uint32_t>());
    // 2. nonzeros in block order (blocks in their new order), inside each tile
    // of that order by output row
    PTI_CUDA(order.alloc(padded(n * 4), s), mod);
    PTI_CUDA(P.lblk.alloc(padded(n * 2), s), mod);
    TileOrderArgs ta{};
    ta.nnz = n;
    ta.nb = nb;
    ta.sb = t->sb;
    ta.tile_block = P.tile_block.as<uint32_t>();
    ta.nbptr = nbptr.as<uint64_t>();
    ta.first = first.as<uint32_t>();
    ta.out_bind = P.binds[mode].as<uint32_t>();
    ta.out_eind = t->einds[mode].as<uint8_t>();
    ta.order = order.as<uint32_t>();
    ta.lblk = P.lblk.as<uint16_t>();
    tile_order_kernel<<<P.ntiles, kSortThreads, 0, s>>>(ta);
    // 3. everything up to here read only bptr and the output mode's arrays;
    // the gathers read every array, after its arrival (with `arr`)
    if (arr) {
        if (arr->vals) PTI_CUDA(cudaStreamWaitEvent(s, arr->vals, 0), mod);
        for (uint32_t k = 0; k < N; ++k)
            if (arr->mode[k]) PTI_CUDA(cudaStreamWaitEvent(s, arr->mode[k], 0), mod);
    }
    PTI_TRY(ensure_err_word(t, s));
    PlanGatherArgs g{};
    g.n = n;
    g.nb = nb;
    g.nmodes = N;
    g.mode = mode;
    g.sb = t->sb;
    g.bperm = bperm.as<uint32_t>();
    g.order = order.as<uint32_t>();
    g.tile_block = P.tile_block.as<uint32_t>();
    g.lblk = P.lblk.as<uint16_t>();
    g.vals_in = t->vals.as<float>();
    for (uint32_t k = 0; k < N; ++k) {
        if (k != mode) PTI_CUDA(P.binds[k].alloc(padded(nb * 4), s), mod);
        PTI_CUDA(P.einds[k].alloc(padded(n), s), mod);
        g.dims[k] = t->ndims[k];
        g.binds_in[k] = t->binds[k].as<uint32_t>();
        g.einds_in[k] = t->einds[k].as<uint8_t>();
        g.binds[k] = P.binds[k].as<uint32_t>();
        g.einds[k] = P.einds[k].as<uint8_t>();
    }
    PTI_CUDA(P.vals.alloc(padded(n * 4), s), mod);
    PTI_CUDA(P.recs.alloc(padded(n * 16), s), mod);
    if (N == 4) {
        PTI_CUDA(P.bquad.alloc(padded(nb * 16), s), mod);
        PTI_CUDA(P.rvals.alloc(padded(n * 4), s), mod);
    }
    g.vals = P.vals.as<float>();
    g.bquad = P.bquad.as<uint4>();
    g.recs = P.recs.as<uint4>();
    g.rvals = P.rvals.as<float>();
    g.err = err_word(t);
    plan_blocks_kernel<<<grid_n(nb), 256, 0, s>>>(g);
    if (N == 2) plan_nonzeros_kernel<2><<<grid_n(n), 256, 0, s>>>(g);
    else if (N == 3) plan_nonzeros_kernel<3><<<grid_n(n), 256, 0, s>>>(g);
    else plan_nonzeros_kernel<4><<<grid_n(n), 256, 0, s>>>(g);
    PTI_CUDA(cudaGetLastError(), mod);
    P.ready = true;
    return 0;
}

bool plan_ready(const ptiB200Tensor *t, uint32_t mode)
{
    return t->hicoo ? t->hicoo_plan[mode].ready : t->coo_plan[mode].ready;
}

static bool capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone;
}

// Builds the schedule of `mode` on first use.  The first call on a handle may
// come from any thread and stream, so the build is under the handle's lock and
// leaves an event behind: a call on another stream than the building one waits
// for it on the device.  (A capturing stream cannot wait for work outside its
// capture; a program captures after the schedules are built.)
int prepare_mode(ptiB200Tensor *t, uint32_t mode, cudaStream_t s, const Arrivals *arr)
{
    const char *mod = "B200 Prepare";
    PTI_CHECK(mode < t->nmodes, PTIERR_VALUE_ERROR, mod, "mode out of range");
    if (t->nnz == 0) return build_plan(t, mode, s, arr);
    std::lock_guard<std::mutex> lock(t->plan_mu);
    PlanOrder &o = t->plan_order[mode];
    if (plan_ready(t, mode)) {
        if (o.event && s != o.stream && !capturing(s)) PTI_CUDA(cudaStreamWaitEvent(s, o.event, 0), mod);
        return 0;
    }
    PTI_TRY(ensure_err_word(t, s));
    const int st = build_plan(t, mode, s, arr);
    if (st) {  // what was allocated of it goes back
        if (t->hicoo) t->hicoo_plan[mode] = HicooModePlan();
        else t->coo_plan[mode] = CooModePlan();
        return st;
    }
    if (!capturing(s)) {
        if (!o.event) PTI_CUDA(cudaEventCreateWithFlags(&o.event, cudaEventDisableTiming), mod);
        PTI_CUDA(cudaEventRecord(o.event, s), mod);
        o.stream = s;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Launch
// ---------------------------------------------------------------------------
// Records in flight per group of the COO walk (FP32, R <= 32) and the CTAs
// per SM its register budget is set for: compile-time choices.
#ifndef PTI_COO_U
#define PTI_COO_U 3
#endif
// ... and for 33 <= R <= 64 (3 fit the same 64-register budget as 2)
#ifndef PTI_COO_U64
#define PTI_COO_U64 3
#endif
#ifndef PTI_COO_MINB
#define PTI_COO_MINB 4
#endif

template <int G, int CPL, int U, class FT, int NIN>
static int launch_coo(const SchedArgs &a, const uint32_t *recs, cudaStream_t s)
{
    constexpr uint32_t RW = Rec<NIN>::words, kTile = coo_tile(RW);
    constexpr size_t smem_max = (size_t)kTile * RW * 4 + (size_t)kSchedThreads * CPL * 4;
    // more operands hold more registers per nonzero in flight
    constexpr int UU = NIN > 4 ? 1 : (NIN >= 3 && U > 2 ? 2 : U);
    auto k = coo_sched_kernel<G, CPL, UU, PTI_COO_MINB, FT, NIN>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max) != cudaSuccess)
        return PTIERR_CUDA_ERROR;
    uint32_t tile = kTile;
    if (a.cut) {
        // 1024 records of 8 words with FP32 rows fit a fourth CTA on an SM (4-D
        // 3M Zipf R = 150, every mode, 1.55 -> 1.21 ms)
        constexpr uint32_t kCut = RW == 8 && CPL == 4 ? kTile / 2 : kTile;
        static const uint64_t slots = cta_slots(k, kSchedThreads, (size_t)kCut * RW * 4 + (size_t)kSchedThreads * CPL * 4);
        tile = tile_for(a.nnz, kCut, slots, Groups<G>::count * 4);
    }
    const size_t smem = (size_t)tile * RW * 4 + (size_t)kSchedThreads * CPL * 4;
    k<<<(unsigned)((a.nnz + tile - 1) / tile), kSchedThreads, smem, s>>>(a, recs, tile);
    return 0;
}

// Which HiCOO kernel runs (a compile-time choice): 0 decodes every tile from
// the staged HiCOO arrays (hicoo_sched_kernel), 2 stages the schedule's
// decoded records (hicoo_rec_kernel), 1 takes the records for 4-D tensors and
// for BF16 factors and decodes 3-D FP32 tiles.
#ifndef PTI_REC_POLICY
#define PTI_REC_POLICY 1
#endif
// CTAs per SM the BF16 record kernels are held to (0: no limit).  Their walk
// is bound by the L1 data pipe and feeds on the L1 that a further CTA's
// shared memory would take.
#ifndef PTI_REC_BF16_CTAS
#define PTI_REC_BF16_CTAS 3
#endif

template <class FT, int NIN>
constexpr bool use_records()
{
    return PTI_REC_POLICY == 2 || (PTI_REC_POLICY == 1 && (NIN == 3 || sizeof(FT) == 2));
}

template <int G, int CPL, class FT, int NIN>
static int launch_hicoo(const SchedArgs &a, unsigned ntiles, cudaStream_t s)
{
    constexpr int U = NIN == 3 || CPL == 8 ? 2 : PTI_HICOO_U;  // nonzeros in flight per group
    if constexpr (!use_records<FT, NIN>()) {
        constexpr size_t smem = HiSmem<NIN, CPL>::total;
        auto k = hicoo_sched_kernel<G, CPL, U, FT, NIN>;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return PTIERR_CUDA_ERROR;
        k<<<ntiles, kSchedThreads, smem, s>>>(a);
        return 0;
    }
    auto kr = hicoo_rec_kernel<G, CPL, U, FT, NIN>;
    size_t rec_smem = RecSmem<NIN, CPL>::total;
    if (sizeof(FT) == 2 && PTI_REC_BF16_CTAS > 0) {
        // more dynamic shared memory than 1/(n+1) of the SM's 228 KB (with
        // the static part and the 1 KB the runtime keeps per CTA)
        const size_t cap = 233472 / (PTI_REC_BF16_CTAS + 1) - 1408 - 1024 + 16;
        rec_smem = rec_smem > cap ? rec_smem : cap;
    }
    if (cudaFuncSetAttribute(kr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rec_smem) != cudaSuccess)
        return PTIERR_CUDA_ERROR;
    kr<<<ntiles, kSchedThreads, rec_smem, s>>>(a);
    return 0;
}

// Lanes per nonzero: 4 columns per lane (FP32 factors, or BF16 factors that
// are not 16-byte addressable by rows) or 8 columns per lane (BF16 with a
// stride that is a multiple of 8); one column pass (R <= 128).
template <class FT, int NIN>
static int launch_r(bool hicoo, bool wide, const SchedArgs &a, const uint32_t *recs, unsigned ntiles, cudaStream_t s)
{
    // lanes a row takes, rounded up to the next group size
    auto go = [&](auto lanes, auto cols) -> int {
        constexpr int G = decltype(lanes)::value, CPL = decltype(cols)::value;
        // records in flight per group of the COO walk
        constexpr int U = CPL == 8 ? 2 : G <= 8 ? PTI_COO_U : G <= 16 ? PTI_COO_U64 : 2;
        return hicoo ? launch_hicoo<G, CPL, FT, NIN>(a, ntiles, s) : launch_coo<G, CPL, U, FT, NIN>(a, recs, s);
    };
    auto pick = [&](auto cols) -> int {
        constexpr int CPL = decltype(cols)::value;
        const uint32_t q = (a.R + CPL - 1) / CPL;
#define PTI_LANES(n) if (q <= n) return go(std::integral_constant<int, n>{}, cols)
        PTI_LANES(1);
        PTI_LANES(2);
        PTI_LANES(4);
        // 6, 9 and 10 lanes beside the powers of two, where that is faster (16 bytes a lane: FP32, wide BF16; 3- and 4-D).  All
        // modes, power of two -> this: 9 and 10 lanes HiCOO 4-D 5M FP32 R = 40
        // 997 -> 687 us, R = 36 995 -> 752; 3-D 8M Zipf R = 40 813 -> 667, BF16
        // R = 80 861 -> 671; COO 3-D 5M Zipf R = 40 516 -> 421; but COO 4-D 3M
        // BF16 R = 80 590 -> 634.  6 lanes COO 3-D 5M Zipf FP32 R = 24 341 ->
        // 303, HiCOO 3-D 8M Zipf BF16 R = 48 527 -> 482; but HiCOO 3-D FP32
        // R = 24 467 -> 477 and every 4-D one slower.  3 and 5 lanes lose more
        // (walks of short rows are bound by their records) than they win.
        if constexpr (CPL * sizeof(FT) == 16 && NIN == 2) {
            if (!hicoo || sizeof(FT) == 2) {
                if (q == 6) return go(std::integral_constant<int, 6>{}, cols);
            }
        }
        PTI_LANES(8);
        if constexpr (CPL * sizeof(FT) == 16 && NIN >= 2) {
            if (hicoo || NIN == 2 || sizeof(FT) == 4) {
                PTI_LANES(9);
                PTI_LANES(10);
            }
        }
        PTI_LANES(16);
        if constexpr (CPL == 4) return go(std::integral_constant<int, 32>{}, cols);
        return PTIERR_VALUE_ERROR;  // not reached: R <= kPanel
#undef PTI_LANES
    };
    if constexpr (sizeof(FT) == 2) {
        if (wide) return pick(std::integral_constant<int, 8>{});
    }
    return pick(std::integral_constant<int, 4>{});
}

// COO schedules of 5 to 8 modes: 4 columns per lane.
template <class FT, int NIN>
static int launch_high(const SchedArgs &a, const uint32_t *recs, cudaStream_t s)
{
    if (a.R <= 8) return launch_coo<2, 4, 2, FT, NIN>(a, recs, s);
    if (a.R <= 16) return launch_coo<4, 4, 2, FT, NIN>(a, recs, s);
    if (a.R <= 32) return launch_coo<8, 4, 2, FT, NIN>(a, recs, s);
    if (a.R <= 64) return launch_coo<16, 4, 2, FT, NIN>(a, recs, s);
    return launch_coo<32, 4, 2, FT, NIN>(a, recs, s);
}

template <class FT>
static int launch_n(int nin, bool hicoo, bool wide, const SchedArgs &a, const uint32_t *recs, unsigned ntiles,
                    cudaStream_t s)
{
    switch (nin) {
        case 1: return launch_r<FT, 1>(hicoo, wide, a, recs, ntiles, s);
        case 2: return launch_r<FT, 2>(hicoo, wide, a, recs, ntiles, s);
        case 3: return launch_r<FT, 3>(hicoo, wide, a, recs, ntiles, s);
        case 4: return launch_high<FT, 4>(a, recs, s);
        case 5: return launch_high<FT, 5>(a, recs, s);
        case 6: return launch_high<FT, 6>(a, recs, s);
        default: return launch_high<FT, 7>(a, recs, s);
    }
}

// Ranks above kPanel run as panels of kPanel columns (the last one narrower),
// one launch each over the same schedule, because a lane group covers at most
// 32 lanes x 4 columns and holds one partial row.  COO records take any order;
// the HiCOO kernels hold three operand rows per record.
constexpr uint32_t kPanel = 128;

bool schedule_supported(const ptiB200Tensor *t, uint32_t mode, uint32_t R, uint32_t stride, bool own_vals,
                        cudaStream_t s)
{
    if (t->nmodes < 2 || t->nmodes > (t->hicoo ? 4u : (uint32_t)kMaxModes) || R < 1) return false;
    if (t->nnz >= 0xFFFFFFFFull && (t->nmodes > 4 || R > kPanel)) return false;  // schedules index nonzeros by 32 bits
    // Building the schedules of 5 modes takes about 0.3 ms, and what they save on
    // small tensors is little: 100,000 nonzeros R = 16, every mode, uniform 93 us
    // direct and 95 scheduled, Zipf 180 and 95; 300,000 111 and 95, 472 and 95.
    constexpr uint64_t kHighOrderFrom = 262144;
    if (t->nmodes > 4 && t->nnz < kHighOrderFrom) return false;
    // One launch of the direct kernel against one per panel: COO, R = 150, three
    // modes, 5,000 nonzeros 51 us against 65, 20,000 Zipf 64 against 65, 50,000
    // Zipf 126 against 64.  (The direct HiCOO kernel is slower at every size.)
    constexpr uint64_t kDirectBelow = 16384;
    if (!t->hicoo && R > kPanel && t->nnz < kDirectBelow) return false;
    // Above 4 modes or one panel the direct kernels stay the choice where a
    // schedule would add state that such calls did not have: substituted
    // values (one reordered copy per mode and handle), and a first use inside
    // a stream capture (the schedule's memory would belong to the graph).
    if ((t->nmodes > 4 || R > kPanel) && (!own_vals || (!plan_ready(t, mode) && capturing(s)))) return false;
    // the HiCOO kernel addresses factor rows by 32-bit element offsets
    if (t->hicoo)
        for (uint32_t m = 0; m < t->nmodes; ++m)
            if ((uint64_t)t->ndims[m] * stride >= ((uint64_t)1 << 32)) return false;
    return true;
}

// Runs the scheduled kernel for `mode` (the schedule must be ready).  Output
// must already be zeroed.
int mttkrp_scheduled(ptiB200Tensor *t, const void *const *mats, int ft, uint32_t R, uint32_t stride,
                     const uint32_t *mats_order, uint32_t mode, float *out, cudaStream_t s,
                     const float *vals_override)
{
    const char *mod = "B200 MTTKRP";
    const uint32_t N = t->nmodes;
    PTI_TRY(ensure_err_word(t, s));
    SchedArgs a{};
    a.nnz = t->nnz;
    a.R = R;
    a.stride = stride;
    a.out_dim = t->ndims[mode];
    a.out = out;
    a.err = err_word(t);
    a.cut = N > 4 || R > kPanel;
    const uint32_t *recs = nullptr;
    unsigned ntiles = 0;
    if (t->hicoo) {
        const HicooModePlan &P = t->hicoo_plan[mode];
        ntiles = P.ntiles;
        a.nb = P.nb;
        a.sb = t->sb;
        a.lblk = P.lblk.as<uint16_t>();
        a.tile_block = P.tile_block.as<uint32_t>();
        a.out_bind = P.binds[mode].as<uint32_t>();
        a.out_eind = P.einds[mode].as<uint8_t>();
        // the operands in increasing mode order: the order of the decoded
        // records and of the 4-D block records (a product of two factors does
        // not depend on the order, of three only in its FP32 rounding)
        (void)mats_order;
        for (uint32_t i = 0, k = 0; k < N; ++k)
            if (k != mode) {
                a.in_bind[i] = P.binds[k].as<uint32_t>();
                a.in_eind[i] = P.einds[k].as<uint8_t>();
                a.in_dim[i] = t->ndims[k];
                a.in_mat[i] = mats[k];
                ++i;
            }
        a.bquad = N == 4 ? P.bquad.as<uint4>() : nullptr;
        a.vals = P.vals.as<float>();
        a.recs = P.recs.as<uint4>();
        a.rvals = P.rvals.as<float>();
    } else {
        // records hold the operand modes in increasing order
        CooModePlan &P = t->coo_plan[mode];
        recs = P.recs.as<uint32_t>();
        // Substituted values are random reads through the permutation.  The walk
        // does them beside its own copies where they and the factors share the
        // L2; otherwise they would push the factor rows out of it, and a pass
        // of their own brings them into record order first.  Loss and gradient,
        // in the walk / in a pass, uniform: 8M R = 40 Zipf (45 MB) 0.97 / 1.02
        // ms, 10M R = 64 (78 MB) 1.29 / 1.34, 18M R = 16 (91 MB) 1.32 / 1.31,
        // 10M R = 64 (101 MB) 1.44 / 1.38, 14M R = 64 (133 MB) 2.25 / 2.00.
        constexpr uint64_t kValsBesideFactors = 96'000'000;
        uint64_t reused = t->nnz * 4;
        for (uint32_t k = 0; k < N; ++k) reused += (uint64_t)t->ndims[k] * stride * (ft == PTI_B200_F32 ? 4 : 2);
        if (vals_override && reused <= kValsBesideFactors) {
            a.vals = vals_override;
            a.perm = P.perm.as<uint32_t>();
        } else if (vals_override) {
            if (!P.alt_vals.ptr) PTI_CUDA(P.alt_vals.alloc(padded(t->nnz * 4), s), mod);
            gather_kernel<<<grid_n(t->nnz), 256, 0, s>>>(vals_override, P.perm.as<uint32_t>(), t->nnz,
                                                         P.alt_vals.as<float>());
            a.vals = P.alt_vals.as<float>();
        }
        for (uint32_t k = 0, i = 0; k < N; ++k)
            if (k != mode) {
                a.in_dim[i] = t->ndims[k];
                a.in_mat[i] = mats[k];
                ++i;
            }
    }
    // BF16 rows are read 8 columns (16 bytes) per lane when every row start
    // is 16-byte aligned.
    bool wide = ft == PTI_B200_BF16 && stride % 8 == 0;
    for (uint32_t k = 0; k < N && wide; ++k)
        if (k != mode && ((uintptr_t)mats[k] & 15) != 0) wide = false;
    const size_t esz = ft == PTI_B200_F32 ? 4 : 2;
    for (uint32_t c0 = 0; c0 < R; c0 += kPanel) {
        SchedArgs p = a;
        p.R = std::min(R - c0, kPanel);
        p.out = out + c0;
        for (uint32_t i = 0; i + 1 < N; ++i)
            p.in_mat[i] = static_cast<const unsigned char *>(a.in_mat[i]) + (size_t)c0 * esz;
        const int r = ft == PTI_B200_F32 ? launch_n<float>((int)N - 1, t->hicoo, false, p, recs, ntiles, s)
                                         : launch_n<__nv_bfloat16>((int)N - 1, t->hicoo, wide, p, recs, ntiles, s);
        PTI_CHECK(r == 0, r, mod, "kernel attribute setup failed");
    }
    PTI_CUDA(cudaGetLastError(), mod);
    return 0;
}

}  // namespace pti
