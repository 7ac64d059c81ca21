// primitives.cuh -- device-wide exclusive scan and a stable LSD radix sort of
// (32- or 64-bit key, 32-bit value) pairs, written for the COO->HiCOO conversion and
// the per-mode schedules.  Both are plain multi-kernel algorithms:
//   scan:  tile reduce -> single-CTA scan of tile sums -> tile rescan + add
//   sort:  per 8-bit digit: tile histograms -> scan (digit-major) -> stable
//          scatter, ranking equal digits within a warp with __match_any_sync
//          and across warps through shared-memory counters.
#pragma once
#include "common.cuh"

namespace pti {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

template <class T>
__device__ __forceinline__ T block_exclusive_scan(T v, T *s_warp, T &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < (int)(blockDim.x >> 5)) s_warp[lane] = w;
    }
    __syncthreads();
    T warp_prefix = warp ? s_warp[warp - 1] : T(0);
    total = s_warp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

template <class T, class In>
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(In in, uint64_t n, T *tile_sums)
{
    __shared__ T s_warp[32];
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    T sum = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j)
        if (base + j < n) sum += in(base + j);
    T total;
    block_exclusive_scan<T>(sum, s_warp, total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Exclusive scan of tile sums by one CTA; writes the grand total at [ntiles].
template <class T>
__global__ void __launch_bounds__(1024) scan_tiles_kernel(T *sums, uint64_t ntiles)
{
    __shared__ T s_warp[32];
    T carry = 0;
    for (uint64_t b = 0; b < ntiles; b += 1024) {
        uint64_t i = b + threadIdx.x;
        T v = i < ntiles ? sums[i] : T(0);
        T total;
        T ex = block_exclusive_scan<T>(v, s_warp, total);
        if (i < ntiles) sums[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) sums[ntiles] = carry;
}

template <class T, class In, class Out>
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(In in, uint64_t n, const T *tile_off, Out out)
{
    __shared__ T s_warp[32];
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    T sum = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        v[j] = base + j < n ? in(base + j) : T(0);
        sum += v[j];
    }
    T total;
    T run = block_exclusive_scan<T>(sum, s_warp, total) + tile_off[blockIdx.x];
#pragma unroll
    for (int j = 0; j < kScanItems; ++j)
        if (base + j < n) {
            out(base + j, run, v[j]);
            run += v[j];
        }
}

// The two halves of an exclusive scan, for a caller that sizes its output by
// the total: scan_sums returns the total through *total_host (synchronous copy)
// if that is non-null; scan_apply then calls out(i, prefix_i, in(i)) for every
// i.  `tmp` must hold ceil(n / kScanTile) + 1 elements of T.
template <class T, class In>
int scan_sums(In in, uint64_t n, T *tmp, T *total_host, cudaStream_t s)
{
    const char *mod = "B200 scan";
    const uint64_t ntiles = (n + kScanTile - 1) / kScanTile;
    if (ntiles == 0) {
        if (total_host) *total_host = 0;
        return 0;
    }
    scan_reduce_kernel<T, In><<<(unsigned)ntiles, kScanThreads, 0, s>>>(in, n, tmp);
    scan_tiles_kernel<T><<<1, 1024, 0, s>>>(tmp, ntiles);
    PTI_CUDA(cudaGetLastError(), mod);
    if (total_host) {
        PTI_CUDA(cudaMemcpyAsync(total_host, tmp + ntiles, sizeof(T), cudaMemcpyDeviceToHost, s), mod);
        PTI_CUDA(cudaStreamSynchronize(s), mod);
    }
    return 0;
}

template <class T, class In, class Out>
int scan_apply(In in, Out out, uint64_t n, const T *tmp, cudaStream_t s)
{
    const uint64_t ntiles = (n + kScanTile - 1) / kScanTile;
    if (ntiles == 0) return 0;
    scan_apply_kernel<T, In, Out><<<(unsigned)ntiles, kScanThreads, 0, s>>>(in, n, tmp, out);
    PTI_CUDA(cudaGetLastError(), "B200 scan");
    return 0;
}

// Exclusive scan: calls out(i, prefix_i, in(i)) for every i; returns the total
// through *total_host (synchronous copy) if non-null.
template <class T, class In, class Out>
int exclusive_scan(In in, Out out, uint64_t n, T *tmp, T *total_host, cudaStream_t s)
{
    PTI_TRY((scan_sums<T, In>(in, n, tmp, nullptr, s)));
    PTI_TRY((scan_apply<T, In, Out>(in, out, n, tmp, s)));
    if (total_host) {
        *total_host = 0;
        const uint64_t ntiles = (n + kScanTile - 1) / kScanTile;
        if (ntiles) {
            PTI_CUDA(cudaMemcpyAsync(total_host, tmp + ntiles, sizeof(T), cudaMemcpyDeviceToHost, s), "B200 scan");
            PTI_CUDA(cudaStreamSynchronize(s), "B200 scan");
        }
    }
    return 0;
}

template <class T>
inline size_t scan_tmp_elems(uint64_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

// ---------------------------------------------------------------------------
// Radix sort
// ---------------------------------------------------------------------------
constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // keys per CTA
constexpr int kSortWarps = kSortThreads / 32;

// Ranks of one warp's keys among equal digits, in order: called with the
// digit of this lane's key, it returns how many of the warp's earlier keys
// (earlier calls, then lower lanes) had that digit, and counts this call's
// keys into cnt (256 counters of the warp's own).
__device__ __forceinline__ uint32_t warp_digit_rank(uint32_t digit, uint32_t *cnt)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t peers = __match_any_sync(0xffffffffu, digit);
    const uint32_t first = __ffs(peers) - 1;
    uint32_t old = 0;
    if (lane == first) {
        old = cnt[digit];
        cnt[digit] = old + __popc(peers);
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, old, first) + __popc(peers & ((1u << lane) - 1u));
}

// Turns the warps' digit counts into where each warp's keys of a digit start
// in the CTA's sorted order, and returns thread d's digit's start (256
// threads, one per digit).
__device__ __forceinline__ uint32_t digit_starts(uint32_t (*cnt)[256], uint32_t *s_warp)
{
    const uint32_t d = threadIdx.x;
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = cnt[w][d];
        cnt[w][d] = sum;
        sum += c;
    }
    uint32_t total;
    const uint32_t start = block_exclusive_scan<uint32_t>(sum, s_warp, total);
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) cnt[w][d] += start;
    return start;
}

template <class K>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const K *keys, uint64_t n, int shift,
                                                                  uint32_t ntiles, uint32_t *hist)
{
    __shared__ uint32_t s_hist[256];
    s_hist[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
    uint32_t digit[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint64_t i = base + (uint64_t)r * kSortThreads + threadIdx.x;
        digit[r] = i < n ? (uint32_t)(keys[i] >> shift) & 0xFFu : 0x100u;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r)
        if (digit[r] < 0x100u) atomicAdd(&s_hist[digit[r]], 1u);
    __syncthreads();
    hist[(uint64_t)threadIdx.x * ntiles + blockIdx.x] = s_hist[threadIdx.x];
}

// Stable scatter of a tile by one digit.  Each warp ranks its 512 consecutive
// keys without a CTA barrier, the tile is brought into digit order in shared
// memory, and then written out, so that the keys of a digit leave as one
// contiguous piece: a pass over 10M 64-bit keys with 32-bit values takes
// 83 us, where one barrier per 256 keys and a write per key from where
// it was read took 125.
template <class K>
__global__ void __launch_bounds__(kSortThreads, 3) radix_scatter_kernel(const K *keys_in, const uint32_t *vals_in,
                                                                        uint64_t n, int shift, uint32_t ntiles,
                                                                        const uint32_t *offsets, K *keys_out,
                                                                        uint32_t *vals_out)
{
    extern __shared__ __align__(16) unsigned char sort_smem[];
    K *s_key = reinterpret_cast<K *>(sort_smem);
    uint32_t *s_val = reinterpret_cast<uint32_t *>(s_key + kSortTile);
    uint32_t(*s_cnt)[256] = reinterpret_cast<uint32_t(*)[256]>(s_val + kSortTile);
    uint32_t *s_base = s_cnt[kSortWarps];
    __shared__ uint32_t s_warp[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
    const uint32_t cnt = (uint32_t)((n - base) < (uint64_t)kSortTile ? (n - base) : (uint64_t)kSortTile);
    const uint32_t off = offsets[(uint64_t)tid * ntiles + blockIdx.x];
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s_cnt[w][tid] = 0;
    const uint32_t i0 = warp * (32 * kSortItems) + lane;
    K key[kSortItems];
    uint32_t rank[kSortItems / 2];  // two 16-bit ranks a word
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t i = i0 + 32 * r;
        // past the end: the largest digit, behind every key of the tile
        key[r] = i < cnt ? keys_in[base + i] : ~K(0);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; r += 2) {
        const uint32_t lo = warp_digit_rank((uint32_t)(key[r] >> shift) & 0xFFu, s_cnt[warp]);
        rank[r / 2] = lo | warp_digit_rank((uint32_t)(key[r + 1] >> shift) & 0xFFu, s_cnt[warp]) << 16;
    }
    uint32_t val[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) val[r] = i0 + 32 * r < cnt ? vals_in[base + i0 + 32 * r] : 0u;
    __syncthreads();
    s_base[tid] = off - digit_starts(s_cnt, s_warp);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t pos = s_cnt[warp][(uint32_t)(key[r] >> shift) & 0xFFu] + (rank[r / 2] >> (16 * (r & 1)) & 0xFFFFu);
        s_key[pos] = key[r];
        s_val[pos] = val[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t i = r * kSortThreads + tid;
        if (i < cnt) {
            const K k = s_key[i];
            const uint32_t out = s_base[(uint32_t)(k >> shift) & 0xFFu] + i;
            keys_out[out] = k;
            vals_out[out] = s_val[i];
        }
    }
}

// Stable LSD sort of (keys, vals) on bits [0, nbits) of the keys (unsigned 32-
// or 64-bit).  The result ends in (keys, vals); (keys_alt, vals_alt) are
// scratch of the same size.
template <class K>
struct RadixScratchT {
    DevBuf keys_alt, vals_alt, hist, scan_tmp;
    int alloc(uint64_t n, cudaStream_t s)
    {
        const char *mod = "B200 sort";
        uint64_t ntiles = (n + kSortTile - 1) / kSortTile;
        PTI_CUDA(keys_alt.alloc(padded(n * sizeof(K)), s), mod);
        PTI_CUDA(vals_alt.alloc(padded(n * 4), s), mod);
        PTI_CUDA(hist.alloc(padded(256 * ntiles * 4), s), mod);
        PTI_CUDA(scan_tmp.alloc(padded(scan_tmp_elems<uint32_t>(256 * ntiles) * 4), s), mod);
        return 0;
    }
};
using RadixScratch = RadixScratchT<uint64_t>;

struct HistIn {
    const uint32_t *h;
    __device__ uint32_t operator()(uint64_t i) const { return h[i]; }
};
struct HistOut {
    uint32_t *h;
    __device__ void operator()(uint64_t i, uint32_t prefix, uint32_t) const { h[i] = prefix; }
};

// Sorts (keys, vals) in place (the buffers may be exchanged with the
// scratch ones, so callers must re-read keys.ptr / vals.ptr afterwards).
template <class K>
int radix_sort_pairs(DevBuf &keys, DevBuf &vals, uint64_t n, int nbits, RadixScratchT<K> &sc, cudaStream_t s)
{
    const char *mod = "B200 sort";
    if (n <= 1 || nbits <= 0) return 0;
    PTI_CHECK(n < 0xFFFFFFFFull, PTIERR_VALUE_ERROR, mod, "too many keys");
    uint32_t ntiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
    uint32_t *hist = sc.hist.template as<uint32_t>();
    constexpr size_t smem = (size_t)kSortTile * (sizeof(K) + 4) + (kSortWarps + 1) * 256 * 4;
    PTI_CUDA(cudaFuncSetAttribute(radix_scatter_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), mod);
    for (int shift = 0; shift < nbits; shift += 8) {
        radix_hist_kernel<K><<<ntiles, kSortThreads, 0, s>>>(keys.as<K>(), n, shift, ntiles, hist);
        PTI_TRY((exclusive_scan<uint32_t>(HistIn{hist}, HistOut{hist}, 256ull * ntiles,
                                          sc.scan_tmp.template as<uint32_t>(), nullptr, s)));
        radix_scatter_kernel<K><<<ntiles, kSortThreads, smem, s>>>(keys.as<K>(), vals.as<uint32_t>(), n, shift, ntiles,
                                                                   hist, sc.keys_alt.template as<K>(),
                                                                   sc.vals_alt.template as<uint32_t>());
        PTI_CUDA(cudaGetLastError(), mod);
        keys.swap(sc.keys_alt);
        vals.swap(sc.vals_alt);
    }
    return 0;
}

}  // namespace pti
