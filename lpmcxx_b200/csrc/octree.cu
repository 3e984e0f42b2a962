// Device octree with the reference's leaf membership.
//
// The reference builds its tree recursively (src/LpmTreeSum.cpp:266-290, src/LpmOctree.cpp:84-143):
// a node whose point count exceeds the leaf capacity is bisected at 0.5*(min+max) along all three
// axes in FP64 (src/LpmBox3d.cpp:140-151), points go to the child whose half-open box contains them
// (src/LpmBox3d.h:37-39), children are ordered ix + 2 iy + 4 iz and empty children are dropped.
//
// Here every point gets a 63-bit key that replays exactly those FP64 midpoint comparisons for 21
// levels (bit 63 set = outside the root box), the (key, index) pairs are radix sorted, and nodes are
// key ranges split level by level on the GPU: a node at level l with more than max_per_leaf points
// splits into the non-empty ranges of its points' level-(l+1) digits.  Sorted order is the
// reference's depth-first order, so leaves sorted by range start are its leaves in DFS order.
//
// The short dependent phases (the passes of a sort of up to 131,072 keys, the levels of the split, the leaf
// numbering) each run as ONE launch of a single thread-block cluster, whose blocks meet at the hardware cluster
// barrier (release / acquire, so the global memory they write is visible across it) instead of at launch boundaries.
#include "octree.h"

#include <algorithm>

namespace lpm {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096 items per block
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int32_t warp_incl_scan(int32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive scan of one value per thread over a block of up to 1024 threads; returns the block total.
__device__ int32_t block_excl_scan(int32_t v, int32_t* total) {
    __shared__ int32_t warp_sums[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    const int32_t incl = warp_incl_scan(v);
    if (lane == 31) warp_sums[w] = incl;
    __syncthreads();
    if (w == 0) {
        int32_t s = lane < nw ? warp_sums[lane] : 0;
        s = warp_incl_scan(s);
        if (lane < nw) warp_sums[lane] = s;
    }
    __syncthreads();
    const int32_t base = w ? warp_sums[w - 1] : 0;
    const int32_t tot = warp_sums[nw - 1];
    __syncthreads();
    if (total) *total = tot;
    return base + incl - v;
}

// ---------------------------------------------------------------------------------- scan
__global__ void scan_block_sums_kernel(const int32_t* __restrict__ in, int64_t n, int32_t* __restrict__ sums) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    int32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + k * kScanThreads + threadIdx.x;
        if (i < n) s += in[i];
    }
    int32_t tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// In-place exclusive scan of m values by one block; writes the total to *total if given.
__global__ void scan_single_block_kernel(int32_t* __restrict__ data, int64_t m, int32_t* __restrict__ total) {
    const int64_t per = (m + blockDim.x - 1) / blockDim.x;
    const int64_t b = threadIdx.x * per, e = min(b + per, m);
    int32_t s = 0;
    for (int64_t i = b; i < e; ++i) s += data[i];
    int32_t tot;
    int32_t run = block_excl_scan(s, &tot);
    for (int64_t i = b; i < e; ++i) {
        const int32_t v = data[i];
        data[i] = run;
        run += v;
    }
    if (threadIdx.x == 0 && total) *total = tot;
}

__global__ void scan_apply_kernel(const int32_t* __restrict__ in, int32_t* __restrict__ out, int64_t n,
                                  const int32_t* __restrict__ sums) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    int32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    int32_t run = block_excl_scan(s, nullptr) + sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
}

// ---------------------------------------------------------------------------------- one cluster
constexpr int kClBlocks = 8;  // portable cluster size
constexpr int kClThreads = 1024;
constexpr int kClWarps = kClBlocks * kClThreads / 32;

// The block's total v over all blocks (*total) and over the blocks of lower rank (returned).  One cluster barrier
// inside; `slot` (one int of shared memory) may be written again only after the next one.
__device__ __forceinline__ int32_t cluster_excl(int32_t v, int32_t* slot, int rank, int32_t* total) {
    if (threadIdx.x == 0) *slot = v;
    cluster_barrier();
    int32_t before = 0, all = 0;
#pragma unroll
    for (int r = 0; r < kClBlocks; ++r) {
        const int32_t t = cluster_load(slot, r);
        all += t;
        before += r < rank ? t : 0;
    }
    *total = all;
    return before;
}

// In-place exclusive scan of m counts (a multiple of 4, 16-byte aligned) by one cluster: a warp's consecutive runs of
// 128 are summed, the warp sums scanned over the block and the cluster, and the runs scanned on their second read.
__global__ void __cluster_dims__(kClBlocks, 1, 1) __launch_bounds__(kClThreads)
    cluster_scan_kernel(int32_t* __restrict__ data, int m) {
    __shared__ int32_t slot, warp_base[kClThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rank = (int)blockIdx.x;
    const int per = (m + 128 * kClWarps - 1) / (128 * kClWarps);  // runs a warp
    const int b = (rank * (kClThreads / 32) + w) * per;
    int4* const d4 = (int4*)data;
    int32_t sum = 0;
    for (int r = b; r < b + per; ++r) {
        const int i = 32 * r + lane;
        const int4 v = 4 * i < m ? d4[i] : make_int4(0, 0, 0, 0);
        sum += v.x + v.y + v.z + v.w;
    }
    sum = warp_incl_scan(sum);
    if (lane == 31) warp_base[w] = sum;
    __syncthreads();
    int32_t block_total = 0, all = 0;
    const int32_t mine = threadIdx.x < kClThreads / 32 ? warp_base[threadIdx.x] : 0;
    int32_t base = block_excl_scan(mine, &block_total);
    base += cluster_excl(block_total, &slot, rank, &all);
    if (threadIdx.x < kClThreads / 32) warp_base[threadIdx.x] = base;
    __syncthreads();
    int32_t run = warp_base[w];
    for (int r = b; r < b + per; ++r) {
        const int i = 32 * r + lane;
        int4 v = 4 * i < m ? d4[i] : make_int4(0, 0, 0, 0);
        const int32_t s = v.x + v.y + v.z + v.w, incl = warp_incl_scan(s);
        int32_t at = run + incl - s;
        const int32_t x = v.x, y = v.y, z = v.z;
        v.x = at;
        v.y = at += x;
        v.z = at += y;
        v.w = at + z;
        if (4 * i < m) d4[i] = v;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    cluster_barrier();  // no block leaves while another reads its total
}

// ---------------------------------------------------------------------------------- radix sort
template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const K* __restrict__ keys, int64_t n, int shift,
                                                                  int32_t* __restrict__ counts, int nblocks) {
    __shared__ int32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    int d[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const int64_t i = base + k * kSortThreads + threadIdx.x;
        d[k] = i < n ? (int)((keys[i] >> shift) & 255) : -1;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; ++k)
        if (d[k] >= 0) atomicAdd(&h[d[k]], 1);
    __syncthreads();
    counts[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter: warp w of a block owns items [w*512, (w+1)*512) of the block's tile and walks them
// in chunks of 32; __match_any_sync groups equal digits inside a chunk.
template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(const K* __restrict__ kin,
                                                                     const int32_t* __restrict__ vin,
                                                                     K* __restrict__ kout, int32_t* __restrict__ vout,
                                                                     int64_t n, int shift,
                                                                     const int32_t* __restrict__ offsets,
                                                                     int nblocks) {
    constexpr int kWarps = kSortThreads / 32;
    constexpr int kPerWarp = kSortTile / kWarps;
    __shared__ int32_t wh[kWarps][256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < kWarps * 256; d += kSortThreads) (&wh[0][0])[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile + (int64_t)w * kPerWarp;
    const unsigned lt = (1u << lane) - 1u;
    for (int c = 0; c < kPerWarp / 32; ++c) {
        const int64_t i = base + c * 32 + lane;
        const bool valid = i < n;
        const int d = valid ? (int)((kin[i] >> shift) & 255) : 256;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        if (valid && lane == __ffs(peers) - 1) wh[w][d] += __popc(peers);
    }
    __syncthreads();
    {
        const int d = threadIdx.x;  // 256 threads, one per digit
        int32_t run = offsets[(int64_t)d * nblocks + blockIdx.x];
#pragma unroll
        for (int q = 0; q < kWarps; ++q) {
            const int32_t t = wh[q][d];
            wh[q][d] = run;
            run += t;
        }
    }
    __syncthreads();
    for (int c = 0; c < kPerWarp / 32; ++c) {
        const int64_t i = base + c * 32 + lane;
        const bool valid = i < n;
        K key = 0;
        int d = 256;
        if (valid) {
            key = kin[i];
            d = (int)((key >> shift) & 255);
        }
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int32_t pos = valid ? wh[w][d] + __popc(peers & lt) : 0;
        __syncwarp();
        if (valid) {
            kout[pos] = key;
            vout[pos] = vin[i];
            if (lane == __ffs(peers) - 1) wh[w][d] += __popc(peers);
        }
        __syncwarp();
    }
}

// ---- packed keys: the sorted bits in the upper 32, the item's index in the lower 32 (morton_keys_kernel writes them so
// where no lower key bit is sorted or read), so that a pass moves 8 bytes an item instead of 12 and reads them once:
// a thread keeps its keys and their ranks in registers, the block orders its tile in shared memory and writes it out in
// runs of equal digits.

// The lanes holding the same 8-bit digit as this one among the lanes of `valid`, from one ballot per bit: the match
// instruction serialises over the distinct digits of a warp (1 us per 32 keys with 32 warps on an SM, 7 of the 12 us of
// a pass over 50,000 keys), eight ballots do not.
__device__ __forceinline__ unsigned digit_peers(int d, unsigned valid) {
    unsigned peers = valid;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool one = (d >> b) & 1;
        const unsigned m = __ballot_sync(0xffffffffu, one);
        peers &= one ? m : ~m;
    }
    return peers;
}

// Ranks of a warp's keys (key[j] at position 32 j + lane of its segment of `per` items, `n` of them valid) among its keys
// of the same digit, in segment order, two 16-bit ranks a word; the warp's digit counts are left in wh (zeroed before).
template <int ITEMS>
__device__ __forceinline__ void warp_ranks(const uint64_t (&key)[ITEMS], int per, int n, int shift, int32_t* wh,
                                           uint32_t (&rank2)[(ITEMS + 1) / 2]) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (j % 2 == 0) rank2[j / 2] = 0;
        if (32 * j >= per) continue;  // warp-uniform
        const bool valid = 32 * j + lane < n;
        const int d = (int)((key[j] >> shift) & 255);
        const unsigned peers = digit_peers(d, __ballot_sync(0xffffffffu, valid));
        const int32_t before = valid ? wh[d] : 0;
        __syncwarp();
        if (valid && (peers & lt) == 0) wh[d] = before + __popc(peers);
        __syncwarp();
        rank2[j / 2] |= (uint32_t)(before + __popc(peers & lt)) << (16 * (j % 2));
    }
}

// The whole LSD sort of n <= ITEMS x 8192 packed keys by one cluster: every pass ranks, exchanges the blocks' digit
// counts through distributed shared memory and writes, two cluster barriers a pass instead of three to five launches.
// The last pass writes perm too.  Bound by the latency of its phases (one global round trip, 256-digit scans, two
// barriers); 8 SMs suffice up to 131,072 keys, above that the many-block passes below are faster.
template <int ITEMS>
struct ClusterSortShape {
    static constexpr int kWarps = kClThreads / 32;
    static constexpr size_t kSmem = sizeof(uint64_t) * ITEMS * kClThreads + sizeof(int32_t) * (kWarps * 256 + 3 * 256);
};
template <int ITEMS>
__global__ void __cluster_dims__(kClBlocks, 1, 1) __launch_bounds__(kClThreads)
    cluster_sort_kernel(uint64_t* __restrict__ keys, uint64_t* __restrict__ tk, int32_t* __restrict__ perm, int n,
                        int bit_lo) {
    constexpr int kW = kClThreads / 32;
    extern __shared__ __align__(16) uint64_t tile[];
    int32_t* const wh = (int32_t*)(tile + ITEMS * kClThreads);  // [warp][digit]
    int32_t* const tot = wh + kW * 256;
    int32_t* const start = tot + 256;  // the block's first position of each digit
    int32_t* const out = start + 256;  // global position of a digit's first key of this block, minus `start`
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rank = (int)blockIdx.x;
    const int per = ((n + kClWarps * 32 - 1) / (kClWarps * 32)) * 32;  // keys per warp, at most 32 ITEMS
    const int b0 = min(n, rank * kW * per), bn = min(n - b0, kW * per);  // this block's keys
    const int wn = max(0, min(bn - w * per, per));                       // this warp's
    uint64_t *ks = keys, *kd = tk;
    for (int shift = bit_lo; shift < 64; shift += 8) {
        for (int d = threadIdx.x; d < kW * 256; d += kClThreads) wh[d] = 0;
        uint64_t key[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            key[j] = 32 * j + lane < wn ? __ldcg(ks + b0 + w * per + 32 * j + lane) : 0;
        __syncthreads();
        uint32_t rank2[(ITEMS + 1) / 2];
        warp_ranks<ITEMS>(key, per, wn, shift, wh + w * 256, rank2);
        __syncthreads();
        if (threadIdx.x < 256) {
            const int d = threadIdx.x;
            int32_t run = 0;
#pragma unroll
            for (int q = 0; q < kW; ++q) {
                const int32_t t = wh[q * 256 + d];
                wh[q * 256 + d] = run;
                run += t;
            }
            tot[d] = run;
        }
        cluster_barrier();
        int32_t before = 0, all = 0, own = 0;
        if (threadIdx.x < 256) {
            own = tot[threadIdx.x];
#pragma unroll
            for (int r = 0; r < kClBlocks; ++r) {
                const int32_t t = cluster_load(&tot[threadIdx.x], r);
                all += t;
                before += r < rank ? t : 0;
            }
        }
        const int32_t base = block_excl_scan(all, nullptr), first = block_excl_scan(own, nullptr);
        if (threadIdx.x < 256) {
            start[threadIdx.x] = first;
            out[threadIdx.x] = base + before - first;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const int d = (int)((key[j] >> shift) & 255);
            if (32 * j + lane < wn)
                tile[start[d] + wh[w * 256 + d] + (int)((rank2[j / 2] >> (16 * (j % 2))) & 0xffffu)] = key[j];
        }
        __syncthreads();
        const bool last = shift + 8 >= 64;
        for (int i = threadIdx.x; i < bn; i += kClThreads) {
            const uint64_t k = tile[i];
            const int pos = out[(int)((k >> shift) & 255)] + i;
            kd[pos] = k;
            if (last) perm[pos] = (int32_t)(uint32_t)k;
        }
        cluster_barrier();  // this pass's output is complete, and every block has read the others' totals
        uint64_t* const kt = ks;
        ks = kd;
        kd = kt;
    }
    if (ks != keys)  // an odd number of passes
        for (int i = rank * kClThreads + threadIdx.x; i < n; i += kClBlocks * kClThreads) keys[i] = __ldcg(ks + i);
}

// One scatter pass over packed keys, many blocks: a tile of kSortTile keys per block, `offsets` (digit-major, scanned)
// its digits' global positions.  perm, if not null (the last pass), receives the indices.
__global__ void __launch_bounds__(kSortThreads) packed_scatter_kernel(const uint64_t* __restrict__ kin,
                                                                      uint64_t* __restrict__ kout,
                                                                      int32_t* __restrict__ perm, int64_t n, int shift,
                                                                      const int32_t* __restrict__ offsets,
                                                                      int nblocks) {
    constexpr int kW = kSortThreads / 32, kPer = kSortTile / kW, kI = kSortItems;
    static_assert(kPer == 32 * kI && kSortThreads == 256, "a warp's segment is kSortItems keys per lane");
    __shared__ uint64_t tile[kSortTile];
    __shared__ int32_t wh[kW][256], start[256], out[256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < kW * 256; d += kSortThreads) (&wh[0][0])[d] = 0;
    const int64_t b0 = (int64_t)blockIdx.x * kSortTile;
    const int bn = (int)min((int64_t)kSortTile, n - b0), wn = max(0, min(bn - w * kPer, kPer));
    uint64_t key[kI];
#pragma unroll
    for (int j = 0; j < kI; ++j) key[j] = 32 * j + lane < wn ? kin[b0 + w * kPer + 32 * j + lane] : 0;
    __syncthreads();
    uint32_t rank2[(kI + 1) / 2];
    warp_ranks<kI>(key, kPer, wn, shift, wh[w], rank2);
    __syncthreads();
    int32_t run = 0;
    {
        const int d = threadIdx.x;
#pragma unroll
        for (int q = 0; q < kW; ++q) {
            const int32_t t = wh[q][d];
            wh[q][d] = run;
            run += t;
        }
    }
    const int32_t first = block_excl_scan(run, nullptr);
    start[threadIdx.x] = first;
    out[threadIdx.x] = offsets[(int64_t)threadIdx.x * nblocks + blockIdx.x] - first;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kI; ++j) {
        const int d = (int)((key[j] >> shift) & 255);
        if (32 * j + lane < wn) tile[start[d] + wh[w][d] + (int)((rank2[j / 2] >> (16 * (j % 2))) & 0xffffu)] = key[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < bn; i += kSortThreads) {
        const uint64_t k = tile[i];
        const int pos = out[(int)((k >> shift) & 255)] + i;
        kout[pos] = k;
        if (perm) perm[pos] = (int32_t)(uint32_t)k;
    }
}

// Digit counts of every tile to global offsets.  One launch where the counts allow it: a block for up to 4096 (4.4 us
// against 6.3 us by a cluster; 10.4 and 20.8 us at 8,192 and 16,384), a cluster up to 2^19 (6.4 us at 65,536 counts, the
// 1M keys of a pass, against 12.4 us back to back by the three launches; equal at 2^19, 20.9 against 16.5 us at 2^20).
constexpr int64_t kBlockScanMax = 4096, kClusterScanMax = 1 << 19;
int digit_offsets(lpm_ctx* ctx, int32_t* counts, int64_t m, int sums_slot) {
    if (m > kClusterScanMax) return scan_exclusive_i32(ctx, counts, counts, m, nullptr, sums_slot);
    if (m > kBlockScanMax)
        LPM_LAUNCH(ctx, "cluster_scan_kernel", cluster_scan_kernel, kClBlocks, kClThreads, 0, counts, (int)m);
    else
        LPM_LAUNCH(ctx, "scan_single_block_kernel", scan_single_block_kernel, 1, 1024, 0, counts, m, (int32_t*)nullptr);
    return LPM_OK;
}

template <int ITEMS>
int cluster_sort(lpm_ctx* ctx, uint64_t* keys, uint64_t* tk, int32_t* perm, int64_t n, int bit_lo) {
    constexpr size_t smem = ClusterSortShape<ITEMS>::kSmem;
    LPM_CUDA_TRY(cudaFuncSetAttribute(cluster_sort_kernel<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    LPM_LAUNCH(ctx, "cluster_sort_kernel", cluster_sort_kernel<ITEMS>, kClBlocks, kClThreads, smem, keys, tk, perm,
               (int)n, bit_lo);
    return LPM_OK;
}

constexpr int64_t kClusterSortMax = 16 * kClBlocks * kClThreads;

template <typename K>
int radix_sort_impl(lpm_ctx* ctx, K* keys, int32_t* vals, K* tk, int32_t* tv, int64_t n, int bit_lo, int bit_hi,
                    int counts_slot, int sums_slot) {
    if (n <= 1) return LPM_OK;
    const int nblocks = (int)((n + kSortTile - 1) / kSortTile);
    int32_t* counts = (int32_t*)scratch(ctx, counts_slot, sizeof(int32_t) * 256 * (size_t)nblocks);
    if (!counts) return LPM_ERR_OOM;
    K* src_k = keys;
    int32_t* src_v = vals;
    K* dst_k = tk;
    int32_t* dst_v = tv;
    for (int shift = bit_lo; shift < bit_hi; shift += 8) {
        LPM_LAUNCH(ctx, "radix_hist_kernel", radix_hist_kernel<K>, nblocks, kSortThreads, 0, src_k, n, shift, counts,
                   nblocks);
        const int rc = digit_offsets(ctx, counts, (int64_t)256 * nblocks, sums_slot);
        if (rc) return rc;
        LPM_LAUNCH(ctx, "radix_scatter_kernel", radix_scatter_kernel<K>, nblocks, kSortThreads, 0, src_k, src_v, dst_k,
                   dst_v, n, shift, counts, nblocks);
        std::swap(src_k, dst_k);
        std::swap(src_v, dst_v);
    }
    if (src_k != keys) {
        LPM_CUDA_TRY(cudaMemcpyAsync(keys, src_k, sizeof(K) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream));
        LPM_CUDA_TRY(cudaMemcpyAsync(vals, src_v, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream));
    }
    return LPM_OK;
}

// ---------------------------------------------------------------------------------- keys
// Packed keys keep 32 bits of the key, which are 11 of the 21 levels' digits.  The count of points inside goes out once
// a block: one addition a warp, all on the same address, took half the time of 1M points (38 -> 24 us with both).
constexpr int kPackedLevels = (31 + 2) / 3;
static_assert(3 * (kKeyLevels - kPackedLevels) <= 32, "the levels left out lie in the lower half of the key");
__global__ void morton_keys_kernel(const double4* __restrict__ pts, int64_t n, RootBox root,
                                   uint64_t* __restrict__ keys, int32_t* __restrict__ vals,
                                   int32_t* __restrict__ counters, int bits, int max_depth, bool packed) {
    const int levels = packed ? kPackedLevels : kKeyLevels;  // (bits == 1 stops at max_depth)
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    root = resolve_root(root);
    bool in = false;
    if (i < n) {
        const double4 p = pts[i];
        const double c[3] = {p.x, p.y, p.z};
        in = root.lo[0] <= c[0] && c[0] < root.hi[0] && root.lo[1] <= c[1] && c[1] < root.hi[1] &&
             root.lo[2] <= c[2] && c[2] < root.hi[2];
        uint64_t key = kKeyOutside;
        if (in && bits == 1) {  // binary: level l bisects axis (l + 1) mod 3 (the Sakajo tree's (j + 2) mod 3, j = l - 1)
            double lo[3] = {root.lo[0], root.lo[1], root.lo[2]};
            double hi[3] = {root.hi[0], root.hi[1], root.hi[2]};
            key = 0;
            for (int l = 1; l <= max_depth; ++l) {
                const int a = (l + 1) % 3;
                const double mid = 0.5 * (lo[a] + hi[a]);  // Box3d::bisectAlongDims midpoint
                if (c[a] < mid) {
                    hi[a] = mid;
                } else {
                    lo[a] = mid;
                    key |= 1ull << (kMaxLevels - l);
                }
            }
        } else if (in) {
            double lo[3] = {root.lo[0], root.lo[1], root.lo[2]};
            double hi[3] = {root.hi[0], root.hi[1], root.hi[2]};
            key = 0;
            for (int l = 1; l <= levels; ++l) {
                uint64_t digit = 0;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const double mid = 0.5 * (lo[a] + hi[a]);  // Box3d::bisectAll midpoint
                    if (c[a] < mid) {
                        hi[a] = mid;
                    } else {
                        lo[a] = mid;
                        digit |= 1ull << a;
                    }
                }
                key |= digit << (3 * (kKeyLevels - l));
            }
        }
        if (packed) {
            keys[i] = (key & ~0xffffffffull) | (uint64_t)i;
        } else {
            keys[i] = key;
            vals[i] = (int32_t)i;
        }
    }
    const int inside = __syncthreads_count(in);
    if (threadIdx.x == 0 && inside) atomicAdd(&counters[0], inside);
}

__global__ void root_extent_kernel(const double4* __restrict__ pts, int64_t first, int64_t n, int mode,
                                   unsigned long long* __restrict__ r_dev) {
    unsigned long long m = 0;  // non-negative doubles order like their bit patterns
    for (int64_t i = first + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double4 p = pts[i];
        const double v = mode == kRootMaxNorm ? fmax(fabs(p.x), fmax(fabs(p.y), fabs(p.z)))
                                              : __dadd_rn(__dadd_rn(__dmul_rn(p.x, p.x), __dmul_rn(p.y, p.y)),
                                                          __dmul_rn(p.z, p.z));
        const unsigned long long b = (unsigned long long)__double_as_longlong(v);
        m = b > m ? b : m;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_xor_sync(0xffffffffu, m, o);
        m = u > m ? u : m;
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax(r_dev, m);
}

__device__ __forceinline__ int level_digit(uint64_t key, int level, int bits) {
    return bits == 1 ? (int)((key >> (kMaxLevels - level)) & 1ull) : (int)((key >> (3 * (kKeyLevels - level))) & 7ull);
}

// Box of child digit d of a level-l node (box pb): all three axes for octrees (ix + 2 iy + 4 iz), axis
// (l + 2) mod 3 for binary trees.
__device__ __forceinline__ void child_box(const double* pb, int l, int d, int bits, double* cb) {
    for (int a = 0; a < 3; ++a) {
        const double mid = 0.5 * (pb[2 * a] + pb[2 * a + 1]);
        const bool split = bits == 3 || a == (l + 2) % 3;
        const bool upper = bits == 3 ? ((d >> a) & 1) : (d & 1);
        cb[2 * a] = split && upper ? mid : pb[2 * a];
        cb[2 * a + 1] = split && !upper ? mid : pb[2 * a + 1];
    }
}

// Box3d::intersectsSphere about the origin (src/LpmBox3d.cpp:79-129): the box's closest point lies inside
// the sphere and its farthest corner outside (distances sqrt((x x + y y) + z z), rounded step by step).
__device__ __forceinline__ double mag3(double x, double y, double z) {
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z)));
}
__device__ bool box_meets_sphere(const double* b, double r) {
    double c[3];
    const bool inside = b[0] <= 0.0 && 0.0 < b[1] && b[2] <= 0.0 && 0.0 < b[3] && b[4] <= 0.0 && 0.0 < b[5];
    for (int a = 0; a < 3; ++a) {
        const double lo = b[2 * a], hi = b[2 * a + 1];
        c[a] = inside ? 0.0 : (lo == hi ? lo : (lo >= 0.0 ? lo : (hi <= 0.0 ? hi : 0.0)));
    }
    double far = 0.0;
    for (int k = 0; k < 8; ++k) {
        const double d = mag3(b[(k & 1) ? 1 : 0], b[(k & 2) ? 3 : 2], b[(k & 4) ? 5 : 4]);
        far = d > far ? d : far;
    }
    return mag3(c[0], c[1], c[2]) <= r && far >= r;
}

// The first position in [s, e) of the sorted keys whose level-l digit is >= d (e if there is none).
__device__ __forceinline__ int digit_bound(const uint64_t* __restrict__ keys, int s, int e, int l, int d, int bits) {
    while (s < e) {
        const int mid = (s + e) >> 1;
        if (level_digit(keys[mid], l, bits) < d) s = mid + 1;
        else e = mid;
    }
    return s;
}
// The same found by a whole warp: a 32-ary search (32 probes per round, ~4 rounds for a million keys instead of ~20
// dependent probes of a binary search).
__device__ __forceinline__ int digit_bound_warp(const uint64_t* __restrict__ keys, int s, int e, int l, int d,
                                                int bits) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    int lo = s, hi = e;  // the boundary b satisfies lo <= b <= hi; positions lo..hi-1 are keys
    while (hi - lo > 32) {
        const int64_t L = hi - lo;
        const int p = lo + (int)(((int64_t)lane * L) >> 5);
        const unsigned below = __ballot_sync(full, level_digit(keys[p], l, bits) < d);
        const int c = __popc(below);  // probes 0..c-1 lie below the boundary (digits are sorted)
        const int nlo = c == 0 ? lo : lo + (int)(((int64_t)(c - 1) * L) >> 5) + 1;
        const int nhi = c == 32 ? hi : lo + (int)(((int64_t)c * L) >> 5);
        lo = nlo;
        hi = nhi;
    }
    const bool less = lane < hi - lo && level_digit(keys[lo + lane], l, bits) < d;
    return lo + __popc(__ballot_sync(full, less));
}

// The nodes of the sorted keys, level by level, and the leaf numbering, by one cluster.  A level takes two steps: the
// boundaries of every split node's child digits (one warp per boundary while the level has few nodes, one thread
// per boundary after), then the child counts' prefix sum (block totals through distributed shared memory) and the
// children.  Levels stop at the first that splits no node.  Then, level by level again, the leaves below every node
// are counted upwards and numbered downwards: leaves in depth-first order are numbered by their nodes' order, no
// pass over the points.  `pending`, if not null, receives every node's number of internal children (-1 for an internal
// node whose children are all leaves).
__global__ void __cluster_dims__(kClBlocks, 1, 1) __launch_bounds__(kClThreads)
    tree_nodes_kernel(Octree t, int32_t* __restrict__ pending) {
    __shared__ int32_t slot[2];
    __shared__ int32_t level_begin[kMaxLevels + 3];
    const int rank = (int)blockIdx.x, tid = rank * kClThreads + (int)threadIdx.x, lane = threadIdx.x & 31;
    constexpr int kAll = kClBlocks * kClThreads;
    const int nd = 1 << t.bits;  // digits per level
    const int n_valid = t.counters[0];
    if (tid == 0) {
        t.node_start[0] = 0;
        t.node_end[0] = n_valid;
        t.node_parent[0] = -1;
        t.node_first_child[0] = -1;
        t.node_nchild[0] = 0;
        t.node_level[0] = 0;
        const RootBox root = resolve_root(t.root);
        for (int a = 0; a < 3; ++a) {
            t.node_box[2 * a] = root.lo[a];
            t.node_box[2 * a + 1] = root.hi[a];
        }
    }
    if (threadIdx.x == 0) {
        level_begin[0] = 0;
        level_begin[1] = 1;
    }
    int lb = 0, le = 1, depth = 0;
    int32_t flags = 0;
    cluster_barrier();
    for (int l = 0; l < t.max_depth; ++l) {
        const int m = le - lb;
        // boundaries 1 .. nd - 1 of every node that splits
        if (m * (nd - 1) <= 2 * kClWarps) {
            for (int q = tid >> 5; q < m * (nd - 1); q += kClWarps) {
                const int i = q / (nd - 1), d = q - i * (nd - 1) + 1;
                const int s = __ldcg(t.node_start + lb + i), e = __ldcg(t.node_end + lb + i);
                if (e - s > t.max_per_leaf) {  // warp-uniform
                    const int at = digit_bound_warp(t.keys, s, e, l + 1, d, t.bits);
                    if (lane == 0) t.child_start[(int64_t)i * 9 + d] = at;
                }
            }
        } else {
            for (int64_t q = tid; q < (int64_t)m * (nd - 1); q += kAll) {
                const int i = (int)(q / (nd - 1)), d = (int)(q - (int64_t)i * (nd - 1)) + 1;
                const int s = __ldcg(t.node_start + lb + i), e = __ldcg(t.node_end + lb + i);
                if (e - s > t.max_per_leaf)
                    t.child_start[(int64_t)i * 9 + d] = digit_bound(t.keys, s, e, l + 1, d, t.bits);
            }
        }
        cluster_barrier();
        // child counts of this block's nodes, block by block in node order, and their prefix sum
        const int chunk = (m + kClBlocks - 1) / kClBlocks, cb = min(m, rank * chunk), ce = min(m, cb + chunk);
        const int per = (ce - cb + kClThreads - 1) / kClThreads;
        const int b = min(ce, cb + (int)threadIdx.x * per), e = min(ce, b + per);
        // the boundaries of node lb + i in cs[0 .. nd]; the kept children, as bits
        auto children = [&](int i, int* cs) -> unsigned {
            const int s = __ldcg(t.node_start + lb + i), en = __ldcg(t.node_end + lb + i);
            if (en - s <= t.max_per_leaf) return 0u;
            cs[0] = s;
            cs[nd] = en;
            for (int d = 1; d < nd; ++d) cs[d] = __ldcg(t.child_start + (int64_t)i * 9 + d);
            unsigned keep = 0;
            for (int d = 0; d < nd; ++d) {
                if (cs[d + 1] <= cs[d]) continue;
                if (t.sphere_r > 0.0) {
                    double pb[6], cbox[6];
                    for (int a = 0; a < 6; ++a) pb[a] = __ldcg(t.node_box + 6 * (int64_t)(lb + i) + a);
                    child_box(pb, l, d, t.bits, cbox);
                    if (!box_meets_sphere(cbox, t.sphere_r)) continue;
                }
                keep |= 1u << d;
            }
            return keep;
        };
        int cs[9];
        unsigned keep = 0;  // of the last node looked at: with one node a thread it is not formed again
        int32_t mine = 0;
        for (int i = b; i < e; ++i) mine += __popc(keep = children(i, cs));
        int32_t block_total = 0, total = 0;
        int32_t run = block_excl_scan(mine, &block_total);
        run += le + cluster_excl(block_total, &slot[l & 1], rank, &total);
        const bool fits = (int64_t)le + total <= t.node_cap;
        if (!fits) flags |= 2;  // node capacity exhausted: the level's nodes stay leaves
        for (int i = b; i < e && fits; ++i) {
            const int node = lb + i;
            if (e - b > 1) keep = children(i, cs);
            const int nc = __popc(keep);
            if (nc == 0) continue;
            t.node_first_child[node] = run;
            t.node_nchild[node] = (int8_t)nc;
            double pb[6], cbox[6];
            for (int a = 0; a < 6; ++a) pb[a] = __ldcg(t.node_box + 6 * (int64_t)node + a);
            int k = run;
            for (int d = 0; d < nd; ++d) {
                if (!((keep >> d) & 1u)) continue;
                child_box(pb, l, d, t.bits, cbox);
                t.node_start[k] = cs[d];
                t.node_end[k] = cs[d + 1];
                t.node_parent[k] = node;
                t.node_first_child[k] = -1;
                t.node_nchild[k] = 0;
                t.node_level[k] = (int8_t)(l + 1);
                for (int a = 0; a < 6; ++a) t.node_box[6 * (int64_t)k + a] = cbox[a];
                ++k;
            }
            run += nc;
        }
        const int next = fits ? total : 0;
        if (threadIdx.x == 0) level_begin[l + 2] = le + next;
        lb = le;
        le += next;
        cluster_barrier();  // the children are visible to every block
        if (next == 0) break;  // uniform over the cluster
        depth = l + 1;
    }
    // leaves below every node, upwards
    for (int l = depth; l >= 0; --l) {
        for (int node = level_begin[l] + tid; node < level_begin[l + 1]; node += kAll) {
            const int nc = __ldcg(t.node_nchild + node), fc = __ldcg(t.node_first_child + node);
            int leaves = nc == 0, internal = 0;
            for (int k = 0; k < nc; ++k) {
                leaves += __ldcg(t.node_leaves + fc + k);
                internal += __ldcg(t.node_nchild + fc + k) > 0;
            }
            t.node_leaves[node] = leaves;
            if (pending) pending[node] = nc > 0 && internal == 0 ? -1 : internal;
        }
        cluster_barrier();
    }
    // leaf numbers, downwards
    if (tid == 0) t.node_leaf0[0] = 0;
    for (int l = 0; l <= depth; ++l) {
        if (l > 0) cluster_barrier();
        for (int node = level_begin[l] + tid; node < level_begin[l + 1]; node += kAll) {
            const int nc = __ldcg(t.node_nchild + node);
            int leaf = l == 0 ? 0 : __ldcg(t.node_leaf0 + node);
            if (nc == 0) {
                t.leaf_node[leaf] = node;
                if (t.max_per_leaf > 0 && __ldcg(t.node_end + node) - __ldcg(t.node_start + node) > t.max_per_leaf)
                    flags |= 1;  // depth limit
            }
            const int fc = __ldcg(t.node_first_child + node);
            for (int k = 0; k < nc; ++k) {
                t.node_leaf0[fc + k] = leaf;
                leaf += __ldcg(t.node_leaves + fc + k);
            }
        }
    }
    if (flags) atomicOr(&t.counters[2], flags);
    if (tid == 0) {
        t.counters[1] = le;
        t.counters[3] = t.n_points > 0 ? __ldcg(t.node_leaves) : 0;
        t.counters[4] = depth;
    }
    cluster_barrier();  // no block leaves while another reads its shared memory
}

// Batch starts of n <= kClusterSortMax sorted keys by one cluster (the rule of batch_flags_kernel and
// batch_first_kernel, treecode.cu): batches start every `batch` positions from the first key of each cell
// (keys >> shift).  Every thread walks a run of consecutive positions, the first one's cell start found by binary search.
__global__ void __cluster_dims__(kClBlocks, 1, 1) __launch_bounds__(kClThreads)
    batch_cut_kernel(const uint64_t* __restrict__ keys, int n, int shift, int batch, int32_t* __restrict__ batch_first,
                     int32_t* __restrict__ nbat, int64_t cap) {
    __shared__ int32_t slot;
    const int rank = (int)blockIdx.x, tid = rank * kClThreads + (int)threadIdx.x;
    constexpr int kAll = kClBlocks * kClThreads;
    const int per = (n + kAll - 1) / kAll, b = (int)min((int64_t)n, (int64_t)tid * per), e = min(n, b + per);
    int pos0 = 0;
    if (b < e) {
        const uint64_t cell = keys[b] >> shift;
        int lo = 0, hi = b;  // smallest j <= b in the same cell
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if ((keys[mid] >> shift) < cell) lo = mid + 1;
            else hi = mid;
        }
        pos0 = (b - lo) % batch;
    }
    auto walk = [&](auto start) {  // start(q) at every batch start of the thread's run
        int pos = pos0;
        uint64_t cell = b < e ? keys[b] >> shift : 0;
        for (int q = b; q < e; ++q) {
            const uint64_t c = keys[q] >> shift;
            if (c != cell) {
                cell = c;
                pos = 0;
            }
            if (pos == 0) start(q);
            if (++pos == batch) pos = 0;
        }
    };
    int32_t count = 0, block_total = 0, total = 0;
    walk([&](int) { ++count; });
    int32_t at = block_excl_scan(count, &block_total);
    at += cluster_excl(block_total, &slot, rank, &total);
    walk([&](int q) {
        if (at <= cap) batch_first[at] = q;
        ++at;
    });
    if (tid == 0) {
        if (total <= cap) batch_first[total] = n;
        nbat[0] = (int32_t)min((int64_t)total, cap);
        nbat[1] = total;
    }
    cluster_barrier();  // no block leaves while another reads its total
}

}  // namespace

int scan_exclusive_i32(lpm_ctx* ctx, const int32_t* in, int32_t* out, int64_t n, int32_t* total_dev, int sums_slot) {
    if (n <= 0) return LPM_OK;
    const int nblocks = (int)((n + kScanTile - 1) / kScanTile);
    int32_t* sums = (int32_t*)scratch(ctx, sums_slot, sizeof(int32_t) * (size_t)(nblocks + 1));
    if (!sums) return LPM_ERR_OOM;
    LPM_LAUNCH(ctx, "scan_block_sums_kernel", scan_block_sums_kernel, nblocks, kScanThreads, 0, in, n, sums);
    LPM_LAUNCH(ctx, "scan_single_block_kernel", scan_single_block_kernel, 1, 1024, 0, sums, (int64_t)nblocks,
               total_dev);
    LPM_LAUNCH(ctx, "scan_apply_kernel", scan_apply_kernel, nblocks, kScanThreads, 0, in, out, n, sums);
    return LPM_OK;
}

int sort_points(lpm_ctx* ctx, const double4* pts, int64_t n, const RootBox& root, int bits, int max_depth, int bit_lo,
                uint64_t* keys, int32_t* perm, uint64_t* tk, int32_t* tv, int32_t* counter, int counts_slot,
                int sums_slot) {
    if (n <= 0) return LPM_OK;
    const bool packed = bit_lo >= 32;
    LPM_LAUNCH(ctx, "morton_keys_kernel", morton_keys_kernel, grid_for(n, 256), 256, 0, pts, n, root, keys, perm, counter,
               bits, max_depth, packed);
    if (!packed) return radix_sort_impl<uint64_t>(ctx, keys, perm, tk, tv, n, bit_lo, 64, counts_slot, sums_slot);
    if (n <= 4 * kClBlocks * kClThreads) return cluster_sort<4>(ctx, keys, tk, perm, n, bit_lo);
    if (n <= 8 * kClBlocks * kClThreads) return cluster_sort<8>(ctx, keys, tk, perm, n, bit_lo);
    if (n <= kClusterSortMax) return cluster_sort<16>(ctx, keys, tk, perm, n, bit_lo);
    const int nblocks = (int)((n + kSortTile - 1) / kSortTile);
    int32_t* counts = (int32_t*)scratch(ctx, counts_slot, sizeof(int32_t) * 256 * (size_t)nblocks);
    if (!counts) return LPM_ERR_OOM;
    uint64_t *ks = keys, *kd = tk;
    for (int shift = bit_lo; shift < 64; shift += 8) {
        LPM_LAUNCH(ctx, "radix_hist_kernel", radix_hist_kernel<uint64_t>, nblocks, kSortThreads, 0, ks, n, shift, counts,
                   nblocks);
        const int rc = digit_offsets(ctx, counts, (int64_t)256 * nblocks, sums_slot);
        if (rc) return rc;
        LPM_LAUNCH(ctx, "packed_scatter_kernel", packed_scatter_kernel, nblocks, kSortThreads, 0, ks, kd,
                   shift + 8 >= 64 ? perm : nullptr, n, shift, counts, nblocks);
        std::swap(ks, kd);
    }
    if (ks != keys)
        LPM_CUDA_TRY(cudaMemcpyAsync(keys, ks, sizeof(uint64_t) * (size_t)n, cudaMemcpyDeviceToDevice, ctx->stream));
    return LPM_OK;
}

bool batch_cut(lpm_ctx* ctx, const uint64_t* keys, int64_t n, int shift, int batch, int32_t* batch_first, int32_t* nbat,
               int64_t cap, int* rc) {
    if (n > kClusterSortMax) return false;
    auto launch = [&]() -> int {
        LPM_LAUNCH(ctx, "batch_cut_kernel", batch_cut_kernel, kClBlocks, kClThreads, 0, keys, (int)n, shift, batch,
                   batch_first, nbat, cap);
        return LPM_OK;
    };
    *rc = launch();
    return true;
}

int root_extent(lpm_ctx* ctx, const double4* pts, int64_t first, int64_t n, int mode, unsigned long long* r_dev) {
    if (n <= first) return LPM_OK;
    const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>(grid_for(n - first, 256), 2 * ctx->num_sms));
    LPM_LAUNCH(ctx, "root_extent_kernel", root_extent_kernel, g, 256, 0, pts, first, n, mode, r_dev);
    return LPM_OK;
}

int radix_sort_u32(lpm_ctx* ctx, uint32_t* keys, int32_t* vals, uint32_t* tk, int32_t* tv, int64_t n, int bits) {
    return radix_sort_impl<uint32_t>(ctx, keys, vals, tk, tv, n, 0, bits, kSlotMisc1, kSlotMisc2);
}

int octree_alloc(Octree& t, int64_t n, int max_per_leaf, int max_depth, int bits, double sphere_r) {
    octree_free(t);
    t.n = n;
    t.max_per_leaf = max_per_leaf;
    t.bits = bits == 1 ? 1 : 3;
    t.levels = t.bits == 1 ? kMaxLevels : kKeyLevels;
    t.max_depth = std::min(std::max(max_depth, 1), t.levels);
    t.sphere_r = t.bits == 1 ? sphere_r : 0.0;
    if (t.bits == 1) {
        // every non-empty node splits to max_depth: level l holds at most min(n, 2^l) nodes
        int64_t cap = 0;
        for (int l = 0; l <= t.max_depth; ++l) cap += l < 62 ? std::min<int64_t>(n, 1ll << l) : n;
        t.node_cap = cap + 16;
    } else {
        // every internal node has >= 2 points in distinct children or splits a range of > max points:
        // n_nodes <= 8 * (internal nodes) + 1 and internal nodes <= depth * n / (max_per_leaf + 1) + 1
        const int64_t internal = (int64_t)t.max_depth * (n / (max_per_leaf + 1) + 1) + 1;
        t.node_cap = std::min<int64_t>(8 * internal + 1, std::max<int64_t>(2 * n + 16, 64));
    }
    const size_t nn = (size_t)std::max<int64_t>(n, 1), nc = (size_t)t.node_cap;
    cudaError_t e = cudaSuccess;
    auto A = [&](void** p, size_t bytes) {
        if (e == cudaSuccess) e = dev_alloc((void**)p, bytes);
    };
    A((void**)&t.keys, nn * 8);
    A((void**)&t.perm, nn * 4);
    A((void**)&t.tmp_keys, nn * 8);
    A((void**)&t.tmp_vals, nn * 4);
    A((void**)&t.node_start, nc * 4);
    A((void**)&t.node_end, nc * 4);
    A((void**)&t.node_parent, nc * 4);
    A((void**)&t.node_first_child, nc * 4);
    A((void**)&t.node_nchild, nc);
    A((void**)&t.node_level, nc);
    A((void**)&t.node_box, nc * 6 * 8);
    A((void**)&t.child_start, nc * 9 * 4);
    A((void**)&t.counters, 16 * 4);
    A((void**)&t.leaf_node, nc * 4);
    A((void**)&t.node_leaf0, nc * 4);
    A((void**)&t.node_leaves, nc * 4);
    if (e != cudaSuccess) {
        octree_free(t);
        return cuda_status(e, "cudaMalloc (octree)");
    }
    return LPM_OK;
}

void octree_free(Octree& t) {
    void* ps[] = {t.keys, t.perm, t.tmp_keys, t.tmp_vals, t.node_start, t.node_end, t.node_parent,
                  t.node_first_child, t.node_nchild, t.node_level, t.node_box, t.child_start, t.counters, t.leaf_node,
                  t.node_leaf0, t.node_leaves};
    for (void* p : ps)
        if (p) cudaFree(p);
    const Octree keep = t;
    t = Octree();
    t.n = keep.n;
    t.max_per_leaf = keep.max_per_leaf;
    t.max_depth = keep.max_depth;
    t.bits = keep.bits;
    t.levels = keep.levels;
    t.sphere_r = keep.sphere_r;
}

int octree_build(lpm_ctx* ctx, Octree& t, const double4* pts, int64_t n, const RootBox& root, int32_t* pending) {
    if (n > t.n || n >= INT32_MAX) {
        set_error("octree_build: %lld points exceed the tree's capacity", (long long)n);
        return LPM_ERR_CAPACITY;
    }
    t.root = root;
    t.n_points = n;
    LPM_CUDA_TRY(cudaMemsetAsync(t.counters, 0, 16 * 4, ctx->stream));
    // the key bits that decide levels 1..max_depth (and the outside flag in bit 63)
    const int bit_lo = std::max(0, t.bits * (t.levels - t.max_depth)) & ~7;
    int rc = sort_points(ctx, pts, n, root, t.bits, t.max_depth, bit_lo, t.keys, t.perm, t.tmp_keys, t.tmp_vals,
                         t.counters);
    if (rc) return rc;
    LPM_LAUNCH(ctx, "tree_nodes_kernel", tree_nodes_kernel, kClBlocks, kClThreads, 0, t, pending);
    return LPM_OK;
}

}  // namespace lpm
