// Dij kernels: compaction of the (spot, voxel) hash table, a stable LSD radix sort, the two CSR
// layouts, and the sparse products dose = D.w and grad = D^T.g.
//
// The reference scores Dij into an open-addressing table keyed by (voxel, spot)
// (insert_hashtable, moqui/kernel_functions/mqi_transport.hpp:68-111) and writes it as a
// spot-row CSR npz in table-scan order (save_to_npz, moqui/base/mqi_io.hpp:251-320).  Here the
// table is compacted and sorted on the device, so both layouts come out in a fixed order:
//   spot rows  (the reference's npz layout, shape [n_spots, n_voxels]): indptr / voxel / value,
//              voxels ascending in a row -- the transposed operator, read by D^T.g;
//   voxel rows (only voxels with an entry, "doubly compressed"): row voxel / row start in its run /
//              spot / value, spots ascending in a row -- read by D.w.
// Both products are gathers with a fixed reduction order: no atomics, reproducible results.
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <utility>

#include <cuda_runtime.h>

#include "mqi_internal.h"

namespace mqi_gpu
{

namespace
{

constexpr int kThreads = 256;   // radix sort and compaction block
constexpr int kItems   = 16;    // keys per thread per radix pass
constexpr int kTile    = kThreads * kItems;
constexpr int kCompactItems = 8;    // table slots per thread and round of the compaction
constexpr int kScanTile = 2048;
static_assert(kScanTile == kRowTile, "the host finds the last tile");

__device__ inline unsigned
lanemask_lt() {
    return (1u << (threadIdx.x & 31)) - 1u;
}

// ---- compaction -----------------------------------------------------------------------------

/// Append every occupied slot as ((spot << vbits) | voxel, FP32 value = FP64 tally x scale, rounded
/// once), in no particular order.  Bound by HBM: 16 B read per slot, 12 B written per entry.  A block
/// gathers its 2048 slots' entries in shared memory, so one atomic on the cursor serves them all
/// (one a warp took 3.3 ms for 2^27 slots, now 0.42: 4 M atomics on one address), the
/// narrow FP64 pipe sees whole warps of entries, and the writes are dense.  `bad` is set where a spot
/// is not below n_spots.
__global__ void __launch_bounds__(kThreads)
k_dij_compact(const DijSlot* __restrict__ tab, uint64_t cap, int vbits, uint32_t n_spots, double scale,
              unsigned long long* __restrict__ keys, uint32_t* __restrict__ vals, uint64_t n_max,
              unsigned long long* __restrict__ cursor, uint32_t* __restrict__ bad) {
    constexpr int kRound = kThreads * kCompactItems;
    __shared__ unsigned long long s_key[kRound];
    __shared__ double             s_val[kRound];
    __shared__ uint32_t           s_n;
    __shared__ unsigned long long s_base;
    const int lane = threadIdx.x & 31;
    for (uint64_t r0 = (uint64_t) blockIdx.x * kRound; r0 < cap; r0 += (uint64_t) gridDim.x * kRound) {
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        ulonglong2 e[kCompactItems];   // DijSlot: key, value
#pragma unroll
        for (int k = 0; k < kCompactItems; ++k) {
            const uint64_t i = r0 + (uint64_t) k * kThreads + threadIdx.x;
            e[k] = i < cap ? reinterpret_cast<const ulonglong2*>(tab)[i] : make_ulonglong2(0ull, 0ull);
        }
        uint32_t mine = 0;
#pragma unroll
        for (int k = 0; k < kCompactItems; ++k) mine += e[k].x != 0ull;
        uint32_t before = mine;   // inclusive, then exclusive, over the warp
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, before, o);
            if (lane >= o) before += y;
        }
        uint32_t warp_base = 0;
        if (lane == 31) warp_base = atomicAdd(&s_n, before);
        uint32_t at = __shfl_sync(0xFFFFFFFFu, warp_base, 31) + before - mine;
#pragma unroll
        for (int k = 0; k < kCompactItems; ++k)
            if (e[k].x != 0ull) {
                s_key[at] = e[k].x - 1ull;
                s_val[at] = __longlong_as_double((long long) e[k].y);
                ++at;
            }
        __syncthreads();
        const uint32_t n = s_n;
        if (threadIdx.x == 0) s_base = n ? atomicAdd(cursor, (unsigned long long) n) : 0ull;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < n; j += kThreads) {
            const uint64_t pos  = s_base + j;
            const uint64_t spot = s_key[j] >> 32;
            if (pos < n_max) {   // the host compares the cursor with n_max afterwards
                keys[pos] = (spot << vbits) | (s_key[j] & 0xFFFFFFFFull);
                vals[pos] = __float_as_uint((float) (s_val[j] * scale));
            }
            if (spot >= n_spots) *bad = 1u;
        }
        __syncthreads();
    }
}

/// *out += the number of occupied slots (nonzero keys) of the table: a grid-stride count, one
/// atomic per warp.
__global__ void
k_dij_count(const DijSlot* __restrict__ tab, uint64_t cap, unsigned long long* __restrict__ out) {
    const uint64_t     stride = (uint64_t) gridDim.x * blockDim.x;
    unsigned long long n      = 0;
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < cap; i += stride) n += tab[i].key != 0ull;
    for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xFFFFFFFFu, n, o);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(out, n);
}

// ---- exclusive scan of u32 ------------------------------------------------------------------

__device__ inline uint32_t
block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t  x    = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < nw ? warp_sums[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) warp_sums[lane] = s;
    }
    __syncthreads();
    const uint32_t warp_off = warp ? warp_sums[warp - 1] : 0u;
    total                   = warp_sums[nw - 1];
    __syncthreads();
    return warp_off + x - v;
}

/// Per-tile exclusive scan (kScanTile elements per 256-thread block, 8 per thread in order);
/// tile totals to `sums`.
__global__ void
k_scan_tiles(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint64_t n, uint32_t* __restrict__ sums) {
    __shared__ uint32_t ws[32];
    const uint64_t t0 = (uint64_t) blockIdx.x * kScanTile + (uint64_t) threadIdx.x * 8;
    uint32_t       v[8], s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        v[k] = (t0 + k < n) ? in[t0 + k] : 0u;
        s += v[k];
    }
    uint32_t total;
    uint32_t run = block_exclusive_scan(s, ws, total);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (t0 + k < n) out[t0 + k] = run;
        run += v[k];
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

/// Exclusive scan of the tile totals by one block, in order.
__global__ void
k_scan_sums(uint32_t* __restrict__ sums, uint64_t n) {
    __shared__ uint32_t ws[32];
    uint32_t carry = 0;
    for (uint64_t b = 0; b < n; b += blockDim.x) {
        const uint64_t i = b + threadIdx.x;
        const uint32_t v = i < n ? sums[i] : 0u;
        uint32_t total;
        const uint32_t e = block_exclusive_scan(v, ws, total);
        if (i < n) sums[i] = carry + e;
        carry += total;
        __syncthreads();
    }
}

__global__ void
k_scan_add(uint32_t* __restrict__ out, uint64_t n, const uint32_t* __restrict__ sums) {
    const uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += sums[i / kScanTile];
}

// ---- radix sort -----------------------------------------------------------------------------

__global__ void __launch_bounds__(kThreads)
k_radix_hist(const unsigned long long* __restrict__ keys, uint64_t n, int shift, uint32_t mask, uint32_t* __restrict__ hist,
             uint32_t n_tiles) {
    __shared__ uint32_t cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t t0 = (uint64_t) blockIdx.x * kTile;
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const uint64_t i = t0 + (uint64_t) r * kThreads + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(uint32_t) (keys[i] >> shift) & mask], 1u);
    }
    __syncthreads();
    if (threadIdx.x <= mask) hist[(uint64_t) threadIdx.x * n_tiles + blockIdx.x] = cnt[threadIdx.x];
}

/// Shared memory of k_radix_scatter.
struct RadixSmem {
    unsigned long long key[kTile];
    uint32_t           val[kTile];
    uint32_t           cnt[kThreads / 32][256];   // per warp and digit: a count, then a place in the tile
    uint32_t           first[256];                // the digit's first place in the tile
    uint32_t           offs[256];                 // and its first place in the output
    uint32_t           ws[32];
};

/// Stable scatter of one digit of at most 8 bits.  A warp takes 512 consecutive elements of the tile,
/// 32 at a time in input order, and ranks each among its equals by warp votes alone; the block then
/// turns the warps' counts into places, puts the tile in order in shared memory and writes it out, a
/// run of each digit's elements at a time.  Bound by HBM (12 B read and written per element).  With
/// the ranking across the block (three barriers per 256 elements) and each element stored from
/// registers, 11.7 M elements took 180 us a pass (now 70).
__global__ void __launch_bounds__(kThreads, 3)
k_radix_scatter(const unsigned long long* __restrict__ kin, const uint32_t* __restrict__ vin,
                unsigned long long* __restrict__ kout, uint32_t* __restrict__ vout, uint64_t n, int shift, uint32_t mask,
                const uint32_t* __restrict__ offs, uint32_t n_tiles) {
    extern __shared__ __align__(16) unsigned char radix_smem[];
    RadixSmem& S    = *reinterpret_cast<RadixSmem*>(radix_smem);
    const int  warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = kThreads / 32;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) S.cnt[w][threadIdx.x] = 0;
    if (threadIdx.x <= mask) S.offs[threadIdx.x] = offs[(uint64_t) threadIdx.x * n_tiles + blockIdx.x];
    __syncthreads();
    const uint64_t t0   = (uint64_t) blockIdx.x * kTile;
    const uint32_t size = (uint32_t) (n - t0 < (uint64_t) kTile ? n - t0 : (uint64_t) kTile);
    const uint32_t w0   = (uint32_t) warp * 32 * kItems;
    unsigned long long k[kItems];
    uint32_t           v[kItems], rank[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const uint32_t i = w0 + (uint32_t) r * 32 + lane;
        k[r] = 0ull;
        v[r] = 0u;
        if (i < size) {
            k[r] = kin[t0 + i];
            v[r] = vin[t0 + i];
        }
    }
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const bool     valid = w0 + (uint32_t) r * 32 + lane < size;
        const uint32_t d     = valid ? (uint32_t) (k[r] >> shift) & mask : 0x100u;   // 0x100 matches no digit
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
        uint32_t       seen  = 0;
        if (valid) seen = S.cnt[warp][d];
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) S.cnt[warp][d] = seen + __popc(peers);
        __syncwarp();
        rank[r] = seen + __popc(peers & lanemask_lt());
    }
    __syncthreads();
    {   // a thread a digit: places of the warps' shares
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c     = S.cnt[w][threadIdx.x];
            S.cnt[w][threadIdx.x] = total;
            total += c;
        }
        uint32_t       all;
        const uint32_t first = block_exclusive_scan(total, S.ws, all);
        S.first[threadIdx.x] = first;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r)
        if (w0 + (uint32_t) r * 32 + lane < size) {
            const uint32_t d   = (uint32_t) (k[r] >> shift) & mask;
            const uint32_t pos = S.first[d] + S.cnt[warp][d] + rank[r];
            S.key[pos] = k[r];
            S.val[pos] = v[r];
        }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < size; j += kThreads) {
        const unsigned long long x = S.key[j];
        const uint32_t           d = (uint32_t) (x >> shift) & mask;
        const uint32_t           o = S.offs[d] + (j - S.first[d]);
        kout[o] = x;
        vout[o] = S.val[j];
    }
}

// ---- CSR assembly ---------------------------------------------------------------------------

/// indptr[r] = lower_bound(keys, r << vbits) for r in [0, n_rows].
__global__ void
k_row_bounds(const unsigned long long* __restrict__ keys, uint64_t n, int vbits, uint64_t n_rows,
             uint64_t* __restrict__ indptr) {
    const uint64_t r = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (r > n_rows) return;
    const unsigned long long target = r << vbits;
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (keys[mid] < target) lo = mid + 1; else hi = mid;
    }
    indptr[r] = lo;
}

/// Spot-row entries: the voxel column and the value of each sorted key.
__global__ void
k_spot_rows(const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals, uint64_t n, uint32_t vmask,
            uint32_t* __restrict__ vox, uint32_t* __restrict__ val) {
    const uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vox[i] = (uint32_t) keys[i] & vmask;
    val[i] = vals[i];
}

/// Whether entry j of the voxel-sorted keys starts a row.
__device__ inline bool
starts_row(const unsigned long long* __restrict__ keys, uint64_t j, uint32_t vmask) {
    return j == 0 || (((uint32_t) keys[j] ^ (uint32_t) keys[j - 1]) & vmask) != 0u;
}

/// Rows that start in each tile of kScanTile entries.
__global__ void __launch_bounds__(kThreads)
k_count_rows(const unsigned long long* __restrict__ keys, uint64_t n, uint32_t vmask, uint32_t* __restrict__ tiles) {
    __shared__ uint32_t sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    const uint64_t t0 = (uint64_t) blockIdx.x * kScanTile;
    uint32_t       c  = 0;
#pragma unroll
    for (int r = 0; r < kScanTile / kThreads; ++r) {
        const uint64_t j = t0 + (uint64_t) r * kThreads + threadIdx.x;
        c += j < n && starts_row(keys, j, vmask);
    }
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&sum, c);
    __syncthreads();
    if (threadIdx.x == 0) tiles[blockIdx.x] = sum;
}

/// Voxel-row entries -- the spot column (Spot: 16 bits where the columns allow) and the value of each
/// sorted key -- and the rows' voxels, first entries (indptr) and those within their stretch of
/// kFwdEntries (off); tiles[b] = the rows that start before tile b.
template<typename Spot>
__global__ void __launch_bounds__(kThreads)
k_voxel_rows(const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals, uint64_t n, int vbits,
             const uint32_t* __restrict__ tiles, uint32_t* __restrict__ row_voxel, uint16_t* __restrict__ off,
             uint64_t* __restrict__ indptr, Spot* __restrict__ spot, uint32_t* __restrict__ val) {
    __shared__ uint32_t ws[32];
    const uint32_t vmask = (uint32_t) ((1ull << vbits) - 1ull);
    const uint64_t t0    = (uint64_t) blockIdx.x * kScanTile;
    uint32_t       row   = tiles[blockIdx.x];
    for (int r = 0; r < kScanTile / kThreads; ++r) {
        const uint64_t j     = t0 + (uint64_t) r * kThreads + threadIdx.x;
        const bool     start = j < n && starts_row(keys, j, vmask);
        uint32_t       total;
        const uint32_t at = row + block_exclusive_scan(start ? 1u : 0u, ws, total);
        if (j < n) {
            const unsigned long long k = keys[j];
            spot[j] = (Spot) (k >> vbits);
            val[j]  = vals[j];
            if (start) {
                row_voxel[at] = (uint32_t) k & vmask;
                indptr[at]    = j;
                off[at]       = (uint16_t) (j % kFwdEntries);
            }
            if (j == n - 1) indptr[at + (start ? 1u : 0u)] = n;
        }
        row += total;
    }
}

// ---- backward segments: their work order ---------------------------------------------------

/// Sort keys of the backward's work order: the voxel of each segment's first entry.
__global__ void
k_seg_keys(const uint64_t* __restrict__ seg_start, uint32_t n_seg, const uint32_t* __restrict__ vox,
           unsigned long long* __restrict__ okeys, uint32_t* __restrict__ oval) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_seg) return;
    okeys[i] = vox[seg_start[i]];
    oval[i]  = i;
}

// ---- products -------------------------------------------------------------------------------

/// Block b of the staged forward owns the voxel rows that start in entries [b * kFwdEntries,
/// (b + 1) * kFwdEntries): row_first[b] = the first row r with indptr[r] >= b * kFwdEntries, and
/// run_k[b] = indptr[row_first[b]], the run's first entry.  One thread per block boundary, a binary
/// search over indptr (once per Dij build).
__global__ void
k_fwd_blocks(const uint64_t* __restrict__ indptr, uint64_t n_rows, uint64_t n_blocks, uint32_t* __restrict__ row_first,
             uint64_t* __restrict__ run_k) {
    const uint64_t b = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (b > n_blocks) return;
    const uint64_t target = b * kFwdEntries;
    uint64_t lo = 0, hi = n_rows;   // first r in [0, n_rows] with indptr[r] >= target
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (indptr[mid] < target) lo = mid + 1; else hi = mid;
    }
    const uint64_t r = b == n_blocks ? n_rows : lo;
    row_first[b]     = (uint32_t) r;
    run_k[b]         = indptr[r];
}

/// Where a voxel row lies: the rows of run b start in entries [b * kFwdEntries, (b + 1) * kFwdEntries),
/// so two bytes a row say where (an 8-byte row pointer was a fifth of what the product read on a
/// plan's matrix, which has about four entries to a row).
__device__ __forceinline__ void
row_span(const uint16_t* __restrict__ off, uint32_t r, uint32_t r1, uint64_t base, uint64_t k1, uint64_t& rb, uint64_t& re) {
    rb = base + off[r];
    re = r + 1 < r1 ? base + off[r + 1] : k1;
}

/// dose[row_voxel[r]] = sum_k val[k] * w[spot[k]] over voxel rows (D.w), in FP64.  Block b stages
/// the products of run b's entries -- at most kFwdEntries + the longest row, read with coalesced
/// loads -- in shared memory, then each thread sums whole rows from there in entry order (a fixed
/// order: the result does not depend on the launch).  A run longer than the staging buffer (a row of
/// more than kFwdStage - kFwdEntries entries) is summed from global memory instead, in the same order.
template<typename Spot>
__global__ void __launch_bounds__(256)
k_dij_forward(const uint32_t* __restrict__ row_voxel, const uint16_t* __restrict__ off,
              const uint32_t* __restrict__ row_first, const uint64_t* __restrict__ run_k, const Spot* __restrict__ spot,
              const float* __restrict__ val, const double* __restrict__ w, double* __restrict__ dose) {
    using Spot4 = typename std::conditional<sizeof(Spot) == 2, ushort4, uint4>::type;
    extern __shared__ __align__(16) unsigned char fwd_smem[];
    double* prod = reinterpret_cast<double*>(fwd_smem);
    const uint32_t r0 = row_first[blockIdx.x], r1 = row_first[blockIdx.x + 1];
    if (r0 >= r1) return;
    const uint64_t base = blockIdx.x * kFwdEntries, k0 = run_k[blockIdx.x], k1 = run_k[blockIdx.x + 1];
    const bool     staged = k1 - k0 <= kFwdStage;
    // the thread's first row is read before the staging, so that its latency overlaps it
    uint32_t r  = r0 + threadIdx.x;
    uint64_t rb = 0, re = 0;
    uint32_t rv = 0;
    if (r < r1) {
        row_span(off, r, r1, base, k1, rb, re);
        rv = row_voxel[r];
    }
    if (staged) {
        // loads of whole groups of four entries (the arrays are padded to whole groups);
        // entries of the group outside [k0, k1) are skipped
        const Spot4*   s4 = reinterpret_cast<const Spot4*>(spot);
        const float4*  v4 = reinterpret_cast<const float4*>(val);
        const uint64_t q1 = (k1 + 3) >> 2;
#pragma unroll 2
        for (uint64_t q = (k0 >> 2) + threadIdx.x; q < q1; q += blockDim.x) {
            const Spot4    ss = s4[q];
            const float4   vv = v4[q];
            const uint64_t k  = q << 2;
            if (k >= k0 && k < k1) prod[k - k0] = (double) vv.x * w[ss.x];
            if (k + 1 >= k0 && k + 1 < k1) prod[k + 1 - k0] = (double) vv.y * w[ss.y];
            if (k + 2 >= k0 && k + 2 < k1) prod[k + 2 - k0] = (double) vv.z * w[ss.z];
            if (k + 3 >= k0 && k + 3 < k1) prod[k + 3 - k0] = (double) vv.w * w[ss.w];
        }
        __syncthreads();
    }
    while (r < r1) {
        double acc = 0.0;
        if (staged)
            for (uint64_t k = rb; k < re; ++k) acc += prod[k - k0];
        else
            for (uint64_t k = rb; k < re; ++k) acc += (double) val[k] * w[spot[k]];
        dose[rv] = acc;
        r += blockDim.x;
        if (r < r1) {
            row_span(off, r, r1, base, k1, rb, re);
            rv = row_voxel[r];
        }
    }
}

// ---- bulk copies: the copy engine (untiled cp.async.bulk) completing on a shared-memory mbarrier

__device__ __forceinline__ uint32_t
smem_u32(const void* p) {
    return (uint32_t) __cvta_generic_to_shared(p);
}

__device__ __forceinline__ void
mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void
mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

/// Global -> shared copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) that
/// completes its bytes on `bar`.
__device__ __forceinline__ void
bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ bool
mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

/// The calling thread's accesses to shared memory so far come before copies that are issued after a
/// barrier: a bulk copy writes through another proxy than the threads do, which barriers alone do not order.
__device__ __forceinline__ void
fence_before_bulk() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

/// The rows and entries of one run of the persistent forward, as thread 0 found them.
struct FwdRun {
    unsigned long long k0, k1, a0;   // entries [k0, k1); staged from a0 (k0 rounded down to a group of eight)
    uint32_t           r0, r1;       // voxel rows [r0, r1)
    uint32_t           staged, pad;
};
static_assert(sizeof(FwdRun) == 40, "FwdRun layout");

constexpr int      kFwdRowsAhead  = 2;     // rows a thread reads ahead
constexpr int      kFwdBatch      = 4;     // products a thread forms at a time
constexpr uint32_t kFwdPipeHeader = 256;   // kFwdStages mbarriers + FwdRuns
static_assert(kFwdStages * (8 + sizeof(FwdRun)) <= kFwdPipeHeader, "forward header");

/// D.w in FP32, persistent, through a ring of kFwdStages shared-memory stages.  Each CTA walks the
/// runs b = blockIdx.x, blockIdx.x + gridDim.x, ... (run b: the voxel rows that start in entries
/// [b * kFwdEntries, (b + 1) * kFwdEntries), row_first[b] to row_first[b + 1], first entry
/// run_k[b]).  While the block forms and sums run i from one stage, the copy engine fills the
/// others with runs i + 1 .. i + kFwdStages - 1: thread 0 issues two untiled bulk copies per run
/// (its spots and values, rounded out to whole groups of eight entries; the arrays are padded)
/// completing on that stage's mbarrier, so each CTA keeps kFwdStages - 1 runs' bytes in flight while
/// it computes.  In a run the block multiplies each value by w[spot] in place, then each thread sums
/// whole rows from there in entry order (as k_dij_forward does): the result does not depend on
/// the grid.  Waits are bounded: a block whose copies have not landed after ~1 s of polling sets
/// bit 8 of `err`, waits (bounded) for its other stages' copies and returns.  A run longer than a
/// stage (kFwdPipeStageEntries entries: a row of more than ~2000 spots) is summed from global memory.
///
/// It reads an entry's spot (2 or 4 bytes) and value and 6 bytes a row, and writes the dose: on a
/// 500-spot CT matrix (9.1e7 entries, 1.5e7 rows) 235 us before the 2-byte spots and row offsets, 195
/// now, 0.55 of the measured copy rate.  What is left is latency between the barriers of a run:
/// neither the product pass, the row sums nor the stores cost more than 25 us by themselves, and
/// weights in shared memory, shorter runs and deeper rings gave nothing.
template<typename Spot>
__global__ void __launch_bounds__(kFwdPipeThreads)
k_dij_forward_pipe(const uint32_t* __restrict__ row_voxel, const uint16_t* __restrict__ off,
                   const uint32_t* __restrict__ row_first, const uint64_t* __restrict__ run_k, uint64_t n_blocks,
                   const Spot* __restrict__ spot, const float* __restrict__ val, const float* __restrict__ w,
                   float* __restrict__ dose, uint32_t* __restrict__ err) {
    constexpr uint32_t kSpotBytes  = (uint32_t) kFwdPipeStageEntries * sizeof(Spot);
    constexpr uint32_t kStageBytes = kSpotBytes + (uint32_t) kFwdPipeStageEntries * sizeof(float);
    extern __shared__ __align__(16) unsigned char fwd_smem[];
    uint64_t*      bar  = reinterpret_cast<uint64_t*>(fwd_smem);
    FwdRun*        runs = reinterpret_cast<FwdRun*>(fwd_smem + 8 * kFwdStages);
    unsigned char* data = fwd_smem + kFwdPipeHeader;
    const int      tid  = threadIdx.x;
    const uint64_t step = gridDim.x;

    // Thread 0 reads a run's bounds one run before it starts that run's copies, so the loads'
    // latency passes while the block computes.
    uint32_t           pf_r0 = 0, pf_r1 = 0;
    unsigned long long pf_k0 = 0, pf_k1 = 0;
    auto fetch = [&](uint64_t b) {
        pf_r0 = row_first[b];
        pf_r1 = row_first[b + 1];
        pf_k0 = run_k[b];
        pf_k1 = run_k[b + 1];
    };
    // thread 0: describe the fetched run in stage s and start its copies
    auto issue = [&](int s) {
        FwdRun R;
        R.r0  = pf_r0;
        R.r1  = pf_r1;
        R.k0  = pf_k0;
        R.k1  = pf_k1;
        R.a0  = R.k0 & ~7ull;
        R.pad = 0;
        const unsigned long long a1 = (R.k1 + 7ull) & ~7ull;
        R.staged = (R.r0 < R.r1 && a1 - R.a0 <= kFwdPipeStageEntries) ? 1u : 0u;
        if (R.staged) {
            const uint32_t m  = (uint32_t) (a1 - R.a0);
            unsigned char* st = data + (size_t) s * kStageBytes;
            mbar_expect_tx(&bar[s], m * (uint32_t) (sizeof(Spot) + sizeof(float)));
            bulk_load(st, spot + R.a0, m * (uint32_t) sizeof(Spot), &bar[s]);
            bulk_load(st + kSpotBytes, val + R.a0, m * (uint32_t) sizeof(float), &bar[s]);
        }
        runs[s] = R;
    };

    if (tid == 0) {
        for (int s = 0; s < kFwdStages; ++s) mbar_init(&bar[s], 1);
        // the first kFwdStages - 1 runs start at once
        uint64_t b = blockIdx.x;
        for (int s = 0; s < kFwdStages - 1 && b < n_blocks; ++s, b += step) {
            fetch(b);
            issue(s);
        }
        if (b < n_blocks) fetch(b);
    }
    __syncthreads();
    uint32_t parity = 0;   // bit s: the phase of stage s's barrier to wait for next
    bool     failed = false;
    int      s      = 0;   // the stage of run i
    uint64_t b      = blockIdx.x;
    for (; b < n_blocks; b += step) {
        const uint64_t ahead = b + (kFwdStages - 1) * step;     // the run that goes into the stage freed last
        const int      sf    = s == 0 ? kFwdStages - 1 : s - 1;
        if (tid == 0 && ahead < n_blocks) {
            issue(sf);
            if (ahead + step < n_blocks) fetch(ahead + step);
        }
        const FwdRun R = runs[s];
        if (R.r0 < R.r1) {
            const uint64_t base = b * kFwdEntries;
            // the thread's first rows, all read before the wait: one latency, and that behind the copies
            uint32_t rv[kFwdRowsAhead], ob[kFwdRowsAhead], oe[kFwdRowsAhead];
#pragma unroll
            for (int i = 0; i < kFwdRowsAhead; ++i) {
                const uint32_t r = R.r0 + tid + i * kFwdPipeThreads;
                if (r < R.r1) {
                    rv[i] = row_voxel[r];
                    ob[i] = off[r];
                    oe[i] = r + 1 < R.r1 ? off[r + 1] : (uint32_t) (R.k1 - base);
                }
            }
            float* s_val = reinterpret_cast<float*>(data + (size_t) s * kStageBytes + kSpotBytes);
            if (R.staged) {
                bool     done  = false;
                uint32_t spins = 0;
                while (!(done = mbar_try_wait(&bar[s], (parity >> s) & 1u)) && ++spins < kBulkSpinLimit) {
                }
                parity ^= 1u << s;
                if (__syncthreads_or(!done)) {
                    failed = true;
                    break;
                }
                const Spot*    s_spot = reinterpret_cast<const Spot*>(data + (size_t) s * kStageBytes);
                const uint32_t m0 = (uint32_t) (R.k0 - R.a0), m1 = (uint32_t) (R.k1 - R.a0);
                for (uint32_t k = m0 + tid; k < m1; k += kFwdBatch * kFwdPipeThreads) {
                    float x[kFwdBatch];
#pragma unroll
                    for (int i = 0; i < kFwdBatch; ++i)
                        x[i] = k + i * kFwdPipeThreads < m1 ? w[s_spot[k + i * kFwdPipeThreads]] : 0.0f;
#pragma unroll
                    for (int i = 0; i < kFwdBatch; ++i)
                        if (k + i * kFwdPipeThreads < m1) s_val[k + i * kFwdPipeThreads] *= x[i];
                }
                __syncthreads();
            }
            auto row_sum = [&](uint32_t o0, uint32_t o1) {
                float acc = 0.0f;
                if (R.staged) {
                    const uint32_t e = (uint32_t) (base + o1 - R.a0);
                    for (uint32_t k = (uint32_t) (base + o0 - R.a0); k < e; ++k) acc += s_val[k];
                } else {
                    for (uint64_t k = base + o0; k < base + o1; ++k) acc += val[k] * w[spot[k]];
                }
                return acc;
            };
#pragma unroll
            for (int i = 0; i < kFwdRowsAhead; ++i)
                if (R.r0 + tid + i * kFwdPipeThreads < R.r1) dose[rv[i]] = row_sum(ob[i], oe[i]);
            for (uint32_t r = R.r0 + tid + kFwdRowsAhead * kFwdPipeThreads; r < R.r1; r += kFwdPipeThreads)
                dose[row_voxel[r]] = row_sum(off[r], r + 1 < R.r1 ? off[r + 1] : (uint32_t) (R.k1 - base));
        }
        fence_before_bulk();
        __syncthreads();   // stage s is free: the next iteration refills it
        s = s + 1 == kFwdStages ? 0 : s + 1;
    }
    if (failed && tid == 0) {
        atomicOr(err, 8u);
        // copies started for the other stages may still be landing: wait for them (bounded) before
        // the block's shared memory is released
        for (int k = 1; k < kFwdStages; ++k) {
            const int      so = (s + k) % kFwdStages;
            const uint64_t bo = b + (uint64_t) k * step;
            if (bo < n_blocks && runs[so].staged)
                for (uint32_t spins = 0; !mbar_try_wait(&bar[so], (parity >> so) & 1u) && spins < kBulkSpinLimit; ++spins) {
                }
        }
    }
}

/// grad[s] = sum_k val[k] * g[voxel[k]] over spot rows (the transposed operator), in two passes
/// with a fixed order.  Pass 1 (k_dij_backward_segments): the entries are cut into segments of at
/// most dij_segment(nnz) entries that never cross a row; one block sums a segment's products (signed
/// terms of a gradient cancel, so plain FP32 sums lose digits: a double-float accumulator per
/// thread for FP32 g, FP64 for FP64 g; FP64 across the block) into one FP64 partial.  Pass 2
/// (k_dij_backward_rows): a warp per row adds its segments' partials in a fixed tree.  Rows of very
/// different lengths (1e4 to 3e6 entries at 2000 spots) thereby spread over every SM.
/// s + c += a * b with no rounding error in the product (TwoProd: one FMA gives the product's
/// rounding error) and Knuth's TwoSum for the addition: a double-float accumulator of about 48
/// significant bits on the FP32 pipes.  GB300's FP64 pipe is far narrower than its FP32 pipes,
/// and an FP64 multiply-add per entry (with two conversions) made the backward FP64-bound.
__device__ __forceinline__ void
df_fma(float& s, float& c, float a, float b) {
    const float p   = __fmul_rn(a, b);
    const float pe  = __fmaf_rn(a, b, -p);
    const float t   = __fadd_rn(s, p);
    const float z   = __fsub_rn(t, s);
    const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(p, z));
    c               = __fadd_rn(c, __fadd_rn(err, pe));
    s               = t;
}

/// A block's share of the products of entries [b, e) of a spot row, per thread, in a fixed order:
/// thread t takes the groups of four q = (b >> 2) + t, + blockDim.x, ... (16-byte loads of voxels
/// and values, four independent gathers of g per group; the arrays are padded to whole groups).
template<typename T>
__device__ __forceinline__ double
segment_sum(uint64_t b, uint64_t e, const uint32_t* __restrict__ vox, const float* __restrict__ val,
            const T* __restrict__ g) {
    const uint4*   v4 = reinterpret_cast<const uint4*>(vox);
    const float4*  a4 = reinterpret_cast<const float4*>(val);
    const uint64_t q1 = (e + 3) >> 2;
    if constexpr (sizeof(T) == sizeof(float)) {
        float s = 0.0f, c = 0.0f;
#pragma unroll 4
        for (uint64_t q = (b >> 2) + threadIdx.x; q < q1; q += blockDim.x) {
            const uint4    vv = v4[q];
            const float4   aa = a4[q];
            const uint64_t k  = q << 2;
            const bool     m0 = k >= b && k < e, m1 = k + 1 >= b && k + 1 < e;
            const bool     m2 = k + 2 >= b && k + 2 < e, m3 = k + 3 >= b && k + 3 < e;
            const float    g0 = m0 ? g[vv.x] : 0.0f, g1 = m1 ? g[vv.y] : 0.0f;
            const float    g2 = m2 ? g[vv.z] : 0.0f, g3 = m3 ? g[vv.w] : 0.0f;
            if (m0) df_fma(s, c, aa.x, g0);
            if (m1) df_fma(s, c, aa.y, g1);
            if (m2) df_fma(s, c, aa.z, g2);
            if (m3) df_fma(s, c, aa.w, g3);
        }
        return (double) s + (double) c;
    } else {
        double d = 0.0;
#pragma unroll 2
        for (uint64_t q = (b >> 2) + threadIdx.x; q < q1; q += blockDim.x) {
            const uint4    vv = v4[q];
            const float4   aa = a4[q];
            const uint64_t k  = q << 2;
            if (k >= b && k < e) d = __fma_rn((double) aa.x, g[vv.x], d);
            if (k + 1 >= b && k + 1 < e) d = __fma_rn((double) aa.y, g[vv.y], d);
            if (k + 2 >= b && k + 2 < e) d = __fma_rn((double) aa.z, g[vv.z], d);
            if (k + 3 >= b && k + 3 < e) d = __fma_rn((double) aa.w, g[vv.w], d);
        }
        return d;
    }
}

/// Pass 1 of D^T.g.  The blocks take segments from a shared cursor in the order of their first
/// voxel (`order`), so the segments in flight at any moment -- of every spot -- cover a narrow
/// band of depth, and their gathers of g come from a few megabytes that stay in L2 instead of each
/// spot's row sweeping the whole dose-gradient vector (a 4-byte gather then costs a 32-byte DRAM
/// sector).  Each segment's partial is written at its spot-major index; which block computes it
/// does not change it, so the result is reproducible.  The cursor is returned to zero by
/// k_dij_backward_rows, which runs after this kernel on the same stream.
template<typename T>
__global__ void __launch_bounds__(256, 8)
k_dij_backward_segments(const uint32_t* __restrict__ order, uint32_t n_seg, const uint64_t* __restrict__ seg_start,
                        const uint32_t* __restrict__ vox, const float* __restrict__ val, const T* __restrict__ g,
                        double* __restrict__ partial, uint32_t* __restrict__ cursor) {
    __shared__ double   part[32];
    __shared__ uint32_t s_next;
    if (threadIdx.x == 0) s_next = atomicAdd(cursor, 1u);
    __syncthreads();
    uint32_t i = s_next;
    while (i < n_seg) {
        __syncthreads();   // everyone has read s_next
        // the next segment is claimed before this one is summed, so the claim's latency overlaps it
        if (threadIdx.x == 0) s_next = atomicAdd(cursor, 1u);
        const uint32_t sg = order[i];
        double         d  = segment_sum<T>(seg_start[sg], seg_start[sg + 1], vox, val, g);
        for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xFFFFFFFFu, d, o);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = d;
        __syncthreads();
        if (threadIdx.x < 32) {
            d = threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0.0;
            for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xFFFFFFFFu, d, o);
            if (threadIdx.x == 0) partial[sg] = d;
        }
        __syncthreads();   // part[] is free again; s_next holds the next claim
        i = s_next;
    }
}

/// A warp a row: its lanes add every 32nd segment's partial, then each other in a fixed tree.  (A
/// thread a row read its partials one after the other: 13.5 us for 500 rows of 14.)
template<typename T>
__global__ void
k_dij_backward_rows(const uint32_t* __restrict__ row_seg, uint32_t n_rows, const double* __restrict__ partial,
                    T* __restrict__ grad, uint32_t* __restrict__ cursor) {
    const uint32_t r    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (r == 0 && lane == 0 && cursor) *cursor = 0u;
    if (r >= n_rows) return;
    double d = 0.0;
    for (uint32_t k = row_seg[r] + lane, e = row_seg[r + 1]; k < e; k += 32) d += partial[k];
    for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xFFFFFFFFu, d, o);
    if (lane == 0) grad[r] = (T) d;
}

__global__ void
k_dij_clear(DijSlot* __restrict__ tab, uint64_t cap) {
    const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < cap; i += stride) {
        tab[i].key   = 0ull;
        tab[i].value = 0.0;
    }
}

unsigned
blocks_for(uint64_t n, int per_block) {
    return (unsigned) ((n + per_block - 1) / per_block);
}

}   // namespace

cudaError_t
dij_clear(DijSlot* tab, uint64_t cap, int sms, cudaStream_t s) {
    k_dij_clear<<<sms * 8, 256, 0, s>>>(tab, cap);
    return cudaGetLastError();
}

cudaError_t
dij_count(const DijSlot* tab, uint64_t cap, unsigned long long* out, int sms, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess || cap == 0) return e;
    k_dij_count<<<(unsigned) std::min<uint64_t>((cap + 255) / 256, (uint64_t) sms * 8), 256, 0, s>>>(tab, cap, out);
    return cudaGetLastError();
}

cudaError_t
dij_compact(const DijSlot* tab, uint64_t cap, int vbits, uint32_t n_spots, double scale, unsigned long long* keys,
            uint32_t* vals, uint64_t n_max, unsigned long long* cursor, uint32_t* bad, int sms, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(cursor, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    const uint64_t rounds = (cap + kThreads * kCompactItems - 1) / (kThreads * kCompactItems);
    k_dij_compact<<<(unsigned) std::min<uint64_t>(rounds, (uint64_t) sms * 6), kThreads, 0, s>>>(tab, cap, vbits, n_spots, scale,
                                                                                              keys, vals, n_max, cursor, bad);
    return cudaGetLastError();
}

uint64_t
scan_scratch_words(uint64_t n) {
    return (n + kScanTile - 1) / kScanTile + 1;
}

cudaError_t
scan_exclusive_u32(const uint32_t* in, uint32_t* out, uint64_t n, uint32_t* scratch, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
    k_scan_tiles<<<(unsigned) tiles, 256, 0, s>>>(in, out, n, scratch);
    k_scan_sums<<<1, 1024, 0, s>>>(scratch, tiles);
    k_scan_add<<<blocks_for(n, 256), 256, 0, s>>>(out, n, scratch);
    return cudaGetLastError();
}

uint64_t
radix_hist_words(uint64_t n) {
    return 256ull * ((n + kTile - 1) / kTile);
}

cudaError_t
radix_sort_pairs(unsigned long long*& keys, uint32_t*& vals, unsigned long long*& keys_alt, uint32_t*& vals_alt,
                 uint64_t n, int first_bit, int bits, uint32_t* hist, uint32_t* offs, uint32_t* scan_scratch,
                 cudaStream_t s) {
    if (n == 0 || bits <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_radix_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(RadixSmem));
    if (e != cudaSuccess) return e;
    const uint32_t n_tiles = (uint32_t) ((n + kTile - 1) / kTile);
    // the fewest passes of at most 8 bits, of nearly equal width: fewer digits make longer runs
    const int passes = (bits + 7) / 8;
    for (int p = 0, bit = first_bit; p < passes; ++p) {
        const int      width = (first_bit + bits - bit + passes - p - 1) / (passes - p);
        const uint32_t mask  = (1u << width) - 1u;
        k_radix_hist<<<n_tiles, kThreads, 0, s>>>(keys, n, bit, mask, hist, n_tiles);
        if ((e = scan_exclusive_u32(hist, offs, (uint64_t) (mask + 1u) * n_tiles, scan_scratch, s)) != cudaSuccess) return e;
        k_radix_scatter<<<n_tiles, kThreads, sizeof(RadixSmem), s>>>(keys, vals, keys_alt, vals_alt, n, bit, mask, offs, n_tiles);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        std::swap(keys, keys_alt);
        std::swap(vals, vals_alt);
        bit += width;
    }
    return cudaSuccess;
}

cudaError_t
dij_row_bounds(const unsigned long long* keys, uint64_t n, int vbits, uint64_t n_rows, uint64_t* indptr, cudaStream_t s) {
    k_row_bounds<<<blocks_for(n_rows + 1, 256), 256, 0, s>>>(keys, n, vbits, n_rows, indptr);
    return cudaGetLastError();
}

cudaError_t
dij_spot_rows(const unsigned long long* keys, const uint32_t* vals, uint64_t n, int vbits, uint32_t* vox, float* val,
              cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_spot_rows<<<blocks_for(n, 256), 256, 0, s>>>(keys, vals, n, (uint32_t) ((1ull << vbits) - 1ull), vox,
                                                  reinterpret_cast<uint32_t*>(val));
    return cudaGetLastError();
}

cudaError_t
dij_count_rows(const unsigned long long* keys, uint64_t n, int vbits, uint32_t* tiles, uint32_t* tile_rows, uint32_t* scratch,
               cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint64_t nt = (n + kScanTile - 1) / kScanTile;
    k_count_rows<<<(unsigned) nt, kThreads, 0, s>>>(keys, n, (uint32_t) ((1ull << vbits) - 1ull), tile_rows);
    return scan_exclusive_u32(tile_rows, tiles, nt, scratch, s);
}

cudaError_t
dij_voxel_rows(const unsigned long long* keys, const uint32_t* vals, uint64_t n, int vbits, const uint32_t* tiles,
               uint32_t* row_voxel, uint16_t* off, uint64_t* indptr, void* spot, bool spot16, float* val, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const unsigned nt = (unsigned) ((n + kScanTile - 1) / kScanTile);
    uint32_t*      v  = reinterpret_cast<uint32_t*>(val);
    if (spot16)
        k_voxel_rows<<<nt, kThreads, 0, s>>>(keys, vals, n, vbits, tiles, row_voxel, off, indptr, (uint16_t*) spot, v);
    else
        k_voxel_rows<<<nt, kThreads, 0, s>>>(keys, vals, n, vbits, tiles, row_voxel, off, indptr, (uint32_t*) spot, v);
    return cudaGetLastError();
}

cudaError_t
dij_forward_blocks(const uint64_t* indptr, uint64_t n_rows, uint64_t nnz, uint32_t* row_first, uint64_t* run_k,
                   uint64_t* n_blocks, cudaStream_t s) {
    const uint64_t nb = (nnz + kFwdEntries - 1) / kFwdEntries;
    *n_blocks         = nb;
    k_fwd_blocks<<<blocks_for(nb + 1, 256), 256, 0, s>>>(indptr, n_rows, nb, row_first, run_k);
    return cudaGetLastError();
}

cudaError_t
dij_seg_order_keys(const uint64_t* seg_start, uint32_t n_seg, const uint32_t* vox, unsigned long long* okeys, uint32_t* oval,
                   cudaStream_t s) {
    if (n_seg == 0) return cudaSuccess;
    k_seg_keys<<<blocks_for(n_seg, 256), 256, 0, s>>>(seg_start, n_seg, vox, okeys, oval);
    return cudaGetLastError();
}

template<typename Spot>
static cudaError_t
forward(const uint32_t* row_voxel, const uint16_t* off, const uint32_t* row_first, const uint64_t* run_k, uint64_t n_blocks,
        const Spot* spot, const float* val, const void* w, void* dose, int fp64, uint32_t* err, int sms, cudaStream_t s) {
    static_assert(kFwdStage * sizeof(double) <= 227 * 1024, "staging buffer exceeds shared memory");
    if (fp64) {
        const size_t sm = kFwdStage * sizeof(double);
        cudaError_t  e  = cudaFuncSetAttribute(k_dij_forward<Spot>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sm);
        if (e != cudaSuccess) return e;
        k_dij_forward<Spot><<<(unsigned) n_blocks, 256, sm, s>>>(row_voxel, off, row_first, run_k, spot, val,
                                                                (const double*) w, (double*) dose);
    } else {
        constexpr size_t sm = kFwdPipeHeader + kFwdStages * kFwdPipeStageEntries * (sizeof(Spot) + sizeof(float));
        constexpr int    per_sm = sizeof(Spot) == 2 ? 3 : 2;
        static_assert(per_sm * (sm + 1024) <= 228 * 1024, "the persistent forward blocks must fit one SM");
        cudaError_t e = cudaFuncSetAttribute(k_dij_forward_pipe<Spot>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sm);
        if (e != cudaSuccess) return e;
        const uint64_t cap  = (uint64_t) sms * per_sm;
        const unsigned grid = (unsigned) (n_blocks < cap ? n_blocks : cap);
        k_dij_forward_pipe<Spot><<<grid, kFwdPipeThreads, sm, s>>>(row_voxel, off, row_first, run_k, n_blocks, spot, val,
                                                                  (const float*) w, (float*) dose, err);
    }
    return cudaGetLastError();
}

cudaError_t
dij_forward(const uint32_t* row_voxel, const uint16_t* off, const uint32_t* row_first, const uint64_t* run_k,
            uint64_t n_blocks, const void* spot, bool spot16, const float* val, const void* w, void* dose, int fp64,
            uint32_t* err, int sms, cudaStream_t s) {
    if (n_blocks == 0) return cudaSuccess;
    return spot16 ? forward(row_voxel, off, row_first, run_k, n_blocks, (const uint16_t*) spot, val, w, dose, fp64, err, sms, s)
                  : forward(row_voxel, off, row_first, run_k, n_blocks, (const uint32_t*) spot, val, w, dose, fp64, err, sms, s);
}

cudaError_t
dij_backward(const uint32_t* order, const uint64_t* seg_start, uint32_t n_seg, const uint32_t* row_seg, uint32_t n_rows,
             const uint32_t* vox, const float* val, double* partial, uint32_t* cursor, const void* g, void* grad,
             int fp64, int sms, cudaStream_t s) {
    if (n_rows == 0) return cudaSuccess;
    if (n_seg) {
        const uint64_t cap  = (uint64_t) sms * 8;   // 8 blocks of 256 threads per SM
        const unsigned grid = (unsigned) std::min<uint64_t>(n_seg, cap);
        if (fp64)
            k_dij_backward_segments<double><<<grid, 256, 0, s>>>(order, n_seg, seg_start, vox, val, (const double*) g,
                                                                 partial, cursor);
        else
            k_dij_backward_segments<float><<<grid, 256, 0, s>>>(order, n_seg, seg_start, vox, val, (const float*) g,
                                                                partial, cursor);
    }
    const unsigned rb = (n_rows + 7) / 8;   // a warp a row
    if (fp64) k_dij_backward_rows<double><<<rb, 256, 0, s>>>(row_seg, n_rows, partial, (double*) grad, cursor);
    else k_dij_backward_rows<float><<<rb, 256, 0, s>>>(row_seg, n_rows, partial, (float*) grad, cursor);
    return cudaGetLastError();
}

}   // namespace mqi_gpu
