// sort.cu -- event records in PackedEvent order per simulation.
//
// Reporters receive events in PackedEvent order (necsim/core/src/event.rs:
// 256-280); the host sorted whole 40- and 56-byte records on one core.  Here
// a stable least-significant-digit radix sort (8-bit digits of the global
// reference, of the prior and the event time's bit patterns, then of the
// simulation) orders 12-byte (key, index) pairs and one gather moves the
// records.  Lineages that have met and not merged yet report the same events:
// with dispersal reporting most records share their time, place and target
// with others and differ in the reference or, where they meet, in the prior
// time.  The places and targets are not sorted by: a pass over the result
// looks for neighbours out of the whole order (unrelated events at the very
// same time), which the host then settles.
// Bound: some sixty short launches, among them a scan by one block per digit,
// not HBM: 600,000 dispersal records of one simulation took 0.42 ms by time
// alone, eight digits of about 30 bytes per pair at 340 GB/s; the ten digits
// more take the place of 30 ms of sorting ties on one core.
#include <cuda_runtime.h>

#include "kernels.h"

namespace necsim {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kSortBlock = 256, kSortWarps = kSortBlock / 32, kSortItems = 8;  // per thread
constexpr uint64_t kSortTile = (uint64_t)kSortBlock * kSortItems;

// Position of item i of a thread: every warp takes a contiguous run of the
// tile, 32 neighbours at a time, so ranks within a warp follow the order.
__device__ __forceinline__ uint64_t item_at(uint64_t tile, int i) {
    return tile * kSortTile + (uint64_t)(threadIdx.x / 32) * (32 * kSortItems) + (uint64_t)i * 32 + (threadIdx.x & 31u);
}

enum SortKey { kByReference, kByPriorTime, kByTime, kBySimulation };

// The next key of every record, in the order so far (`idx`; null: as stored).
template <typename Record, SortKey BY>
__global__ void sort_keys_kernel(const Record *rec, uint64_t n, const uint32_t *idx, unsigned long long *key,
                                 uint32_t *idx_out) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t k = idx ? idx[j] : (uint32_t)j;
        const Record &r = rec[k];
        key[j] = BY == kByReference   ? r.gref
                 : BY == kByPriorTime ? time_bits(r.prior_time)
                 : BY == kByTime      ? time_bits(r.event_time)
                                      : r.sim;
        if (!idx) idx_out[j] = k;
    }
}

// Sets *unordered if a record belongs before its predecessor.
template <typename Record>
__global__ void sort_check_kernel(const Record *rec, uint64_t n, uint32_t *unordered) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x + 1; j < n;
         j += (uint64_t)gridDim.x * blockDim.x)
        if (time_bits(rec[j].event_time) == time_bits(rec[j - 1].event_time) && event_less(rec[j], rec[j - 1]))
            *unordered = 1u;
}

// Digit counts of every tile: hist[digit * tiles + tile].
__global__ void __launch_bounds__(kSortBlock) sort_count_kernel(const unsigned long long *key, uint64_t n, int shift,
                                                                uint32_t *hist, uint32_t tiles) {
    __shared__ uint32_t count[256];
    count[threadIdx.x] = 0;
    __syncthreads();
    for (int i = 0; i < kSortItems; ++i) {
        const uint64_t j = item_at(blockIdx.x, i);
        if (j < n) atomicAdd(&count[(key[j] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[(uint64_t)threadIdx.x * tiles + blockIdx.x] = count[threadIdx.x];
}

// Exclusive prefix sums of m counts, in place, by one block.
__global__ void __launch_bounds__(1024) sort_scan_kernel(uint32_t *v, uint64_t m) {
    __shared__ uint32_t warp_sum[32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
    uint32_t carry = 0;
    for (uint64_t base = 0; base < m; base += 4096) {
        uint32_t x[4], sum = 0;
        const uint64_t at = base + (uint64_t)threadIdx.x * 4;
        for (int i = 0; i < 4; ++i) {
            x[i] = at + i < m ? v[at + i] : 0u;
            sum += x[i];
        }
        uint32_t inc = sum;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, inc, off);
            if ((int)lane >= off) inc += y;
        }
        if (lane == 31) warp_sum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = warp_sum[lane];
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(kAll, w, off);
                if ((int)lane >= off) w += y;
            }
            warp_sum[lane] = w;
        }
        __syncthreads();
        uint32_t run = carry + inc - sum + (warp ? warp_sum[warp - 1] : 0u);
        for (int i = 0; i < 4; ++i) {
            if (at + i < m) v[at + i] = run;
            run += x[i];
        }
        carry += warp_sum[31];
        __syncthreads();
    }
}

// Moves every pair to its digit's place, keeping the order of equal digits.
__global__ void __launch_bounds__(kSortBlock) sort_scatter_kernel(const unsigned long long *key, const uint32_t *idx,
                                                                  uint64_t n, int shift, const uint32_t *offset,
                                                                  uint32_t tiles, unsigned long long *key_out,
                                                                  uint32_t *idx_out) {
    __shared__ uint32_t count[kSortWarps][256];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
    for (int w = 0; w < kSortWarps; ++w) count[w][threadIdx.x] = 0;
    __syncthreads();
    uint32_t rank[kSortItems];
    unsigned long long k[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const uint64_t j = item_at(blockIdx.x, i);
        const bool in = j < n;
        k[i] = in ? key[j] : 0;
        const unsigned d = in ? (unsigned)(k[i] >> shift) & 255u : 256u;  // absent items match only one another
        const unsigned same = __match_any_sync(kAll, d);
        const int leader = __ffs(same) - 1;
        uint32_t before = 0;
        if (in && (int)lane == leader) {
            before = count[warp][d];
            count[warp][d] = before + (uint32_t)__popc(same);
        }
        __syncwarp();
        rank[i] = __shfl_sync(kAll, before, leader) + (uint32_t)__popc(same & ((1u << lane) - 1u));
    }
    __syncthreads();
    {  // this thread's digit: the tile's offset, then the warps' in order
        uint32_t run = offset[(uint64_t)threadIdx.x * tiles + blockIdx.x];
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = count[w][threadIdx.x];
            count[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const uint64_t j = item_at(blockIdx.x, i);
        if (j >= n) continue;
        const uint32_t d = count[warp][(unsigned)(k[i] >> shift) & 255u] + rank[i];
        key_out[d] = k[i];
        idx_out[d] = idx[j];
    }
}

// Records in sorted order, one 8-byte word per thread.
template <typename Record>
__global__ void sort_gather_kernel(const Record *rec, const uint32_t *idx, uint64_t n, Record *out) {
    constexpr uint64_t kWords = sizeof(Record) / 8;
    const uint64_t *src = reinterpret_cast<const uint64_t *>(rec);
    uint64_t *dst = reinterpret_cast<uint64_t *>(out);
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n * kWords;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t j = t / kWords;
        dst[t] = src[(uint64_t)idx[j] * kWords + (t - j * kWords)];
    }
}

size_t up(size_t bytes) { return (bytes + 255) & ~(size_t)255; }

template <typename Record>
cudaError_t sort_records_t(const Record *rec, uint64_t n, uint32_t n_sims, uint64_t references, void *scratch,
                           unsigned grid, Record **sorted, uint32_t **unordered, cudaStream_t st) {
    static_assert(sizeof(Record) % 8 == 0, "records are whole words");
    unsigned char *p = static_cast<unsigned char *>(scratch);
    auto take = [&](size_t bytes) {
        unsigned char *q = p;
        p += up(bytes);
        return q;
    };
    const uint32_t tiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
    Record *out = reinterpret_cast<Record *>(take(n * sizeof(Record)));
    unsigned long long *key[2];
    uint32_t *idx[2];
    for (int b = 0; b < 2; ++b) {
        key[b] = reinterpret_cast<unsigned long long *>(take(n * 8));
        idx[b] = reinterpret_cast<uint32_t *>(take(n * 4));
    }
    uint32_t *hist = reinterpret_cast<uint32_t *>(take((size_t)tiles * 256 * 4));
    *unordered = reinterpret_cast<uint32_t *>(take(4));
    int from = 0;
    auto pass = [&](int shift) {
        sort_count_kernel<<<tiles, kSortBlock, 0, st>>>(key[from], n, shift, hist, tiles);
        sort_scan_kernel<<<1, 1024, 0, st>>>(hist, (uint64_t)tiles * 256);
        sort_scatter_kernel<<<tiles, kSortBlock, 0, st>>>(key[from], idx[from], n, shift, hist, tiles, key[1 - from],
                                                          idx[1 - from]);
        from = 1 - from;
    };
    sort_keys_kernel<Record, kByReference><<<grid, 256, 0, st>>>(rec, n, nullptr, key[0], idx[0]);
    for (int shift = 0; shift < 64 && ((references - 1) >> shift) != 0; shift += 8) pass(shift);
    sort_keys_kernel<Record, kByPriorTime><<<grid, 256, 0, st>>>(rec, n, idx[from], key[from], nullptr);
    for (int shift = 0; shift < 64; shift += 8) pass(shift);
    sort_keys_kernel<Record, kByTime><<<grid, 256, 0, st>>>(rec, n, idx[from], key[from], nullptr);
    for (int shift = 0; shift < 64; shift += 8) pass(shift);
    if (n_sims > 1) {
        sort_keys_kernel<Record, kBySimulation><<<grid, 256, 0, st>>>(rec, n, idx[from], key[from], nullptr);
        for (int shift = 0; shift < 32 && ((n_sims - 1) >> shift) != 0; shift += 8) pass(shift);
    }
    sort_gather_kernel<<<grid, 256, 0, st>>>(rec, idx[from], n, out);
    const cudaError_t set = cudaMemsetAsync(*unordered, 0, 4, st);
    if (set != cudaSuccess) return set;
    sort_check_kernel<<<grid, 256, 0, st>>>(out, n, *unordered);
    *sorted = out;
    return cudaGetLastError();
}

}  // namespace

size_t sort_scratch_bytes(uint64_t n, size_t record) {
    const uint64_t tiles = (n + kSortTile - 1) / kSortTile;
    return up(n * record) + 2 * (up(n * 8) + up(n * 4)) + up((size_t)tiles * 256 * 4) + up(4);
}

cudaError_t sort_records(const DevSpeciationEvent *rec, uint64_t n, uint32_t n_sims, uint64_t references, void *scratch,
                         unsigned grid, DevSpeciationEvent **sorted, uint32_t **unordered, cudaStream_t st) {
    return sort_records_t(rec, n, n_sims, references, scratch, grid, sorted, unordered, st);
}

cudaError_t sort_records(const DevDispersalEvent *rec, uint64_t n, uint32_t n_sims, uint64_t references, void *scratch,
                         unsigned grid, DevDispersalEvent **sorted, uint32_t **unordered, cudaStream_t st) {
    return sort_records_t(rec, n, n_sims, references, scratch, grid, sorted, unordered, st);
}

}  // namespace necsim
