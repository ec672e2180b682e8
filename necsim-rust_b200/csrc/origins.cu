// origins.cu -- the simulations' origin lineages, written by the device.
//
// Every run starts from its scenario's origins (OriginPreSampler::all()
// through origin_sampler/{non_spatial,in_memory,spatially_implicit,
// singleton_demes/{circle,rectangle}}.rs).  They are closed forms of the
// origin's position, or positions in a prefix sum over rows or cells, so the
// host hands over a description per simulation instead of 32 bytes per
// lineage.  A NonSpatial call with ten million lineages took 296 ms with
// origins enumerated and copied by the host and some forty allocations, and
// takes 83 ms with this and one allocation; the kernel is bound by the 42
// bytes written per lineage (46 with the learned schedule).
// The WrappingNoise sample is filtered by its noise on the device too (the
// host and the device compute the same bits); its order is immaterial: a
// lineage's outcome depends on its own state, merges on global references.
#include <cuda_runtime.h>

#include "../../include/necsim_b200.h"
#include "kernels.h"
#include "wrapping_noise.h"

namespace necsim {

namespace {

// The last r in [0, rows) with prefix[r] <= k (prefix[0] = 0 <= k < prefix[rows]).
__device__ __forceinline__ uint64_t row_of(const uint64_t *prefix, uint64_t rows, uint64_t k) {
    uint64_t lo = 0, hi = rows;
    while (hi - lo > 1) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (prefix[mid] <= k)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

}  // namespace

// blockIdx.y strides over the simulations, the rest over their lineages.
__global__ void origins_kernel(const OriginSpec *specs, uint32_t n_sims, LineageSoA out, uint8_t *state) {
    for (uint32_t s = blockIdx.y; s < n_sims; s += gridDim.y) {
        const OriginSpec o = specs[s];
        for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < o.n;
             k += (uint64_t)gridDim.x * blockDim.x) {
            uint32_t x = 0, y = 0, i = 0;
            uint64_t g = k;
            double last = 0.0;
            if (o.form == kOriginGrid) {
                const uint64_t cell = k / o.deme;
                i = (uint32_t)(k - cell * o.deme);
                const uint64_t row = cell / o.width;
                x = (uint32_t)(cell - row * o.width);
                y = (uint32_t)row;
            } else if (o.form == kOriginPlane) {
                const uint64_t row = k / o.width;
                x = o.x0 + (uint32_t)(k - row * o.width);
                y = o.y0 + (uint32_t)row;
                g = ((uint64_t)y << 32) | x;
            } else if (o.form == kOriginCircle) {
                const uint64_t row = row_of(o.prefix, o.rows, k);
                const uint64_t first = o.prefix[row], half = (o.prefix[row + 1] - first) / 2;
                x = o.x0 - (uint32_t)half + (uint32_t)(k - first);
                y = o.y0 + (uint32_t)row;
                g = ((uint64_t)y << 32) | x;
            } else if (o.form == kOriginCells) {
                const uint64_t cell = row_of(o.prefix, o.rows, k);
                i = (uint32_t)(k - o.prefix[cell]);
                x = (uint32_t)(cell % o.width);
                y = (uint32_t)(cell / o.width);
            } else {
                const necsim_lineage l = o.given[k];
                x = l.x;
                y = l.y;
                i = l.index;
                g = l.global_reference;
                last = l.last_event_time;
            }
            const uint64_t d = o.offset + k;
            out.x[d] = x;
            out.y[d] = y;
            out.idx[d] = i;
            out.sim[d] = s;
            out.last[d] = last;
            out.gref[d] = g;
            out.steps[d] = 0;
            out.has_next[d] = 0;
            state[d] = 0;
            if (out.pred_end) out.pred_end[d] = 0.f;
        }
    }
}

cudaError_t launch_origins(const OriginSpec *specs, uint32_t n_sims, uint64_t n_total, const LineageSoA &out,
                           uint8_t *state, unsigned grid, cudaStream_t st) {
    if (n_sims == 0 || n_total == 0) return cudaSuccess;
    // about `grid` blocks in all, at least one per simulation (y <= 65,535)
    const uint32_t rows = n_sims < 65535u ? n_sims : 65535u;
    const uint64_t per_sim = (n_total / n_sims + 255) / 256 + 1;
    uint64_t cols = (grid + rows - 1) / rows;
    if (cols > per_sim) cols = per_sim;
    origins_kernel<<<dim3((unsigned)(cols ? cols : 1), rows), 256, 0, st>>>(specs, n_sims, out, state);
    return cudaGetLastError();
}

// The habitable locations of a WrappingNoise Rectangle sample
// (singleton_demes/rectangle.rs:93-120): counted, and appended to `out` when
// it is given.  `count` starts at zero.
__global__ void noise_origins_kernel(const NoiseHabitat *habitat, uint32_t x0, uint32_t y0, uint64_t width,
                                     uint64_t first_k, uint64_t n, necsim_lineage *out,
                                     unsigned long long *count) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = first_k + (uint64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint64_t k = base + threadIdx.x;
        uint32_t x = 0, y = 0;
        bool in = false;
        if (k < n) {
            const uint64_t row = k / width;
            x = x0 + (uint32_t)(k - row * width);
            y = y0 + (uint32_t)row;
            in = noise::habitat_at(*habitat, x, y) != 0;
        }
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        if (!mask) continue;
        unsigned long long first = 0;
        const unsigned lane = threadIdx.x & 31u;
        const int leader = __ffs(mask) - 1;
        if ((int)lane == leader) first = atomicAdd(count, (unsigned long long)__popc(mask));
        first = __shfl_sync(0xffffffffu, first, leader);
        if (in && out) {
            necsim_lineage l;
            l.global_reference = ((uint64_t)y << 32) | x;
            l.last_event_time = 0.0;
            l.x = x;
            l.y = y;
            l.index = 0;
            l.pad = 0;
            out[first + __popc(mask & ((1u << lane) - 1u))] = l;
        }
    }
}

cudaError_t launch_noise_origins(const NoiseHabitat *habitat, uint32_t x0, uint32_t y0, uint64_t width, uint64_t n,
                                 necsim_lineage *out, unsigned long long *count, unsigned grid, cudaStream_t st) {
    // launches of at most 2^26 locations, so none is long
    constexpr uint64_t kMost = 1ULL << 26;
    for (uint64_t k = 0; k < n; k += kMost) {
        const uint64_t end = n - k < kMost ? n : k + kMost, blocks = (end - k + 127) / 128;
        noise_origins_kernel<<<(unsigned)(blocks < grid ? blocks : grid), 128, 0, st>>>(habitat, x0, y0, width, k, end,
                                                                                      out, count);
    }
    return cudaGetLastError();
}

}  // namespace necsim
