// mpm_edit.cu — COMPACT (deleteNear) and RAYCAST (raycastFluid) passes.
//
// The reference compacts with one atomic counter (shaders.js:542), so its
// survivor order depends on thread scheduling.  Here the survivors keep their
// index order (a deterministic order the reference can also produce): one pass
// counts survivors per block of kCompactTile particles, and a second writes
// each survivor at its block offset plus its rank inside the block (warp
// ballots).  A block adds up the counts before its own by itself up to
// kSelfScanBlocks blocks; beyond, where those reads would grow with the square
// of n, one block scans the counts in between.  Both passes stream the inputs
// with coalesced 16-byte loads, a thread's eight particles in flight at once:
// the work is HBM-bound (72 B per particle kept; the second read of the
// positions comes from L2 as far as they fit).
#include <cuda_runtime.h>

#include "mpm_device.cuh"
#include "mpm_edit.h"

namespace mpm {
namespace {

// shaders.js:80-84
__device__ __forceinline__ float ray_perp_dist(f3 pos, f3 origin, f3 dir) {
    const f3 to_p = sub(pos, origin);
    const float d = dot3(to_p, dir);
    const f3 perp = mk(to_p.x - d * dir.x, to_p.y - d * dir.y, to_p.z - d * dir.z);
    return len3(perp);
}

// shaders.js:536-540: a particle survives unless it lies inside the cylinder.
__device__ __forceinline__ bool survives(const float4 q, const mpm_ray_params& del) {
    return !(ray_perp_dist(mk(q.x, q.y, q.z), mk(del.ox, del.oy, del.oz), mk(del.dx, del.dy, del.dz)) < del.radius);
}

constexpr uint32_t kCompactWarps = kCompactThreads / 32;

// The positions of this thread's kCompactRounds particles (index base + r *
// kCompactThreads + thread) and which of them survive, as a ballot per round.
__device__ __forceinline__ void compact_load(const mpm_ray_params& del, uint32_t n, uint64_t base,
                                             const float4* __restrict__ pos, float4* q, uint32_t* keep) {
#pragma unroll
    for (uint32_t r = 0; r < kCompactRounds; ++r) {
        const uint64_t p = base + r * kCompactThreads + threadIdx.x;
        q[r] = p < n ? pos[p] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (uint32_t r = 0; r < kCompactRounds; ++r)
        keep[r] = __ballot_sync(0xffffffffu,
                                base + r * kCompactThreads + threadIdx.x < n && survives(q[r], del));
}

__global__ void __launch_bounds__(kCompactThreads) k_compact_count(mpm_ray_params del, uint32_t n,
                                                                   const float4* __restrict__ pos,
                                                                   uint32_t* __restrict__ counts) {
    __shared__ uint32_t ws[kCompactWarps];
    float4 q[kCompactRounds];
    uint32_t keep[kCompactRounds];
    compact_load(del, n, (uint64_t)blockIdx.x * kCompactTile, pos, q, keep);
    uint32_t total = 0;
#pragma unroll
    for (uint32_t r = 0; r < kCompactRounds; ++r) total += __popc(keep[r]);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        total = 0;
        for (uint32_t w = 0; w < kCompactWarps; ++w) total += ws[w];
        counts[blockIdx.x] = total;
    }
}

// One block: exclusive scan of the per-block counts in place; the total goes
// to *count_dev.
__global__ void __launch_bounds__(1024) k_compact_scan(uint32_t nblocks, uint32_t* __restrict__ counts,
                                                       uint32_t* __restrict__ count_dev) {
    __shared__ uint32_t ws[33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < nblocks; b0 += 1024) {
        const uint32_t b = b0 + threadIdx.x;
        const uint32_t x = b < nblocks ? counts[b] : 0u;
        uint32_t sc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, sc, o);
            if (lane >= o) sc += y;
        }
        if (lane == 31) ws[wid] = sc;
        __syncthreads();
        if (wid == 0) {
            const uint32_t w = ws[lane];
            uint32_t ww = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, ww, o);
                if (lane >= o) ww += y;
            }
            ws[lane] = ww - w;
            if (lane == 31) ws[32] = ww;
        }
        __syncthreads();
        if (b < nblocks) counts[b] = carry + ws[wid] + sc - x;
        carry += ws[32];
        __syncthreads();
    }
    if (threadIdx.x == 0) *count_dev = carry;
}

// counts: the survivors per block (scanned: their exclusive prefixes).
template <bool kScanned>
__global__ void __launch_bounds__(kCompactThreads) k_compact_write(mpm_ray_params del, uint32_t n,
                                                                   const float4* __restrict__ pos_in,
                                                                   const float4* __restrict__ vel_in,
                                                                   const float* __restrict__ mass_in,
                                                                   float4* __restrict__ pos_out,
                                                                   float4* __restrict__ vel_out,
                                                                   float* __restrict__ mass_out,
                                                                   const uint32_t* __restrict__ counts,
                                                                   uint32_t* __restrict__ count_dev) {
    __shared__ uint32_t wsum[kCompactRounds][kCompactWarps];
    __shared__ uint32_t part[kCompactWarps];
    const uint64_t base = (uint64_t)blockIdx.x * kCompactTile;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    float4 q[kCompactRounds];
    uint32_t keep[kCompactRounds];
    compact_load(del, n, base, pos_in, q, keep);
    if (lane == 0) {
#pragma unroll
        for (uint32_t r = 0; r < kCompactRounds; ++r) wsum[r][wid] = __popc(keep[r]);
    }
    uint32_t off = 0;
    if (kScanned) {
        off = counts[blockIdx.x];
    } else {
        for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kCompactThreads) off += counts[b];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) off += __shfl_xor_sync(0xffffffffu, off, d);
        if (lane == 0) part[wid] = off;
    }
    __syncthreads();
    if (!kScanned) {
        off = 0;
#pragma unroll
        for (uint32_t w = 0; w < kCompactWarps; ++w) off += part[w];
    }
    // first places of this warp's rounds
    uint32_t at[kCompactRounds];
#pragma unroll
    for (uint32_t r = 0; r < kCompactRounds; ++r) {
#pragma unroll
        for (uint32_t w = 0; w < kCompactWarps; ++w) {
            if (w == wid) at[r] = off;
            off += wsum[r][w];
        }
    }
    if (!kScanned && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *count_dev = off;
    // four rounds' velocities and masses in flight at a time
#pragma unroll
    for (uint32_t r0 = 0; r0 < kCompactRounds; r0 += 4) {
        float4 v[4];
        float m[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint64_t p = base + (r0 + k) * kCompactThreads + threadIdx.x;
            if ((keep[r0 + k] >> lane) & 1u) {
                v[k] = vel_in[p];
                m[k] = mass_in[p];
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if ((keep[r0 + k] >> lane) & 1u) {
                const uint32_t idx = at[r0 + k] + __popc(keep[r0 + k] & ((1u << lane) - 1u));
                pos_out[idx] = q[r0 + k];
                vel_out[idx] = v[k];
                mass_out[idx] = m[k];
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_raycast(mpm_ray_params ray, uint32_t n, const float4* __restrict__ pos,
                                                 uint32_t* __restrict__ hit) {
    const f3 origin = mk(ray.ox, ray.oy, ray.oz), dir = mk(ray.dx, ray.dy, ray.dz);
    uint32_t best = 0xFFFFFFFFu;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (uint64_t)gridDim.x * blockDim.x) {
        const float4 q = pos[p];
        const f3 pp = mk(q.x, q.y, q.z);
        const float t = dot3(sub(pp, origin), dir);            // shaders.js:570
        if (t <= 0.0f) continue;                                 // shaders.js:571
        if (ray_perp_dist(pp, origin, dir) >= ray.radius) continue;   // shaders.js:572
        const uint32_t bits = __float_as_uint(t);
        best = bits < best ? bits : best;                        // atomicMin on the bits (shaders.js:574)
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if ((threadIdx.x & 31) == 0 && best != 0xFFFFFFFFu) atomicMin(hit, best);
}

}  // namespace

cudaError_t launch_compact(const mpm_ray_params& del, uint32_t n, const float4* pos_in, const float4* vel_in,
                           const float* mass_in, float4* pos_out, float4* vel_out, float* mass_out,
                           uint32_t* scratch, uint32_t* count_dev, cudaStream_t stream) {
    if (n == 0) return cudaMemsetAsync(count_dev, 0, 4, stream);
    const uint32_t nblocks = (uint32_t)((n + (uint64_t)kCompactTile - 1) / kCompactTile);
    k_compact_count<<<nblocks, kCompactThreads, 0, stream>>>(del, n, pos_in, scratch);
    if (nblocks <= kSelfScanBlocks) {
        k_compact_write<false><<<nblocks, kCompactThreads, 0, stream>>>(del, n, pos_in, vel_in, mass_in, pos_out, vel_out,
                                                                        mass_out, scratch, count_dev);
    } else {
        k_compact_scan<<<1, 1024, 0, stream>>>(nblocks, scratch, count_dev);
        k_compact_write<true><<<nblocks, kCompactThreads, 0, stream>>>(del, n, pos_in, vel_in, mass_in, pos_out, vel_out,
                                                                       mass_out, scratch, count_dev);
    }
    return cudaGetLastError();
}

cudaError_t launch_raycast(const mpm_ray_params& ray, uint32_t n, const float4* pos_in, uint32_t* hit_dev,
                           cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(hit_dev, 0xFF, 4, stream);   // fluid-gpu.js:601 sentinel
    if (e != cudaSuccess || n == 0) return e;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t want = (n + 255u) / 256u;
    const uint32_t blocks = (uint32_t)(want < (uint64_t)sms * 8 ? want : (uint64_t)sms * 8);
    k_raycast<<<blocks, 256, 0, stream>>>(ray, n, pos_in, hit_dev);
    return cudaGetLastError();
}

}  // namespace mpm
