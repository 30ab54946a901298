// shade_kernels.cuh — the shade-stage kernels (k_shade, k_shade_batch), included by
// the translation units that instantiate them: shade_kernels.cu (with the sampler,
// light sampling and hit record inlined) and shade_cache_kernels.cu (the radiance-cache
// instantiation, with them out of line). Internal linkage: each unit emits only the
// instantiations it uses.
#pragma once
#include "wavefront.cuh"

namespace luz {
namespace {


// Resident blocks per SM the register allocator is asked to allow. The kernels are bound by
// latency (path state, spills, instruction fetch): 1080p glossy frame at 64 spp, shade stage
// of the kernels without cold code: 6 blocks (80 registers) 56.1 ms, 5 (96) 56.5, 4 (128)
// 58.6, 8 (64) 61.0; Cornell box 300x300 at 50 spp 2.03, 1.96, 2.04, 2.55 ms. (Blocks of 768
// threads that start each 32 paths together, so that the warps of an SM share the
// instruction cache: 49.1 ms on that frame, but 2.15 ms on the box and 0.44 instead of
// 0.37 ms on a 96x64 preview.)
#ifndef LUZ_SHADE_MIN_BLOCKS
#define LUZ_SHADE_MIN_BLOCKS 6
#endif

// Path of shade slot i: slots run through the class segments in class order, from `first` on.
template <int FIRST>
__device__ __forceinline__ uint32_t binned_path(const PathBuf& P, const uint32_t* bin, uint32_t i)
{
    uint32_t k = FIRST, start = 0;
    while (k < kShadeClasses - 1 && i >= start + bin[k]) {
        start += bin[k];
        k++;
    }
    return P.bins[k * P.bin_stride + (i - start)];
}

// Paths of the part at this bounce.
template <int PART>
__device__ __forceinline__ uint32_t shade_count(const Ctrl* C, int bounce)
{
    if (PART == SHADE_MISSES) return C->bin[bounce][0];
    return C->count[bounce] - (PART == SHADE_HITS ? C->bin[bounce][0] : 0u);
}

template <int MODE, int PART, bool COLD>
__global__ void __launch_bounds__(kBlock, LUZ_SHADE_MIN_BLOCKS) k_shade(const DScene* __restrict__ Sp, WaveArgs w, PathBuf P, Ctrl* C, int bounce)
{
    const DScene& S = *Sp;
    const uint32_t count = shade_count<PART>(C, bounce);
    uint32_t* nq = (bounce & 1) ? P.queue0 : P.queue1;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    // a queue shorter than the grid is spread over all of its blocks
    const uint32_t wid = count >= warps * 32u ? (blockIdx.x * blockDim.x + threadIdx.x) >> 5
                                              : (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    for (uint32_t first = 0; first < count; first += warps * 32u) {
        const uint32_t base = first + wid * 32u;
        if (base >= count) break;
        const uint32_t i = base + lane_id();
        const bool valid = i < count;
        ShadeOut o;
        o.cont = false;
        o.sh[0] = o.sh[1] = false;
        uint32_t p = 0;
        if (valid) {
            p = binned_path<PART == SHADE_HITS ? 1 : 0>(P, C->bin[bounce], i);
            shade_path<MODE, PART, COLD>(S, w, P, p, bounce, o);
        }
        __syncwarp();
        const uint32_t qi = warp_append(&C->count[bounce + 1], o.cont);
        if (o.cont) nq[qi] = p;
        for (int slot = 0; slot < 2; slot++) {
            const uint32_t si = warp_append(&C->shadow[bounce], o.sh[slot]);
            if (o.sh[slot]) {
                P.sh_o[si] = make_float4(o.sh_o[slot].x, o.sh_o[slot].y, o.sh_o[slot].z, o.sh_t[slot]);
                P.sh_d[si] = make_float4(o.sh_d[slot].x, o.sh_d[slot].y, o.sh_d[slot].z,
                                         __uint_as_float(p | ((uint32_t)slot << 31)));
                P.sh_x[si] = make_int2(o.xobj, o.xprim);
            }
        }
    }
}

// The missed paths of a bounce: the sky, and the path ends. Half of the vertices of an open
// scene are misses, and their code needs 56 registers and no local memory where a hit's
// takes 80 and 416 bytes (kSplitShadePaths says when they get a launch of their own).
template <int MODE, bool COLD>
__global__ void __launch_bounds__(kBlock, 8) k_shade_misses(const DScene* __restrict__ Sp, WaveArgs w,
                                                                                 PathBuf P, Ctrl* C, int bounce)
{
    const DScene& S = *Sp;
    const uint32_t count = shade_count<SHADE_MISSES>(C, bounce);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        ShadeOut o;
        shade_path<MODE, SHADE_MISSES, COLD>(S, w, P, P.bins[i], bounce, o);
    }
}

// k_shade over a multi-scene wave: the scene and wave arguments are the path's segment's.
template <int MODE, bool COLD>
__global__ void __launch_bounds__(kBlock, LUZ_SHADE_MIN_BLOCKS) k_shade_batch(const DScene* __restrict__ scenes,
                                                                             const WaveArgs* __restrict__ segs,
                                                                             PathBuf P, Ctrl* C, int bounce)
{
    const uint32_t count = C->count[bounce];
    uint32_t* nq = (bounce & 1) ? P.queue0 : P.queue1;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    // a queue shorter than the grid is spread over all of its blocks
    const uint32_t wid = count >= warps * 32u ? (blockIdx.x * blockDim.x + threadIdx.x) >> 5
                                              : (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    for (uint32_t first = 0; first < count; first += warps * 32u) {
        const uint32_t base = first + wid * 32u;
        if (base >= count) break;
        const uint32_t i = base + lane_id();
        const bool valid = i < count;
        ShadeOut o;
        o.cont = false;
        o.sh[0] = o.sh[1] = false;
        uint32_t p = 0;
        if (valid) {
            p = binned_path<0>(P, C->bin[bounce], i);
            const WaveArgs& w = segs[P.seg[p]];
            shade_path<MODE, SHADE_ALL, COLD>(scenes[w.batch_scene], w, P, p, bounce, o);
        }
        __syncwarp();
        const uint32_t qi = warp_append(&C->count[bounce + 1], o.cont);
        if (o.cont) nq[qi] = p;
        for (int slot = 0; slot < 2; slot++) {
            const uint32_t si = warp_append(&C->shadow[bounce], o.sh[slot]);
            if (o.sh[slot]) {
                P.sh_o[si] = make_float4(o.sh_o[slot].x, o.sh_o[slot].y, o.sh_o[slot].z, o.sh_t[slot]);
                P.sh_d[si] = make_float4(o.sh_d[slot].x, o.sh_d[slot].y, o.sh_d[slot].z,
                                         __uint_as_float(p | ((uint32_t)slot << 31)));
                P.sh_x[si] = make_int2(o.xobj, o.xprim);
            }
        }
    }
}

}  // namespace
}  // namespace luz
