// shade_kernels.cu — the shade stage of the wavefront integrator, in a
// translation unit of its own built with FMA contraction (-fmad=true).
//
// Traversal (trace.cuh), ray generation and the film stay in integrator.cu,
// built with -fmad=false: there every FP32 expression rounds as written, so
// the GPU hits equal the FP32 restatement's bit for bit. Shading is compared
// with the FP64 reference within a relative tolerance, where contracting a
// product and a sum into one rounding only removes error; the sampler's FP64
// lattice arithmetic (dmath.cuh) is written with explicit round-to-nearest
// intrinsics, so it stays bit-exact with the reference in either unit.
#define LUZ_NO_CACHE_KERNELS
// Inlined here, out of line elsewhere: the sampler, the environment and light
// sampling / pdf functions and the hit record. With the paths binned by material
// class the shade kernel's instruction footprint no longer stalls it, and these
// calls' argument traffic through local memory cost more (1080p glossy frame, 16
// spp: shade stage 29.5 -> 25.8 ms). Inlining the BSDF functions as well made it
// slower (37.7 ms: 128 registers could no longer hold the larger body).
#define LUZ_SAMPLER_ATTR __forceinline__
#define LUZ_LIGHT_ATTR __forceinline__
#define LUZ_HIT_ATTR __forceinline__
#include "shade_kernels.cuh"

namespace luz {

// The gradients of a wave's visits of the differentiated texture, its paths ended.
__global__ void k_adjoint_vertices(const DScene* __restrict__ Sp, WaveArgs w, PathBuf P)
{
    const DScene& S = *Sp;
    const unsigned long long n = min(*w.adj_count, w.adj_cap), step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const AdjVertex v = w.adj_vertices[i];
        const float4 r = P.rad[v.path], a = P.pend0[v.path], b = P.pend1[v.path];
        const F3 L = (F3{r.x, r.y, r.z} + F3{a.x, a.y, a.z}) + F3{b.x, b.y, b.z};
        adjoint_texture(S, w, P.pixel[v.path], L, v.u, v.v, F3{v.before[0], v.before[1], v.before[2]});
    }
}

AdjointVerticesKernel adjoint_vertices_kernel() { return k_adjoint_vertices; }

BatchShadeKernel batch_shade_kernel(int mode, bool cold)
{
    return mode == 1 ? k_shade_batch<1, true> : cold ? k_shade_batch<0, true> : k_shade_batch<0, false>;
}

ShadeKernel shade_kernel(int mode, int part, bool cold)
{
    if (mode == 2) return shade_kernel_cached(cold);
    if (mode == 3) return cold ? k_shade<3, SHADE_ALL, true> : k_shade<3, SHADE_ALL, false>;
    if (part == SHADE_MISSES) return cold ? k_shade_misses<0, true> : k_shade_misses<0, false>;
    if (mode == 1)
        return part == SHADE_HITS       ? k_shade<1, SHADE_HITS, true>
               : part == SHADE_FEATURES ? k_shade<1, SHADE_FEATURES, true>
                                        : k_shade<1, SHADE_ALL, true>;
    if (cold)
        return part == SHADE_HITS       ? k_shade<0, SHADE_HITS, true>
               : part == SHADE_FEATURES ? k_shade<0, SHADE_FEATURES, true>
                                        : k_shade<0, SHADE_ALL, true>;
    return part == SHADE_HITS       ? k_shade<0, SHADE_HITS, false>
           : part == SHADE_FEATURES ? k_shade<0, SHADE_FEATURES, false>
                                    : k_shade<0, SHADE_ALL, false>;
}

}  // namespace luz
