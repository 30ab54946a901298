// trace.cuh — closest-hit and any-hit traversal of the two-level scene.
//
// Semantics follow the reference exactly (tie order included):
//   Renderer::internal::_checkHits          src/renderer/HitHelper.cpp:5-32
//   isShadowOccluded                        src/renderer/ColorHelper.cpp:801-829
//   BVHNode::hit / hitAny                   src/core/Hittables/BVHNode.cpp:221-380
//     1 or 3 children: index order, each child does its own test;
//     2 children: near-first, swap only on strict <, second needs near < closest;
//     >= 4 children: stable insertion sort by near, skip near >= closest.
//   Mesh::hit / hitAny                      src/core/Hittables/Mesh.cpp:578-735
//     explicit stack, prune near >= closest, ties push the right child last
//     (visited first); leaf triangles in order, later equal-t triangle wins.
//   Triangle::hit (Moller-Trumbore)         src/core/Hittables/Triangle.cpp:196-305
//   MeshInstance::hit / hitAny              src/core/Hittables/MeshInstance.cpp:251-327
//   Rectangle / Sphere / Cube / Plane / ConstantVolume intersectors.
// Arithmetic is FP32 with the reference's operation order (-fmad=false), so
// oracle/restate.cpp reproduces every hit bit for bit on the same packed arrays.
#pragma once
#include "dmath.cuh"

namespace luz {

// Caustic photon map of the current render (caustics.cuh): photons in grid-cell
// order, three float4 each, and an open-addressing table from packed cell key
// to the cell's [begin, end) photon range. count = 0: no map.
struct DCaustics {
    const float4* photons;
    const unsigned long long* cell_keys;
    const uint2* cell_ranges;
    uint32_t mask;
    uint32_t count;
};

struct DScene {
    const GRect* rects;
    const GObject* objects;
    const GTopNode* top_nodes;
    const GTopChild* top_children;
    const GNode4* nodes4;      // collapsed mesh BVH
    const GTri* tris;
    const GTriShade* tri_shade;
    const float* vnormals;
    const float* vuvs;
    const GMesh* meshes;
    const GMaterial* materials;
    const GTexture* textures;
    const float4* texels;
    const GLight* lights;
    const GIes* ies;
    const double* cdf;
    const int32_t* index_pool;
    const float4* env_texels;
    const uint8_t* obj_class;  // material type a hit on each object shades with (shade binning)
    uint32_t* error;          // device error word (bit flags)
    unsigned long long* counters;   // LUZ_RENDER_COUNT: ext nodes/tris/top, shadow nodes/tris/top,
                                    // ext / shadow binary-node visits (read by the counting
                                    // instantiations of the trace kernels only)
    int32_t mesh_stack_limit;       // traversal stack bounds enforced (<= kMeshStack4 / kTopStack;
    int32_t top_stack_limit;        // lowered only by luz_gpu_scene_set_traversal_limits)
    uint32_t top4_base;             // staged nodes: [top4_base, top4_base + top4_count) of nodes4, the
    uint32_t top4_count;            // breadth-first top of the scene's largest mesh (0: none)
    DCaustics cm;
    GSceneConst k;
};

enum ErrBits : uint32_t { ERR_TOP_STACK = 1u, ERR_MESH_STACK = 2u, ERR_CAUSTIC_GRID = 4u };

// Scene features a traversal kernel is instantiated for (GSceneConst.features).
// A kernel compiled without a feature never meets that object kind in its
// scene. (Analytic primitives are always compiled in: an instantiation with
// meshes as its only kind measured 2.3x slower in the any-hit kernel, at 2.4
// instead of 6.1 active threads per warp instruction.)
// TF_STAGED: the kernel has staged the scene's top collapsed nodes in shared
// memory (stage_top_nodes) and the mesh walks read them there.
enum TraceFeature : uint32_t { TF_INSTANCE = 1u, TF_VOLUME = 2u, TF_ALL = 3u, TF_STAGED = 4u };

// The staged nodes of a trace kernel's block.
static __shared__ __align__(128) float4 s_top4[kTopNodes4 * 8];

// Copies the staged node range into shared memory; every thread of the block calls it
// once, before its first traversal.
__device__ __forceinline__ void stage_top_nodes(const DScene& S)
{
    const float4* src = reinterpret_cast<const float4*>(S.nodes4 + S.top4_base);
    for (uint32_t i = threadIdx.x; i < S.top4_count * 8u; i += blockDim.x) s_top4[i] = __ldg(src + i);
    __syncthreads();
}

// xobj / xprim name the primitive a secondary ray leaves from. A ray that
// starts on a planar primitive cannot meet it again at t > 0 in exact
// arithmetic (the reference's FP64 hits never do, they fall below T_MIN), so
// the FP32 traversal skips that primitive instead of re-hitting it through
// rounding error at grazing angles; for the source sphere an outgoing ray
// skips it and an entering ray keeps only the far root.
struct TRay {
    F3 o, d, inv;
    bool zero;
    bool axis0;      // some inverse-direction component is 0 (axis-parallel ray)
    int32_t xobj, xprim;
};

__device__ __forceinline__ float inv_component(float c)
{
    if (c == 0.0f || !isfinite(c)) return 0.0f;
    const float i = 1.0f / c;
    return isfinite(i) ? i : 0.0f;
}
__device__ __forceinline__ TRay make_ray(F3 o, F3 d)
{
    TRay r;
    r.o = o;
    r.d = d;
    r.inv = F3{inv_component(d.x), inv_component(d.y), inv_component(d.z)};
    r.zero = (d.x == 0.0f && d.y == 0.0f && d.z == 0.0f);
    r.axis0 = r.inv.x == 0.0f || r.inv.y == 0.0f || r.inv.z == 0.0f;
    r.xobj = -1;
    r.xprim = -1;
    return r;
}
__device__ __forceinline__ TRay make_ray_x(F3 o, F3 d, int32_t xobj, int32_t xprim)
{
    TRay r = make_ray(o, d);
    r.xobj = xobj;
    r.xprim = xprim;
    return r;
}

struct THit {
    float t;
    int32_t obj;     // GObject index, -1 = miss
    int32_t prim;    // mesh: leaf slot of the triangle; cube: face; else 0
    float u, v;
};

// Per-ray traversal context: the volume distance sample (evaluated once, on first use).
struct VolSample {
    const Key* key;
    double u;
    bool have;
    __device__ __forceinline__ double get()
    {
        if (!have) {
            u = sample1d(*key, DIM_VOLUME_DISTANCE);
            have = true;
        }
        return u;
    }
};

// boxHitDistance / AABB::hit (Mesh.cpp:99-139, BVHNode.cpp:20-60, AABB.cpp:37-71).
// For a ray with no zero inverse component the per-axis swap and the running
// max/min are written as selects (same values as the reference's sequence: the
// early exit on tmax <= tmin is monotone, so testing once at the end is equal).
__device__ __forceinline__ bool box_hit(const float* mn, const float* mx, const TRay& r, float tmax, float& tnear)
{
    if (r.zero) return false;
    float tmin = kTMin;
    const float o[3] = {r.o.x, r.o.y, r.o.z};
    const float iv[3] = {r.inv.x, r.inv.y, r.inv.z};
    if (!r.axis0) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float t0 = (mn[a] - o[a]) * iv[a];
            const float t1 = (mx[a] - o[a]) * iv[a];
            tmin = fmaxf(tmin, fminf(t0, t1));
            tmax = fminf(tmax, fmaxf(t0, t1));
        }
        tnear = tmin;
        return !(tmax <= tmin);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float inv = iv[a];
        if (inv == 0.0f) {
            if (o[a] < mn[a] || o[a] > mx[a]) return false;
            continue;
        }
        float t0 = (mn[a] - o[a]) * inv;
        float t1 = (mx[a] - o[a]) * inv;
        if (inv < 0.0f) {
            const float sw = t0;
            t0 = t1;
            t1 = sw;
        }
        tmin = t0 > tmin ? t0 : tmin;
        tmax = t1 < tmax ? t1 : tmax;
        if (tmax <= tmin) return false;
    }
    tnear = tmin;
    return true;
}

__device__ __forceinline__ float fmax3f(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3f(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Mesh-box slab test in the form t = plane * inv + noi with noi = -(o * inv)
// rounded once per ray: one FMA per plane instead of a subtraction and a
// product, and three-input min/max for the running interval. Equal to
// box_hit in real arithmetic; in FP32 each distance is off by less than
// 2^-24 (|o| + |t d|) / |d| along its axis, below the T_MIN padding of every
// mesh box (Triangle.cpp:114-125) while |o| < 4096 and the mesh lies within
// 8192 units of the origin: mesh_fast_slabs checks both.
__device__ __forceinline__ bool mesh_fast_slabs(const GMesh& M, const TRay& r)
{
    const float om = fmax3f(fabsf(r.o.x), fabsf(r.o.y), fabsf(r.o.z));
    const float mm = fmaxf(fmax3f(fabsf(M.bmin[0]), fabsf(M.bmin[1]), fabsf(M.bmin[2])),
                           fmax3f(fabsf(M.bmax[0]), fabsf(M.bmax[1]), fabsf(M.bmax[2])));
    return !r.zero && !r.axis0 && om < 4096.0f && mm < 8192.0f;
}
__device__ __forceinline__ F3 neg_o_inv(const TRay& r)
{
    return F3{-(r.o.x * r.inv.x), -(r.o.y * r.inv.y), -(r.o.z * r.inv.z)};
}
__device__ __forceinline__ bool box_hit_fast(const float* mn, const float* mx, const TRay& r, const F3& noi, float tmax,
                                             float& tnear)
{
    const float t0x = fmaf(mn[0], r.inv.x, noi.x), t1x = fmaf(mx[0], r.inv.x, noi.x);
    const float t0y = fmaf(mn[1], r.inv.y, noi.y), t1y = fmaf(mx[1], r.inv.y, noi.y);
    const float t0z = fmaf(mn[2], r.inv.z, noi.z), t1z = fmaf(mx[2], r.inv.z, noi.z);
    const float lo = fmax3f(fmaxf(kTMin, fminf(t0x, t1x)), fminf(t0y, t1y), fminf(t0z, t1z));
    const float hi = fmin3f(fminf(tmax, fmaxf(t0x, t1x)), fmaxf(t0y, t1y), fmaxf(t0z, t1z));
    tnear = lo;
    return !(hi <= lo);
}
// Mesh box test: the FMA form (FAST) or box_hit. noi = neg_o_inv(r) (FAST only).
template <bool FAST>
__device__ __forceinline__ bool mesh_box(const float* mn, const float* mx, const TRay& r, const F3& noi, float tmax,
                                         float& tnear)
{
    if constexpr (FAST) return box_hit_fast(mn, mx, r, noi, tmax, tnear);
    else return box_hit(mn, mx, r, tmax, tnear);
}

__device__ __forceinline__ bool tri_test(const GTri& T, const TRay& r, float tmin, float tmax, float& t, float& u, float& v)
{
    const F3 e1 = f3(T.e1), e2 = f3(T.e2), v0 = f3(T.v0);
    const F3 p = cross(r.d, e2);
    const float det = dot(e1, p);
    if (fabsf(det) < 1e-12f) return false;
    const float inv_det = 1.0f / det;
    const F3 tv = r.o - v0;
    u = dot(tv, p) * inv_det;
    if (u < 0.0f || u > 1.0f) return false;
    const F3 q = cross(tv, e1);
    v = dot(r.d, q) * inv_det;
    if (v < 0.0f || u + v > 1.0f) return false;
    t = dot(e2, q) * inv_det;
    return !(t > tmax || t < tmin);
}

__device__ __forceinline__ GTri load_tri(const GTri* tris, uint32_t i)
{
    const float4* p = reinterpret_cast<const float4*>(tris + i);
    const float4 a = ld4(p), b = ld4(p + 1), c = ld4(p + 2);
    GTri t;
    t.v0[0] = a.x; t.v0[1] = a.y; t.v0[2] = a.z; t.orig = __float_as_uint(a.w);
    t.e1[0] = b.x; t.e1[1] = b.y; t.e1[2] = b.z; t.area = b.w;
    t.e2[0] = c.x; t.e2[1] = c.y; t.e2[2] = c.z; t.pad = 0;
    return t;
}
// Address of a collapsed node: the staged copy when it lies in the staged range, else
// global memory (the same bytes either way).
template <uint32_t F>
__device__ __forceinline__ const char* node4_at(const DScene& S, uint32_t ref)
{
    if constexpr ((F & TF_STAGED) != 0) {
        const uint32_t j = ref - S.top4_base;
        if (j < S.top4_count) return reinterpret_cast<const char*>(s_top4 + 8 * j);
    }
    return reinterpret_cast<const char*>(S.nodes4 + ref);
}
template <uint32_t F, class T>
__device__ __forceinline__ T node4_ld(const char* p)
{
    if constexpr ((F & TF_STAGED) != 0) return *reinterpret_cast<const T*>(p);
    else return __ldg(reinterpret_cast<const T*>(p));
}

// The four entry boxes of a collapsed node against a ray: which are met before tmax,
// their entry distances and, for the visit order, those of the two sides (nl: slots 0
// and 1, nr: slots 2 and 3; meaningful where the side holds an accepted entry).
struct Node4Test {
    bool ha[4];
    float na[4];
    float nl, nr;
    bool hl, hr;   // SIDES: the side boxes themselves are met
    uint32_t ref[4];
};

// FAST: the ray's sign picks each axis's near and far planes at the load, so that a box
// costs six FMAs, a three-input max and min each with one more, and a comparison, with no
// per-plane min / max: the fma is monotone in the plane, so near <= far as box_hit_fast's
// min and max would order them. A side's entry distance follows from its slots' near
// distances (the side's box is the union of its slots' boxes and the fma is monotone, so
// its near distance along an axis is the smaller of the slots'): the same values as a test
// of the stored side box, for five operations instead of eleven and three loads less.
template <bool FAST, uint32_t F, bool ORDER, bool SIDES>
__device__ __forceinline__ void node4_test(const DScene& S, uint32_t nref, const TRay& r, float tmax, Node4Test& T)
{
    const char* p = node4_at<F>(S, nref);
    const uint4 rf = node4_ld<F, uint4>(p + 48);
    T.ref[0] = rf.x;
    T.ref[1] = rf.y;
    T.ref[2] = rf.z;
    T.ref[3] = rf.w;
    if constexpr (FAST) {
        const F3 noi = neg_o_inv(r);
        const uint32_t sx = (__float_as_uint(r.inv.x) >> 31) << 6, sy = (__float_as_uint(r.inv.y) >> 31) << 6,
                       sz = (__float_as_uint(r.inv.z) >> 31) << 6;
        const float4 ax = node4_ld<F, float4>(p + sx), ay = node4_ld<F, float4>(p + 16 + sy),
                     az = node4_ld<F, float4>(p + 32 + sz);
        const float4 bx = node4_ld<F, float4>(p + (64u - sx)), by = node4_ld<F, float4>(p + 16 + (64u - sy)),
                     bz = node4_ld<F, float4>(p + 32 + (64u - sz));
        const float nx[4] = {fmaf(ax.x, r.inv.x, noi.x), fmaf(ax.y, r.inv.x, noi.x), fmaf(ax.z, r.inv.x, noi.x),
                             fmaf(ax.w, r.inv.x, noi.x)};
        const float ny[4] = {fmaf(ay.x, r.inv.y, noi.y), fmaf(ay.y, r.inv.y, noi.y), fmaf(ay.z, r.inv.y, noi.y),
                             fmaf(ay.w, r.inv.y, noi.y)};
        const float nz[4] = {fmaf(az.x, r.inv.z, noi.z), fmaf(az.y, r.inv.z, noi.z), fmaf(az.z, r.inv.z, noi.z),
                             fmaf(az.w, r.inv.z, noi.z)};
        const float fx[4] = {fmaf(bx.x, r.inv.x, noi.x), fmaf(bx.y, r.inv.x, noi.x), fmaf(bx.z, r.inv.x, noi.x),
                             fmaf(bx.w, r.inv.x, noi.x)};
        const float fy[4] = {fmaf(by.x, r.inv.y, noi.y), fmaf(by.y, r.inv.y, noi.y), fmaf(by.z, r.inv.y, noi.y),
                             fmaf(by.w, r.inv.y, noi.y)};
        const float fz[4] = {fmaf(bz.x, r.inv.z, noi.z), fmaf(bz.y, r.inv.z, noi.z), fmaf(bz.z, r.inv.z, noi.z),
                             fmaf(bz.w, r.inv.z, noi.z)};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            T.na[k] = fmax3f(fmaxf(kTMin, nx[k]), ny[k], nz[k]);
            T.ha[k] = !(fmin3f(fminf(tmax, fx[k]), fy[k], fz[k]) <= T.na[k]);
        }
        if constexpr (ORDER) {
            T.nl = fmax3f(fmaxf(kTMin, fminf(nx[0], nx[1])), fminf(ny[0], ny[1]), fminf(nz[0], nz[1]));
            T.nr = fmax3f(fmaxf(kTMin, fminf(nx[2], nx[3])), fminf(ny[2], ny[3]), fminf(nz[2], nz[3]));
        }
        if constexpr (SIDES) {
            T.hl = !(fmin3f(fminf(tmax, fmaxf(fx[0], fx[1])), fmaxf(fy[0], fy[1]), fmaxf(fz[0], fz[1])) <= T.nl);
            T.hr = !(fmin3f(fminf(tmax, fmaxf(fx[2], fx[3])), fmaxf(fy[2], fy[3]), fmaxf(fz[2], fz[3])) <= T.nr);
        }
    } else {
        const float4 lo[3] = {node4_ld<F, float4>(p), node4_ld<F, float4>(p + 16), node4_ld<F, float4>(p + 32)};
        const float4 hi[3] = {node4_ld<F, float4>(p + 64), node4_ld<F, float4>(p + 80), node4_ld<F, float4>(p + 96)};
        const float mn[4][3] = {{lo[0].x, lo[1].x, lo[2].x}, {lo[0].y, lo[1].y, lo[2].y},
                                {lo[0].z, lo[1].z, lo[2].z}, {lo[0].w, lo[1].w, lo[2].w}};
        const float mx[4][3] = {{hi[0].x, hi[1].x, hi[2].x}, {hi[0].y, hi[1].y, hi[2].y},
                                {hi[0].z, hi[1].z, hi[2].z}, {hi[0].w, hi[1].w, hi[2].w}};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            T.na[k] = 0.f;
            T.ha[k] = T.ref[k] != kEmptySlot && box_hit(mn[k], mx[k], r, tmax, T.na[k]);
        }
        if constexpr (ORDER) {
#pragma unroll
            for (int s = 0; s < 2; s++) {
                float umn[3], umx[3], n = 0.f;
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    umn[a] = fminf(mn[2 * s][a], mn[2 * s + 1][a]);
                    umx[a] = fmaxf(mx[2 * s][a], mx[2 * s + 1][a]);
                }
                const bool h = box_hit(umn, umx, r, tmax, n);
                if (s) {
                    T.nr = n;
                    T.hr = h;
                } else {
                    T.nl = n;
                    T.hl = h;
                }
            }
        }
    }
}

// The accepted entries of a collapsed node in visit order: the nearer side first (ties:
// the right one), and on a side the nearer entry first (ties: the right one).
struct Node4Order {
    uint32_t ref[4];
    float near[4];
    bool on[4];   // first side's first, its second, the other side's first, its second
};
__device__ __forceinline__ void node4_order(const Node4Test& T, Node4Order& O)
{
    // second entry of a side first unless the first is accepted and strictly nearer
    const bool lswap = T.ha[1] && !(T.ha[0] && T.na[0] < T.na[1]);
    const bool rswap = T.ha[3] && !(T.ha[2] && T.na[2] < T.na[3]);
    const bool l1 = T.ha[0] || T.ha[1], l2 = T.ha[0] && T.ha[1];
    const bool r1 = T.ha[2] || T.ha[3], r2 = T.ha[2] && T.ha[3];
    const bool rf = r1 && !(l1 && T.nl < T.nr);
    const uint32_t la = lswap ? T.ref[1] : T.ref[0], lb = lswap ? T.ref[0] : T.ref[1];
    const uint32_t ra = rswap ? T.ref[3] : T.ref[2], rb = rswap ? T.ref[2] : T.ref[3];
    const float lan = lswap ? T.na[1] : T.na[0], lbn = lswap ? T.na[0] : T.na[1];
    const float ran = rswap ? T.na[3] : T.na[2], rbn = rswap ? T.na[2] : T.na[3];
    O.ref[0] = rf ? ra : la;
    O.near[0] = rf ? ran : lan;
    O.on[0] = l1 || r1;
    O.ref[1] = rf ? rb : lb;
    O.near[1] = rf ? rbn : lbn;
    O.on[1] = rf ? r2 : l2;
    O.ref[2] = rf ? la : ra;
    O.near[2] = rf ? lan : ran;
    O.on[2] = l1 && r1;
    O.ref[3] = rf ? lb : rb;
    O.near[3] = rf ? lbn : rbn;
    O.on[3] = l1 && r1 && (rf ? l2 : r2);
}

// Visit order of a collapsed node's entries, as the binary near-first
// traversal (Mesh::hit, Mesh.cpp:578-660) would reach them: the nearer of L
// and R first (ties: R), and within each the nearer child first (ties: the
// right one): node4_order.
//
// Testing all boxes at N's visit instead of at L's and R's gives the same
// visits: L is visited right after N (nothing changes `closest` in between),
// and an entry of R's side that the binary traversal would reject later,
// because `closest` shrank meanwhile, has near >= closest by then and is
// pruned when popped. Child boxes lie inside their parent's (the node boxes
// are unions of their triangles' boxes, rounded outward), so a grandchild's
// entry distance is never below its parent's and a grandchild of a rejected
// child is itself rejected.

// Mesh traversal stack in the thread's local memory: node or leaf reference
// and near distance per entry.
struct LocalStack {
    uint32_t r[kMeshStack4];
    float n[kMeshStack4];
    __device__ __forceinline__ void set(int d, uint32_t ref, float near)
    {
        r[d] = ref;
        n[d] = near;
    }
    __device__ __forceinline__ uint32_t ref(int d) const { return r[d]; }
    __device__ __forceinline__ float near(int d) const { return n[d]; }
};

// Mesh::hit — closest triangle; closest is updated in place.
template <bool FAST, uint32_t F, class Stk>
__device__ __forceinline__ bool mesh_closest_walk(const DScene& S, const GMesh& M, const TRay& r, float tmin,
                                                  float& closest, int32_t& slot, float& bu, float& bv, int32_t skip,
                                                  Stk& st)
{
    float root_near;
    if (!mesh_box<FAST>(M.bmin, M.bmax, r, neg_o_inv(r), closest, root_near)) return false;
    // Walks the collapsed BVH. The entry about to be visited stays in
    // registers (ref, near); a node visit pushes the other accepted entries in
    // reverse visit order. Pruning (near >= closest) happens when an entry is
    // reached, as in the reference.
    uint32_t ref = (uint32_t)M.root4_ref;
    float near = root_near;
    int sp = 0;
    bool hit = false;
    while (true) {
        if (!(near >= closest)) {
            if (ref & kLeafBit) {
                const uint32_t first = (ref & 0x7fffffffu) >> 3;
                const uint32_t cnt = (ref & 7u) + 1u;
                for (uint32_t i = first; i < first + cnt; i++) {
                    if ((int32_t)i == skip) continue;
                    const GTri T = load_tri(S.tris, i);
                    float t, u, v;
                    if (tri_test(T, r, tmin, closest, t, u, v)) {
                        closest = t;
                        slot = (int32_t)i;
                        bu = u;
                        bv = v;
                        hit = true;
                    }
                }
            } else {
                Node4Test T;
                node4_test<FAST, F, true, false>(S, ref, r, closest, T);
                const int ne = (int)T.ha[0] + (int)T.ha[1] + (int)T.ha[2] + (int)T.ha[3];
                if (sp + ne > S.mesh_stack_limit) {
                    atomicOr(S.error, ERR_MESH_STACK);
                    break;
                }
                if (ne > 0) {
                    Node4Order o;
                    node4_order(T, o);
#pragma unroll
                    for (int k = 3; k > 0; k--)
                        if (o.on[k]) st.set(sp++, o.ref[k], o.near[k]);
                    ref = o.ref[0];
                    near = o.near[0];
                    continue;
                }
            }
        }
        if (sp == 0) break;
        sp--;
        ref = st.ref(sp);
        near = st.near(sp);
    }
    return hit;
}

template <uint32_t F, class Stk>
__device__ __forceinline__ bool mesh_closest(const DScene& S, const GMesh& M, const TRay& r, float tmin, float& closest,
                                             int32_t& slot, float& bu, float& bv, int32_t skip, Stk& st)
{
    if (mesh_fast_slabs(M, r)) return mesh_closest_walk<true, F>(S, M, r, tmin, closest, slot, bu, bv, skip, st);
    return mesh_closest_walk<false, F>(S, M, r, tmin, closest, slot, bu, bv, skip, st);
}

// Rectangle::hit geometric test (Rectangle.cpp:212-249); returns t.
__device__ __forceinline__ bool rect_test(const GRect& R, const TRay& r, float tmin, float tmax, float& t)
{
    if (R.w <= 0.0f || R.h <= 0.0f) return false;
    const F3 p = f3(R.p), n = f3(R.n);
    const float a = dot(r.o - p, n);
    const float b = dot(r.d, n);
    if (b == 0.0f || (a < 0.0f && b < 0.0f) || (a > 0.0f && b > 0.0f)) return false;
    t = -a / b;
    if (t > tmax || t < tmin) return false;
    const F3 d = (r.o + (t * r.d)) - p;
    const float wd = dot(d, f3(R.wa));
    const float hd = dot(d, f3(R.ha));
    return !(fabsf(wd) > R.hw || fabsf(hd) > R.hh);
}

// Sphere::hit / hitAny root selection (Sphere.cpp:227-302).
__device__ __forceinline__ bool sphere_test(const GObject& O, const TRay& r, float tmin, float tmax, float& t,
                                            bool source = false)
{
    if (O.f[4] == 0.0f || r.zero) return false;
    const F3 c = f3(O.f);
    const float rad = O.f[3];
    const F3 oc = r.o - c;
    const float b = dot(oc, r.d);
    if (source && b >= 0.0f) return false;   // leaving the source sphere
    // b^2 - (|oc|^2 - r^2) as r^2 - |oc - b d|^2: equal for a unit direction, free of cancellation.
    const F3 f = oc - b * r.d;
    const float disc = (rad * rad) - len2(f);
    if (disc < 0.0f) return false;
    const float sq = sqrtf(disc);
    float root = -b - sq;
    if (source || root < tmin || root > tmax) {
        root = -b + sq;
        if (root < tmin || root > tmax) return false;
    }
    t = root;
    return true;
}

__device__ __forceinline__ bool plane_test(const GObject& O, const TRay& r, float tmin, float tmax, float& t)
{
    const F3 n = f3(O.f + 1);
    const F3 pos = F3{0.0f, O.f[0], 0.0f};
    const float d = dot(r.d, n);
    if (d == 0.0f) return false;
    t = dot(pos - r.o, n) / d;
    return !(t > tmax || t < tmin);
}

// MeshInstance::_localRay (MeshInstance.cpp:245-265) with InstanceTransform inverses.
__device__ __forceinline__ F3 inv_rotate(const GObject& O, F3 v)
{
    const float cx = O.f[6], sx = O.f[7], cy = O.f[8], sy = O.f[9], cz = O.f[10], sz = O.f[11];
    float x = v.x, y = v.y, z = v.z;
    float nx = (x * cz) + (y * sz);
    float ny = (-x * sz) + (y * cz);
    x = nx;
    y = ny;
    nx = (x * cy) - (z * sy);
    float nz = (x * sy) + (z * cy);
    x = nx;
    z = nz;
    ny = (y * cx) + (z * sx);
    nz = (-y * sx) + (z * cx);
    return F3{x, ny, nz};
}
__device__ __forceinline__ F3 fwd_rotate(const GObject& O, F3 v)
{
    const float cx = O.f[6], sx = O.f[7], cy = O.f[8], sy = O.f[9], cz = O.f[10], sz = O.f[11];
    float x = v.x, y = v.y, z = v.z;
    float ny = (y * cx) - (z * sx);
    float nz = (y * sx) + (z * cx);
    y = ny;
    z = nz;
    float nx = (x * cy) + (z * sy);
    nz = (-x * sy) + (z * cy);
    x = nx;
    z = nz;
    nx = (x * cz) - (y * sz);
    ny = (x * sz) + (y * cz);
    return F3{nx, ny, z};
}
__device__ __forceinline__ bool instance_invertible(const GObject& O)
{
    return fabsf(O.f[3]) > 1e-12f && fabsf(O.f[4]) > 1e-12f && fabsf(O.f[5]) > 1e-12f;
}
__device__ __forceinline__ bool local_ray(const GObject& O, const TRay& r, TRay& lr, float& scale)
{
    if (!instance_invertible(O)) return false;
    const F3 s = f3(O.f + 3);
    const F3 ur = inv_rotate(O, r.d);
    const F3 ld = F3{ur.x / s.x, ur.y / s.y, ur.z / s.z};
    scale = sqrtf(len2(ld));
    if (!isfinite(scale) || scale <= 0.0f) return false;
    const F3 uo = inv_rotate(O, r.o - f3(O.f));
    const F3 lo = F3{uo.x / s.x, uo.y / s.y, uo.z / s.z};
    if (!isfinite(lo.x) || !isfinite(lo.y) || !isfinite(lo.z)) return false;
    lr = make_ray_x(lo, vdiv(ld, scale), r.xobj, r.xprim);
    return true;
}

// ConstantVolume::sampleScatteringDistance (ConstantVolume.cpp:62-121) with the
// boundary's hitInterval(-T_MAX, T_MAX) (Cube.cpp:134-175, Sphere.cpp:304-343).
// Length (scene units along the ray) of the part of [tmin, tmax] inside the
// boundary of volume O: the interval volume_distance samples in.
static __device__ float volume_overlap(const GObject& O, F3 o, F3 d, float tmin, float tmax)
{
    float entry, exit;
    if (O.aux == 3 /* LUZ_OBJ_CUBE */) {
        float imin = -kInf, imax = kInf;
        const float oo[3] = {o.x, o.y, o.z}, dd[3] = {d.x, d.y, d.z};
        for (int a = 0; a < 3; a++) {
            if (dd[a] == 0.0f) {
                if (oo[a] < O.f[a] || oo[a] > O.f[3 + a]) return 0.0f;
                continue;
            }
            const float inv = 1.0f / dd[a];
            const float t0 = (O.f[a] - oo[a]) * inv, t1 = (O.f[3 + a] - oo[a]) * inv;
            imin = fmaxf(imin, fminf(t0, t1));
            imax = fminf(imax, fmaxf(t0, t1));
            if (imin >= imax) return 0.0f;
        }
        entry = imin;
        exit = imax;
    } else {
        if (d.x == 0.0f && d.y == 0.0f && d.z == 0.0f) return 0.0f;
        const F3 oc = o - f3(O.f);
        const float b = dot(oc, d);
        const F3 f = oc - b * d;
        const float disc = (O.f[3] * O.f[3]) - len2(f);
        if (disc < 0.0f) return 0.0f;
        const float sq = sqrtf(disc);
        entry = fminf(-b - sq, -b + sq);
        exit = fmaxf(-b - sq, -b + sq);
    }
    entry = fmaxf(fmaxf(entry, tmin), 0.0f);
    exit = fminf(exit, tmax);
    if (!(exit > entry)) return 0.0f;
    return (exit - entry) * sqrtf(len2(d));
}

template <class VS>
__device__ bool volume_distance(const GObject& O, const TRay& r, float tmin, float tmax, VS& vs, float& t)
{
    float entry, exit;
    if (O.aux == 3 /* LUZ_OBJ_CUBE */) {
        float imin = -kInf, imax = kInf;
        const float o[3] = {r.o.x, r.o.y, r.o.z};
        const float d[3] = {r.d.x, r.d.y, r.d.z};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (d[a] == 0.0f) {
                if (o[a] < O.f[a] || o[a] > O.f[3 + a]) return false;
                continue;
            }
            const float inv = 1.0f / d[a];
            float t0 = (O.f[a] - o[a]) * inv;
            float t1 = (O.f[3 + a] - o[a]) * inv;
            if (t0 > t1) {
                const float s = t0;
                t0 = t1;
                t1 = s;
            }
            imin = fmaxf(imin, t0);
            imax = fminf(imax, t1);
            if (imin >= imax) return false;
        }
        entry = imin;
        exit = imax;
    } else {
        if (r.zero) return false;
        const F3 oc = r.o - f3(O.f);
        const float b = dot(oc, r.d);
        const F3 f = oc - b * r.d;
        const float disc = (O.f[3] * O.f[3]) - len2(f);
        if (disc < 0.0f) return false;
        const float sq = sqrtf(disc);
        float r0 = -b - sq, r1 = -b + sq;
        if (r0 > r1) {
            const float s = r0;
            r0 = r1;
            r1 = s;
        }
        if (r0 >= r1) return false;
        entry = r0;
        exit = r1;
    }
    if (entry < tmin) entry = tmin;
    if (exit > tmax) exit = tmax;
    if (entry >= exit) return false;
    if (entry < 0.0f) entry = 0.0f;
    const float len = sqrtf(len2(r.d));
    if (len <= 0.0f || !isfinite(len)) return false;
    const float inside = (exit - entry) * len;
    const float hd = (float)((double)O.f[6] * log(fmax(vs.get(), 1e-12)));
    if (hd > inside) return false;
    t = entry + hd / len;
    return true;
}

// One object's closest hit; updates closest/hit when it wins.
template <uint32_t F, class Stk>
__device__ __forceinline__ void object_closest(const DScene& S, int32_t oi, const TRay& r, float tmin, float& closest,
                                               THit& h, VolSample& vs, Stk& st)
{
    const GObject O = S.objects[oi];
    const bool src = oi == r.xobj;
    float t;
    switch (O.kind) {
    case OK_RECT:
        if (!src && rect_test(S.rects[O.aux], r, tmin, closest, t)) {
            closest = t;
            h = THit{t, oi, 0, 0.f, 0.f};
        }
        break;
    case OK_CUBE:
        for (int f = 0; f < 6; f++)
            if (!(src && f == r.xprim) && rect_test(S.rects[O.aux + f], r, tmin, closest, t)) {
                closest = t;
                h = THit{t, oi, f, 0.f, 0.f};
            }
        break;
    case OK_SPHERE:
        if (sphere_test(O, r, tmin, closest, t, src)) {
            closest = t;
            h = THit{t, oi, 0, 0.f, 0.f};
        }
        break;
    case OK_PLANE:
        if (!src && plane_test(O, r, tmin, closest, t)) {
            closest = t;
            h = THit{t, oi, 0, 0.f, 0.f};
        }
        break;
    case OK_MESH: {
        int32_t slot;
        float u, v;
        if (mesh_closest<F>(S, S.meshes[O.aux], r, tmin, closest, slot, u, v, src ? r.xprim : -1, st))
            h = THit{closest, oi, slot, u, v};
        break;
    }
    case OK_INSTANCE: {
        if constexpr (!(F & TF_INSTANCE)) break;
        TRay lr;
        float s;
        if (!local_ray(O, r, lr, s)) break;
        float lc = closest * s;
        int32_t slot;
        float u, v;
        if (!mesh_closest<F>(S, S.meshes[O.aux], lr, tmin * s, lc, slot, u, v, src ? r.xprim : -1, st)) break;
        const float wt = lc / s;
        if (!isfinite(wt) || wt < tmin || wt > closest) break;
        closest = wt;
        h = THit{wt, oi, slot, u, v};
        break;
    }
    case OK_VOLUME:
        if constexpr (!(F & TF_VOLUME)) break;
        if (volume_distance(O, r, tmin, closest, vs, t)) {
            closest = t;
            h = THit{t, oi, 0, 0.f, 0.f};
        }
        break;
    default:
        break;
    }
}

// Top-level stack entries: ref | kind << 30; kind 0 = node (near check),
// 1 = node (own box test), 2 = object (near check), 3 = object (no check).
#define TOP_PUSH(ref_, kind_, near_)                       \
    do {                                                   \
        if (sp >= S.top_stack_limit) {                     \
            atomicOr(S.error, ERR_TOP_STACK);              \
            sp = 0;                                        \
            break;                                         \
        }                                                  \
        sref[sp] = (uint32_t)(ref_) | ((uint32_t)(kind_) << 30); \
        snear[sp] = (near_);                               \
        sp++;                                              \
    } while (0)

// Renderer::internal::_checkHits with explicit [tmin, tmax].
template <uint32_t F, class Stk>
__device__ __forceinline__ THit closest_hit(const DScene& S, const TRay& r, float tmin, float tmax, VolSample& vs, Stk& st)
{
    THit h{kInf, -1, 0, 0.f, 0.f};
    float closest = tmax;
    if (S.k.accel_kind == 2) {
        object_closest<F>(S, S.k.accel_object, r, tmin, closest, h, vs, st);
    } else if (S.k.accel_kind == 1) {
        uint32_t sref[kTopStack];
        float snear[kTopStack];
        int sp = 0;
        TOP_PUSH(0, 1, -kInf);
        while (sp > 0) {
            sp--;
            const uint32_t e = sref[sp];
            const float near = snear[sp];
            const uint32_t kind = e >> 30;
            const int32_t idx = (int32_t)(e & 0x3fffffffu);
            if (kind >= 2) {
                if (kind == 2 && near >= closest) continue;
                object_closest<F>(S, idx, r, tmin, closest, h, vs, st);
                continue;
            }
            const GTopNode N = S.top_nodes[idx];
            float dummy;
            if (kind == 1) {
                if (!box_hit(N.bmin, N.bmax, r, closest, dummy)) continue;
            } else if (near >= closest) {
                continue;
            }
            const int n = N.child_count;
            const GTopChild* C = S.top_children + N.child_start;
            if (n != 2 && n <= 3) {
                for (int i = n - 1; i >= 0; i--) {
                    if (C[i].is_node) TOP_PUSH(C[i].ref, 1, -kInf);
                    else TOP_PUSH(C[i].ref, 3, -kInf);
                }
            } else if (n == 2) {
                float na = 0.f, nb = 0.f;
                const bool ha = box_hit(C[0].bmin, C[0].bmax, r, closest, na);
                const bool hb = box_hit(C[1].bmin, C[1].bmax, r, closest, nb);
                int first = 0, second = 1;
                bool hf = ha, hs = hb;
                float nf = na, ns = nb;
                if (ha && hb && nb < na) {
                    first = 1;
                    second = 0;
                    hf = hb;
                    hs = ha;
                    nf = nb;
                    ns = na;
                }
                if (hs) TOP_PUSH(C[second].ref, C[second].is_node ? 0 : 2, ns);
                if (hf) TOP_PUSH(C[first].ref, C[first].is_node ? 0 : 2, nf);
            } else {
                int ord[16];
                float on[16];
                int cnt = 0;
                for (int i = 0; i < n && i < 16; i++) {
                    float cn;
                    if (!box_hit(C[i].bmin, C[i].bmax, r, closest, cn)) continue;
                    int j = cnt;
                    while (j > 0 && on[j - 1] > cn) {
                        on[j] = on[j - 1];
                        ord[j] = ord[j - 1];
                        j--;
                    }
                    on[j] = cn;
                    ord[j] = i;
                    cnt++;
                }
                for (int j = cnt - 1; j >= 0; j--) {
                    const GTopChild& c = C[ord[j]];
                    TOP_PUSH(c.ref, c.is_node ? 0 : 2, on[j]);
                }
            }
        }
    }
    for (int i = 0; i < S.k.unaccel_count; i++)
        object_closest<F>(S, S.index_pool[S.k.unaccel_offset + i], r, tmin, closest, h, vs, st);
    return h;
}

}  // namespace luz
