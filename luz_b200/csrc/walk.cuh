// walk.cuh — the traversal of the trace kernels: one ray per lane, the 32 lanes of a warp
// in step.
//
// A ray's walk of the two-level scene (trace.cuh gives its semantics and its order) is a
// state machine of four kinds of step: a collapsed mesh node, the triangles of a leaf, a
// top-level node, an object. One stack holds the entries of both levels: those of the mesh
// being walked lie above `base`, the top level's below it, so a lane whose mesh walk ends
// goes on with its top-level entries while its neighbours are still inside a mesh. walk()
// runs one kind of step at a time for all lanes that wait at that kind, chosen by warp
// votes, and brings the warp together after each step.
//
// What bounds it: SIMT divergence and the instructions of a step (two thirds of the issue
// slots are used), then the latency of a step's loads. Written as nested per-thread loops
// (mesh walk inside object inside top-level node) the lanes of a warp part at their first
// divergent branch and are not brought together again before the loop ends: 8 active lanes
// per instruction on the 1080p glossy frame against 17-23 here, its extension stage 126.0 ->
// 82.2 ms and its shadow stage 68.9 -> 46.7 ms at 64 spp, with the shared launch and the
// collapsed nodes of one cache line.
#pragma once
#include "trace.cuh"

namespace luz {

enum WalkState : uint32_t { WS_NODE = 0, WS_LEAF = 1, WS_TOP = 2, WS_OBJECT = 3, WS_DONE = 4 };

constexpr int kWalkBlock = 128;                         // threads per block of the walking kernels
constexpr int kWalkStack = kMeshStack4 + kTopStack;     // entries of both levels

// The world rays of the lanes inside an instance, while they walk with its local ray.
struct WorldRays {
    float v[9][kWalkBlock];
};

// F: TF_* bits; ANY: any hit (an occlusion test) instead of the closest one; COUNT: counts
// the records read (mesh nodes, triangles, top-level records, and the binary-node visits
// that the collapsed nodes stand for); VS: the volume sample's source.
template <uint32_t F, bool ANY, bool COUNT, class VS>
struct Walk {
    TRay r;              // the ray of the current step: the world's, or an instance's local one
    float tmin;          // of r
    float closest;       // the closest hit along r so far (ANY: the ray's end)
    THit h;              // the world's hit; ANY: obj >= 0 when occluded
    uint32_t state, ref; // ref: mesh node or leaf (NODE, LEAF); stack reference with its kind (TOP, OBJECT)
    int sp, base;        // stack entries; those of the mesh being walked start at base
    int next_unaccel;    // next entry of the unaccelerated object list
    int32_t obj, skip;   // object whose mesh is walked; triangle the ray leaves from
    bool fast;           // mesh_fast_slabs of that mesh and r
    bool inside;         // inside an instance
    float scale, world_closest, world_tmin, lu, lv;
    int32_t lslot;       // closest local triangle, -1 = none
    uint32_t n_nodes, n_tris, n_top, n_bnodes;
    uint2* st;           // kWalkStack entries: reference, near distance (bits)

    __device__ __forceinline__ float tnear(uint2 e) const { return __uint_as_float(e.y); }

    __device__ __forceinline__ void start(const DScene& S, const TRay& ray, float t0, float t1)
    {
        r = ray;
        tmin = t0;
        closest = t1;
        h = THit{kInf, -1, 0, 0.f, 0.f};
        sp = base = 0;
        next_unaccel = 0;
        inside = false;
        if constexpr (COUNT) n_nodes = n_tris = n_top = n_bnodes = 0;
        if (ANY && t1 <= kTMin) {
            state = WS_DONE;
        } else if (S.k.accel_kind == 2) {
            ref = (uint32_t)S.k.accel_object | (3u << 30);
            state = WS_OBJECT;
        } else if (S.k.accel_kind == 1) {
            ref = 1u << 30;
            state = WS_TOP;
        } else {
            pop_top(S);
        }
    }

    // Top-level references: ref | kind << 30; kind 0 = node (near distance checked when
    // reached), 1 = node (own box test), 2 = object (near distance checked), 3 = object.
    __device__ __forceinline__ void go_top(uint32_t e)
    {
        ref = e;
        state = (e >> 31) ? WS_OBJECT : WS_TOP;
    }
    __device__ __forceinline__ void pop_top(const DScene& S)
    {
        while (sp > 0) {
            sp--;
            const uint2 e = st[sp];
            if (!ANY && !((e.x >> 30) & 1u) && tnear(e) >= closest) continue;
            go_top(e.x);
            return;
        }
        if (next_unaccel < S.k.unaccel_count) {
            ref = (uint32_t)S.index_pool[S.k.unaccel_offset + next_unaccel] | (3u << 30);
            next_unaccel++;
            state = WS_OBJECT;
        } else {
            state = WS_DONE;
        }
    }
    __device__ __forceinline__ void push_top(uint32_t e, float near)
    {
        st[sp] = make_uint2(e, __float_as_uint(near));
        sp++;
    }
    // True (and the walk at its end, the error set) when n more entries overflow the top-level stack.
    __device__ __forceinline__ bool top_full(const DScene& S, int n)
    {
        if (sp + n <= S.top_stack_limit) return false;
        atomicOr(S.error, ERR_TOP_STACK);
        sp = 0;
        state = WS_DONE;
        return true;
    }

    __device__ __forceinline__ void go_mesh(uint32_t e)
    {
        ref = e;
        state = (e & kLeafBit) ? WS_LEAF : WS_NODE;
    }
    __device__ __forceinline__ void pop_mesh(const DScene& S, WorldRays* W)
    {
        while (sp > base) {
            sp--;
            const uint2 e = st[sp];
            if (!ANY && tnear(e) >= closest) continue;
            go_mesh(e.x);
            return;
        }
        leave_mesh(S, W);
    }
    // The mesh of `obj` is walked: back to the world ray when it was an instance's, and on.
    __device__ __forceinline__ void leave_mesh(const DScene& S, WorldRays* W)
    {
        if constexpr ((F & TF_INSTANCE) != 0) {
            if (inside) {
                inside = false;
                const int t = (int)threadIdx.x;
                r.o = F3{W->v[0][t], W->v[1][t], W->v[2][t]};
                r.d = F3{W->v[3][t], W->v[4][t], W->v[5][t]};
                r.inv = F3{W->v[6][t], W->v[7][t], W->v[8][t]};
                r.zero = (r.d.x == 0.0f && r.d.y == 0.0f && r.d.z == 0.0f);
                r.axis0 = r.inv.x == 0.0f || r.inv.y == 0.0f || r.inv.z == 0.0f;
                const float lc = closest;
                closest = world_closest;
                tmin = world_tmin;
                if (!ANY && lslot >= 0) {
                    const float wt = lc / scale;
                    if (isfinite(wt) && !(wt < tmin) && !(wt > closest)) {
                        closest = wt;
                        h = THit{wt, obj, lslot, lu, lv};
                    }
                }
            }
        }
        pop_top(S);
    }

    // Starts the walk of a mesh with the current ray (an instance's local one when inside).
    __device__ __forceinline__ void enter_mesh(const DScene& S, const GMesh& M, WorldRays* W)
    {
        base = sp;
        fast = mesh_fast_slabs(M, r);
        float near;
        const bool in = fast ? box_hit_fast(M.bmin, M.bmax, r, neg_o_inv(r), closest, near)
                             : box_hit(M.bmin, M.bmax, r, closest, near);
        if (in && (ANY || !(near >= closest))) go_mesh((uint32_t)M.root4_ref);
        else leave_mesh(S, W);
    }

    __device__ __forceinline__ void node_step(const DScene& S, WorldRays* W)
    {
        Node4Test T;
        if (fast) node4_test<true, F, !ANY, COUNT && !ANY>(S, ref, r, closest, T);
        else node4_test<false, F, !ANY, COUNT && !ANY>(S, ref, r, closest, T);
        if constexpr (COUNT) {
            // binary-node visits this node stands for: N itself, and each side that is an
            // interior node of the binary tree (two entries) and that the walk enters
            n_nodes++;
            if (ANY)
                n_bnodes += 1u + (uint32_t)(T.ref[1] != kEmptySlot && (T.ha[0] || T.ha[1]))
                            + (uint32_t)(T.ref[3] != kEmptySlot && (T.ha[2] || T.ha[3]));
            else
                n_bnodes += 1u + (uint32_t)(T.hl && T.ref[1] != kEmptySlot) + (uint32_t)(T.hr && T.ref[3] != kEmptySlot);
        }
        const int ne = (int)T.ha[0] + (int)T.ha[1] + (int)T.ha[2] + (int)T.ha[3];
        if (sp - base + ne > S.mesh_stack_limit) {
            atomicOr(S.error, ERR_MESH_STACK);
            sp = base;
            leave_mesh(S, W);
            return;
        }
        if (ne == 0) {
            pop_mesh(S, W);
            return;
        }
        if constexpr (ANY) {
            // Any accepted entry may hold an occluder and the first one found ends the walk,
            // so the entries are taken in slot order; the answer does not depend on it.
            uint32_t first = 0;
            bool have = false;
#pragma unroll
            for (int k = 3; k >= 0; k--)
                if (T.ha[k]) {
                    if (have) st[sp++].x = first;
                    first = T.ref[k];
                    have = true;
                }
            go_mesh(first);
        } else {
            Node4Order o;
            node4_order(T, o);
#pragma unroll
            for (int k = 3; k > 0; k--)
                if (o.on[k]) st[sp++] = make_uint2(o.ref[k], __float_as_uint(o.near[k]));
            go_mesh(o.ref[0]);
        }
    }

    __device__ __forceinline__ void leaf_step(const DScene& S, WorldRays* W)
    {
        const uint32_t first = (ref & 0x7fffffffu) >> 3, end = first + (ref & 7u) + 1u;
        for (uint32_t i = first; i < end; i++) {
            if ((int32_t)i == skip) continue;
            const GTri T = load_tri(S.tris, i);
            if constexpr (COUNT) n_tris++;
            float t, u, v;
            if (!tri_test(T, r, tmin, closest, t, u, v)) continue;
            if constexpr (ANY) {
                h.obj = obj;
                break;
            } else {
                accept(t, (int32_t)i, u, v);
            }
        }
        if (ANY && h.obj >= 0) state = WS_DONE;
        else pop_mesh(S, W);
    }

    // leaf_step of the lanes in `owners`, eight lanes to a leaf (a leaf holds at most eight
    // triangles): every lane of the warp calls it. A leaf's triangles are tested side by
    // side against the owner's interval; the nearest wins, at equal distances the last in
    // leaf order, which is what testing them one after another comes to.
    // SCENES: the lanes' scenes may differ.
    template <bool SCENES>
    __device__ __forceinline__ void leaf_step_grouped(const DScene& S, unsigned owners, WorldRays* W)
    {
        constexpr unsigned full = 0xffffffffu;
        const int lane = (int)(threadIdx.x & 31u), j = lane & 7, g = lane >> 3;
        const bool owner = (owners >> lane) & 1u;
        const int rank = __popc(owners & ((1u << lane) - 1u));   // of an owner: its round and group
        bool again = false;
        int r0 = 0;
        for (unsigned left = owners; left; r0 += 4) {
            int src = -1;   // owner of this lane's group in this round
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (g == k) src = __ffs(left) - 1;
                left &= left - 1u;
            }
            const bool has = src >= 0;
            src = has ? src : lane;
            const uint32_t oref = __shfl_sync(full, ref, src);
            TRay q;
            q.o = F3{__shfl_sync(full, r.o.x, src), __shfl_sync(full, r.o.y, src), __shfl_sync(full, r.o.z, src)};
            q.d = F3{__shfl_sync(full, r.d.x, src), __shfl_sync(full, r.d.y, src), __shfl_sync(full, r.d.z, src)};
            const float t0 = __shfl_sync(full, tmin, src), t1 = __shfl_sync(full, closest, src);
            const int32_t sk = __shfl_sync(full, skip, src);
            const GTri* tris = S.tris;
            if constexpr (SCENES)
                tris = reinterpret_cast<const GTri*>(__shfl_sync(full, reinterpret_cast<unsigned long long>(tris), src));
            const uint32_t i = ((oref & 0x7fffffffu) >> 3) + (uint32_t)j;
            float t = kInf, u = 0.f, v = 0.f;
            bool ok = false;
            if (has && (uint32_t)j <= (oref & 7u) && (int32_t)i != sk) {
                const GTri T = load_tri(tris, i);
                ok = tri_test(T, q, t0, t1, t, u, v);
            }
            const bool mine = owner && (rank >> 2) == (r0 >> 2);
            const int gl = 8 * (rank & 3);
            const unsigned hits = __ballot_sync(full, ok);
            if constexpr (COUNT)
                if (mine) {   // as one after another: ANY ends at the first hit; the skipped triangle is not read
                    const unsigned h8 = (hits >> gl) & 0xffu;
                    const uint32_t last = ANY && h8 ? (uint32_t)__ffs(h8) - 1u : ref & 7u;
                    n_tris += last + 1u - (uint32_t)((uint32_t)(skip - (int32_t)((ref & 0x7fffffffu) >> 3)) <= last);
                }
            if constexpr (ANY) {
                if (mine && ((hits >> gl) & 0xffu)) h.obj = obj;
            } else {
                if (!hits) continue;
                const unsigned odd = __ballot_sync(full, ok && !(t < kInf));   // not a distance: one after another
                if (!ok) t = kInf;
                int best = lane;
#pragma unroll
                for (int off = 4; off > 0; off >>= 1) {
                    const float t2 = __shfl_xor_sync(full, t, off);
                    const int b2 = __shfl_xor_sync(full, best, off);
                    if (t2 < t || (t2 == t && b2 > best)) {
                        t = t2;
                        best = b2;
                    }
                }
                const float rt = __shfl_sync(full, t, gl);
                const int rb = __shfl_sync(full, best, gl);
                const float ru = __shfl_sync(full, u, rb), rv = __shfl_sync(full, v, rb);
                if (mine && ((hits >> gl) & 0xffu)) {
                    if ((odd >> gl) & 0xffu) again = true;
                    else accept(rt, (int32_t)((ref & 0x7fffffffu) >> 3) + (rb & 7), ru, rv);
                }
            }
        }
        if (owner) {
            if (again) leaf_step(S, W);
            else if (ANY && h.obj >= 0) state = WS_DONE;
            else pop_mesh(S, W);
        }
    }
    __device__ __forceinline__ void accept(float t, int32_t i, float u, float v)
    {
        closest = t;
        if ((F & TF_INSTANCE) && inside) {
            lslot = i;
            lu = u;
            lv = v;
        } else {
            h = THit{t, obj, i, u, v};
        }
    }

    __device__ __forceinline__ void top_step(const DScene& S)
    {
        const GTopNode N = S.top_nodes[ref & 0x3fffffffu];
        const int n = N.child_count;
        if constexpr (COUNT) n_top += 1u + (uint32_t)n;
        float near;
        if ((ref >> 30) == 1u && !box_hit(N.bmin, N.bmax, r, closest, near)) {
            pop_top(S);
            return;
        }
        const GTopChild* C = S.top_children + N.child_start;
        if (n != 2 && n <= 3) {   // index order, each child does its own test
            if (n == 0) {
                pop_top(S);
                return;
            }
            if (top_full(S, n)) return;
            for (int i = n - 1; i > 0; i--)
                push_top((uint32_t)C[i].ref | (C[i].is_node ? 1u : 3u) << 30, -kInf);
            go_top((uint32_t)C[0].ref | (C[0].is_node ? 1u : 3u) << 30);
        } else if (ANY) {   // accepted children in index order
            uint32_t first = 0;
            bool have = false;
            for (int i = n - 1; i >= 0; i--) {
                if (!box_hit(C[i].bmin, C[i].bmax, r, closest, near)) continue;
                if (top_full(S, have ? 2 : 1)) return;
                if (have) push_top(first, 0.f);
                first = (uint32_t)C[i].ref | (C[i].is_node ? 0u : 3u) << 30;
                have = true;
            }
            if (have) go_top(first);
            else pop_top(S);
        } else if (n == 2) {   // nearer child first, swapped only when strictly nearer
            float na = 0.f, nb = 0.f;
            const bool ha = box_hit(C[0].bmin, C[0].bmax, r, closest, na);
            const bool hb = box_hit(C[1].bmin, C[1].bmax, r, closest, nb);
            const uint32_t ea = (uint32_t)C[0].ref | (C[0].is_node ? 0u : 2u) << 30;
            const uint32_t eb = (uint32_t)C[1].ref | (C[1].is_node ? 0u : 2u) << 30;
            if (!ha && !hb) {
                pop_top(S);
                return;
            }
            if (top_full(S, (int)ha + (int)hb)) return;
            const bool b_first = hb && !(ha && !(nb < na));
            if (ha && hb) push_top(b_first ? ea : eb, b_first ? na : nb);
            go_top(b_first ? eb : ea);
        } else {
            // four and more: by entry distance, ties in index order. The accepted children are
            // inserted into the stack itself, the nearest on top.
            int cnt = 0;
            for (int i = 0; i < n && i < 16; i++) {
                if (!box_hit(C[i].bmin, C[i].bmax, r, closest, near)) continue;
                if (top_full(S, cnt + 1)) return;
                const uint32_t e = (uint32_t)C[i].ref | (C[i].is_node ? 0u : 2u) << 30;
                int j = sp + cnt;
                while (j > sp) {
                    const uint2 q = st[j - 1];
                    if (tnear(q) > near) break;
                    st[j] = q;
                    j--;
                }
                st[j] = make_uint2(e, __float_as_uint(near));
                cnt++;
            }
            if (cnt == 0) {
                pop_top(S);
                return;
            }
            sp += cnt - 1;
            go_top(st[sp].x);
        }
    }

    __device__ __forceinline__ void hit_object(float t, int32_t oi, int32_t prim)
    {
        if constexpr (ANY) {
            h.obj = oi;
        } else {
            closest = t;
            h = THit{t, oi, prim, 0.f, 0.f};
        }
    }

    __device__ __forceinline__ void object_step(const DScene& S, WorldRays* W, VS& vs)
    {
        const int32_t oi = (int32_t)(ref & 0x3fffffffu);
        const GObject& O = S.objects[oi];
        if constexpr (COUNT) n_top++;
        const bool src = oi == r.xobj;
        float t;
        obj = oi;
        switch (O.kind) {
        case OK_RECT:
            if (!src && rect_test(S.rects[O.aux], r, tmin, closest, t)) hit_object(t, oi, 0);
            break;
        case OK_CUBE:
            for (int f = 0; f < 6; f++)
                if (!(src && f == r.xprim) && rect_test(S.rects[O.aux + f], r, tmin, closest, t)) {
                    hit_object(t, oi, f);
                    if (ANY) break;
                }
            break;
        case OK_SPHERE:
            if (sphere_test(O, r, tmin, closest, t, src)) hit_object(t, oi, 0);
            break;
        case OK_PLANE:
            if (!src && plane_test(O, r, tmin, closest, t)) hit_object(t, oi, 0);
            break;
        case OK_MESH:
            skip = src ? r.xprim : -1;
            enter_mesh(S, S.meshes[O.aux], W);
            return;
        case OK_INSTANCE:
            if constexpr ((F & TF_INSTANCE) != 0) {
                TRay lr;
                float s;
                if (!local_ray(O, r, lr, s)) break;
                const int i = (int)threadIdx.x;
                W->v[0][i] = r.o.x;
                W->v[1][i] = r.o.y;
                W->v[2][i] = r.o.z;
                W->v[3][i] = r.d.x;
                W->v[4][i] = r.d.y;
                W->v[5][i] = r.d.z;
                W->v[6][i] = r.inv.x;
                W->v[7][i] = r.inv.y;
                W->v[8][i] = r.inv.z;
                world_closest = closest;
                world_tmin = tmin;
                scale = s;
                closest = closest * s;
                tmin = tmin * s;
                r = lr;
                inside = true;
                lslot = -1;
                skip = src ? r.xprim : -1;
                enter_mesh(S, S.meshes[O.aux], W);
                return;
            }
            break;
        case OK_VOLUME:
            if constexpr ((F & TF_VOLUME) != 0)
                if (volume_distance(O, r, tmin, closest, vs, t)) hit_object(t, oi, 0);
            break;
        default:
            break;
        }
        if (ANY && h.obj >= 0) state = WS_DONE;
        else pop_top(S);
    }
};

// Up to this many lanes at leaves are tested in groups (leaf_step_grouped: a round of four
// leaves costs about as much as one and a half triangles tested by all lanes); above it each
// lane tests its own leaf's triangles one after another. 1080p glossy frame at 64 spp, in
// groups up to 0, 8, 16, 32 lanes: 241.4, 225.2, 223.5, 232.4 ms; draft 3.25, 2.83, 2.81, 2.84;
// with instances one kind alone is better than both: Cornell box 7.33, 7.68, 7.51, 7.20 ms.
#ifndef LUZ_LEAF_GROUP_MAX
#define LUZ_LEAF_GROUP_MAX 16
#endif
#ifndef LUZ_LEAF_GROUP_MAX_INST
#define LUZ_LEAF_GROUP_MAX_INST 32
#endif
template <uint32_t F>
constexpr int kLeafGroupMax = (F & TF_INSTANCE) ? LUZ_LEAF_GROUP_MAX_INST : LUZ_LEAF_GROUP_MAX;

// Runs the walks of a warp's lanes to their ends; every lane of the warp calls it (a lane
// without a ray with its state at WS_DONE). Node steps run while at least half of the live
// lanes wait at one; then each other kind that some lane waits at runs once. With instances
// the lanes spread over leaves, top-level nodes and objects, and only the kind that most of
// them wait at runs (leaves before top-level nodes before objects at equal numbers): 1e5
// instances at 8 spp 198.4 -> 185.5 ms, the Cornell box 4.98 -> 4.91 ms (spheres without
// instances 1.38 -> 1.42 ms, so not there). SCENES: the lanes' scenes may differ.
template <bool SCENES, uint32_t F, bool ANY, bool COUNT, class VS>
__device__ __forceinline__ void walk_warp(const DScene& S, Walk<F, ANY, COUNT, VS>& w, WorldRays* wr, VS& vs)
{
    constexpr unsigned full = 0xffffffffu;
    while (true) {
        const int live = __popc(__ballot_sync(full, w.state != WS_DONE));
        if (live == 0) break;
        const int enough = (live + 1) >> 1;
        while (__popc(__ballot_sync(full, w.state == WS_NODE)) >= enough) {
            if (w.state == WS_NODE) w.node_step(S, wr);
            __syncwarp();
        }
        const unsigned leaves = __ballot_sync(full, w.state == WS_LEAF);
        const unsigned objects = __ballot_sync(full, w.state == WS_OBJECT);
        bool do_leaf = leaves != 0, do_object = objects != 0, do_top = true;
        if constexpr ((F & TF_INSTANCE) != 0) {
            const int n_leaf = __popc(leaves), n_object = __popc(objects),
                      n_top = __popc(__ballot_sync(full, w.state == WS_TOP));
            do_leaf = n_leaf > 0 && n_leaf >= max(n_top, n_object);
            do_top = !do_leaf && n_top > 0 && n_top >= n_object;
            do_object = !do_leaf && !do_top;
        }
        if (do_leaf) {
            if (__popc(leaves) > kLeafGroupMax<F>) {
                if (w.state == WS_LEAF) w.leaf_step(S, wr);
            } else {
                w.template leaf_step_grouped<SCENES>(S, leaves, wr);
            }
            __syncwarp();
        }
        if (do_object) {
            if (w.state == WS_OBJECT) w.object_step(S, wr, vs);
            __syncwarp();
        }
        if (do_top) {
            if (w.state == WS_TOP) w.top_step(S);
            __syncwarp();
        }
    }
}

}  // namespace luz
