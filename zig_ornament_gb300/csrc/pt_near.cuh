// pt_near.cuh — closest-hit traversal nearest child first, with the
// reference's results.
//
// The reference walks its tree right child first, whatever the ray's
// direction (bvh.hip.h:145-276), over splits at medians of random axes.  Its
// result, though, is a function of the ray and the primitives alone, but for
// rounding: among the primitives whose own test accepts the ray, and whose
// own and ancestors' boxes the ray hits, the one with the smallest t.  This
// traversal finds that primitive in other trees over the same primitives
// (tree_build.cu: fewer visits), nearest box first (fewer still), and shows
// from the candidates it saw that the reference's walk ends with the same
// one.  Where it cannot show it, the ray is walked again the reference's way
// (`redo`).
//
// Why the results agree.  Let t(P) be the parameter that the reference's
// test computes for primitive P (it does not depend on the t_max of the
// moment), and let "P's own boxes" be the leaf's box in its BLAS and the
// shape's box in the TLAS.  All boxes are tested with the reference's
// arithmetic (aabb_hit_fast).  Every stored box holds the boxes below it
// (checked when the trees are built) and float multiplication, addition, min
// and max are monotonic, so an ancestor's computed interval holds P's own, in
// the reference's tree as in these: a ray that passes P's own boxes with
// t_max = infinity passes all ancestors' too.  Let B be the best candidate
// (smallest t among those that pass), and T = max(t(B), entry of B's own
// boxes).  If every other candidate has t > T, the reference's t_max is above
// T whenever it tests one of B's boxes or B itself, so B is reached and
// accepted, and nothing replaces it.  A second candidate within T (a tie, or
// two surfaces within a rounding step) sets `unsure`.
//
// What is pruned.  A box entered beyond `lim` is skipped: T, plus what the
// computed t of a primitive in there can lie in front of the computed entry of
// its boxes.  That is, in units of t,
//   * rounding of the slab test: 2^-23 of the origin's and the box's
//     coordinates in the space of the test, times 1/d of the axis, for each of
//     the two boxes compared.  A ray that runs along a box's face (|d| down to
//     safe_invdir's 1e-5) and a mesh far from its own origin (survey data, that
//     its transform brings back) make it large: the margin of a mesh is taken
//     from the ray's origin in its space (near_move), the TLAS's from the ray's
//     own (walker_begin, near_turn).
//   * rounding of the shape's transform, which moves the hit against the box of
//     the shape in the TLAS: near_turn and near_reach (tree_build.cu,
//     shapes_kernel; also a box that is not quite around its shape).
//   * rounding of the primitive's own test, across the ray (triangle_pad, in the
//     place of a mesh leaf's type; near_reach) and along it (kNearSlide times
//     that; kNearMargin of t).  Triangles whose shape alone can magnify rounding
//     a thousandfold (edges parallel to one part in 2^10) are given their whole
//     tree's box by the builder.
// With a margin of 2^-10 of the world origin's coordinates alone, 215 of 1.6 M
// rays at instances of a mesh modelled 10^6 from its origin missed what the
// reference hits, and 41 of 0.7 M from the sphere field's surfaces with epsilon
// zero; the margins cost 1 to 2 % of a frame (1080p scene 314 -> 320 ms).
//
// What is left: a ray in a triangle's plane, to within rounding, is given a t by
// Möller and Trumbore's test that is rounding alone, anywhere along the ray, and
// the reference's result is then a matter of whether it came to that triangle
// before the true hit.  (0 of 10^8 rays in random directions and off surfaces; of
// rays aimed along the planes of triangles in a random soup, 6 in 10^4.)
#pragma once

#include "pt_device.cuh"
#include "pt_kernels.h"

namespace orn {

constexpr float kNearMargin = 0.0625f;   // pruning margin relative to t
constexpr uint32_t kNearNone = 0xffffffffu;   // no shape
constexpr uint32_t kNearLeave = 0xffffffffu;  // NearWalker::node: nothing is left in this space

// Traversal state of one ray.
struct NearWalker {
    uint32_t node;             // next node (typed reference), or kNearLeave
    float near;                // entry of its box
    int sp, floor;             // entries on the stack; those that are not of this space
    f3 o, d, inv, oxinv;       // (of the TLAS only while inner nodes of it are visited)
    float t, tie;              // best hit; T of the comment above
    float lim;                 // boxes entered beyond are skipped
    float margin, tlas_margin; // the share of it that does not grow with t: in this space, and in the TLAS
    uint32_t shape;            // current shape's node; kNearNone in the TLAS
    float entry;               // entry of its box
    uint32_t hit_shape, hit_tri;
    float u, v;
    bool unsure;               // the candidates seen do not settle the reference's result
    bool redo;                 // walking the reference's tree in its order
    bool away;                 // back in the TLAS with the space of a mesh
};

// The stack of nodes to visit, each with the entry of its box: the first SS / 2
// in shared memory (as TravStack, 8 bytes an access), the rest in local memory.
template <int SS>
struct NearStack {
    static_assert(SS % 2 == 0 && SS / 2 < kNearStackSize, "near stack");
    uint2* sstack;
    int sstride;
    uint2 lstack[kNearStackSize - SS / 2];
    // `base` (8-byte aligned): SS * stride words that `stride` threads share
    __device__ __forceinline__ void init(uint32_t* base, uint32_t thread, int stride) {
        sstack = reinterpret_cast<uint2*>(base) + thread;
        sstride = stride;
    }
    __device__ __forceinline__ void put(int i, uint32_t node, float near) {
        const uint2 v = make_uint2(node, __float_as_uint(near));
        if (i < SS / 2) sstack[i * sstride] = v;
        else lstack[i - SS / 2] = v;
    }
    __device__ __forceinline__ uint2 get(int i) const {
        if (i < SS / 2) return sstack[i * sstride];
        return lstack[i - SS / 2];
    }
};

// Moves the ray into a space.
__device__ __forceinline__ void near_space(NearWalker& w, f3 o, f3 d) {
    w.o = o;
    w.d = d;
    w.inv = safe_invdir(d);
    w.oxinv = mul(neg(o), w.inv);
}

__device__ __forceinline__ float max_abs(f3 a) { return fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)); }

__device__ __forceinline__ float min_abs(f3 a) { return fminf(fminf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)); }

// The limit for the best hit of the moment.
__device__ __forceinline__ float near_limit(const NearWalker& w) {
    return w.tie + (w.tie * kNearMargin + w.margin);
}

__device__ __forceinline__ void near_start(NearWalker& w, uint32_t root, f3 ro, f3 rd) {
    w.node = root;
    w.near = -INFINITY;
    w.sp = w.floor = 0;
    near_space(w, ro, rd);
    w.t = w.tie = (float)3.40282e+38;
    w.lim = INFINITY;
    w.shape = kNearNone;
    w.entry = -INFINITY;
    w.hit_shape = kNearNone;
    w.unsure = w.redo = w.away = false;
}

__device__ __forceinline__ void walker_begin(NearWalker& w, const SceneDev& sc, f3 ro, f3 rd) {
    near_start(w, sc.nroot, ro, rd);
    // (in units of t)
    w.margin = w.tlas_margin = sc.near_slide * min_abs(w.inv) +
                               (max_abs(ro) * (2.0f * sc.near_turn) + sc.near_reach) * max_abs(w.inv);
}

// aabb_hit_fast that also gives the entry.
// (mul.rn.f32x2 and add.rn.f32x2 are no way to do two at a time: the compiler
// makes one fma of them, and a box that the reference misses by a rounding is
// hit.  Products alone in pairs: no gain.)
__device__ __forceinline__ bool near_box(float4 mn, float4 mx, f3 inv, f3 oxinv, float t_min, float t_max,
                                         float* entry) {
    const float fx = mx.x * inv.x + oxinv.x, fy = mx.y * inv.y + oxinv.y, fz = mx.z * inv.z + oxinv.z;
    const float nx = mn.x * inv.x + oxinv.x, ny = mn.y * inv.y + oxinv.y, nz = mn.z * inv.z + oxinv.z;
    const float out = fminf(fminf(fminf(fmaxf(fx, nx), fmaxf(fy, ny)), fmaxf(fz, nz)), t_max);
    *entry = fmaxf(fmaxf(fmaxf(fminf(fx, nx), fminf(fy, ny)), fminf(fz, nz)), t_min);
    return *entry <= out;
}

// A candidate at parameter t whose leaf's box is entered at `near`; true
// when it is the best so far.
__device__ __forceinline__ bool near_accept(NearWalker& w, float t, float near) {
    if (!(t < w.t)) {
        if (t <= w.tie) w.unsure = !w.redo;   // a tie, or a second surface within the first one's T
        return false;
    }
    const float tie = fmaxf(t, fmaxf(near, w.entry));
    w.unsure = w.t <= tie && !w.redo;
    w.t = t;
    w.tie = tie;
    // (redo: the reference's own t_max)
    w.lim = w.redo ? t : near_limit(w);
    return true;
}

// The next node of this space from the stack, or kNearLeave.
template <int SS>
__device__ __forceinline__ void near_pop(NearWalker& w, NearStack<SS>& stack) {
    for (;;) {
        if (w.sp == w.floor) {
            w.node = kNearLeave;
            return;
        }
        const uint2 top = stack.get(--w.sp);
        w.node = top.x;
        w.near = __uint_as_float(top.y);
        if (w.near <= w.lim) return;
    }
}

// Tests the two boxes of the lane's inner node and goes on with the nearer.
template <int SS>
__device__ __forceinline__ void near_inner(NearWalker& w, const SceneDev& sc, float t_min, NearStack<SS>& stack) {
    Node nd;
    nd.load(sc.nodes + 4 * (size_t)w.node);
    float nl, nr;
    const bool hl = near_box(nd.a, nd.b, w.inv, w.oxinv, t_min, w.lim, &nl);
    const bool hr = near_box(nd.c, nd.e, w.inv, w.oxinv, t_min, w.lim, &nr);
    const uint32_t lref = bits(nd.a.w), rref = bits(nd.b.w);
    const bool right = hr && (!hl || nr < nl || w.redo);
    if (hl && hr) {
        stack.put(w.sp++, right ? lref : rref, w.redo ? -INFINITY : (right ? nl : nr));
    }
    if (hl || hr) {
        w.node = right ? rref : lref;
        w.near = right ? nr : nl;
    } else {
        near_pop(w, stack);
    }
}

// Tests the lane's triangle and takes up the next node.
template <int SS>
__device__ __forceinline__ void near_triangle(NearWalker& w, const SceneDev& sc, float t_min, NearStack<SS>& stack) {
    Node nd;
    nd.load(sc.nodes + 4 * (size_t)(w.node & kRefIndexMask));
    const f3 v0 = mk(nd.a.x, nd.a.y, nd.a.z);
    float t = 0.0f, u = 0.0f, v = 0.0f;
    bool hit;
    if (sc.watertight) {
        float wt = 0.0f, wu = 0.0f, wv = 0.0f;   // (in memory: the test is out of line)
        hit = tri_watertight(w.o, w.d, v0, mk(nd.b.x, nd.b.y, nd.b.z), mk(nd.c.x, nd.c.y, nd.c.z), t_min, INFINITY, &wt,
                             &wu, &wv);
        t = wt;
        u = wu;
        v = wv;
    } else {
        hit = tri_mt_edges(w.o, w.d, v0, mk(nd.e.x, nd.e.y, nd.e.z), mk(nd.b.w, nd.c.w, nd.e.w), t_min, INFINITY, &t,
                           &u, &v);
    }
    if (hit && (bits(nd.a.w) & kNearOwnBox) != 0u) {
        const float4 lo = make_float4(fminf(fminf(v0.x, nd.b.x), nd.c.x), fminf(fminf(v0.y, nd.b.y), nd.c.y),
                                      fminf(fminf(v0.z, nd.b.z), nd.c.z), 0.0f);
        const float4 hi = make_float4(fmaxf(fmaxf(v0.x, nd.b.x), nd.c.x), fmaxf(fmaxf(v0.y, nd.b.y), nd.c.y),
                                      fmaxf(fmaxf(v0.z, nd.b.z), nd.c.z), 0.0f);
        hit = near_box(lo, hi, w.inv, w.oxinv, t_min, (float)3.40282e+38, &w.near);
    }
    if (hit && near_accept(w, t, w.near)) {
        w.hit_shape = w.shape;
        w.hit_tri = bits(nd.a.w) & ~kNearOwnBox;
        w.u = u;
        w.v = v;
    }
    near_pop(w, stack);
}

// Tests the lane's sphere, enters its mesh, or leaves the mesh it is in (and
// enters the next, where that follows at once).  False when the ray is
// finished.
template <int SS>
__device__ __forceinline__ bool near_move(NearWalker& w, const SceneDev& sc, f3 ro, f3 rd, float t_min,
                                          NearStack<SS>& stack) {
    if (w.node == kNearLeave) {
        if (w.shape != kNearNone) {
            w.shape = kNearNone;
            w.entry = -INFINITY;
            w.floor = 0;
            w.away = true;
            w.margin = w.tlas_margin;
            if (!w.redo) w.lim = near_limit(w);
            near_pop(w, stack);
        }
        if (w.node == kNearLeave) {
            if (!w.unsure) return false;
            // few rays: ties and near-ties.  The same steps over the
            // reference's nodes, right child first, boxes tested against the
            // best t of the moment and never again
            near_start(w, sc.root_ref, ro, rd);
            w.redo = true;
            w.lim = w.t;
            return true;
        }
    }
    const uint32_t type = w.node >> 30;
    f3 o = ro, d = rd;
    float across = 0.0f;
    if (type != ORN_NODE_INTERNAL) {
        Node nd;
        nd.load(sc.nodes + 4 * (size_t)(w.node & kRefIndexMask));
        const float4 r2 = make_float4(nd.c.x, nd.c.y, nd.c.z, nd.e.x);
        o = mk(dot4(nd.a, ro.x, ro.y, ro.z, 1.0f), dot4(nd.b, ro.x, ro.y, ro.z, 1.0f), dot4(r2, ro.x, ro.y, ro.z, 1.0f));
        d = mk(dot4(nd.a, rd.x, rd.y, rd.z, 0.0f), dot4(nd.b, rd.x, rd.y, rd.z, 0.0f), dot4(r2, rd.x, rd.y, rd.z, 0.0f));
        if (type == ORN_NODE_SPHERE) {
            // sphere_hit with the initial t_max: the root it takes does not
            // depend on a smaller one
            const float far = (float)3.40282e+38;
            const float aa = d.x * d.x + d.y * d.y + d.z * d.z;
            const float half_b = dot(o, d);
            const float cc = (o.x * o.x + o.y * o.y + o.z * o.z) - 1.0f * 1.0f;
            const float disc = half_b * half_b - aa * cc;
            if (!(disc < 0.0f)) {
                const float sq = sqrtf(disc);
                float t = (-half_b - sq) / aa;
                if (t < t_min || far < t) {
                    t = (-half_b + sq) / aa;
                    if (t < t_min || far < t) t = far;
                }
                if (t < far && near_accept(w, t, w.near)) w.hit_shape = w.node;
            }
            near_pop(w, stack);
            if (!w.away || (w.node >> 30) != ORN_NODE_INTERNAL) return true;
            o = ro;
            d = rd;
        } else {
            w.shape = w.node;
            w.entry = w.near;
            w.floor = w.sp;
            w.node = bits(nd.e.w);
            w.near = -INFINITY;
            across = nd.c.w;
        }
    }
    w.away = false;
    near_space(w, o, d);
    if (w.shape != kNearNone && !w.redo) {   // (a mesh was entered)
        w.margin = max_abs(w.oxinv) * 0x1p-21f + across * (max_abs(w.inv) + kNearSlide * min_abs(w.inv));
        w.lim = near_limit(w);
    }
    return true;
}

// A few node visits, then a triangle, then a move between spaces, each by the
// lanes that have come to one; false when the lane's ray is finished.  Five of
// six are node visits (1080p scene, a ray: 66, 5 triangles, 8 moves; the
// reference's walk 108, 5, 5): with a triangle's and a shape's code run after
// every one of them (walker_step) for two or three lanes, most issue slots
// went there; kNearInner visits between halve that against the wait.
template <int SS>
__device__ __forceinline__ bool near_step(NearWalker& w, const SceneDev& sc, f3 ro, f3 rd, float t_min,
                                          NearStack<SS>& stack) {
#pragma unroll 1
    for (int i = 0; i < kNearInner; ++i) {
        if ((w.node >> 30) == ORN_NODE_INTERNAL) near_inner(w, sc, t_min, stack);
        else break;
    }
    if ((w.node >> 30) == ORN_NODE_TRIANGLE && w.node != kNearLeave) near_triangle(w, sc, t_min, stack);
    const uint32_t type = w.node >> 30;
    if (w.node == kNearLeave || type == ORN_NODE_SPHERE || type == ORN_NODE_MESH)
        return near_move(w, sc, ro, rd, t_min, stack);
    return true;
}

// The finished ray's hit record; false when it hit nothing.
__device__ __forceinline__ bool near_finish(const NearWalker& w, const SceneDev& sc, HitRec* h) {
    if (w.hit_shape == kNearNone) return false;
    const float4 e = ldg4(sc.nodes + 4 * (size_t)(w.hit_shape & kRefIndexMask) + 3);
    h->t = w.t;
    h->material = bits(e.y);
    h->type = w.hit_shape >> 30;
    h->inv = bits(e.z) * 2u;
    h->tri = w.hit_tri * 3u;
    h->u = w.u;
    h->v = w.v;
    return true;
}

}  // namespace orn
