// mc_traverse.cuh - BVH traversal over the library's node layout.
//
// Binary layout: one 64-byte record per internal node holding BOTH children's
// boxes and references (leaf child k -> ~k), so a traversal step is one
// contiguous 64-byte read instead of the reference's node read plus two child
// box reads (PT:1276-1321). Leaves are 64-byte primitive records in leaf
// (sorted Morton) order: a triangle's three vertices, id, type and unit normal.
//
// The visit order and every test follow the reference's stepTraversal /
// traverseAnyHit (PT:1152-1321): both child boxes are tested against the
// current closest distance, a leaf child is intersected on the spot (left then
// right), internal children are descended left first with the right one
// pushed. Closest hits keep the first primitive found at equal t (strict <).
#pragma once
#include "mc_internal.h"
#include "mc_math.cuh"

namespace mc {

enum { STEP_CONTINUE = 0, STEP_DONE = 1, STEP_OCCLUDED = 2, STEP_OVERFLOW = 3 };

struct TraceScene {
    const float4* __restrict__ nodes;   // binary: 4 float4 per internal node; wide: 8
    const float4* __restrict__ prims;   // primitive records, 4 float4 per leaf
    int root;                           // root node of this scene (batched builds share the arrays)
};

// A lane's traversal stack in shared memory: entry i of the block's thread t
// at word i * STRIDE + t, so a warp's accesses fall in 32 distinct banks at
// any depths. Positions are byte offsets from the block's array, so a push or
// a pop is one access and one addition.
template <int STRIDE>
struct SharedStack {
    char* base;   // the block's array
    int bottom;   // this lane's entry 0
    int limit;    // one past this lane's last entry
    MC_D SharedStack(int* array, int cap)
        : base(reinterpret_cast<char*>(array)), bottom((int)threadIdx.x * 4), limit((int)threadIdx.x * 4 + cap * STRIDE * 4) {}
    static constexpr int kStep = STRIDE * 4;
    MC_D void put(int at, int v) const { *reinterpret_cast<int*>(base + at) = v; }
    MC_D int get(int at) const { return *reinterpret_cast<const int*>(base + at); }
};

// Traversal state of one ray in one lane.
struct TravState {
    RayInv r;
    float time;
    float tmax;     // closest distance so far (closest) or the segment length (any hit)
    int hitLeaf;    // leaf slot of the closest hit, -1 none
    int node;
    int sp;         // stack position (SharedStack byte offset)
    int xy, z;      // octant nodes: where the near planes of this ray's octant sit (float4 index)
};

template <class Stack>
MC_D void trav_restart(TravState& s, const Stack& stack, float tmax, int root) {
    s.tmax = tmax;
    s.hitLeaf = -1;
    s.node = root;
    s.sp = stack.bottom;
}

template <class Stack>
MC_D void trav_begin(TravState& s, const Stack& stack, const V3& o, const V3& d, float time, float tmax, int root) {
    s.r = make_ray_inv(o, d);
    const bool nx = s.r.ix < 0.0f, ny = s.r.iy < 0.0f;
    s.xy = nx ? (ny ? 2 : 6) : (ny ? 4 : 0);
    s.z = s.r.iz < 0.0f ? 10 : 8;
    s.time = time;
    trav_restart(s, stack, tmax, root);
}

MC_D float4 ldg4(const float4* p) { return __ldg(p); }
// 32 bytes (32-byte aligned) as one load.
MC_D void ldg8(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// A leaf's 64-byte record (two sectors of one line): a triangle's three
// vertices, its id and type, and its unit normal; a sphere's centers, radius
// and motion flag in the vertices' place.
MC_D const float4* leaf_record(const TraceScene& sc, int k) { return sc.prims + (size_t)((unsigned)k * 4u); }

// Intersects leaf slot k; returns true and t when the primitive is hit with
// t in the reference's accepted range (hit_* internal checks).
template <int ISECT>
MC_D bool leaf_hit(const TraceScene& sc, int k, const TravState& s, const WatertightRay& w, float& t) {
    const float4* rec = leaf_record(sc, k);
    float4 a, b, c, n;
    ldg8(rec, a, b);
    ldg8(rec + 2, c, n);
    int type = __float_as_int(c.z);
    if (type == 1) {
        V3 v0(a.x, a.y, a.z), v1(a.w, b.x, b.y), v2(b.z, b.w, c.x);
        if (ISECT == 0) return hit_triangle_ref(v0, v1, v2, V3(n.x, n.y, n.z), s.r.o, s.r.d, s.tmax, t);
        return hit_triangle_watertight(w, v0, v1, v2, s.r.o, t);
    }
    bool front;
    V3 outward;
    return hit_sphere_ref(V3(a.x, a.y, a.z), V3(a.w, b.x, b.y), b.w != 0.f, b.z, s.r.o, s.r.d, s.time, t, front, outward);
}

// One traversal step. ANY: any-hit semantics (PT:1152-1207): boxes are tested
// against the fixed segment length and the first blocker in (1e-4, tmax) ends
// the ray. Otherwise closest hit (PT:1276-1321 + testPrimitiveClosest 1537-1551).
// Counters of the instrumented variant: node visits and primitive tests.
struct TravCount {
    int visits = 0;
    int leaves = 0;
};

// A push beyond the lane's stack ends the ray and sets MC_DEVERR_STACK.
template <bool ANY, int ISECT, bool COUNT, class Stack>
MC_D int trav_step(const TraceScene& sc, TravState& s, const Stack& stack, const WatertightRay& w, int* err,
                   TravCount* cnt) {
    const float4* nd = sc.nodes + (size_t)((unsigned)s.node * 4u);
    float4 a, b, c, d;
    ldg8(nd, a, b);
    ldg8(nd + 2, c, d);
    int lref = __float_as_int(d.x), rref = __float_as_int(d.y);
    bool oL = hit_box(s.r, a.x, a.y, a.z, a.w, b.x, b.y, s.tmax);
    bool oR = hit_box(s.r, b.z, b.w, c.x, c.y, c.z, c.w, s.tmax);
    bool lLeaf = lref < 0, rLeaf = rref < 0;
    if (COUNT) {
        cnt->visits++;
        cnt->leaves += (oL && lLeaf ? 1 : 0) + (oR && rLeaf ? 1 : 0);
    }
    if (oL && lLeaf) {
        float t;
        if (leaf_hit<ISECT>(sc, ~lref, s, w, t)) {
            if (ANY) {
                if (t > 0.0001f && t < s.tmax) return STEP_OCCLUDED;
            } else if (t < s.tmax && t > 0.0001f) {
                s.tmax = t;
                s.hitLeaf = ~lref;
            }
        }
    }
    if (oR && rLeaf) {
        float t;
        if (leaf_hit<ISECT>(sc, ~rref, s, w, t)) {
            if (ANY) {
                if (t > 0.0001f && t < s.tmax) return STEP_OCCLUDED;
            } else if (t < s.tmax && t > 0.0001f) {
                s.tmax = t;
                s.hitLeaf = ~rref;
            }
        }
    }
    bool tL = oL && !lLeaf, tR = oR && !rLeaf;
    if (!tL && !tR) {
        if (s.sp == stack.bottom) return STEP_DONE;
        s.sp -= Stack::kStep;
        s.node = stack.get(s.sp);
    } else {
        if (tL && tR) {
            if (s.sp >= stack.limit) {
                atomicOr(err, MC_DEVERR_STACK);
                return STEP_DONE;
            }
            stack.put(s.sp, rref);
            s.sp += Stack::kStep;
        }
        s.node = tL ? lref : rref;
    }
    return STEP_CONTINUE;
}

// ---------------------------------------------------------------------------
// 4-wide layout: 128 bytes per node = child boxes as six float4 (lo.x, lo.y,
// lo.z, hi.x, hi.y, hi.z of the four children), the four child references
// (internal: wide-node index; leaf: ~rank; empty: MC_WIDE_EMPTY) and a spare
// float4. Leaves are stored in the reference's static visit order (their rank),
// so "first found at equal t" becomes "smallest rank at equal t" whatever order
// this traversal visits them in; every box is an exact box of the binary tree,
// tested with the reference's slab arithmetic (no per-axis early exit is needed:
// the three-axis test returns the same boolean).
// ---------------------------------------------------------------------------
// (plane - o) * (1 / d) of the four children's planes on one axis, two values
// per instruction (the same roundings as four subtractions and four
// multiplications).
MC_D float2 slab_t2(float u, float v, float o, float i) {
    float2 r;
    asm("{\n\t.reg .b64 a, b, c;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %5};\n\t"
        "add.rn.ftz.f32x2 a, a, b;\n\tmul.rn.ftz.f32x2 a, a, c;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(u), "f"(v), "f"(-o), "f"(i));
    return r;
}
MC_D float4 slab_t4(const float4& p, float o, float i) {
    const float2 a = slab_t2(p.x, p.y, o, i), b = slab_t2(p.z, p.w, o, i);
    return make_float4(a.x, a.y, b.x, b.y);
}

// The reference's slab test from a box's entry (e) and exit (x) distances per
// axis, already swapped by the sign of the direction.
MC_D bool slab_hit(float e0, float e1, float e2, float x0, float x1, float x2, float tfar, float& tnear) {
    tnear = fmaxf(max3(0.0001f, e0, e1), e2);
    return !(fminf(min3(tfar, x0, x1), x2) <= tnear);
}

MC_D void cswap(float& ka, int& va, float& kb, int& vb) {
    if (kb < ka) {
        float tk = ka; ka = kb; kb = tk;
        int tv = va; va = vb; vb = tv;
    }
}

// Child planes of a quantised node (MC_BVH_LAYOUT_WIDE4Q): plane = origin +
// byte * 2^e, one byte per child in each word.
MC_D float4 q_planes(float origin, float scale, unsigned bytes) {
    return make_float4(fmaf((float)(bytes & 0xFFu), scale, origin), fmaf((float)((bytes >> 8) & 0xFFu), scale, origin),
                       fmaf((float)((bytes >> 16) & 0xFFu), scale, origin), fmaf((float)(bytes >> 24), scale, origin));
}

MC_D float q_scale(unsigned exps, int axis) {
    const int e = (int)((exps >> (8 * axis)) & 0xFFu) - 128;
    return __int_as_float((e + 127) << 23);
}

MC_D float4 pick(bool c, const float4& a, const float4& b) {
    return make_float4(c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z, c ? a.w : b.w);
}

// FORM: MC_BVH_LAYOUT_WIDE4 (128-byte nodes, near and far planes by select),
// MC_LAYOUT_OCTANT (the same nodes in 192 bytes, by address: float4 0..7 the x
// and y planes as low low, high high, low high, high low; 8..11 low z and high
// z, each followed by the references) or MC_BVH_LAYOUT_WIDE4Q (64-byte
// quantised nodes with conservative boxes: more boxes pass, the leaf tests and
// the rank rule decide the hit as with exact boxes); with MC_LAYOUT_ORDERED for
// launches whose stack may be too short.
template <bool ANY, int ISECT, bool COUNT, class Stack, int FORM>
MC_D int trav_step4(const TraceScene& sc, TravState& s, const Stack& stack, const WatertightRay& w, int* err,
                    TravCount* cnt) {
    constexpr int NODES = FORM & 3;
    constexpr bool ORDERED = (FORM & MC_LAYOUT_ORDERED) != 0;
    float4 ax, ay, az, bx, by, bz, rf;  // near and far planes of the four children, their references
    if (NODES == MC_BVH_LAYOUT_WIDE4Q) {
        const float4* nd = sc.nodes + (size_t)((unsigned)s.node * 4u);
        float4 h, q0, q1;
        ldg8(nd, h, q0);
        ldg8(nd + 2, q1, rf);
        const unsigned ex = (unsigned)__float_as_int(h.w);
        const float sx = q_scale(ex, 0), sy = q_scale(ex, 1), sz = q_scale(ex, 2);
        const unsigned lx = (unsigned)__float_as_int(q0.x), hx = (unsigned)__float_as_int(q0.w);
        const unsigned ly = (unsigned)__float_as_int(q0.y), hy = (unsigned)__float_as_int(q1.x);
        const unsigned lz = (unsigned)__float_as_int(q0.z), hz = (unsigned)__float_as_int(q1.y);
        const bool nx = s.r.ix < 0.0f, ny = s.r.iy < 0.0f, nz = s.r.iz < 0.0f;
        ax = q_planes(h.x, sx, nx ? hx : lx);
        bx = q_planes(h.x, sx, nx ? lx : hx);
        ay = q_planes(h.y, sy, ny ? hy : ly);
        by = q_planes(h.y, sy, ny ? ly : hy);
        az = q_planes(h.z, sz, nz ? hz : lz);
        bz = q_planes(h.z, sz, nz ? lz : hz);
    } else if (NODES == MC_BVH_LAYOUT_WIDE4) {
        const float4* nd = sc.nodes + (size_t)((unsigned)s.node * 8u);
        float4 lx, ly, lz, hx, hy, hz;
        ldg8(nd, lx, ly);
        ldg8(nd + 2, lz, hx);
        ldg8(nd + 4, hy, hz);
        rf = ldg4(nd + 6);
        const bool nx = s.r.ix < 0.0f, ny = s.r.iy < 0.0f, nz = s.r.iz < 0.0f;
        ax = pick(nx, hx, lx);
        bx = pick(nx, lx, hx);
        ay = pick(ny, hy, ly);
        by = pick(ny, ly, hy);
        az = pick(nz, hz, lz);
        bz = pick(nz, lz, hz);
    } else {
        const unsigned nd = (unsigned)s.node * 12u;
        ldg8(sc.nodes + (nd + (unsigned)s.xy), ax, ay);
        ldg8(sc.nodes + (nd + ((unsigned)s.xy ^ 2u)), bx, by);
        ldg8(sc.nodes + (nd + (unsigned)s.z), az, rf);
        bz = ldg4(sc.nodes + (nd + 18u - (unsigned)s.z));
    }
    ax = slab_t4(ax, s.r.o.x, s.r.ix);
    bx = slab_t4(bx, s.r.o.x, s.r.ix);
    ay = slab_t4(ay, s.r.o.y, s.r.iy);
    by = slab_t4(by, s.r.o.y, s.r.iy);
    az = slab_t4(az, s.r.o.z, s.r.iz);
    bz = slab_t4(bz, s.r.o.z, s.r.iz);
    const int ref[4] = {__float_as_int(rf.x), __float_as_int(rf.y), __float_as_int(rf.z), __float_as_int(rf.w)};
    float tn[4];
    bool hit[4];
    hit[0] = slab_hit(ax.x, ay.x, az.x, bx.x, by.x, bz.x, s.tmax, tn[0]);
    hit[1] = slab_hit(ax.y, ay.y, az.y, bx.y, by.y, bz.y, s.tmax, tn[1]);
    hit[2] = slab_hit(ax.z, ay.z, az.z, bx.z, by.z, bz.z, s.tmax, tn[2]);
    hit[3] = slab_hit(ax.w, ay.w, az.w, bx.w, by.w, bz.w, s.tmax, tn[3]);
    if (COUNT) cnt->visits++;
    unsigned lm = (hit[0] && ref[0] < 0 ? 1u : 0u) | (hit[1] && ref[1] < 0 ? 2u : 0u) |
                  (hit[2] && ref[2] < 0 ? 4u : 0u) | (hit[3] && ref[3] < 0 ? 8u : 0u);
    // internal children by distance; misses, leaves and empty slots
    // (MC_WIDE_EMPTY, the largest int) as +inf
    constexpr unsigned kLeafOrEmpty = (unsigned)MC_WIDE_EMPTY;
    float k0 = (hit[0] && (unsigned)ref[0] < kLeafOrEmpty) ? tn[0] : INFINITY;
    float k1 = (hit[1] && (unsigned)ref[1] < kLeafOrEmpty) ? tn[1] : INFINITY;
    float k2 = (hit[2] && (unsigned)ref[2] < kLeafOrEmpty) ? tn[2] : INFINITY;
    float k3 = (hit[3] && (unsigned)ref[3] < kLeafOrEmpty) ? tn[3] : INFINITY;
    int v0 = ref[0], v1 = ref[1], v2 = ref[2], v3 = ref[3];
    cswap(k0, v0, k1, v1);
    cswap(k2, v2, k3, v3);
    cswap(k0, v0, k2, v2);
    // The ones to push stay in part order where the stack holds all that a ray of
    // the tree can push: the full sort costs 6 % of 1M scattered rays. In a shorter
    // stack (stack_entries) the order decides how many entries a ray needs, and
    // the farthest goes first.
    if (ORDERED) {
        cswap(k1, v1, k3, v3);
        cswap(k1, v1, k2, v2);
    }
    int step = STEP_CONTINUE;
    if (k0 == INFINITY) {
        if (s.sp == stack.bottom) step = STEP_DONE;
        else {
            s.sp -= Stack::kStep;
            s.node = stack.get(s.sp);
        }
    } else {
        // push the others, continue with the nearest
        const int extra = (k1 != INFINITY) + (k2 != INFINITY) + (k3 != INFINITY);
        if (s.sp + extra * Stack::kStep > stack.limit) {
            // ordered: reported after the leaves, one of which may end an occlusion ray
            if (!ORDERED) atomicOr(err, MC_DEVERR_STACK);
            step = ORDERED ? STEP_OVERFLOW : STEP_DONE;
        } else {
            if (k3 != INFINITY) { stack.put(s.sp, v3); s.sp += Stack::kStep; }
            if (ORDERED && k2 != INFINITY) { stack.put(s.sp, v2); s.sp += Stack::kStep; }
            if (k1 != INFINITY) { stack.put(s.sp, v1); s.sp += Stack::kStep; }
            if (!ORDERED && k2 != INFINITY) { stack.put(s.sp, v2); s.sp += Stack::kStep; }
            s.node = v0;
        }
    }
    // the leaf children: one loop over this lane's hit leaf children (a warp
    // runs as many iterations as its busiest lane, not one predicated block per
    // child slot)
    while (lm) {
        const int c = __ffs(lm) - 1;
        lm &= lm - 1;
        const int k = ~(c == 0 ? ref[0] : c == 1 ? ref[1] : c == 2 ? ref[2] : ref[3]);
        float t;
        if (COUNT) cnt->leaves++;
        if (leaf_hit<ISECT>(sc, k, s, w, t)) {
            if (ANY) {
                if (t > 0.0001f && t < s.tmax) return STEP_OCCLUDED;
            } else if (t > 0.0001f && (t < s.tmax || (t == s.tmax && s.hitLeaf >= 0 && k < s.hitLeaf))) {
                s.tmax = t;
                s.hitLeaf = k;
            }
        }
    }
    if (ORDERED && step == STEP_OVERFLOW) {
        atomicOr(err, MC_DEVERR_STACK);
        step = STEP_DONE;
    }
    return step;
}

// LAY: MC_BVH_LAYOUT_BINARY, or a FORM of trav_step4.
template <bool ANY, int ISECT, bool COUNT, int LAY, class Stack>
MC_D int trav_step_layout(const TraceScene& sc, TravState& s, const Stack& stack, const WatertightRay& w, int* err,
                          TravCount* cnt) {
    if (LAY != MC_BVH_LAYOUT_BINARY) return trav_step4<ANY, ISECT, COUNT, Stack, LAY>(sc, s, stack, w, err, cnt);
    return trav_step<ANY, ISECT, COUNT, Stack>(sc, s, stack, w, err, cnt);
}

// The hit record fields a leaf slot stands for.
MC_D void leaf_identity(const TraceScene& sc, int k, int& type, int& id) {
    float4 c = ldg4(leaf_record(sc, k) + 2);
    id = __float_as_int(c.y);
    type = __float_as_int(c.z);
}

}  // namespace mc
