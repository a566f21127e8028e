// Two-level BVH4 traversal on the device: one thread per ray, the traversal stack in
// shared memory (entry k of thread t at smem[k * BLOCK + t], bank-conflict free), hit
// children pushed farthest-first so the nearest is visited next.
//
// Arithmetic follows the reference bit for bit (the file is compiled without FMA
// contraction): the slab test of bvhTraversal.h:57-72 including its NaN behaviour
// (min/max return the second operand when a lane is NaN, as SSE minps/maxps do), the
// Moller-Trumbore test of mesh.cpp:259-291, the world-to-object ray transform of
// primitive.cpp:48-59 (object-space tMin reset to 1e-4, direction not renormalised),
// and the sphere / cube tests of sphere.cpp:15-39 and cube.cpp:16-46.
// Visit order differs from the reference (which pushes children in index order
// without sorting), so among hits at exactly equal t a different primitive may win.
#pragma once
#include "gnd/layout.h"
#include "gnd/motion.h"

namespace gnd {

struct TRay {
    V3 o, d;
    float tmin, tmax;
    float time = 0.0f;   // shutter time; moves animated instances (primitive.cpp:48-50)
};

struct THit {
    float t, u, v;
    int32_t inst;     // instance (primitive in scene-file order), -1 on a miss
    uint32_t slot;    // leaf-order triangle slot (meshes); 0xFFFFFFFF for analytic shapes
};

enum TraceError : int { kTraceOk = 0, kTraceStackOverflow = 1, kTraceIterLimit = 2, kTraceBadRef = 4 };

constexpr uint32_t kSentinel = 0xFFFFFFFEu;
constexpr uint32_t kMaxIterations = 1u << 22;

__device__ __forceinline__ float4 ldg4(const void* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ uint4 ldgu4(const void* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }

// Reference-exact lane min / max (SSE semantics).
__device__ __forceinline__ float lmin(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float lmax(float a, float b) { return a > b ? a : b; }

// Work counters of the counting variants: node visits and triangle tests per lane, and
// for the phases of the persistent loop (persistentTrace) the warp steps of each phase
// (counted by lane 0; a triangle pass and a step into instances are one each) and the lanes
// that test a triangle or an instance in them, so that lanes busy per step = lane steps
// / (32 x warp steps).
struct TraceCounters {
    uint32_t nodes, tris;
    uint32_t nodeWarpSteps, leafSteps, leafWarpSteps;
};

// Moller-Trumbore against the object-space ray (mesh.cpp:259-291). Returns true when the
// triangle is hit with tmin < t < tmax; writes t, u, v.
__device__ __forceinline__ bool triTest(const Tri* tp, V3 o, V3 d, float tmin, float tmax, float& t, float& u,
                                        float& v, uint32_t& prim) {
    float4 a = ldg4(&tp->v0x), b = ldg4(&tp->v1x), c = ldg4(&tp->v2x);
    float e1x = b.x - a.x, e1y = b.y - a.y, e1z = b.z - a.z;
    float e2x = c.x - a.x, e2y = c.y - a.y, e2z = c.z - a.z;
    float px = d.y * e2z - d.z * e2y;
    float py = d.z * e2x - d.x * e2z;
    float pz = d.x * e2y - d.y * e2x;
    float det = (e1x * px + e1y * py) + e1z * pz;
    bool ok = fabsf(det) > 1e-8f;
    float invDet = __frcp_rn(det);
    float tx = o.x - a.x, ty = o.y - a.y, tz = o.z - a.z;
    u = ((tx * px + ty * py) + tz * pz) * invDet;
    ok = ok && (u >= 0.0f) && (u <= 1.0f);
    float qx = ty * e1z - tz * e1y;
    float qy = tz * e1x - tx * e1z;
    float qz = tx * e1y - ty * e1x;
    v = ((d.x * qx + d.y * qy) + d.z * qz) * invDet;
    ok = ok && (v >= 0.0f) && (u + v <= 1.0f);
    t = ((e2x * qx + e2y * qy) + e2z * qz) * invDet;
    ok = ok && (t > tmin) && (t < tmax);
    prim = __float_as_uint(a.w);
    return ok;
}

// sphere.cpp:15-39 (object space)
__device__ __forceinline__ bool sphereTest(float radius, V3 o, V3 d, float tmin, float tmax, float& tHit) {
    float A = dot(d, d);
    float B = 2.0f * dot(o, d);
    float C = dot(o, o) - (radius * radius);
    float discrim = B * B - 4.0f * A * C;
    if (discrim < 0) return false;
    float rd = sqrtf(discrim);
    float t0 = (-B - rd) / (2.0f * A);
    float t1 = (-B + rd) / (2.0f * A);
    if (t0 > tmin && t0 < tmax) { tHit = t0; return true; }
    if (t1 > tmin && t1 < tmax) { tHit = t1; return true; }
    return false;
}

// cube.cpp:16-46 (object space, extents ex)
__device__ __forceinline__ bool cubeTest(V3 ex, V3 o, V3 d, float tmin, float tmax, float& tHit) {
    float t0 = 0.0f, t1 = tmax;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float inv = 1.0f / comp(d, i);
        float oi = comp(o, i), e = comp(ex, i);
        float tn = (-e - oi) * inv;
        float tf = (e - oi) * inv;
        if (tn > tf) { float s = tn; tn = tf; tf = s; }
        t0 = tn > t0 ? tn : t0;
        t1 = tf < t1 ? tf : t1;
        if (t0 > t1) return false;
    }
    float th = t0;
    if (th < tmin) {
        th = t1;
        if (th < tmin) return false;
    }
    tHit = th;
    return true;
}

// True for a ray that can hit nothing although it enters every box: one with a NaN in its
// origin or direction (a degenerate BSDF sample). A NaN slab term never excludes a child,
// so such a ray would visit every node and triangle of the scene (4.8 s for one path of the
// 5.2M-triangle sphere grid, ended by the iteration limit). The object-space ray has NaN in
// every component of the one that held it; det or u of a triangle is then NaN and its
// comparison false (mesh.cpp:259-291), and both roots of a sphere are NaN. A cube reports a
// hit at tMax (its interval is never narrowed), which is accepted when finite.
__device__ __forceinline__ bool missesAll(const SceneView& s, const TRay& r) {
    const bool bad = isnan(r.o.x) || isnan(r.o.y) || isnan(r.o.z) || isnan(r.d.x) || isnan(r.d.y) || isnan(r.d.z);
    return bad && !(s.hasCubes && r.tmax < 3.402823466e38f);
}

// World-to-object rows of animated instance `id` at `time` (primitive.cpp:49:
// m_objectToWorld.interpolate(time).inverse()); r0..r2 hold the start transform's rows on
// entry, which stay for time <= 0. Only the MOTION variants of the traversal call it
// (scenes with animated instances); rays at time 0 (user ray batches) need none.
__device__ __forceinline__ void animatedW2ORows(const SceneView& s, uint32_t id, float time, float4& r0, float4& r1, float4& r2) {
    if (time <= 0.0f) return;
    Xf34 w;
    if (time >= 1.0f) {
        w = s.motion[id].endW2O;
    } else {
        Xf34 m;
        motionCompose(s.motion[id], (time - 0.0f) / (1.0f - 0.0f), m, w);
    }
    r0 = make_float4(w.r[0][0], w.r[0][1], w.r[0][2], w.r[0][3]);
    r1 = make_float4(w.r[1][0], w.r[1][1], w.r[1][2], w.r[1][3]);
    r2 = make_float4(w.r[2][0], w.r[2][1], w.r[2][2], w.r[2][3]);
}

// ---------------------------------------------------------------- persistent traversal
// Traversal as an incremental per-lane state machine (traceOne below runs it for one ray per
// thread) for persistent warps: lanes that finish a ray fetch the next one (warp-aggregated atomic on
// a per-launch counter), and each round runs a node phase (every lane tests inner nodes
// until it holds a leaf) and a leaf pass (the warp's lanes share out the pending triangles),
// so the warp executes one code path at a time.
//
// What bounds it: instructions issued for the lanes that still have work (about 12 of 32 on
// random rays), not bytes. Hence packed fp32 arithmetic for the slabs, a child entered or
// popped in the same step as the test before it, inner nodes dropped at the pop when a hit
// found meanwhile is nearer, and triangles of all lanes tested side by side.
constexpr int kSmemStack = 16;
constexpr int kPStackMax = 128;   // entries per ray, shared + local

// Stack entry: a child reference and, for closest-hit queries, its visit key (entry
// distance, see packKey; 0 for entries that are always taken).
template <bool KEYED>
struct TEntry;
template <>
struct TEntry<true> {
    uint32_t ref, key;
};
template <>
struct TEntry<false> {
    uint32_t ref;
};

// SMEM: entries kept in shared memory (the block's array holds SMEM * BLOCK entries, entry k
// of thread t at [k * BLOCK + t]: bank-conflict free); the remaining kPStackMax - SMEM live
// in a per-lane local array.
template <int BLOCK, int SMEM, bool KEYED>
struct TStack {
    static_assert(SMEM > 0 && SMEM < kPStackMax, "shared part of the stack out of range");
    using Entry = TEntry<KEYED>;
    Entry* smem;                 // this lane's column in the block's shared array
    Entry local[kPStackMax - SMEM];
    __device__ __forceinline__ void put(int k, uint32_t ref, uint32_t key) {
        Entry e;
        e.ref = ref;
        if constexpr (KEYED) e.key = key;
        if (k < SMEM) smem[k * BLOCK] = e;
        else local[k - SMEM] = e;
    }
    __device__ __forceinline__ Entry get(int k) const { return k < SMEM ? smem[k * BLOCK] : local[k - SMEM]; }
};

struct Trav {
    V3 o, d, inv;       // current ray (world, or object space inside a bottom-level tree)
    float tmin, tmax;   // tmax: the ray's, then the nearest hit's distance
    int curInst;        // -1 at the top level
    int sp;
    uint32_t cur;       // inner node to test, kEmpty when none
    uint32_t leaf;      // pending primitives (a leaf reference advanced past those done), kEmpty when none
    bool fast, wfast;   // current / world ray: nodeKeysFast applies (see there)
    float u, v;         // hit
    int32_t inst;
    uint32_t slot;
};

// True when (bound - o) * inv cannot be NaN for any finite or infinite node bound: the
// origin is finite and every inverse direction component is finite and non-zero.
__device__ __forceinline__ bool slabFinite(const SceneView& s, V3 o, V3 inv) {
    const bool f = isfinite(o.x) && isfinite(o.y) && isfinite(o.z) && isfinite(inv.x) && isfinite(inv.y) &&
                   isfinite(inv.z) && inv.x != 0.0f && inv.y != 0.0f && inv.z != 0.0f;
    return s.fastBoxes && f;
}

__device__ __forceinline__ void travInit(Trav& t, const SceneView& s, const TRay& ray) {
    t.o = ray.o; t.d = ray.d;
    t.inv = v3(__frcp_rn(ray.d.x), __frcp_rn(ray.d.y), __frcp_rn(ray.d.z));
    t.fast = t.wfast = slabFinite(s, t.o, t.inv) && !isnan(ray.tmin) && !isnan(ray.tmax);
    t.tmin = ray.tmin; t.tmax = ray.tmax;
    t.curInst = -1;
    t.leaf = kEmpty;
    t.sp = 0;
    t.u = t.v = 0.0f;
    t.inst = -1;
    t.slot = 0xFFFFFFFFu;
    t.cur = s.tlasRoot;   // kEmpty for a scene without primitives
}

// Visit-order key of a hit child: the entry distance's bits with the child slot in the
// two lowest bits, so that unsigned comparison orders children nearest first (distances
// within 3 ulp fall back to slot order; a negative distance, possible only with a
// negative tMin, sorts by magnitude). Order affects only which of several hits at
// exactly equal t is reported, never whether or where a hit is found.
constexpr uint32_t kMissKey = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t packKey(float a, int slot) {
    return (__float_as_uint(a) & 0x7FFFFFFCu) | (uint32_t)slot;
}
// Inner nodes on the stack with a key above this begin beyond the nearest hit: none of their
// children would be entered, since a child's box lies within its node's and the rounded slab
// distances keep that order. So they are dropped. A leaf is tested wherever its box begins: a
// triangle seen almost edge-on, or an instance far from the origin, reports distances that are
// not bounded by its box to any fixed number of ulps. (Dropping leaves beyond the hit too, with
// a margin of 2^-15: 16.8M random rays 6.56 ms instead of 6.62, microfacet 170.5 instead of 172.7,
// volumetric 29.6 instead of 31.0, and another hit at such triangles.) Keys are distances only when no entry
// distance can be negative (tMin >= 0), tMax is a positive number and the slab test is the plain
// one (a NaN term of the exact one may leave an infinite entry distance); otherwise everything is kept.
__device__ __forceinline__ uint32_t cullKey(const Trav& t) {
    return t.fast && t.tmin >= 0.0f && t.tmax > 0.0f ? __float_as_uint(t.tmax) : kMissKey;
}

// Child entry distances of one node for the current ray (bvhTraversal.h:57-72) as visit
// keys; kMissKey for a missed or empty child. nodeKeysExact is the reference's lane arithmetic with
// SSE min/max (the second operand when either is NaN), for any ray and any bounds.
__device__ __forceinline__ void nodeKeysExact(const Node4* nd, const Trav& t, uint32_t key[4]) {
    const uint4 ch = ldgu4(nd->child);
    const uint32_t ref[4] = {ch.x, ch.y, ch.z, ch.w};
    float4 lx = ldg4(nd->lox), hx = ldg4(nd->hix);
    float t1[4] = {(lx.x - t.o.x) * t.inv.x, (lx.y - t.o.x) * t.inv.x, (lx.z - t.o.x) * t.inv.x, (lx.w - t.o.x) * t.inv.x};
    float t2[4] = {(hx.x - t.o.x) * t.inv.x, (hx.y - t.o.x) * t.inv.x, (hx.z - t.o.x) * t.inv.x, (hx.w - t.o.x) * t.inv.x};
    float tn[4], tf[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { tn[i] = lmin(t1[i], t2[i]); tf[i] = lmax(t1[i], t2[i]); }
    float4 ly = ldg4(nd->loy), hy = ldg4(nd->hiy);
    float u1[4] = {(ly.x - t.o.y) * t.inv.y, (ly.y - t.o.y) * t.inv.y, (ly.z - t.o.y) * t.inv.y, (ly.w - t.o.y) * t.inv.y};
    float u2[4] = {(hy.x - t.o.y) * t.inv.y, (hy.y - t.o.y) * t.inv.y, (hy.z - t.o.y) * t.inv.y, (hy.w - t.o.y) * t.inv.y};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        tn[i] = lmax(tn[i], lmin(u1[i], u2[i]));
        tf[i] = lmin(tf[i], lmax(u1[i], u2[i]));
    }
    float4 lz = ldg4(nd->loz), hz = ldg4(nd->hiz);
    float w1[4] = {(lz.x - t.o.z) * t.inv.z, (lz.y - t.o.z) * t.inv.z, (lz.z - t.o.z) * t.inv.z, (lz.w - t.o.z) * t.inv.z};
    float w2[4] = {(hz.x - t.o.z) * t.inv.z, (hz.y - t.o.z) * t.inv.z, (hz.z - t.o.z) * t.inv.z, (hz.w - t.o.z) * t.inv.z};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // bvhTraversal.h:69-72: max(max(x, y), max(z, tMin)) <= min(min(x, y), min(z, tMax))
        float a = lmax(tn[i], lmax(lmin(w1[i], w2[i]), t.tmin));
        float b = lmin(tf[i], lmin(lmax(w1[i], w2[i]), t.tmax));
        key[i] = (a <= b && ref[i] != kEmpty) ? packKey(a, i) : kMissKey;
    }
}

// Two fp32 operations per instruction (sm_100), each rounded as its scalar form is.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// (bound - o) * inv of four bounds
__device__ __forceinline__ void slab4(float4 b, uint64_t no, uint64_t iv, float t[4]) {
    unpack2(mul2(add2(pack2(b.x, b.y), no), iv), t[0], t[1]);
    unpack2(mul2(add2(pack2(b.z, b.w), no), iv), t[2], t[3]);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The same distances with less work, for rays and nodes where it gives the same values
// (t.fast: finite origin, finite non-zero inverse direction; fastBoxes: no NaN bound, lo <= hi
// for every non-empty child, and lo = inf, hi = -inf for an empty one). Then no slab term is
// NaN, so min/max are the hardware ones, and because (bound - o) * inv is monotone in the
// bound, the smaller of the two planes of an axis is the lo plane when inv > 0 and the hi
// plane when inv < 0: the near and far planes are chosen once per axis from the direction's
// sign instead of by a min/max per child. An empty child has near = inf > far = -inf. The
// result may differ from nodeKeysExact only in the sign of a zero key, which no
// comparison sees.
__device__ __forceinline__ void nodeKeysFast(const Node4* nd, const Trav& t, uint32_t key[4]) {
    const bool sx = t.inv.x < 0.0f, sy = t.inv.y < 0.0f, sz = t.inv.z < 0.0f;
    const float4 nx = ldg4(sx ? nd->hix : nd->lox), fx = ldg4(sx ? nd->lox : nd->hix);
    const float4 ny = ldg4(sy ? nd->hiy : nd->loy), fy = ldg4(sy ? nd->loy : nd->hiy);
    const float4 nz = ldg4(sz ? nd->hiz : nd->loz), fz = ldg4(sz ? nd->loz : nd->hiz);
    float n0[4], f0[4], n1[4], f1[4], n2[4], f2[4];
    {
        const uint64_t no = pack2(-t.o.x, -t.o.x), iv = pack2(t.inv.x, t.inv.x);
        slab4(nx, no, iv, n0);
        slab4(fx, no, iv, f0);
    }
    {
        const uint64_t no = pack2(-t.o.y, -t.o.y), iv = pack2(t.inv.y, t.inv.y);
        slab4(ny, no, iv, n1);
        slab4(fy, no, iv, f1);
    }
    {
        const uint64_t no = pack2(-t.o.z, -t.o.z), iv = pack2(t.inv.z, t.inv.z);
        slab4(nz, no, iv, n2);
        slab4(fz, no, iv, f2);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = fmaxf(max3(n0[i], n1[i], n2[i]), t.tmin);
        const float b = fminf(min3(f0[i], f1[i], f2[i]), t.tmax);
        key[i] = a <= b ? packKey(a, i) : kMissKey;
    }
}

// The same direction bit for bit: 0 and -0 have reciprocals of opposite sign, and the exact slab
// test tells them apart when the origin lies on a box plane.
__device__ __forceinline__ bool sameDir(V3 a, V3 b) {
    return ((__float_as_uint(a.x) ^ __float_as_uint(b.x)) | (__float_as_uint(a.y) ^ __float_as_uint(b.y)) |
            (__float_as_uint(a.z) ^ __float_as_uint(b.z))) == 0u;
}

// Gives the lane reference `e` to work on: an inner node, or a leaf to hold.
__device__ __forceinline__ void travTake(Trav& t, uint32_t e) {
    const bool leaf = isLeaf(e);
    t.leaf = leaf ? e : kEmpty;
    t.cur = leaf ? kEmpty : e;
}

// Takes the next stack entry but the inner nodes beyond the nearest hit; a sentinel on the way
// restores the world ray (Src::world). With an empty stack the lane holds nothing.
template <bool CULL, typename Stack, typename Src>
__device__ __forceinline__ void travPop(Trav& t, const Stack& st, const Src& src) {
    t.cur = kEmpty;
    t.leaf = kEmpty;
    uint32_t cull = kMissKey;
    if constexpr (CULL) cull = cullKey(t);
    while (t.sp > 0) {
        const auto e = st.get(--t.sp);
        if (e.ref == kSentinel) {
            const V3 od = t.d;
            src.world(t.o, t.d, t.tmin);
            if (!sameDir(od, t.d)) t.inv = v3(__frcp_rn(t.d.x), __frcp_rn(t.d.y), __frcp_rn(t.d.z));
            t.fast = t.wfast;
            t.curInst = -1;
            if constexpr (CULL) cull = cullKey(t);
            continue;
        }
        if constexpr (CULL) {
            if (e.key > cull && !isLeaf(e.ref)) continue;
        }
        travTake(t, e.ref);
        return;
    }
}

// Tests the lane's inner node: the nearest hit child is taken, the others are pushed
// nearest last; without a hit the next stack entry is taken. Returns an error bitmask.
// Without ORDER (any-hit queries, whose answer does not depend on the visit order) the hit
// children are visited in slot order, which saves the sort.
template <bool COUNT, bool CULL, bool ORDER, typename Stack, typename Src>
__device__ __forceinline__ int travNodeStep(Trav& t, const Node4* __restrict__ nodes, Stack& st, const Src& src, TraceCounters* cnt) {
    const Node4* nd = nodes + t.cur;
    if (COUNT) cnt->nodes++;
    uint32_t key[4];
    const uint4 ch = ldgu4(nd->child);   // with the boxes: a load after the sort would be another L1 latency
    if (t.fast) nodeKeysFast(nd, t, key);
    else nodeKeysExact(nd, t, key);
    if (!ORDER) {
        const uint32_t ref[4] = {ch.x, ch.y, ch.z, ch.w};
        const int nhit = (key[0] != kMissKey) + (key[1] != kMissKey) + (key[2] != kMissKey) + (key[3] != kMissKey);
        if (nhit == 0) {
            travPop<CULL>(t, st, src);
            return 0;
        }
        if (t.sp + nhit - 1 > kPStackMax) return kTraceStackOverflow;
        uint32_t pending = kEmpty;
#pragma unroll
        for (int i = 3; i >= 0; --i) {
            if (key[i] == kMissKey) continue;
            if (pending != kEmpty) st.put(t.sp++, pending, 0u);
            pending = ref[i];
        }
        travTake(t, pending);
        return 0;
    }
    // ascending sort network on the packed keys (unsigned min / max)
#define GND_CSWAP(a, b)                                     \
    {                                                       \
        const uint32_t lo = min(key[a], key[b]);            \
        key[b] = max(key[a], key[b]);                       \
        key[a] = lo;                                        \
    }
    GND_CSWAP(0, 1) GND_CSWAP(2, 3) GND_CSWAP(0, 2) GND_CSWAP(1, 3) GND_CSWAP(1, 2)
#undef GND_CSWAP
    if (key[0] == kMissKey) {
        travPop<CULL>(t, st, src);
        return 0;
    }
    if (t.sp + 3 > kPStackMax && t.sp + (key[1] != kMissKey) + (key[2] != kMissKey) + (key[3] != kMissKey) > kPStackMax)
        return kTraceStackOverflow;
    // farther children on the stack (farthest deepest)
    auto refOf = [&](uint32_t k) {
        const uint32_t lo = (k & 1u) ? ch.y : ch.x, hi = (k & 1u) ? ch.w : ch.z;
        return (k & 2u) ? hi : lo;
    };
#pragma unroll
    for (int i = 3; i >= 1; --i)
        if (key[i] != kMissKey) st.put(t.sp++, refOf(key[i]), key[i]);
    travTake(t, refOf(key[0]));
    return 0;
}

__device__ __forceinline__ void travStop(Trav& t) {
    t.sp = 0;
    t.cur = t.leaf = kEmpty;
}

// One instance of the pending top-level leaf; the rest of the leaf stays pending, or goes to
// the stack when a mesh is entered. For ANY, a hit ends the ray.
template <bool ANY, bool MOTION, typename Stack>
__device__ __forceinline__ int travInstStep(Trav& t, const SceneView& s, Stack& st, const uint8_t* nullMask, float time) {
    const uint32_t first = leafFirst(t.leaf), count = leafCount(t.leaf);
    t.leaf = count > 1u ? makeLeaf(first + 1u, count - 1u) : kEmpty;
    uint32_t id = __ldg(s.tlasList + first);
    if (nullMask && nullMask[id]) return 0;
    const InstTrav* it = s.instT + id;
    float4 r0 = ldg4(&it->w2o.r[0][0]), r1 = ldg4(&it->w2o.r[1][0]), r2 = ldg4(&it->w2o.r[2][0]);
    float4 meta = ldg4(&it->kind);
    uint32_t kind = __float_as_uint(meta.x);
    if (MOTION && (kind & kInstAnimated)) animatedW2ORows(s, id, time, r0, r1, r2);
    kind &= ~kInstAnimated;
    V3 lo, ld;
    lo.x = (r0.x * t.o.x + r0.y * t.o.y) + (r0.z * t.o.z + r0.w);
    lo.y = (r1.x * t.o.x + r1.y * t.o.y) + (r1.z * t.o.z + r1.w);
    lo.z = (r2.x * t.o.x + r2.y * t.o.y) + (r2.z * t.o.z + r2.w);
    ld.x = (r0.x * t.d.x + r0.y * t.d.y) + (r0.z * t.d.z + r0.w * 0.0f);
    ld.y = (r1.x * t.d.x + r1.y * t.d.y) + (r1.z * t.d.z + r1.w * 0.0f);
    ld.z = (r2.x * t.d.x + r2.y * t.d.y) + (r2.z * t.d.z + r2.w * 0.0f);
    if (kind == kShapeMesh) {
        uint32_t root = __float_as_uint(meta.y);
        if (root == kEmpty) return 0;
        if (t.sp + 1 + (t.leaf != kEmpty) > kPStackMax) return kTraceStackOverflow;
        if (t.leaf != kEmpty) {
            // the rest of this leaf comes back after the bottom-level tree
            st.put(t.sp++, t.leaf, 0u);
            t.leaf = kEmpty;
        }
        st.put(t.sp++, kSentinel, 0u);
        t.cur = root;
        // a translation keeps the direction, and with it the three reciprocals
        if (!sameDir(ld, t.d)) t.inv = v3(__frcp_rn(ld.x), __frcp_rn(ld.y), __frcp_rn(ld.z));
        t.o = lo; t.d = ld;
        t.fast = t.wfast && slabFinite(s, lo, t.inv);
        t.tmin = kEpsilon;
        t.curInst = (int)id;
        return 0;
    }
    float th;
    bool h;
    if (kind == kShapeSphere) h = sphereTest(meta.z, lo, ld, kEpsilon, t.tmax, th);
    else h = cubeTest(v3(meta.z, meta.w, __ldg(&s.instS[id].ext[2])), lo, ld, kEpsilon, t.tmax, th);
    // bvh.cpp:39: the nearest distance starts at FLT_MAX
    if (h && th < (t.inst >= 0 ? t.tmax : 3.402823466e38f)) {
        t.tmax = th;
        t.u = t.v = 0.0f;
        t.inst = (int)id;
        t.slot = 0xFFFFFFFFu;
        if (ANY) travStop(t);
    }
    return 0;
}

// Tests triangles of the lanes' pending bottom-level leaves: up to four of each lane's leaf,
// up to 32 in all, one per lane of the warp (all lanes call it; `mine`: this lane holds such
// a leaf). The owner's ray comes by shuffle; the owner then takes the nearest hit of its
// triangles, the first of equal ones as a loop over them would. Lanes whose triangles do not
// fit keep their leaf for the next pass. `map`: this warp's 32 words of shared memory.
// On random rays a leaf holds 1.8 triangles: one pass of 21 busy lanes takes the place of 3.5
// steps with 6.
template <bool ANY, bool COUNT>
__device__ __forceinline__ void travTriPass(Trav& t, const SceneView* sv, bool mine, uint32_t* map, TraceCounters* cnt) {
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const uint32_t first = leafFirst(t.leaf), count = mine ? leafCount(t.leaf) : 0u;
    const uint32_t take = min(count, 4u);
    const uint32_t m = __ballot_sync(0xffffffffu, mine);
    const uint32_t c0 = __ballot_sync(0xffffffffu, mine && ((take - 1u) & 1u)), c1 = __ballot_sync(0xffffffffu, mine && ((take - 1u) & 2u));
    const uint32_t at = (uint32_t)__popc(m & below) + (uint32_t)__popc(c0 & below) + 2u * (uint32_t)__popc(c1 & below);
    const bool fits = mine && at + take <= 32u;
    // owner of pair p: the lane whose range starts at the last start at or below p
    const uint32_t starts = __reduce_or_sync(0xffffffffu, fits ? 1u << at : 0u);
    const uint32_t total = __reduce_max_sync(0xffffffffu, fits ? at + take : 0u);
    if (fits) map[at] = lane;
    __syncwarp();
    const bool busy = lane < total;
    const int start = 31 - __clz((int)(starts & (below | (1u << lane))));
    const uint32_t owner = busy ? map[start] : lane;
    __syncwarp();
    TRay r;
    r.o.x = __shfl_sync(0xffffffffu, t.o.x, owner); r.o.y = __shfl_sync(0xffffffffu, t.o.y, owner);
    r.o.z = __shfl_sync(0xffffffffu, t.o.z, owner);
    r.d.x = __shfl_sync(0xffffffffu, t.d.x, owner); r.d.y = __shfl_sync(0xffffffffu, t.d.y, owner);
    r.d.z = __shfl_sync(0xffffffffu, t.d.z, owner);
    r.tmin = __shfl_sync(0xffffffffu, t.tmin, owner);
    r.tmax = __shfl_sync(0xffffffffu, t.tmax, owner);
    const Tri* tris = reinterpret_cast<const Tri*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(mine ? sv->tris + first : nullptr), owner));
    float th = INFINITY, u = 0.0f, v = 0.0f;
    if (COUNT && busy) cnt->leafSteps++;
    if (busy) {
        float tt;
        uint32_t prim;
        if (triTest(tris + (lane - (uint32_t)start), r.o, r.d, r.tmin, r.tmax, tt, u, v, prim)) th = tt;
    }
    uint32_t best = 32u;
    if (__any_sync(0xffffffffu, th < INFINITY)) {
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            const float c = __shfl_sync(0xffffffffu, th, (at + k) & 31u);
            if (fits && k < take && c < t.tmax) { t.tmax = c; best = k; }
        }
        const uint32_t from = (at + best) & 31u;
        const float bu = __shfl_sync(0xffffffffu, u, from), bv = __shfl_sync(0xffffffffu, v, from);
        if (best < 4u) {
            t.u = bu; t.v = bv;
            t.inst = t.curInst;
            t.slot = first + best;
        }
    }
    if (fits) {
        if (COUNT) cnt->tris += take;
        t.leaf = count > take ? makeLeaf(first + take, count - take) : kEmpty;
        if (ANY && best < 4u) travStop(t);
    }
}

// The hit a finished query reports.
__device__ __forceinline__ THit travHit(const Trav& t) {
    THit h;
    h.t = t.inst >= 0 ? t.tmax : INFINITY;
    h.u = t.u; h.v = t.v;
    h.inst = t.inst;
    h.slot = t.slot;
    return h;
}

// Warp-aggregated fetch of the next work index for lanes in `want`.
__device__ __forceinline__ uint32_t warpFetch(uint32_t* counter, bool want) {
    uint32_t mask = __ballot_sync(0xffffffffu, want);
    uint32_t base = 0;
    int lane = threadIdx.x & 31;
    if (mask) {
        int leader = __ffs(mask) - 1;
        if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
        base = __shfl_sync(0xffffffffu, base, leader);
    }
    return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

// One ray per thread to its closest hit (the transmittance queries: a few short segments each,
// in small scenes; a thread's own loop costs less than the persistent loop's phases there).
struct OneRay {
    const TRay* r;
    __device__ __forceinline__ void world(V3& o, V3& d, float& tmin) const { o = r->o; d = r->d; tmin = r->tmin; }
};
template <bool MOTION, int BLOCK, int SMEM>
__device__ __forceinline__ int traceOne(const SceneView& s, const TRay& ray, THit& hit, TStack<BLOCK, SMEM, true>& st) {
    Trav t;
    const OneRay src{&ray};
    travInit(t, s, ray);
    if (!t.fast && missesAll(s, ray)) t.cur = kEmpty;
    const Node4* nodes = s.nodes;
    int err = 0;
    uint32_t iter = 0;
    while (t.cur != kEmpty || t.leaf != kEmpty) {
        while (t.cur != kEmpty) {
            const int e = travNodeStep<false, true, true>(t, nodes, st, src, nullptr);
            if (e || ++iter > kMaxIterations) {
                err |= e ? e : (int)kTraceIterLimit;
                travStop(t);
            }
        }
        if (t.leaf == kEmpty) break;   // the stack is empty
        if (t.curInst >= 0) {
            const uint32_t first = leafFirst(t.leaf), count = leafCount(t.leaf);
            for (uint32_t k = 0; k < count; ++k) {
                float tt, u, v;
                uint32_t prim;
                if (triTest(s.tris + first + k, t.o, t.d, t.tmin, t.tmax, tt, u, v, prim)) {
                    t.tmax = tt;
                    t.u = u; t.v = v;
                    t.inst = t.curInst;
                    t.slot = first + k;
                }
            }
            travPop<true>(t, st, src);
        } else {
            const int e = travInstStep<false, MOTION>(t, s, st, nullptr, ray.time);
            if (e) {
                err |= e;
                travStop(t);
            } else if (t.cur == kEmpty && t.leaf == kEmpty) {
                travPop<true>(t, st, src);
            }
        }
    }
    hit = travHit(t);
    return err;
}

// Persistent traversal loop. Every lane of every warp runs it to the end (the block size
// is a multiple of 32 and no lane exits early). Src provides:
//   uint32_t count()                      number of rays
//   kPlainWalk                            true: what the plain traversal visits is visited (and counted): no
//                                         distance check at the pop, rays that miss everything walked too
//   bool load(uint32_t i, TRay&, const SceneView*&, const uint8_t*& nullMask)
//   void world(V3& o, V3& d, float& tmin) const   the ray in flight again (leaving a mesh)
//   void store(uint32_t i, const THit&, const SceneView&)   (the query's scene)
// SLOT_ORDER_ANY: any-hit queries visit hit children in slot order instead of nearest
// first (faster for the bounded shadow segments of the path tracer; rays to infinity find
// an occluder sooner nearest first).
// leafBatch (1..32): the node phase ends as soon as that many lanes hold a leaf (32: when
// no lane can take another node step); lanes still traversing keep their state and go on
// in the next round. Only the interleaving of the lanes' steps changes.
// `map`: 32 words of shared memory per warp.
// Measured (one B200; 4.2M random rays on 2^20 triangles / 32 passes of the 1024^2 sphere grid):
// full node phases, refill of any idle lane 2.30 ms / 101.6 ms, one child per step, triangle by
// triangle; this loop 1.77 / 88.5 while it dropped leaves beyond the hit as well (1% more
// without, see cullKey). Its parts: kPassLanes 32, 24, 16, 12: - / 98.9, 95.3, 94.1,
// 95.9; kRefill 1, 4, 8, 12: 1.94, 1.90, 1.88, 1.94 / -, 93.0, 91.5, -; child references loaded
// with the boxes instead of after the sort -4% / -0.7%; reciprocals kept across a translation
// -1.5% / -2%. Two steps per vote, 7 or 6 blocks per SM: no gain on the small scenes.
constexpr int kPassLanes = 16;
constexpr int kRefill = 8;
template <int BLOCK, bool ANY, bool COUNT, int SMEM = kSmemStack, bool MOTION = false, bool SLOT_ORDER_ANY = false, typename Src>
__device__ __forceinline__ int persistentTrace(Src& src, uint32_t* fetchCounter, TEntry<!ANY>* smemStack, uint32_t* smemMap,
                                               TraceCounters* cnt, uint32_t leafBatch = 32) {
    constexpr bool kCull = !ANY && !Src::kPlainWalk;
    // a leaf pass takes 32 triangles: waiting for more than kPassLanes lanes gains nothing
    leafBatch = min(leafBatch, (uint32_t)kPassLanes);
    TStack<BLOCK, SMEM, !ANY> st;
    st.smem = smemStack + threadIdx.x;
    uint32_t* map = smemMap + (threadIdx.x & ~31u);
    Trav t;
    travStop(t);
    const SceneView* sv = nullptr;
    const Node4* nodes = nullptr;
    const uint8_t* nm = nullptr;
    float time = 0.0f;
    bool active = false;
    bool drained = false;   // warp-uniform: the counter has passed n
    uint32_t idx = 0;
    int err = 0;
    const uint32_t n = src.count();
    uint32_t iter = 0;
    // Fewer rays than lanes: spread over all warps, since a warp's steps grow with the number
    // of its lanes that diverge. (1000 rays: a warp each.)
    const uint32_t warps = gridDim.x * (BLOCK / 32);
    // At least one lane takes rays, to see that there are none left.
    const bool takes = (threadIdx.x & 31u) < (n < warps * 32u ? max((n + warps - 1u) / warps, 1u) : 32u);
    for (;;) {
        // new rays when kRefill lanes are out of work (or all): setting up a ray costs about
        // a node step, whatever the number of lanes doing it
        const uint32_t busy = __ballot_sync(0xffffffffu, active);
        if (!drained && __popc(busy) <= 32 - kRefill) {
            const bool idle = !active && takes;
            const uint32_t got = warpFetch(fetchCounter, idle);
            if (__any_sync(0xffffffffu, idle && got >= n)) drained = true;
            if (idle && got < n) {
                idx = got;
                TRay r;
                // a source may decline an item (it belongs to another kernel of the launch)
                if (src.load(idx, r, sv, nm)) {
                    travInit(t, *sv, r);
                    if (!Src::kPlainWalk && !t.fast && missesAll(*sv, r)) t.cur = kEmpty;
                    nodes = sv->nodes;
                    if (MOTION) time = r.time;
                    active = true;
                    iter = 0;
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) {
            if (drained) break;
            continue;
        }
        // node phase: a lane steps until it holds a leaf. Whether it steps depends only on
        // its own state, so each ray's sequence of visits, and its result, is the same
        // whatever the other rays of the warp do.
        for (;;) {
            const bool want = t.cur != kEmpty;
            const uint32_t wants = __ballot_sync(0xffffffffu, want);
            if (!wants) break;
            if ((uint32_t)__popc(__ballot_sync(0xffffffffu, t.leaf != kEmpty)) >= leafBatch) break;
            if (COUNT && (threadIdx.x & 31) == 0) cnt->nodeWarpSteps++;
            if (want) {
                const int e = travNodeStep<COUNT, kCull, !(ANY && SLOT_ORDER_ANY)>(t, nodes, st, src, cnt);
                if (e || ++iter > kMaxIterations) {
                    err |= e ? e : (int)kTraceIterLimit;
                    travStop(t);
                }
            }
        }
        // leaf pass
        const bool held = t.leaf != kEmpty;
        const bool tri = held && t.curInst >= 0;
        if (COUNT) {   // the triangle pass counts its own lanes
            const bool anyTri = __any_sync(0xffffffffu, tri), anyInst = __any_sync(0xffffffffu, held && !tri);
            if ((threadIdx.x & 31) == 0) cnt->leafWarpSteps += (anyTri ? 1u : 0u) + (anyInst ? 1u : 0u);
            if (held && !tri) cnt->leafSteps++;
        }
        if (__any_sync(0xffffffffu, tri)) travTriPass<ANY, COUNT>(t, sv, tri, map, cnt);
        if (held && !tri) {
            const int e = travInstStep<ANY, MOTION>(t, *sv, st, nm, time);
            if (e) {
                err |= e;
                travStop(t);
            }
        }
        if (t.leaf == kEmpty && t.cur == kEmpty) {
            if (t.sp > 0) travPop<kCull>(t, st, src);
            if (active && t.sp == 0 && t.leaf == kEmpty && t.cur == kEmpty) {
                src.store(idx, travHit(t), *sv);
                active = false;
            }
        }
    }
    return err;
}

}  // namespace gnd
