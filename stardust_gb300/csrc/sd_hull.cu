// sd_hull.cu -- convex-hull rigid bodies: world AABBs, GJK/EPA narrow
// phase with atomic-free force reduction, quaternion integration.
//
// Narrow phase: sandbox/testGJK.cu:52-315 (support mapping of a vertex soup,
// Minkowski difference B - A, simplex cases, termination dot(w, d) < 0,
// at most 64 support evaluations) in the standard GJK formulation
// (Gilbert, Johnson, Keerthi 1988) with the full line/triangle/tetrahedron
// case analysis; EPA (van den Bergen 2001) for the penetration depth,
// normal and witness points, which the reference lacks.
//
// Work split: a few lanes per unique pair (A, B) = (min, max) of the per-body
// partner lists built by the LBVH (four for the first support, eight for the
// rest of GJK, a warp for EPA); what they find goes to the pair's entry in
// A's list and to its mirror in B's with the opposite sign -- exact action =
// reaction with no atomics.  One thread per body then sums its entries in list
// order (the segmented reduction), adds walls and gravity and integrates.
//
// Every float operation follows oracle/sd_oracle_hull.c in order
// (-fmad=false), so results are bit-identical to the CPU restatement.
#include "sd_common.cuh"

namespace sd {

namespace {

constexpr int kHullThreads = 128;
constexpr int kSeedThreads = 256;
constexpr int kFirstLanes = 4, kGjkLanes = 8;  // lanes of a pair in parts 1 and 2 of the narrow phase
// EPA's blocks per SM (the margin's come first), all resident at once: 4 (118
// registers) ten steps of 32,768 hulls 2314 us, 5 (96) 2325, 6 (80, spilling)
// 2357, 8 (64) 2381.
constexpr uint32_t kMarginBlocks = 152;
constexpr int kEpaBlocks = 4;
constexpr int kEpaWarps = 4;  // warps per block of the EPA kernel
constexpr int kGjkMaxIt = 64;
// support evaluations a seeded GJK run gets to certify separation before the
// plain run takes over
constexpr int kSeedMaxIt = 2;
constexpr int kEpaMaxV = 48;
constexpr int kEpaMaxF = 96;
constexpr int kEpaMaxIt = 48;
enum : int { kSep = 0, kHit = 1, kTouch = 2, kNoConv = 3 };

struct v3 {
    float x, y, z;
};
__device__ __forceinline__ v3 mk(float x, float y, float z) { return v3{x, y, z}; }
__device__ __forceinline__ v3 vadd(v3 a, v3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ v3 vsub(v3 a, v3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ v3 vneg(v3 a) { return mk(-a.x, -a.y, -a.z); }
__device__ __forceinline__ v3 vscale(v3 a, float s) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float vdot(v3 a, v3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
__device__ __forceinline__ v3 vcross(v3 a, v3 b) {
    return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ bool vzero(v3 a) { return a.x == 0.0f && a.y == 0.0f && a.z == 0.0f; }
__device__ __forceinline__ v3 f3(float4 a) { return mk(a.x, a.y, a.z); }

struct Mat {
    float r[9];
};

__device__ __forceinline__ Mat qrot(float4 q) {
    const float qs = q.x, qx = q.y, qy = q.z, qz = q.w;
    Mat R;
    R.r[0] = 1.0f - 2.0f * (qy * qy + qz * qz);
    R.r[1] = 2.0f * (qx * qy - qs * qz);
    R.r[2] = 2.0f * (qx * qz + qs * qy);
    R.r[3] = 2.0f * (qx * qy + qs * qz);
    R.r[4] = 1.0f - 2.0f * (qx * qx + qz * qz);
    R.r[5] = 2.0f * (qy * qz - qs * qx);
    R.r[6] = 2.0f * (qx * qz - qs * qy);
    R.r[7] = 2.0f * (qy * qz + qs * qx);
    R.r[8] = 1.0f - 2.0f * (qx * qx + qy * qy);
    return R;
}
__device__ __forceinline__ v3 rot(const Mat& R, v3 v) {
    return mk((R.r[0] * v.x + R.r[1] * v.y) + R.r[2] * v.z, (R.r[3] * v.x + R.r[4] * v.y) + R.r[5] * v.z,
              (R.r[6] * v.x + R.r[7] * v.y) + R.r[8] * v.z);
}
__device__ __forceinline__ v3 rotT(const Mat& R, v3 d) {
    return mk((R.r[0] * d.x + R.r[3] * d.y) + R.r[6] * d.z, (R.r[1] * d.x + R.r[4] * d.y) + R.r[7] * d.z,
              (R.r[2] * d.x + R.r[5] * d.y) + R.r[8] * d.z);
}

struct HBody {
    Mat R;
    const float4* V;
    uint32_t nv;
};

struct Cso {
    v3 w, a, b;
    uint32_t key;
};

struct HPair {
    HBody A, B;
    v3 off;  // x_B - x_A
};

// G neighbouring lanes that work on one pair: all of them hold the same
// values, and take the same branches, outside the points they split.
template <int G>
struct Group {
    uint32_t mask, sub, lead;  // the group's lanes, this one's place, the first's lane
};
template <int G>
__device__ __forceinline__ Group<G> lane_group() {
    const uint32_t lane = threadIdx.x & 31u, lead = lane & ~(uint32_t)(G - 1);
    return Group<G>{(0xffffffffu >> (32 - G)) << lead, lane - lead, lead};
}

// The supports of A in -d and of B in d: the first point (lowest index) of
// largest dot product, as a scan with a strict '>' from point 0 picks (a NaN
// product never wins, and a NaN at point 0 keeps point 0).  Past the last point
// a lane looks at the last one again, which changes nothing.
struct Best {
    float bd;
    uint32_t k;
};
__device__ __forceinline__ void take_point(Best& r, float t, uint32_t k) {
    if (t > r.bd) {
        r.bd = t;
        r.k = k;
    }
}
template <int G>
__device__ __forceinline__ void join_best(const Group<G>& g, Best& r, int o) {
    const float ob = __shfl_xor_sync(g.mask, r.bd, o);
    const uint32_t oi = __shfl_xor_sync(g.mask, r.k, o);
    if (ob > r.bd || (ob == r.bd && oi < r.k)) {
        r.bd = ob;
        r.k = oi;
    }
}
template <int G>
__device__ __forceinline__ Cso cso(const HPair& P, v3 d, const Group<G>& g) {
    const v3 da = rotT(P.A.R, vneg(d)), db = rotT(P.B.R, d);
    const uint32_t la = P.A.nv - 1u, lb = P.B.nv - 1u, last = max(la, lb);
    Best a{-INFINITY, 0u}, b = a;
    float a0 = 0.0f, b0 = 0.0f;
#pragma unroll 4
    for (uint32_t k = g.sub; k <= last; k += G) {  // both bodies' loads in flight together
        const uint32_t ka = min(k, la), kb = min(k, lb);
        const float ta = vdot(da, f3(__ldg(P.A.V + ka))), tb = vdot(db, f3(__ldg(P.B.V + kb)));
        if (k == 0u) {
            a0 = ta;
            b0 = tb;
        }
        take_point(a, ta, ka);
        take_point(b, tb, kb);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        join_best(g, a, o);
        join_best(g, b, o);
    }
    const uint32_t nan = __shfl_sync(g.mask, (a0 != a0 ? 1u : 0u) | (b0 != b0 ? 2u : 0u), g.lead);
    if (nan & 1u) a.k = 0u;
    if (nan & 2u) b.k = 0u;
    Cso r;
    r.a = rot(P.A.R, f3(__ldg(P.A.V + a.k)));
    r.b = vadd(rot(P.B.R, f3(__ldg(P.B.V + b.k))), P.off);
    r.w = vsub(r.b, r.a);
    r.key = a.k * 1024u + b.k;
    return r;
}

struct Simplex {
    float4* s;
    uint32_t order;
    int n;
};
__device__ __forceinline__ float4 point(const Simplex& S, uint32_t k) { return S.s[(S.order >> (8 * k)) & 3u]; }

// Puts p first.
__device__ __forceinline__ void add_point(Simplex* S, const Cso& p, const Group<kGjkLanes>& g) {
    uint32_t used = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (k < S->n) used |= 1u << ((S->order >> (8 * k)) & 3u);
    const uint32_t slot = (uint32_t)__ffs((int)~used) - 1u;
    __syncwarp(g.mask);  // (the other lanes are done with what the slot held)
    if (g.sub == 0) S->s[slot] = make_float4(p.w.x, p.w.y, p.w.z, __uint_as_float(p.key));
    __syncwarp(g.mask);
    S->order = (S->order << 8) | slot;
    S->n += 1;
}

// A support key (ia * 1024 + ib, both indices below 256) in 16 bits.
__device__ __forceinline__ uint16_t key16(uint32_t key) { return (uint16_t)(((key >> 10) << 8) | (key & 1023u)); }

// Closest point of a triangle to the origin (Ericson, Real-Time Collision
// Detection, 5.1.5); mask = the vertices of the closest feature.  The region is
// selected, not branched to, with one division for all of them: the groups of a
// warp are rarely in one region.
__device__ __forceinline__ v3 closest_tri(v3 A, v3 B, v3 C, int* mask) {
    const v3 ab = vsub(B, A), ac = vsub(C, A), ap = vneg(A), bp = vneg(B), cp = vneg(C);
    const float d1 = vdot(ab, ap), d2 = vdot(ac, ap), d3 = vdot(ab, bp), d4 = vdot(ac, bp), d5 = vdot(ab, cp),
                d6 = vdot(ac, cp);
    const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
    const float e4 = d4 - d3, e5 = d5 - d6;
    const int m = (d1 <= 0.0f && d2 <= 0.0f)                    ? 1
                  : (d3 >= 0.0f && d4 <= d3)                    ? 2
                  : (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f)    ? 3
                  : (d6 >= 0.0f && d5 <= d6)                    ? 4
                  : (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f)    ? 5
                  : (va <= 0.0f && e4 >= 0.0f && e5 >= 0.0f)    ? 6
                                                                : 7;
    const float num = m == 3 ? d1 : (m == 5 ? d2 : (m == 6 ? e4 : 1.0f));
    const float den = m == 3 ? d1 - d3 : (m == 5 ? d2 - d6 : (m == 6 ? e4 + e5 : (va + vb) + vc));
    const float t = num / den, s = m == 7 ? vb * t : t;
    const v3 base = (m == 2 || m == 6) ? B : (m == 4 ? C : A);
    const v3 dir = m == 6 ? vsub(C, B) : (m == 5 ? ac : ab);
    const v3 edge = vadd(base, vscale(dir, s)), inner = vadd(edge, vscale(ac, vc * t));
    *mask = m;
    return m == 7 ? inner : ((m == 3 || m == 5 || m == 6) ? edge : base);
}

/* Closest point to the origin of the simplex S (Ericson, Real-Time Collision
 * Detection, 5.1.2, 5.1.5, 5.1.6: Voronoi-region tests of the segment,
 * triangle and tetrahedron).  Reduces the simplex to the vertices of the
 * closest feature (kept in their order) and returns the point in *v; for a
 * tetrahedron that contains the origin returns true and leaves S whole.  Lane f
 * takes a tetrahedron's face f; the first face of least distance wins. */
__device__ __forceinline__ bool closest_simplex(Simplex* S, v3* v, const Group<kGjkLanes>& g) {
    if (S->n == 1) {
        *v = f3(point(*S, 0));
        return false;
    }
    if (S->n == 2) {
        const v3 A = f3(point(*S, 0)), B = f3(point(*S, 1)), ab = vsub(B, A);
        const float t = vdot(vneg(A), ab);
        if (t <= 0.0f) {
            S->n = 1;
            *v = A;
            return false;
        }
        const float den = vdot(ab, ab);
        if (t >= den) {
            S->order >>= 8;
            S->n = 1;
            *v = B;
            return false;
        }
        *v = vadd(A, vscale(ab, t / den));
        return false;
    }
    // faces with the opposite vertex: 0123, 0231, 0312, 1320 (a nibble each); a
    // triangle is 012 in every lane
    uint32_t face = 0x3210u;
    if (S->n == 4) {
        const uint32_t f = g.sub & 3u;
        face = f == 0 ? 0x3210u : (f == 1 ? 0x1320u : (f == 2 ? 0x2130u : 0x0231u));
    }
    const v3 p = f3(point(*S, face & 3u)), q = f3(point(*S, (face >> 4) & 3u)), r = f3(point(*S, (face >> 8) & 3u));
    int mask;
    v3 cv = closest_tri(p, q, r, &mask);
    if (S->n == 4) {
        const v3 o = f3(point(*S, face >> 12));
        const v3 nrm = vcross(vsub(q, p), vsub(r, p));
        const float sp = vdot(vneg(p), nrm), so = vdot(vsub(o, p), nrm);
        const bool outside = (sp > 0.0f && so < 0.0f) || (sp < 0.0f && so > 0.0f) || so == 0.0f;
        const uint32_t out = __ballot_sync(g.mask, outside) >> g.lead;
        const float dd = vdot(cv, cv);
        int best = -1;
        float best_d = 0.0f;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const float d = __shfl_sync(g.mask, dd, g.lead + f);
            if (((out >> f) & 1u) && (best < 0 || d < best_d)) {
                best = f;
                best_d = d;
            }
        }
        if (best < 0) return true;
        const uint32_t from = g.lead + (uint32_t)best;
        face = __shfl_sync(g.mask, face, from);
        mask = __shfl_sync(g.mask, mask, from);
        cv = mk(__shfl_sync(g.mask, cv.x, from), __shfl_sync(g.mask, cv.y, from), __shfl_sync(g.mask, cv.z, from));
    }
    uint32_t order = 0;
    int m = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (mask & (1 << k)) {
            order |= ((S->order >> (8 * ((face >> (4 * k)) & 3u))) & 3u) << (8 * m);
            ++m;
        }
    S->order = order;
    S->n = m;
    *v = cv;
    return false;
}

/* GJK (distance form) on B - A from a seed direction d0: v is the closest
 * point of the current simplex to the origin, the next support is taken in
 * -v, and the reference's test dot(w, d) < 0 ends it as separated; a
 * support point seen before in the run ends it as touching (no further
 * progress is possible: the origin is on the boundary of B - A within
 * rounding); a simplex that encloses the origin ends it as a hit; a zero
 * |v| as touching; max_it supports without an end as not converged.
 *
 * Run over a sequence of attempts: attempt a starts from d0[a] and may take
 * max_it[a] supports; the first attempt that certifies separation, or the
 * last attempt, decides.  Each attempt is a whole GJK run from its seed
 * (its own simplex and seen supports), but all attempts run in one loop
 * with one support call per pass, so the threads of a warp in different
 * attempts still share that call.  Returns the status; *iters =
 * supports over all attempts run, *which = the deciding attempt, *dir and
 * *S of the deciding attempt. */
struct GjkAttempts {
    v3 d0[3];
    int max_it[3];
    int n;
    // selects, not indexing, so that the attempts stay in registers
    __device__ __forceinline__ v3 seed(int a) const { return a == 0 ? d0[0] : (a == 1 ? d0[1] : d0[2]); }
    __device__ __forceinline__ int limit(int a) const {
        return a == 0 ? max_it[0] : (a == 1 ? max_it[1] : max_it[2]);
    }
};

__device__ int gjk_attempts(const HPair& P, const GjkAttempts& at, Simplex* S, int* iters, v3* dir, int* which,
                            uint16_t* seen, const Group<kGjkLanes>& g, int a, int total) {
    int it = 0;
    bool first = true;
    v3 v = mk(0.f, 0.f, 0.f);
    float vv = 0.0f;
    for (;;) {
        v3 d;
        if (first) {
            d = at.seed(a);
            if (vzero(d)) d = mk(1.0f, 0.0f, 0.0f);
            it = 0;
        } else {
            d = vneg(v);
        }
        *dir = d;
        const Cso p = cso(P, d, g);
        ++it;
        int st = -1;
        if (vdot(p.w, d) < 0.0f) {
            st = kSep;
        } else {
            const uint16_t key = key16(p.key);
            if (first) {
                S->n = 0;
                add_point(S, p, g);
                v = p.w;
            } else {
                bool met = false;
                for (int k = (int)g.sub; k < it - 1; k += kGjkLanes) met |= seen[k] == key;
                if (__any_sync(g.mask, met)) {
                    st = kTouch;
                } else {
                    add_point(S, p, g);
                    if (closest_simplex(S, &v, g)) st = kHit;
                }
            }
            if (g.sub == 0) seen[it - 1] = key;
            __syncwarp(g.mask);
            if (st < 0) vv = vdot(v, v);
            first = false;
        }
        if (st < 0) {  // the tests made before the next support
            if (vv == 0.0f) st = kTouch;
            else if (it >= at.limit(a)) st = kNoConv;
        }
        if (st >= 0) {
            total += it;
            if (st == kSep || a + 1 >= at.n) {
                *iters = total;
                *which = a;
                return st;
            }
            ++a;
            first = true;
        }
    }
}

/* The separating direction of largest margin, for training the warm-start
 * network: distance-form GJK run to convergence (|v|^2 - v.w <= 1e-5 |v|^2,
 * at most kGjkMaxIt supports) from d0; returns false when the pair is not
 * cleanly separated.  *out = -v / |v|, the direction of the closest points. */
__device__ bool gjk_margin_dir(const HPair& P, v3 d0, v3* out, Simplex* S, const Group<kGjkLanes>& g) {
    v3 d = vzero(d0) ? mk(1.0f, 0.0f, 0.0f) : d0;
    Cso p = cso(P, d, g);
    S->n = 0;
    add_point(S, p, g);
    v3 v = p.w;
    for (int it = 1; it < kGjkMaxIt; ++it) {
        const float vv = vdot(v, v);
        if (!(vv > 0.0f)) return false;
        d = vneg(v);
        p = cso(P, d, g);
        if (vv - vdot(v, p.w) <= 1e-5f * vv) break;  // converged: v is (nearly) the closest point
        if (S->n >= 4) return false;  // (closest_simplex keeps at most 3 points unless it reports a hit)
        add_point(S, p, g);
        if (closest_simplex(S, &v, g)) return false;
    }
    const float vv = vdot(v, v);
    if (!(vv > 0.0f)) return false;
    const float inv = 1.0f / sqrtf(vv);
    *out = mk(-v.x * inv, -v.y * inv, -v.z * inv);
    return true;
}

struct Face {
    uint8_t i[3];
    v3 n;
    float dist;
};

__device__ __forceinline__ bool face_make(const Cso* V, uint8_t a, uint8_t b, uint8_t c, Face* f) {
    const v3 nn = vcross(vsub(V[b].w, V[a].w), vsub(V[c].w, V[a].w));
    const float len = sqrtf(vdot(nn, nn));
    if (!(len > 0.0f)) return false;
    f->i[0] = a;
    f->i[1] = b;
    f->i[2] = c;
    f->n = mk(nn.x / len, nn.y / len, nn.z / len);
    f->dist = vdot(f->n, V[a].w);
    return true;
}

struct Contact {
    float depth;
    v3 n, c;
    int epa_iters;
    bool ok;
};

// ---------------------------------------------------------------- EPA
// One warp per intersecting pair; the polytope lives in shared memory.  The
// warp splits the scans (faces, vertices of the support calls, duplicate
// keys, face visibility, new faces) and keeps the sequential algorithm's
// choices exactly: the first face of least distance, the first vertex of
// largest dot product, kept faces and new faces in list order; lane 0 alone
// builds the horizon edge list (its order decides the new faces' order).

constexpr uint32_t kFull = 0xffffffffu;

struct EpaShared {
    Cso V[kEpaMaxV];
    Face F[kEpaMaxF];
    uint8_t E[3 * kEpaMaxF][2];
};

// The support point a key names (key = ia * 1024 + ib): the same arithmetic
// as cso(), so the same bits.
__device__ __forceinline__ Cso cso_of_key(const HPair& P, uint32_t key) {
    Cso r;
    r.a = rot(P.A.R, f3(__ldg(P.A.V + (key >> 10))));
    const v3 bb = rot(P.B.R, f3(__ldg(P.B.V + (key & 1023u))));
    r.b = vadd(bb, P.off);
    r.w = vsub(r.b, r.a);
    r.key = key;
    return r;
}

// The sequential "best = 0; if (F[k].dist < F[best].dist) best = k" by a
// warp: the first face of least distance (NaN never wins; NaN at face 0
// keeps face 0).
__device__ __forceinline__ int closest_face_warp(const Face* F, int nf) {
    const int lane = threadIdx.x & 31;
    float bd = 0.0f;
    int best = -1;
    for (int k = lane; k < nf; k += 32) {
        const float t = F[k].dist;
        if (t != t) continue;
        if (best < 0 || t < bd) {
            bd = t;
            best = k;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(kFull, bd, o);
        const int oi = __shfl_xor_sync(kFull, best, o);
        if (oi >= 0 && (best < 0 || ob < bd || (ob == bd && oi < best))) {
            bd = ob;
            best = oi;
        }
    }
    const float d0 = F[0].dist;
    return (d0 != d0 || best < 0) ? 0 : best;
}

/* EPA from GJK's enclosing tetrahedron s[0..3] (every lane holds it):
 * expands the polytope of B - A towards the origin's closest face until the
 * support gains at most tol (or repeats a vertex, or a capacity is reached);
 * the contact is that face's plane (normal -n, depth) and the midpoint of
 * the witness points at the origin's projection.  Every lane returns the
 * same *out. */
__device__ void epa_warp(const HPair& P, uint32_t key, float tol, EpaShared& sh, Contact* out) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    int nv = 4, nf = 0;
    __syncwarp();  // the previous pair's reads of the polytope are done
    if (lane < 4) sh.V[lane] = cso_of_key(P, key);
    __syncwarp();
    {  // the tetrahedron's faces, lane k the k-th: 012, 023, 031, 132
        const uint32_t i = lane == 0 ? 0x210u : (lane == 1 ? 0x320u : (lane == 2 ? 0x130u : 0x231u));
        Face f;
        bool ok = lane < 4 && face_make(sh.V, (uint8_t)(i & 15u), (uint8_t)((i >> 4) & 15u), (uint8_t)(i >> 8), &f);
        if (ok && f.dist < 0.0f) {
            const uint8_t t = f.i[1];
            f.i[1] = f.i[2];
            f.i[2] = t;
            f.n = vneg(f.n);
            f.dist = -f.dist;
        }
        const uint32_t m = __ballot_sync(kFull, ok);
        if (ok) sh.F[__popc(m & lt)] = f;
        nf = __popc(m);
    }
    out->ok = false;
    out->epa_iters = 0;
    __syncwarp();
    if (nf == 0) return;
    int best = 0;
    for (int it = 0;; ++it) {
        best = closest_face_warp(sh.F, nf);
        out->epa_iters = it + 1;
        if (it >= kEpaMaxIt || nv >= kEpaMaxV) break;
        const Face fb = sh.F[best];
        const Cso p = cso(P, fb.n, lane_group<32>());
        bool dup = false;
        for (int k = lane; k < nv; k += 32) dup |= sh.V[k].key == p.key;
        if (__any_sync(kFull, dup) || vdot(p.w, fb.n) - fb.dist <= tol) break;
        const uint8_t q = (uint8_t)nv;
        // faces that see p (before any face moves)
        constexpr int kVis = (kEpaMaxF + 31) / 32;
        uint32_t vis[kVis];
#pragma unroll
        for (int c = 0; c < kVis; ++c) {
            const int k = 32 * c + lane;
            bool v = false;
            vis[c] = 0u;
            if (32 * c >= nf) continue;
            if (k < nf) v = vdot(sh.F[k].n, vsub(p.w, sh.V[sh.F[k].i[0]].w)) > 0.0f;
            vis[c] = __ballot_sync(kFull, v);
        }
        __syncwarp();
        if (lane == 0) sh.V[nv] = p;
        ++nv;
        // horizon: edges of the visible faces in face order, an edge met
        // again reversed cancels (the last edge moves into its place)
        int ne = 0;
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < kVis; ++c)
                for (uint32_t left = vis[c]; left; left &= left - 1u) {
                    const int k = 32 * c + __ffs((int)left) - 1;
                    for (int e = 0; e < 3; ++e) {
                        const uint8_t a = sh.F[k].i[e], b = sh.F[k].i[e == 2 ? 0 : e + 1];
                        int found = -1;
                        for (int m = 0; m < ne; ++m)
                            if (sh.E[m][0] == b && sh.E[m][1] == a) {
                                found = m;
                                break;
                            }
                        if (found >= 0) {
                            sh.E[found][0] = sh.E[ne - 1][0];
                            sh.E[found][1] = sh.E[ne - 1][1];
                            --ne;
                        } else {
                            sh.E[ne][0] = a;
                            sh.E[ne][1] = b;
                            ++ne;
                        }
                    }
                }
        }
        ne = __shfl_sync(kFull, ne, 0);
        __syncwarp();
        // the faces that do not see p, compacted in order (a face moves to
        // an index at or below its own: read a chunk, then write it)
        int keep = 0;
#pragma unroll
        for (int c = 0; c < kVis; ++c) {
            if (32 * c >= nf) break;
            const int k = 32 * c + lane;
            const bool kept = k < nf && !((vis[c] >> lane) & 1u);
            Face f;
            if (kept) f = sh.F[k];
            const uint32_t m = __ballot_sync(kFull, kept);
            __syncwarp();
            if (kept) sh.F[keep + __popc(m & lt)] = f;
            keep += __popc(m);
            __syncwarp();
        }
        nf = keep;
        if (nf + ne > kEpaMaxF) break;
        // new faces (edge, p) in edge order; degenerate ones are dropped
        for (int c = 0; 32 * c < ne; ++c) {
            const int m = 32 * c + lane;
            Face f;
            const bool ok = m < ne && face_make(sh.V, sh.E[m][0], sh.E[m][1], q, &f);
            const uint32_t mk_ = __ballot_sync(kFull, ok);
            if (ok) sh.F[nf + __popc(mk_ & lt)] = f;
            nf += __popc(mk_);
        }
        __syncwarp();
        if (nf == 0) return;
    }
    Cso t[3] = {sh.V[sh.F[best].i[0]], sh.V[sh.F[best].i[1]], sh.V[sh.F[best].i[2]]};
    __syncwarp();  // the polytope is read: the next pair may overwrite it
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2 - a; ++b)
            if (t[b].key > t[b + 1].key) {
                const Cso s2 = t[b];
                t[b] = t[b + 1];
                t[b + 1] = s2;
            }
    const v3 e0 = vsub(t[1].w, t[0].w), e1 = vsub(t[2].w, t[0].w);
    const v3 nn = vcross(e0, e1);
    const float len = sqrtf(vdot(nn, nn));
    if (!(len > 0.0f)) return;
    v3 n = mk(nn.x / len, nn.y / len, nn.z / len);
    float depth = vdot(n, t[0].w);
    if (depth < 0.0f) {
        n = vneg(n);
        depth = -depth;
    }
    const v3 pp = vscale(n, depth);
    const v3 e2 = vsub(pp, t[0].w);
    const float d00 = vdot(e0, e0), d01 = vdot(e0, e1), d11 = vdot(e1, e1);
    const float d20 = vdot(e2, e0), d21 = vdot(e2, e1);
    const float den = d00 * d11 - d01 * d01;
    float l1 = 0.0f, l2 = 0.0f;
    if (den != 0.0f) {
        l1 = (d11 * d20 - d01 * d21) / den;
        l2 = (d00 * d21 - d01 * d20) / den;
    }
    const float l0 = (1.0f - l1) - l2;
    const v3 a = vadd(vadd(vscale(t[0].a, l0), vscale(t[1].a, l1)), vscale(t[2].a, l2));
    const v3 b = vadd(vadd(vscale(t[0].b, l0), vscale(t[1].b, l1)), vscale(t[2].b, l2));
    out->depth = depth;
    out->n = vneg(n);
    out->c = vscale(vadd(a, b), 0.5f);
    out->ok = true;
}

__device__ __forceinline__ void make_pair(const HullBuffers& H, uint32_t A, uint32_t B, HPair* P) {
    P->A.R = qrot(H.quat[A]);
    P->B.R = qrot(H.quat[B]);
    P->A.V = H.verts + H.vstart[A];
    P->A.nv = H.vcount[A];
    P->B.V = H.verts + H.vstart[B];
    P->B.nv = H.vcount[B];
    P->off = vsub(f3(H.pos[B]), f3(H.pos[A]));
}

__device__ __forceinline__ v3 contact_force(const HullParams& p, float delta, v3 m, v3 vr, float meff) {
    const float vn = vdot(vr, m);
    const float gn = p.damp * sqrtf(meff);
    const float fn = p.kn * delta - gn * vn;
    const float fc = fn > 0.0f ? fn : 0.0f;
    const v3 vt = mk(vr.x - vn * m.x, vr.y - vn * m.y, vr.z - vn * m.z);
    const float vt2 = vdot(vt, vt);
    v3 f = mk(fn * m.x, fn * m.y, fn * m.z);
    if (vt2 > 0.0f) {
        const float vtm = sqrtf(vt2);
        const float ftm = fminf(p.mu * fc, gn * vtm);
        const float s = ftm / vtm;
        f.x += -(s * vt.x);
        f.y += -(s * vt.y);
        f.z += -(s * vt.z);
    }
    return f;
}

// ------------------------------------------------------------- kernels

// kAabbLanes lanes to a hull, each with every kAabbLanes-th point (all of them
// start from the first, so a NaN there stays as it does in one pass); equal
// extremes go to the lower point, the one a single pass keeps.  Also clears
// the step's counters.  A chain of dependent loads: 32,768 hulls of 8 to 32
// points 12.3 us with one lane, 8.7 with four (cold caches).
constexpr int kAabbLanes = 4;

__global__ void __launch_bounds__(128) hull_aabb_kernel(HullBuffers H) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, b = t / kAabbLanes, sub = t % kAabbLanes;
    if (t < 4) H.stats[t] = 0ull;
    if (t < kHullCounters) H.counters[t] = 0u;
    const bool in = b < H.nb;
    const uint32_t bb = in ? b : 0u;
    const Mat R = qrot(H.quat[bb]);
    const float4* V = H.verts + H.vstart[bb];
    const uint32_t nv = H.vcount[bb];
    v3 w = rot(R, f3(V[0]));
    float mn[3] = {w.x, w.y, w.z}, mx[3] = {w.x, w.y, w.z};
    uint32_t imn[3] = {0, 0, 0}, imx[3] = {0, 0, 0};
#pragma unroll 4
    for (uint32_t k = sub ? sub : kAabbLanes; k < nv; k += kAabbLanes) {
        w = rot(R, f3(V[k]));
        const float c[3] = {w.x, w.y, w.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (c[a] < mn[a]) {
                mn[a] = c[a];
                imn[a] = k;
            }
            if (c[a] > mx[a]) {
                mx[a] = c[a];
                imx[a] = k;
            }
        }
    }
#pragma unroll
    for (int o = 1; o < kAabbLanes; o <<= 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float ln = __shfl_xor_sync(0xffffffffu, mn[a], o), lx = __shfl_xor_sync(0xffffffffu, mx[a], o);
            const uint32_t in_ = __shfl_xor_sync(0xffffffffu, imn[a], o), ix = __shfl_xor_sync(0xffffffffu, imx[a], o);
            if (ln < mn[a] || (ln == mn[a] && in_ < imn[a])) {
                mn[a] = ln;
                imn[a] = in_;
            }
            if (lx > mx[a] || (lx == mx[a] && ix < imx[a])) {
                mx[a] = lx;
                imx[a] = ix;
            }
        }
    }
    if (!in || sub != 0) return;
    const float4 x = H.pos[b];
    H.lo[b] = make_float4(x.x + mn[0], x.y + mn[1], x.z + mn[2], 0.f);
    H.hi[b] = make_float4(x.x + mx[0], x.y + mx[1], x.z + mx[2], 0.f);
    H.ext[2 * b] = imn[0] | (imn[1] << 8) | (imn[2] << 16);
    H.ext[2 * b + 1] = imx[0] | (imx[1] << 8) | (imx[2] << 16);
}

// Seeds from the previous step's final directions (seed mode 2): the pair's
// entry in the previous partner list of A (binary search) carries the
// direction in A's body frame.  feat (may be null) receives the 12 MLP
// inputs and w of seeds the previous-contact flag.  The entries of the unique
// pairs (self < partner) are listed on the way, a block's together: what each
// pair gets does not depend on its place.  (Counting them per body, scanning
// and filling was five launches, 20 us a step of 32,768 hulls.)
__global__ void hull_prev_seed_kernel(HullBuffers H, uint32_t mode) {
    __shared__ uint32_t s_at[kSeedThreads / 32 + 1];
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x, total = H.off[H.nb];
    // (an overflowed step is reported, not evaluated)
    if (blockIdx.x * blockDim.x >= total || (uint64_t)total > H.cap) return;
    const uint32_t self = e < total ? H.self[e] : 0u, other = e < total ? H.partners[e] : 0u;
    {
        const bool uniq = self < other;
        const uint32_t m = __ballot_sync(0xffffffffu, uniq), warp = threadIdx.x >> 5;
        if (lane_id() == 0) s_at[warp] = (uint32_t)__popc(m);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t c = 0;
            for (uint32_t k = 0; k < kSeedThreads / 32; ++k) {
                const uint32_t x = s_at[k];
                s_at[k] = c;
                c += x;
            }
            s_at[kSeedThreads / 32] = c ? atomicAdd(H.counters + kUniquePairs, c) : 0u;
        }
        __syncthreads();
        const uint32_t u = s_at[kSeedThreads / 32] + s_at[warp] + (uint32_t)__popc(m & ((1u << lane_id()) - 1u));
        if (uniq && u < H.cap / 2 + 1) H.ulist[u] = e;
    }
    if (e >= total) return;
    const uint32_t A = min(self, other), B = max(self, other);
    // previous entry of (A, B); a previous list that overflowed is ignored
    float4 prev = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t lo = H.prev_off[A];
    const uint32_t end = (uint64_t)H.prev_off[H.nb] > H.cap ? lo : H.prev_off[A + 1];
    uint32_t hi = end;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        const uint32_t v = H.prev_partners[mid];
        if (v < B) lo = mid + 1;
        else hi = mid;
    }
    const bool found = lo < end && H.prev_partners[lo] == B;
    if (found) prev = H.prev_dir[lo];
    const bool have = found && prev.w != 0.0f;
    // mode 2 seeds from the previous direction; mode 1's seeds are written by
    // the network afterwards; mode 0 runs plain GJK (the inputs are still
    // recorded, for training)
    H.seeds[e] = (mode == 2u && have) ? make_float4(prev.x, prev.y, prev.z, 1.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (H.feat) {
        // 12 inputs in A's body frame: relative quaternion conj(qA) (x) qB,
        // centre offset / (rhoA + rhoB), previous-contact flag, previous
        // direction (unit), |offset| / (rhoA + rhoB)
        const float4 qa = H.quat[A], qb = H.quat[B];
        const float as = qa.x, ax = -qa.y, ay = -qa.z, az = -qa.w;
        const float rs = as * qb.x - ((ax * qb.y + ay * qb.z) + az * qb.w);
        const float rx = as * qb.y + qb.x * ax + (ay * qb.w - az * qb.z);
        const float ry = as * qb.z + qb.x * ay + (az * qb.y - ax * qb.w);
        const float rz = as * qb.w + qb.x * az + (ax * qb.z - ay * qb.y);
        const Mat R = qrot(qa);
        const float scale = 1.0f / (H.iinv[A].w + H.iinv[B].w);
        const v3 o = vscale(rotT(R, vsub(f3(H.pos[B]), f3(H.pos[A]))), scale);
        float4* f = reinterpret_cast<float4*>(H.feat + 16 * (size_t)e);
        f[0] = make_float4(rs, rx, ry, rz);
        f[1] = make_float4(o.x, o.y, o.z, have ? 1.0f : 0.0f);
        const float pn = sqrtf((prev.x * prev.x + prev.y * prev.y) + prev.z * prev.z);
        const float pi = (have && pn > 0.0f) ? 1.0f / pn : 0.0f;
        f[2] = make_float4(prev.x * pi, prev.y * pi, prev.z * pi, sqrtf(vdot(o, o)));
        f[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// The start of a pair's first attempt.  A seeded run gets kSeedMaxIt support
// evaluations to certify separation; only that certificate is taken from it --
// any other outcome is the plain run's, so contact sets, forces and states do
// not depend on seeds.  Learned seeds (keep_anchor): the pair's anchor
// direction (its last certificate, inputs 8..10) is tried first with one
// support, and the network's direction -- trained on the pairs whose anchor
// failed -- with one more only when the anchor fails.
struct GjkSeed {
    v3 seed, anchor;  // in A's frame
    bool seeded, learned;
};
__device__ __forceinline__ GjkSeed gjk_seed(const HullBuffers& H, uint32_t e) {
    const float4 sd = H.seeds ? H.seeds[e] : make_float4(0.f, 0.f, 0.f, 0.f);
    GjkSeed r{f3(sd), mk(0.f, 0.f, 0.f), sd.w == 1.0f, false};
    r.learned = r.seeded && H.keep_anchor && H.feat;
    if (r.learned) r.anchor = f3(*reinterpret_cast<const float4*>(H.feat + 16 * (size_t)e + 8));
    return r;
}

// A pair that ends without a hit: status, direction and no force (only entries
// with a hit are summed) for its entry e and the mirror in B's list; dA is the
// final direction in A's frame (seed of the next step).  No training sample yet.
__device__ __forceinline__ void end_pair(const HullBuffers& H, uint32_t e, uint32_t em, v3 dA, bool sep) {
    const float4 d4 = make_float4(dA.x, dA.y, dA.z, sep ? 1.0f : 0.0f);
    H.dir[e] = d4;
    if (em != e) H.dir[em] = d4;
    if (H.teach && *H.teach_on) {
        H.teach[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (em != e) H.teach[em] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// The mirror entry (B, A) of the unique entry e = (A, B), found by a group in
// B's list (e where there is none: never with consistent lists).
template <int G>
__device__ __forceinline__ uint32_t mirror_entry(const HullBuffers& H, uint32_t e, uint32_t A, uint32_t B,
                                                 const Group<G>& g) {
    const uint32_t b0 = H.off[B], b1 = H.off[B + 1];
    for (uint32_t at = b0; at < b1; at += G) {
        const bool hit = at + g.sub < b1 && H.partners[at + g.sub] == A;
        const uint32_t m = __ballot_sync(g.mask, hit);
        if (m) return at + (uint32_t)__ffs((int)m) - 1u - g.lead;
    }
    return e;
}

// Narrow phase, part 1, kFirstLanes lanes per unique pair (A, B), A < B, from its
// entry in A's list: the first support of GJK, which certifies most pairs'
// separation (of 43,500 pairs of 32,768 packed hulls 33,800); the others are
// listed for part 2, where they fill whole warps.
__global__ void __launch_bounds__(kHullThreads) hull_gjk_first_kernel(HullBuffers H) {
    const Group g = lane_group<kFirstLanes>();
    if ((uint64_t)H.off[H.nb] > H.cap) return;  // an overflowed step is reported, not evaluated
    const uint32_t pairs = min(H.counters[kUniquePairs], (uint32_t)(H.cap / 2 + 1));
    const uint32_t first = (blockIdx.x * blockDim.x + threadIdx.x) / kFirstLanes, step = gridDim.x * blockDim.x / kFirstLanes;
    for (uint32_t u0 = first - g.lead / kFirstLanes; u0 < pairs; u0 += step) {  // (a warp's groups together)
        const uint32_t u = u0 + g.lead / kFirstLanes;
        bool open = false;
        if (u < pairs) {
            const uint32_t e = H.ulist[u], A = H.self[e], B = H.partners[e];
            HPair P;
            make_pair(H, A, B, &P);
            const GjkSeed sd = gjk_seed(H, e);
            v3 d = sd.seeded ? rot(P.A.R, sd.learned ? sd.anchor : sd.seed) : vneg(P.off);
            if (vzero(d)) d = mk(1.0f, 0.0f, 0.0f);
            const Cso p = cso(P, d, g);
            open = !(vdot(p.w, d) < 0.0f);
            if (!open) {
                const uint32_t em = mirror_entry(H, e, A, B, g);
                if (g.sub == 0) {
                    end_pair(H, e, em, sd.learned ? sd.anchor : rotT(P.A.R, d), true);
                    H.info[e] = H.info[em] = (uint32_t)kSep | (1u << 8);
                }
            }
        }
        const uint32_t m = __ballot_sync(0xffffffffu, open && g.sub == 0);
        uint32_t at = 0;
        if (lane_id() == 0 && m) at = atomicAdd(H.counters + kOpenPairs, (uint32_t)__popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (open && g.sub == 0) H.open[at + (uint32_t)__popc(m & ((1u << lane_id()) - 1u))] = u;
    }
}

// Part 2 for one pair.
__device__ __forceinline__ void gjk_pair(const HullBuffers& H, uint32_t u, float4* slots, uint16_t* seen, const Group<kGjkLanes>& g) {
    Simplex S{slots, 0u, 0};
    const uint32_t e = H.ulist[u], A = H.self[e], B = H.partners[e];
    HPair P;
    make_pair(H, A, B, &P);
    const GjkSeed sd = gjk_seed(H, e);
    // the plain run decides whenever no seed certifies
    GjkAttempts at;
    const v3 plain = vneg(P.off), seed = rot(P.A.R, sd.seed);
    if (sd.learned) at = {{seed, seed, plain}, {1, 1, kGjkMaxIt}, 3};  // (the anchor, attempt 0, has failed)
    else if (sd.seeded) at = {{seed, plain, plain}, {kSeedMaxIt, kGjkMaxIt, kGjkMaxIt}, 2};
    else at = {{plain, plain, plain}, {kGjkMaxIt, kGjkMaxIt, kGjkMaxIt}, 1};
    int which = 0, iters = 0;
    v3 dir;
    const int st = gjk_attempts(P, at, &S, &iters, &dir, &which, seen, g, sd.learned ? 1 : 0, sd.learned ? 1 : 0);
    const uint32_t em = mirror_entry(H, e, A, B, g);
    if (g.sub != 0) return;
    end_pair(H, e, em, rotT(P.A.R, dir), st == kSep);
    // a training step: a separated pair whose anchor failed (the cases the
    // network's seed is tried on) gets its max-margin direction beside EPA
    if (H.teach && *H.teach_on && st == kSep && sd.learned)
        H.margin[atomicAdd(H.counters + kMarginPairs, 1u)] = make_float4(dir.x, dir.y, dir.z, __uint_as_float(e));
    if (st == kHit) {  // EPA and the contact force in hull_epa_kernel
        const uint32_t k = atomicAdd(H.counters + kHitPairs, 1u);  // k < unique pairs <= cap / 2 + 1
        H.hits[k] = make_uint2(u, (uint32_t)iters);
        H.hit_keys[k] = make_uint4(__float_as_uint(point(S, 0).w), __float_as_uint(point(S, 1).w),
                                   __float_as_uint(point(S, 2).w), __float_as_uint(point(S, 3).w));
        return;
    }
    H.info[e] = H.info[em] = (uint32_t)st | ((uint32_t)iters << 8);
}

// Part 2, kGjkLanes lanes per pair left: GJK (seeded or plain).  A separated or
// touching pair is finished here; a pair found intersecting goes to the hit
// list for hull_epa_kernel.  Split so that GJK does not carry EPA's registers
// and polytope.  "hull_blocks" of its blocks per SM (109 registers, so four fit).
// 43,500 pairs of 32,768 packed hulls, 9,600 of them intersecting: the two
// parts 13 + 30 us a step; one thread per pair, 32 pairs of all kinds to a
// warp, took 62 (its simplex walked through local memory, its loads served a
// point at a time), and 219 on a training step, where a few lanes of a warp had
// the margin to find.  Latency still bounds both: part 2's chain is up to 13
// supports.  Lanes per pair: part 1 takes
// 13 us with four, 16 with eight; part 2 34 and 30.
__global__ void __launch_bounds__(kHullThreads, 4) hull_gjk_kernel(HullBuffers H) {
    // the simplex and the supports seen, per group in shared memory
    __shared__ float4 s_simplex[kHullThreads / kGjkLanes][4];
    __shared__ uint16_t s_seen[kHullThreads / kGjkLanes][kGjkMaxIt];
    const Group g = lane_group<kGjkLanes>();
    float4* const slots = s_simplex[threadIdx.x / kGjkLanes];
    uint16_t* const seen = s_seen[threadIdx.x / kGjkLanes];
    const uint32_t pairs = H.counters[kOpenPairs];
    constexpr uint32_t kTake = 32 / kGjkLanes;  // pairs a warp takes at a time, the next while it works
    uint32_t take = 0;
    if (lane_id() == 0) take = atomicAdd(H.counters + kNextPair, kTake);
    for (;;) {
        const uint32_t base = __shfl_sync(0xffffffffu, take, 0);
        if (base >= pairs) return;
        if (lane_id() == 0) take = atomicAdd(H.counters + kNextPair, kTake);
        const uint32_t k = base + g.lead / kGjkLanes;
        if (k < pairs) gjk_pair(H, H.open[k], slots, seen, g);
        __syncwarp();
    }
}

// Part 3, one warp per pair GJK found intersecting: EPA from
// GJK's enclosing tetrahedron (rebuilt from its support keys), the contact
// force at the EPA point; A's entry and B's mirror get forces of opposite
// sign -- exact action = reaction, no atomics.  Warps stride over the hit
// count.
//
// The first kMarginBlocks blocks take a training step's separated pairs (none on
// other steps), kGjkLanes lanes each: the max-margin direction in A's frame, a
// chain of up to 64 supports.  As the end of GJK it took 94 us more (ten steps,
// two of them training, 2133 us); beside EPA 2072 (76 blocks 2077, 38 2251).
__global__ void __launch_bounds__(kEpaWarps * 32, kEpaBlocks) hull_epa_kernel(HullParams p, HullBuffers H) {
    __shared__ __align__(16) EpaShared polytope[kEpaWarps];
    if (blockIdx.x < kMarginBlocks) {
        constexpr uint32_t kGroups = kEpaWarps * 32 / kGjkLanes;
        static_assert(sizeof polytope >= kGroups * 4 * sizeof(float4), "the groups' simplexes fit");
        const Group<kGjkLanes> g = lane_group<kGjkLanes>();
        const uint32_t at = threadIdx.x / kGjkLanes, n = H.counters[kMarginPairs];
        float4* const slots = reinterpret_cast<float4*>(polytope) + 4 * at;
        for (uint32_t k = blockIdx.x * kGroups + at; k < n; k += kMarginBlocks * kGroups) {
            const float4 d = H.margin[k];
            const uint32_t e = __float_as_uint(d.w);
            HPair P;
            make_pair(H, H.self[e], H.partners[e], &P);
            Simplex S{slots, 0u, 0};
            v3 m;
            if (gjk_margin_dir(P, f3(d), &m, &S, g) && g.sub == 0) {
                const v3 mA = rotT(P.A.R, m);
                H.teach[e] = make_float4(mA.x, mA.y, mA.z, 1.0f);
            }
        }
        return;
    }
    EpaShared& sh = polytope[threadIdx.x >> 5];
    const uint32_t n_hits = H.counters[kHitPairs];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nwarps = ((gridDim.x - kMarginBlocks) * blockDim.x) >> 5;
    for (uint32_t k = ((blockIdx.x - kMarginBlocks) * blockDim.x + threadIdx.x) >> 5; k < n_hits; k += nwarps) {
        const uint2 hit = H.hits[k];
        const uint32_t key = reinterpret_cast<const uint32_t*>(H.hit_keys + k)[lane & 3u];
        const uint32_t e = H.ulist[hit.x];
        const uint32_t A = H.self[e], B = H.partners[e];
        HPair P;
        make_pair(H, A, B, &P);
        const uint32_t em = mirror_entry(H, e, A, B, lane_group<32>());
        int st = kHit;
        v3 fa = mk(0.f, 0.f, 0.f), ta = mk(0.f, 0.f, 0.f), fbv = mk(0.f, 0.f, 0.f), tb = mk(0.f, 0.f, 0.f);
        Contact c;
        epa_warp(P, key, (H.iinv[A].w + H.iinv[B].w) * 1e-7f, sh, &c);
        // contact skin: overlaps within it (float GJK cannot resolve them
        // reliably) carry no force and the spring acts on depth - skin
        const float skin = (H.iinv[A].w + H.iinv[B].w) * 1e-4f;
        if (!c.ok || !(c.depth > skin)) {
            st = kTouch;
        } else {
            const float4 pa = H.pos[A], pb = H.pos[B];
            const float mA = pa.w, mB = pb.w;
            const v3 rA = c.c, rB = vsub(c.c, P.off);
            const v3 vA = vadd(f3(H.vel[A]), vcross(f3(H.omg[A]), rA));
            const v3 vB = vadd(f3(H.vel[B]), vcross(f3(H.omg[B]), rB));
            const float meff = (mA * mB) / (mA + mB);
            fbv = contact_force(p, c.depth - skin, c.n, vsub(vB, vA), meff);
            tb = vcross(rB, fbv);
            fa = vneg(fbv);
            ta = vcross(rA, fa);
        }
        if (lane == 0) {
            const uint32_t info = (uint32_t)st | (hit.y << 8) | ((uint32_t)c.epa_iters << 16);
            H.ef[e] = make_float4(fa.x, fa.y, fa.z, 0.f);
            H.et[e] = make_float4(ta.x, ta.y, ta.z, 0.f);
            H.info[e] = info;
            if (em != e) {
                H.ef[em] = make_float4(fbv.x, fbv.y, fbv.z, 0.f);
                H.et[em] = make_float4(tb.x, tb.y, tb.z, 0.f);
                H.info[em] = info;
            }
        }
    }
}

// Per body: segmented sum of its entries (list order), walls, integration;
// and the step statistics over the unique pairs (entries with self < other):
// [0] pairs, [1] GJK support evaluations, [2] intersecting pairs, [3] EPA
// iterations.  A sum that starts at +0 is never -0, so the entries without a
// hit, whose force is +0, are left out of it with the same bits.  The entries'
// states are read kEntryBatch at a time; latency bounds it
// (10 us for 32,768 hulls, and the separate statistics took 7).
constexpr int kEntryBatch = 8;

__global__ void __launch_bounds__(64) hull_integrate_kernel(HullParams p, HullBuffers H) {
    __shared__ uint32_t s_count[4];
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (threadIdx.x < 4) s_count[threadIdx.x] = 0u;
    __syncthreads();
    v3 f = mk(0.f, 0.f, 0.f), t = mk(0.f, 0.f, 0.f);
    uint32_t c[4] = {0u, 0u, 0u, 0u};
    if (b < H.nb && (uint64_t)H.off[H.nb] <= H.cap) {
        const uint32_t e0 = H.off[b], e1 = H.off[b + 1];
        for (uint32_t e = e0; e < e1; e += kEntryBatch) {
            uint32_t inf[kEntryBatch], other[kEntryBatch];
#pragma unroll
            for (int k = 0; k < kEntryBatch; ++k) {
                inf[k] = e + k < e1 ? H.info[e + k] : 0u;
                other[k] = e + k < e1 ? H.partners[e + k] : 0u;
            }
#pragma unroll
            for (int k = 0; k < kEntryBatch; ++k) {
                const bool hit = e + k < e1 && (inf[k] & 0xffu) == (uint32_t)kHit;
                if (hit) {
                    f = vadd(f, f3(H.ef[e + k]));
                    t = vadd(t, f3(H.et[e + k]));
                }
                if (e + k < e1 && b <= other[k]) {
                    c[0] += 1;
                    c[1] += (inf[k] >> 8) & 0xffu;
                    c[2] += hit;
                    c[3] += (inf[k] >> 16) & 0xffu;
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t w = __reduce_add_sync(0xffffffffu, c[k]);
        if (lane_id() == 0 && w) atomicAdd(&s_count[k], w);
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_count[threadIdx.x]) atomicAdd(H.stats + threadIdx.x, (unsigned long long)s_count[threadIdx.x]);
    if (b >= H.nb) return;
    const float4 x4 = H.pos[b], v4 = H.vel[b], w4 = H.omg[b], q4 = H.quat[b];
    const Mat R = qrot(q4);
    if (p.walls) {
        const float4* V = H.verts + H.vstart[b];
        const uint32_t ex[2] = {H.ext[2 * b], H.ext[2 * b + 1]};
        const float xs[3] = {x4.x, x4.y, x4.z};
        for (int a = 0; a < 3; ++a) {
            for (int side = 0; side < 2; ++side) {
                if (!(p.walls & (1 << (2 * a + side)))) continue;
                const uint32_t k = (ex[side] >> (8 * a)) & 0xffu;
                const v3 r = rot(R, f3(V[k]));
                const float rc[3] = {r.x, r.y, r.z};
                const float xa = xs[a] + rc[a];
                const float gap = side == 0 ? xa - p.lo[a] : p.hi[a] - xa;
                if (!(gap < 0.0f)) continue;
                float nn[3] = {0.0f, 0.0f, 0.0f};
                nn[a] = side == 0 ? 1.0f : -1.0f;
                const v3 vc = vadd(f3(v4), vcross(f3(w4), r));
                const v3 fw = contact_force(p, -gap, mk(nn[0], nn[1], nn[2]), vc, x4.w);
                f = vadd(f, fw);
                t = vadd(t, vcross(r, fw));
            }
        }
    }
    if (H.force) H.force[b] = make_float4(f.x, f.y, f.z, 0.f);
    if (H.torque) H.torque[b] = make_float4(t.x, t.y, t.z, 0.f);
    const float dt = p.dt, m = x4.w;
    const float vx = v4.x + dt * (f.x / m + p.g[0]);
    const float vy = v4.y + dt * (f.y / m + p.g[1]);
    const float vz = v4.z + dt * (f.z / m + p.g[2]);
    const float px = x4.x + dt * vx, py = x4.y + dt * vy, pz = x4.z + dt * vz;
    const float4 L4 = H.ang[b];
    const float Lx = L4.x + dt * t.x, Ly = L4.y + dt * t.y, Lz = L4.z + dt * t.z;
    const float4 ii = H.iinv[b];
    v3 lb = rotT(R, mk(Lx, Ly, Lz));
    lb = mk(lb.x * ii.x, lb.y * ii.y, lb.z * ii.z);
    const v3 om = rot(R, lb);
    const float wx = om.x, wy = om.y, wz = om.z;
    const float qs = q4.x, qx = q4.y, qy = q4.z, qz = q4.w;
    const float h = 0.5f * dt;
    const float ds = -((wx * qx + wy * qy) + wz * qz);
    const float dx = qs * wx + (wy * qz - wz * qy);
    const float dy = qs * wy + (wz * qx - wx * qz);
    const float dz = qs * wz + (wx * qy - wy * qx);
    const float ns = qs + h * ds, nx = qx + h * dx, ny = qy + h * dy, nz = qz + h * dz;
    const float nrm = sqrtf((ns * ns + nx * nx) + (ny * ny + nz * nz));
    H.pos[b] = make_float4(px, py, pz, m);
    H.vel[b] = make_float4(vx, vy, vz, 0.f);
    H.ang[b] = make_float4(Lx, Ly, Lz, 0.f);
    H.quat[b] = make_float4(ns / nrm, nx / nrm, ny / nrm, nz / nrm);
    H.omg[b] = make_float4(wx, wy, wz, 0.f);
}

inline uint32_t grid_for(uint64_t n, int threads) { return (uint32_t)((n + threads - 1) / threads); }

}  // namespace

cudaError_t hull_aabb_async(HullBuffers& H, cudaStream_t st) {
    if (H.nb == 0) return cudaSuccess;
    hull_aabb_kernel<<<grid_for((uint64_t)H.nb * kAabbLanes, 128), 128, 0, st>>>(H);
    return cudaGetLastError();
}

cudaError_t hull_seed_async(HullBuffers& H, uint32_t mode, cudaStream_t st) {
    if (H.nb == 0 || H.cap == 0) return cudaSuccess;
    hull_prev_seed_kernel<<<grid_for(H.cap, kSeedThreads), kSeedThreads, 0, st>>>(H, mode);
    return cudaGetLastError();
}

// A training step's samples (w = 1 in teach) gathered in entry order: flags,
// their scan, the copies.  Threads past the step's entry count return at once.
__global__ void hull_teach_flags_kernel(const float4* __restrict__ teach, const uint32_t* __restrict__ d_count,
                                        uint32_t cap, uint32_t* __restrict__ flags) {
    stream_wait();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= cap) return;
    const uint32_t n = min(*d_count, cap);
    flags[e] = e < n && teach[e].w == 1.0f ? 1u : 0u;
}

__global__ void hull_teach_gather_kernel(const float* __restrict__ feat, const float4* __restrict__ teach,
                                         const uint32_t* __restrict__ flags, const uint32_t* __restrict__ pos,
                                         uint32_t cap, uint32_t rows_cap, float* __restrict__ feat_c,
                                         float4* __restrict__ teach_c, uint32_t* __restrict__ d_total) {
    stream_wait();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= cap) return;
    if (e == cap - 1) *d_total = min(pos[e] + flags[e], rows_cap);
    if (!flags[e]) return;
    const uint32_t r = pos[e];
    if (r >= rows_cap) return;  // one sample per unique pair fits; inconsistent lists could exceed it
    const float4* src = reinterpret_cast<const float4*>(feat + 16 * (size_t)e);
    float4* dst = reinterpret_cast<float4*>(feat_c + 16 * (size_t)r);
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[k] = src[k];
    teach_c[r] = teach[e];
}

static int g_hull_blocks = 4;
void hull_set_blocks(int b) { g_hull_blocks = b == 3 ? 3 : 4; }
int hull_blocks() { return g_hull_blocks; }

cudaError_t hull_teach_compact_async(const HullBuffers& H, const uint32_t* d_count, float* feat_c, float4* teach_c,
                                     uint32_t* flags, uint32_t* pos, uint32_t* scan, uint32_t* d_total,
                                     cudaStream_t st) {
    const uint32_t cap = (uint32_t)H.cap;
    if (cap == 0) return cudaMemsetAsync(d_total, 0, 4, st);
    launch_after(st, grid_for(cap, 256), 256, 0, hull_teach_flags_kernel, H.teach, d_count, cap, flags);
    cudaError_t e = scan_exclusive_async(flags, pos, cap, scan, st);
    if (e != cudaSuccess) return e;
    launch_after(st, grid_for(cap, 256), 256, 0, hull_teach_gather_kernel, H.feat, H.teach, flags, pos, cap,
                 cap / 2 + 1, feat_c, teach_c, d_total);
    return cudaGetLastError();
}

cudaError_t hull_narrow_async(const HullParams& p, HullBuffers& H, cudaStream_t st) {
    if (H.nb == 0 || H.cap == 0) return cudaSuccess;
    hull_gjk_first_kernel<<<152 * 8, kHullThreads, 0, st>>>(H);
    hull_gjk_kernel<<<152 * g_hull_blocks, kHullThreads, 0, st>>>(H);
    hull_epa_kernel<<<kMarginBlocks + 152 * kEpaBlocks, kEpaWarps * 32, 0, st>>>(p, H);
    return cudaGetLastError();
}

cudaError_t hull_integrate_async(const HullParams& p, HullBuffers& H, cudaStream_t st) {
    if (H.nb == 0) return cudaSuccess;
    hull_integrate_kernel<<<grid_for(H.nb, 64), 64, 0, st>>>(p, H);
    return cudaGetLastError();
}

}  // namespace sd
