// Warp-cooperative exact FP64 closest-point queries on the 32-wide tree.
//
// The per-thread FP64 query (nearest64) walks the binary tree alone: about 30
// dependent node visits, and the 32 lanes of a warp take 32 different paths.
// Here the whole warp answers one query: the FP32 boxes and slabs of the wide
// tree only decide which leaf clusters can hold the nearest primitive, and
// the primitives themselves are compared in FP64 with the reference's
// expressions, so the winning distance is the minimum over all primitives and
// has the same bits whichever tree found it.
//
// What makes the FP32 pruning safe: boxes and slabs are rounded outward when
// they are built, and `margin` (a few tens of ulps of the largest coordinate)
// covers the rounding of the point to FP32 and of the bound arithmetic.  A
// cluster is skipped only when its bound exceeds the best distance found plus
// twice that margin.  wide64_usable() says for which scenes the margin is
// meaningful; others keep the per-thread query, and so does a point too far
// away for FP32 distances (fp32_reaches).
#pragma once
#include "scene.cuh"
#include "wide.cuh"

namespace wosb {

// FP32 bounds of a scene with this box can steer FP64 queries: coordinates
// whose squares stay normal FP32 numbers, and a margin small against the
// scene (a box far from the origin would make every cluster a candidate).
inline bool wide64_usable(const double bbox[6], int dim, float margin) {
    double ext = 0.0, mag = 0.0;
    for (int k = 0; k < dim; ++k) {
        const double lo = bbox[2 * k], hi = bbox[2 * k + 1];
        ext = ext > hi - lo ? ext : hi - lo;
        mag = mag > (lo < 0 ? -lo : lo) ? mag : (lo < 0 ? -lo : lo);
        mag = mag > (hi < 0 ? -hi : hi) ? mag : (hi < 0 ? -hi : hi);
    }
    return ext > 1e-9 && mag < 1e9 && static_cast<double>(margin) < 1e-3 * ext;
}

// Whether FP32 distances from p to such a scene are finite numbers: squares of
// up to 2e9 and the triangle test's products of two of them stay below 3.4e38.
// False for a NaN coordinate as well.
__device__ __forceinline__ bool fp32_reaches(float px, float py, float pz) {
    return fabsf(px) < 1e9f && fabsf(py) < 1e9f && fabsf(pz) < 1e9f;
}
// A traversal's first limit: none of the tree's nodes is below -1.
__device__ __forceinline__ float first_limit(float px, float py, float pz) {
    return fp32_reaches(px, py, pz) ? INFINITY : -1.0f;
}

// Up to this many primitives a lane's own FP64 query (nearest64) beats the
// warp's when all 32 lanes have one.  FAST_FP64 walk kernel on a B200, ms per
// thread / by the warp: 2D annulus, 12 M steps: 128 segments 2.26 / 2.98, 200
// 3.31 / 3.06, 512 4.81 / 3.18; 3D sphere, 1.5 M steps: 64 triangles 2.11 /
// 2.96, 144 3.60 / 3.21, 256 4.64 / 2.78, 3600 18.8 / 4.38.
__host__ __device__ __forceinline__ int thread_query_prims(int dim) { return dim == 2 ? 160 : 128; }

// Squared FP64 distance from p to the primitive in binary slot k and its
// closest point (the leaf test of nearest64).
template <int DIM>
__device__ __forceinline__ double slot_dist64(const SceneView &s, int k, double px, double py,
                                              double pz, double &nx, double &ny, double &nz) {
    if (DIM == 2) {
        const double2 a = s.seg64[2 * k], c = s.seg64[2 * k + 1];
        nz = 0.0;
        return npq_seg64(a.x, a.y, c.x, c.y, px, py, nx, ny);
    }
    const double2 *r = s.tri64 + 7 * k;
    const double2 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3], r4 = r[4], r5 = r[5], r6 = r[6];
    return eberly<double>(px, py, pz, r0.x, r0.y, r1.x, r1.y, r2.x, r2.y, r3.x, r3.y, r4.x, r4.y,
                          r5.x, r5.y, r6.x, r6.y, nx, ny, nz);
}

// Visits the leaf clusters whose FP32 lower bound is below `limit` (which
// leaf(cluster) lowers), nearest child first.  All 32 lanes call it with the
// same point and `limit` at first_limit.  The comparisons are strict: infinity
// is the distance of a node's padding children, which have no nodes or clusters
// of their own, and (for a point that FP32 does not reach) of real ones.
template <int DIM, class Leaf>
__device__ __forceinline__ void visit_clusters(const WideView &w, float px, float py, float pz,
                                               const float &limit, Leaf &&leaf) {
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    auto take_nearest = [&](unsigned &m, float d) -> int {
        const unsigned key = ((m >> lane) & 1u) ? order_key(d, lane) : 0xffffffffu;
        const unsigned k = __reduce_min_sync(kAll, key) & 31u;
        m &= ~(1u << k);
        return static_cast<int>(k);
    };
    if (w.H == 1) {
        leaf(0);
        return;
    }
    if (w.H == 2) {
        const float d = wide_box_dist<DIM>(w, 1, 0, px, py, pz);
        unsigned m = __ballot_sync(kAll, d < limit);
        while (m) {
            leaf(take_nearest(m, d));
            m &= __ballot_sync(kAll, d < limit);
        }
        return;
    }
    // taller trees: above the two lowest levels, children in lane order with
    // one pending mask per level; the two lowest nearest first
    unsigned mask[8];
    int parent[8];
    int h = w.H - 1;
    int node = 0;
    float top = wide_box_dist<DIM>(w, h, 0, px, py, pz);
    unsigned m2 = __ballot_sync(kAll, top < limit);
    for (;;) {
        if (h == 2) {
            while (m2) {
                const int n2 = node * 32 + take_nearest(m2, top);
                const float d1 = wide_box_dist<DIM>(w, 1, n2, px, py, pz);
                unsigned m1 = __ballot_sync(kAll, d1 < limit);
                while (m1) {
                    leaf(n2 * 32 + take_nearest(m1, d1));
                    m1 &= __ballot_sync(kAll, d1 < limit);
                }
                m2 &= __ballot_sync(kAll, top < limit);
            }
        } else if (m2) {
            const int child = node * 32 + take_nearest(m2, top);
            mask[h] = m2;
            parent[h] = node;
            node = child;
            --h;
            top = wide_box_dist<DIM>(w, h, node, px, py, pz);
            m2 = __ballot_sync(kAll, top < limit);
            continue;
        }
        // this node is done: back to its parent's pending children, whose
        // bounds are formed again against the limit of now
        if (h == w.H - 1) return;
        ++h;
        node = parent[h];
        top = wide_box_dist<DIM>(w, h, node, px, py, pz);
        m2 = mask[h] & __ballot_sync(kAll, top < limit);
    }
}

// The squared radius that still counts as a candidate once `best2` (a squared
// FP32 distance, rounded up) has been found.
__device__ __forceinline__ float candidate_limit(float best2, float margin) {
    float r;  // approximate root: the last factor covers its few ulps
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(best2));
    r += 2.0f * margin;
    return r * r * (1.0f + 0x1p-18f);
}

// Lane minimum of non-negative doubles across the warp.
__device__ __forceinline__ double warp_min_double(double v) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
    const unsigned hi = static_cast<unsigned>(b >> 32), lo = static_cast<unsigned>(b);
    const unsigned mh = __reduce_min_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? lo : 0xffffffffu);
    return __longlong_as_double(static_cast<long long>(
        (static_cast<unsigned long long>(mh) << 32) | ml));
}

// Whether two equally near primitives must be told apart as the reference's
// traversal does: their closest points are not one point (a shared vertex or
// edge, found through either, differs by ulps), or their boundaries differ.
// Grid points on a symmetry plane of a box, say, are as far from its top as
// from its bottom.
template <int DIM>
__device__ __forceinline__ bool tie_matters(const SceneView &s, int a, int b, double dx, double dy,
                                            double dz, float margin) {
    const double tol = 1e-3 * static_cast<double>(margin);
    if (dx * dx + dy * dy + (DIM == 3 ? dz * dz : 0.0) > tol * tol) return true;
    return DIM == 2 && s.segid[a].x != s.segid[b].x;
}

// This lane's nearest primitive so far (slot -1: none), its squared distance
// and closest point; `split`: another one ties with it in a way that matters.
struct LaneNearest {
    double d2, x, y, z;
    int slot;
    bool split;
};

// The winner among the lanes' primitives.  Equally near ones: the lowest
// slot, or where the choice matters what nearest64 picks, so that boundary
// points and values are the per-thread query's.  Without any (a point that
// FP32 does not reach) the per-thread query answers.
template <int DIM>
__device__ __forceinline__ int winning_slot(const SceneView &s, double px, double py, double pz,
                                            const LaneNearest &c, float margin) {
    constexpr unsigned kAll = 0xffffffffu;
    const double m = warp_min_double(c.d2);
    const bool mine = c.slot >= 0 && c.d2 == m;
    const unsigned ties = __ballot_sync(kAll, mine);
    bool per_thread = ties == 0u;
    int win = -1;
    if (ties) {
        const int from = __ffs(static_cast<int>(ties)) - 1;
        win = __shfl_sync(kAll, c.slot, from);
        if ((ties & (ties - 1u)) || __any_sync(kAll, mine && c.split)) {
            const double dx = c.x - __shfl_sync(kAll, c.x, from);
            const double dy = c.y - __shfl_sync(kAll, c.y, from);
            const double dz = DIM == 3 ? c.z - __shfl_sync(kAll, c.z, from) : 0.0;
            per_thread = __any_sync(
                kAll, mine && (c.split || tie_matters<DIM>(s, c.slot, win, dx, dy, dz, margin)));
            win = static_cast<int>(
                __reduce_min_sync(kAll, mine ? static_cast<unsigned>(c.slot) : 0xffffffffu));
        }
    }
    if (per_thread) {
        win = nearest64<DIM>(s, px, py, pz, __longlong_as_double(0x7ff0000000000000LL)).slot;
    }
    return win;
}

// Binary slot of the primitive nearest to (px, py, pz), every primitive of
// the visited clusters compared in FP64.  The same for all 32 lanes, which
// call it with the same point.
template <int DIM>
__device__ __forceinline__ int warp_nearest64_full(const SceneView &s, const WideView &w,
                                                   double px, double py, double pz,
                                                   float margin) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = static_cast<int>(threadIdx.x & 31u);
    LaneNearest c{__longlong_as_double(0x7ff0000000000000LL), 0.0, 0.0, 0.0, -1, false};
    const float fx = static_cast<float>(px), fy = static_cast<float>(py);
    const float fz = static_cast<float>(pz);
    float limit = first_limit(fx, fy, fz), ubest = INFINITY;
    visit_clusters<DIM>(w, fx, fy, fz, limit, [&](int cluster) {
        const int ws = cluster * 32 + lane;
        double d2 = __longlong_as_double(0x7ff0000000000000LL);
        if (ws < w.n) {
            const int k = __ldg(w.wide2bin + ws);
            double nx, ny, nz;
            d2 = slot_dist64<DIM>(s, k, px, py, pz, nx, ny, nz);
            const bool tie = d2 == c.d2 && c.slot >= 0;
            const bool split =
                tie && (c.split || tie_matters<DIM>(s, k, c.slot, nx - c.x, ny - c.y,
                                                    DIM == 3 ? nz - c.z : 0.0, margin));
            if (d2 < c.d2 || (tie && k < c.slot)) c = LaneNearest{d2, nx, ny, nz, k, split};
            if (tie) c.split = split;
        }
        const float u = __uint_as_float(
            __reduce_min_sync(kAll, __float_as_uint(__double2float_ru(d2))));
        if (u < ubest) {
            ubest = u;
            limit = candidate_limit(u, margin);
        }
    });
    return winning_slot<DIM>(s, px, py, pz, c, margin);
}

// The primitives that can be nearest to a point: binary slots a and, when
// FP32 distances cannot tell two apart, b (else -1).
struct Candidates {
    int a, b;
};

// This lane's primitive of leaf cluster `cluster`: its squared FP32 distance
// from p (within the margin of, or above, the true one) and a lower bound of
// the true squared distance up to the margin.
//
// 2D: the two are the same.  Point, vertices and offsets are rounded by at
// most 2^-23 of the largest coordinate, and the foot's parameter is one
// quotient, whose error moves the foot by a few 2^-24 of the offset: in all
// within half the scene's margin.
//
// 3D: Eberly's barycentric coordinates divide by det = |e1 x e2|^2.  Their
// rounding moves the computed closest point inside the triangle by at most
// about 4 2^-24 (|p - v0| L^4 / det), L the longest edge, and by up to
// (L^4 / det)^(1/2) times that where it flips the choice of an edge next to
// an obtuse corner.  A displacement delta from a minimum raises the squared
// distance by at most delta^2, so the bound subtracts
// (32 2^-24)^2 k^3 (d^2 + 4 L^2), k = L^4 / det: nothing for ordinary
// triangles, everything for slivers, which are then compared in FP64.
template <int DIM>
__device__ __forceinline__ float lane_distance(const WideView &w, int cluster, float px, float py,
                                               float pz, float &lower) {
    if (DIM == 2) {
        lower = wide_prim_dist<2>(w, cluster, px, py, pz);
        return lower;
    }
    const float *r = w.prim + cluster * (16 * 32) + (threadIdx.x & 31u);
    float4 rec[4];
    float *f = reinterpret_cast<float *>(rec);
#pragma unroll
    for (int k = 0; k < 16; ++k) f[k] = r[k * 32];
    const float d = eberly32(px, py, pz, rec);
    const float a = rec[0].w, b = rec[1].w, c = rec[2].w;
    const float l2 = fmaxf(a, fmaxf(c, a - 2.0f * b + c));
    const float k = l2 * l2 * rec[3].y;
    // fmaxf drops a NaN (a triangle too thin for FP32): bound 0
    lower = fmaxf(d - 3.7e-12f * (k * k * k) * (d + 4.0f * l2), 0.0f);
    return d;
}

// Candidates for the primitive nearest to (px, py, pz), the same for all 32
// lanes, which call it with the same point; pick_nearest64 decides between
// them.  FP32 distances choose: a primitive whose lower bound exceeds the
// smallest distance by more than two margins is not the nearest.  Mostly one
// primitive is left, sometimes two (next to a vertex of a finely divided
// curve, or an edge of a surface); the caller forms their FP64 distances for
// all its lanes at once.  More than two are compared here, and a lane that
// met two falls back to comparing every primitive in FP64.
template <int DIM>
__device__ __forceinline__ Candidates warp_candidates64(const SceneView &s, const WideView &w,
                                                        double px, double py, double pz) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = static_cast<int>(threadIdx.x & 31u);
    const float fx = static_cast<float>(px), fy = static_cast<float>(py);
    const float fz = static_cast<float>(pz);
    // points outside the scene's box (classification) carry larger ulps
    const float margin =
        fmaxf(w.margin64, 4e-6f * fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))));
    const float reach = DIM == 2 ? 0.5f * margin : margin;
    float first = INFINITY, second = INFINITY;  // this lane's two smallest bounds
    int ws = 0;
    float limit = first_limit(fx, fy, fz), ubest = INFINITY;
    visit_clusters<DIM>(w, fx, fy, fz, limit, [&](int cluster) {
        float lower;
        const float d = lane_distance<DIM>(w, cluster, fx, fy, fz, lower);
        second = fminf(second, fmaxf(first, lower));
        if (lower < first) {
            first = lower;
            ws = cluster * 32 + lane;
        }
        const float u = __uint_as_float(__reduce_min_sync(kAll, __float_as_uint(d)));
        if (u < ubest) {
            ubest = u;
            limit = candidate_limit(u, reach);
        }
    });
    const unsigned near = __ballot_sync(kAll, first <= limit && ws < w.n);
    if (__any_sync(kAll, second <= limit) || near == 0u || !(ubest < INFINITY)) {
        return Candidates{warp_nearest64_full<DIM>(s, w, px, py, pz, margin), -1};
    }
    const int k = __ldg(w.wide2bin + min(ws, w.n - 1));
    const unsigned rest = near & (near - 1u);
    const int a = __shfl_sync(kAll, k, __ffs(near) - 1);
    if (rest == 0u) return Candidates{a, -1};
    if ((rest & (rest - 1u)) == 0u) return Candidates{a, __shfl_sync(kAll, k, __ffs(rest) - 1)};
    LaneNearest c{__longlong_as_double(0x7ff0000000000000LL), 0.0, 0.0, 0.0, -1, false};
    if ((near >> lane) & 1u) {
        c.slot = k;
        c.d2 = slot_dist64<DIM>(s, k, px, py, pz, c.x, c.y, c.z);
    }
    return Candidates{winning_slot<DIM>(s, px, py, pz, c, margin), -1};
}

// The nearest of a point's candidates: its squared FP64 distance, closest
// point and binary slot.  Equally near: as winning_slot decides.
template <int DIM>
__device__ __forceinline__ double pick_nearest64(const SceneView &s, float margin, Candidates c,
                                                 double px, double py, double pz, int &slot,
                                                 double &nx, double &ny, double &nz) {
    slot = c.a;
    if (c.a < 0) {  // no finite distance (a point too far away to square)
        nx = ny = nz = 0.0;
        return __longlong_as_double(0x7ff0000000000000LL);
    }
    double d2 = slot_dist64<DIM>(s, c.a, px, py, pz, nx, ny, nz);
    if (c.b >= 0) {
        double bx, by, bz;
        const double e2 = slot_dist64<DIM>(s, c.b, px, py, pz, bx, by, bz);
        bool second = e2 < d2 || (e2 == d2 && c.b < c.a);
        if (e2 == d2 && tie_matters<DIM>(s, c.a, c.b, bx - nx, by - ny,
                                         DIM == 3 ? bz - nz : 0.0, margin)) {
            second = nearest64<DIM>(s, px, py, pz, __longlong_as_double(0x7ff0000000000000LL))
                         .slot == c.b;
        }
        if (second) {
            slot = c.b;
            d2 = e2;
            nx = bx;
            ny = by;
            nz = bz;
        }
    }
    return d2;
}

// Winding numbers of the mesh around G points, the segments spread over the
// lanes (winding_number's sum, in any order); a segment is read once for all
// G points.
template <int G>
struct WindingPoints {
    double x[G], y[G];
    int wn[G];
};
template <int G>
__device__ __forceinline__ void warp_winding_numbers(const SceneView &s, WindingPoints<G> &q) {
    const int lane = static_cast<int>(threadIdx.x & 31u);
#pragma unroll
    for (int g = 0; g < G; ++g) q.wn[g] = 0;
    for (int k = lane; k < s.n_prims; k += 32) {
        const double2 a = s.seg64[2 * k], c = s.seg64[2 * k + 1];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const double area =
                (c.x - a.x) * (q.y[g] - a.y) - (q.x[g] - a.x) * (c.y - a.y);
            if (a.y <= q.y[g]) {
                if (c.y > q.y[g] && area > 0) ++q.wn[g];
            } else {
                if (c.y <= q.y[g] && area < 0) --q.wn[g];
            }
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) q.wn[g] = __reduce_add_sync(0xffffffffu, q.wn[g]);
}

// Whether the ray meets the padded box of every node from the root to the
// leaf of binary slot k, i.e. whether count_ray_hits tests that triangle.
__device__ __forceinline__ bool ray_reaches(const SceneView &s, const double *p,
                                            const double *ray, int k) {
    int j = static_cast<int>(((static_cast<long long>(k) + 1) * (1ll << s.depth) - 1) / s.n_prims);
    while (leaf_first(j, s.n_prims, s.depth) > k) --j;
    while (leaf_first(j + 1, s.n_prims, s.depth) <= k) ++j;
    for (unsigned id = (1u << s.depth) + static_cast<unsigned>(j); id >= 1u; id >>= 1) {
        if (!ray_box(s.box64 + 6 * id, p, ray)) return false;
    }
    return true;
}

// 1 / the ray's component, which is finite also where the component is zero or
// vanishes in FP32: with an infinite reciprocal a box whose padded face holds
// the origin would be lost to 0 * inf.
__host__ __device__ __forceinline__ float ray_reciprocal(double ray) {
    const float r = static_cast<float>(ray);
    return 1.0f / (fabsf(r) < 1e-30f ? copysignf(1e-30f, r) : r);
}

// Narrows the ray's interval [t0, t1] to the slab between lo and hi (relative
// to the origin).  Along the slab an origin in it keeps the interval, and one
// off it leaves t0 > t1 for every t that the other slabs allow.
__host__ __device__ __forceinline__ void clip_to_slab(float lo, float hi, float inv, float &t0,
                                                      float &t1) {
    const float ta = lo * inv, tb = hi * inv;
    t0 = fmaxf(t0, fminf(ta, tb));
    t1 = fminf(t1, fmaxf(ta, tb));
}

// count_ray_hits by the whole warp: FP32 tests of the wide tree's boxes,
// padded by `pad` for their rounding, choose the leaf clusters, and the lanes
// test a cluster's triangles in FP64.  A triangle that is crossed plainly is
// one whose boxes the ray meets; one met at a grazing angle or ambiguously is
// counted only if the reference's traversal reaches it (ray_reaches).
__device__ __forceinline__ int warp_ray_hits(const SceneView &s, const WideView &w,
                                             const double *p, const double *ray, float pad,
                                             bool &ambiguous) {
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    float o[3], inv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o[k] = static_cast<float>(p[k]);
        inv[k] = ray_reciprocal(ray[k]);
    }
    auto meets = [&](int h, int parent) -> bool {
        const float *b = w.box + w.off[h] + parent * (11 * 32) + lane;
        float t0 = 0.0f, t1 = INFINITY;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            clip_to_slab(b[32 * k] - pad - o[k], b[32 * (3 + k)] + pad - o[k], inv[k], t0, t1);
        }
        // (padding children have lo = inf, hi = -inf)
        return t0 <= t1 * (1.0f + 0x1p-20f) && b[0] < INFINITY;
    };
    int hits = 0;
    ambiguous = false;
    auto leaf = [&](int cluster) -> bool {
        const int ws = cluster * 32 + static_cast<int>(lane);
        int h = kMiss;
        if (ws < w.n) {
            const int k = __ldg(w.wide2bin + ws);
            bool grazing;
            h = moller_trumbore(p, ray, s.tri64 + 7 * k, grazing);
            if ((h == kAmbiguous || (h == kHit && grazing)) && !ray_reaches(s, p, ray, k)) {
                h = kMiss;
            }
        }
        if (__any_sync(kAll, h == kAmbiguous)) return true;
        hits += __popc(__ballot_sync(kAll, h == kHit));
        return false;
    };
    if (w.H == 1) {
        ambiguous = leaf(0);
        return hits;
    }
    // mask[h]: children of height h (of the node parent[h]) still to visit
    unsigned mask[8];
    int parent[8];
    int h = w.H - 1;
    parent[h] = 0;
    mask[h] = __ballot_sync(kAll, meets(h, 0));
    for (;;) {
        if (mask[h] == 0u) {
            if (h == w.H - 1) return hits;
            ++h;
            continue;
        }
        const int k = __ffs(static_cast<int>(mask[h])) - 1;
        mask[h] &= mask[h] - 1u;
        const int child = parent[h] * 32 + k;
        if (h == 1) {
            if (leaf(child)) {
                ambiguous = true;
                return hits;
            }
        } else {
            --h;
            parent[h] = child;
            mask[h] = __ballot_sync(kAll, meets(h, child));
        }
    }
}

}  // namespace wosb
