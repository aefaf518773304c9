// Exact-path kernels: classification, PLAIN_FP64 walks and the FP64
// closest-point / PRNG checks.  This translation unit is compiled with
// --fmad=false so double expressions round exactly like the reference's
// C++17 x86-64 build (no FMA contraction); expression shapes in the device
// headers follow the reference for the same reason.
#include <algorithm>
#include <cmath>

#include "kernels.h"

namespace wosb {

namespace {

constexpr int kExactThreads = 128;

__device__ __forceinline__ double dinf() { return __longlong_as_double(0x7ff0000000000000LL); }

// 3D inside test with the reference's ray budget and majority vote
// (src/inside.cpp:228-260).  Returns the location code; counts retries.
template <class Count>
__device__ __forceinline__ int classify_3d(double bdist, double btol, int max_ray_attempts,
                                           Xoshiro &rng, int &retries, Count &&count) {
    retries = 0;
    if (bdist <= btol) return 2;
    int valid = 0, votes = 0;
    for (int a = 0; a < max_ray_attempts && valid < 3; ++a) {
        // random_unit_direction, src/inside.cpp:18-25
        const double u = rng.unit();
        const double v = rng.unit();
        const double z = 2 * u - 1;
        const double phi = 2 * kPi * v;
        const double r = sqrt(1 - z * z);
        const double ray[3] = {r * cos(phi), r * sin(phi), z};
        bool amb;
        const int hits = count(ray, amb);
        if (amb) {
            ++retries;
            continue;
        }
        votes += hits & 1;
        ++valid;
    }
    if (valid < 3) return 3;
    return votes > 1 ? 1 : 0;
}

// The start record of a point whose distance is known to be at least `lo`,
// beyond what its exact value could decide (FastStart): no nearest point
// (slot -1), which no walk reads, since such a point is neither on the
// boundary nor inside the shell.
template <int DIM>
__device__ __forceinline__ StartRecord far_start(const double *p, double lo) {
    StartRecord st;
    st.radius = lo;
    st.nx = p[0];
    st.ny = p[1];
    st.nz = DIM == 3 ? p[2] : 0.0;
    st.boundary_id = -1;
    st.slot = -1;
    return st;
}

// Location and (non-inside) fields of point t (include/wos/runner.hpp:
// 170-206), by one lane.
template <int DIM>
__device__ __forceinline__ void write_class(long long t, int where, int retries,
                                            const StartRecord &st, const EqDesc &eq,
                                            const Fields &out, uint8_t *location,
                                            StartRecord *start, DeviceCounters *ctr) {
    if (retries) atomicAdd(&ctr->ambiguous_ray_retries, static_cast<unsigned long long>(retries));
    if (where == 3) atomicAdd(&ctr->indeterminate_points, 1ull);
    location[t] = static_cast<uint8_t>(where);
    start[t] = st;
    if (out.location) out.location[t] = static_cast<uint8_t>(where);
    if (where != 1) {
        double m = __longlong_as_double(0x7ff8000000000000LL), zero = m;
        if (where == 2) {
            m = boundary_value<DIM>(eq, V3<double>{st.nx, st.ny, st.nz}, st.boundary_id);
            zero = 0.0;
        }
        if (out.mean) out.mean[t] = m;
        if (out.variance) out.variance[t] = zero;
        if (out.standard_error) out.standard_error[t] = zero;
        if (out.mean_steps) out.mean_steps[t] = zero;
    }
}

// Classification of point t by one thread alone.  A lower bound `lo` of its
// distance above `exact_below` (FastStart) becomes the start radius without
// the exact query.
template <int DIM>
__device__ __forceinline__ void classify_point(const SceneView &s, const PointSet &ps,
                                               long long t, uint64_t seed, int max_ray_attempts,
                                               double btol, const EqDesc &eq, const Fields &out,
                                               uint8_t *location, StartRecord *start,
                                               DeviceCounters *ctr, double lo = -1.0,
                                               double exact_below = 0.0) {
    double p[3];
    uint64_t linear;
    point_at(ps, t, p[0], p[1], p[2], linear);
    StartRecord st;
    if (exact_below >= 0.0 && lo > exact_below) {
        st = far_start<DIM>(p, lo);
    } else {
        const Nearest<double> q = nearest64<DIM>(s, p[0], p[1], p[2], dinf());
        st.radius = sqrt(q.best);
        st.nx = q.x;
        st.ny = q.y;
        st.nz = DIM == 3 ? q.z : 0.0;
        st.boundary_id = (DIM == 2 && q.slot >= 0) ? s.segid[q.slot].x : -1;
        st.slot = q.slot;
    }
    int where, retries = 0;
    if (DIM == 2) {
        where = st.radius <= btol ? 2 : (winding_number(s, p[0], p[1]) != 0 ? 1 : 0);
    } else {
        Xoshiro rng(splitmix64(point_seed(seed, linear) ^ kInsideStream));
        where = classify_3d(st.radius, btol, max_ray_attempts, rng, retries,
                            [&](const double *ray, bool &amb) {
                                return count_ray_hits(s, p, ray, amb);
                            });
    }
    write_class<DIM>(t, where, retries, st, eq, out, location, start, ctr);
}

template <int DIM>
__global__ void __launch_bounds__(kExactThreads)
    classify_kernel(SceneView s, PointSet ps, uint64_t seed, int max_ray_attempts, double btol,
                    EqDesc eq, Fields out, uint8_t *location, StartRecord *start,
                    DeviceCounters *ctr) {
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < ps.n;
         t += stride) {
        classify_point<DIM>(s, ps, t, seed, max_ray_attempts, btol, eq, out, location, start, ctr);
    }
}

// FastStart lower bounds of the points of a warp: lane j's point (when
// `want`) is queried by the whole warp with the lattice build's conservative
// wide-tree query, on scene w_of(j).  Returns this lane's bound, or -1.
template <int DIM, int HC, class WOf, class MarginOf>
__device__ __forceinline__ float start_bounds(bool want, double x, double y, double z, WOf w_of,
                                              MarginOf margin_of) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr float kShrink = 1.0f - 0x1p-10f;
    const int lane = static_cast<int>(threadIdx.x & 31u);
    float lo = -1.0f;
    unsigned todo = __ballot_sync(kAll, want);
    while (todo) {
        const int j = __ffs(todo) - 1;
        todo &= todo - 1u;
        const float qx = __shfl_sync(kAll, static_cast<float>(x), j);
        const float qy = __shfl_sync(kAll, static_cast<float>(y), j);
        const float qz = DIM == 3 ? __shfl_sync(kAll, static_cast<float>(z), j) : 0.0f;
        // both lookups may shuffle: every lane takes them here, converged
        const WideView &wj = w_of(j);
        const float mj = margin_of(j);
        const WideResult q = wide_nearest<DIM, HC>(wj, qx, qy, qz, kShrink * kShrink, 0.0f);
        if (lane == j && q.slot >= 0) {
            // the rounding of the point to FP32 and of the distance
            // arithmetic stay within the margin (the lattice's bound)
            const float d = (sqrtf(q.best) * kShrink - mj) * (1.0f - 0x1p-20f);
            lo = d > 0.0f ? d : 0.0f;
        }
    }
    return lo;
}

// classify_kernel with FastStart: one warp per 32 consecutive points (scenes
// whose exact queries stay per thread).
template <int DIM>
__global__ void __launch_bounds__(kExactThreads)
    classify_fast_kernel(SceneView s, WideView w, PointSet ps, uint64_t seed, int max_ray_attempts,
                         double btol, double exact_below, float margin, EqDesc eq, Fields out,
                         uint8_t *location, StartRecord *start, DeviceCounters *ctr) {
    const long long lane = threadIdx.x & 31;
    const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
    for (long long base = warp * 32; base < ps.n; base += warps * 32) {
        const long long t = base + lane;
        const bool valid = t < ps.n;
        double x = 0.0, y = 0.0, z = 0.0;
        uint64_t linear = 0;
        if (valid) point_at(ps, t, x, y, z, linear);
        const float lo = start_bounds<DIM, kHeightAny>(
            valid, x, y, z, [&](int) -> const WideView & { return w; },
            [&](int) { return margin; });
        if (valid) {
            classify_point<DIM>(s, ps, t, seed, max_ray_attempts, btol, eq, out, location, start,
                                ctr, static_cast<double>(lo), exact_below);
        }
    }
}

// Start record of point p by the whole warp: with `exact_below` >= 0 first
// FastStart's conservative query, the exact one where that does not settle it.
template <int DIM, int HC>
__device__ __forceinline__ StartRecord warp_start(const SceneView &s, const WideView &w,
                                                  const double *p, double exact_below,
                                                  float margin) {
    constexpr float kShrink = 1.0f - 0x1p-10f;
    if (exact_below >= 0.0) {
        // the lattice build's conservative query; the rounding of the point
        // to FP32 and of the distance arithmetic stay within the margin
        const WideResult q = wide_nearest<DIM, HC>(
            w, static_cast<float>(p[0]), static_cast<float>(p[1]),
            DIM == 3 ? static_cast<float>(p[2]) : 0.0f, kShrink * kShrink, 0.0f);
        double lo = -1.0;
        if (q.slot >= 0) {
            const float d = (sqrtf(q.best) * kShrink - margin) * (1.0f - 0x1p-20f);
            lo = d > 0.0f ? d : 0.0f;
        }
        if (lo > exact_below) return far_start<DIM>(p, lo);
    }
    StartRecord st;
    const double z = DIM == 3 ? p[2] : 0.0;
    const Candidates c = warp_candidates64<DIM>(s, w, p[0], p[1], z);
    st.radius = sqrt(
        pick_nearest64<DIM>(s, w.margin64, c, p[0], p[1], z, st.slot, st.nx, st.ny, st.nz));
    st.boundary_id = DIM == 2 && st.slot >= 0 ? s.segid[st.slot].x : -1;
    return st;
}

// Location of a 3D point at distance `bdist` from the boundary, its rays
// cast by the whole warp.
__device__ __forceinline__ int warp_classify_3d(const SceneView &s, const WideView &w,
                                                const double *p, double bdist, double btol,
                                                int max_ray_attempts, Xoshiro &rng,
                                                int &retries) {
    const float far = static_cast<float>(fmax(fabs(p[0]), fmax(fabs(p[1]), fabs(p[2]))));
    const float pad = fmaxf(w.margin64, 4e-6f * far);
    const bool reach = fp32_reaches(static_cast<float>(p[0]), static_cast<float>(p[1]),
                                    static_cast<float>(p[2]));
    auto count = [&](const double *ray, bool &amb) {
        return reach ? warp_ray_hits(s, w, p, ray, pad, amb) : count_ray_hits(s, p, ray, amb);
    };
    return classify_3d(bdist, btol, max_ray_attempts, rng, retries, count);
}

// Classification of points [t0, t0 + G) of `ps` (those below ps.n) by the
// whole warp: the start queries, and the winding numbers (2D, G points
// together) or the rays (3D, one point), each spread over the lanes.
template <int DIM, int HC, int G>
__device__ __forceinline__ void classify_points_warp(const SceneView &s, const WideView &w,
                                                     const PointSet &ps, long long t0,
                                                     uint64_t seed, int max_ray_attempts,
                                                     double btol, double exact_below,
                                                     float margin, const EqDesc &eq,
                                                     const Fields &out, uint8_t *location,
                                                     StartRecord *start, DeviceCounters *ctr) {
    const int lane = threadIdx.x & 31;
    StartRecord mine{};  // lane g: point t0 + g
    WindingPoints<G> q{};
    uint64_t linear = 0;
    double p[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int g = 0; g < G; ++g) {
        point_at(ps, min(t0 + g, ps.n - 1), p[0], p[1], p[2], linear);
        const StartRecord st = warp_start<DIM, HC>(s, w, p, exact_below, margin);
        if (lane == g) mine = st;
    }
    int where = 0, retries = 0;
    if (DIM == 2) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            point_at(ps, min(t0 + g, ps.n - 1), q.x[g], q.y[g], p[2], linear);
        }
        warp_winding_numbers<G>(s, q);
#pragma unroll
        for (int g = 0; g < G; ++g) where = lane == g ? (q.wn[g] != 0 ? 1 : 0) : where;
        if (mine.radius <= btol) where = 2;
    } else {
        Xoshiro rng(splitmix64(point_seed(seed, linear) ^ kInsideStream));
        const double bdist = __shfl_sync(0xffffffffu, mine.radius, 0);
        where = warp_classify_3d(s, w, p, bdist, btol, max_ray_attempts, rng, retries);
    }
    if (lane < G && t0 + lane < ps.n) {
        write_class<DIM>(t0 + lane, where, retries, mine, eq, out, location, start, ctr);
    }
}

// G points per warp (scenes whose FP32 bounds can steer FP64 queries).  A
// thread per point left the chip to a few warps of diverging FP64 traversals
// and a point's winding number to one lane.  ms, thread / warp: 48 points of a
// 256-segment star 0.036 / 0.011, 9177 of a blob of 3968 triangles 0.65 / 0.08
// (exact starts 2.58 / 0.11), 64^3 of a sphere of 16 128 triangles 3.2 / 2.2
// (exact starts 16.8 / 9.9: most of it the points on the sphere's symmetry
// planes, whose ties go through nearest64).
template <int DIM, int HC, int G>
__global__ void __launch_bounds__(kExactThreads)
    classify_warp_kernel(SceneView s, WideView w, PointSet ps, uint64_t seed, int max_ray_attempts,
                         double btol, double exact_below, float margin, EqDesc eq, Fields out,
                         uint8_t *location, StartRecord *start, DeviceCounters *ctr) {
    __shared__ int s_off[8];
    if (threadIdx.x < 8) s_off[threadIdx.x] = w.off[threadIdx.x];
    __syncthreads();
    w.off = s_off;
    const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
    for (long long t = warp * G; t < ps.n; t += warps * G) {
        classify_points_warp<DIM, HC, G>(s, w, ps, t, seed, max_ray_attempts, btol, exact_below,
                                         margin, eq, out, location, start, ctr);
    }
}

// Classification of a batch: global point g in [base, base + n) belongs to
// the item with the largest point_begin <= g.  One warp per point, as in a
// lone solve (items[i].exact_below >= 0: FastStart), or one lane where the
// item's scene asks for per-thread queries.
template <int DIM>
__global__ void __launch_bounds__(kExactThreads)
    classify_batch_kernel(const BatchItem *__restrict__ items, int n_items, long long base,
                          long long n) {
    const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
    for (long long t = warp; t < n; t += warps) {
        const long long g = base + t;
        int lo = 0, hi = n_items - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (items[mid].point_begin <= g) lo = mid;
            else hi = mid - 1;
        }
        const BatchItem &it = items[lo];
        const long long pt = g - it.point_begin;
        auto *location = const_cast<uint8_t *>(it.a.location);
        auto *start = const_cast<StartRecord *>(it.a.start);
        if (it.a.w.margin64 >= 0.0f) {
            classify_points_warp<DIM, kHeightAny, 1>(it.a.s, it.a.w, it.a.ps, pt, it.a.seed,
                                                     it.max_ray_attempts, it.btol,
                                                     it.exact_below, it.start_margin, it.eq,
                                                     it.out, location, start, it.a.ctr);
            continue;
        }
        double x, y, z;
        uint64_t linear;
        point_at(it.a.ps, pt, x, y, z, linear);
        const float bound = start_bounds<DIM, kHeightAny>(
            (threadIdx.x & 31) == 0 && it.exact_below >= 0.0, x, y, z,
            [&](int) -> const WideView & { return it.a.w; }, [&](int) { return it.start_margin; });
        if ((threadIdx.x & 31) == 0) {
            classify_point<DIM>(it.a.s, it.a.ps, pt, it.a.seed, it.max_ray_attempts, it.btol,
                                it.eq, it.out, location, start, it.a.ctr,
                                static_cast<double>(bound), it.exact_below);
        }
        __syncwarp();
    }
}

// Stands in for source draws that were taken from the stream beforehand and
// whose sample has no effect (3D sources are zero).
struct SkippedDraws {
    __device__ __forceinline__ double unit() { return 0.5; }
    __device__ __forceinline__ double unit_open() { return 0.5; }
};

// Takes one step's draws from a point's walk stream: in 3D, where one stream
// serves both, the source sample's first (six for a Green sample, three for a
// uniform one), then the direction's.
template <int DIM, class Eq>
__device__ __forceinline__ void step_draws(const Eq &eq, Xoshiro &rng, double &u, double &v) {
    if constexpr (DIM == 3 && Eq::kSource) {
        if (eq.mode == kGreen) {
            for (int k = 0; k < 4; ++k) rng.unit_open();
            rng.unit();
            rng.unit();
        } else {
            rng.unit();
            rng.unit();
            rng.unit_open();
        }
    }
    direction_draws<DIM>(rng, u, v);
}

// The walks of one point, one step of the current walk at a time.  A point's
// walks run one after another on its streams (where a walk's draws begin
// depends on every walk before it), so the point is the unit of parallel work.
template <int DIM, class Eq>
struct PlainWalks {
    V3<double> x0, p, np;
    double R0, R, sample, weight;
    double mean, m2, total_steps;
    unsigned long long steps_sum;
    long long t;
    int bid, i, steps, hits;
    bool overflow;
    Xoshiro walk, src;

    __device__ PlainWalks(const PointSet &ps, long long point, uint64_t seed,
                          const StartRecord *__restrict__ start)
        : walk(0), src(0) {
        t = point;
        uint64_t linear;
        point_at(ps, t, x0.x, x0.y, x0.z, linear);
        const uint64_t pseed = point_seed(seed, linear);
        walk = Xoshiro(splitmix64(pseed ^ kWalkStream));
        src = Xoshiro(DIM == 2 ? splitmix64(pseed ^ kSourceStream) : 0ull);
        R0 = start[t].radius;
        mean = m2 = total_steps = 0.0;
        steps_sum = 0;
        i = hits = 0;
        overflow = false;
        begin();
    }

    // wos_sample, include/wos/wos.hpp:54-138
    __device__ __forceinline__ void begin() {
        p = x0;
        R = R0;
        sample = 0.0;
        weight = 1.0;
        steps = 0;
    }
    __device__ __forceinline__ bool stepping(double eps, int max_steps) const {
        return R > eps && steps < max_steps;
    }
    // A step whose direction was drawn ahead (draw_ahead); in 3D the source
    // sample, whose draws were skipped then, is that of a zero source.
    __device__ __forceinline__ void step(const Eq &eq, const Direction &d) {
        if constexpr (DIM == 2) {
            p = walk_body<2, true, double>(eq, p, R, sample, weight, d, src, overflow);
        } else {
            SkippedDraws none;
            p = walk_body<3, true, double>(eq, p, R, sample, weight, d, none, overflow);
        }
        ++steps;
    }
    __device__ __forceinline__ void step(const Eq &eq) {
        if (DIM == 2) {
            p = walk_body<2, true, double>(eq, p, R, sample, weight, walk, src, overflow);
        } else {
            p = walk_body<3, true, double>(eq, p, R, sample, weight, walk, walk, overflow);
        }
        ++steps;
    }
    // The walk ends at its last nearest point (the start's, after no step).
    __device__ __forceinline__ void end(const Eq &eq, double eps,
                                        const StartRecord *__restrict__ start) {
        if (steps == 0) {
            np = V3<double>{start[t].nx, start[t].ny, start[t].nz};
            bid = start[t].boundary_id;
        }
        if (R > eps) ++hits;
        sample += weight * eq.boundary(np, bid);
        // Welford update, include/wos/wos.hpp:169-180
        const double count = static_cast<double>(i + 1);
        const double before = sample - mean;
        mean += before / count;
        const double after = sample - mean;
        m2 += before * after;
        total_steps += steps;
        steps_sum += static_cast<unsigned long long>(steps);
        ++i;
    }
    __device__ void write(int n_walks, const Fields &out, DeviceCounters *ctr) const {
        const double variance = n_walks > 1 ? m2 / static_cast<double>(n_walks - 1) : 0.0;
        const double se = n_walks > 0 ? sqrt(variance / static_cast<double>(n_walks)) : 0.0;
        const double mean_steps = n_walks > 0 ? total_steps / static_cast<double>(n_walks) : 0.0;
        if (out.mean) out.mean[t] = mean;
        if (out.variance) out.variance[t] = variance;
        if (out.standard_error) out.standard_error[t] = se;
        if (out.mean_steps) out.mean_steps[t] = mean_steps;
        if (hits) atomicAdd(&ctr->max_steps_hits, static_cast<unsigned long long>(hits));
        atomicAdd(&ctr->total_steps, steps_sum);
        atomicAdd(&ctr->exact_queries, steps_sum);  // one FP64 BVH query per step
        atomicAdd(&ctr->total_walks, static_cast<unsigned long long>(n_walks));
        if (overflow) atomicOr(&ctr->error_flags, kErrRejectionCap);
    }
};

// One thread per point, each with its own FP64 tree queries: the form for
// scenes whose FP32 bounds cannot steer a query (wide64_usable).
template <int DIM, class Eq>
__global__ void __launch_bounds__(kExactThreads)
    walk_plain_kernel(SceneView s, PointSet ps, uint64_t seed, Eq eq, int n_walks, double eps,
                      int max_steps, const uint8_t *__restrict__ location,
                      const StartRecord *__restrict__ start, Fields out, DeviceCounters *ctr) {
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < ps.n;
         t += stride) {
        if (location[t] != 1) continue;
        PlainWalks<DIM, Eq> k(ps, t, seed, start);
        while (k.i < n_walks) {
            k.begin();
            while (k.stepping(eps, max_steps)) {
                k.step(eq);
                const Nearest<double> q = nearest64<DIM>(s, k.p.x, k.p.y, k.p.z, dinf());
                k.R = sqrt(q.best);
                k.np = V3<double>{q.x, q.y, q.z};
                if (DIM == 2) k.bid = q.slot >= 0 ? s.segid[q.slot].x : -1;
            }
            k.end(eq, eps, start);
        }
        k.write(n_walks, out, ctr);
    }
}

// `per_warp` consecutive points per warp, each owned by the first lane of its
// group of 32 / per_warp lanes.  Every iteration steps each point's walk and
// the whole warp then answers the points' queries one after another
// (warp_candidates64).  A point's walks are serial, so the kernel waits on one
// step's chain (draw, sine and cosine, query, square root) rather than on issue
// slots.  Per-thread queries made that chain 30 dependent tree nodes long in 32
// diverging lanes.  The draws do not depend on the walk, so a group takes its
// point's next draws together, one step's per lane, and forms all their sines
// and cosines at once (each lane keeps the stream and picks its own draws).
// 1360 inside points of an annulus of 256 segments, 1000 walks: 144.8 ms by
// threads, 10.4 by warps, 8.6 ms with directions drawn ahead; 0.41 M walks in a
// blob of 3968 triangles 425, 9.4 and 8.9 ms (same results, bit for bit).
template <int DIM, class Eq>
__global__ void __launch_bounds__(kExactThreads, 4)
    walk_plain_warp_kernel(SceneView s, WideView w, int per_warp, PointSet ps, uint64_t seed,
                           Eq eq, int n_walks, double eps, int max_steps,
                           const uint8_t *__restrict__ location,
                           const StartRecord *__restrict__ start, Fields out,
                           DeviceCounters *ctr) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ int s_off[8];
    if (threadIdx.x < 8) s_off[threadIdx.x] = w.off[threadIdx.x];
    __syncthreads();
    w.off = s_off;
    const int lane = threadIdx.x & 31;
    const int group = 32 / per_warp, sub = lane % group;
    const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long long t = warp * per_warp + lane / group;
    const bool mine = t < ps.n && location[t] == 1;  // the group has a point to walk
    bool active = mine && sub == 0;
    if (!__any_sync(kAll, active)) return;
    PlainWalks<DIM, Eq> k(ps, mine ? t : 0, seed, start);
    Direction ahead{0.0, 0.0, 0.0, 0.0};  // the group's step `used` + sub
    int used = group;                     // directions of the batch taken so far
    while (__any_sync(kAll, active)) {
        const bool query = active && k.stepping(eps, max_steps);
        // groups whose batch is used up draw the next one
        const bool refill =
            __shfl_sync(kAll, static_cast<int>(query && used == group), lane - sub) != 0;
        if (__any_sync(kAll, refill)) {
            if (refill) {
                double u = 0.0, v = 0.0;
                for (int i = 0; i < group; ++i) {
                    double ui, vi;
                    step_draws<DIM>(eq, k.walk, ui, vi);
                    if (i == sub) {
                        u = ui;
                        v = vi;
                    }
                }
                ahead = direction_of<DIM>(u, v);
                used = 0;
            }
            __syncwarp();
        }
        const int from = lane - sub + (query ? used : 0);
        Direction d;
        d.c = __shfl_sync(kAll, ahead.c, from);
        d.s = __shfl_sync(kAll, ahead.s, from);
        d.r = DIM == 3 ? __shfl_sync(kAll, ahead.r, from) : 1.0;
        d.z = DIM == 3 ? __shfl_sync(kAll, ahead.z, from) : 0.0;
        if (query) {
            k.step(eq, d);
            ++used;
        }
        unsigned pending = __ballot_sync(kAll, query);
        Candidates cand{0, -1};
        while (pending) {
            const int j = __ffs(pending) - 1;
            pending &= pending - 1u;
            const double qx = __shfl_sync(kAll, k.p.x, j), qy = __shfl_sync(kAll, k.p.y, j);
            const double qz = DIM == 3 ? __shfl_sync(kAll, k.p.z, j) : 0.0;
            const Candidates c = warp_candidates64<DIM>(s, w, qx, qy, qz);
            if (lane == j) cand = c;
        }
        if (query) {
            int slot;
            k.R = sqrt(pick_nearest64<DIM>(s, w.margin64, cand, k.p.x, k.p.y, k.p.z, slot, k.np.x,
                                           k.np.y, k.np.z));
            if (DIM == 2) k.bid = slot >= 0 ? s.segid[slot].x : -1;
        }
        if (active && !k.stepping(eps, max_steps)) {
            k.end(eq, eps, start);
            if (k.i < n_walks) {
                k.begin();
            } else {
                active = false;
                k.write(n_walks, out, ctr);
            }
        }
    }
}

__global__ void prng_kernel(const uint64_t *seeds, long long n, int count, uint64_t *out) {
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < n;
         t += stride) {
        Xoshiro rng(seeds[t]);
        for (int i = 0; i < count; ++i) out[t * count + i] = rng.u64();
    }
}

template <int DIM>
__global__ void closest64_kernel(SceneView s, const double *pts, long long n, double *dist,
                                 double *nearest, int *bid) {
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < n;
         t += stride) {
        const double px = pts[DIM * t], py = pts[DIM * t + 1];
        const double pz = DIM == 3 ? pts[DIM * t + 2] : 0.0;
        const Nearest<double> q = nearest64<DIM>(s, px, py, pz, dinf());
        dist[t] = sqrt(q.best);
        nearest[DIM * t] = q.x;
        nearest[DIM * t + 1] = q.y;
        if (DIM == 3) nearest[DIM * t + 2] = q.z;
        if (bid) bid[t] = (DIM == 2 && q.slot >= 0) ? s.segid[q.slot].x : -1;
    }
}

int blocks_for(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > (1ll << 30)) b = 1ll << 30;
    return static_cast<int>(b);
}

// Points per warp of walk_plain_warp_kernel.  A warp answers its lanes'
// queries in turn, so few points per warp give short steps, and many share
// the cost of the step's arithmetic (one instruction stream for all lanes).
// Measured on a B200, walk kernel in ms at 1 / 2 / 4 / 8 points per warp: 2D
// circle of 1024 segments, 64 walks: 32^2 points 0.69 / 0.94 / 1.47 / 2.33; 64^2
// 1.19 / 1.05 / 1.58 / 2.50; 128^2 3.46 / 2.86 / 2.99 / 2.86; 256^2 12.8 / 10.1 /
// 8.71 / 7.89.  3D sphere of 16 128 triangles, 16 walks (queries dominate the
// step): 24^3 3.08 / 3.10 / 3.08 / 5.06; 40^3 12.2 / 10.9 / 10.6 / 11.7.
int points_per_warp(int dim, long long n) {
    if (dim == 3) return n >= 32768 ? 2 : 1;
    int p = 1;
    while (p < 8 && n / (2 * p) >= 2048) p *= 2;
    return p;
}

template <int DIM, class Eq>
void launch_plain_typed(const SceneView &s, const WideView &w, const PointSet &ps, uint64_t seed,
                        const Eq &eq, int n_walks, double eps, int max_steps, const uint8_t *location,
                        const StartRecord *start, Fields out, DeviceCounters *ctr,
                        cudaStream_t stream) {
    if (w.margin64 >= 0.0f) {
        const int per_warp = points_per_warp(DIM, ps.n);
        const long long warps = (ps.n + per_warp - 1) / per_warp;
        walk_plain_warp_kernel<DIM, Eq>
            <<<blocks_for(32 * warps, kExactThreads), kExactThreads, 0, stream>>>(
                s, w, per_warp, ps, seed, eq, n_walks, eps, max_steps, location, start, out, ctr);
        return;
    }
    walk_plain_kernel<DIM, Eq><<<blocks_for(ps.n, kExactThreads), kExactThreads, 0, stream>>>(
        s, ps, seed, eq, n_walks, eps, max_steps, location, start, out, ctr);
}

template <int DIM>
void launch_plain_dim(const SceneView &s, const WideView &w, const PointSet &ps, uint64_t seed,
                      EqDesc e, int n_walks, double eps, int max_steps, const uint8_t *location,
                      const StartRecord *start, Fields out, DeviceCounters *ctr,
                      cudaStream_t stream) {
    switch (e.kind) {
        case kLaplace:
            launch_plain_typed<DIM>(s, w, ps, seed, Laplace<DIM>{}, n_walks, eps, max_steps,
                                    location, start, out, ctr, stream);
            break;
        case kPoisson:
            launch_plain_typed<DIM>(s, w, ps, seed, Poisson<DIM>{e.mode, e.alpha}, n_walks, eps,
                                    max_steps, location, start, out, ctr, stream);
            break;
        case kScreened:
            launch_plain_typed<DIM>(s, w, ps, seed, Screened<DIM>{e.mode, e.alpha}, n_walks, eps,
                                    max_steps, location, start, out, ctr, stream);
            break;
        case kTransient:
            if (DIM == 2) {
                launch_plain_typed<2>(s, w, ps, seed, Transient<2>{kGreen, e.alpha, e.tr}, n_walks,
                                      eps, max_steps, location, start, out, ctr, stream);
            }
            break;
        case kPlate:
            if (DIM == 2) {
                launch_plain_typed<2>(s, w, ps, seed, Plate<2>{e.mode, *e.pl}, n_walks, eps,
                                      max_steps, location, start, out, ctr, stream);
            }
            break;
        default:
            launch_plain_typed<DIM>(s, w, ps, seed, Helmholtz<DIM>{}, n_walks, eps, max_steps,
                                    location, start, out, ctr, stream);
            break;
    }
}

}  // namespace

cudaError_t launch_classify(const SceneView &s, const WideView &wide, const PointSet &ps,
                            uint64_t seed, int max_ray_attempts, double btol, EqDesc eq,
                            Fields out, uint8_t *location, StartRecord *start,
                            DeviceCounters *counters, cudaStream_t stream,
                            const FastStart &fast) {
    if (ps.n <= 0) return cudaSuccess;
    const int blocks = blocks_for(ps.n, kExactThreads);
    if (wide.margin64 >= 0.0f) {
        // 2D: eight points per warp share the segments' loads when that still
        // gives every scheduler several warps (disk of 1024 segments, 256^2
        // points: 0.158 ms at 1, 0.101 at 8, 0.118 by threads)
        const int group = s.dim == 2 && ps.n >= 8 * 148 * 16 ? 8 : 1;
        const long long warps = (ps.n + group - 1) / group;
        const int b = blocks_for(std::min<long long>(32 * warps, 32ll * 148 * 64), kExactThreads);
        const double below = fast.on ? fast.exact_below : -1.0;
        // 2D: one kernel for all heights (256^2 points of a 256-segment star 0.069
        // ms with a class each, 0.071); 3D: 64^3 of a sphere of 16 128 triangles
        // 2.01 with, 2.26 without
        if (s.dim == 2) {
            auto k = group == 8 ? classify_warp_kernel<2, kHeightAny, 8>
                                : classify_warp_kernel<2, kHeightAny, 1>;
            k<<<b, kExactThreads, 0, stream>>>(s, wide, ps, seed, max_ray_attempts, btol, below,
                                               fast.margin, eq, out, location, start, counters);
            return cudaGetLastError();
        }
        return with_height_class(height_class(wide.H), [&](auto h) -> cudaError_t {
            constexpr int HC = decltype(h)::value;
            classify_warp_kernel<3, HC, 1><<<b, kExactThreads, 0, stream>>>(
                s, wide, ps, seed, max_ray_attempts, btol, below, fast.margin, eq, out, location,
                start, counters);
            return cudaGetLastError();
        });
    }
    if (fast.on && fast.w.n > 0) {
        auto k = s.dim == 2 ? classify_fast_kernel<2> : classify_fast_kernel<3>;
        k<<<blocks, kExactThreads, 0, stream>>>(s, fast.w, ps, seed, max_ray_attempts, btol,
                                                fast.exact_below, fast.margin, eq, out, location,
                                                start, counters);
        return cudaGetLastError();
    }
    if (s.dim == 2) {
        classify_kernel<2><<<blocks, kExactThreads, 0, stream>>>(s, ps, seed, max_ray_attempts,
                                                                 btol, eq, out, location, start,
                                                                 counters);
    } else {
        classify_kernel<3><<<blocks, kExactThreads, 0, stream>>>(s, ps, seed, max_ray_attempts,
                                                                 btol, eq, out, location, start,
                                                                 counters);
    }
    return cudaGetLastError();
}

cudaError_t launch_classify_batch(int dim, const BatchItem *items, int n_items,
                                  long long point_base, long long n_points, cudaStream_t stream) {
    if (n_items <= 0 || n_points <= 0) return cudaSuccess;
    // a warp per point
    long long b = (n_points + 3) / 4;
    if (b > 148 * 64) b = 148 * 64;
    if (dim == 2) {
        classify_batch_kernel<2><<<static_cast<int>(b), kExactThreads, 0, stream>>>(
            items, n_items, point_base, n_points);
    } else {
        classify_batch_kernel<3><<<static_cast<int>(b), kExactThreads, 0, stream>>>(
            items, n_items, point_base, n_points);
    }
    return cudaGetLastError();
}

cudaError_t launch_walk_plain(const SceneView &s, const WideView &w, const PointSet &ps,
                              uint64_t seed, EqDesc eq, int n_walks, double eps, int max_steps,
                              const uint8_t *location, const StartRecord *start, Fields out,
                              DeviceCounters *counters, cudaStream_t stream) {
    if (ps.n <= 0) return cudaSuccess;
    if (s.dim == 2) {
        launch_plain_dim<2>(s, w, ps, seed, eq, n_walks, eps, max_steps, location, start, out,
                            counters, stream);
    } else {
        launch_plain_dim<3>(s, w, ps, seed, eq, n_walks, eps, max_steps, location, start, out,
                            counters, stream);
    }
    return cudaGetLastError();
}

namespace {
__global__ void special64_kernel(const double *x, long long n, double *li0, double *lk0) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    li0[i] = log_i0(x[i]);
    lk0[i] = log_k0(x[i]);
}
}  // namespace

cudaError_t launch_special64(const double *x, long long n, double *log_i0, double *log_k0,
                             cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    special64_kernel<<<blocks_for(n, 128), 128, 0, stream>>>(x, n, log_i0, log_k0);
    return cudaGetLastError();
}

cudaError_t launch_prng(const uint64_t *seeds, long long n, int count, uint64_t *out,
                        cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    prng_kernel<<<blocks_for(n, 128), 128, 0, stream>>>(seeds, n, count, out);
    return cudaGetLastError();
}

cudaError_t launch_closest64(const SceneView &s, const double *pts, long long n, double *dist,
                             double *nearest, int *bid, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    if (s.dim == 2) {
        closest64_kernel<2><<<blocks_for(n, 128), 128, 0, stream>>>(s, pts, n, dist, nearest, bid);
    } else {
        closest64_kernel<3><<<blocks_for(n, 128), 128, 0, stream>>>(s, pts, n, dist, nearest, bid);
    }
    return cudaGetLastError();
}

}  // namespace wosb
