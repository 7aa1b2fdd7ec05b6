// mrt_gridwalk.cuh - persistent closest-hit and any-hit engines for the RegularGrid
// (RegularGrid.hpp:157-465).
//
// grid_trace() walks one ray from its first cell to its last in one thread, so a warp waits for
// its longest walk (a camera ray that leaves the grid after a few cells shares the warp with one
// that crosses the dense soup for a hundred).  Here every lane keeps a resumable walk and the warp
// loops:
//   1. refill: idle lanes take new work items from a global counter (one atomicAdd per warp);
//   2. advance: lanes without a reference to test step from cell to cell until most have one;
//   3. test: lanes with references test them until most have none;
//   4. completion: the area lights (Scene::traceLights, after the accelerators) and the work item's
//      finish(), which may start the item's next ray in the same lane.
// Every ray takes grid_trace's steps in grid_trace's order and meets the references in that order, so
// the answer is the reference's bit for bit.  Two kinds of work whose outcome is known are left out:
//   * Tests.  A triangle is listed in every cell it may touch and in the next one along each axis (nine
//     references a triangle on the 1,000,000-triangle soup).  A walk has tested the whole list of the cell
//     it comes from, and a triangle that failed there fails again: its test does not depend on the cell,
//     and the length it is held against only shrinks.  So is the second look at a cell that the
//     reference's testloop begins with.  The build marks such references per direction of the step (skip
//     bits), and the lane goes past them without reading the triangle.  A distance that is not a number
//     breaks the argument (it passes any length test, and any length passes a test against it): from the
//     first such distance on, the ray's walk tests everything as the reference does.
//   * Cell records.  An empty cell's record says how many steps further every cell is empty (up to
//     kEmptyReach); those steps read nothing.
// On the 1080p frame of the soup at G = 128 a camera ray steps through 152 cells, 134 of them empty, and
// meets 159 references, 79 of which are left to test.  Bound by the lanes' differing walks (11.8 of 32
// active) and the latency of the triangle records; 6.48 -> 3.51 ms a frame, the any-hit rays above
// 0.93 -> 0.59 ms (one ray a thread before).
#pragma once

#include "mrt_persistent.cuh"

namespace mrt {

// resident blocks of 128 threads per SM for the kernels of the persistent grid walk (the 1080p soup frame:
// 8 blocks, 64 registers 3.58 ms, 7 blocks 3.92 ms; any-hit rays: the same at 8, 10 and 12)
constexpr int kGridBlocksPerSm = 8;

// flags: bits 0-1 the phase (1 first walk, 2 testloop, 0 finished), bits 8-15 the steps that are known to
// come to empty cells, bits kSkipShift.. the ray's skip bits, one for each axis (none: a distance was not a
// number, or the references carry no skip bits).
struct GridWalk {
    float tx, ty, tz, dx, dy, dz;   // as Dda
    int32_t sx, sy, sz;             // change of the record index by a step
    uint32_t c;                     // record of the cell
    uint32_t flags;
    uint32_t skip;                  // skip bit of the step that led to the cell (0: test everything)
    float len;
    uint32_t id;
    uint32_t k, e;                  // the cell's references: next to test, end
};
constexpr uint32_t kWalkPhase = 3u, kWalkReach = 0xFF00u, kWalkSkip = ~0u << kSkipShift;

__device__ __forceinline__ bool grid_walking(const GridWalk &w) { return (w.flags & kWalkPhase) != 0u; }

// the current cell's references; the walk ends on the border
__device__ __forceinline__ void grid_walk_load(const DevGrid &g, GridWalk &w) {
    const uint2 r = __ldg(&g.cells[w.c]);
    w.k = r.x;
    w.e = r.y;
    if (r.x == kEmptyCell) {
        w.e = 0u;   // (k >= e: nothing to test)
        w.flags = r.y ? w.flags + ((r.y - 1u) << 8) : w.flags & ~kWalkPhase;
    }
}

__device__ __forceinline__ void grid_walk_setup(const DevGrid &g, const Ray &r, GridWalk &w) {
    Dda st;
    dda_setup(g, r, st);
    w.tx = st.tx; w.ty = st.ty; w.tz = st.tz;
    w.dx = st.dx; w.dy = st.dy; w.dz = st.dz;
    w.sx = st.sx;
    w.sy = st.sy * (g.G + 2);
    w.sz = st.sz * (g.G + 2) * (g.G + 2);
    if (w.flags & kWalkSkip)
        w.flags = (st.sx < 0 ? 2u : 1u) << kSkipShift | (st.sy < 0 ? 8u : 4u) << kSkipShift | (st.sz < 0 ? 32u : 16u) << kSkipShift;
    w.flags |= 1u;
    w.skip = 0u;
    w.c = grid_cell(g, st.X, st.Y, st.Z);
    grid_walk_load(g, w);
}

// A, AB, AC of triangle i from the grid's packed records
__device__ __forceinline__ void grid_tri_load(const DevGrid &g, uint32_t i, V3 &a, V3 &ab, V3 &ac) {
    const float *rec = g.trec + 16 * (size_t)i;
    uint4 p0, p1;
    ldg_32b(reinterpret_cast<const uint4 *>(rec), p0, p1);
    const float acz = __ldg(rec + 8);
    a = V3{__uint_as_float(p0.x), __uint_as_float(p0.y), __uint_as_float(p0.z)};
    ab = V3{__uint_as_float(p0.w), __uint_as_float(p1.x), __uint_as_float(p1.y)};
    ac = V3{__uint_as_float(p1.z), __uint_as_float(p1.w), acz};
}

// Certain to fail tri_test's (and tri_occ's) test of u = (1 / np) q, found without the division: u is off
// q / np by at most 2^-23 of its value, so it is above 1 where |q| > 1.000001 |np| (or below 0 with the
// signs apart), and below 0, not -0, where the signs differ and neither factor is near the ends of the
// range.  Most references that a walk tests end here.
__device__ __forceinline__ bool misses_u(const V3 &a, const V3 &ab, const V3 &ac, const Ray &r) {
    const V3 perp = cross(r.d, ac);
    const float np = dot(ab, perp), q = dot(r.o - a, perp);
    const float n = fabsf(np), m = fabsf(q);
    const bool apart = ((__float_as_uint(np) ^ __float_as_uint(q)) >> 31) != 0u;
    return n >= kEpsilon && n <= 1.0e10f && (m > n * 1.000001f || (apart && m >= 1.0e-30f));
}

// triangle i of the grid with the reference accept rule (triangle_hit), its edges from the grid's
// packed record when the build made them
__device__ __forceinline__ bool grid_tri_hit(const DevScene &s, const DevGrid &g, uint32_t i, const Ray &r, float &len,
                                             uint32_t &id) {
    if (!g.trec) return triangle_hit(s, i, r, len, id);
    const uint32_t self = hid(MRT_PRIM_TRIANGLE, i);
    if (r.exclude == self) return false;
    V3 a, ab, ac;
    grid_tri_load(g, i, a, ab, ac);
    if (misses_u(a, ab, ac, r)) return false;
    float t, u, v;
    if (!tri_test(a, ab, ac, r, t, u, v)) return false;
    if (t >= len) return false;
    len = t;
    id = self;
    return true;
}

__device__ __forceinline__ bool grid_tri_occ(const DevScene &s, const DevGrid &g, uint32_t i, const Ray &r, float dist) {
    if (!g.trec) return triangle_occ(s, i, r, dist);
    if (r.exclude == hid(MRT_PRIM_TRIANGLE, i)) return false;
    V3 a, ab, ac;
    grid_tri_load(g, i, a, ab, ac);
    return !misses_u(a, ab, ac, r) && tri_occ(a, ab, ac, r, dist);
}

// planes and spheres walk their own grids first (Shader.cpp:124-150), whole, in this lane
__device__ __forceinline__ void grid_walk_begin(const DevScene &s, const Ray &r, GridWalk &w) {
    w.len = kRayLengthMax;
    w.id = MRT_HIT_NONE;
    grid_trace<kPlane>(s, r, w.len, w.id);
    grid_trace<kSphere>(s, r, w.len, w.id);
    const DevGrid &g = s.grid[kTriangle];
    w.flags = (g.id_mask == 0xFFFFFFFFu || !(w.len == w.len)) ? 0u : kWalkSkip;
    w.k = w.e = 0u;
    if (g.has) grid_walk_setup(g, r, w);
}

// the move to the next cell (RegularGrid.hpp:251-279, 299-333): the testloop ends when the hit lies before
// the next cell boundary, either walk when the next cell is on the border.  (A walk takes at most 3 G steps.)
template <bool kTestloop>
__device__ __forceinline__ void grid_walk_step(const DevGrid &g, GridWalk &w) {
    const bool x = w.tx < w.ty && w.tx < w.tz, y = !(w.tx < w.ty) && w.ty < w.tz;
    if (kTestloop && (w.flags & 2u) && w.len < (x ? w.tx : y ? w.ty : w.tz)) { w.flags &= ~kWalkPhase; return; }
    w.c += (uint32_t)(x ? w.sx : y ? w.sy : w.sz);
    if (x) w.tx = w.tx + w.dx;
    else if (y) w.ty = w.ty + w.dy;
    else w.tz = w.tz + w.dz;
    if (w.flags & kWalkReach) { w.flags -= 0x100u; return; }
    w.skip = w.flags & ((x ? 3u : y ? 12u : 48u) << kSkipShift);
    grid_walk_load(g, w);
}

// the next reference of the cell that is not skipped; false when none is left
__device__ __forceinline__ bool grid_walk_ref(const DevGrid &g, GridWalk &w, uint32_t &i) {
    uint32_t ref;
    do { ref = __ldg(&g.refs[w.k++]); } while ((ref & w.skip) && w.k < w.e);
    i = ref & g.id_mask;
    return !(ref & w.skip);
}

__device__ __forceinline__ void grid_walk_test(const DevScene &s, const DevGrid &g, const Ray &r, GridWalk &w) {
    uint32_t i;
    if (!grid_walk_ref(g, w, i) || !grid_tri_hit(s, g, i, r, w.len, w.id)) return;
    const bool first = (w.flags & kWalkPhase) == 1u;
    w.flags = (w.flags & ~kWalkPhase) | 2u;
    if (!(w.len == w.len)) {
        w.flags &= ~kWalkSkip;
        w.skip = 0u;
        if (first) grid_walk_load(g, w);   // the testloop starts over this same cell
    }
}

// Votes of a warp: the advance phase ends when fewer than kGridAdvance lanes have to step while others
// wait, the test phase when fewer than kGridTest lanes have references while others wait (12 both; 4, 8, 16
// and 24 are slower); between two votes a lane takes up to so many steps and references.  Camera rays walk
// alike, so many are worth a vote: the 1080p soup frame takes 3.51 ms at 16 steps and 8 references, 3.58
// at 8 and 4, 3.77 at 4 and 2, 4.12 at 1 and 1.  Shadow rays in all directions do not: 300,007 any-hit rays
// in a soup of 100,003 take 0.59 ms at 1 and 1, 0.61 at 2 and 2, 0.64 at 4 and 2.
constexpr int kGridAdvance = 12, kGridTest = 12;
constexpr int kGridSteps = 16, kGridTests = 8, kGridAnySteps = 1, kGridAnyTests = 1;

// the advance and the test phase of a warp, at least one step of each
template <int kSteps, int kTests, class Step, class Test>
__device__ __forceinline__ void grid_phases(bool active, const GridWalk &w, Step step, Test test) {
    const uint32_t FULL = 0xFFFFFFFFu;
    for (;;) {
        bool go = active && grid_walking(w) && w.k >= w.e;
#pragma unroll 1
        for (int u = 0; go && u < kSteps; ++u) {
            step();
            go = grid_walking(w) && w.k >= w.e;
        }
        __syncwarp();
        const uint32_t m = __ballot_sync(FULL, go);
        if (m == 0u || (__popc(m) < kGridAdvance && __any_sync(FULL, active && !go))) break;
    }
    for (;;) {
        bool go = active && grid_walking(w) && w.k < w.e;
#pragma unroll 1
        for (int u = 0; go && u < kTests; ++u) {
            test();
            go = grid_walking(w) && w.k < w.e;
        }
        __syncwarp();
        const uint32_t m = __ballot_sync(FULL, go);
        if (m == 0u || (__popc(m) < kGridTest && __any_sync(FULL, active && !go))) break;
    }
}

// Work provides total(), counter(), begin(item, lane, r) and
// finish(lane, r, hit, t, id, const FastTrav &) -> true: r holds the item's next ray (as persistent_closest)
template <class Work, class Lane>
__device__ void persistent_grid_closest(const DevScene &s, Work &work, Lane &lane) {
    const uint32_t FULL = 0xFFFFFFFFu;
    const int lane_id = threadIdx.x & 31;
    const uint32_t total = work.total();
    bool active = false;
    bool exhausted = false;
    Ray r;
    GridWalk w;
    const FastTrav none{};
    for (;;) {
        const uint32_t idle = __ballot_sync(FULL, !active);
        if (!exhausted && (__popc(idle) >= 8 || idle == FULL)) {
            const int leader = __ffs(idle) - 1;
            uint32_t base = 0;
            if (lane_id == leader) base = atomicAdd(work.counter(), (uint32_t)__popc(idle));
            base = __shfl_sync(FULL, base, leader);
            if (base + (uint32_t)__popc(idle) >= total) exhausted = true;
            if (!active) {
                const uint32_t item = base + __popc(idle & ((1u << lane_id) - 1u));
                if (item < total && work.begin(item, lane, r)) {
                    grid_walk_begin(s, r, w);
                    active = true;
                }
            }
        }
        if (__ballot_sync(FULL, active) == 0) {
            if (exhausted) break;
            continue;
        }
        grid_phases<kGridSteps, kGridTests>(active, w, [&] { grid_walk_step<true>(s.grid[kTriangle], w); },
                    [&] { grid_walk_test(s, s.grid[kTriangle], r, w); });
        if (active && !grid_walking(w)) {
            lights_trace(s, r, w.len, w.id);
            // an accepted plane, sphere, triangle or light leaves its id
            if (work.finish(lane, r, w.id != MRT_HIT_NONE, w.len, w.id, none)) grid_walk_begin(s, r, w);
            else active = false;
        }
    }
}

// any-hit (RegularGrid.hpp:341-465): planes and spheres in order, then the triangle grid; the first
// occluder ends the ray.  Work provides total(), counter(), begin(item, lane, r, dist) and
// finish(lane, occluded) (as persistent_any).
template <class Work, class Lane>
__device__ void persistent_grid_any(const DevScene &s, Work &work, Lane &lane) {
    const uint32_t FULL = 0xFFFFFFFFu;
    const int lane_id = threadIdx.x & 31;
    const uint32_t total = work.total();
    const DevGrid &g = s.grid[kTriangle];
    bool active = false, exhausted = false, occluded = false;
    Ray r;
    GridWalk w;
    float dist = 0.0f;
    for (;;) {
        const uint32_t idle = __ballot_sync(FULL, !active);
        if (!exhausted && (__popc(idle) >= 8 || idle == FULL)) {
            const int leader = __ffs(idle) - 1;
            uint32_t base = 0;
            if (lane_id == leader) base = atomicAdd(work.counter(), (uint32_t)__popc(idle));
            base = __shfl_sync(FULL, base, leader);
            if (base + (uint32_t)__popc(idle) >= total) exhausted = true;
            if (!active) {
                const uint32_t item = base + __popc(idle & ((1u << lane_id) - 1u));
                if (item < total && work.begin(item, lane, r, dist)) {
                    active = true;
                    occluded = grid_occ<kPlane>(s, r, dist) || grid_occ<kSphere>(s, r, dist);
                    w.flags = g.id_mask == 0xFFFFFFFFu ? 0u : kWalkSkip;
                    w.k = w.e = 0u;
                    if (!occluded && g.has) grid_walk_setup(g, r, w);
                }
            }
        }
        if (__ballot_sync(FULL, active) == 0) {
            if (exhausted) break;
            continue;
        }
        grid_phases<kGridAnySteps, kGridAnyTests>(active, w, [&] { grid_walk_step<false>(g, w); },
                    [&] {
                        uint32_t i;
                        if (grid_walk_ref(g, w, i) && grid_tri_occ(s, g, i, r, dist)) { occluded = true; w.flags &= ~kWalkPhase; }
                    });
        if (active && !grid_walking(w)) {
            work.finish(lane, occluded);
            active = false;
        }
    }
}

}  // namespace mrt
