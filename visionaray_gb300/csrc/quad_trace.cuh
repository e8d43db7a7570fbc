// Warp-stepped traversal of the quad nodes (bvh_layout.cuh, quads.cu), shared by the ray
// queries (traverse.cu) and the path tracer (pathtrace.cu).
//
// What bounded the node-pair loop (traverse_core.cuh): a warp of incoherent rays ran it
// with 7.9 of 32 lanes active, since lanes that reach a leaf wait for the lanes still
// descending and ended rays wait for the warp's longest one, and its 64-byte node fetches
// kept the load/store pipe 62 % busy (two wavefronts per lane and visit).  Here
//   - a node visit tests four descendants out of one 64-byte record, so a ray takes half
//     the visits (and half the wavefronts);
//   - every round runs the leaf tests of the lanes that stand at a leaf, then advances each
//     busy lane by two or three nodes, so no lane waits for a whole descent;
//   - a warp refills its idle lanes from its rays, and takes more of them when they run out.
// Measured, heightfield 2048^2 with 4,194,304 sorted secondary rays: 19 lanes active, the
// query 3.36 -> 1.78 ms; 8.4 M ambient-occlusion rays over 1024^2: 3.63 -> 2.15 ms.  What
// bounds it now (a bounce of a 1920 x 1080 path-traced frame): the load/store pipe's
// wavefronts (80 %), two per lane and node, then issue slots (72 %).
//
// The answers are the node-pair loop's, bit for bit but for one case, although the visits
// differ:
//   - Boxes only get larger (quantised outward, and the distances below carry a margin
//     for every rounding), so each leaf whose own box the pair loop's slab test accepts is
//     reached, and triangles are tested with the same arithmetic.
//   - The pair loop returns some triangle T that hits within [tmin, tmax] and whose leaf
//     box the ray hits (the boxes of a tree are nested and the slab test is monotone, so
//     an accepted leaf box implies accepted ancestors).  Among those let T* be the one of
//     smallest t.  The pair loop can return another one only if it dropped T* for a triangle
//     with t <= the entry distance of T*'s leaf box, or met an equal t first.  So if no
//     other hit has t <= max(t*, entry distance of T*'s leaf box), T* is its answer;
//     otherwise (a ray through a shared edge, coincident triangles) the ray is traced
//     again by the pair loop.  Nodes are culled 1/256 beyond the best t, so such a second
//     hit is met whatever the order, unless its t is off by more than that from where its
//     own box begins: a triangle seen edge-on, whose t is made of rounding errors.  A ray
//     that tested such a triangle (kQuadEdgeOn), as one in the plane of a surface does, is
//     not culled by its best t from there on.  The case that is left: an edge-on triangle
//     beyond the culling distance of an ordinary hit that was found before any other edge-on
//     one, with a computed t in front of that hit.  The pair loop reports it or not, as its
//     own order falls.
//   - Any hit, unordered: the pair loop reports the first hit of a depth-first walk in
//     child order, and the quads' slots are in that order.  Any hit, near first (shadow
//     rays): only whether there is a hit is used.
//   - A ray with non-finite or extreme components, and one whose walk needs more than the
//     shared stack, is traced by the pair loop too.
#pragma once

#include "traverse_core.cuh"

namespace gbrt {

// Threads of a block and shared stack entries per thread of every kernel that runs
// quad_trace: 32 x 128 x 4 B = 16 KB per block.  A visit pushes up to three entries; 16
// entries sent 125 of the 4.2 M heightfield rays to the pair loop, 24 none, but a path
// tracer's long tails wait for such rays (high-definition frame 60.2 ms at 20 entries, 49.7
// at 24, 49.0 at 32).
constexpr int kQuadBlock = 128;
constexpr int kQuadStack = 32;
// Resident blocks the register allocation must allow: 9 (36 warps, 56 registers, no
// spills).  Heightfield closest hit 1.79 ms; 1.86 at 8 blocks; with fixed spans 2.10, 2.18 at
// 10 blocks (48 registers, spilling).
constexpr int kQuadMinBlocks = 9;
// Idle lanes of a warp that trigger a refill (6 and 11 within 1 %, 4 up to 3 % slower).
constexpr int kQuadRefill = 8;
// Node steps per round, after the leaf tests of the lanes that stand at one (waiting for
// several such lanes costs more than it saves: any 44.4 ms per high-definition frame, two
// 44.6, three 44.9).  Ray queries take three (heightfield closest hit 1.84 ms at two, 1.79 at
// three, 1.78 at four; 8.4 M ambient-occlusion rays 2.20, 2.16, 2.18), the path tracer two
// (three: high-definition frame 41.4 -> 41.5 ms, forward and backward 31.4 -> 32.2, batch of
// scenes 7.72 -> 7.63).
constexpr int kQuadQuerySteps = 3;
constexpr int kQuadPathSteps = 2;
// A triangle is edge-on to a ray if its determinant, other than 0 (no hit), is at most this
// times the largest components of the direction and the two edges.  Answers that differed
// from the pair loop's in a restatement of both on the CPU, 34 million rays in planes turned
// against the axes with vertices 0 to 3e-6 off them: 6,360 without the rule, 2 at 2^-13, 0
// at 2^-11.  Rays that are not culled for it at 2^-13: 1e-4 to 4e-4 of them (heightfield, box
// and random triangles), 2 to 4 % of the time of
// closest-hit queries with the tests themselves (1.4 %).
constexpr float kQuadEdgeOn = 1.220703125e-4f;   // 2^-13
// Added to best_tri (-1 for none yet) of such a ray: triangles are below 2^29 + 1.
constexpr int kQuadOpen = 1 << 30;

// Rays per warp for n rays on a GPU that holds `resident` warps of the kernel (5,472 on 152
// SMs).  As many warps as rays while they fit: a warp's time is its slowest chain of
// dependent node loads, and rays of other warps do not lengthen it (4,096 camera rays over
// 65,536 triangles 65 us one per warp, 87 us four per warp).  Beyond that, lanes that
// advance together pay more than warps (16,384 rays: 88 us sixteen per warp, 100 three per
// warp; 65,536: 104 us 32 per warp, 132 twelve): about 3/4 of the resident warps, at least
// half to fully occupied ones.  Where no counter is there to share long queries by
// (quad_share), they go in up to 2 1/4 waves of spans of 128 to 256, which the block
// scheduler balances (1,048,576 secondary rays: 637 us at 128, 684 at 64, 687 at 256; 4.2 M:
// 2.60 ms at 128, 2.49 at 256).
__host__ __device__ __forceinline__ uint32_t quad_span(uint32_t n, uint32_t resident)
{
    if (n <= resident) return 1;
    const uint32_t full = resident * 3 / 4, sparse = resident * 3 / 16, waves = resident * 9 / 4;
    const uint32_t one = (n + full - 1) / full;
    if (one <= 128)
    {
        const uint32_t lanes = (n + sparse - 1) / sparse;
        const uint32_t least = lanes < 32 ? lanes : 32;
        return one > least ? one : least;
    }
    const uint32_t many = (n + waves - 1) / waves;
    return many < 128 ? 128 : (many > 256 ? 256 : many);
}

// Rays that a warp takes at a time off a shared counter when there are more than kQuadChunk
// for each resident warp: a warp that got long rays takes fewer, and the launch ends
// together.  Against fixed spans: 400,000 sorted secondary rays 378 -> 351 us, 1,000,000 636
// -> 549, 4,194,304 2,096 -> 1,810; high-definition frame 44.3 -> 41.5 ms, batch of scenes
// 8.83 -> 7.70.  48 and 64 at a time are up to 5 % slower at a few hundred thousand rays, 1 %
// faster on ambient occlusion; 128 slower.  The counter is part of the memory that sorted
// queries, host-buffer queries, frames and batches have; a device query in input order has
// none (trace_device in api.cu) and keeps the spans (with a counter camera rays would take
// 163 us for 200 at 640^2, 281 for 320 at 1024^2, 1,037 for 1,022 at 2048^2).
constexpr uint32_t kQuadChunk = 32;

// A warp's rays: next .. end - 1 first, then, unless shared is 0, chunks below `shared`
// (the number of rays) from `first` + what the counter says.
struct quad_work
{
    uint32_t next, end, shared, first;
    uint32_t* taken;
};

__host__ __device__ __forceinline__ bool quad_shared(uint32_t n, uint32_t resident)
{
    return n > resident * kQuadChunk && n < 0xF0000000u;   // chunks past the end do not wrap
}

// The work of one warp (empty: next >= end).  taken: a zeroed counter, or null.
__device__ __forceinline__ quad_work quad_share(uint32_t warp, uint32_t n, uint32_t resident, uint32_t* taken)
{
    if (taken && quad_shared(n, resident))
    {
        if (warp >= resident) return { 0, 0, 0, 0, nullptr };
        return { warp * kQuadChunk, (warp + 1) * kQuadChunk, n, resident * kQuadChunk, taken };
    }
    const uint32_t span = quad_span(n, resident);
    const uint64_t first = uint64_t(warp) * span;
    if (first >= n) return { 0, 0, 0, 0, nullptr };
    const uint32_t next = uint32_t(first);
    return { next, n - next < span ? n : next + span, 0, 0, nullptr };
}

__device__ __forceinline__ float max3f(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// A triangle's own leaf box (tri_box in lbvh_device.cuh, for finite input) against a ray
// by the pair loop's slab test: whether it is hit, and its entry distance.
__device__ __forceinline__ bool leaf_box_hit(f3 o, f3 id, float tmin, float tmax, f3 v, f3 e1, f3 e2, float& tn)
{
    const f3 p = { __fadd_rn(v.x, e1.x), __fadd_rn(v.y, e1.y), __fadd_rn(v.z, e1.z) };
    const f3 q = { __fadd_rn(v.x, e2.x), __fadd_rn(v.y, e2.y), __fadd_rn(v.z, e2.z) };
    const float lx = (ref_min(ref_min(v.x, p.x), q.x) - o.x) * id.x, hx = (ref_max(ref_max(v.x, p.x), q.x) - o.x) * id.x;
    const float ly = (ref_min(ref_min(v.y, p.y), q.y) - o.y) * id.y, hy = (ref_max(ref_max(v.y, p.y), q.y) - o.y) * id.y;
    const float lz = (ref_min(ref_min(v.z, p.z), q.z) - o.z) * id.z, hz = (ref_max(ref_max(v.z, p.z), q.z) - o.z) * id.z;
    tn = fmaxf(tmin, fmaxf(fminf(lx, hx), fmaxf(fminf(ly, hy), fminf(lz, hz))));
    return fminf(tmax, fminf(fmaxf(lx, hx), fminf(fmaxf(ly, hy), fmaxf(lz, hz)))) >= tn;
}

// The reciprocal of a zero direction component.  The pair loop takes FLT_MAX, with which an
// axis is entered at -inf and left at inf for any origin between its planes; here the
// distances have to stay finite, and quad_ray_ok sees to it that they are still beyond
// those of the other axes.
constexpr float kQuadZeroRcp = 7.555786372591432e22f;   // 2^76
__device__ __forceinline__ float quad_rcp(float d) { return d != 0.0f ? __frcp_rn(d) : kQuadZeroRcp; }

// Whether the quads' conservative arithmetic covers a ray that starts from node `root`:
// components finite and moderate, each direction component zero or not below 2^-40 of the
// largest.  What overflows within these bounds becomes an infinity or a NaN that leaves its
// axis unbounded.  With a zero component, an origin between the planes of that axis is
// inside them by the margin of a step, at least 2^-6.5 cell * 2^76 as a distance; cells are
// at least 2^-40 of the tree's largest coordinate M (quads.cu), so that is above 2^29.4 M,
// and the distances along the largest component d are at most (M + |o|) / d: not more than
// 2^28.1 M for an origin within 2^14 M and d above 2^-14.
__device__ __forceinline__ bool quad_ray_ok(f3 o, f3 d, bvh_view const& v, int root)
{
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    const float md = fmaxf(fmaxf(ax, ay), az), low = md * 9.094947017729282e-13f;
    const float mo = fabsf(o.x) + fabsf(o.y) + fabsf(o.z);
    const bool ok = md >= 9.094947017729282e-13f && md <= 1.099511627776e12f && mo <= 1.152921504606847e18f &&
                    (ax >= low || ax == 0.0f) && (ay >= low || ay == 0.0f) && (az >= low || az == 0.0f);
    if (uint32_t(root) >= uint32_t(v.num_inner) || (ax != 0.0f && ay != 0.0f && az != 0.0f)) return ok;
    return ok && md >= 6.103515625e-05f && mo <= 16384.0f * tree_reach(v.nodes + root);
}

// Traces the rays index(k) of `rays` for the k of `work` with the calling warp (every lane
// must call it with the same work) and calls done(ray, result) for each, in any order
// and from any lane.  index(k) below n is a ray, root(ray) the link its walk starts from.
// stack_mem: kQuadStack * kQuadBlock shared words of the block.  bad: null when the host
// knows the quads valid, else their validity word (the last record's org[0]): when it is
// set every ray takes the pair loop.
template <bool AnyHit, bool NearFirst, int Steps, class Root, class Index, class Done>
__device__ __forceinline__ void quad_trace(int* stack_mem, bvh_view const& v, const float* __restrict__ bad,
                                           const gbrt_ray* __restrict__ rays, uint32_t n, quad_work work,
                                           uint32_t* __restrict__ status, Root root, Index index, Done done)
{
    uint32_t next = work.next, end = work.end;
    constexpr int kDeep = INT32_MAX;   // best_tri of a ray that the pair loop answers
    const uint32_t full = 0xFFFFFFFFu, none = 0xFFFFFFFFu;
    const uint32_t lane_bit = 1u << (threadIdx.x & 31u);
    // the lane's stack column as shared-memory addresses; the entry at col ends the walk
    const uint32_t col = uint32_t(__cvta_generic_to_shared(stack_mem)) + 4u * threadIdx.x;
    const uint32_t top_limit = col + 4u * kQuadBlock * (kQuadStack - 4);
    uint32_t ray = none, top = col;
    int node = kEmptyLink, best_tri = -1;
    f3 o = { 0.0f, 0.0f, 0.0f }, d = { 0.0f, 0.0f, 0.0f }, id = { 0.0f, 0.0f, 0.0f };
    float tmin = 0.0f, tmax = 0.0f, limit = 0.0f, best_t = 0.0f, second_t = 0.0f;

    // One quad: the nearest (or first) hit child becomes `node`, the others are pushed; with
    // no hit the stack is popped.
    auto step = [&]() {
        float a[8], b[8];
        ld8(v.quads + node, a);
        ld8(reinterpret_cast<const char*>(v.quads + node) + 32, b);
        // the distance to plane value f = 1 + q 2^-16 of an axis is f * S + O with S =
        // 2^16 cell / d and O = (org - o) / d - S; the margin 2^-21 (|org - o| / |d| + |S|)
        // is more than the roundings here and those of the pair loop's test together
        const float k21 = 4.76837158203125e-07f;
        const float Sx = a[3] * id.x, Sy = b[6] * id.y, Sz = b[7] * id.z;
        const float Ax = (a[0] - o.x) * id.x, Ay = (a[1] - o.y) * id.y, Az = (a[2] - o.z) * id.z;
        const float Ox = Ax - Sx, Oy = Ay - Sy, Oz = Az - Sz;
        const float mx = fabsf(Ax) + fabsf(Sx), my = fabsf(Ay) + fabsf(Sy), mz = fabsf(Az) + fabsf(Sz);
        const float nxo = __fmaf_rn(-k21, mx, Ox), fxo = __fmaf_rn(k21, mx, Ox);
        const float nyo = __fmaf_rn(-k21, my, Oy), fyo = __fmaf_rn(k21, my, Oy);
        const float nzo = __fmaf_rn(-k21, mz, Oz), fzo = __fmaf_rn(k21, mz, Oz);
        // near and far planes by the direction's sign: one select per four planes
        const bool sx = id.x < 0.0f, sy = id.y < 0.0f, sz = id.z < 0.0f;
        const uint32_t nx4 = __float_as_uint(sx ? b[1] : b[0]), fx4 = __float_as_uint(sx ? b[0] : b[1]);
        const uint32_t ny4 = __float_as_uint(sy ? b[3] : b[2]), fy4 = __float_as_uint(sy ? b[2] : b[3]);
        const uint32_t nz4 = __float_as_uint(sz ? b[5] : b[4]), fz4 = __float_as_uint(sz ? b[4] : b[5]);
        float tn[4], tf[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            // byte k of the planes into bits 7..14 of 1.0f: the float 1 + q 2^-16.  The
            // dot product runs on the FMA pipe; a byte permute, as the rest of the visit
            // (selects, minima, compares), on the ALU pipe, which was the narrowest one (camera
            // rays 337 -> 306 us, ambient occlusion 2.51 -> 2.30 ms, high-definition frame
            // 47.1 -> 44.3).
            auto plane = [&](uint32_t q) { return __uint_as_float(__dp4a(q, 0x80u << (8 * k), 0x3F800000u)); };
            const float nx = __fmaf_rn(plane(nx4), Sx, nxo), fx = __fmaf_rn(plane(fx4), Sx, fxo);
            const float ny = __fmaf_rn(plane(ny4), Sy, nyo), fy = __fmaf_rn(plane(fy4), Sy, fyo);
            const float nz = __fmaf_rn(plane(nz4), Sz, nzo), fz = __fmaf_rn(plane(fz4), Sz, fzo);
            tn[k] = max3f(fmaxf(nx, ny), nz, tmin);
            tf[k] = min3f(fminf(fx, fy), fz, limit);
        }
        // Selection, pushes and pop as predicated PTX: as C++ they became branches that
        // split the warp (401 -> 361 instructions per ray).  Only the nearest child is
        // chosen; the others keep slot order (sorting them saves 1 % of the visits).  A
        // child equal to the chosen one (an empty slot repeats the last link, if its
        // inverted box passes) is not pushed.
        if constexpr (NearFirst)
            asm volatile(
                "{\n\t.reg .pred h0,h1,h2,h3,p,q;\n\t.reg .f32 t0,t1,t2,t3,ta,tb;\n\t.reg .b32 la,lb;\n\t"
                "setp.le.f32 h0, %2, %6;\n\tsetp.le.f32 h1, %3, %7;\n\t"
                "setp.le.f32 h2, %4, %8;\n\tsetp.le.f32 h3, %5, %9;\n\t"
                "selp.f32 t0, %2, 0f7F800000, h0;\n\tselp.f32 t1, %3, 0f7F800000, h1;\n\t"
                "selp.f32 t2, %4, 0f7F800000, h2;\n\tselp.f32 t3, %5, 0f7F800000, h3;\n\t"
                "setp.lt.f32 p, t1, t0;\n\tselp.b32 la, %11, %10, p;\n\tmin.f32 ta, t0, t1;\n\t"
                "setp.lt.f32 q, t3, t2;\n\tselp.b32 lb, %13, %12, q;\n\tmin.f32 tb, t2, t3;\n\t"
                "setp.lt.f32 p, tb, ta;\n\tselp.b32 %0, lb, la, p;\n\tmin.f32 ta, ta, tb;\n\t"
                "setp.ne.and.s32 q, %13, %0, h3;\n\t@q add.u32 %1, %1, %14;\n\t@q st.shared.b32 [%1], %13;\n\t"
                "setp.ne.and.s32 q, %12, %0, h2;\n\t@q add.u32 %1, %1, %14;\n\t@q st.shared.b32 [%1], %12;\n\t"
                "setp.ne.and.s32 q, %11, %0, h1;\n\t@q add.u32 %1, %1, %14;\n\t@q st.shared.b32 [%1], %11;\n\t"
                "setp.ne.and.s32 q, %10, %0, h0;\n\t@q add.u32 %1, %1, %14;\n\t@q st.shared.b32 [%1], %10;\n\t"
                "setp.eq.f32 p, ta, 0f7F800000;\n\t@p ld.shared.b32 %0, [%1];\n\t@p sub.u32 %1, %1, %14;\n\t}"
                : "=&r"(node), "+r"(top)
                : "f"(tn[0]), "f"(tn[1]), "f"(tn[2]), "f"(tn[3]), "f"(tf[0]), "f"(tf[1]), "f"(tf[2]), "f"(tf[3]),
                  "r"(__float_as_int(a[4])), "r"(__float_as_int(a[5])), "r"(__float_as_int(a[6])),
                  "r"(__float_as_int(a[7])), "n"(4 * kQuadBlock)
                : "memory");
        else
            asm volatile(
                "{\n\t.reg .pred h0,h1,h2,h3,p,q;\n\t"
                "setp.le.f32 h0, %2, %6;\n\tsetp.le.f32 h1, %3, %7;\n\t"
                "setp.le.f32 h2, %4, %8;\n\tsetp.le.f32 h3, %5, %9;\n\t"
                "selp.b32 %0, %12, %13, h2;\n\tselp.b32 %0, %11, %0, h1;\n\tselp.b32 %0, %10, %0, h0;\n\t"
                "setp.ne.and.s32 q, %13, %0, h3;\n\t@q add.u32 %1, %1, %14;\n\t@q st.shared.b32 [%1], %13;\n\t"
                "setp.ne.and.s32 q, %12, %0, h2;\n\t@q add.u32 %1, %1, %14;\n\t@q st.shared.b32 [%1], %12;\n\t"
                "setp.ne.and.s32 q, %11, %0, h1;\n\t@q add.u32 %1, %1, %14;\n\t@q st.shared.b32 [%1], %11;\n\t"
                "or.pred p, h0, h1;\n\tor.pred q, h2, h3;\n\tor.pred p, p, q;\n\t"
                "@!p ld.shared.b32 %0, [%1];\n\t@!p sub.u32 %1, %1, %14;\n\t}"
                : "=&r"(node), "+r"(top)
                : "f"(tn[0]), "f"(tn[1]), "f"(tn[2]), "f"(tn[3]), "f"(tf[0]), "f"(tf[1]), "f"(tf[2]), "f"(tf[3]),
                  "r"(__float_as_int(a[4])), "r"(__float_as_int(a[5])), "r"(__float_as_int(a[6])),
                  "r"(__float_as_int(a[7])), "n"(4 * kQuadBlock)
                : "memory");
        const bool deep = top > top_limit;   // at least one free entry short of a visit's three
        node = deep ? kEmptyLink : node;
        best_tri = deep ? kDeep : best_tri;
    };

    for (;;)
    {
        // a link outside both ranges (the end of a walk, or a corrupt one) leaves a lane idle
        const bool leaf = uint32_t(~node) < uint32_t(v.num_tris);
        const uint32_t leaves = __ballot_sync(full, leaf);
        const uint32_t busy = __ballot_sync(full, leaf || uint32_t(node) < uint32_t(v.num_inner));
        if (next >= end && end < work.shared && 32 - __popc(busy) >= kQuadRefill)
        {
            // end == shared once the rays are out
            uint32_t taken = 0;
            if (lane_bit == 1u) taken = atomicAdd(work.taken, kQuadChunk);
            taken = __shfl_sync(full, taken, 0);
            next = min(work.first + taken, work.shared);
            end = min(next + kQuadChunk, work.shared);
        }
        if (busy == 0 || (next < end && 32 - __popc(busy) >= kQuadRefill))
        {
            if (!(busy & lane_bit))
            {
                if (ray != none)
                {
                    if (node != kEmptyLink) atomicOr(status, kStatusBadIndex);
                    if (!AnyHit && best_tri >= kQuadOpen - 1 && best_tri != kDeep) best_tri -= kQuadOpen;
                    trace_result res{ best_tri, best_t, 0.0f, 0.0f };
                    bool exact = best_tri == kDeep;
                    if (best_tri >= 0 && !exact)
                    {
                        const tri48* tp = v.tris + best_tri;
                        const float4 t0 = ldg4(&tp->t0), t1 = ldg4(&tp->t1), t2 = ldg4(&tp->t2);
                        const f3 v1 = { t0.x, t0.y, t0.z }, e1 = { t1.x, t1.y, t1.z }, e2 = { t2.x, t2.y, t2.z };
                        float tn;
                        const bool in_box = leaf_box_hit(o, { safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z) }, tmin, tmax,
                                                         v1, e1, e2, tn);
                        // a box entered beyond the culling distance (a sliver's t is far off)
                        // may have hidden such a second hit
                        exact = !in_box || (!AnyHit && (tn > limit || second_t <= fmaxf(best_t, tn)));
                        // u and v by the same test on the same inputs: the same values
                        const tri_hit h = intersect_triangle(o, d, v1, e1, e2);
                        res.u = h.u;
                        res.v = h.v;
                    }
                    if (exact)
                    {
                        local_stack<kStackSize> stack;
                        res = traverse_bvh_with<AnyHit, decltype(stack), NearFirst>(
                            stack, v.nodes, v.tris, root(ray), v.num_inner, v.num_tris, o, d, tmin, tmax, status);
                    }
                    done(ray, res);
                    ray = none;
                }
                node = kEmptyLink;
                const uint32_t k = next + __popc(~busy & (lane_bit - 1u));
                if (k < end)
                {
                    ray = index(k);
                    if (ray < n)
                    {
                        const float4 r0 = ldg4(&rays[ray]);
                        const float4 r1 = ldg4(reinterpret_cast<const float4*>(&rays[ray]) + 1);
                        o = { r0.x, r0.y, r0.z };
                        d = { r0.w, r1.x, r1.y };
                        id = { quad_rcp(d.x), quad_rcp(d.y), quad_rcp(d.z) };
                        tmin = r1.z;
                        limit = tmax = r1.w;
                        best_t = second_t = FLT_MAX;
                        top = col;
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(top), "r"(kEmptyLink) : "memory");
                        const int start = root(ray);
                        const bool ok = quad_ray_ok(o, d, v, start) && !(bad && *bad != 0.0f);
                        node = ok ? start : kEmptyLink;
                        best_tri = ok ? -1 : kDeep;
                    }
                    else
                    {
                        atomicOr(status, kStatusBadIndex);
                        ray = none;
                    }
                }
            }
            const bool last = busy == 0 && next >= end;
            next = min(end, next + __popc(~busy));
            if (last) break;
            continue;
        }
        if (leaves != 0)
        {
            if (leaf)
            {
                const int t = ~node;
                const tri48* tp = v.tris + t;
                // the record's aligned 32 bytes and the other 16: two loads per lane, not three
                const bool odd = reinterpret_cast<uintptr_t>(tp) & 16;
                float w[8];
                ld8(reinterpret_cast<const char*>(tp) + (odd ? 16 : 0), w);
                const float4 x4 = ldg4(reinterpret_cast<const float4*>(tp) + (odd ? 0 : 2));
                const f3 t0 = { odd ? x4.x : w[0], odd ? x4.y : w[1], odd ? x4.z : w[2] };
                const f3 t1 = { odd ? w[0] : w[4], odd ? w[1] : w[5], odd ? w[2] : w[6] };
                const f3 t2 = { odd ? w[4] : x4.x, odd ? w[5] : x4.y, odd ? w[6] : x4.z };
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(node) : "r"(top) : "memory");
                top -= 4u * kQuadBlock;
                const tri_hit h = intersect_triangle(o, d, t0, t1, t2);
                const bool hit = h.hit && h.t >= tmin && h.t <= tmax;
                if constexpr (AnyHit)
                {
                    if (hit)
                    {
                        best_tri = t;
                        best_t = h.t;
                        node = kEmptyLink;
                    }
                }
                else
                {
                    const float size = max3f(fabsf(d.x), fabsf(d.y), fabsf(d.z)) *
                                       (max3f(fabsf(t1.x), fabsf(t1.y), fabsf(t1.z)) *
                                        max3f(fabsf(t2.x), fabsf(t2.y), fabsf(t2.z)));
                    bool open = best_tri >= kQuadOpen - 1;
                    if (!open && h.det != 0.0f && !(fabsf(h.det) > kQuadEdgeOn * size))
                    {
                        open = true;
                        best_tri += kQuadOpen;
                    }
                    if (hit)
                    {
                        second_t = fminf(second_t, fmaxf(h.t, best_t));
                        best_tri = h.t < best_t ? (open ? t + kQuadOpen : t) : best_tri;
                        best_t = fminf(h.t, best_t);
                    }
                    limit = open ? tmax : fminf(tmax, best_t + fabsf(best_t) * (1.0f / 256.0f));
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int k = 0; k < Steps; ++k)
        {
            if (uint32_t(node) < uint32_t(v.num_inner)) step();
            __syncwarp();
        }
    }
}

} // namespace gbrt
