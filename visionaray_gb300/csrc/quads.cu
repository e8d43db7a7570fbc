// Quad nodes: up to four descendants of a node pair in one 64-byte record with outward
// quantised boxes (layout in bvh_layout.cuh), made from a finished tree in one pass.  The
// ray queries and the path tracer traverse them (quad_trace.cuh).
//
// One thread per node pair starts from its two children and twice opens the inner one of
// the largest box area, in place, so the slots stay in depth-first order (which any-hit
// queries depend on).  A quad is then full wherever its subtree has four leaves, and the
// boxes most likely to be hit are the ones replaced.  Against opening both children
// always: sorted secondary rays over a 2048^2 heightfield 2.27 -> 2.18 ms, ambient
// occlusion 2.61 -> 2.51, preview frame 237 -> 217 us, high-definition frame 48.2 -> 46.8
// ms, at the same build time.
//
// No queue, no compaction, no level-by-level launches, and a quad has its node pair's
// index, so the pairs' links serve unchanged.  Every pair gets a quad although a walk from
// the root meets fewer: which ones those are is not known bottom-up, and the pass is bound
// by HBM traffic either way (64 B read and 64 B written per pair).

#include "traverse_core.cuh"

namespace gbrt {
namespace {

constexpr int kBlock = 256;

// The coordinates a quantised tree covers: beyond them (or for a non-finite box) queries
// keep the node pairs.
constexpr float kQuadMaxCoord = 1.152921504606847e18f;   // 2^60

struct slot
{
    float lo[3], hi[3];
    int link;
};

__device__ __forceinline__ slot child(bvh2_node const& p, int s)
{
    return s ? slot{ { p.xy1.x, p.xy1.z, p.z01.z }, { p.xy1.y, p.xy1.w, p.z01.w }, p.link.y }
             : slot{ { p.xy0.x, p.xy0.z, p.z01.x }, { p.xy0.y, p.xy0.w, p.z01.y }, p.link.x };
}

__device__ __forceinline__ slot pick(bool first, slot const& a, slot const& b)
{
    return { { first ? a.lo[0] : b.lo[0], first ? a.lo[1] : b.lo[1], first ? a.lo[2] : b.lo[2] },
             { first ? a.hi[0] : b.hi[0], first ? a.hi[1] : b.hi[1], first ? a.hi[2] : b.hi[2] },
             first ? a.link : b.link };
}

// Half the surface of an inner slot's box (at most FLT_MAX, 0 for a NaN), -1 for a leaf.
__device__ __forceinline__ float open_area(slot const& s, uint32_t num_inner)
{
    const float x = s.hi[0] - s.lo[0], y = s.hi[1] - s.lo[1], z = s.hi[2] - s.lo[2];
    const float area = x * y + y * z + z * x;
    return uint32_t(s.link) < num_inner ? fminf(fmaxf(area, 0.0f), FLT_MAX) : -1.0f;
}

// roots: null, or the first node pairs of num_scenes trees (batches); root: the only tree's.
__global__ void __launch_bounds__(kBlock) make_quad_nodes(const bvh2_node* __restrict__ nodes, uint32_t num_inner,
                                                          const uint32_t* __restrict__ roots, uint32_t num_scenes,
                                                          uint32_t root, quad_node* __restrict__ quads,
                                                          uint32_t* __restrict__ host_bad)
{
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= num_inner) return;
    const bvh2_node p = nodes[i];
    const float reach = tree_reach(nodes + (roots ? __ldg(&roots[upper_segment(roots, num_scenes, i)]) : root));
    // named values: an array indexed by the choice goes to local memory (0.28 -> 0.70 ms for
    // 8.4 M triangles)
    slot s0 = child(p, 0), s1 = child(p, 1), s2 = s1, s3;
    const float blo[3] = { fminf(s0.lo[0], s1.lo[0]), fminf(s0.lo[1], s1.lo[1]), fminf(s0.lo[2], s1.lo[2]) };
    const float bhi[3] = { fmaxf(s0.hi[0], s1.hi[0]), fmaxf(s0.hi[1], s1.hi[1]), fmaxf(s0.hi[2], s1.hi[2]) };
    int count = 2;
    const float a0 = open_area(s0, num_inner), a1 = open_area(s1, num_inner);
    if (a0 >= 0.0f || a1 >= 0.0f)
    {
        const bool left = a0 >= a1;
        const bvh2_node q = nodes[left ? s0.link : s1.link];
        const slot f = child(q, 0), l = child(q, 1);
        s2 = pick(left, s1, l);
        s1 = pick(left, l, f);
        s0 = pick(left, f, s0);
        count = 3;
    }
    s3 = s2;
    const float b0 = open_area(s0, num_inner), b1 = open_area(s1, num_inner);
    const float b2 = count == 3 ? open_area(s2, num_inner) : -1.0f;
    if (b0 >= 0.0f || b1 >= 0.0f || b2 >= 0.0f)
    {
        const bool first = b0 >= b1 && b0 >= b2, last = !first && b2 > b1;
        const bvh2_node q = nodes[first ? s0.link : (last ? s2.link : s1.link)];
        const slot f = child(q, 0), l = child(q, 1);
        s3 = pick(last, l, s2);
        s2 = pick(first, s1, pick(last, f, l));
        s1 = pick(first, l, pick(last, s1, f));
        s0 = pick(first, f, s0);
        count = 4;
    }
    const slot c[4] = { s0, s1, s2, s3 };
    uint32_t qlo[3], qhi[3], scale[3];
    float org[3];
    bool fits = true;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        // cell: the smallest power of two that covers the box with 252 of them and is at
        // least 2^-20 of its largest coordinate, so that org = low corner - cell is below
        // the corner by about a cell after rounding and every plane below stays in 0..255;
        // at least 2^-40 of the tree's largest coordinate for rays along the planes
        // (quad_ray_ok)
        const float far_coord = fmaxf(fabsf(blo[a]), fabsf(bhi[a]));
        float t = fmaxf(__fdiv_ru(__fsub_ru(bhi[a], blo[a]), 252.0f), far_coord * 9.5367431640625e-07f);
        t = fmaxf(t, reach * 9.094947017729282e-13f);
        t = fminf(fmaxf(t, 8.271806125530277e-25f), kQuadMaxCoord);   // 2^-80
        const int e = int((__float_as_uint(t) + 0x7FFFFFu) >> 23) - 127;
        const float cell = __int_as_float((e + 127) << 23);
        const float inv = __int_as_float((127 - e) << 23);   // exact
        scale[a] = uint32_t(e + 127 + 16) << 23;
        org[a] = __fsub_rd(blo[a], cell);
        qlo[a] = qhi[a] = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            float l = 255.0f, h = 0.0f;
            if (k < count)
            {
                l = floorf(__fsub_rd(c[k].lo[a], org[a]) * inv);
                h = ceilf(__fsub_ru(c[k].hi[a], org[a]) * inv);
                // every box of the record is finite and moderate, or the tree is not
                // traversed through its quads (fminf / fmaxf above would hide a NaN)
                fits = fits && fabsf(c[k].lo[a]) <= kQuadMaxCoord && fabsf(c[k].hi[a]) <= kQuadMaxCoord && l >= 0.0f &&
                       h <= 255.0f;
            }
            qlo[a] |= uint32_t(fminf(fmaxf(l, 0.0f), 255.0f)) << (8 * k);
            qhi[a] |= uint32_t(fminf(fmaxf(h, 0.0f), 255.0f)) << (8 * k);
        }
    }
    uint4* w = reinterpret_cast<uint4*>(quads + i);
    w[0] = make_uint4(__float_as_uint(org[0]), __float_as_uint(org[1]), __float_as_uint(org[2]), scale[0]);
    w[1] = make_uint4(c[0].link, c[1].link, c[2].link, c[3].link);
    w[2] = make_uint4(qlo[0], qhi[0], qlo[1], qhi[1]);
    w[3] = make_uint4(qlo[2], qhi[2], scale[1], scale[2]);
    if (!fits)
    {
        quads[num_inner].org[0] = 1.0f;
        if (host_bad) *host_bad = 1u;
    }
}

} // namespace

gbrt_status make_quads(gbrt_context* ctx, bvh2_node const* nodes, uint32_t num_inner, uint32_t const* roots,
                       uint32_t num_scenes, uint32_t root, quad_node* quads, uint32_t* host_bad, cudaStream_t stream)
{
    make_quad_nodes<<<(num_inner + kBlock - 1) / kBlock, kBlock, 0, stream>>>(nodes, num_inner, roots, num_scenes, root,
                                                                            quads, host_bad);
    GBRT_LAUNCH_CHECK(ctx, "make_quad_nodes");
    return GBRT_OK;
}

} // namespace gbrt
