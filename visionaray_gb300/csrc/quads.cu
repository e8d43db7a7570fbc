// Quad nodes: two levels of the node pairs in one 64-byte record with outward quantised
// boxes (layout in bvh_layout.cuh), made from a finished tree in one pass.  The ray
// queries and the path tracer traverse them (quad_trace.cuh).
//
// One thread per node pair reads its own record and its two inner children's and writes
// one record: no queue, no compaction, no level-by-level launches, and a quad has its
// node pair's index, so the pairs' links serve unchanged.  Every pair gets a quad although
// a walk from the root meets every second level only: which levels those are is not known
// bottom-up, and the pass is bound by HBM traffic either way (64 B read and 64 B written
// per pair).

#include "api_internal.h"
#include "device_math.cuh"

namespace gbrt {
namespace {

constexpr int kBlock = 256;

// The coordinates a quantised tree covers: beyond them (or for a non-finite box) queries
// keep the node pairs.
constexpr float kQuadMaxCoord = 1.152921504606847e18f;   // 2^60

__global__ void __launch_bounds__(kBlock) make_quad_nodes(const bvh2_node* __restrict__ nodes, uint32_t num_inner,
                                                          quad_node* __restrict__ quads,
                                                          uint32_t* __restrict__ host_bad)
{
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= num_inner) return;
    const bvh2_node p = nodes[i];
    float lo[3][4], hi[3][4];
    int link[4];
    uint32_t empty = 0;
#pragma unroll
    for (int s = 0; s < 2; ++s)
    {
        const int c = s ? p.link.y : p.link.x;
        if (c >= 0 && uint32_t(c) < num_inner)
        {
            const bvh2_node q = nodes[c];
            lo[0][2 * s] = q.xy0.x, hi[0][2 * s] = q.xy0.y, lo[1][2 * s] = q.xy0.z, hi[1][2 * s] = q.xy0.w;
            lo[2][2 * s] = q.z01.x, hi[2][2 * s] = q.z01.y;
            lo[0][2 * s + 1] = q.xy1.x, hi[0][2 * s + 1] = q.xy1.y, lo[1][2 * s + 1] = q.xy1.z;
            hi[1][2 * s + 1] = q.xy1.w, lo[2][2 * s + 1] = q.z01.z, hi[2][2 * s + 1] = q.z01.w;
            link[2 * s] = q.link.x;
            link[2 * s + 1] = q.link.y;
        }
        else
        {
            const float4 xy = s ? p.xy1 : p.xy0;
            lo[0][2 * s] = xy.x, hi[0][2 * s] = xy.y, lo[1][2 * s] = xy.z, hi[1][2 * s] = xy.w;
            lo[2][2 * s] = s ? p.z01.z : p.z01.x, hi[2][2 * s] = s ? p.z01.w : p.z01.y;
            link[2 * s] = link[2 * s + 1] = c;
            empty |= 2u << (2 * s);
        }
    }
    const float blo[3] = { fminf(p.xy0.x, p.xy1.x), fminf(p.xy0.z, p.xy1.z), fminf(p.z01.x, p.z01.z) };
    const float bhi[3] = { fmaxf(p.xy0.y, p.xy1.y), fmaxf(p.xy0.w, p.xy1.w), fmaxf(p.z01.y, p.z01.w) };
    uint32_t qlo[3], qhi[3], scale[3];
    float org[3];
    bool fits = true;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        // cell: the smallest power of two that covers the box with 252 of them and is at
        // least 2^-20 of its largest coordinate, so that org = low corner - cell is below
        // the corner by about a cell after rounding and every plane below stays in 0..255
        const float far_coord = fmaxf(fabsf(blo[a]), fabsf(bhi[a]));
        float t = fmaxf(__fdiv_ru(__fsub_ru(bhi[a], blo[a]), 252.0f), far_coord * 9.5367431640625e-07f);
        t = fminf(fmaxf(t, 8.271806125530277e-25f), kQuadMaxCoord);   // 2^-80
        const int e = int((__float_as_uint(t) + 0x7FFFFFu) >> 23) - 127;
        const float cell = __int_as_float((e + 127) << 23);
        const float inv = __int_as_float((127 - e) << 23);   // exact
        scale[a] = uint32_t(e + 127 + 15) << 23;
        org[a] = __fsub_rd(blo[a], cell);
        qlo[a] = qhi[a] = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            float l = 255.0f, h = 0.0f;
            if (!(empty >> k & 1u))
            {
                l = floorf(__fsub_rd(lo[a][k], org[a]) * inv);
                h = ceilf(__fsub_ru(hi[a][k], org[a]) * inv);
                // every box of the record is finite and moderate, or the tree is not
                // traversed through its quads (fminf / fmaxf above would hide a NaN)
                fits = fits && fabsf(lo[a][k]) <= kQuadMaxCoord && fabsf(hi[a][k]) <= kQuadMaxCoord && l >= 0.0f &&
                       h <= 255.0f;
            }
            qlo[a] |= uint32_t(fminf(fmaxf(l, 0.0f), 255.0f)) << (8 * k);
            qhi[a] |= uint32_t(fminf(fmaxf(h, 0.0f), 255.0f)) << (8 * k);
        }
    }
    uint4* w = reinterpret_cast<uint4*>(quads + i);
    w[0] = make_uint4(__float_as_uint(org[0]), __float_as_uint(org[1]), __float_as_uint(org[2]), scale[0]);
    w[1] = make_uint4(link[0], link[1], link[2], link[3]);
    w[2] = make_uint4(qlo[0], qhi[0], qlo[1], qhi[1]);
    w[3] = make_uint4(qlo[2], qhi[2], scale[1], scale[2]);
    if (!fits)
    {
        quads[num_inner].org[0] = 1.0f;
        if (host_bad) *host_bad = 1u;
    }
}

} // namespace

gbrt_status make_quads(gbrt_context* ctx, bvh2_node const* nodes, uint32_t num_inner, quad_node* quads,
                       uint32_t* host_bad, cudaStream_t stream)
{
    make_quad_nodes<<<(num_inner + kBlock - 1) / kBlock, kBlock, 0, stream>>>(nodes, num_inner, quads, host_bad);
    GBRT_LAUNCH_CHECK(ctx, "make_quad_nodes");
    return GBRT_OK;
}

} // namespace gbrt
