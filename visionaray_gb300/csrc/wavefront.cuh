// The wavefront path tracer's state, shared by the single-scene renderer (pathtrace.cu) and
// the batch renderer (batch_wf.cu): ray and shadow queues, path state, vertex records.
// Units including this header are compiled with --fmad=false.
#pragma once

#include "pt_shade.cuh"
#include "quad_trace.cuh"

namespace gbrt {
namespace {

// Paths of a pass: 2^22 (0.8 GB of path state).  One sample per pixel and pass left a
// small frame's launches short of the GPU and every bounce's tail idle.  Measured against
// that: 641x479x4 over instances 8.30 -> 4.70 ms (its extend and shadow in one launch too),
// 512x512x16 forward frame 30.1 -> 19.7 ms, 1920x1080x8 box 76.0 -> 63.5 ms.
constexpr uint64_t kPassPaths = 1ull << 22;

struct frame_buffers
{
    gbrt_ray* rays[2];
    uint32_t* path[2];
    uint4* hits;
    gbrt_ray* shadow_rays;
    uint32_t* shadow_path;
    float4* shadow_contrib;
    float4* throughput;
    float4* radiance;
    uint2* rng_flags;   // draw counter, flags
    float4* sum;
    uint32_t* counts;   // per bounce: its ray queue's length, its shadow queue's
    uint32_t* taken;    // per queue: rays taken by warps beyond their first (quad_share)
    // path p of the pass is sample first_sample + p % samples of pixel first_pixel + p / samples
    uint32_t first_pixel, samples, first_sample;
    // the adjoint's replay: per bounce and path a vertex_rec in kRecWords float4
    // (rec[(bounce * paths + p) * kRecWords]), and each path's number of vertices; null for
    // a frame
    float4* rec;
    uint32_t* num_rec;
    uint32_t paths;
    // queue order by origin cell (GBRT_TRACE_SORT_RAYS): keys / values and their
    // double buffers, the sort's scratch
    uint32_t* keys;
    uint32_t* vals;
    uint32_t* keys_alt;
    uint32_t* vals_alt;
    void* sort_scratch;
};

constexpr int kRecWords = 5;

// The pixel and sample of path p of a pass.
__device__ __forceinline__ uint2 path_sample(frame_buffers const& fb, uint32_t p)
{
    return make_uint2(fb.first_pixel + p / fb.samples, fb.first_sample + p % fb.samples);
}

// Appends the lanes with `take` to a queue: one atomic per warp.  Every lane of the
// warp must call it.
__device__ __forceinline__ uint32_t warp_append(bool take, uint32_t* counter)
{
    const uint32_t full = 0xFFFFFFFFu;
    uint32_t mask = __ballot_sync(full, take);
    if (mask == 0) return 0;
    int lane = threadIdx.x & 31;
    int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, uint32_t(__popc(mask)));
    base = __shfl_sync(full, base, leader);
    return base + uint32_t(__popc(mask & ((1u << lane) - 1u)));
}

__device__ __forceinline__ void store_ray(gbrt_ray* dst, v3 o, v3 d, float tmin, float tmax)
{
    float4* p = reinterpret_cast<float4*>(dst);
    p[0] = make_float4(o.x, o.y, o.z, d.x);
    p[1] = make_float4(d.y, d.z, tmin, tmax);
}

// The answer of shadow queue entry j of a bounce: an unoccluded contribution is added to
// its path's radiance; in a replay an occluded one is taken out of its vertex record.
__device__ __forceinline__ void finish_shadow(frame_buffers const& fb, uint32_t j, uint32_t bounce, bool occluded)
{
    if (fb.rec)
    {
        if (occluded)
        {
            float* kind = &fb.rec[(uint64_t(bounce) * fb.paths + fb.shadow_path[j]) * kRecWords].x;
            *kind = __uint_as_float(__float_as_uint(*kind) & 0xFFu);
        }
        return;
    }
    if (occluded) return;
    const uint32_t p = fb.shadow_path[j];
    const float4 c = fb.shadow_contrib[j];
    const float4 r = fb.radiance[p];
    fb.radiance[p] = make_float4(r.x + c.x, r.y + c.y, r.z + c.z, 0.0f);
}

// vertex_rec in kRecWords float4 (the kind and the next-event flag share a word).
__device__ __forceinline__ void store_rec(frame_buffers const& fb, uint32_t bounce, uint32_t p, vertex_rec const& r)
{
    float4* o = fb.rec + (uint64_t(bounce) * fb.paths + p) * kRecWords;
    o[0] = make_float4(__uint_as_float(r.kind | r.nee << 8), __uint_as_float(r.geom), __uint_as_float(r.lgeom), r.rr);
    o[1] = make_float4(r.thr.x, r.thr.y, r.thr.z, r.w);
    o[2] = make_float4(r.x, r.b0, r.kl, r.lint.x);
    o[3] = make_float4(r.lint.y, r.lint.z, r.gnee.x, r.gnee.y);
    o[4] = make_float4(r.gnee.z, r.f.spec.x, r.f.spec.y, r.f.spec.z);
}

__device__ __forceinline__ vertex_rec load_rec(frame_buffers const& fb, uint32_t bounce, uint32_t p)
{
    const float4* o = fb.rec + (uint64_t(bounce) * fb.paths + p) * kRecWords;
    const float4 a = o[0], b = o[1], c = o[2], d = o[3], e = o[4];
    vertex_rec r;
    r.kind = __float_as_uint(a.x) & 0xFFu;
    r.nee = __float_as_uint(a.x) >> 8;
    r.geom = __float_as_uint(a.y);
    r.lgeom = __float_as_uint(a.z);
    r.rr = a.w;
    r.thr = { b.x, b.y, b.z };
    r.w = b.w;
    r.x = c.x;
    r.b0 = c.y;
    r.kl = c.z;
    r.lint = { c.w, d.x, d.y };
    r.gnee = { d.z, d.w, e.x };
    r.f.spec = { e.y, e.z, e.w };
    return r;
}

inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

// The buffers of a pass of n paths over npix pixels with num_counts queue lengths; sort: with
// the queue order's keys; record_bounces: with the vertex records of that many bounces.
// Returns their bytes; with base non-null sets fb to them.
inline size_t layout_frame_buffers(uint32_t npix, uint32_t n, uint64_t num_counts, bool sort, uint32_t record_bounces,
                                   void* base, frame_buffers& fb)
{
    const size_t key = sort ? size_t(n) * 4 : 0;
    size_t sizes[] = { size_t(n) * 32, size_t(n) * 32, size_t(n) * 4, size_t(n) * 4, size_t(n) * 16,
                       size_t(n) * 32, size_t(n) * 4,  size_t(n) * 16, size_t(n) * 16, size_t(n) * 16,
                       size_t(n) * 8,  size_t(npix) * 16, size_t(num_counts) * 8, key, key, key,
                       key, sort ? radix_sort_scratch_bytes(n) : 0,
                       size_t(n) * record_bounces * kRecWords * 16, record_bounces ? size_t(n) * 4 : 0 };
    constexpr int kParts = int(sizeof(sizes) / sizeof(sizes[0]));
    size_t total = 0;
    for (size_t s : sizes) total += align256(s);
    if (!base) return total;
    void* ptr[kParts];
    size_t off = 0;
    for (int k = 0; k < kParts; ++k)
    {
        ptr[k] = static_cast<char*>(base) + off;
        off += align256(sizes[k]);
    }
    fb.rays[0] = static_cast<gbrt_ray*>(ptr[0]);
    fb.rays[1] = static_cast<gbrt_ray*>(ptr[1]);
    fb.path[0] = static_cast<uint32_t*>(ptr[2]);
    fb.path[1] = static_cast<uint32_t*>(ptr[3]);
    fb.hits = static_cast<uint4*>(ptr[4]);
    fb.shadow_rays = static_cast<gbrt_ray*>(ptr[5]);
    fb.shadow_path = static_cast<uint32_t*>(ptr[6]);
    fb.shadow_contrib = static_cast<float4*>(ptr[7]);
    fb.throughput = static_cast<float4*>(ptr[8]);
    fb.radiance = static_cast<float4*>(ptr[9]);
    fb.rng_flags = static_cast<uint2*>(ptr[10]);
    fb.sum = static_cast<float4*>(ptr[11]);
    fb.counts = static_cast<uint32_t*>(ptr[12]);
    fb.taken = fb.counts + num_counts;
    fb.keys = static_cast<uint32_t*>(ptr[13]);
    fb.vals = static_cast<uint32_t*>(ptr[14]);
    fb.keys_alt = static_cast<uint32_t*>(ptr[15]);
    fb.vals_alt = static_cast<uint32_t*>(ptr[16]);
    fb.sort_scratch = ptr[17];
    fb.rec = record_bounces ? static_cast<float4*>(ptr[18]) : nullptr;
    fb.num_rec = static_cast<uint32_t*>(ptr[19]);
    fb.paths = n;
    fb.first_pixel = 0;
    fb.first_sample = 0;
    return total;
}

} // namespace
} // namespace gbrt
