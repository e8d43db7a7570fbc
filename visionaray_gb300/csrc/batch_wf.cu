// The batch renderer's wavefront frame: every scene's paths in the queues of one frame.
//
// The persistent kernel (batch_pt.cuh) runs a pixel's samples and bounces in one thread:
// its traversal diverges across pixels of different path lengths, and its registers hold
// the path beside the walk.  Here the frame goes in passes of up to kPassPaths paths of
// consecutive pixels of any scenes, through the stages of the single-scene renderer
// (pathtrace.cu): camera rays, closest hits over the arena's quad nodes from each ray's
// scene's root, shading with that scene's constants, shadow rays.  The arithmetic and the
// random numbers are the persistent kernel's, so the images are equal bit for bit.
// Measured: 64 scenes of 1 k to 1 M triangles, 6.7 M one-sample pixels of 3 bounces: frame
// 10.1 ms in the persistent kernel (launch {128, 32, 64, BLOCKS}), 6.6 here, 0.32 of them the
// quad nodes of the 9.6 M triangles.
//
// Used for launches on the node pairs, unsorted, with the full 64-entry stack (a shorter
// one reports trees it does not hold, which the quads' walk would not), where it is the
// faster one (batch_wavefront_applies).  Enqueue only: the buffers belong to the
// batch, so its captured frame stays valid whatever the context does.
// A frame that the caller captures goes through the persistent kernel: its replays must
// allow later calls to change the frames, and to need larger buffers.

#include "batch_pt.cuh"
#include "wavefront.cuh"

#include <algorithm>

namespace gbrt {
namespace {

constexpr int kBlock = 128;
constexpr int kShadeMinBlocks = 8;

struct batch_wf_args
{
    const batch_frame* __restrict__ frames;
    const uint32_t* pixel_offsets;
    uint32_t num_scenes, order;
    const gbrt_material* materials;
    uint32_t num_materials;
    const float4* lights;            // 4 float4 per light; null without lights
    const uint32_t* light_offsets;
    const float2* trig;
    // per path: its scene and its pixel in the scene's image
    uint32_t* scene;
    uint32_t* pixel;
};

// Path p of the pass is sample first_sample + p % samples of the first_pixel + p / samples-th
// pixel of the batch; those within their scene's sample count are queued.
__global__ void __launch_bounds__(kBlock) bp_raygen(batch_wf_args a, frame_buffers fb, uint32_t n)
{
    const uint32_t p = blockIdx.x * kBlock + threadIdx.x;
    bool live = p < n;
    v3 o = { 0.0f, 0.0f, 0.0f }, d = { 0.0f, 0.0f, 0.0f };
    if (live)
    {
        const uint2 ps = path_sample(fb, p);
        const uint32_t s = upper_segment(a.pixel_offsets, a.num_scenes, ps.x);
        const batch_frame& f = a.frames[s];
        uint32_t pixel = ps.x - __ldg(&a.pixel_offsets[s]);
        if (a.order == GBRT_BATCH_ORDER_BLOCKS && f.blocks)
        {
            const uint32_t blk = pixel >> 5, w = pixel & 31u, bw = f.width >> 3;
            pixel = ((blk / bw) * 4u + (w >> 3)) * f.width + (blk % bw) * 8u + (w & 7u);
        }
        a.scene[p] = s;
        a.pixel[p] = pixel;
        fb.throughput[p] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
        fb.radiance[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        fb.rng_flags[p] = make_uint2(2u, kLastSpecular);
        live = ps.y < f.spp && f.num_bounces > 0;
        o = { f.cam.eye.x, f.cam.eye.y, f.cam.eye.z };
        if (live) d = primary_dir(f.cam, f.width, f.height, f.frame_id, pixel, ps.y);
    }
    const uint32_t slot = warp_append(live, &fb.counts[0]);
    if (live)
    {
        store_ray(&fb.rays[0][slot], o, d, 0.0f, FLT_MAX);
        fb.path[0][slot] = p;
    }
}

// As pt_trace_quads (pathtrace.cu): the closest hits of the bounce's ray queue and the
// shadow rays of the bounce before, each ray from its scene's root.
__global__ void __launch_bounds__(kQuadBlock, kQuadMinBlocks) bp_trace_quads(batch_wf_args a, frame_buffers fb, int q,
                                                                             uint32_t bounce, uint32_t extend,
                                                                             bvh_view v, const float* bad,
                                                                             uint32_t resident,
                                                                             uint32_t* __restrict__ status)
{
    __shared__ int stack_mem[kQuadStack * kQuadBlock];
    const bool closest = extend != 0 && blockIdx.y == 0;
    const uint32_t n = closest ? fb.counts[2 * bounce] : fb.counts[2 * bounce - 1];
    const quad_work work = quad_share(blockIdx.x * (kQuadBlock / 32) + (threadIdx.x >> 5), n, resident,
                                      fb.taken + (closest ? 2 * bounce : 2 * bounce - 1));
    if (work.next >= work.end) return;
    auto index = [](uint32_t k) { return k; };
    if (closest)
        quad_trace<false, true, kQuadPathSteps>(
            stack_mem, v, bad, fb.rays[q], n, work, status,
            [&](uint32_t j) { return a.frames[a.scene[fb.path[q][j]]].root; }, index,
            [&](uint32_t j, trace_result const& h) {
                fb.hits[j] = make_uint4(uint32_t(h.tri), __float_as_uint(h.t), 0u, 0u);
            });
    else
        quad_trace<true, true, kQuadPathSteps>(
            stack_mem, v, bad, fb.shadow_rays, n, work, status,
            [&](uint32_t j) { return a.frames[a.scene[fb.shadow_path[j]]].root; }, index,
            [&](uint32_t j, trace_result const& h) { finish_shadow(fb, j, bounce - 1, h.tri >= 0); });
}

template <bool Extended>
__global__ void __launch_bounds__(kBlock, kShadeMinBlocks) bp_shade(batch_wf_args a, frame_buffers fb, int q,
                                                                    uint32_t bounce, const tri48* tris,
                                                                    int32_t num_tris, uint32_t* __restrict__ status)
{
    const uint32_t n = fb.counts[2 * bounce];
    for (uint32_t base = blockIdx.x * kBlock; base < n; base += gridDim.x * kBlock)
    {
        const uint32_t i = base + threadIdx.x;
        vertex_out out;
        out.cont = false;
        out.shadow = false;
        uint32_t p = 0;
        float epsilon = 0.0f;
        if (i < n)
        {
            p = fb.path[q][i];
            const batch_frame& f = a.frames[a.scene[p]];
            shade_params sp;
            sp.materials = a.materials;
            sp.num_materials = a.num_materials;
            sp.lights = nullptr;
            sp.num_lights = 0;
            if (a.lights)
            {
                const uint32_t s = a.scene[p], l0 = __ldg(&a.light_offsets[s]);
                sp.lights = a.lights + 4 * uint64_t(l0);
                sp.num_lights = __ldg(&a.light_offsets[s + 1]) - l0;
            }
            sp.tris = tris;
            sp.num_tris = num_tris;
            sp.epsilon = epsilon = f.epsilon;
            sp.ambient = f.ambient;
            sp.frame = f.frame_id;
            sp.sample = path_sample(fb, p).y;
            sp.bounce = bounce;
            sp.flags = f.flags;
            sp.albedo = nullptr;
            sp.emission = nullptr;
            sp.trig = a.trig;
            const float4* rp = reinterpret_cast<const float4*>(&fb.rays[q][i]);
            const float4 r0 = rp[0], r1 = rp[1];
            const uint4 hh = fb.hits[i];
            const uint2 rf = fb.rng_flags[p];
            path_state st{ xyz(fb.throughput[p]), xyz(fb.radiance[p]), rf.x, rf.y };
            shade_vertex<Extended, false>(sp, a.pixel[p], bounce, { r0.x, r0.y, r0.z }, { r0.w, r1.x, r1.y }, r1.z,
                                          r1.w, int(hh.x), __uint_as_float(hh.y), st, out, status);
            fb.throughput[p] = make_float4(st.thr.x, st.thr.y, st.thr.z, 0.0f);
            fb.radiance[p] = make_float4(st.rad.x, st.rad.y, st.rad.z, 0.0f);
            fb.rng_flags[p] = make_uint2(st.k, st.flags);
            out.cont = out.cont && bounce + 1 < f.num_bounces;
        }
        const uint32_t slot = warp_append(out.cont, &fb.counts[2 * bounce + 2]);
        if (out.cont)
        {
            store_ray(&fb.rays[q ^ 1][slot], out.next_o, out.next_d, 0.0f, FLT_MAX);
            fb.path[q ^ 1][slot] = p;
        }
        const uint32_t sslot = warp_append(out.shadow, &fb.counts[2 * bounce + 1]);
        if (out.shadow)
        {
            store_ray(&fb.shadow_rays[sslot], out.sh_o, out.sh_d, epsilon, out.sh_tmax);
            fb.shadow_path[sslot] = p;
            fb.shadow_contrib[sslot] = make_float4(out.contrib.x, out.contrib.y, out.contrib.z, 0.0f);
        }
    }
}

// The pass's samples of pixel first_pixel + i added in sample order; the pass that holds the
// pixel's last sample writes its average (rr.color += result.color, then rr.color /= spp and
// the blend with sfactor 1 and dfactor 0, as batch_pt).
__global__ void __launch_bounds__(kBlock) bp_accumulate(batch_wf_args a, frame_buffers fb, uint32_t pixels,
                                                        float4* __restrict__ images)
{
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= pixels) return;
    const uint64_t p0 = uint64_t(i) * fb.samples;
    const uint32_t s = a.scene[p0];
    const batch_frame& f = a.frames[s];
    if (fb.first_sample >= f.spp) return;
    float4 sum = fb.first_sample == 0 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : fb.sum[i];
    const uint32_t count = min(fb.samples, f.spp - fb.first_sample);
    for (uint32_t k = 0; k < count; ++k)
    {
        const float4 r = fb.radiance[p0 + k];
        const float4 c = (fb.rng_flags[p0 + k].y & kFirstHit) ? make_float4(r.x, r.y, r.z, 1.0f) : f.bg;
        sum = make_float4(sum.x + c.x, sum.y + c.y, sum.z + c.z, sum.w + c.w);
    }
    if (fb.first_sample + count < f.spp)
    {
        fb.sum[i] = sum;
        return;
    }
    const float spp = float(f.spp);
    const float4 av = make_float4(sum.x / spp, sum.y / spp, sum.z / spp, sum.w / spp);
    const float sf = 1.0f, df = 0.0f, dz = 0.0f;
    images[uint64_t(__ldg(&a.pixel_offsets[s])) + a.pixel[p0]] =
        make_float4(av.x * sf + dz * df, av.y * sf + dz * df, av.z * sf + dz * df, av.w * sf + dz * df);
}

// A pass's pixels and samples per pixel.
struct pass_shape
{
    uint32_t pixels, samples;
};

pass_shape shape_of(gbrt_batch const* b)
{
    const uint32_t pixels = uint32_t(std::min<uint64_t>(b->total_pixels, kPassPaths));
    return { pixels, uint32_t(std::min<uint64_t>(b->max_spp, kPassPaths / pixels)) };
}

} // namespace

// Where the persistent kernel is the faster one (measured against it, ms wavefront and
// persistent, one sample unless stated):
//   - Every bounce is two launches for all paths, however few are left (6 us when none is),
//     where the persistent kernel's threads end with their paths, but take a pixel's samples
//     one after the other.  Trees of 2,000 triangles in the open: 65,536 pixels 0.31 and 0.31
//     at 8 bounces, 0.39 and 0.32 at 16, 2.4 and 0.30 at 256; 1,048,576 pixels 0.84 and 0.92 at
//     16, 1.01 and 0.92 at 32; 4,194,304 pixels 2.27 and 2.86 at 32, 4.55 and 2.85 at 256;
//     4,096 pixels of 256 samples at 8 bounces 0.76 and 40.8.
//   - Small trees are not worth the queues' traffic.  4,194,304 pixels, 1, 2 and 3 bounces:
//     34 triangles (room with a blob) 0.50, 1.01, 1.61 and 0.26, 0.45, 0.71; 734 triangles 0.60,
//     1.25, 1.93 and 0.34, 0.90, 1.91; 20,494 triangles 0.90, 1.84, 2.77 and 0.79, 2.42, 4.60;
//     2,000 triangles in the open 1.02 and 1.23 at one bounce.  65,536 pixels, which do not fill
//     the GPU: 34 triangles 0.04, 0.06, 0.08 and 0.02, 0.04, 0.06; 200 in the open 0.048 and
//     0.071 at one bounce.
bool batch_wavefront_applies(gbrt_batch const* b)
{
    if (b->launch.width != 2 || b->launch.sort != 0 || b->launch.stack != uint32_t(kStackSize) || b->total_pixels == 0 ||
        b->total_inner == 0)
        return false;
    const pass_shape ps = shape_of(b);
    if (b->max_bounces > 8ull * ps.samples + uint64_t(ps.pixels) * ps.samples / (1u << 17)) return false;
    uint32_t least_triangles = b->max_bounces <= 1 ? 2048 : b->max_bounces == 2 ? 1024 : 256;
    if (ps.pixels < (1u << 19)) least_triangles = ps.samples >= 4 ? 0 : 128;
    return b->total / b->num_scenes >= least_triangles;
}

bool ensure_batch_wavefront(gbrt_context* ctx, gbrt_batch* b)
{
    auto allocate = [&](void** p, size_t bytes) {
        if (device_malloc(ctx, p, bytes) == cudaSuccess) return true;
        cudaGetLastError();
        return false;
    };
    if (!b->quads)
    {
        void* quads = nullptr;
        if (!allocate(&quads, (size_t(b->total_inner) + 1) * sizeof(quad_node))) return false;
        b->quads = static_cast<quad_node*>(quads);
    }
    const pass_shape ps = shape_of(b);
    const uint32_t n = ps.pixels * ps.samples;
    frame_buffers fb;
    const size_t bytes = layout_frame_buffers(ps.pixels, n, 2 * (b->max_bounces + 1), false, 0, nullptr, fb) +
                         2 * align256(size_t(n) * 4);
    if (b->path_bytes >= bytes) return true;
    // frames in flight may still use the old buffers
    if (b->path_buf && cudaStreamSynchronize(ctx->stream) != cudaSuccess) return false;
    cudaFree(b->path_buf);
    b->path_buf = nullptr;
    b->path_bytes = 0;
    b->graph_dirty = true;
    if (!allocate(&b->path_buf, bytes)) return false;
    b->path_bytes = bytes;
    return true;
}

gbrt_status batch_wavefront(gbrt_context* ctx, gbrt_batch* b, float* d_images, cudaStream_t s, bool force_quads)
{
    if (!b->quads || !b->path_buf) return fail(ctx, GBRT_ERR_INVALID_ARG, "batch_pathtrace: path buffers not allocated");
    const float* bad = &b->quads[b->total_inner].org[0];
    if (force_quads || b->quads_gen != b->build_gen)
    {
        GBRT_CUDA(ctx, cudaMemsetAsync(b->quads + b->total_inner, 0, sizeof(quad_node), s));
        gbrt_status st = make_quads(ctx, b->nodes, b->total_inner, b->d_inner_offsets, b->num_scenes, 0, b->quads,
                                    nullptr, s);
        if (st != GBRT_OK) return st;
        // only captured here: a graph that fails to come about has made none
        if (!is_capturing(s)) b->quads_gen = b->build_gen;
    }
    const pass_shape ps = shape_of(b);
    const uint32_t num_counts = 2 * (b->max_bounces + 1);
    frame_buffers fb;
    const size_t used = layout_frame_buffers(ps.pixels, ps.pixels * ps.samples, num_counts, false, 0, b->path_buf, fb);
    batch_wf_args a;
    a.frames = static_cast<const batch_frame*>(b->d_frames);
    a.pixel_offsets = b->d_pixel_offsets;
    a.num_scenes = b->num_scenes;
    a.order = b->launch.order;
    a.materials = b->d_materials;
    a.num_materials = b->num_materials;
    a.lights = b->num_lights > 0 ? b->d_lights : nullptr;
    a.light_offsets = b->d_light_offsets;
    a.trig = ctx->d_trig;
    a.scene = reinterpret_cast<uint32_t*>(static_cast<char*>(b->path_buf) + used);
    a.pixel = a.scene + align256(size_t(ps.pixels) * ps.samples * 4) / 4;
    bvh_view v{};
    v.nodes = b->nodes;
    v.quads = b->quads;
    v.tris = b->tris;
    v.num_inner = int32_t(b->total_inner);
    v.num_tris = int32_t(b->total);
    const uint32_t resident = uint32_t(ctx->num_sms) * kQuadMinBlocks * (kQuadBlock / 32);
    const bool lit = b->num_lights > 0;
    for (uint32_t px = 0; px < b->total_pixels; px += ps.pixels)
    {
        const uint32_t pixels = std::min(ps.pixels, b->total_pixels - px);
        fb.first_pixel = px;
        for (uint32_t smp = 0; smp < b->max_spp; smp += ps.samples)
        {
            fb.first_sample = smp;
            fb.samples = std::min(ps.samples, b->max_spp - smp);
            const uint32_t n = pixels * fb.samples, blocks = (n + kBlock - 1) / kBlock;
            const uint32_t shade_blocks = std::min(blocks, uint32_t(ctx->num_sms) * kShadeMinBlocks * 4);
            const uint32_t grid = (std::min(n, resident) + kQuadBlock / 32 - 1) / (kQuadBlock / 32);
            auto trace = [&](int q, uint32_t bounce, bool extend, bool shadow) -> gbrt_status {
                bp_trace_quads<<<dim3(grid, extend && shadow ? 2 : 1), kQuadBlock, 0, s>>>(
                    a, fb, q, bounce, extend ? 1u : 0u, v, bad, resident, ctx->d_status);
                GBRT_LAUNCH_CHECK(ctx, "bp_trace_quads");
                return GBRT_OK;
            };
            GBRT_CUDA(ctx, cudaMemsetAsync(fb.counts, 0, size_t(num_counts) * 8, s));
            bp_raygen<<<blocks, kBlock, 0, s>>>(a, fb, n);
            GBRT_LAUNCH_CHECK(ctx, "bp_raygen");
            int q = 0;
            for (uint32_t bounce = 0; bounce < b->max_bounces; ++bounce)
            {
                gbrt_status st = trace(q, bounce, true, bounce > 0 && lit);
                if (st != GBRT_OK) return st;
                auto shade = b->extended_materials ? bp_shade<true> : bp_shade<false>;
                shade<<<shade_blocks, kBlock, 0, s>>>(a, fb, q, bounce, b->tris, int32_t(b->total), ctx->d_status);
                GBRT_LAUNCH_CHECK(ctx, "bp_shade");
                q ^= 1;
            }
            if (lit && b->max_bounces > 0)
            {
                gbrt_status st = trace(q, b->max_bounces, false, true);
                if (st != GBRT_OK) return st;
            }
            bp_accumulate<<<(pixels + kBlock - 1) / kBlock, kBlock, 0, s>>>(a, fb, pixels,
                                                                          reinterpret_cast<float4*>(d_images));
            GBRT_LAUNCH_CHECK(ctx, "bp_accumulate");
        }
    }
    return GBRT_OK;
}

} // namespace gbrt
