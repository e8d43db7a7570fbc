// Bottom-up LBVH construction from sorted Morton codes: hierarchy, boxes, node records and
// leaf triangles in one pass (lbvh.cu: one scene; batch.cu: many scenes in one
// arena).
//
// The tree is Karras' (lbvh.h:120-185, 281-330) but found from below, after Apetrei,
// "Fast and Simple Agglomerative LBVH Construction" (2014): a node over the keys [l, r]
// is the left child of its parent if the keys r, r + 1 share a longer prefix than l - 1, l,
// else the right child, and the parent is made by whichever of the two children arrives
// last at the split between them.  Karras' numbering follows without knowing the rest of
// the tree: a left child has index r, a right child index l, the root 0.  The thread that
// makes a node has both children's boxes and its index and writes the 64-byte record once.
//
// Almost all of that happens inside a block: it starts from kAggBlock consecutive leaves,
// and nodes whose keys lie in the block meet through shared memory.  What is left when no
// thread of the block can go on -- the O(log kAggBlock) nodes that wait for a neighbour
// block -- is written to mailboxes in global memory, and a second kernel takes it up from
// there with one warp per block of the first (both sides' data written before an atomic on
// the split's flag; the second arrival reads the other side's).  No thread waits for
// another one.  In one kernel, each block's few climbing threads held its registers and
// shared memory through a chain of fences and atomics: 1,151 us for 8.4 M triangles.
//
// Measured on 8,388,608 triangles (heightfield 2048^2): in-place rebuild 1.76 -> 1.11 ms;
// a refit (these two kernels and a memset of the flags) 0.67 ms.  Bound by the load/store
// pipe (56 %: the triangle gather, 112 B of stores per triangle, the mail in shared memory)
// and by the divergence of the climb (9 of 32 lanes, issue slots 44 %).
#pragma once

#include "lbvh_device.cuh"
#include "traverse_core.cuh"

namespace gbrt {

constexpr int kAggBlock = 512;

// One side's data at a split: the child's box, the end of its key range away from the
// split, and its height.
struct __align__(16) agg_mail
{
    float4 a;   // lo.x, lo.y, lo.z, hi.x
    float4 b;   // hi.y, hi.z, far end, height (the last two as bits)
};
// Per split and scene-wide split position: left and right child.  n of these.
struct agg_slot
{
    agg_mail side[2];
};

struct agg_args
{
    gbrt_triangle const* tris_in;
    const uint32_t* sorted_ids;
    const uint32_t* codes;
    uint32_t n;
    // segmented: scene s owns the leaves [offsets[s], offsets[s + 1]) and the inner nodes
    // from inner_offsets[s]
    const uint32_t* offsets;
    const uint32_t* inner_offsets;
    uint32_t num_scenes;
    bvh2_node* nodes;
    int2* ranges;            // null, or the leaf range of every inner node
    agg_slot* slots;         // n
    uint32_t* flags;         // n, zero
    // nodes of block b that wait for another block: waiting[b * (kAggBlock + 1) ...], each
    // (split << 1) | side, and their number
    uint32_t* waiting;
    uint32_t* num_waiting;
    tri48* tris_out;
    uint32_t* root_height;   // the root's height (segmented: the largest by atomicMax)
    uint32_t* status;
};

// A 44-byte triangle at a 4-byte aligned address as five 64-bit loads and one 32-bit one
// (the words before or after the 8-byte aligned ones): half the load instructions, and
// every one of them touches another line per lane when the triangles are gathered.
__device__ __forceinline__ tri_in load_tri_gather(gbrt_triangle const* __restrict__ tris, uint64_t i)
{
    const uint32_t* w = reinterpret_cast<const uint32_t*>(tris + i);
    const bool odd = (reinterpret_cast<uintptr_t>(w) & 4u) != 0;
    const uint2* p = reinterpret_cast<const uint2*>(w + (odd ? 1 : 0));
    const uint2 v0 = __ldg(p), v1 = __ldg(p + 1), v2 = __ldg(p + 2), v3 = __ldg(p + 3), v4 = __ldg(p + 4);
    const uint32_t s = __ldg(w + (odd ? 0 : 10));
    tri_in t;
    t.geom_id = odd ? s : v0.x;
    t.prim_id = odd ? v0.x : v0.y;
    t.v1 = { __uint_as_float(odd ? v0.y : v1.x), __uint_as_float(odd ? v1.x : v1.y), __uint_as_float(odd ? v1.y : v2.x) };
    t.e1 = { __uint_as_float(odd ? v2.x : v2.y), __uint_as_float(odd ? v2.y : v3.x), __uint_as_float(odd ? v3.x : v3.y) };
    t.e2 = { __uint_as_float(odd ? v3.y : v4.x), __uint_as_float(odd ? v4.x : v4.y), __uint_as_float(odd ? v4.y : s) };
    return t;
}

__device__ __forceinline__ agg_mail pack_mail(box3 const& b, int far_end, int height)
{
    return { make_float4(b.lo.x, b.lo.y, b.lo.z, b.hi.x),
             make_float4(b.hi.y, b.hi.z, __int_as_float(far_end), __int_as_float(height)) };
}

// Common-prefix length of the neighbouring sorted keys j and j + 1 of the segment [lo, hi)
// (Karras' delta, with segment-local indices as the tie-break), -1 across its ends.
__device__ __forceinline__ int neighbour_delta(const uint32_t* __restrict__ codes, int j, int lo, int hi)
{
    if (j < lo || j + 1 >= hi) return -1;
    const uint32_t x = __ldg(&codes[j]) ^ __ldg(&codes[j + 1]);
    return x == 0 ? 32 + __clz(uint32_t(j - lo) ^ uint32_t(j + 1 - lo)) : __clz(x);
}

// Words of agg_args::waiting and num_waiting for n leaves.
constexpr uint64_t agg_blocks(uint64_t n) { return (n + kAggBlock - 1) / kAggBlock; }
constexpr uint64_t agg_waiting_words(uint64_t n) { return agg_blocks(n) * (kAggBlock + 2); }

__device__ __forceinline__ void store8(void* p, float a, float b, float c, float d, float e, float f, float g, float h)
{
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d), "f"(e),
                 "f"(f), "f"(g), "f"(h)
                 : "memory");
}

// The node over [l, r] whose children are the left one up to split m and the right one, in
// the segment that starts at leaf lo and at inner node inner_base: its record; its box in
// `b`, its height in `height`.
template <bool Segmented>
__device__ __forceinline__ void agg_make_node(agg_args const& a, int lo, int inner_base, int l, int r, int m, bool root,
                                              bool is_left, agg_mail const& lm, agg_mail const& rm, box3& b,
                                              int& height)
{
    const int index = inner_base + (root ? 0 : (is_left ? r : l) - lo);
    height = max(__float_as_int(lm.b.w), __float_as_int(rm.b.w)) + 1;
    const int cl = l == m ? ~m : inner_base + (m - lo);
    const int cr = m + 1 == r ? ~r : inner_base + (m + 1 - lo);
    // xy0, xy1 | z01, link: two 256-bit stores
    store8(a.nodes + index, lm.a.x, lm.a.w, lm.a.y, lm.b.x, rm.a.x, rm.a.w, rm.a.y, rm.b.x);
    store8(reinterpret_cast<char*>(a.nodes + index) + 32, lm.a.z, lm.b.y, rm.a.z, rm.b.y, __int_as_float(cl),
           __int_as_float(cr), __int_as_float(height), __int_as_float(-1));
    if (a.ranges) a.ranges[index] = make_int2(l, r);
    b = box_union_cas({ { lm.a.x, lm.a.y, lm.a.z }, { lm.a.w, lm.b.x, lm.b.y } },
                      { { rm.a.x, rm.a.y, rm.a.z }, { rm.a.w, rm.b.x, rm.b.y } });
    if (root)
    {
        if (Segmented)
            atomicMax(a.root_height, uint32_t(height));
        else
            *a.root_height = uint32_t(height);
    }
}

template <bool Segmented>
__global__ void __launch_bounds__(kAggBlock) agg_in_blocks(agg_args a)
{
    // split kk of the block is the one between its leaves b0 + kk - 1 and b0 + kk; kk = 0 and
    // kAggBlock are the block's ends
    // (mail halves as separate arrays: neighbouring lanes' accesses hit different banks)
    __shared__ float4 mail_a[2][kAggBlock + 1], mail_b[2][kAggBlock + 1];
    __shared__ uint32_t flags[kAggBlock + 1];
    __shared__ int delta[kAggBlock + 1];
    __shared__ uint32_t waiting;

    const int n = int(a.n);
    const int b0 = int(blockIdx.x) * kAggBlock;
    const int tid = int(threadIdx.x);
    const int j = b0 + tid;
    int lo = 0, hi = n, inner_base = 0;
    bool active = j < n;
    if (Segmented && active)
    {
        const uint32_t s = upper_segment(a.offsets, a.num_scenes, uint32_t(j));
        lo = int(__ldg(&a.offsets[s]));
        hi = int(__ldg(&a.offsets[s + 1]));
        inner_base = int(__ldg(&a.inner_offsets[s]));
    }
    for (int k = tid; k <= kAggBlock; k += kAggBlock) flags[k] = 0;
    if (active)
    {
        if (tid == 0) delta[0] = neighbour_delta(a.codes, j - 1, lo, hi);
        delta[tid + 1] = neighbour_delta(a.codes, j, lo, hi);
    }

    box3 box;
    if (active)
    {
        uint32_t id = __ldg(&a.sorted_ids[j]);
        if (id >= a.n)
        {
            atomicOr(a.status, kStatusBadIndex);
            id = 0;
        }
        const tri_in t = load_tri_gather(a.tris_in, id);
        float4* o = reinterpret_cast<float4*>(a.tris_out + j);
        o[0] = make_float4(t.v1.x, t.v1.y, t.v1.z, __uint_as_float(t.prim_id));
        o[1] = make_float4(t.e1.x, t.e1.y, t.e1.z, __uint_as_float(t.geom_id));
        o[2] = make_float4(t.e2.x, t.e2.y, t.e2.z, __uint_as_float(kLastInLeaf));
        box = tri_box(t);
    }
    __syncthreads();

    // inside the block
    if (active && hi - lo > 1)
    {
        int l = j, r = j, height = 0;
        for (;;)
        {
            const int dl = delta[l - b0], dr = delta[r - b0 + 1];
            const bool left = dr > dl;
            const int kk = left ? r - b0 + 1 : l - b0;
            const agg_mail mine = pack_mail(box, left ? l : r, height);
            mail_a[left ? 0 : 1][kk] = mine.a;
            mail_b[left ? 0 : 1][kk] = mine.b;
            __threadfence_block();
            if (atomicOr(&flags[kk], left ? 1u : 2u) == 0) break;   // the other side goes on
            __threadfence_block();
            const agg_mail other = { mail_a[left ? 1 : 0][kk], mail_b[left ? 1 : 0][kk] };
            const agg_mail lm = left ? mine : other, rm = left ? other : mine;
            const int m = b0 + kk - 1;
            l = __float_as_int(lm.b.z);
            r = __float_as_int(rm.b.z);
            const int pl = delta[l - b0], pr = delta[r - b0 + 1];
            const bool root = pl < 0 && pr < 0;
            agg_make_node<Segmented>(a, lo, inner_base, l, r, m, root, pr > pl, lm, rm, box, height);
            if (root) break;
        }
    }
    if (tid == 0) waiting = 0;
    __syncthreads();

    // the nodes that wait at a split for a node that leaves the block
    for (int kk = tid; kk <= kAggBlock; kk += kAggBlock)
    {
        const uint32_t f = flags[kk];
        if (f != 1u && f != 2u) continue;
        const int side = f == 1u ? 0 : 1, m = b0 + kk - 1;
        a.slots[m].side[side] = { mail_a[side][kk], mail_b[side][kk] };
        a.waiting[uint64_t(blockIdx.x) * (kAggBlock + 1) + atomicAdd(&waiting, 1u)] = uint32_t(m) << 1 | uint32_t(side);
    }
    __syncthreads();
    if (tid == 0) a.num_waiting[blockIdx.x] = waiting;
}

constexpr int kAggTopBlock = 128;

template <bool Segmented>
__global__ void __launch_bounds__(kAggTopBlock) agg_across_blocks(agg_args a, uint32_t num_blocks)
{
    const uint32_t block = blockIdx.x * (kAggTopBlock / 32) + (threadIdx.x >> 5);
    if (block >= num_blocks) return;
    const uint32_t count = min(a.num_waiting[block], uint32_t(kAggBlock + 1));
    for (uint32_t i = threadIdx.x & 31u; i < count; i += 32)
    {
        const uint32_t w = a.waiting[uint64_t(block) * (kAggBlock + 1) + i];
        int m = int(w >> 1);
        bool left = !(w & 1u);
        int lo = 0, hi = int(a.n), inner_base = 0;
        if (Segmented)
        {
            const uint32_t s = upper_segment(a.offsets, a.num_scenes, uint32_t(left ? m : m + 1));
            lo = int(__ldg(&a.offsets[s]));
            hi = int(__ldg(&a.offsets[s + 1]));
            inner_base = int(__ldg(&a.inner_offsets[s]));
        }
        // (the mail written by the kernel before needs no fence)
        for (;;)
        {
            agg_slot* slot = a.slots + m;
            if (atomicOr(&a.flags[m], left ? 1u : 2u) == 0) break;   // the other side goes on
            __threadfence();
            const agg_mail lm = { __ldcg(&slot->side[0].a), __ldcg(&slot->side[0].b) };
            const agg_mail rm = { __ldcg(&slot->side[1].a), __ldcg(&slot->side[1].b) };
            const int l = __float_as_int(lm.b.z), r = __float_as_int(rm.b.z);
            const int pl = neighbour_delta(a.codes, l - 1, lo, hi), pr = neighbour_delta(a.codes, r, lo, hi);
            const bool root = pl < 0 && pr < 0;
            left = pr > pl;
            box3 b;
            int height;
            agg_make_node<Segmented>(a, lo, inner_base, l, r, m, root, left, lm, rm, b, height);
            if (root) break;
            m = left ? r : l - 1;
            a.slots[m].side[left ? 0 : 1] = pack_mail(b, left ? l : r, height);
            __threadfence();
        }
    }
}

// Both kernels on `stream`.
template <bool Segmented>
inline gbrt_status agglomerate(gbrt_context* ctx, agg_args const& a, cudaStream_t stream)
{
    const uint32_t blocks = uint32_t(agg_blocks(a.n));
    agg_in_blocks<Segmented><<<blocks, kAggBlock, 0, stream>>>(a);
    GBRT_LAUNCH_CHECK(ctx, "agg_in_blocks");
    if (blocks > 1)
    {
        agg_across_blocks<Segmented><<<(blocks + kAggTopBlock / 32 - 1) / (kAggTopBlock / 32), kAggTopBlock, 0, stream>>>(
            a, blocks);
        GBRT_LAUNCH_CHECK(ctx, "agg_across_blocks");
    }
    return GBRT_OK;
}

} // namespace gbrt
