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
// Almost all of that happens inside a block: it starts from kAggBlock consecutive leaves and
// goes in rounds over the list of subtrees made so far.  A split whose delta is larger than
// those at the outer ends of its two subtrees is their parent's, so every such pair becomes
// a node and the list is compacted; no round needs more than its neighbours' entries.  What
// is left when no pair of the block can go on -- the O(log kAggBlock) nodes that wait for a
// neighbour block -- is written to mailboxes in global memory, and a second kernel takes it
// up from there with one warp per block of the first (both sides' data written before an
// atomic on the split's flag; the second arrival reads the other side's).  No thread waits
// for another one.  In one kernel, each block's few climbing threads held its registers and
// shared memory through a chain of fences and atomics: 1,151 us for 8.4 M triangles.
//
// Measured on 8,388,608 triangles (heightfield 2048^2): a refit (these two kernels, the quads
// and a memset of the flags) 799 us, of which the first kernel 406 us at 41 % of the DRAM
// bandwidth.  With each leaf's thread climbing through atomics on shared flags (9 of 32
// lanes at work, against 23) and gathering its triangle alone it was 511 us.  Bound now by
// the barriers of the rounds and by the load/store pipe (64 %).  Rounds inside each warp
// first save barriers but lose the lanes (refit 854 -> 964 us); blocks of 128 and 512
// leaves 911 and 872 us.
#pragma once

#include "lbvh_device.cuh"
#include "traverse_core.cuh"

namespace gbrt {

// One side's data at a split: the child's box, the end of its key range away from the
// split, its height, and between blocks the delta (+ 1) at the far end.
struct __align__(16) agg_mail
{
    float4 a;   // lo.x, lo.y, lo.z, hi.x
    float4 b;   // hi.y, hi.z, far end, height | far delta << 8 (the last two as bits)
};
// Per split and scene-wide split position: left and right child.  n of these.
struct agg_slot
{
    agg_mail side[2];
};
static_assert(sizeof(agg_slot) == 64, "lbvh_scratch_layout_for counts 64 bytes per slot");

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
    height = max(__float_as_int(lm.b.w) & 0xFF, __float_as_int(rm.b.w) & 0xFF) + 1;
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

constexpr int kTriWords = sizeof(gbrt_triangle) / 4;
// Resident blocks the registers must allow (40, a spilled word in the segmented form): five
// 898 us per refit, eight 891.
constexpr int kAggMinBlocks = 6;

template <bool Segmented>
__global__ void __launch_bounds__(kAggBlock, kAggMinBlocks) agg_in_blocks(agg_args a)
{
    // The subtrees made so far, in key order: entry t of a list is the t-th one's first leaf
    // in the block | (delta at its left end + 1) << 16, and one more entry for the block's end.
    // A subtree's box and height stand at its first leaf's element (halves as separate
    // arrays: neighbouring lanes' accesses hit different banks).
    __shared__ uint32_t list[2][kAggBlock + 1];
    __shared__ float4 box_a[kAggBlock], box_b[kAggBlock];
    __shared__ int seg_lo[Segmented ? kAggBlock : 1], seg_inner[Segmented ? kAggBlock : 1];
    __shared__ uint32_t tri_words[kAggBlock / 32][32 * kTriWords];
    __shared__ uint32_t kept[kAggBlock / 32];
    __shared__ uint32_t left_over, waiting;

    const int n = int(a.n);
    const int b0 = int(blockIdx.x) * kAggBlock;
    const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
    const uint32_t full = 0xFFFFFFFFu, lanes_below = (1u << lane) - 1u;
    const int j = b0 + tid;
    const bool active = j < n;
    uint32_t m = uint32_t(n - b0 < kAggBlock ? n - b0 : kAggBlock);
    uint32_t id = 0;
    if (active)
    {
        int lo = 0, hi = n;
        if (Segmented)
        {
            const uint32_t s = upper_segment(a.offsets, a.num_scenes, uint32_t(j));
            lo = int(__ldg(&a.offsets[s]));
            hi = int(__ldg(&a.offsets[s + 1]));
            seg_lo[tid] = lo;
            seg_inner[tid] = int(__ldg(&a.inner_offsets[s]));
        }
        if (tid == 0) list[0][0] = uint32_t(neighbour_delta(a.codes, j - 1, lo, hi) + 1) << 16;
        list[0][tid + 1] = uint32_t(tid + 1) | uint32_t(neighbour_delta(a.codes, j, lo, hi) + 1) << 16;

        id = __ldg(&a.sorted_ids[j]);
        if (id >= a.n)
        {
            atomicOr(a.status, kStatusBadIndex);
            id = 0;
        }
    }
    // The warp's triangles word by word, consecutive lanes on one triangle, and out again as
    // records: an access touches the lines of three triangles, not of 32.
    uint32_t* words = tri_words[warp];
    const uint32_t* in = reinterpret_cast<const uint32_t*>(a.tris_in);
#pragma unroll
    for (int k = 0; k < kTriWords; ++k)
    {
        const int w = 32 * k + lane, t = w / kTriWords;
        words[w] = __ldg(&in[uint64_t(__shfl_sync(full, id, t)) * kTriWords + (w - kTriWords * t)]);
    }
    __syncwarp();
    {
        const float* w = reinterpret_cast<const float*>(words + kTriWords * lane);
        const tri_in t = { { w[2], w[3], w[4] }, { w[5], w[6], w[7] }, { w[8], w[9], w[10] }, 0, 0 };
        const agg_mail mine = pack_mail(tri_box(t), 0, 0);
        box_a[tid] = mine.a;
        box_b[tid] = mine.b;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        const int q = 32 * k + lane, t = q / 3, part = q - 3 * t;
        const float* w = reinterpret_cast<const float*>(words + kTriWords * t);
        const float* v = w + 2 + 3 * part;
        if (j - lane + t < n)
            reinterpret_cast<float4*>(a.tris_out + (j - lane))[q] =
                make_float4(v[0], v[1], v[2], part == 2 ? __uint_as_float(kLastInLeaf) : w[1 - part]);
    }
    if (tid == 0) waiting = 0;
    __syncthreads();

    // One round on list `cur`: where the delta between two subtrees is larger than at their
    // outer ends, they are the children of one node.  Returns whether subtree t stays on
    // the list (a right child does not), its entry in e1.
    auto round = [&](int cur, int t, uint32_t& e1) -> bool {
        if (t >= int(m)) return false;
        const uint32_t* e = list[cur] + t;
        e1 = e[0];
        const uint32_t e2 = e[1];
        const uint32_t d1 = e1 >> 16, d2 = e2 >> 16;   // + 1: 0 is no common prefix
        if (t > 0 && d1 > d2 && d1 > e[-1] >> 16) return false;
        if (t + 1 < int(m) && d2 > d1)
        {
            const uint32_t e3 = e[2], d3 = e3 >> 16;
            if (d2 > d3)
            {
                const int l = int(e1 & 0xFFFFu), mid = int(e2 & 0xFFFFu), r = int(e3 & 0xFFFFu) - 1;
                agg_mail lm = { box_a[l], box_b[l] }, rm = { box_a[mid], box_b[mid] };
                const int lo = Segmented ? seg_lo[l] : 0, inner_base = Segmented ? seg_inner[l] : 0;
                box3 box;
                int height;
                agg_make_node<Segmented>(a, lo, inner_base, b0 + l, b0 + r, b0 + mid - 1, d1 == 0 && d3 == 0, d3 > d1, lm,
                                         rm, box, height);
                const agg_mail made = pack_mail(box, 0, height);
                box_a[l] = made.a;
                box_b[l] = made.b;
            }
        }
        return true;
    };
    int cur = 0;
    bool more = true;
    while (more && m > 32)
    {
        uint32_t e1 = 0;
        const bool stays = round(cur, tid, e1);
        const uint32_t mask = __ballot_sync(full, stays);
        if (lane == 0) kept[warp] = __popc(mask);
        __syncthreads();
        const uint32_t of_lane = lane < kAggBlock / 32 ? kept[lane] : 0u;
        const uint32_t all = __reduce_add_sync(full, of_lane);
        const uint32_t at = __reduce_add_sync(full, lane < warp ? of_lane : 0u) + __popc(mask & lanes_below);
        if (stays) list[cur ^ 1][at] = e1;
        if (tid == 0) list[cur ^ 1][all] = list[cur][m];
        more = all != m;
        m = all;
        cur ^= 1;
        __syncthreads();
    }
    if (warp == 0)
    {
        while (more)
        {
            uint32_t e1 = 0;
            const bool stays = round(cur, lane, e1);
            const uint32_t mask = __ballot_sync(full, stays);
            const uint32_t all = __popc(mask);
            if (stays) list[cur ^ 1][__popc(mask & lanes_below)] = e1;
            if (lane == 0) list[cur ^ 1][all] = list[cur][m];
            more = all != m;
            m = all;
            cur ^= 1;
            __syncwarp();
        }
        if (lane == 0) left_over = m | uint32_t(cur) << 16;
    }
    __syncthreads();

    // what is left and not a root waits at a split for a node that leaves the block
    m = left_over & 0xFFFFu;
    if (uint32_t(tid) < m)
    {
        const uint32_t* e = list[left_over >> 16] + tid;
        const uint32_t d1 = e[0] >> 16, d2 = e[1] >> 16;
        if (d1 != 0 || d2 != 0)
        {
            const bool left = d2 > d1;
            const int l = int(e[0] & 0xFFFFu), end = int(e[1] & 0xFFFFu);
            const int split = b0 + (left ? end : l) - 1;
            agg_mail mail = { box_a[l], box_b[l] };
            mail.b.z = __int_as_float(left ? b0 + l : b0 + end - 1);
            mail.b.w = __int_as_float(__float_as_int(mail.b.w) | int(left ? d1 : d2) << 8);
            a.slots[split].side[left ? 0 : 1] = mail;
            a.waiting[uint64_t(blockIdx.x) * (kAggBlock + 1) + atomicAdd(&waiting, 1u)] =
                uint32_t(split) << 1 | uint32_t(left ? 0 : 1);
        }
    }
    __syncthreads();
    if (tid == 0) a.num_waiting[blockIdx.x] = waiting;
}

constexpr int kAggTopBlock = 128;

// Bound by the chain of dependent memory accesses of a step, so a step is two of them: the
// atomic, which is also the fence, and the other side's mail, which carries the delta at
// its far end.  With fences around the atomic and the deltas from the codes a refit of
// 5,003 triangles took 58.8 us, now 49.9; of 1,000,000 174 -> 153 us.
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
        int lo = 0, inner_base = 0;
        if (Segmented)
        {
            const uint32_t s = upper_segment(a.offsets, a.num_scenes, uint32_t(left ? m : m + 1));
            lo = int(__ldg(&a.offsets[s]));
            inner_base = int(__ldg(&a.inner_offsets[s]));
        }
        for (;;)
        {
            agg_slot* slot = a.slots + m;
            // releases this side's mail (the kernel before wrote the first), acquires the other's
            uint32_t seen;
            asm volatile("atom.acq_rel.gpu.global.or.b32 %0, [%1], %2;"
                         : "=r"(seen)
                         : "l"(&a.flags[m]), "r"(left ? 1u : 2u)
                         : "memory");
            if (seen == 0) break;   // the other side goes on
            const agg_mail lm = { __ldcg(&slot->side[0].a), __ldcg(&slot->side[0].b) };
            const agg_mail rm = { __ldcg(&slot->side[1].a), __ldcg(&slot->side[1].b) };
            const int l = __float_as_int(lm.b.z), r = __float_as_int(rm.b.z);
            const int pl = __float_as_int(lm.b.w) >> 8, pr = __float_as_int(rm.b.w) >> 8;   // + 1
            const bool root = pl == 0 && pr == 0;
            left = pr > pl;
            box3 b;
            int height;
            agg_make_node<Segmented>(a, lo, inner_base, l, r, m, root, left, lm, rm, b, height);
            if (root) break;
            m = left ? r : l - 1;
            a.slots[m].side[left ? 0 : 1] = pack_mail(b, left ? l : r, height | (left ? pl : pr) << 8);
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
