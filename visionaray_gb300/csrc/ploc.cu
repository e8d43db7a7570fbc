// High-quality BVH build by parallel locally-ordered clustering (PLOC: D. Meister and
// J. Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume Hierarchy
// Construction", IEEE TVCG 24(3), 2018).  Not a visionaray builder: the reference's GPU
// builder is the LBVH (lbvh.cu), whose Morton splits cost the heightfield rays about
// 1.8x the node visits of its binned-SAH tree; this build reaches SAH-like trees on the
// GPU in a few milliseconds and feeds the same node-pair traversal.
//
// Clusters start as the triangles in Morton order (the LBVH's first stages).  Each
// iteration, every cluster finds the neighbour within kRadius positions whose union box
// has the smallest surface area (ties to the lower index); mutual nearest neighbours
// merge into a new node pair at the lower position, and a prefix sum compacts the
// surviving clusters in order and numbers the new nodes.  Iterations repeat until one
// cluster -- the root -- is left.  Node pairs carry both children's boxes, parent links
// and subtree heights, so refits and every traversal kernel apply unchanged; the leaf
// triangles are the Morton-ordered tri48 records of the LBVH.
//
// An iteration is two launches (ploc_nearest, ploc_merge); how many clusters are left stays
// on the device, and the host looks at it two iterations late, while the next ones run.
// The last kTail clusters take more than half of the iterations: one block does them all in
// shared memory (ploc_tail).  982,802 heightfield triangles: 55 iterations of 5 or 7
// launches and a synchronisation each took 2.1 ms, bound by the host, now 0.6 ms.

#include "lbvh_device.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace gbrt {
namespace {

constexpr int kBlock = 256;
constexpr int kRadius = 16;   // neighbours searched on each side

// Clusters per tile of an iteration.  A ploc_nearest block searches its tile and kRadius
// positions on each side, so that it knows which of its own pairs are mutual, four adjacent
// clusters per thread: they share most of their 36 neighbours' boxes, whose reads from
// shared memory bounded the search (982,802 clusters: one per thread 60.8 us, two 36.7, four
// 29.4; 10,000 are 2 us faster with two, which does not show beside the launches).
constexpr int kTile = 608;
constexpr int kSearch = kTile + 2 * kRadius;
constexpr int kItems = 4;
constexpr int kSearchThreads = kSearch / kItems;
constexpr int kStage = kTile + 4 * kRadius;
// Tiles per group of the prefix sum: a ploc_merge block adds up the groups before its own
// and the tiles before it in the group.
constexpr uint32_t kGroup = 64;
// Clusters that one block finishes, two per thread while there are more than threads.  Its
// first iteration is about as long as two launches.
constexpr int kTail = 2048;
constexpr int kTailThreads = 1024;

// Where the clustering stands, read by an iteration and written for the next one.
struct ploc_state
{
    uint32_t clusters, nodes;   // left, made
    uint32_t stuck;             // an iteration merged nothing
};

// Elements of a staged box array, padded so that lanes four (or two) apart read different
// banks.
__host__ __device__ constexpr int padded(int e) { return e + (e >> 3); }

inline uint32_t blocks_for(uint64_t n) { return uint32_t((n + kBlock - 1) / kBlock); }
inline size_t align_up(size_t v) { return (v + 255) & ~size_t(255); }

// Leaf clusters: the box of the j-th triangle in Morton order (id ~j, height 0), and
// that triangle's tri48 record.  Also starts the state and clears the groups' sums.
__global__ void __launch_bounds__(kBlock) ploc_leaves(gbrt_triangle const* __restrict__ tris_in,
                                                      const uint32_t* __restrict__ sorted_ids, uint32_t n,
                                                      float4* __restrict__ lo, float4* __restrict__ hi,
                                                      tri48* __restrict__ tris_out, ploc_state* __restrict__ state,
                                                      unsigned long long* __restrict__ groups, uint32_t num_groups,
                                                      uint32_t* __restrict__ status)
{
    uint32_t j = blockIdx.x * kBlock + threadIdx.x;
    if (j >= n) return;
    if (j == 0) *state = { n, 0, 0 };
    if (j < num_groups) groups[j] = 0;
    uint32_t id = __ldg(&sorted_ids[j]);
    if (id >= n)
    {
        atomicOr(status, kStatusBadIndex);
        id = 0;
    }
    tri_in t = load_tri(tris_in, id);
    tri48 o;
    o.t0 = make_float4(t.v1.x, t.v1.y, t.v1.z, __uint_as_float(t.prim_id));
    o.t1 = make_float4(t.e1.x, t.e1.y, t.e1.z, __uint_as_float(t.geom_id));
    o.t2 = make_float4(t.e2.x, t.e2.y, t.e2.z, __uint_as_float(kLastInLeaf));
    tris_out[j] = o;
    box3 b = tri_box(t);
    lo[j] = make_float4(b.lo.x, b.lo.y, b.lo.z, __int_as_float(~int(j)));
    hi[j] = make_float4(b.hi.x, b.hi.y, b.hi.z, __int_as_float(0));
}

__device__ __forceinline__ float union_area(float4 alo, float4 ahi, float4 blo, float4 bhi)
{
    float dx = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x);
    float dy = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y);
    float dz = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
    return dx * dy + dy * dz + dz * dx;
}

// The kItems adjacent clusters from stage element e0, each against its neighbours in
// ascending order (a tie keeps the lower one): the stage elements of the nearest, -1 for none.
// Elements outside the clusters are boxes from -inf to inf, which are nobody's nearest.
template <int Items>
__device__ __forceinline__ void nearest_of(const float4* __restrict__ slo, const float4* __restrict__ shi, int e0,
                                           int nearest[Items])
{
    float4 alo[Items], ahi[Items];
    float best[Items];
#pragma unroll
    for (int r = 0; r < Items; ++r)
    {
        alo[r] = slo[padded(e0 + r)];
        ahi[r] = shi[padded(e0 + r)];
        best[r] = FLT_MAX;
        nearest[r] = -1;
    }
    auto against = [&](int r, int e, float4 const& blo, float4 const& bhi) {
        const float a = union_area(alo[r], ahi[r], blo, bhi);
        if (a < best[r])
        {
            best[r] = a;
            nearest[r] = e;
        }
    };
#pragma unroll
    for (int k = 0; k < Items - 1; ++k)   // neighbours of the first items only
    {
        const int e = e0 - kRadius + k;
        const float4 blo = slo[padded(e)], bhi = shi[padded(e)];
#pragma unroll
        for (int r = 0; r <= k; ++r) against(r, e, blo, bhi);
    }
    for (int e = e0 + Items - 1 - kRadius; e < e0; ++e)
    {
        const float4 blo = slo[padded(e)], bhi = shi[padded(e)];
#pragma unroll
        for (int r = 0; r < Items; ++r) against(r, e, blo, bhi);
    }
#pragma unroll
    for (int k = 0; k < Items; ++k)
    {
#pragma unroll
        for (int r = 0; r < Items; ++r)
            if (r != k) against(r, e0 + k, alo[k], ahi[k]);
    }
    for (int e = e0 + Items; e <= e0 + kRadius; ++e)
    {
        const float4 blo = slo[padded(e)], bhi = shi[padded(e)];
#pragma unroll
        for (int r = 0; r < Items; ++r) against(r, e, blo, bhi);
    }
#pragma unroll
    for (int k = 1; k < Items; ++k)   // of the last items only
    {
        const int e = e0 + kRadius + k;
        const float4 blo = slo[padded(e)], bhi = shi[padded(e)];
#pragma unroll
        for (int r = k; r < Items; ++r) against(r, e, blo, bhi);
    }
}

__device__ __forceinline__ void stage_outside(float4& lo, float4& hi)
{
    const float inf = __int_as_float(0x7F800000);
    lo = make_float4(-inf, -inf, -inf, 0.0f);
    hi = make_float4(inf, inf, inf, 0.0f);
}

// Nearest neighbour of every cluster within kRadius positions (smallest union area), and
// the merges (high half) and surviving clusters (low half) of every tile and group of
// tiles.  A cluster merges (and owns the new node) when its nearest neighbour is mutual
// and lies after it; it disappears when the mutual neighbour lies before it.
__global__ void __launch_bounds__(kSearchThreads) ploc_nearest(const float4* __restrict__ lo,
                                                               const float4* __restrict__ hi,
                                                               const ploc_state* __restrict__ state,
                                                               int* __restrict__ nn,
                                                               unsigned long long* __restrict__ tiles,
                                                               unsigned long long* __restrict__ groups)
{
    __shared__ float4 slo[padded(kStage)];
    __shared__ float4 shi[padded(kStage)];
    __shared__ int snn[kSearch];
    __shared__ uint32_t counts[2];
    const int64_t m = state->clusters;
    const int64_t b0 = int64_t(blockIdx.x) * kTile;
    if (b0 >= m || m <= kTail) return;
    if (threadIdx.x < 2) counts[threadIdx.x] = 0;
    for (int e = threadIdx.x; e < kStage; e += kSearchThreads)
    {
        const int64_t g = b0 - 2 * kRadius + e;
        float4 l, h;
        stage_outside(l, h);
        if (g >= 0 && g < m)
        {
            l = lo[g];
            h = hi[g];
        }
        slo[padded(e)] = l;
        shi[padded(e)] = h;
    }
    __syncthreads();
    {
        // element x of snn is cluster b0 - kRadius + x, stage element x + kRadius
        const int x = int(threadIdx.x) * kItems;
        int nearest[kItems];
        nearest_of<kItems>(slo, shi, x + kRadius, nearest);
#pragma unroll
        for (int r = 0; r < kItems; ++r) snn[x + r] = nearest[r] >= 0 ? nearest[r] - kRadius : -1;
    }
    __syncthreads();
    uint32_t merges = 0, keeps = 0;
    for (int k = threadIdx.x; k < kTile && b0 + k < m; k += kSearchThreads)
    {
        const int x = k + kRadius, j = snn[x];
        const bool mutual = j >= 0 && snn[j] == x;
        nn[b0 + k] = j >= 0 ? int(b0 + j - kRadius) : -1;
        merges += mutual && x < j;
        keeps += !(mutual && x > j);
    }
    merges = __reduce_add_sync(0xFFFFFFFFu, merges);
    keeps = __reduce_add_sync(0xFFFFFFFFu, keeps);
    if ((threadIdx.x & 31) == 0)
    {
        atomicAdd(&counts[0], merges);
        atomicAdd(&counts[1], keeps);
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        const unsigned long long sum = (static_cast<unsigned long long>(counts[0]) << 32) | counts[1];
        tiles[blockIdx.x] = sum;
        atomicAdd(&groups[blockIdx.x / kGroup], sum);
    }
}

// The node pair of clusters a and b (boxes with the id in lo.w and the height in hi.w); a
// becomes the merged cluster.
__device__ __forceinline__ bool make_pair(float4& alo, float4& ahi, float4 const& blo, float4 const& bhi, uint32_t node,
                                          uint32_t num_inner, bvh2_node* __restrict__ nodes,
                                          uint32_t* __restrict__ status)
{
    const int ca = __float_as_int(alo.w), cb = __float_as_int(blo.w);
    if (node >= num_inner || ca >= int(node) || cb >= int(node))   // children were made in earlier steps
    {
        atomicOr(status, kStatusBadIndex);
        return false;
    }
    const int height = max(__float_as_int(ahi.w), __float_as_int(bhi.w)) + 1;
    bvh2_node nd;
    nd.xy0 = make_float4(alo.x, ahi.x, alo.y, ahi.y);
    nd.xy1 = make_float4(blo.x, bhi.x, blo.y, bhi.y);
    nd.z01 = make_float4(alo.z, ahi.z, blo.z, bhi.z);
    nd.link = make_int4(ca, cb, height, -1);
    nodes[node] = nd;
    if (ca >= 0) nodes[ca].link.w = int(node << 1) | 0;
    if (cb >= 0) nodes[cb].link.w = int(node << 1) | 1;
    // merged as the LBVH merges (NaN and outward infinities of a leaf box skipped)
    alo = make_float4(ref_min(cas_lo(alo.x), cas_lo(blo.x)), ref_min(cas_lo(alo.y), cas_lo(blo.y)),
                      ref_min(cas_lo(alo.z), cas_lo(blo.z)), __int_as_float(int(node)));
    ahi = make_float4(ref_max(cas_hi(ahi.x), cas_hi(bhi.x)), ref_max(cas_hi(ahi.y), cas_hi(bhi.y)),
                      ref_max(cas_hi(ahi.z), cas_hi(bhi.z)), __int_as_float(height));
    return true;
}

// One clustering step: merging clusters create the next node pairs in order, survivors are
// compacted in order into (out_lo, out_hi).  With kTail clusters or fewer left the step
// only copies them, since the host may launch a few steps too many.  The block of the last
// tile writes the next state, for the host too; block 0 clears the next step's group sums.
__global__ void __launch_bounds__(kTile) ploc_merge(const float4* __restrict__ lo, const float4* __restrict__ hi,
                                                    const int* __restrict__ nn, const ploc_state* __restrict__ state,
                                                    ploc_state* __restrict__ next,
                                                    const unsigned long long* __restrict__ tiles,
                                                    const unsigned long long* __restrict__ groups,
                                                    unsigned long long* __restrict__ next_groups, uint32_t num_groups,
                                                    uint32_t num_inner, bvh2_node* __restrict__ nodes,
                                                    float4* __restrict__ out_lo, float4* __restrict__ out_hi,
                                                    uint32_t* __restrict__ host_clusters,
                                                    uint32_t* __restrict__ status)
{
    __shared__ unsigned long long warp_before[kTile / 32];
    __shared__ uint32_t warp_own[kTile / 32];
    const ploc_state now = *state;
    const int64_t m = now.clusters;
    const int64_t b0 = int64_t(blockIdx.x) * kTile;
    if (blockIdx.x == 0)
        for (uint32_t k = threadIdx.x; k < num_groups; k += kTile) next_groups[k] = 0;
    const int64_t i = b0 + threadIdx.x;
    if (m <= kTail)
    {
        if (i < m)
        {
            out_lo[i] = lo[i];
            out_hi[i] = hi[i];
        }
        if (i == 0) *next = now;
        return;
    }
    if (b0 >= m) return;
    const int j = i < m ? nn[i] : -1;
    const bool mutual = j >= 0 && j < m && nn[j] == int(i);
    const bool merges = mutual && i < j, keeps = i < m && !(mutual && i > j);
    // (merges << 32 | survivors) of the tiles before this one
    unsigned long long before = 0;
    const uint32_t group = blockIdx.x / kGroup;
    for (uint32_t g = threadIdx.x; g < group; g += kTile) before += groups[g];
    if (group * kGroup + threadIdx.x < blockIdx.x) before += tiles[group * kGroup + threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lanes_below = (1u << lane) - 1u;
    const uint32_t mm = __ballot_sync(0xFFFFFFFFu, merges), kk = __ballot_sync(0xFFFFFFFFu, keeps);
    if (lane == 0)
    {
        warp_before[warp] = before;
        warp_own[warp] = uint32_t(__popc(mm)) << 16 | uint32_t(__popc(kk));
    }
    __syncthreads();
    before = 0;
    uint32_t own = 0, all = 0;
    for (int w = 0; w < kTile / 32; ++w)
    {
        before += warp_before[w];
        all += warp_own[w];
        if (w < warp) own += warp_own[w];
    }
    if (threadIdx.x == 0 && b0 + kTile >= m)
    {
        const uint32_t made = uint32_t(before >> 32) + (all >> 16), left = uint32_t(before) + (all & 0xFFFFu);
        *next = { made ? left : 0u, now.nodes + made, made ? 0u : 1u };
        *host_clusters = made ? left : 0u;
    }
    if (!keeps) return;
    float4 alo = lo[i], ahi = hi[i];
    if (merges)
    {
        const uint32_t node = now.nodes + uint32_t(before >> 32) + (own >> 16) + uint32_t(__popc(mm & lanes_below));
        if (!make_pair(alo, ahi, lo[j], hi[j], node, num_inner, nodes, status)) return;
    }
    const uint32_t dst = uint32_t(before) + (own & 0xFFFFu) + uint32_t(__popc(kk & lanes_below));
    out_lo[dst] = alo;
    out_hi[dst] = ahi;
}

// One step of m clusters in shared memory (cluster k at element k + kRadius), Items per
// thread.  Returns (merges << 16 | survivors).
template <int Items>
__device__ __forceinline__ uint32_t tail_step(float4* slo, float4* shi, int* snn, uint32_t* warp_own, int m,
                                              uint32_t made, uint32_t num_inner, bvh2_node* __restrict__ nodes,
                                              uint32_t* __restrict__ status)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k0 = int(threadIdx.x) * Items;
    if (k0 < m)
    {
        int nearest[Items];
        nearest_of<Items>(slo, shi, k0 + kRadius, nearest);
#pragma unroll
        for (int r = 0; r < Items; ++r) snn[k0 + r] = nearest[r] >= 0 ? nearest[r] - kRadius : -1;
    }
    __syncthreads();
    int other[Items];
    uint32_t what[Items], mine = 0;   // as the return value, of one cluster
#pragma unroll
    for (int r = 0; r < Items; ++r)
    {
        const int k = k0 + r;
        other[r] = k < m ? snn[k] : -1;
        const bool mutual = other[r] >= 0 && snn[other[r]] == k;
        what[r] = (mutual && k < other[r] ? 1u << 16 : 0u) + (k < m && !(mutual && k > other[r]) ? 1u : 0u);
        mine += what[r];
    }
    uint32_t incl = mine;
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_own[warp] = incl;
    __syncthreads();
    const uint32_t of_lane = warp_own[lane];   // kTailThreads / 32 == 32 warps
    const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, of_lane);
    uint32_t at = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? of_lane : 0u) + incl - mine;
    float4 alo[Items], ahi[Items];
    uint32_t dst[Items];
#pragma unroll
    for (int r = 0; r < Items; ++r)
    {
        dst[r] = at & 0xFFFFu;
        if (what[r] & 1u)
        {
            alo[r] = slo[padded(k0 + r + kRadius)];
            ahi[r] = shi[padded(k0 + r + kRadius)];
            if (what[r] >> 16)
                make_pair(alo[r], ahi[r], slo[padded(other[r] + kRadius)], shi[padded(other[r] + kRadius)],
                          made + (at >> 16), num_inner, nodes, status);
        }
        at += what[r];
    }
    __syncthreads();
    const int left = int(all & 0xFFFFu);
#pragma unroll
    for (int r = 0; r < Items; ++r)
    {
        const int k = k0 + r;
        if (what[r] & 1u)
        {
            slo[padded(int(dst[r]) + kRadius)] = alo[r];
            shi[padded(int(dst[r]) + kRadius)] = ahi[r];
        }
        if (k >= left && k < m) stage_outside(slo[padded(k + kRadius)], shi[padded(k + kRadius)]);
    }
    __syncthreads();
    return all;
}

// Every step from kTail or fewer clusters to the root, in one block, and the report.
constexpr size_t kTailBytes = 2 * size_t(padded(kTail + 2 * kRadius)) * sizeof(float4);

__global__ void __launch_bounds__(kTailThreads) ploc_tail(const float4* __restrict__ lo, const float4* __restrict__ hi,
                                                          const ploc_state* __restrict__ state, uint32_t num_inner,
                                                          bvh2_node* __restrict__ nodes,
                                                          build_result* __restrict__ report,
                                                          uint32_t* __restrict__ status)
{
    extern __shared__ float4 tail_mem[];
    float4* slo = tail_mem;
    float4* shi = tail_mem + padded(kTail + 2 * kRadius);
    __shared__ int snn[kTail];
    __shared__ uint32_t warp_own[kTailThreads / 32];
    int m = int(state->clusters);
    uint32_t made = state->nodes;
    bool stuck = state->stuck != 0 || m > kTail;
    for (int e = threadIdx.x; e < kTail + 2 * kRadius; e += kTailThreads)
    {
        float4 l, h;
        stage_outside(l, h);
        if (!stuck && e >= kRadius && e - kRadius < m)
        {
            l = lo[e - kRadius];
            h = hi[e - kRadius];
        }
        slo[padded(e)] = l;
        shi[padded(e)] = h;
    }
    __syncthreads();
    while (!stuck && m > 1)
    {
        const uint32_t step = m > kTailThreads ? tail_step<2>(slo, shi, snn, warp_own, m, made, num_inner, nodes, status)
                                               : tail_step<1>(slo, shi, snn, warp_own, m, made, num_inner, nodes, status);
        made += step >> 16;
        stuck = step >> 16 == 0;
        m = int(step & 0xFFFFu);
    }
    if (threadIdx.x == 0)
    {
        const float4 l = slo[padded(kRadius)], h = shi[padded(kRadius)];
        report->lo[0] = l.x, report->lo[1] = l.y, report->lo[2] = l.z;
        report->hi[0] = h.x, report->hi[1] = h.y, report->hi[2] = h.z;
        report->root = __float_as_int(l.w);
        report->height = uint32_t(__float_as_int(h.w));
        report->made = made;
        report->stuck = stuck ? 1u : 0u;
    }
}

// Steps between a launch and the host's look at the cluster count: the GPU has two queued
// while it looks, and at most that many run on kTail clusters for nothing.
constexpr uint32_t kLate = 2;

struct event_ring
{
    cudaEvent_t events[kLate + 1] = {};
    ~event_ring()
    {
        for (cudaEvent_t e : events)
            if (e) cudaEventDestroy(e);
    }
    cudaError_t at(uint32_t i, cudaEvent_t** out)
    {
        *out = &events[i % (kLate + 1)];
        return **out ? cudaSuccess : cudaEventCreateWithFlags(*out, cudaEventDisableTiming);
    }
};

} // namespace

gbrt_status build_ploc(gbrt_context* ctx, gbrt_triangle const* d_tris, uint32_t n, gbrt_bvh* bvh)
{
    bvh->kind = bvh_kind::ploc;
    bvh->num_prims = n;
    bvh->num_inner = n > 0 ? n - 1 : 0;
    bvh->root = n > 1 ? int32_t(n - 2) : ~0;
    bvh->height = 0;
    if (n == 0) return GBRT_OK;
    cudaStream_t s = ctx->stream;
    gbrt_status st = alloc_tree(ctx, bvh, n);
    if (st != GBRT_OK) return st;
    st = morton_order(ctx, d_tris, n, bvh->sorted_codes, bvh->sorted_ids);
    if (st != GBRT_OK) return st;

    // scratch (after the sort): clusters twice, neighbours, tile and group sums, states
    const uint32_t max_tiles = (n + kTile - 1) / kTile, num_groups = max_tiles / kGroup + 1;
    size_t off_lo0 = 0, off_hi0 = align_up(size_t(n) * 16), off_lo1 = off_hi0 + align_up(size_t(n) * 16);
    size_t off_hi1 = off_lo1 + align_up(size_t(n) * 16), off_nn = off_hi1 + align_up(size_t(n) * 16);
    size_t off_tiles = off_nn + align_up(size_t(n) * 4), off_groups = off_tiles + align_up(size_t(max_tiles) * 8);
    size_t off_state = off_groups + align_up(size_t(num_groups) * 16);
    st = ensure_scratch(ctx, off_state + 256);
    if (st != GBRT_OK) return st;
    build_result* result = nullptr;
    st = ensure_result(ctx, &result);
    if (st != GBRT_OK) return st;
    char* base = static_cast<char*>(ctx->scratch);
    float4* lo[2] = { reinterpret_cast<float4*>(base + off_lo0), reinterpret_cast<float4*>(base + off_lo1) };
    float4* hi[2] = { reinterpret_cast<float4*>(base + off_hi0), reinterpret_cast<float4*>(base + off_hi1) };
    int* nn = reinterpret_cast<int*>(base + off_nn);
    auto* tiles = reinterpret_cast<unsigned long long*>(base + off_tiles);
    auto* group_mem = reinterpret_cast<unsigned long long*>(base + off_groups);
    unsigned long long* groups[2] = { group_mem, group_mem + num_groups };
    auto* state = reinterpret_cast<ploc_state*>(base + off_state);

    ploc_leaves<<<blocks_for(n), kBlock, 0, s>>>(d_tris, bvh->sorted_ids, n, lo[0], hi[0], bvh->tris, state, groups[0],
                                                 num_groups, ctx->d_status);
    GBRT_LAUNCH_CHECK(ctx, "ploc_leaves");
    auto* host = const_cast<volatile build_result*>(ctx->h_result);
    host->clusters = n;
    host->quads_bad = 0;
    event_ring done;
    uint32_t iter = 0;
    for (uint32_t clusters = n; clusters > uint32_t(kTail); ++iter)
    {
        const int cur = int(iter & 1);
        const uint32_t grid = (clusters + kTile - 1) / kTile;
        ploc_nearest<<<grid, kSearchThreads, 0, s>>>(lo[cur], hi[cur], state + cur, nn, tiles, groups[cur]);
        GBRT_LAUNCH_CHECK(ctx, "ploc_nearest");
        ploc_merge<<<grid, kTile, 0, s>>>(lo[cur], hi[cur], nn, state + cur, state + (cur ^ 1), tiles, groups[cur],
                                          groups[cur ^ 1], num_groups, bvh->num_inner, bvh->nodes, lo[cur ^ 1],
                                          hi[cur ^ 1], &result->clusters, ctx->d_status);
        GBRT_LAUNCH_CHECK(ctx, "ploc_merge");
        cudaEvent_t* mark = nullptr;
        GBRT_CUDA(ctx, done.at(iter, &mark));
        GBRT_CUDA(ctx, cudaEventRecord(*mark, s));
        if (iter >= kLate)
        {
            GBRT_CUDA(ctx, done.at(iter - kLate, &mark));
            GBRT_CUDA(ctx, cudaEventSynchronize(*mark));
            clusters = host->clusters;
        }
    }
    GBRT_CUDA(ctx, cudaFuncSetAttribute(ploc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTailBytes)));
    ploc_tail<<<1, kTailThreads, kTailBytes, s>>>(lo[iter & 1], hi[iter & 1], state + (iter & 1), bvh->num_inner,
                                                  bvh->nodes, result, ctx->d_status);
    GBRT_LAUNCH_CHECK(ctx, "ploc_tail");
    if (bvh->quads)
    {
        GBRT_CUDA(ctx, cudaMemsetAsync(bvh->quads + bvh->num_inner, 0, sizeof(quad_node), s));
        st = make_quads(ctx, bvh->nodes, bvh->num_inner, nullptr, 0, uint32_t(bvh->root), bvh->quads,
                        &result->quads_bad, s);
        if (st != GBRT_OK) return st;
    }
    GBRT_CUDA(ctx, cudaStreamSynchronize(s));
    const build_result r = *ctx->h_result;
    if (r.stuck) return fail(ctx, GBRT_ERR_CUDA, "PLOC build: inconsistent merge step");
    if (r.made != n - 1) return fail(ctx, GBRT_ERR_CUDA, "PLOC build: wrong node count");
    if (r.root != bvh->root) return fail(ctx, GBRT_ERR_CUDA, "PLOC build: unexpected root");
    bvh->quads_ok = bvh->quads && r.quads_bad == 0;
    bvh->height = r.height;
    for (int a = 0; a < 3; ++a)
    {
        bvh->lo[a] = r.lo[a];
        bvh->hi[a] = r.hi[a];
    }
    if (bvh->height + 1 > uint32_t(kStackSize))
        return fail(ctx, GBRT_ERR_STACK_OVERFLOW, "PLOC tree height exceeds the traversal stack");
    return GBRT_OK;
}

// The tree in visionaray's index_bvh layout (bvh.h:70-141): nodes numbered breadth
// first with the two children of a node adjacent, one primitive per leaf (first_prim
// = the original index, indices = 0, 1, 2, ...).  Built on the host from the node pairs.
gbrt_status export_generic(gbrt_context* ctx, gbrt_bvh const* bvh, gbrt_bvh_node* d_nodes, uint32_t* d_indices)
{
    const uint32_t n = bvh->num_prims;
    if (n == 0) return GBRT_OK;
    std::vector<bvh2_node> pairs(bvh->num_inner);
    std::vector<uint32_t> ids(n);
    cudaStream_t s = ctx->stream;
    if (bvh->num_inner)
        GBRT_CUDA(ctx, cudaMemcpyAsync(pairs.data(), bvh->nodes, pairs.size() * sizeof(bvh2_node),
                                       cudaMemcpyDeviceToHost, s));
    GBRT_CUDA(ctx, cudaMemcpyAsync(ids.data(), bvh->sorted_ids, size_t(n) * 4, cudaMemcpyDeviceToHost, s));
    GBRT_CUDA(ctx, cudaStreamSynchronize(s));
    std::vector<gbrt_bvh_node> out(2 * size_t(n) - 1);
    auto put = [](gbrt_bvh_node& d, float lx, float hx, float ly, float hy, float lz, float hz, uint32_t first,
                  uint16_t count) {
        d.bbox_min[0] = lx;
        d.bbox_max[0] = hx;
        d.bbox_min[1] = ly;
        d.bbox_max[1] = hy;
        d.bbox_min[2] = lz;
        d.bbox_max[2] = hz;
        d.first_child_or_prim = first;
        d.num_prims = count;
        d.ordered_traversal_axis = 0;
        d.ordered_traversal_sign = 0;
    };
    if (n == 1)
    {
        put(out[0], bvh->lo[0], bvh->hi[0], bvh->lo[1], bvh->hi[1], bvh->lo[2], bvh->hi[2], ids[0], 1);
    }
    else
    {
        put(out[0], bvh->lo[0], bvh->hi[0], bvh->lo[1], bvh->hi[1], bvh->lo[2], bvh->hi[2], 1u, 0);
        // (pair node, output slot of its first child)
        std::vector<std::pair<int, uint32_t>> queue{ { bvh->root, 1u } };
        uint32_t next = 3;
        for (size_t q = 0; q < queue.size(); ++q)
        {
            bvh2_node const& nd = pairs[size_t(queue[q].first)];
            const uint32_t slot = queue[q].second;
            const int child[2] = { nd.link.x, nd.link.y };
            const float4 xy[2] = { nd.xy0, nd.xy1 };
            const float zl[2] = { nd.z01.x, nd.z01.z }, zh[2] = { nd.z01.y, nd.z01.w };
            for (int c = 0; c < 2; ++c)
            {
                gbrt_bvh_node& d = out[slot + c];
                if (child[c] < 0)
                {
                    put(d, xy[c].x, xy[c].y, xy[c].z, xy[c].w, zl[c], zh[c], ids[size_t(~child[c])], 1);
                }
                else
                {
                    put(d, xy[c].x, xy[c].y, xy[c].z, xy[c].w, zl[c], zh[c], next, 0);
                    queue.push_back({ child[c], next });
                    next += 2;
                }
            }
        }
    }
    std::vector<uint32_t> idx(n);
    for (uint32_t k = 0; k < n; ++k) idx[k] = k;
    GBRT_CUDA(ctx, cudaMemcpyAsync(d_nodes, out.data(), out.size() * sizeof(gbrt_bvh_node), cudaMemcpyHostToDevice, s));
    GBRT_CUDA(ctx, cudaMemcpyAsync(d_indices, idx.data(), size_t(n) * 4, cudaMemcpyHostToDevice, s));
    GBRT_CUDA(ctx, cudaStreamSynchronize(s));
    return GBRT_OK;
}

} // namespace gbrt
