// Internal octree linkage and node geometry (tree/octree.hpp:55-196, tree/octree_gpu.cu:41-203,
// focus/source_center_gpu.cu:212-240).
//
//  1. the nodes in (level, key) order with their links, by counting: the nodes that begin at a leaf are known from its
//     neighbours in the array, so a node's place is its level's start plus the nodes of that level before it
//  2. node geometric centres and half sizes from the decoded integer box, unfused arithmetic
#include "cs_common.cuh"
#include "octree_link.cuh"

#include <algorithm>
#include <vector>

namespace csg
{

template<class K>
__device__ __forceinline__ int binaryKeyWeight(K key, unsigned level)
{
    int ret = 0;
    for (unsigned l = 1; l <= level + 1; ++l)
        ret += digitWeight(int(octalDigit<K>(key, l)));
    return ret;
}

// L, I, N from the host, or from a leaf count in device memory (then the launch covers a capacity and the slots
// [N, capacity) of the node arrays are padding)
struct LinkSizes
{
    int L, I, N;
};
__device__ __forceinline__ LinkSizes linkSizes(const int* Ldev, int Lhost)
{
    int L = Ldev ? *Ldev : Lhost;
    int I = (L - 1) / 7;
    return {L, I, L + I};
}

/* The placeholder prefixes in ascending order are the nodes level by level, in key order within a level. Leaf t begins
 * the nodes of the levels first..last: its own, and its ancestors that leaf t - 1 is not in. So the place of such a
 * node is the start of its level plus the count of leaves before t that begin a node of that level: one ballot per
 * level and warp. First children and parents need no search, as a node and its first child begin at the same leaf.
 * The nodes' numbers in internal_to_leaf follow the boundaries between their children 3 and 4; the leaf before that
 * boundary knows the number and, being inside the node, the node's place: the last one of its level that begins at or
 * before the leaf. Bound by its three launches and one read and write of the arrays. Against a radix sort of the
 * prefixes, its inversion and binary searches for the children, about ten launches, whole passes went from 877 to
 * 799 us (120k FP32 Plummer), 1026 to 978 (1M uniform) and 14.11 to 13.97 ms (16M Plummer). */
constexpr int LINK_TILE = 1024; // leaves of a block: a warp per level for the sums over its 32 warps

struct LeafNodes
{
    int first, last; // levels of the nodes that begin at the leaf; none: first > last
    int mid;         // level of the node whose children 3 and 4 meet at the leaf's end, or -1
};

template<class K>
__device__ __forceinline__ LeafNodes leafNodes(const K* __restrict__ leaves, int t, int L, K& key)
{
    constexpr int maxL = KeyTraits<K>::maxLevel;
    if (t >= L) return {1, 0, -1};
    key          = leaves[t];
    const K next = leaves[t + 1];
    LeafNodes r;
    r.last       = int(min(treeLevel<K>(next - key), unsigned(maxL)));
    r.first      = t ? commonPrefix<K>(leaves[t - 1], key) / 3 + 1 : 0;
    const int cp = commonPrefix<K>(key, next);
    r.mid        = t < L - 1 && cp >= 0 && cp % 3 == 0 && cp / 3 < maxL ? cp / 3 : -1;
    return r;
}

//! what no node of a valid tree is written to stays in range for every later reader
__device__ __forceinline__ void clearLinks(int Ncap, int N, int32_t* childOffsets, int32_t* i2l, int32_t* l2i)
{
    const int step = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= Ncap; i += step)
    {
        childOffsets[i] = 0;
        if (i < N) i2l[i] = l2i[i] = 0;
    }
}

//! counts[level][tile]: the nodes of a level that begin in a tile
template<class K>
__global__ void __launch_bounds__(LINK_TILE) linkCountKernel(const K* __restrict__ leaves, const int* Ldev, int Lhost,
                                                             int Ncap, int32_t* __restrict__ counts,
                                                             int32_t* __restrict__ childOffsets,
                                                             int32_t* __restrict__ i2l, int32_t* __restrict__ l2i)
{
    constexpr int levels = KeyTraits<K>::maxLevel + 1;
    __shared__ int cnt[levels];
    const LinkSizes z = linkSizes(Ldev, Lhost);
    if (threadIdx.x < levels) cnt[threadIdx.x] = 0;
    clearLinks(Ncap, z.N, childOffsets, i2l, l2i);
    K key             = 0;
    const LeafNodes b = leafNodes<K>(leaves, blockIdx.x * LINK_TILE + threadIdx.x, z.L, key);
    __syncthreads();
#pragma unroll
    for (int l = 0; l < levels; ++l)
    {
        const unsigned m = __ballot_sync(0xffffffffu, b.first <= l && l <= b.last);
        if (m && threadIdx.x % 32 == 0) atomicAdd(&cnt[l], __popc(m));
    }
    __syncthreads();
    if (threadIdx.x < levels) counts[size_t(threadIdx.x) * gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

//! one block per level: the sums before each tile, and the level's total
__global__ void __launch_bounds__(1024) linkScanKernel(int32_t* __restrict__ counts, int tiles,
                                                       int32_t* __restrict__ totals)
{
    __shared__ int warpSum[32];
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    int32_t* c = counts + size_t(blockIdx.x) * tiles;
    int carry  = 0;
    for (int base = 0; base < tiles; base += 1024)
    {
        const int i = base + threadIdx.x;
        const int v = i < tiles ? c[i] : 0;
        int incl    = v;
#pragma unroll
        for (int d = 1; d < 32; d *= 2)
        {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane == 31) warpSum[warp] = incl;
        __syncthreads();
        int before = lane < warp ? warpSum[lane] : 0, all = warpSum[lane];
        before = __reduce_add_sync(0xffffffffu, before);
        all    = __reduce_add_sync(0xffffffffu, all);
        if (i < tiles) c[i] = carry + before + incl - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

template<class K>
__global__ void __launch_bounds__(LINK_TILE)
    linkNodesKernel(const K* __restrict__ leaves, const int* Ldev, int Lhost, int Ncap,
                    const int32_t* __restrict__ counts, const int32_t* __restrict__ totals, K* __restrict__ prefixes,
                    int32_t* childOffsets, int32_t* __restrict__ parents, int32_t* __restrict__ levelRange,
                    int32_t* i2l, int32_t* l2i)
{
    constexpr int levels = KeyTraits<K>::maxLevel + 1;
    __shared__ unsigned mask[levels][32];
    __shared__ int place[levels][32]; // of a warp's first node of the level
    __shared__ int total[levels];
    const LinkSizes z = linkSizes(Ldev, Lhost);
    const int L = z.L, I = z.I, N = z.N;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int t       = blockIdx.x * LINK_TILE + threadIdx.x;
    const bool single = gridDim.x == 1; // then no counts: the tile's own are all
    if (single) clearLinks(Ncap, N, childOffsets, i2l, l2i);
    for (int i = N + t; i < Ncap; i += gridDim.x * LINK_TILE)
        prefixes[i] = ~K(0); // a capacity's padding: behind every real prefix

    K key             = 0;
    const LeafNodes b = leafNodes<K>(leaves, t, L, key);
#pragma unroll
    for (int l = 0; l < levels; ++l)
    {
        const unsigned m = __ballot_sync(0xffffffffu, b.first <= l && l <= b.last);
        if (lane == l) mask[l][warp] = m;
    }
    __syncthreads();
    if (warp < levels)
    {
        const int v = __popc(mask[warp][lane]);
        int incl    = v;
#pragma unroll
        for (int d = 1; d < 32; d *= 2)
        {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        place[warp][lane] = incl - v + (single ? 0 : counts[size_t(warp) * gridDim.x + blockIdx.x]);
        if (lane == 31) total[warp] = single ? incl : totals[warp];
    }
    __syncthreads();
    if (warp < levels)
    {
        const int start = __reduce_add_sync(0xffffffffu, lane < warp ? total[lane] : 0);
        place[warp][lane] += start;
        if (blockIdx.x == 0 && lane == 0)
        {
            levelRange[warp] = min(start, N);
            if (warp == levels - 1) levelRange[levels] = N;
        }
    }
    __syncthreads();

    const unsigned below = (1u << lane) - 1u;
    auto at = [&](int l) { return place[l][warp] + __popc(mask[l][warp] & below); };
    int parent = -1;
    for (int l = b.first; l <= b.last; ++l)
    {
        const int pos = at(l);
        if (pos >= N) break; // not a valid tree
        prefixes[pos] = encodePlaceholderBit<K>(key, 3 * l);
        if (parent >= 0 && pos > 0 && pos + 8 <= N)
        {
            childOffsets[parent]   = pos;
            parents[(pos - 1) / 8] = parent;
        }
        parent = pos;
        if (l == b.last)
        {
            i2l[pos]   = t;
            l2i[t + I] = pos;
        }
    }
    if (b.mid >= 0)
    {
        const int pos = at(b.mid) + int(mask[b.mid][warp] >> lane & 1u) - 1;
        const int num = (t + binaryKeyWeight<K>(key, b.mid)) / 7;
        if (pos >= 0 && pos < N && num >= 0 && num < I)
        {
            i2l[pos] = num - I;
            l2i[num] = pos;
        }
    }
}

template<class K>
size_t buildLinkWorkspaceBytes(int L)
{
    constexpr size_t levels = KeyTraits<K>::maxLevel + 1;
    Arena a;
    a.take<int32_t>(levels * iceil(std::max(L, 1), LINK_TILE));
    a.take<int32_t>(levels);
    return a.size + 512;
}

template<class K>
int buildLink(cudaStream_t s, const K* leaves, int L, const cs_octree_view& v, void* ws, size_t wsBytes,
              const int* Ldev)
{
    constexpr int levels = KeyTraits<K>::maxLevel + 1;
    if (L < 1)
    {
        setLastError("build octree: need at least one leaf");
        return CS_ERR_INVALID;
    }
    // with Ldev, L is the leaf capacity and the arrays of v hold the capacity's node count
    int I = (L - 1) / 7, N = L + I;
    if (v.num_leaf_nodes != L || v.num_internal_nodes != I || v.num_nodes != N)
    {
        setLastError("build octree: view sizes (%d, %d, %d) do not match L = %d", v.num_leaf_nodes,
                     v.num_internal_nodes, v.num_nodes, L);
        return CS_ERR_INVALID;
    }
    const int tiles = iceil(L, LINK_TILE);
    Arena a{static_cast<char*>(ws), 0, wsBytes};
    int32_t* counts = a.take<int32_t>(size_t(levels) * tiles);
    int32_t* totals = a.take<int32_t>(levels);
    if (!a.ok())
    {
        setLastError("build octree: workspace too small");
        return CS_ERR_INVALID;
    }
    if (tiles > 1)
    {
        linkCountKernel<K><<<tiles, LINK_TILE, 0, s>>>(leaves, Ldev, L, N, counts, v.child_offsets, v.internal_to_leaf,
                                                       v.leaf_to_internal);
        CSG_CHECK_LAUNCH();
        linkScanKernel<<<levels, 1024, 0, s>>>(counts, tiles, totals);
        CSG_CHECK_LAUNCH();
    }
    linkNodesKernel<K><<<tiles, LINK_TILE, 0, s>>>(leaves, Ldev, L, N, counts, totals, static_cast<K*>(v.prefixes),
                                                   v.child_offsets, v.parents, v.level_range, v.internal_to_leaf,
                                                   v.leaf_to_internal);
    CSG_CHECK_LAUNCH();
    return CS_OK;
}

template size_t buildLinkWorkspaceBytes<uint32_t>(int);
template size_t buildLinkWorkspaceBytes<uint64_t>(int);
template int buildLink<uint32_t>(cudaStream_t, const uint32_t*, int, const cs_octree_view&, void*, size_t, const int*);
template int buildLink<uint64_t>(cudaStream_t, const uint64_t*, int, const cs_octree_view&, void*, size_t, const int*);

// ---------------------------------------------------------------------------------------------------------------
// node geometry: centerAndSize (sfc/box.hpp:318-335) of hilbertIBox / mortonIBox
// ---------------------------------------------------------------------------------------------------------------
template<class T>
struct GeoParams
{
    T lo[3];
    T half[3]; // 0.5 * (1 / 2^L) * box length, rounded in T as the reference does
};

template<class K, class T, int Kind>
__global__ void geoCentersKernel(const K* __restrict__ prefixes, int Nhost, const int* Ldev, T* __restrict__ centers,
                                 T* __restrict__ sizes, GeoParams<T> g)
{
    int i       = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = Ldev ? linkSizes(Ldev, 0).N : Nhost;
    if (i >= N) return;
    K prefix          = prefixes[i];
    K start           = decodePlaceholderBit<K>(prefix);
    unsigned level    = decodePrefixLength<K>(prefix) / 3;
    unsigned maxCoord = 1u << KeyTraits<K>::maxLevel;
    unsigned cube     = maxCoord >> level;
    unsigned ix, iy, iz;
    if (Kind == CS_HILBERT)
    {
        decodeHilbert<K>(start, ix, iy, iz);
        unsigned mask = ~(cube - 1u);
        ix &= mask;
        iy &= mask;
        iz &= mask;
    }
    else { decodeMorton<K>(start, ix, iy, iz); }
    unsigned imin[3] = {ix, iy, iz};
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        int a                = int(imin[k]);
        int b                = a + int(cube);
        centers[3 * i + k]   = RN<T>::add(g.lo[k], RN<T>::mul(T(b + a), g.half[k]));
        sizes[3 * i + k]     = RN<T>::mul(T(b - a), g.half[k]);
    }
}

template<class K, class T>
int geoCenters(cudaStream_t s, const K* prefixes, int N, T* centers, T* sizes, const cs_box& box, int kind,
               const int* Ldev)
{
    if (N <= 0) return CS_OK;
    auto bp = makeBoxParams<T>(box);
    GeoParams<T> g;
    const T uL = T(1) / T(int(1u << KeyTraits<K>::maxLevel));
    for (int k = 0; k < 3; ++k)
    {
        g.lo[k]   = bp.lo[k];
        g.half[k] = T(0.5) * uL * bp.len[k];
    }
    if (kind == CS_HILBERT)
        geoCentersKernel<K, T, CS_HILBERT><<<iceil(N, 256), 256, 0, s>>>(prefixes, N, Ldev, centers, sizes, g);
    else geoCentersKernel<K, T, CS_MORTON><<<iceil(N, 256), 256, 0, s>>>(prefixes, N, Ldev, centers, sizes, g);
    CSG_CHECK_LAUNCH();
    return CS_OK;
}

// batched sets in one 64-bit tree: node key = (set << 30) | the set's 32-bit key, set roots at level rootLevel; every
// node at or below a set root gets the geometry the set's own 32-bit tree gives it (its box, its levels); the nodes
// above the set roots and the empty filler nodes get a zero box (never traversed)
template<class T, int Kind>
__global__ void geoCentersBatchKernel(const uint64_t* __restrict__ prefixes, int N, T* __restrict__ centers,
                                      T* __restrict__ sizes, const GeoParams<T>* __restrict__ sets, int numSets,
                                      unsigned rootLevel)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    uint64_t prefix = prefixes[i];
    uint64_t start  = decodePlaceholderBit<uint64_t>(prefix);
    unsigned level  = decodePrefixLength<uint64_t>(prefix) / 3;
    uint64_t set    = start >> 30;
    if (level < rootLevel || set >= uint64_t(numSets))
    {
#pragma unroll
        for (int k = 0; k < 3; ++k)
            centers[3 * size_t(i) + k] = sizes[3 * size_t(i) + k] = T(0);
        return;
    }
    const uint32_t rel = uint32_t(start & ((uint64_t(1) << 30) - 1));
    unsigned cube      = (1u << KeyTraits<uint32_t>::maxLevel) >> (level - rootLevel);
    unsigned ix, iy, iz;
    if (Kind == CS_HILBERT)
    {
        decodeHilbert<uint32_t>(rel, ix, iy, iz);
        unsigned mask = ~(cube - 1u);
        ix &= mask;
        iy &= mask;
        iz &= mask;
    }
    else { decodeMorton<uint32_t>(rel, ix, iy, iz); }
    const GeoParams<T> g = sets[set];
    unsigned imin[3]     = {ix, iy, iz};
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        int a0                     = int(imin[k]);
        int b0                     = a0 + int(cube);
        centers[3 * size_t(i) + k] = RN<T>::add(g.lo[k], RN<T>::mul(T(b0 + a0), g.half[k]));
        sizes[3 * size_t(i) + k]   = RN<T>::mul(T(b0 - a0), g.half[k]);
    }
}

template<class T>
size_t geoParamsBytes(int numSets)
{
    return size_t(numSets) * sizeof(GeoParams<T>) + 256;
}

template<class T>
int geoCentersBatched(cudaStream_t s, const uint64_t* prefixes, int N, T* centers, T* sizes, const cs_box* boxes,
                      int numSets, int kind, void* paramsDev, unsigned rootLevel)
{
    if (N <= 0) return CS_OK;
    std::vector<GeoParams<T>> g(numSets);
    const T uL = T(1) / T(int(1u << KeyTraits<uint32_t>::maxLevel));
    for (int j = 0; j < numSets; ++j)
    {
        auto bp = makeBoxParams<T>(boxes[j]);
        for (int k = 0; k < 3; ++k)
        {
            g[j].lo[k]   = bp.lo[k];
            g[j].half[k] = T(0.5) * uL * bp.len[k];
        }
    }
    auto* gd = static_cast<GeoParams<T>*>(paramsDev);
    CSG_CUDA_TRY(cudaMemcpyAsync(gd, g.data(), g.size() * sizeof(GeoParams<T>), cudaMemcpyHostToDevice, s));
    if (kind == CS_HILBERT)
        geoCentersBatchKernel<T, CS_HILBERT><<<iceil(N, 256), 256, 0, s>>>(prefixes, N, centers, sizes, gd, numSets,
                                                                           rootLevel);
    else
        geoCentersBatchKernel<T, CS_MORTON><<<iceil(N, 256), 256, 0, s>>>(prefixes, N, centers, sizes, gd, numSets,
                                                                          rootLevel);
    CSG_CHECK_LAUNCH();
    return CS_OK;
}

template size_t geoParamsBytes<float>(int);
template size_t geoParamsBytes<double>(int);
template int geoCentersBatched<float>(cudaStream_t, const uint64_t*, int, float*, float*, const cs_box*, int, int,
                                      void*, unsigned);
template int geoCentersBatched<double>(cudaStream_t, const uint64_t*, int, double*, double*, const cs_box*, int, int,
                                       void*, unsigned);

template int geoCenters<uint32_t, float>(cudaStream_t, const uint32_t*, int, float*, float*, const cs_box&, int,
                                         const int*);
template int geoCenters<uint32_t, double>(cudaStream_t, const uint32_t*, int, double*, double*, const cs_box&, int,
                                          const int*);
template int geoCenters<uint64_t, float>(cudaStream_t, const uint64_t*, int, float*, float*, const cs_box&, int,
                                         const int*);
template int geoCenters<uint64_t, double>(cudaStream_t, const uint64_t*, int, double*, double*, const cs_box&, int,
                                          const int*);

} // namespace csg

using namespace csg;

extern "C" size_t cs_build_octree_workspace_bytes(int32_t num_leaves, int key_bits)
{
    return key_bits == 32 ? buildLinkWorkspaceBytes<uint32_t>(num_leaves) : buildLinkWorkspaceBytes<uint64_t>(num_leaves);
}

template<class K>
static int buildOctreeEntry(cs_stream_t stream, const K* leaves, int32_t L, const cs_octree_view* view,
                            int32_t* levelRangeHost, void* ws, size_t wsb)
{
    if (!leaves || !view || !view->prefixes || !view->child_offsets || !view->parents || !view->level_range ||
        !view->internal_to_leaf || !view->leaf_to_internal)
    {
        setLastError("build octree: null pointer");
        return CS_ERR_INVALID;
    }
    cudaStream_t s = cudaStream_t(stream);
    Workspace w;
    size_t need = buildLinkWorkspaceBytes<K>(L);
    int rc      = w.acquire(ws, wsb, need, s);
    if (rc) return rc;
    rc = buildLink<K>(s, leaves, L, *view, w.ptr, need);
    if (rc) return rc;
    if (levelRangeHost)
    {
        CSG_CUDA_TRY(cudaMemcpyAsync(levelRangeHost, view->level_range, (KeyTraits<K>::maxLevel + 2) * sizeof(int32_t),
                                     cudaMemcpyDeviceToHost, s));
        CSG_CUDA_TRY(cudaStreamSynchronize(s));
    }
    return CS_OK;
}

extern "C" int cs_build_octree_u32(cs_stream_t stream, const uint32_t* leaves, int32_t L, const cs_octree_view* view,
                                   int32_t* lr, void* ws, size_t wsb)
{
    return buildOctreeEntry<uint32_t>(stream, leaves, L, view, lr, ws, wsb);
}
extern "C" int cs_build_octree_u64(cs_stream_t stream, const uint64_t* leaves, int32_t L, const cs_octree_view* view,
                                   int32_t* lr, void* ws, size_t wsb)
{
    return buildOctreeEntry<uint64_t>(stream, leaves, L, view, lr, ws, wsb);
}

#define CS_GEO_ENTRY(kb, K, tb, T)                                                                                     \
    extern "C" int cs_geo_centers_##kb##_##tb(cs_stream_t stream, const K* prefixes, int32_t n, T* c, T* sz,           \
                                              const cs_box* box, int kind)                                             \
    {                                                                                                                  \
        if (!box || (n > 0 && (!prefixes || !c || !sz)))                                                               \
        {                                                                                                              \
            setLastError("geo centers: null pointer");                                                                 \
            return CS_ERR_INVALID;                                                                                     \
        }                                                                                                              \
        return geoCenters<K, T>(cudaStream_t(stream), prefixes, n, c, sz, *box, kind);                                \
    }
CS_GEO_ENTRY(u32, uint32_t, f32, float)
CS_GEO_ENTRY(u32, uint32_t, f64, double)
CS_GEO_ENTRY(u64, uint64_t, f32, float)
CS_GEO_ENTRY(u64, uint64_t, f64, double)
