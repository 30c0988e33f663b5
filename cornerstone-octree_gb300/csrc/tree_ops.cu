// Tree operations around the octree path: upsweeps of node counts and source centres, target groups, SFC gap
// filling and spanning trees.
//
// Upsweeps (upsweepSumGpu, tree/octree_gpu.cu:218-236; upsweepCentersGpu, focus/source_center_gpu.cu:173-205). The
// reference launches one kernel per tree level, deepest first, with the level boundaries read on the host. Here one
// launch does the whole upsweep: a warp per group of eight siblings counts the leaves among them at once; each internal
// node has an arrival counter, and the warp whose arrival completes the eight combines them (in child order, so
// floating-point results equal the level-by-level evaluation) and carries on upwards. For centres the lanes hold (child,
// component) and only the eight additions of a component are serial. Bound: the chain of levels (latency). 4M particles,
// 240k nodes: 109 -> 68 us for centres, 29 -> 28 us for counts, against one thread per leaf and a serial combine. The level-by-level form is kept for callers that hold only
// levelRange (no parents array), as the reference's signature does.
//
// Source centres (computeLeafSourceCenterGpu, focus/source_center_gpu.cu:103-170). Mass centres are evaluated in the
// CPU reference's order (massCenter, focus/source_center.hpp:70-81: a serial sum over the leaf's particles, then one
// division) with round-to-nearest intrinsics, so the results equal the CPU path bit for bit; the reference's own GPU
// kernel sums 8-way interleaved partial sums with fused multiply-adds and differs from its CPU path in the last bits.
//
// Target groups (computeFixedGroups / computeGroupSplits, traversal/groups_gpu.cu, groupSplitsKernel and findSplits in
// traversal/groups_gpu.cuh). Fixed groups of 32 or 64 consecutive particles are cut where consecutive particles are
// farther apart than min(tol * edge of the smallest leaf among the group's first 32 particles, 2h / minExtent), in
// unit-box coordinates. One warp per fixed group computes the cut mask and the count; an exclusive scan gives each
// group's first output slot, and a second pass writes the group starts directly (the reference scans twice with a
// host synchronisation in between).
//
// SFC gaps (countSfcGapsGpu / fillSfcGapsGpu, tree/csarray_gpu.cu:238-270) and computeSpanningTree
// (tree/csarray.hpp:482-506): spanSfcRange per interval, an exclusive scan, and the keys written per interval.
#include "cs_common.cuh"
#include "octree_link.cuh"

#include <algorithm>
#include <type_traits>

namespace csg
{

int exclusiveScanI32(cudaStream_t s, const int32_t* in, int32_t* out, size_t n, int32_t init, void* ws, size_t wsb);
size_t exclusiveScanWorkspaceBytes(size_t n);

// ---------------------------------------------------------------------------------------------------------------
// upsweeps
// ---------------------------------------------------------------------------------------------------------------

// NodeCount (tree/octree.hpp:603-615): min(2^32 - 1, sum of the 8 children)
struct CountCombine
{
    using V                   = uint32_t;
    static constexpr int WARP = 1; // threads per sibling group of the one-launch upsweep
    __device__ static void combine(V* q, int node, int child)
    {
        unsigned long long sum = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            sum += __ldcg(q + child + k);
        q[node] = uint32_t(min(sum, 0xFFFFFFFFull));
    }
};

// addBody / normalizeMass / CombineSourceCenter (focus/source_center.hpp:46-98) in the reference's order, no fusion
template<class T>
__device__ __forceinline__ void addBody(T c[4], T x, T y, T z, T m)
{
    T w  = RN<T>::abs_(m);
    c[0] = RN<T>::add(c[0], RN<T>::mul(w, x));
    c[1] = RN<T>::add(c[1], RN<T>::mul(w, y));
    c[2] = RN<T>::add(c[2], RN<T>::mul(w, z));
    c[3] = RN<T>::add(c[3], w);
}

template<class T>
__device__ __forceinline__ T rdiv(T a, T b)
{
    if constexpr (std::is_same_v<T, double>) return __ddiv_rn(a, b);
    else return __fdiv_rn(a, b);
}

template<class T>
__device__ __forceinline__ void normalizeMass(T c[4])
{
    T inv = (c[3] != T(0)) ? rdiv<T>(T(1), c[3]) : T(1);
    c[0]  = RN<T>::mul(c[0], inv);
    c[1]  = RN<T>::mul(c[1], inv);
    c[2]  = RN<T>::mul(c[2], inv);
}

template<class T>
struct CenterCombine
{
    using V                   = T; // 4 per node
    static constexpr int WARP = 32;
    __device__ static void combine(T* q, int node, int child)
    {
        T c[4] = {0, 0, 0, 0};
        for (int k = 0; k < 8; ++k)
        {
            const T* s = q + 4 * size_t(child + k);
            addBody<T>(c, __ldcg(s), __ldcg(s + 1), __ldcg(s + 2), __ldcg(s + 3));
        }
        normalizeMass<T>(c);
        T* o = q + 4 * size_t(node);
        o[0] = c[0], o[1] = c[1], o[2] = c[2], o[3] = c[3];
    }
    // lane 4 k + c holds component c of child k; the operations and their order are those of combine
    __device__ static void combineWarp(T* q, int node, int child, int lane)
    {
        const int c  = lane & 3;
        const T v    = __ldcg(q + 4 * size_t(child) + lane);
        const T m    = RN<T>::abs_(__shfl_sync(0xffffffffu, v, lane | 3));
        const T term = c < 3 ? RN<T>::mul(m, v) : m;
        T sum        = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            sum = RN<T>::add(sum, __shfl_sync(0xffffffffu, term, 4 * k + c));
        const T mass = __shfl_sync(0xffffffffu, sum, 3);
        if (lane < 4)
        {
            const T inv               = mass != T(0) ? rdiv<T>(T(1), mass) : T(1);
            q[4 * size_t(node) + c] = c < 3 ? RN<T>::mul(sum, inv) : sum;
        }
    }
};

// one launch, a warp (centres) or a thread (counts) per sibling group g (nodes 8 g + 1 .. 8 g + 8, children of
// parents[g]) that holds leaves
template<class Op>
__global__ void __launch_bounds__(256) upsweepLinkedKernel(const int32_t* __restrict__ childOffsets,
                                                           const int32_t* __restrict__ parents, int numGroups,
                                                           typename Op::V* q, unsigned* arrivals)
{
    constexpr bool WARP    = Op::WARP == 32;
    constexpr unsigned ALL = 0xffffffffu;
    const int lane         = WARP ? threadIdx.x & 31 : 0;
    int group              = int((size_t(blockIdx.x) * blockDim.x + threadIdx.x) / Op::WARP);
    if (group >= numGroups) return;
    unsigned add = 0;
    if constexpr (WARP) add = __popc(__ballot_sync(ALL, lane < 8 && childOffsets[8 * group + 1 + lane] == 0));
    else
    {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            add += childOffsets[8 * group + 1 + k] == 0;
    }
    if (add == 0) return;
    for (;;)
    {
        const int p  = __ldg(parents + group);
        unsigned old = 0;
        if (lane == 0)
        {
            __threadfence(); // this group's values before the arrival that may let another one read them
            old = atomicAdd(arrivals + p, add);
            __threadfence(); // the other children's values after their arrivals
        }
        if constexpr (WARP) old = __shfl_sync(ALL, old, 0);
        if (old + add != 8u) return;
        if constexpr (WARP)
        {
            __syncwarp();
            Op::combineWarp(q, p, __ldg(childOffsets + p), lane);
            __threadfence();
            __syncwarp();
        }
        else Op::combine(q, p, __ldg(childOffsets + p));
        if (p == 0) return;
        group = (p - 1) / 8;
        add   = 1;
    }
}

template<class Op>
__global__ void upsweepLevelKernel(int first, int last, const int32_t* __restrict__ childOffsets, typename Op::V* q)
{
    int i = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= last) return;
    int c = childOffsets[i];
    if (c) Op::combine(q, i, c);
}

template<class Op>
static int upsweep(cudaStream_t s, int numLevels, const int32_t* levelRangeHost, const int32_t* childOffsets,
                   const int32_t* parents, int numNodes, typename Op::V* q, void* ws, size_t wsb)
{
    if (numNodes <= 1) return CS_OK;
    if (!childOffsets || !q)
    {
        setLastError("upsweep: null pointer");
        return CS_ERR_INVALID;
    }
    if (parents)
    {
        Workspace w;
        int rc = w.acquire(ws, wsb, size_t(numNodes) * sizeof(unsigned), s);
        if (rc) return rc;
        unsigned* arr = static_cast<unsigned*>(w.ptr);
        CSG_CUDA_TRY(cudaMemsetAsync(arr, 0, size_t(numNodes) * sizeof(unsigned), s));
        const int groups = (numNodes - 1) / 8;
        upsweepLinkedKernel<Op><<<iceil(size_t(groups) * Op::WARP, 256), 256, 0, s>>>(childOffsets, parents, groups, q, arr);
        CSG_CHECK_LAUNCH();
        return CS_OK;
    }
    if (!levelRangeHost || numLevels < 1)
    {
        setLastError("upsweep: need parents or the host level range");
        return CS_ERR_INVALID;
    }
    for (int level = numLevels - 1; level >= 0; --level)
    {
        int a = levelRangeHost[level], b = levelRangeHost[level + 1];
        if (b > a)
        {
            upsweepLevelKernel<Op><<<iceil(size_t(b - a), 256), 256, 0, s>>>(a, b, childOffsets, q);
            CSG_CHECK_LAUNCH();
        }
    }
    return CS_OK;
}

// Leaf mass centres, the reference's serial sums. A warp reads the particles of eight consecutive leaves in order and
// forms the products |m| x, |m| y, |m| z with all lanes, into shared memory; then four lanes per leaf add up one component
// each; the block normalises its 64 sums together. Bound by the FP64 pipe (2 lanes per clock and SM): three full
// multiplies per 32 particles, one addition per particle of the fullest leaf of eight, one division per 32 leaves. One
// thread per leaf ran 32 leaves as long as the fullest and read 32 scattered lines per load: 4M particles in 210k leaves
// 174 -> 137 us (four lanes per leaf straight from global memory: 196 us, the same lines).
constexpr int LC_WARPS = 8;
constexpr int LC_CAP   = 192; // particles staged at a time

template<class Tc, class Tm, class T>
__global__ void __launch_bounds__(32 * LC_WARPS) leafCentersKernel(const Tc* __restrict__ x, const Tc* __restrict__ y,
                                                                   const Tc* __restrict__ z, const Tm* __restrict__ m,
                                                                   const int32_t* __restrict__ l2i, int numLeaves,
                                                                   const uint32_t* __restrict__ layout, T* centers)
{
    __shared__ T sTerm[LC_WARPS][4][LC_CAP + 1];
    __shared__ T sSum[8 * LC_WARPS][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane & 3;
    const int leaf0 = blockIdx.x * 8 * LC_WARPS, own = 8 * warp + (lane >> 2);
    const int leaf  = min(numLeaves, leaf0 + own);
    uint32_t i = layout[leaf];
    const uint32_t end = leaf < numLeaves ? layout[leaf + 1] : i;
    uint32_t b         = __shfl_sync(0xffffffffu, i, 0);
    const uint32_t stop = __shfl_sync(0xffffffffu, end, 31);
    T sum = 0;
    for (; b < stop; b += LC_CAP)
    {
        const uint32_t n = min(uint32_t(LC_CAP), stop - b);
#pragma unroll 2
        for (uint32_t k = lane; k < n; k += 32)
        {
            const T a         = RN<T>::abs_(T(m[b + k]));
            sTerm[warp][0][k] = RN<T>::mul(a, T(x[b + k]));
            sTerm[warp][1][k] = RN<T>::mul(a, T(y[b + k]));
            sTerm[warp][2][k] = RN<T>::mul(a, T(z[b + k]));
            sTerm[warp][3][k] = a;
        }
        __syncwarp();
        for (const uint32_t e = min(end, b + n); i < e; ++i)
            sum = RN<T>::add(sum, sTerm[warp][c][i - b]);
        __syncwarp();
    }
    sSum[own][c] = sum;
    __syncthreads();
    for (int l = threadIdx.x; l < 8 * LC_WARPS && leaf0 + l < numLeaves; l += 32 * LC_WARPS)
    {
        T s[4] = {sSum[l][0], sSum[l][1], sSum[l][2], sSum[l][3]};
        normalizeMass<T>(s);
        T* o = centers + 4 * size_t(l2i[leaf0 + l]);
        o[0] = s[0], o[1] = s[1], o[2] = s[2], o[3] = s[3];
    }
}

// ---------------------------------------------------------------------------------------------------------------
// target groups
// ---------------------------------------------------------------------------------------------------------------

template<class T>
__device__ __forceinline__ T fmaRn(T a, T b, T c)
{
    if constexpr (std::is_same_v<T, double>) return __fma_rn(a, b, c);
    else return __fmaf_rn(a, b, c);
}

template<class T, class K>
struct GroupArgs
{
    uint32_t first, last;
    const T *x, *y, *z, *h;
    const K* leaves;
    int numLeaves;
    const uint32_t* layout;
    T ilx, ily, ilz, minExt;
    float tol;
};

// deepest level among the leaves of particles [p0, p1], by the whole warp: the leaf of p0 (upper_bound(layout, p0) - 1)
// by a 32-way search, then the leaves from there that hold particles up to p1
template<class K>
__device__ __forceinline__ unsigned deepestLeaf(const K* __restrict__ leaves, const uint32_t* __restrict__ layout,
                                                int numLeaves, uint32_t p0, uint32_t p1, int lane)
{
    int lo = 0, hi = numLeaves;
    for (;;)
    {
        const int chunk = (hi - lo + 31) / 32, at = lo + lane * chunk;
        const int below = __popc(__ballot_sync(0xffffffffu, at < hi && __ldg(layout + at) <= p0));
        lo += max(0, below - 1) * chunk;
        if (chunk <= 1) break;
        hi = min(hi, lo + chunk);
    }
    unsigned lev = 0;
    for (;; lo += 32)
    {
        const int l     = lo + lane;
        const bool in   = l < numLeaves && __ldg(layout + l) <= p1;
        if (in && __ldg(layout + l + 1) > __ldg(layout + l)) lev = max(lev, treeLevel<K>(leaves[l + 1] - leaves[l]));
        if (!__all_sync(0xffffffffu, in)) break;
    }
    return __reduce_max_sync(0xffffffffu, lev);
}

// FP32 decision of d2 > min(dc2, (2 h / minExt)^2) for FP64 particles: 1 cut, 0 no cut, -1 undecided. u: the FP64
// difference of the particles per axis (unscaled); its truncated float is within 2^-20, so is h's; the reference's own
// difference of the two scaled coordinates is within 2^-51 (|x| il + |u| il) of u il. Per axis e = |u| il with an error
// of at most 2^-18 e + delta, so |d2_f - d2| <= 2^-16 d2_f + 2 (ex + ey + ez) delta + 3 delta^2 (the slack covers the
// FP32 roundings), and (2 h / minExt)^2 is known to 2^-16.
__device__ __forceinline__ int cutScreen(const double (&u)[3], const double (&x)[3], const double* h, const float (&il)[3],
                                         float minExt, float dcLo, float dcHi)
{
    float e[3], delta = 1e-30f;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        float f = 0.f, s = 0.f;
        ok    = truncEstimate(u[k], f) && ok;
        ok    = truncEstimate(x[k], s) && ok;
        e[k]  = fabsf(f) * il[k];
        delta = fmaxf(delta, fmaf(0x1p-49f, fabsf(s) * il[k] + e[k], 0x1p-119f * il[k]));
    }
    float h2 = 1.f;
    if (h)
    {
        float hf = 0.f;
        ok       = truncEstimate(*h, hf) && ok && hf > 0.f;
        hf       = 2.f * hf / minExt;
        h2       = hf * hf;
    }
    const float d2  = fmaf(e[2], e[2], fmaf(e[1], e[1], e[0] * e[0]));
    const float err = 0x1p-16f * d2 + 2.5f * delta * (e[0] + e[1] + e[2]) + 4.f * delta * delta + 1e-30f;
    if (!ok) return -1;
    const float lo = d2 - err, hi = d2 + err;
    if (lo > dcHi || lo > h2 * (1.f + 0x1p-15f) + 1e-30f) return 1;
    if (hi < dcLo && hi < h2 * (1.f - 0x1p-15f) - 1e-30f) return 0;
    return -1;
}

// one warp per fixed group of NW * 32 particles: cut masks (bit k of segment w: cut after particle 32 w + k) and the
// number of groups it becomes. FP64 particles are decided in FP32 (cutScreen) but for those near the criterion: the FP64
// pipe (2 lanes per clock and SM) saw 28 instructions per particle, a division among them, and sees three; 4M particles,
// with the 32-way search of the leaf: 213 -> 88 us
template<int NW, class T, class K>
__global__ void groupSplitsKernel(GroupArgs<T, K> a, uint32_t numFixed, uint32_t* masks, int32_t* numSplits)
{
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane      = threadIdx.x & 31;
    if (warp >= numFixed) return;
    const uint32_t b0 = a.first + warp * 32u * NW;
    // smallest leaf volume among the first segment's particles; leaf volumes in the unit box are 2^(-3 level), and
    // their cube root is exactly 2^(-level): distCrit = 2^(-deepest level) * tol
    const unsigned lev = deepestLeaf<K>(a.leaves, a.layout, a.numLeaves, min(b0, a.last - 1), min(b0 + 31u, a.last - 1), lane);
    T dc         = RN<T>::mul(T(ldexp(1.0, -int(lev))), T(a.tol));
    T dc2        = RN<T>::mul(dc, dc);
    float dcLo = 0.f, dcHi = 0.f;
    const float il[3] = {float(a.ilx), float(a.ily), float(a.ilz)}, minExtF = float(a.minExt);
    if constexpr (std::is_same_v<T, double>)
    {
        dcLo = __double2float_rd(dc2);
        dcHi = __double2float_ru(dc2);
    }
    int count = 1;
#pragma unroll
    for (int w = 0; w < NW; ++w)
    {
        uint32_t j  = min(b0 + 32u * w + lane, a.last - 1);
        uint32_t jn = min(b0 + 32u * w + lane + 1, a.last - 1);
        // the last particle of the fixed group is compared with itself (no cut)
        if (w == NW - 1 && lane == 31) jn = j;
        const T p[3] = {a.x[j], a.y[j], a.z[j]}, q[3] = {a.x[jn], a.y[jn], a.z[jn]};
        int cut = -1;
        if constexpr (std::is_same_v<T, double>)
        {
            const double u[3] = {q[0] - p[0], q[1] - p[1], q[2] - p[2]};
            cut               = cutScreen(u, p, a.h ? a.h + j : nullptr, il, minExtF, dcLo, dcHi);
        }
        if (cut < 0)
        {
            T dx   = RN<T>::sub(RN<T>::mul(q[0], a.ilx), RN<T>::mul(p[0], a.ilx));
            T dy   = RN<T>::sub(RN<T>::mul(q[1], a.ily), RN<T>::mul(p[1], a.ily));
            T dz   = RN<T>::sub(RN<T>::mul(q[2], a.ilz), RN<T>::mul(p[2], a.ilz));
            T d2   = fmaRn<T>(dz, dz, fmaRn<T>(dy, dy, RN<T>::mul(dx, dx)));
            T hr   = a.h ? rdiv<T>(RN<T>::mul(T(2), a.h[j]), a.minExt) : T(1);
            T h2   = RN<T>::mul(hr, hr);
            T crit = dc2 < h2 ? dc2 : h2;
            cut    = d2 > crit;
        }
        unsigned m = __ballot_sync(0xffffffffu, cut > 0);
        if (lane == 0) masks[size_t(warp) * NW + w] = m;
        count += __popc(m);
    }
    if (lane == 0) numSplits[warp] = count;
}

template<int NW>
__global__ void groupWriteKernel(const uint32_t* __restrict__ masks, const int32_t* __restrict__ offsets,
                                 uint32_t numFixed, uint32_t first, uint32_t last, uint32_t* groups, size_t capacity)
{
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= numFixed) return;
    const uint32_t b0 = first + g * 32u * NW;
    size_t o          = size_t(offsets[g]);
    if (o < capacity) groups[o] = b0;
    ++o;
#pragma unroll
    for (int w = 0; w < NW; ++w)
    {
        unsigned m = masks[size_t(g) * NW + w];
        while (m)
        {
            int k = __ffs(m) - 1;
            m &= m - 1;
            if (o < capacity) groups[o] = b0 + 32u * w + uint32_t(k) + 1u;
            ++o;
        }
    }
    if (g == numFixed - 1 && o < capacity) groups[o] = last;
}

// ---------------------------------------------------------------------------------------------------------------
// SFC gaps and spanning trees
// ---------------------------------------------------------------------------------------------------------------

template<class K>
__device__ __forceinline__ int lastNzPlace(K x)
{
    return x ? KeyTraits<K>::maxLevel - ctzKey<K>(x) / 3 : KeyTraits<K>::maxLevel;
}

// spanSfcRange (sfc/common.hpp:422-460): the cornerstone keys covering [a, b); counts them, stores them if out != 0
template<class K>
__device__ int spanSfcRange(K a, K b, K* out)
{
    int n         = 0;
    const int ub  = KeyTraits<K>::bits - 3 * KeyTraits<K>::maxLevel;
    int firstDiff = (clzKey<K>(a ^ b) + 3 - ub) / 3;
    int aLast = lastNzPlace<K>(a), bLast = lastNzPlace<K>(b);
    for (int pos = aLast; pos > firstDiff; --pos)
    {
        int digits = (8 - int(octalDigit<K>(a, unsigned(pos)))) % 8;
        n += digits;
        while (digits--)
        {
            if (out) *out++ = a;
            a += K(1) << (3 * (KeyTraits<K>::maxLevel - pos));
        }
    }
    for (int pos = firstDiff; pos <= bLast; ++pos)
    {
        int digits = int(octalDigit<K>(b, unsigned(pos))) - int(octalDigit<K>(a, unsigned(pos)));
        n += digits;
        while (digits--)
        {
            if (out) *out++ = a;
            a += K(1) << (3 * (KeyTraits<K>::maxLevel - pos));
        }
    }
    return n;
}

template<class K>
__global__ void countSfcGapsKernel(const K* __restrict__ tree, int numNodes, int32_t* ops)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < numNodes) ops[i] = spanSfcRange<K>(tree[i], tree[i + 1], nullptr);
}

template<class K>
__global__ void fillSfcGapsKernel(const K* __restrict__ tree, int numNodes, const int32_t* __restrict__ ops,
                                  K* newTree, int64_t capacity)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < numNodes)
    {
        int64_t o = ops[i], e = ops[i + 1];
        if (e <= capacity) spanSfcRange<K>(tree[i], tree[i + 1], newTree + o);
    }
    if (i == numNodes && int64_t(ops[numNodes]) < capacity) newTree[ops[numNodes]] = tree[numNodes];
}

} // namespace csg

using namespace csg;

// ---- upsweeps ----
extern "C" size_t cs_upsweep_workspace_bytes(int32_t num_nodes) { return size_t(num_nodes) * 4 + 256; }

extern "C" int cs_upsweep_sum(cs_stream_t stream, int num_levels, const int32_t* level_range_host,
                              const int32_t* child_offsets, const int32_t* parents, int32_t num_nodes,
                              uint32_t* node_counts, void* ws, size_t wsb)
{
    return upsweep<CountCombine>(cudaStream_t(stream), num_levels, level_range_host, child_offsets, parents,
                                 num_nodes, node_counts, ws, wsb);
}

#define CS_CENTER_ENTRIES(SUF, Tc, Tm, T)                                                                              \
    extern "C" int cs_leaf_source_centers_##SUF(cs_stream_t stream, const Tc* x, const Tc* y, const Tc* z,            \
                                               const Tm* m, const int32_t* leaf_to_internal, int32_t num_leaves,      \
                                               const uint32_t* layout, T* centers)                                   \
    {                                                                                                                  \
        if (num_leaves <= 0) return CS_OK;                                                                             \
        if (!x || !y || !z || !m || !leaf_to_internal || !layout || !centers)                                          \
        {                                                                                                              \
            setLastError("leaf source centres: null pointer");                                                         \
            return CS_ERR_INVALID;                                                                                     \
        }                                                                                                              \
        leafCentersKernel<Tc, Tm, T><<<iceil(size_t(num_leaves), 8 * LC_WARPS), 32 * LC_WARPS, 0,                    \
                                       cudaStream_t(stream)>>>(                                                       \
            x, y, z, m, leaf_to_internal, num_leaves, layout, centers);                                                \
        CSG_CHECK_LAUNCH();                                                                                            \
        return CS_OK;                                                                                                  \
    }

CS_CENTER_ENTRIES(f64, double, double, double)
CS_CENTER_ENTRIES(f64_m32, double, float, double)
CS_CENTER_ENTRIES(f32, float, float, float)

extern "C" int cs_upsweep_source_centers_f64(cs_stream_t stream, int num_levels, const int32_t* level_range_host,
                                             const int32_t* child_offsets, const int32_t* parents, int32_t num_nodes,
                                             double* centers, void* ws, size_t wsb)
{
    return upsweep<CenterCombine<double>>(cudaStream_t(stream), num_levels, level_range_host, child_offsets, parents,
                                          num_nodes, centers, ws, wsb);
}
extern "C" int cs_upsweep_source_centers_f32(cs_stream_t stream, int num_levels, const int32_t* level_range_host,
                                             const int32_t* child_offsets, const int32_t* parents, int32_t num_nodes,
                                             float* centers, void* ws, size_t wsb)
{
    return upsweep<CenterCombine<float>>(cudaStream_t(stream), num_levels, level_range_host, child_offsets, parents,
                                         num_nodes, centers, ws, wsb);
}

// ---- target groups ----
extern "C" size_t cs_group_splits_workspace_bytes(uint32_t num_particles, unsigned group_size)
{
    size_t nf = (size_t(num_particles) + group_size - 1) / std::max(1u, group_size);
    return nf * (2 * 4 + 4 + 4) + exclusiveScanWorkspaceBytes(nf + 1) + 1024;
}

template<class T>
static int groupSplits(cudaStream_t s, uint32_t first, uint32_t last, const T* x, const T* y, const T* z, const T* h,
                       const uint64_t* leaves, int32_t numLeaves, const uint32_t* layout, const cs_box* box,
                       unsigned groupSize, float tol, uint32_t* groups, size_t capacity, uint32_t* numGroupsHost,
                       void* ws, size_t wsb)
{
    if (groupSize != 32 && groupSize != 64)
    {
        setLastError("group splits: group size must be 32 or 64 (got %u)", groupSize);
        return CS_ERR_INVALID;
    }
    if (last < first || !box || !numGroupsHost || (last > first && (!x || !y || !z || !leaves || !layout)) ||
        (capacity && !groups) || numLeaves < 1)
    {
        setLastError("group splits: invalid arguments");
        return CS_ERR_INVALID;
    }
    const uint32_t nfix = (last - first + groupSize - 1) / groupSize;
    if (nfix == 0)
    {
        *numGroupsHost = 0;
        if (capacity) CSG_CUDA_TRY(cudaMemcpyAsync(groups, &last, sizeof(uint32_t), cudaMemcpyHostToDevice, s));
        return CS_OK;
    }
    Workspace w;
    int rc = w.acquire(ws, wsb, cs_group_splits_workspace_bytes(last - first, groupSize), s);
    if (rc) return rc;
    Arena ar{static_cast<char*>(w.ptr), 0, cs_group_splits_workspace_bytes(last - first, groupSize)};
    uint32_t* masks  = ar.take<uint32_t>(size_t(nfix) * 2);
    int32_t* nsplit  = ar.take<int32_t>(size_t(nfix) + 1);
    int32_t* offsets = ar.take<int32_t>(size_t(nfix) + 1);
    size_t scanBytes = exclusiveScanWorkspaceBytes(size_t(nfix) + 1);
    void* scanWs     = ar.take<char>(scanBytes);
    BoxParams<T> bp  = makeBoxParams<T>(*box);
    GroupArgs<T, uint64_t> a{first, last, x, y, z, h, leaves, numLeaves, layout, bp.ilen[0], bp.ilen[1], bp.ilen[2],
                             std::min(std::min(bp.len[0], bp.len[1]), bp.len[2]), tol};
    CSG_CUDA_TRY(cudaMemsetAsync(nsplit + nfix, 0, sizeof(int32_t), s));
    unsigned blocks = iceil(size_t(nfix) * 32, 256);
    if (groupSize == 32) groupSplitsKernel<1, T, uint64_t><<<blocks, 256, 0, s>>>(a, nfix, masks, nsplit);
    else groupSplitsKernel<2, T, uint64_t><<<blocks, 256, 0, s>>>(a, nfix, masks, nsplit);
    CSG_CHECK_LAUNCH();
    if ((rc = exclusiveScanI32(s, nsplit, offsets, size_t(nfix) + 1, 0, scanWs, scanBytes))) return rc;
    if (groupSize == 32)
        groupWriteKernel<1><<<iceil(nfix, 256), 256, 0, s>>>(masks, offsets, nfix, first, last, groups, capacity);
    else groupWriteKernel<2><<<iceil(nfix, 256), 256, 0, s>>>(masks, offsets, nfix, first, last, groups, capacity);
    CSG_CHECK_LAUNCH();
    int32_t total = 0;
    CSG_CUDA_TRY(cudaMemcpyAsync(&total, offsets + nfix, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    CSG_CUDA_TRY(cudaStreamSynchronize(s));
    *numGroupsHost = uint32_t(total);
    if (size_t(total) + 1 > capacity)
    {
        setLastError("group splits: %d groups need %d entries, capacity %zu", total, total + 1, capacity);
        return CS_ERR_CAPACITY;
    }
    return CS_OK;
}

extern "C" int cs_group_splits_f64(cs_stream_t stream, uint32_t first, uint32_t last, const double* x,
                                   const double* y, const double* z, const double* h, const uint64_t* leaves,
                                   int32_t num_leaves, const uint32_t* layout, const cs_box* box, unsigned group_size,
                                   float tol, uint32_t* groups, size_t groups_capacity, uint32_t* num_groups,
                                   void* ws, size_t wsb)
{
    return groupSplits<double>(cudaStream_t(stream), first, last, x, y, z, h, leaves, num_leaves, layout, box,
                               group_size, tol, groups, groups_capacity, num_groups, ws, wsb);
}
extern "C" int cs_group_splits_f32(cs_stream_t stream, uint32_t first, uint32_t last, const float* x, const float* y,
                                   const float* z, const float* h, const uint64_t* leaves, int32_t num_leaves,
                                   const uint32_t* layout, const cs_box* box, unsigned group_size, float tol,
                                   uint32_t* groups, size_t groups_capacity, uint32_t* num_groups, void* ws,
                                   size_t wsb)
{
    return groupSplits<float>(cudaStream_t(stream), first, last, x, y, z, h, leaves, num_leaves, layout, box,
                              group_size, tol, groups, groups_capacity, num_groups, ws, wsb);
}

// ---- SFC gaps and spanning trees ----
template<class K>
static int countGaps(cudaStream_t s, const K* tree, int32_t numNodes, int32_t* ops)
{
    if (numNodes <= 0) return CS_OK;
    if (!tree || !ops)
    {
        setLastError("count sfc gaps: null pointer");
        return CS_ERR_INVALID;
    }
    countSfcGapsKernel<K><<<iceil(size_t(numNodes), 256), 256, 0, s>>>(tree, numNodes, ops);
    CSG_CHECK_LAUNCH();
    return CS_OK;
}

template<class K>
static int fillGaps(cudaStream_t s, const K* tree, int32_t numNodes, const int32_t* ops, K* newTree, int64_t cap)
{
    if (numNodes < 0 || !tree || !ops || !newTree)
    {
        setLastError("fill sfc gaps: invalid arguments");
        return CS_ERR_INVALID;
    }
    fillSfcGapsKernel<K><<<iceil(size_t(numNodes) + 1, 128), 128, 0, s>>>(tree, numNodes, ops, newTree, cap);
    CSG_CHECK_LAUNCH();
    return CS_OK;
}

template<class K>
static int spanningTree(cudaStream_t s, const K* keys, int32_t numKeys, K* out, int32_t capacity, int32_t* outSize,
                        void* ws, size_t wsb)
{
    if (numKeys < 2 || !keys || !outSize)
    {
        setLastError("spanning tree: need at least 2 keys");
        return CS_ERR_INVALID;
    }
    const int32_t nn  = numKeys - 1;
    size_t scanBytes  = exclusiveScanWorkspaceBytes(size_t(nn) + 1);
    size_t need       = (size_t(nn) + 1) * 4 * 2 + scanBytes + 1024;
    Workspace w;
    int rc = w.acquire(ws, wsb, need, s);
    if (rc) return rc;
    Arena ar{static_cast<char*>(w.ptr), 0, need};
    int32_t* cnt = ar.take<int32_t>(size_t(nn) + 1);
    int32_t* off = ar.take<int32_t>(size_t(nn) + 1);
    void* sws    = ar.take<char>(scanBytes);
    CSG_CUDA_TRY(cudaMemsetAsync(cnt + nn, 0, sizeof(int32_t), s));
    if ((rc = countGaps<K>(s, keys, nn, cnt))) return rc;
    if ((rc = exclusiveScanI32(s, cnt, off, size_t(nn) + 1, 0, sws, scanBytes))) return rc;
    if ((rc = fillGaps<K>(s, keys, nn, off, out, int64_t(capacity)))) return rc;
    int32_t total = 0;
    CSG_CUDA_TRY(cudaMemcpyAsync(&total, off + nn, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    CSG_CUDA_TRY(cudaStreamSynchronize(s));
    *outSize = total + 1;
    if (total + 1 > capacity)
    {
        setLastError("spanning tree: %d keys needed, capacity %d", total + 1, capacity);
        return CS_ERR_CAPACITY;
    }
    return CS_OK;
}

extern "C" int cs_count_sfc_gaps_u32(cs_stream_t stream, const uint32_t* tree, int32_t num_nodes, int32_t* node_ops)
{
    return countGaps<uint32_t>(cudaStream_t(stream), tree, num_nodes, node_ops);
}
extern "C" int cs_count_sfc_gaps_u64(cs_stream_t stream, const uint64_t* tree, int32_t num_nodes, int32_t* node_ops)
{
    return countGaps<uint64_t>(cudaStream_t(stream), tree, num_nodes, node_ops);
}
extern "C" int cs_fill_sfc_gaps_u32(cs_stream_t stream, const uint32_t* tree, int32_t num_nodes,
                                    const int32_t* node_ops, uint32_t* new_tree)
{
    return fillGaps<uint32_t>(cudaStream_t(stream), tree, num_nodes, node_ops, new_tree, INT64_MAX);
}
extern "C" int cs_fill_sfc_gaps_u64(cs_stream_t stream, const uint64_t* tree, int32_t num_nodes,
                                    const int32_t* node_ops, uint64_t* new_tree)
{
    return fillGaps<uint64_t>(cudaStream_t(stream), tree, num_nodes, node_ops, new_tree, INT64_MAX);
}
extern "C" size_t cs_spanning_tree_workspace_bytes(int32_t num_keys)
{
    return (size_t(num_keys) + 1) * 8 + exclusiveScanWorkspaceBytes(size_t(num_keys) + 1) + 1024;
}
extern "C" int cs_spanning_tree_u32(cs_stream_t stream, const uint32_t* keys, int32_t num_keys, uint32_t* out,
                                    int32_t capacity, int32_t* out_size, void* ws, size_t wsb)
{
    return spanningTree<uint32_t>(cudaStream_t(stream), keys, num_keys, out, capacity, out_size, ws, wsb);
}
extern "C" int cs_spanning_tree_u64(cs_stream_t stream, const uint64_t* keys, int32_t num_keys, uint64_t* out,
                                    int32_t capacity, int32_t* out_size, void* ws, size_t wsb)
{
    return spanningTree<uint64_t>(cudaStream_t(stream), keys, num_keys, out, capacity, out_size, ws, wsb);
}
