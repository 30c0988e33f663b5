// Stable LSD radix sort of (key, uint32 value) pairs: one histogram kernel for all digit positions, then one
// "onesweep" kernel per 8-bit digit (Adinets & Merrill, "Onesweep: a faster least significant digit radix sort for
// GPUs", 2022). Each block takes the next tile (256 threads x 16 or 12 keys: a runtime choice, SortShape) from an
// atomic counter, ranks its keys by digit in input
// order (ballots + per-warp counters), publishes its per-digit counts and obtains the counts of all earlier tiles
// by decoupled look-back, then scatters through shared memory so that global writes are runs of consecutive
// addresses. Traffic per pass: 2 * (sizeof(K) + 4) bytes per pair; the histogram reads the keys once.
//
// What bounds it: latency and issue in equal parts (55 % of the issue slots at 24 warps per SM; a pass moves 2.3 to 2.9
// TB/s, 34 to 43 % of the measured copy rate). 16M 64-bit keys 1.47 -> 1.15 ms, 20M 32-bit keys 1.02 -> 0.70 ms with the
// ballots in the ranking (a match instruction per key had bound every pass at 100 cycles each), pipelined counter
// additions and four keys in flight per thread of the histogram (103 -> 52 us for 20M 32-bit keys).
//
// Look-back waits spin on a flag that an earlier tile (which has already started, because tiles are handed out in
// order) will publish; every wait is bounded, and a wait that gives up sets ERRBIT_SORT_TIMEOUT and continues.
#include "radix_sort.cuh"

#include <algorithm>
#include <cstdio>

namespace csg
{

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS   = RS_THREADS / 32;
constexpr int RS_MIN_TILE = RS_THREADS * 12; // the smaller of the two tile shapes sizes the workspace
constexpr int RS_BINS    = 256;
constexpr int RS_MAXPASS = 8;

constexpr uint32_t ST_AGG   = 1u << 30;
constexpr uint32_t ST_INC   = 2u << 30;
constexpr uint32_t ST_FLAGS = 3u << 30;
constexpr uint32_t ST_COUNT = (1u << 30) - 1;


// resident blocks per SM of the 16-key tiles: what shared memory holds for 64-bit keys; 20M 32-bit keys 0.71 ms with 3,
// 0.68 with 4, 0.93 with 5 (spilling)
template<class K>
constexpr int RS_BLOCKS16 = sizeof(K) == 4 ? 4 : 3;

struct SortLayout
{
    uint32_t* hist;        // [passes][256]
    uint32_t* status;      // [passes][tiles][256]
    uint32_t* tileCounter; // [passes]
    size_t tiles;
    int passes;
};

static inline int numPasses(int beginBit, int endBit) { return (endBit - beginBit + 7) / 8; }

template<class K>
static SortLayout sortLayout(Arena& a, size_t n, int beginBit, int endBit, int tile)
{
    SortLayout L;
    L.passes      = numPasses(beginBit, endBit);
    L.tiles       = (n + tile - 1) / tile;
    L.hist        = a.take<uint32_t>(size_t(RS_MAXPASS) * RS_BINS);
    L.tileCounter = a.take<uint32_t>(RS_MAXPASS);
    L.status      = a.take<uint32_t>(size_t(L.passes) * L.tiles * RS_BINS + 1);
    return L;
}

template<class K>
size_t radixSortWorkspaceBytes(size_t n, int beginBit, int endBit)
{
    Arena a;
    sortLayout<K>(a, n, beginBit, endBit, RS_MIN_TILE);
    return a.size + 256;
}

template<class K>
__device__ __forceinline__ uint32_t digitOf(K key, int shift, uint32_t mask)
{
    return uint32_t(key >> shift) & mask;
}

// all digit histograms in one read of the keys
template<class K>
__global__ void __launch_bounds__(256) radixHistogramKernel(const K* __restrict__ keys, size_t n, int beginBit,
                                                            int endBit, int passes, uint32_t* __restrict__ hist)
{
    __shared__ uint32_t sh[2][RS_MAXPASS][RS_BINS];
    for (int i = threadIdx.x; i < 2 * RS_MAXPASS * RS_BINS; i += blockDim.x)
        (&sh[0][0][0])[i] = 0;
    __syncthreads();

    const int copy = (threadIdx.x >> 5) & 1;
    const int lane = threadIdx.x & 31;
    // four keys per thread and round, loaded before any is counted
    constexpr int U     = 4;
    const size_t stride = size_t(gridDim.x) * 256 * U;
    for (size_t i0 = size_t(blockIdx.x) * 256 * U; i0 < n; i0 += stride)
    {
        K key[U];
        const bool full = i0 + 256 * U <= n;
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const size_t i = i0 + u * 256 + threadIdx.x;
            key[u]         = full || i < n ? keys[i] : K(0);
        }
        for (int p = 0; p < passes; ++p)
        {
            const int shift     = beginBit + 8 * p;
            const uint32_t mask = (1u << min(8, endBit - shift)) - 1u;
#pragma unroll
            for (int u = 0; u < U; ++u)
            {
                const bool valid = full || i0 + u * 256 + threadIdx.x < n;
                const uint32_t d = digitOf(key[u], shift, mask);
                // one addition for a warp whose keys share the digit (the high digits of clustered or sorted keys)
                int same;
                __match_all_sync(0xffffffffu, valid ? d : ~0u, &same);
                if (same)
                {
                    if (lane == 0 && valid) atomicAdd(&sh[copy][p][d], 32u);
                }
                else if (valid) { atomicAdd(&sh[copy][p][d], 1u); }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * RS_BINS; i += blockDim.x)
    {
        uint32_t c = (&sh[0][0][0])[i] + (&sh[1][0][0])[i];
        if (c) atomicAdd(hist + i, c);
    }
}

// exclusive scan of 256 values held one per thread (blockDim.x == 256)
__device__ __forceinline__ uint32_t blockExclusiveScan256(uint32_t v, uint32_t* sWarpSums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x     = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sWarpSums[warp] = x;
    __syncthreads();
    if (warp == 0)
    {
        uint32_t w = lane < RS_WARPS ? sWarpSums[lane] : 0;
#pragma unroll
        for (int o = 1; o < RS_WARPS; o <<= 1)
        {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < RS_WARPS) sWarpSums[lane] = w; // inclusive warp sums
    }
    __syncthreads();
    uint32_t warpPrefix = warp > 0 ? sWarpSums[warp - 1] : 0;
    return warpPrefix + x - v;
}

// the lanes of the warp whose digit equals this lane's, by eight ballots: a match instruction takes time in proportion to
// the distinct values (100 cycles of the shared-memory pipe for random digits)
__device__ __forceinline__ unsigned digitPeers(uint32_t d)
{
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; ++b)
    {
        const int set    = int(d << (31 - b)) >> 31; // all ones if bit b is set
        const unsigned m = __ballot_sync(0xffffffffu, set != 0);
        peers &= ~(m ^ unsigned(set));
    }
    return peers;
}

// rank of each of a warp's keys among the warp's keys of the same digit, in input order (item-major); hist (zero before)
// then holds the warp's digit counts
template<class K, int Items>
__device__ __forceinline__ void rankItems(const K (&k)[Items], int shift, uint32_t mask, int lane, uint32_t* hist,
                                          uint32_t (&rank)[Items])
{
    constexpr int Group   = 4; // items in flight
    const unsigned ltMask = (1u << lane) - 1u;
    static_assert(Items % Group == 0);
#pragma unroll
    for (int j0 = 0; j0 < Items; j0 += Group)
    {
        uint32_t old[Group];
        unsigned peers[Group];
#pragma unroll
        for (int u = 0; u < Group; ++u)
            peers[u] = digitPeers(digitOf(k[j0 + u], shift, mask));
#pragma unroll
        for (int u = 0; u < Group; ++u)
        {
            old[u] = 0;
            if ((peers[u] >> lane) == 1u) old[u] = atomicAdd(hist + digitOf(k[j0 + u], shift, mask), __popc(peers[u]));
            __syncwarp();
        }
#pragma unroll
        for (int u = 0; u < Group; ++u)
            rank[j0 + u] = __shfl_sync(0xffffffffu, old[u], 31 - __clz(peers[u])) + __popc(peers[u] & ltMask);
    }
}

template<class K, bool Iota, int Items, int MinBlocks>
__global__ void __launch_bounds__(RS_THREADS, MinBlocks) onesweepKernel(const K* __restrict__ keysIn,
                                                             const uint32_t* __restrict__ valsIn,
                                                             K* __restrict__ keysOut, uint32_t* __restrict__ valsOut,
                                                             size_t n, int shift, uint32_t mask,
                                                             const uint32_t* __restrict__ passHist,
                                                             uint32_t* status, uint32_t* tileCounter,
                                                             uint32_t* errWord, uint32_t spinLimit, int stallTile1)
{
    constexpr int Tile = RS_THREADS * Items;
    extern __shared__ __align__(16) unsigned char smem[];
    K* sKeys        = reinterpret_cast<K*>(smem);
    uint32_t* sVals = reinterpret_cast<uint32_t*>(smem + Tile * sizeof(K));

    __shared__ uint32_t sWarpHist[RS_WARPS][RS_BINS];
    __shared__ uint32_t sTileOff[RS_BINS];
    __shared__ uint32_t sGlobalBase[RS_BINS];
    __shared__ uint32_t sWarpSums[RS_WARPS];
    __shared__ uint32_t sTile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) sTile = atomicAdd(tileCounter, 1u);
    for (int i = tid; i < RS_WARPS * RS_BINS; i += RS_THREADS)
        (&sWarpHist[0][0])[i] = 0;
    __syncthreads();

    const uint32_t tile   = sTile;
    const size_t tileBase = size_t(tile) * Tile;
    const size_t warpBase = tileBase + size_t(warp) * Items * 32;

    K k[Items];
    uint32_t v[Items];
#pragma unroll
    for (int j = 0; j < Items; ++j)
    {
        size_t idx = warpBase + j * 32 + lane;
        if (idx < n)
        {
            k[j] = keysIn[idx];
            v[j] = Iota ? uint32_t(idx) : valsIn[idx];
        }
        else
        {
            k[j] = ~K(0); // padding ranks after every real key in the last digit bucket, lands at positions >= n
            v[j] = 0;
        }
    }

    // rank within the warp's sub-tile, in input order: the last lane of each digit's peers adds their number to the
    // warp's counter and gets the count of earlier items back, several items in flight
    uint32_t rank[Items];
    rankItems<K, Items>(k, shift, mask, lane, sWarpHist[warp], rank);
    __syncthreads();

    // per digit (one thread per digit): tile total and per-warp exclusive prefixes
    const uint32_t dg = tid;
    uint32_t total    = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w)
    {
        uint32_t c        = sWarpHist[w][dg];
        sWarpHist[w][dg]  = total;
        total            += c;
    }
    volatile uint32_t* vstatus = status;
    size_t myIdx               = size_t(tile) * RS_BINS + dg;
    if (tile == 0) { vstatus[myIdx] = ST_INC | total; }
    else { vstatus[myIdx] = ST_AGG | total; }

    uint32_t excl = blockExclusiveScan256(total, sWarpSums);
    sTileOff[dg]  = excl;

    // decoupled look-back for this digit
    uint32_t prefix = 0;
    if (tile > 0)
    {
        // four predecessors per round (independent loads), consumed in order down to the first inclusive entry;
        // an unpublished entry ends the round and is read again. Below tile 0 reads as an empty inclusive entry.
        constexpr int LB = 4;
        long t          = long(tile) - 1;
        uint32_t spins  = 0;
        bool timedOut   = false;
        while (true)
        {
            uint32_t st[LB];
#pragma unroll
            for (int u = 0; u < LB; ++u)
                st[u] = t - u >= 0 ? uint32_t(vstatus[size_t(t - u) * RS_BINS + dg]) : uint32_t(ST_INC);
            // test mode: tile 1 waits for an entry that is never published, until the spin limit
            if (stallTile1 && tile == 1) st[0] = 0;
            int used  = 0;
            bool done = false, wait = false;
#pragma unroll
            for (int u = 0; u < LB; ++u)
            {
                if (done || wait) continue;
                if ((st[u] & ST_FLAGS) == 0)
                {
                    wait = true;
                    continue;
                }
                prefix += st[u] & ST_COUNT;
                used++;
                if (st[u] & ST_INC) done = true;
            }
            if (done) break;
            t -= used;
            if (wait)
            {
                if (++spins > spinLimit)
                {
                    timedOut = true;
                    break;
                }
                __nanosleep(20);
            }
        }
        if (timedOut) atomicOr(errWord, ERRBIT_SORT_TIMEOUT);
        vstatus[myIdx] = ST_INC | (prefix + total);
    }
    sGlobalBase[dg] = passHist[dg] + prefix - excl; // global position of the tile's slot 0 were it of this digit
    __syncthreads();

    // scatter into shared memory in (digit, input order) order
#pragma unroll
    for (int j = 0; j < Items; ++j)
    {
        uint32_t d   = digitOf(k[j], shift, mask);
        uint32_t pos = sTileOff[d] + sWarpHist[warp][d] + rank[j];
        sKeys[pos]   = k[j];
        sVals[pos]   = v[j];
    }
    __syncthreads();

    // coalesced write-out: consecutive shared slots of one digit go to consecutive global positions
#pragma unroll 4
    for (int i = tid; i < Tile; i += RS_THREADS)
    {
        K key      = sKeys[i];
        uint32_t d = digitOf(key, shift, mask);
        const uint32_t out = sGlobalBase[d] + uint32_t(i); // modulo 2^32, n < 2^30
        if (out < n)
        {
            keysOut[out] = key;
            valsOut[out] = sVals[i];
        }
    }
}

// Small sorts in one block: every pass in shared memory, 256 keys per warp, 8 per lane. The general path is ten dependent
// launches of one or two tiles (4096 64-bit keys: 93 us of kernels, 27 us here), each a look-back, a histogram and a
// trip through global memory; up to 8192 keys the block is faster, and its shared memory ends there.
constexpr int SS_ITEMS = 8;
constexpr int SS_MAX   = 32 * 32 * SS_ITEMS;

template<class K>
__global__ void __launch_bounds__(1024) smallSortKernel(K* keys, uint32_t* vals, int n, int beginBit, int endBit, int iota)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int slots = blockDim.x * SS_ITEMS, warps = blockDim.x >> 5;
    K* sKeys        = reinterpret_cast<K*>(smem);
    uint32_t* sVals = reinterpret_cast<uint32_t*>(sKeys + slots);
    uint32_t* sHist = sVals + slots; // [warps][256]
    __shared__ uint32_t sTileOff[RS_BINS];
    __shared__ uint32_t sWarpSums[RS_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, base = warp * 32 * SS_ITEMS;
    K k[SS_ITEMS];
    uint32_t v[SS_ITEMS];
#pragma unroll
    for (int j = 0; j < SS_ITEMS; ++j)
    {
        const int i = base + j * 32 + lane;
        k[j]        = i < n ? keys[i] : ~K(0); // padding stays behind every key
        v[j]        = i < n ? (iota ? uint32_t(i) : vals[i]) : 0u;
    }
    for (int shift = beginBit; shift < endBit; shift += 8)
    {
        const uint32_t mask = (1u << min(8, endBit - shift)) - 1u;
        for (int b = tid; b < warps * RS_BINS; b += blockDim.x)
            sHist[b] = 0;
        __syncthreads();
        uint32_t rank[SS_ITEMS];
        rankItems<K, SS_ITEMS>(k, shift, mask, lane, sHist + warp * RS_BINS, rank);
        __syncthreads();
        uint32_t total = 0;
        if (tid < RS_BINS)
            for (int w = 0; w < warps; ++w)
            {
                const uint32_t c           = sHist[w * RS_BINS + tid];
                sHist[w * RS_BINS + tid] = total;
                total += c;
            }
        // exclusive scan of the 256 totals by the first eight warps
        uint32_t x = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31 && warp < RS_WARPS) sWarpSums[warp] = x;
        __syncthreads();
        if (tid < RS_BINS)
        {
            uint32_t before = 0;
            for (int w = 0; w < warp; ++w)
                before += sWarpSums[w];
            sTileOff[tid] = before + x - total;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < SS_ITEMS; ++j)
        {
            const uint32_t d   = digitOf(k[j], shift, mask);
            const uint32_t pos = sTileOff[d] + sHist[warp * RS_BINS + d] + rank[j];
            sKeys[pos]         = k[j];
            sVals[pos]         = v[j];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < SS_ITEMS; ++j)
        {
            k[j] = sKeys[base + j * 32 + lane];
            v[j] = sVals[base + j * 32 + lane];
        }
    }
#pragma unroll
    for (int j = 0; j < SS_ITEMS; ++j)
    {
        const int i = base + j * 32 + lane;
        if (i < n) keys[i] = k[j], vals[i] = v[j];
    }
}

template<class K>
static int smallSort(cudaStream_t s, K* keys, uint32_t* vals, size_t n, int beginBit, int endBit, bool iota)
{
    const int warps    = std::max(RS_WARPS, int((n + 32 * SS_ITEMS - 1) / (32 * SS_ITEMS)));
    const size_t bytes = size_t(warps) * (32 * SS_ITEMS * (sizeof(K) + sizeof(uint32_t)) + RS_BINS * sizeof(uint32_t));
    CSG_CUDA_TRY(cudaFuncSetAttribute(smallSortKernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(32 * (32 * SS_ITEMS * (sizeof(K) + sizeof(uint32_t)) + RS_BINS * sizeof(uint32_t)))));
    smallSortKernel<K><<<1, warps * 32, bytes, s>>>(keys, vals, int(n), beginBit, endBit, iota ? 1 : 0);
    CSG_CHECK_LAUNCH();
    return CS_OK;
}

__global__ void iotaKernel(uint32_t* v, size_t n)
{
    size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) v[i] = uint32_t(i);
}

// exclusive scan of each pass's 256-bin histogram, in place (one block per pass)
__global__ void histScanKernel(uint32_t* hist)
{
    __shared__ uint32_t sWarpSums[RS_WARPS];
    uint32_t* h = hist + size_t(blockIdx.x) * RS_BINS;
    uint32_t v  = h[threadIdx.x];
    uint32_t e  = blockExclusiveScan256(v, sWarpSums);
    h[threadIdx.x] = e;
}

// the onesweep passes with one tile shape (Items keys per thread, MinBlocks resident blocks per SM); on return kin /
// vin point at the buffers holding the result
template<class K, int Items, int MinBlocks>
static int onesweepPasses(cudaStream_t s, K*& kin, uint32_t*& vin, K* keysAlt, uint32_t* valsAlt, size_t n,
                          int beginBit, int endBit, bool iota, const SortLayout& L, uint32_t* err)
{
    const size_t smemBytes = size_t(RS_THREADS) * Items * (sizeof(K) + sizeof(uint32_t));
    CSG_CUDA_TRY(cudaFuncSetAttribute(onesweepKernel<K, true, Items, MinBlocks>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, int(smemBytes)));
    CSG_CUDA_TRY(cudaFuncSetAttribute(onesweepKernel<K, false, Items, MinBlocks>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, int(smemBytes)));
    const WaitLimits wl = waitLimits();
    const int stall     = (wl.stall & CS_WAIT_STALL_SORT) ? 1 : 0;
    K* kout             = keysAlt;
    uint32_t* vout      = valsAlt;
    for (int p = 0; p < L.passes; ++p)
    {
        int shift     = beginBit + 8 * p;
        int bitsHere  = std::min(8, endBit - shift);
        uint32_t mask = (1u << bitsHere) - 1u;
        uint32_t* st  = L.status + size_t(p) * L.tiles * RS_BINS;
        if (p == 0 && iota)
            onesweepKernel<K, true, Items, MinBlocks><<<unsigned(L.tiles), RS_THREADS, smemBytes, s>>>(
                kin, vin, kout, vout, n, shift, mask, L.hist + p * RS_BINS, st, L.tileCounter + p, err, wl.sortSpins,
                stall);
        else
            onesweepKernel<K, false, Items, MinBlocks><<<unsigned(L.tiles), RS_THREADS, smemBytes, s>>>(
                kin, vin, kout, vout, n, shift, mask, L.hist + p * RS_BINS, st, L.tileCounter + p, err, wl.sortSpins,
                stall);
        CSG_CHECK_LAUNCH();
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    return CS_OK;
}

template<class K>
int radixSortPairs(cudaStream_t s, K* keys, uint32_t* vals, K* keysAlt, uint32_t* valsAlt, size_t n, int beginBit,
                   int endBit, bool iota, void* ws, size_t wsBytes, uint32_t* errWord, bool* resultInAlt,
                   int sortItems)
{
    constexpr int KB = 8 * sizeof(K);
    if (beginBit < 0 || endBit > KB || beginBit > endBit)
    {
        setLastError("sort: invalid bit range [%d, %d)", beginBit, endBit);
        return CS_ERR_INVALID;
    }
    if (n >= (size_t(1) << 30))
    {
        setLastError("sort: n = %zu exceeds the 2^30 limit", n);
        return CS_ERR_INVALID;
    }
    if (resultInAlt) *resultInAlt = false;
    if (n == 0) return CS_OK;
    int passes = numPasses(beginBit, endBit);
    if (passes == 0 || n == 1)
    {
        // nothing to reorder; the values still become 0..n-1 when asked for
        if (iota)
        {
            iotaKernel<<<iceil(n, 256), 256, 0, s>>>(vals, n);
            CSG_CHECK_LAUNCH();
        }
        return CS_OK;
    }

    if (sortItems != 0 && sortItems != 12 && sortItems != 16)
    {
        setLastError("sort: keys per thread must be 12 or 16 (0: the default, 16)");
        return CS_ERR_INVALID;
    }
    Arena a{static_cast<char*>(ws), 0, wsBytes};
    SortLayout L = sortLayout<K>(a, n, beginBit, endBit, RS_THREADS * (sortItems == 12 ? 12 : 16));
    if (!a.ok())
    {
        setLastError("sort: workspace too small");
        return CS_ERR_INVALID;
    }
    if (!errWord)
    {
        setLastError("sort: internal error word missing");
        return CS_ERR_INVALID;
    }
    uint32_t* err = errWord;
    // (the test mode that stalls a look-back needs one)
    if (n <= size_t(SS_MAX) && !(waitLimits().stall & CS_WAIT_STALL_SORT))
        return smallSort<K>(s, keys, vals, n, beginBit, endBit, iota);

    size_t zeroBytes = (reinterpret_cast<char*>(L.status + size_t(L.passes) * L.tiles * RS_BINS) -
                        reinterpret_cast<char*>(L.hist));
    CSG_CUDA_TRY(cudaMemsetAsync(L.hist, 0, zeroBytes, s));

    {
        unsigned grid = unsigned(std::min<size_t>((n + 1023) / 1024, size_t(smCount()) * 8));
        radixHistogramKernel<K><<<grid, 256, 0, s>>>(keys, n, beginBit, endBit, passes, L.hist);
        CSG_CHECK_LAUNCH();
        histScanKernel<<<passes, RS_BINS, 0, s>>>(L.hist);
        CSG_CHECK_LAUNCH();
    }

    K* kin        = keys;
    uint32_t* vin = vals;
    int rc        = sortItems == 12
                        ? onesweepPasses<K, 12, 4>(s, kin, vin, keysAlt, valsAlt, n, beginBit, endBit, iota, L, err)
                        : onesweepPasses<K, 16, RS_BLOCKS16<K>>(s, kin, vin, keysAlt, valsAlt, n, beginBit, endBit, iota, L, err);
    if (rc) return rc;
    bool inAlt = (kin == keysAlt);
    if (resultInAlt) { *resultInAlt = inAlt; }
    else if (inAlt)
    {
        CSG_CUDA_TRY(cudaMemcpyAsync(keys, keysAlt, n * sizeof(K), cudaMemcpyDeviceToDevice, s));
        CSG_CUDA_TRY(cudaMemcpyAsync(vals, valsAlt, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    }
    return CS_OK;
}

template<class K>
int radixSortPreload()
{
    cudaFuncAttributes fa;
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, radixHistogramKernel<K>));
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, histScanKernel));
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, iotaKernel));
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, smallSortKernel<K>));
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, onesweepKernel<K, true, 16, RS_BLOCKS16<K>>));
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, onesweepKernel<K, false, 16, RS_BLOCKS16<K>>));
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, onesweepKernel<K, true, 12, 4>));
    CSG_CUDA_TRY(cudaFuncGetAttributes(&fa, onesweepKernel<K, false, 12, 4>));
    return CS_OK;
}

template int radixSortPreload<uint32_t>();
template int radixSortPreload<uint64_t>();
template size_t radixSortWorkspaceBytes<uint32_t>(size_t, int, int);
template size_t radixSortWorkspaceBytes<uint64_t>(size_t, int, int);
template int radixSortPairs<uint32_t>(cudaStream_t, uint32_t*, uint32_t*, uint32_t*, uint32_t*, size_t, int, int, bool,
                                      void*, size_t, uint32_t*, bool*, int);
template int radixSortPairs<uint64_t>(cudaStream_t, uint64_t*, uint32_t*, uint64_t*, uint32_t*, size_t, int, int, bool,
                                      void*, size_t, uint32_t*, bool*, int);

} // namespace csg

using namespace csg;

extern "C" size_t cs_sort_pairs_workspace_bytes(size_t n, int key_bits)
{
    size_t b = key_bits == 32 ? radixSortWorkspaceBytes<uint32_t>(n, 0, 32) : radixSortWorkspaceBytes<uint64_t>(n, 0, 64);
    return b + 512; // + error word
}

template<class K>
static int sortEntry(cs_stream_t stream, K* keys, uint32_t* values, size_t n, K* keysAlt, uint32_t* valuesAlt,
                     int beginBit, int endBit, int iota, void* ws, size_t wsBytes)
{
    if (n == 0) return CS_OK;
    if (!keys || !values || !keysAlt || !valuesAlt)
    {
        setLastError("sort: null pointer");
        return CS_ERR_INVALID;
    }
    cudaStream_t s = cudaStream_t(stream);
    size_t need    = radixSortWorkspaceBytes<K>(n, beginBit, endBit) + 512;
    Workspace w;
    int rc = w.acquire(ws, wsBytes, need, s);
    if (rc) return rc;
    char* base     = static_cast<char*>(w.ptr);
    uint32_t* err  = reinterpret_cast<uint32_t*>(base + need - 256);
    CSG_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(uint32_t), s));
    rc = radixSortPairs<K>(s, keys, values, keysAlt, valuesAlt, n, beginBit, endBit, iota != 0, base, need - 512, err,
                           nullptr);
    if (rc) return rc;
    // the reference's sortByKey synchronises the stream on return (primitives/primitives_gpu.h:152); so does this
    uint32_t herr = 0;
    CSG_CUDA_TRY(cudaMemcpyAsync(&herr, err, sizeof(herr), cudaMemcpyDeviceToHost, s));
    CSG_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr)
    {
        setLastError("sort: a look-back wait timed out");
        return CS_ERR_TIMEOUT;
    }
    return CS_OK;
}

extern "C" int cs_sort_pairs_u32(cs_stream_t stream, uint32_t* keys, uint32_t* values, size_t n, uint32_t* keys_alt,
                                 uint32_t* values_alt, int begin_bit, int end_bit, int iota, void* ws, size_t wsb)
{
    return sortEntry<uint32_t>(stream, keys, values, n, keys_alt, values_alt, begin_bit, end_bit, iota, ws, wsb);
}
extern "C" int cs_sort_pairs_u64(cs_stream_t stream, uint64_t* keys, uint32_t* values, size_t n, uint64_t* keys_alt,
                                 uint32_t* values_alt, int begin_bit, int end_bit, int iota, void* ws, size_t wsb)
{
    return sortEntry<uint64_t>(stream, keys, values, n, keys_alt, values_alt, begin_bit, end_bit, iota, ws, wsb);
}
