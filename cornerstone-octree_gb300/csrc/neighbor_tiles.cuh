// Neighbour search, 32 targets per warp with the pair tests on the tensor cores. Included by neighbors.cu, whose file
// header defines the semantics, the path-safe threshold Tsafe and the FP32 thresholds that the exact decisions rest on.
//
// A warp owns 32 consecutive (SFC-ordered) targets. Coordinates are floats relative to P, the centre of the targets.
//
// 1. Nodes. A stack of node codes in shared memory, lowest (in SFC order) on top. A step takes the leaves that lie on
//    top (up to 32, one per lane) and expands the internal ones among the next four entries, one child per lane: a
//    child survives if the distance of its box to the box of one of the four sub-groups of 8 targets is within that
//    sub-group's largest radius (every rounding widens the test). Leaves whose particles adjoin form one run.
// 2. Candidates. A run is read 32 particles at a time; a particle is kept if it lies in one of the four spheres that
//    enclose a sub-group's search spheres, and appended to a queue. The leaves that a warp's spheres touch hold about
//    three times as many particles as the spheres do, so this test (12 packed FP32 instructions) removes half of the
//    pair tests and, above all, fills the tiles.
// 3. Tiles. 32 queued candidates against the 32 targets: D = |a - b|^2 - Tin + E as eight mma.sync m16n8k16. Per axis
//    a coordinate is hi + lo in fp16 (22 bits), and the four products fill four of the 16 k; |a|^2 as hi + lo (against
//    ones) fills two more, |b|^2 - Tin + E as hi + lo another two. Sign bits become masks (one funnel shift per
//    value), and a 4 x 4 byte transpose among the four lanes of a quad gives every lane the 32-bit mask of its own
//    target, in candidate order. (tcgen05 needs 64 or 128 rows that share their candidates and a round trip through
//    shared memory, a barrier and TMEM per tile; a warp's candidates are its own, and the products are 4 % of the
//    issue slots here.)
//    Scale and error: coordinates are scaled by a power of two so that every kept |a| and every |b| is below 64. With
//    products exact, the two fp16 parts of a value v within 2^-22 |v|, |a|^2 and |b|^2 rounded in fp32, and the tensor
//    core's accumulation rounded (possibly truncated) to fp32 after each of 16 terms whose absolute sum is below 2^14:
//      2 * 2 * 64^2 * 2^-22 + 3 * 2^-24 * 2^12 * 2 + 2^-22 * (2^12 + 2^13) + 16 * 2^-23 * 2^14 < 0.045 < E = 1/16,
//    so D < 0 proves d2_f < Tin, and D >= W = max(Tup - Tin) + 2 E (scaled) proves d2_f >= Tup. |b|^2 - Tin + E is
//    within 2^12 + E because 0 <= Tin <= Tup (a negative Tin is raised to zero) and every target's sqrt(Tup) is a part
//    of its sphere's radius; with Tin = 0 a tile accepts no pair and leaves all below Tup undecided. The values between
//    (about two per warp of 32 targets x 100 neighbours) are tested again in FP32 on the frame coordinates and, where
//    that cannot decide either, in the reference's arithmetic.
// 4. Output. Every lane appends its target's hits in ascending candidate order, eight tiles at a time.
//
// Warps whose targets spread over more than eight of the smallest radius would lose the scaled precision; they take
// the leaves one by one, the warp looping over the targets that may reach the leaf with two ballots each (FP32,
// thresholds Tin and Tup). Those, and warps with a sub-group much larger than its radii or with many expansions, test
// nodes against the 32 search spheres.
//
// What bounds it: instruction issue (62 % of the slots) together with latency (fixed-latency chains, shared memory, L2)
// at 28 warps per SM; DRAM is at 10 %. 16M FP64 Plummer particles, 100 neighbours: 11.3 ms, where one lane per target
// with packed FP32 tests (two candidates per instruction, the output loop run per batch) took 17.0 ms; 15.9 against 31
// thousand warp instructions per 32 targets, of which nodes 3.7, rounds 3.8, tiles 3.8, output 3.9 thousand. 32M uniform FP32
// particles in a periodic box, 57 neighbours: 18.6 against 28.3 ms. 7 blocks of 4 warps per SM measured best (6: 11.9,
// 8: 12.0 ms, spilling); hits written after every tile: 14.9 ms, after 4 tiles: 11.9 ms.
//
// Stack bound: a step replaces at most four entries by at most 32 while fewer than NT_WIDE entries lie on the stack,
// and a single entry by at most 8 above, where the depth-first order adds at most 7 per level (21 levels) and one more:
// NT_WIDE + 28 + 7 * 21 + 8.
#pragma once

constexpr int NT_WIDE        = 128;
constexpr int NT_LOOSE_AFTER = 96; // node expansions
constexpr int NT_STACK       = NT_WIDE + 28 + 7 * 21 + 9;
// tiles whose hits are written together
constexpr int NT_DEFER      = 8;
constexpr int NT_MIN_BLOCKS = 7;

struct TileWarp
{
    int stack[NT_STACK];
    float4 queue[64];        // kept candidates: frame coordinates and index; a full half becomes fp16 records in place
    uint32_t tileJ[NT_DEFER][32];   // per tile: its candidate indices, the first one last
    uint32_t mask[NT_DEFER + 2][32]; // per lane: the hits of the tiles that have any (bit 31 - k: candidate k)
    float4 tgt[32];          // per lane: the target's frame coordinates, its node test radius squared
    float4 thr[32];          // per lane: Tin, Tup, Tsafe
    float4 boxLo[4];         // per sub-group: box of its targets; lo.w: its node test radius squared
    float4 boxHi[4];
    float4 sph[4];           // two sub-groups' spheres per pair of vectors: -x x' -y y' | -z z' r2 r2'
    uint32_t self[32];       // queue position of the warp's own particles
};

__device__ __forceinline__ float reduxMinF(float v)
{
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float reduxMaxF(float v)
{
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
// over the eight lanes of a sub-group (the lanes with the same lane % 4)
__device__ __forceinline__ float subMinF(float v)
{
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
        v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float subMaxF(float v)
{
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// v = hi + lo, hi and lo in fp16 (each rounded to nearest), hi in the low half
__device__ __forceinline__ uint32_t splitHalf(float v)
{
    const __half h  = __float2half_rn(v);
    const __half2 p = __floats2half2_rn(v, __fsub_rn(v, __half2float(h)));
    return *reinterpret_cast<const uint32_t*>(&p);
}

// D = A B for 16 targets (rows) x 8 candidates (columns)
__device__ __forceinline__ void tileMma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// byte s of lane t (of a quad, bytes counted from the top) becomes byte t of lane s
__device__ __forceinline__ uint32_t quadTranspose(uint32_t x, int lane)
{
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, 1);
    x                = __byte_perm(x, y, (lane & 1) ? 0x6240 : 0x3715);
    const uint32_t z = __shfl_xor_sync(0xffffffffu, x, 2);
    return __byte_perm(x, z, (lane & 2) ? 0x5410 : 0x3276);
}

// d2 < r2 of a pair, and the reference's cell tests on the path from a leaf to the root, exact in T, of a target whose
// search sphere may cross a periodic boundary (pbc: it does, and the differences are folded)
template<class T>
struct FoldTarget
{
    TargetRef<T> t;
    bool pbc;
};

template<class T>
__device__ __noinline__ bool foldPairWithin(FoldTarget<T> f, const BoxParams<T>& b, uint32_t j)
{
    T xi, yi, zi, r2, cellR2;
    loadTarget(f.t, xi, yi, zi, r2, cellR2);
    return pairDist2Exact<T>(xi, yi, zi, f.pbc, f.t.x[j], f.t.y[j], f.t.z[j], b) < r2;
}

template<class T>
__device__ __noinline__ bool foldPath(FoldTarget<T> f, const BoxParams<T>& b, int leafNode, const int32_t* parents,
                                      const T* centers, const T* sizes, int rootNode)
{
    T xi, yi, zi, r2, cellR2;
    loadTarget(f.t, xi, yi, zi, r2, cellR2);
    for (int n = leafNode;;)
    {
        if (!cellOverlapsExact<T>(xi, yi, zi, f.pbc, cellR2, centers + 3 * size_t(n), sizes + 3 * size_t(n), b)) return false;
        if (n <= rootNode) return true;
        n = parents[(n - 1) / 8];
    }
}

// Fold: the warps that hold a target whose search sphere crosses a periodic boundary (the other instance leaves them).
// Everything is folded to its image nearest to P. That is the image the reference takes for every pair within reach as
// long as a target's offset and radius together stay below half a period (foldSafe, with room to spare; the remaining
// warps go to the path kernel). The folds round at the period's scale: A and the node margin grow by 12 eps L; the pairs
// in the wider band are decided by the reference's folded expressions. 32M uniform FP32 particles: the 8 % of the warps
// at the boundary took 5.1 ms lane by lane in the path kernel; 2.7 ms here, and 0.6 ms for the path kernel, whose few
// remaining warps (targets on both sides of a jump of the curve) are one chain each.
template<class T, bool Stats, bool Fold>
__global__ void __launch_bounds__(NB_THREADS, NT_MIN_BLOCKS) findNeighborsTileKernel(NbArgs<T> a, NbPrep prep)
{
    constexpr bool F64  = std::is_same_v<T, double>;
    constexpr float EPS = EPS32;
    // rounding slack of the key quantisation / node boxes, and of the cell test, in units of C
    constexpr float KAPPA_REL = F64 ? 32.f * 2.220446e-16f : 32.f * 1.1920929e-7f;
    constexpr float RHO       = F64 ? 9.5367432e-7f : 7.6293945e-6f; // 2^-20, 2^-17
    constexpr float TILE_E    = 0.0625f;
    constexpr unsigned ALL    = 0xffffffffu;
    constexpr float INF       = INFINITY;

    __shared__ TileWarp sWarp[NB_WARPS];
    int tid; // volatile: kept in registers instead of read again from the special register
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    const int lane     = tid & 31;
    TileWarp& w        = sWarp[tid >> 5];
    const size_t wid   = size_t(blockIdx.x) * NB_WARPS + (tid >> 5);
    const size_t base0 = size_t(a.first) + wid * 32;
    if (base0 >= size_t(a.last)) return;
    if constexpr (Fold)
        if (a.nc[base0 - a.first] != NB_DEFERRED) return;
    // lane 4 g + t owns target g + 8 t: the row whose mask the quad transpose hands to it
    const int tau      = (lane >> 2) | ((lane & 3) << 3);
    const size_t i64   = base0 + tau;
    const bool active  = i64 < size_t(a.last);
    const uint32_t i   = active ? uint32_t(i64) : uint32_t(base0);
    const T xi = a.x[i], yi = a.y[i], zi = a.z[i];
    T r2, cellR2, twoh;
    targetRadii<T>(a.h, a.hf, i, a.ext, r2, cellR2, twoh);
    bool pbc = false;
    if (Fold || a.anyPbc)
    {
        const bool inside = RN<T>::sub(xi, twoh) >= a.b.lo[0] && RN<T>::sub(yi, twoh) >= a.b.lo[1] &&
                            RN<T>::sub(zi, twoh) >= a.b.lo[2] && RN<T>::add(xi, twoh) <= a.b.hi[0] &&
                            RN<T>::add(yi, twoh) <= a.b.hi[1] && RN<T>::add(zi, twoh) <= a.b.hi[2];
        pbc = !inside;
        if constexpr (!Fold)
            if (__any_sync(ALL, active && pbc))
            {
                if (lane == 0) a.nc[base0 - a.first] = NB_DEFERRED;
                return;
            }
    }
    float len[3] = {}, ilen[3] = {}, lenMax = 0.f; // Fold: the periods (0: not periodic)
    if constexpr (Fold)
    {
        if (!foldSafe<T>(xi, yi, zi, r2, a.b)) return; // stays deferred
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (a.b.pbc[k])
            {
                len[k]  = float(a.b.len[k]);
                ilen[k] = 1.f / len[k];
                lenMax  = fmaxf(lenMax, len[k]);
            }
    }
    // a target that is not finite (in FP32, the frame's type) has no neighbours and takes no part in the frame
    const bool live = active && fabsf(float(xi)) < INF && fabsf(float(yi)) < INF && fabsf(float(zi)) < INF;
    auto foldF = [&](float d, int k) { return Fold ? fmaf(-len[k], rintf(d * ilen[k]), d) : d; };
    const FoldTarget<T> ftarget{TargetRef<T>{a.x, a.y, a.z, a.h, a.hf, a.ext, i}, pbc};
    const TargetRef<T> tref = ftarget.t;
    const float C     = __fmul_ru(*prep.cmax, 1.f + 64 * EPS);
    const float delta = __fmul_ru(KAPPA_REL * 0.5f, C); // particle outside its node's float box by at most delta
    const float kappa = __fmul_ru(KAPPA_REL, C);
    const unsigned ngmax = a.ngmax;
    uint32_t* myNb       = a.nb + size_t(i - a.first) * ngmax;
    unsigned nc          = 0;
    const unsigned ltMask = (1u << lane) - 1u;
    unsigned long long stNodes = 0, stLeaves = 0, stCand = 0, stKept = 0, stTiles = 0, stAmb = 0, stExact = 0,
                       stRounds = 0, stDirect = 0, stSteps = 0;

    // one pass per set among the warp's targets (batched trees; a single pass otherwise)
    int mySet = 0, passSet = 0, lastSet = 0;
    if (a.numSets)
    {
        int lo = 0, hi = a.numSets;
        while (lo + 1 < hi)
        {
            int mid = (lo + hi) >> 1;
            if (__ldg(a.setOffsets + mid) <= i) lo = mid;
            else hi = mid;
        }
        mySet   = lo;
        passSet = __reduce_min_sync(ALL, active ? unsigned(mySet) : ALL);
        lastSet = int(__reduce_max_sync(ALL, active ? unsigned(mySet) : 0u));
    }
    for (;; ++passSet)
    {
        const bool inPass       = live && (!a.numSets || mySet == passSet);
        const unsigned passMask = __ballot_sync(ALL, inPass);
        const int rootNode      = a.numSets ? __ldg(a.setRoots + passSet) : 0;

        // ---- frame, radii and thresholds of the pass ----
        float P[3], b[3];
        {
            float f[3] = {float(xi), float(yi), float(zi)};
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                // Fold: the positions nearest to the first target's
                const float f0 = __shfl_sync(ALL, f[k], 0);
                if constexpr (Fold) f[k] = f0 + foldF(f[k] - f0, k);
                const float lo = reduxMinF(inPass ? f[k] : INF), hi = reduxMaxF(inPass ? f[k] : -INF);
                P[k] = fmaf(0.5f, hi - lo, lo);
            }
        }
        if constexpr (Fold)
        {
            const T q[3] = {xi, yi, zi};
#pragma unroll
            for (int k = 0; k < 3; ++k)
                b[k] = float(pbcFoldNb<T>(RN<T>::sub(q[k], T(P[k])), a.b.pbc[k], a.b.len[k], a.b.ilen[k]));
        }
        else if constexpr (F64)
        {
            b[0] = __double2float_rn(__dsub_rn(xi, double(P[0])));
            b[1] = __double2float_rn(__dsub_rn(yi, double(P[1])));
            b[2] = __double2float_rn(__dsub_rn(zi, double(P[2])));
        }
        else
        {
            b[0] = __fsub_rn(xi, P[0]);
            b[1] = __fsub_rn(yi, P[1]);
            b[2] = __fsub_rn(zi, P[2]);
        }
        const float R = __fmul_ru(reduxMaxF(inPass ? fmaxf(fabsf(b[0]), fmaxf(fabsf(b[1]), fabsf(b[2]))) : 0.f),
                                  1.f + 4 * EPS);
        const float A = __fmaf_ru(4 * EPS, R, __fmaf_ru(4 * EPS * EPS, C, 12 * EPS * lenMax));
        float rr, Tin, Tup;
        {
            float r2lo, r2hi, cLo, cHi;
            if constexpr (F64)
            {
                r2lo = __double2float_rd(r2);
                r2hi = __double2float_ru(r2);
                cLo  = __double2float_rd(cellR2);
                cHi  = __double2float_ru(cellR2);
            }
            else { r2lo = r2hi = r2; cLo = cHi = cellR2; }
            rr = __fsqrt_ru(r2hi);
            // Fold: a target whose sphere lies inside the box meets everything where it is. Below r - 2 kappa the folded
            // distance is that one (for particles and leaves in the box, up to its faces' rounding)
            if (Fold && !pbc) cLo = fminf(cLo, r2lo);
            const float tsafe =
                __fadd_rd(__fadd_rd(__fmul_rd(cLo, 1.f - RHO), -__fmul_ru(__fmul_ru(4.f, kappa), __fsqrt_ru(cHi))),
                          -__fmul_ru(__fmul_ru(4.f, kappa), kappa));
            const float m = __fmul_ru(__fmul_ru(8.f, A), rr), q = __fmul_ru(__fmul_ru(32.f, A), A);
            Tin = __fadd_rd(__fadd_rd(__fmul_rd(fminf(r2lo, tsafe), 1.f - 24 * EPS), -m), -q);
            Tup = __fadd_ru(__fadd_ru(__fmul_ru(r2hi, 1.f + 24 * EPS), m), q);
            if constexpr (!F64) // subnormal results of the reference's FP32 sums
            {
                Tin = __fsub_rd(Tin, 0x1p-146f);
                Tup = __fadd_ru(Tup, 0x1p-146f);
            }
            // no distance is below zero: the same decisions, and the tiles' sums stay within their bound (tsafe is far
            // below zero where the radius is small against kappa)
            Tin = fmaxf(Tin, 0.f);
            // nodes within the cell radius are visited too where it is the larger one: a particle outside its leaf's
            // box can be within r although the box is not
            const float rad = __fmul_ru(a.ext > 1.f ? fmaxf(rr, __fsqrt_ru(cHi)) : rr, 1.f + 64 * EPS);
            __syncwarp();
            w.tgt[lane]  = make_float4(b[0], b[1], b[2], inPass ? __fmul_ru(__fmul_ru(rad, rad), 1.f + 8 * EPS) : -1.f);
            w.thr[lane]  = make_float4(Tin, Tup, tsafe, 0.f);
            w.self[lane] = ALL;
        }

        // ---- sub-groups of 8 consecutive targets: box, largest radius, and the sphere around its search spheres ----
        bool spread;
        float gS;
        {
            float lo[3], hi[3], gc[3], d2 = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                lo[k] = subMinF(inPass ? b[k] : INF);
                hi[k] = subMaxF(inPass ? b[k] : -INF);
                gc[k] = lo[k] <= hi[k] ? 0.5f * (lo[k] + hi[k]) : 0.f;
                d2    = __fmaf_ru(b[k] - gc[k], b[k] - gc[k], d2);
            }
            const float rmax  = subMaxF(inPass ? rr : 0.f);
            const float reach = __fadd_ru(__fsqrt_ru(d2), __fsqrt_ru(fmaxf(Tup, 0.f)));
            const float gr    = subMaxF(inPass ? __fmul_ru(reach, 1.f + 16 * EPS) : -1.f);
            const float rad2  = subMaxF(w.tgt[lane].w);
            if (lane < 4)
            {
                w.boxLo[lane] = make_float4(lo[0], lo[1], lo[2], rad2);
                w.boxHi[lane] = make_float4(hi[0], hi[1], hi[2], 0.f);
                float* s      = reinterpret_cast<float*>(w.sph) + 8 * (lane >> 1) + (lane & 1);
                s[0] = -gc[0], s[2] = -gc[1], s[4] = -gc[2];
                s[6] = gr >= 0.f ? __fmul_ru(__fmul_ru(gr, gr), 1.f + 16 * EPS) : -1.f;
            }
            spread         = __any_sync(ALL, gr > 3.f * rmax);
            const float gl = __fsqrt_ru(__fmaf_ru(gc[2], gc[2], __fmaf_ru(gc[1], gc[1], __fmul_ru(gc[0], gc[0]))));
            gS             = __fmul_ru(reduxMaxF(gr >= 0.f ? __fadd_ru(gl, gr) : 0.f), 1.f + 16 * EPS);
        }
        const float rmin = reduxMinF(inPass ? rr : INF);
        // a power of two that brings the largest kept coordinate into [32, 64)
        const int ex     = 5 - ((__float_as_int(gS) >> 23) - 127);
        const bool mma   = gS <= 8.f * rmin && ex >= -60 && ex <= 60;
        const float sc   = __int_as_float((127 + (mma ? ex : 0)) << 23);
        bool loose       = spread || !mma;

        // ---- the targets as the rows of A, and the accumulator's start values ----
        uint32_t aLo[4] = {}, aHi[4] = {};
        uint32_t wBits = 0;
        if (mma)
        {
            uint32_t* tmp    = reinterpret_cast<uint32_t*>(w.queue);
            const float sc2  = sc * sc;
            const float tinS = Tin * sc2;
            float n2         = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                const float v      = b[k] * sc;
                n2                 = fmaf(v, v, n2);
                const uint32_t p   = inPass ? splitHalf(-2.f * v) : 0u;
                tmp[k * 32 + tau]       = __byte_perm(p, p, 0x1010);
                tmp[(3 + k) * 32 + tau] = __byte_perm(p, p, 0x3232);
            }
            tmp[6 * 32 + tau] = splitHalf(inPass ? n2 - tinS + TILE_E : 32768.f);
            wBits = __float_as_uint(reduxMaxF(inPass ? fmaf(Tup, sc2, 2.f * TILE_E) - tinS : 0.f) * (1.f + 16 * EPS));
            __syncwarp();
            const int t = lane & 3;
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                const int row = (lane >> 2) + 8 * k;
                aLo[k]        = t < 3 ? tmp[t * 32 + row] : 0x3c003c00u; // (1, 1) for |a|^2 = hi + lo
                aHi[k]        = tmp[(3 + t) * 32 + row];                 // lane 3: |b|^2 - Tin + E = hi + lo
            }
        }

        // particle j in the frame
        auto frame = [&](uint32_t j, float& ax, float& ay, float& az) {
            if constexpr (F64)
            {
                const float4 ph = prep.phi[j], pl = prep.plo[j];
                ax = foldF(__fadd_rn(__fsub_rn(ph.x, P[0]), pl.x), 0);
                ay = foldF(__fadd_rn(__fsub_rn(ph.y, P[1]), pl.y), 1);
                az = foldF(__fadd_rn(__fsub_rn(ph.z, P[2]), pl.z), 2);
            }
            else
            {
                ax = foldF(__fsub_rn(a.x[j], P[0]), 0);
                ay = foldF(__fsub_rn(a.y[j], P[1]), 1);
                az = foldF(__fsub_rn(a.z[j], P[2]), 2);
            }
        };
        // an upper bound of |x_i - leaf box|^2 below Tsafe proves that this target's path to the leaf passes the
        // reference's cell tests (the ancestors contain the leaf)
        auto pathSafe = [&](int leafNode) -> bool {
            const float4* r = prep.nrec + 3 * size_t(leafNode);
            const float4 ch = r[0], cl = r[1], s4 = r[2], tg = w.tgt[lane];
            const float cc[3] = {__fadd_rn(__fsub_rn(ch.x, P[0]), cl.x), __fadd_rn(__fsub_rn(ch.y, P[1]), cl.y),
                                 __fadd_rn(__fsub_rn(ch.z, P[2]), cl.z)};
            const float sz[3] = {s4.x, s4.y, s4.z}, bb[3] = {tg.x, tg.y, tg.z};
            float n2u = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                const float D = fabsf(foldF(__fsub_rn(cc[k], bb[k]), k));
                const float u = __fmaf_ru(4.5f * EPS, D + sz[k], __fmaf_ru(1.05f, A, delta));
                const float d = fmaxf(__fadd_ru(__fsub_ru(D, sz[k]), u), 0.f);
                n2u           = __fmaf_ru(d, d, n2u);
            }
            return n2u < w.thr[lane].z;
        };

        // exact decisions
        auto within = [&](uint32_t j) {
            if constexpr (Fold) return foldPairWithin<T>(ftarget, a.b, j);
            else return pairWithinAt(tref, j);
        };
        auto path = [&](int node) {
            if constexpr (Fold) return foldPath<T>(ftarget, a.b, node, a.parents, a.centers, a.sizes, rootNode);
            else return leafPathAt<T>(tref, node, a.parents, a.centers, a.sizes, rootNode);
        };

        // ---- traversal ----
        const float nodeMargin = __fmaf_ru(
            16 * EPS, R, __fadd_ru(__fadd_ru(delta, delta), __fmaf_ru(2 * EPS, C, 12 * EPS * lenMax)));
        int top                = passMask ? 1 : 0;
        if (lane == 0)
        {
            const int c0 = __float_as_int(prep.nrec[3 * size_t(rootNode)].w);
            w.stack[0]   = c0 > 0 ? c0 : -(2 * rootNode + (c0 < 0 ? 1 : 0)) - 1;
        }
        __syncwarp();
        uint32_t curBase = 0, curEnd = 0; // the run being read
        bool runOut = false;              // it holds particles outside their leaf's box
        unsigned rem = 0, outM = 0;       // runs of the leaves taken last that are not yet read (bit: first leaf's lane)
        int nl       = 0;
        uint32_t lf = 0, le = 0; // this lane's leaf
        int lnode         = 0;
        unsigned needMask = 0;         // target by target: the lanes whose spheres may reach the leaf
        int expanded      = 0;         // entries taken by the steps of this pass
        int qn = 0, qoff = 0;          // queued candidates, and the half of the queue that holds the first of them
        uint32_t qabs = 0;             // candidates queued before the current tile
        int outPend = 0, selfPend = 0; // tiles that may hold outside candidates / the warp's own particles
        int nDefer    = 0;             // tiles whose hits are not yet written
        unsigned held = 0;             // this lane's hits in them,
        unsigned tileOf = 0;          // the masks that hold them
        int words       = 0;
        for (;;)
        {
            // ---- candidates, until a tile is full (target by target: one round) ----
            bool end = false;
            do
            {
                while (curBase >= curEnd)
                {
                    while (rem == 0 && top > 0)
                    {
                        const int n          = min(top, 32);
                        const int cod        = w.stack[top - 1 - min(lane, n - 1)];
                        const unsigned inner = __ballot_sync(ALL, cod > 0 || lane >= n);
                        nl                   = __popc((inner - 1u) & ~inner); // leaves on top: the zeros below
                        if (nl > 0)
                        {
                            const bool leaf = lane < nl;
                            lnode           = leaf ? ~cod >> 1 : 0;
                            const float4* r = prep.nrec + 3 * size_t(lnode);
                            lf              = __float_as_uint(r[1].w);
                            le              = __float_as_uint(r[2].w);
                            const uint32_t prev = __shfl_up_sync(ALL, le, 1);
                            rem  = __ballot_sync(ALL, leaf && (lane == 0 || lf != prev || !mma));
                            outM = __ballot_sync(ALL, leaf && (~cod & 1));
                            top -= nl;
                            if constexpr (Stats) stLeaves += nl;
                        }
                        if constexpr (Stats) stSteps++;
                        const int wnd = min(n - nl, top > NT_WIDE ? 1 : 4);
                        if (wnd > 0)
                        {
                            const int c      = __shfl_sync(ALL, cod, (nl + (lane >> 3)) & 31);
                            const bool in    = (lane >> 3) < wnd;
                            const int child  = in && c > 0 ? c + (lane & 7) : 0;
                            const float4* r  = prep.nrec + 3 * size_t(child);
                            const float4 rA = r[0], rC = r[2];
                            float cl[3], ch[3];
                            {
                                const float cc[3] = {rA.x, rA.y, rA.z}, sz[3] = {rC.x, rC.y, rC.z};
#pragma unroll
                                for (int k = 0; k < 3; ++k)
                                {
                                    // the box widened by its own roundings, the targets' and the centre's low part
                                    const float q = foldF(__fsub_rn(cc[k], P[k]), k);
                                    const float s = sz[k] + fmaf(8 * EPS, fabsf(q) + sz[k], nodeMargin);
                                    cl[k]         = Fold ? q : q - s;
                                    ch[k]         = Fold ? s : q + s;
                                }
                            }
                            bool hit  = false;
                            auto test = [&](const float4& lo, const float4& hi) {
                                if constexpr (Fold)
                                {
                                    // the image nearest to the targets' box, which is not always the one nearest to P
                                    const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
                                    float n2 = 0.f;
#pragma unroll
                                    for (int k = 0; k < 3; ++k)
                                    {
                                        float d = fabsf(cl[k] - 0.5f * (l[k] + h[k]));
                                        if (len[k] > 0.f) d = fminf(d, fabsf(len[k] - d));
                                        d  = fmaxf(d - ch[k] - 0.5f * (h[k] - l[k]), 0.f);
                                        n2 = fmaf(d, d, n2);
                                    }
                                    hit = hit || n2 <= lo.w;
                                    return;
                                }
                                const float dx = fmaxf(fmaxf(lo.x - ch[0], cl[0] - hi.x), 0.f);
                                const float dy = fmaxf(fmaxf(lo.y - ch[1], cl[1] - hi.y), 0.f);
                                const float dz = fmaxf(fmaxf(lo.z - ch[2], cl[2] - hi.z), 0.f);
                                hit            = hit || fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= lo.w;
                            };
                            if (loose)
                            {
#pragma unroll 4
                                for (int g = 0; g < 32; ++g)
                                    test(w.tgt[g], w.tgt[g]);
                            }
                            else
                            {
#pragma unroll
                                for (int g = 0; g < 4; ++g)
                                    test(w.boxLo[g], w.boxHi[g]);
                            }
                            // a leaf stays as it is
                            hit              = in && (c > 0 ? hit : (lane & 7) == 0);
                            const int c0     = __float_as_int(rA.w);
                            const int ccod   = c > 0 ? (c0 > 0 ? c0 : ~(2 * child - c0)) : c; // c0 of a leaf: 0 or -1
                            const unsigned m = __ballot_sync(ALL, hit);
                            if constexpr (Stats) stNodes += in && c > 0 && (lane & 7) == 0;
                            expanded += wnd;
                            loose = loose || expanded > NT_LOOSE_AFTER;
                            top -= wnd;
                            if (top + __popc(m) > NT_STACK)
                            {
                                if (lane == 0 && a.errWord) atomicOr(a.errWord, 4u);
                                top = 0;
                                break;
                            }
                            __syncwarp();
                            // the lowest survivor on top
                            if (hit) w.stack[top + __popc((m >> lane) >> 1)] = ccod;
                            top += __popc(m);
                            __syncwarp();
                        }
                    }
                    end = rem == 0;
                    if (end) break;
                    const int s = __ffs(rem) - 1;
                    rem &= rem - 1;
                    const int e = mma ? (rem ? __ffs(rem) - 2 : nl - 1) : s;
                    curBase     = __shfl_sync(ALL, lf, s);
                    curEnd      = __shfl_sync(ALL, le, e);
                    runOut      = ((outM >> s) & ((2u << (e - s)) - 1u)) != 0u;
                    if (!mma)
                    {
                        // the targets whose search sphere may reach the leaf
                        const float4* r = prep.nrec + 3 * size_t(__shfl_sync(ALL, lnode, s));
                        const float4 rA = r[0], rC = r[2], tg = w.tgt[lane];
                        const float cc[3] = {rA.x, rA.y, rA.z}, sz[3] = {rC.x, rC.y, rC.z}, bb[3] = {tg.x, tg.y, tg.z};
                        float n2 = 0.f;
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                        {
                            const float q = foldF(__fsub_rn(cc[k], P[k]), k);
                            const float u = sz[k] + fmaf(8 * EPS, fabsf(q) + sz[k], nodeMargin);
                            const float d = fmaxf(fabsf(foldF(q - bb[k], k)) - u, 0.f);
                            n2            = fmaf(d, d, n2);
                        }
                        needMask = __ballot_sync(ALL, n2 <= tg.w);
                        if (needMask == 0u) curBase = curEnd;
                    }
                    if constexpr (Stats) stCand += curEnd - curBase;
                }
                if (end || !mma) break;
                do
                {
                    const uint32_t j = curBase + lane;
                    float ax, ay, az;
                    frame(min(j, curEnd - 1u), ax, ay, az);
                    bool keep       = false;
                    const float2 x2 = make_float2(ax, ax), y2 = make_float2(ay, ay), z2 = make_float2(az, az);
#pragma unroll
                    for (int p = 0; p < 2; ++p)
                    {
                        const float4 s0 = w.sph[2 * p], s1 = w.sph[2 * p + 1];
                        const float2 dx = __fadd2_rn(x2, make_float2(s0.x, s0.y));
                        const float2 dy = __fadd2_rn(y2, make_float2(s0.z, s0.w));
                        const float2 dz = __fadd2_rn(z2, make_float2(s1.x, s1.y));
                        const float2 e  = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                        keep            = keep || e.x <= s1.z || e.y <= s1.w;
                    }
                    keep             = keep && j < curEnd;
                    const unsigned m = __ballot_sync(ALL, keep);
                    const int pos    = qn + __popc(m & ltMask);
                    if (keep) w.queue[(qoff + pos) & 63] = make_float4(ax, ay, az, __uint_as_float(j));
                    // uniform: the run meets the warp's own particles (a round before or after them is harmless)
                    if (curBase - uint32_t(base0) + 31u < 63u)
                    {
                        const uint32_t rel = j - uint32_t(base0);
                        if (keep && rel < 32u) w.self[rel] = qabs + uint32_t(pos);
                        selfPend = 2;
                    }
                    if (runOut && __any_sync(ALL, keep && (prep.pnode[j] >> 31))) outPend = 2;
                    qn += __popc(m);
                    curBase += 32;
                    if constexpr (Stats) stKept += __popc(m), stRounds++;
                } while (curBase < curEnd && qn < 32);
            } while (qn < 32);
            const bool done = end && qn == 0;
            if (!done)
            {
                unsigned inM = 0, ambM = 0; // bit 31 - k: candidate k is a neighbour / is not decided
                uint32_t jv;                // this lane's candidate of the tile
                int cnt;
                uint32_t selfAt; // candidate 0 of the tile, in the numbering of w.self (mma) or of the particles
                if (mma)
                {
                    // ---- one tile: up to 32 queued candidates against the 32 targets ----
                    __syncwarp();
                    cnt            = min(qn, 32);
                    const float4 q = w.queue[qoff + lane];
                    jv             = __float_as_uint(q.w);
                    const float x = q.x * sc, y = q.y * sc, z = q.z * sc;
                    uint4 rec     = make_uint4(splitHalf(x), splitHalf(y), splitHalf(z),
                                               splitHalf(fmaf(z, z, fmaf(y, y, x * x))));
                    // beyond the queue's end (the last tile): |a|^2 = 57344, no neighbour
                    if (lane >= cnt) rec = make_uint4(0u, 0u, 0u, 0x00007b00u);
                    __syncwarp();
                    // slot 8 s + 2 n + c is column 2 s + c of column block n: the mask bits of lane s of a quad are
                    // then the candidates 8 s .. 8 s + 7 in order
                    reinterpret_cast<uint4*>(w.queue)[qoff + (((lane & 6) << 2) | ((lane >> 2) & 6) | (lane & 1))] = rec;
                    w.tileJ[nDefer][31 - lane] = jv;
                    __syncwarp();
                    const uint32_t* bw   = reinterpret_cast<const uint32_t*>(w.queue) + 4 * qoff + lane;
                    const uint32_t b0[4]  = {bw[0], bw[32], bw[64], bw[96]};
                    const bool last       = (lane & 3) == 3; // its upper k: (1, 1) for |b|^2 - Tin + E
                    const uint32_t b1[4]  = {last ? 0x3c003c00u : b0[0], last ? 0x3c003c00u : b0[1],
                                             last ? 0x3c003c00u : b0[2], last ? 0x3c003c00u : b0[3]};
                    uint32_t part[2] = {}, lowest = ALL;
#pragma unroll
                    for (int m = 0; m < 2; ++m)
                    {
                        float d[4][4];
#pragma unroll
                        for (int n = 0; n < 4; ++n)
                            tileMma(d[n], aLo[2 * m], aLo[2 * m + 1], aHi[2 * m], aHi[2 * m + 1], b0[n], b1[n]);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int n = 0; n < 4; ++n)
                            {
                                const uint32_t u = __float_as_uint(d[n][2 * h]), v = __float_as_uint(d[n][2 * h + 1]);
                                part[m] = __funnelshift_l(u, part[m], 1);
                                part[m] = __funnelshift_l(v, part[m], 1);
                                lowest  = min(min(lowest, u), v);
                            }
                    }
                    inM = quadTranspose(__byte_perm(part[0], part[1], 0x1054), lane);
                    // as unsigned integers the values in [0, W) are exactly those below W's bits (a tile in ten has
                    // one: the products are formed again there rather than kept)
                    if (__any_sync(ALL, lowest < wBits))
                    {
                        uint32_t mAmb = 0;
#pragma unroll
                        for (int m = 0; m < 2; ++m)
#pragma unroll
                            for (int n = 0; n < 4; ++n)
                            {
                                float d[4];
                                tileMma(d, aLo[2 * m], aLo[2 * m + 1], aHi[2 * m], aHi[2 * m + 1], b0[n], b1[n]);
#pragma unroll
                                for (int c = 0; c < 4; ++c)
                                    if (__float_as_uint(d[c]) < wBits)
                                        mAmb |= 1u << (31 - (16 * m + 8 * (c >> 1) + 2 * n + (c & 1)));
                            }
                        ambM = quadTranspose(mAmb, lane);
                    }
                    if (!inPass) inM = ambM = 0;
                    qn -= cnt;
                    qoff ^= 32;
                    selfAt = qabs;
                    qabs += 32;
                    if constexpr (Stats) stTiles++;
                }
                else
                {
                    // lanes hold the candidates, the warp loops over the targets that need the leaf
                    jv = curBase + lane;
                    float ax, ay, az;
                    frame(min(jv, curEnd - 1u), ax, ay, az);
                    if (jv >= curEnd) ax = INF;
                    cnt    = int(min(32u, curEnd - curBase));
                    selfAt = curBase;
                    for (unsigned mm = needMask; mm; mm &= mm - 1)
                    {
                        const int L     = __ffs(mm) - 1;
                        const float4 tg = w.tgt[L];
                        const float2 th = *reinterpret_cast<const float2*>(&w.thr[L]);
                        const float dx = ax - tg.x, dy = ay - tg.y, dz = az - tg.z;
                        const float e     = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                        const unsigned mi = __ballot_sync(ALL, e < th.x);
                        const unsigned ma = __ballot_sync(ALL, e < th.y);
                        if (lane == L)
                        {
                            inM  = __brev(mi);
                            ambM = __brev(ma & ~mi);
                        }
                    }
                    __syncwarp();
                    w.tileJ[nDefer][31 - lane] = jv;
                    __syncwarp();
                    selfPend = outPend = 1;
                    curBase += 32;
                    if constexpr (Stats) stRounds++, stDirect++;
                }

                // ---- exceptions ----
                if (selfPend)
                {
                    const uint32_t k = (mma ? w.self[tau] : i) - selfAt;
                    if (k < 32u)
                    {
                        inM &= ~(0x80000000u >> k);
                        ambM &= ~(0x80000000u >> k);
                    }
                    --selfPend;
                }
                if (outPend)
                {
                    --outPend;
                    // candidates outside their leaf's box have no path-safe shortcut of their own: a neighbour iff
                    // within r and this target's path to the leaf passes the reference's cell tests, walked exactly
                    // if need be. Leaf by leaf: with coarse keys most particles of a leaf can be outside
                    const uint32_t pn = lane < cnt ? prep.pnode[jv] : 0u;
                    for (unsigned ob = __ballot_sync(ALL, (pn >> 31) != 0u); ob;)
                    {
                        const uint32_t code = __shfl_sync(ALL, pn, __ffs(ob) - 1);
                        const unsigned mine = __ballot_sync(ALL, pn == code);
                        ob &= ~mine;
                        const unsigned bits = __brev(mine);
                        unsigned f          = (inM | ambM) & bits;
                        if (f == 0u) continue;
                        const int node = int(code & 0x7fffffffu);
                        if (pathSafe(node) || path(node))
                        {
                            // (one outside the periodic box is not where it is folded to)
                            f = (Fold && !pbc ? inM | ambM : ambM) & bits;
                            inM &= ~f;
                            while (f)
                            {
                                const int k = __clz(f);
                                f ^= 0x80000000u >> k;
                                if (within(w.tileJ[nDefer][31 - k])) inM |= 0x80000000u >> k;
                            }
                        }
                        else { inM &= ~bits; }
                        ambM &= ~bits;
                    }
                }
                while (ambM)
                {
                    const int k = __clz(ambM);
                    ambM ^= 0x80000000u >> k;
                    const uint32_t j = w.tileJ[nDefer][31 - k];
                    float ax, ay, az;
                    frame(j, ax, ay, az);
                    const float4 tg = w.tgt[lane], th = w.thr[lane];
                    const float dx = ax - tg.x, dy = ay - tg.y, dz = az - tg.z;
                    const float e  = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    bool in        = e < th.x;
                    if (!in && e < th.y)
                    {
                        if constexpr (Stats) stExact++;
                        const int node = int(prep.pnode[j] & 0x7fffffffu);
                        if (pathSafe(node)) in = within(j);
                        else if constexpr (Fold) in = within(j) && path(node);
                        else
                            in = slowPairAt<T>(tref, kappa, th.z, j, node, a.parents, a.centers, a.sizes, true, rootNode);
                    }
                    if constexpr (Stats) stAmb++;
                    if (in) inM |= 0x80000000u >> k;
                }
                // the lane's masks that are not empty, one below the other, and the tile of each (4 bits)
                if (inM)
                {
                    w.mask[words][lane] = inM;
                    tileOf |= unsigned(nDefer) << (4 * words);
                    ++words;
                }
                held += __popc(inM);
                ++nDefer;
            }

            // ---- the hits of up to NT_DEFER tiles, each lane its own in ascending order. In a single tile the hits of
            // a target cluster (its candidates are neighbours along the curve: a lane has 5 of 32 on average, the
            // busiest one 20), over several tiles they balance ----
            if (nDefer == NT_DEFER || done)
            {
                int left    = nc < ngmax ? int(min(held, ngmax - nc)) : 0; // the count is not capped
                uint32_t* p = myNb + nc;
                nc += held;
                const uint32_t* mt = &w.mask[0][lane];
                const uint32_t* jt = w.tileJ[tileOf & 15u];
                uint32_t m         = *mt;
                // selects instead of a branch (some lane ends a word in nearly every round), the next word read ahead
                uint32_t nx = mt[32];
                while (left > 0)
                {
                    const int k = 31 - __clz(m);
                    *p          = jt[k];
                    m ^= 1u << k;
                    const bool z = m == 0u;
                    mt += z ? 32 : 0;
                    m = z ? nx : m;
                    tileOf >>= z ? 4 : 0;
                    jt = w.tileJ[tileOf & 15u];
                    nx = mt[32];
                    ++p;
                    --left;
                }
                held = tileOf = 0;
                words         = 0;
                nDefer = 0;
                __syncwarp();
                if (done) break;
            }
        }
        if (!a.numSets || passSet >= lastSet) break;
    }
    if (active) a.nc[i - a.first] = nc;
    if constexpr (Stats)
    {
        // [2] FP32 re-tests, [3] exact decisions (per lane); [4] leaves, [5] candidates read, [6] node expansions, [7]
        // warps, [8] candidates kept, [9] tiles, [10] rounds, [11] rounds tested target by target, [12] steps (per warp)
        unsigned long long v[3] = {stAmb, stExact, stNodes};
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            for (int o = 16; o > 0; o >>= 1)
                v[k] += __shfl_xor_sync(ALL, v[k], o);
        }
        if (lane == 0)
        {
            const unsigned long long s[11] = {v[0], v[1], stLeaves, stCand, v[2], 1ull, stKept, stTiles, stRounds, stDirect, stSteps};
            for (int k = 0; k < 11; ++k)
                atomicAdd(a.stats + 2 + k, s[k]);
        }
    }
}
