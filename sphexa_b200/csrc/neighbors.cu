// Neighbour search on sm_100a: one warp per target group of 32 consecutive (SFC-ordered) particles.
//
// Per group: (1) the search box = union over the group's still-active particles of [x - 2h, x + 2h];
// (2) a depth-first traversal of the focus octree in child (= SFC) order, warp-cooperative with 8 lanes testing the
// 8 children of a node against the box (periodic axes use the minimum image), collecting overlapping leaves in
// ascending order in shared memory; (3) each buffered leaf is cut into the 8-particle SFC blocks it covers, every
// block's bounding box (precomputed once per step) is tested against the search box 32 blocks at a time, and the
// particles of surviving blocks are streamed 32 at a time through shared memory; (4) every lane tests the staged
// candidates against its own particle, two candidates per packed FP32x2 instruction on coordinates relative to the
// group centre, and runs the exact FP64 test of the reference (cstone/findneighbors.hpp:33-51,77-147: squared
// minimum-image distance < (2h)^2, j != i) only for candidates within a narrow band around the radius.
// Candidates arrive in ascending particle order, so each list equals the reference CPU list, which is also ascending
// (depth-first octree traversal over SFC-ordered leaves), including which neighbours are kept when more than ngmax
// qualify. The smoothing-length iteration of sph/include/sph/find_neighbors.hpp:10-41 is fused: lanes whose count
// left [ng0/4, ngmax+1] update h and search again, at most maxIterations times; settled lanes keep their lists.
#include <algorithm>

#include "neighbors.cuh"
#include "primitives.cuh"

namespace sphb
{

namespace
{

constexpr int kNbWarps   = 4;
constexpr int kNbThreads = kNbWarps * kWarp;
constexpr int kStackWide = 44;  // entries up to which the traversal takes four of them at a time
constexpr int kStackCap  = 220; // kStackWide + 28, and 7 per level for those taken one at a time
constexpr int kLeafCap   = 256; // candidate leaves buffered before they are streamed

/*! Lanes that share a target. One lane per target tests and appends for its own particle, 32 targets per warp. A group's
 *  traversal, staging and tests run one after another, so a launch of few groups takes as long as its slowest one, with
 *  most of the GPU idle. With four (eight) lanes per target a warp serves eight (four) targets: each lane tests and
 *  appends its part of the staged candidates, and the smaller search box admits fewer of them. But each box is traversed
 *  and staged by itself, so a launch that fills the GPU is slower with it: hence the limits below.
 *  Neighbour phase, us. Whole searches with four and eight lanes: 16^3 particles 64 and 49, 36^3 (a sphere of them)
 *  99 and 108, 30^3 FP64 103 and 117; with one and four, before the traversal took four nodes a round: 30^3 167 and 122,
 *  50^3 327 and 426, 63^3 394 and 579.
 *  Searches of listed groups, a small part of all, choose by the length of the list, which only the device knows. Neighbour
 *  phase with one lane, with eight, and with eight for lists of up to 1,500 groups (1,350 to 1,700 do the same): block
 *  time steps of 64^3 334, 248 and 248, 81^3 414, 300 and 301, 90^3 378, 496 and 388, 100^3 468, 609 and 476, 100^3 with a
 *  wide blast 757, 1480 and 760, global steps of 128^3 934, 1193 and 935. */
constexpr int kFewLanes             = 4;
constexpr int kManyLanes            = 8;
constexpr size_t kManyLanesAll      = 10000;
constexpr size_t kFewLanesAll       = 40000;
constexpr size_t kManyLanesListed   = 1500; // groups of the list

template<int kPer, bool kSkin>
struct NbShared
{
    //! list entries a target buffers: the chunk being filled and up to 8 more neighbours (kPer 1) or 32
    static constexpr int kRing = (kPer == 1 ? 2 : 5) * kNbChunk;
    int stack[kNbWarps][kStackCap];
    int leafFirst[kNbWarps][kLeafCap]; // the buffered leaves, then the first particle of each
    int leafEnd[kNbWarps][kLeafCap];   // one past its last particle
    int blkPre[kNbWarps][kLeafCap + 1]; // exclusive prefix of the number of blocks per buffered leaf
    int pStart[kNbWarps][kWarp];       // surviving pieces (block and leaf intersections) of one round
    int pPre[kNbWarps][kWarp + 1];     // exclusive prefix of their lengths
    uint8_t pieceOf[kNbWarps][kWarp * kBlockSize]; // candidate of the round -> its piece
    // staged candidates: position relative to the group centre (FP32, pairs loaded as float2) and index
    alignas(16) float cx[kNbWarps][kWarp];
    alignas(16) float cy[kNbWarps][kWarp];
    alignas(16) float cz[kNbWarps][kWarp];
    int cj[kNbWarps][kWarp];
    // per target: the neighbours of the list chunks being filled, written out as 32-byte sectors when full; target minor,
    // so that the appends of a warp fall into distinct banks
    uint32_t nbuf[kNbWarps][kRing * kWarp / kPer];
    uint16_t dbuf[kNbWarps][kSkin ? kRing * kWarp / kPer : 1]; // skin rows: the quantised build distance of each entry
};

/*! Half width of the band |d^2 - (2h)^2| < band * (2h)^2 in which the FP32 distance cannot decide and the exact FP64
 *  test runs. Relative coordinates are formed in FP64 and rounded once to FP32, so each has an error of at most
 *  2^-24 S, S = the largest distance from the group centre at which a neighbour of the group can lie. For a pair at
 *  distance ~2h that bounds the FP32 squared-distance error by about 2^-21 (S / 2h + 1) (2h)^2 including the FP32
 *  arithmetic; the band is four times that. */
__device__ inline float bandOf(float S, float twoH) { return 2.0e-6f * (S / twoH + 1.0f); }

__device__ inline double warpMin(double v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
    {
        v = fmin(v, __shfl_xor_sync(0xffffffffu, v, off));
    }
    return v;
}

__device__ inline double warpMax(double v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
    {
        v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
    }
    return v;
}

//! warp-wide exclusive prefix of one value per lane; *total receives the sum
__device__ inline int warpExclusive(int v, int lane, int* total)
{
    int incl = v;
#pragma unroll
    for (int off = 1; off < kWarp; off <<= 1)
    {
        int t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) { incl += t; }
    }
    *total = __shfl_sync(0xffffffffu, incl, kWarp - 1);
    return incl - v;
}

//! largest r in [0, n) with pre[r] <= t (pre ascending, pre[0] = 0 <= t)
__device__ inline int findSlot(const int* pre, int n, int t)
{
    int lo = 0, hi = n;
    while (hi - lo > 1)
    {
        int mid = (lo + hi) >> 1;
        if (pre[mid] <= t) { lo = mid; }
        else { hi = mid; }
    }
    return lo;
}

//! 32-byte read-only load of a packed position (two 16-byte loads of one sector)
__device__ inline double4 ldPos(const double4* p)
{
    const double2* q = reinterpret_cast<const double2*>(p);
    double2 lo = __ldg(q), hi = __ldg(q + 1);
    return make_double4(lo.x, lo.y, hi.x, hi.y);
}

//! what one launch of the search computes
enum SearchKind : int
{
    kSearchAll,    // neighbour lists of every group, with the smoothing-length iteration
    kSearchListed, // the same for the groups of a device-side list
    kSearchSkin    // skin lists: every j within 2 h (1 + skin), no iteration, h read only
};

//! launch inputs of the listed and skin searches
struct SearchExtras
{
    const unsigned* groups;
    const unsigned* numListed;
    SkinLists sl;
    double onePlusSkin;
    const unsigned* gate; // if set: the launch runs only when bit *gate of gateMask is set (a device-side mode)
    unsigned gateMask;
};

/*! Blocks that stay resident on an SM: eight by their registers, fewer where the buffers do not fit into its shared memory
 *  (228 KB, 1 KB of it per block for the system). Row builds with one lane per target keep seven. The other kinds keep
 *  eight: a stack of 256 entries instead of 220 left them seven (neighbour phase of 101^3 FP64 1064 us, now 1029, of Noh
 *  81^3 498, now 482, of 128^3 with a wide blast 2272, now 2191). */
template<int kPer, bool kSkin>
constexpr int residentBlocks()
{
    constexpr int fit = int(228 * 1024 / (sizeof(NbShared<kPer, kSkin>) + 1024));
    return fit < 8 ? fit : 8;
}
static_assert(residentBlocks<1, false>() == 8 && residentBlocks<kFewLanes, true>() == 8, "the launches count on eight");

/*! One warp's unit of the search: kWarp / kPer targets of a group of 32 (unit = kPer group + part; of a listed search,
 *  group is the place in the list). */
template<bool kBatched, int kKind, int kPer>
__device__ __forceinline__ void searchUnit(NbShared<kPer, kKind == kSearchSkin>& sh, size_t unit,
                                           const double* __restrict__ x, const double* __restrict__ y,
                                           const double* __restrict__ z, const double4* __restrict__ pos, double* h,
                                           size_t n, const TreeView& tree, const DevBox& box, const NeighborParams& prm,
                                           uint32_t* __restrict__ nidx, unsigned* __restrict__ ncOut, unsigned* status,
                                           const TreeView* __restrict__ views, const uint8_t* __restrict__ inst,
                                           const SearchExtras& ex)
{
    constexpr int kTargets = kWarp / kPer; // targets of a warp
    const int warp         = threadIdx.x / kWarp;
    const int lane         = threadIdx.x & (kWarp - 1);
    const int piece        = lane % kPer; // which of the lanes that share the target
    const size_t numGroups = (n + kWarp - 1) / kWarp;
    size_t group = unit / kPer;
    if constexpr (kKind == kSearchListed) { group = ex.groups[group]; }
    if (group >= numGroups) { return; }
    const unsigned slot = unsigned(unit % kPer) * kTargets + lane / kPer; // the target's place in its group
    constexpr bool kSkin = kKind == kSearchSkin;
    // the lists written: neighbour lists (ngmax entries) or skin rows (cap entries)
    uint32_t* const outList  = kSkin ? ex.sl.rows : nidx;
    const unsigned listCap   = kSkin ? ex.sl.cap : prm.ngmax;

    const size_t i = group * kWarp + slot;
    // an ensemble: the group's instance (its first slot is never padding) selects the tree; padding slots idle
    TreeView tv = tree;
    if constexpr (kBatched) { tv = views[inst[group * kWarp]]; }
    const bool valid = i < n && !(kBatched && inst[i] == kGhost);
    const double xi  = valid ? x[i] : 0.0;
    const double yi  = valid ? y[i] : 0.0;
    const double zi  = valid ? z[i] : 0.0;
    double hi        = valid ? h[i] : 0.0;

    const unsigned ngmin = prm.ng0 / 4;
    const unsigned ngPad = kSkin ? ex.sl.cap : paddedNgmax(prm.ngmax);
    bool active          = valid;
    int updates          = 0;
    unsigned count       = 0;
    bool overflow        = false;

    int* stack     = sh.stack[warp];
    int* leafFirst = sh.leafFirst[warp];
    int* leafEnd   = sh.leafEnd[warp];
    int* blkPre    = sh.blkPre[warp];
    int* pStart    = sh.pStart[warp];
    int* pPre      = sh.pPre[warp];

    while (__ballot_sync(0xffffffffu, active) != 0u && !overflow)
    {
        const double r        = kSkin ? __dmul_rn(2.0 * hi, ex.onePlusSkin) : 2.0 * hi;
        // the exact test: (2h)^2 as the reference computes it, or R^2 for skin rows
        const double radiusSq = kSkin ? __dmul_rn(r, r) : searchRadiusSq(hi);
        double blo[3], bhi[3];
        blo[0] = warpMin(active ? xi - r : INFINITY);
        blo[1] = warpMin(active ? yi - r : INFINITY);
        blo[2] = warpMin(active ? zi - r : INFINITY);
        bhi[0] = warpMax(active ? xi + r : -INFINITY);
        bhi[1] = warpMax(active ? yi + r : -INFINITY);
        bhi[2] = warpMax(active ? zi + r : -INFINITY);
        double gc[3], gs[3];
        float gcb[3], gsb[3], lenf[3], ilenf[3]; // group box in the block-box frame (relative to the box corner)
        for (int k = 0; k < 3; ++k)
        {
            gc[k]    = 0.5 * (blo[k] + bhi[k]);
            gs[k]    = 0.5 * (bhi[k] - blo[k]) * (1.0 + 1e-12) + 1e-14 * box.len[k];
            gcb[k]   = float(gc[k] - box.lo[k]);
            gsb[k]   = __double2float_ru(gs[k] + 4e-7 * box.len[k]);
            lenf[k]  = float(box.len[k]);
            ilenf[k] = float(box.ilen[k]);
        }
        // this particle relative to the group centre in FP32, and the FP32 acceptance band
        const float rix  = float(minImage(xi - gc[0], box.len[0], box.ilen[0], box.periodic[0]));
        const float riy  = float(minImage(yi - gc[1], box.len[1], box.ilen[1], box.periodic[1]));
        const float riz  = float(minImage(zi - gc[2], box.len[2], box.ilen[2], box.periodic[2]));
        const float twoH = float(r);
        const float r2f  = twoH * twoH;
        float reach      = active ? sqrtf(rix * rix + riy * riy + riz * riz) * 1.001f + twoH : 0.f;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
        {
            reach = fmaxf(reach, __shfl_xor_sync(0xffffffffu, reach, off));
        }
        // Differences of two coordinates that were each folded to the nearest image of the group centre are the
        // minimum image of the pair only while 2h + (offset from the centre) < L/2 on every periodic axis. Groups
        // whose reach exceeds that (search radii comparable to the box) test every candidate exactly instead.
        bool wrapTest = false;
        float maxSpan = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            if (box.periodic[k])
            {
                wrapTest = wrapTest || reach >= 0.5f * lenf[k];
                maxSpan  = fmaxf(maxSpan, 0.5f * lenf[k]);
            }
        }
        const float band = active ? bandOf(wrapTest ? fmaxf(reach, maxSpan) : reach, twoH) : 0.f;
        const float r2lo = r2f * (1.f - band);
        const float r2hi = r2f * (1.f + band);

        if (active) { count = 0; }
        int numLeaves = 0;

        // this target's ring of list chunks, entry e at ring[(e mod kRing) * kStride], and the store of a full chunk to the
        // chunked list layout (nidxAt)
        constexpr int kRing   = NbShared<kPer, kSkin>::kRing;
        constexpr int kStride = kTargets;
        uint32_t* ring        = &sh.nbuf[warp][lane / kPer];
        uint16_t* dring       = &sh.dbuf[warp][lane / kPer];
        // skin rows: distance -> units of R / kSkinDistUnits. The FP32 distance of the pair serves where it is known
        // to kSkinDistSlack units: both coordinates are rounded once relative to the group centre, 2^-24 reach each,
        // and the FP32 arithmetic adds at most 4 * 2^-24 R, together 2^-24 (3.5 reach + 4 R) < 1.3e-6 R = 0.084 units
        // for reach <= 5 R (a compact group reaches 2 to 3 R)
        const double qScale  = kSkinDistUnits / r;
        const float qScaleF  = float(qScale);
        const bool exactDist = wrapTest || reach > 5.f * twoH;
        auto storeChunk = [&](unsigned c) {
            uint32_t* dst         = outList + nidxAt(group, ngPad, c * kNbChunk, slot);
            const uint32_t* chunk = ring + (c * kNbChunk % kRing) * kStride;
            if constexpr (kSkin)
            {
                const uint16_t* dchunk = dring + (c * kNbChunk % kRing) * kStride;
                uint4 d;
                d.x = unsigned(dchunk[0]) | (unsigned(dchunk[kStride]) << 16);
                d.y = unsigned(dchunk[2 * kStride]) | (unsigned(dchunk[3 * kStride]) << 16);
                d.z = unsigned(dchunk[4 * kStride]) | (unsigned(dchunk[5 * kStride]) << 16);
                d.w = unsigned(dchunk[6 * kStride]) | (unsigned(dchunk[7 * kStride]) << 16);
                *reinterpret_cast<uint4*>(ex.sl.dist + nidxAt(group, ngPad, c * kNbChunk, slot)) = d;
            }
            // one 256-bit streaming store of the whole sector (the lists are next read once per J-loop)
            asm volatile("st.global.cs.v8.u32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(chunk[0]),
                         "r"(chunk[kStride]), "r"(chunk[2 * kStride]), "r"(chunk[3 * kStride]), "r"(chunk[4 * kStride]),
                         "r"(chunk[5 * kStride]), "r"(chunk[6 * kStride]), "r"(chunk[7 * kStride])
                         : "memory");
        };
        // neighbour k of the staged candidates as entry e of the list
        auto put = [&](int k, int j, unsigned e) {
            if constexpr (kSkin)
            {
                // the build distance, for the refilter's bounds
                uint16_t q16;
                if (exactDist)
                {
                    double4 pj = ldPos(pos + j);
                    double q   = rint(sqrt(exactDistSq(pj.x, pj.y, pj.z, xi, yi, zi, box)) * qScale);
                    q16        = uint16_t(fmin(q, kSkinDistUnits));
                }
                else
                {
                    float dx = sh.cx[warp][k] - rix, dy = sh.cy[warp][k] - riy, dz = sh.cz[warp][k] - riz;
                    float q  = rintf(sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx))) * qScaleF);
                    q16      = uint16_t(fminf(q, float(kSkinDistUnits)));
                }
                dring[(e % kRing) * kStride] = q16;
            }
            ring[(e % kRing) * kStride] = uint32_t(j);
        };

        // test the staged 32 candidates (this lane's part of them where lanes share a target) against the target and
        // append the neighbours in index order
        constexpr int kShare = kWarp / kPer; // candidates per lane
        auto testStaged = [&](int numReal) {
            if (!active) { return; }
            // bit k of sure: candidate first + k lies inside the sphere by its FP32 distance (below the band); of maybe:
            // it may (below the upper edge of the band)
            const int first = piece * kShare;
            unsigned maybe = 0u, sure = 0u;
            if (!wrapTest)
            {
                const float2 mx = make_float2(-rix, -rix), my = make_float2(-riy, -riy), mz = make_float2(-riz, -riz);
#pragma unroll
                for (int k = 0; k < kShare; k += 2)
                {
                    float2 X  = *reinterpret_cast<const float2*>(&sh.cx[warp][first + k]);
                    float2 Y  = *reinterpret_cast<const float2*>(&sh.cy[warp][first + k]);
                    float2 Z  = *reinterpret_cast<const float2*>(&sh.cz[warp][first + k]);
                    float2 dx = __fadd2_rn(X, mx);
                    float2 dy = __fadd2_rn(Y, my);
                    float2 dz = __fadd2_rn(Z, mz);
                    float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                    maybe |= (unsigned(d2.x < r2hi) << k) | (unsigned(d2.y < r2hi) << (k + 1));
                    sure |= (unsigned(d2.x < r2lo) << k) | (unsigned(d2.y < r2lo) << (k + 1));
                }
            }
            else
            {
                // every real candidate of the chunk goes through the exact FP64 test below, which folds the pair
                // difference itself (padding sits at the end of the last chunk)
                int real = min(max(numReal - first, 0), kShare);
                maybe    = real >= 32 ? 0xffffffffu : ((1u << real) - 1u);
            }
            // candidates too close to the search radius for FP32: the exact test of the reference (rare)
            unsigned band = maybe & ~sure;
            while (band)
            {
                int k = __ffs(band) - 1;
                band &= band - 1u;
                int j      = sh.cj[warp][first + k];
                double4 pj = ldPos(pos + j);
                if (exactDistSq(pj.x, pj.y, pj.z, xi, yi, zi, box) < radiusSq) { sure |= 1u << k; }
            }
            if constexpr (kPer == 1)
            {
                // append the neighbours in candidate (= index) order, up to eight before the chunk that filled up is
                // stored: the warp's lanes store together instead of at every append that fills a chunk (neighbour phase of
                // 101^3 FP64 1096 -> 1052 us, of 63^3 332 -> 315)
                while (sure)
                {
                    const unsigned from = count;
                    while (sure && count - from < kNbChunk)
                    {
                        int k = __ffs(sure) - 1;
                        sure &= sure - 1u;
                        int j = sh.cj[warp][k];
                        if (size_t(j) == i) { continue; }
                        if (count < listCap) { put(k, j, count); }
                        ++count;
                    }
                    const unsigned c = min(from, listCap) / kNbChunk;
                    if (min(count, listCap) / kNbChunk != c) { storeChunk(c); }
                }
            }
            else
            {
                // every lane of the target appends its own, after those of the lanes before it
                const unsigned team = ((1u << kPer) - 1u) << (lane - piece);
#pragma unroll
                for (int k = 0; k < kShare; ++k)
                {
                    if (((sure >> k) & 1u) && size_t(sh.cj[warp][first + k]) == i) { sure &= ~(1u << k); }
                }
                unsigned hits = __popc(sure), before = 0u, all = hits;
#pragma unroll
                for (int off = 1; off < kPer; off <<= 1)
                {
                    unsigned o = __shfl_xor_sync(team, all, off);
                    before += (piece & off) ? o : 0u;
                    all += o;
                }
                unsigned e = count + before;
                while (sure)
                {
                    int k = __ffs(sure) - 1;
                    sure &= sure - 1u;
                    if (e < listCap) { put(first + k, sh.cj[warp][first + k], e); }
                    ++e;
                }
                __syncwarp(team);
                // the chunks that filled up: at most five, and no entry past the list's capacity is stored
                const unsigned now = min(count + all, listCap);
                for (unsigned c = min(count, listCap) / kNbChunk + piece; c < now / kNbChunk; c += kPer)
                {
                    storeChunk(c);
                }
                __syncwarp(team);
                count += all;
            }
        };

        // stream the buffered candidate leaves, pruned to the 8-particle blocks that meet the search box
        auto flush = [&]() {
            int local[kLeafCap / kWarp];
            int sum = 0;
#pragma unroll
            for (int q = 0; q < kLeafCap / kWarp; ++q)
            {
                int t   = lane * (kLeafCap / kWarp) + q;
                int nbk = 0;
                if (t < numLeaves)
                {
                    int leaf = leafFirst[t];
                    int b    = tv.layout[leaf];
                    int e    = tv.layout[leaf + 1];
                    leafFirst[t] = b;
                    leafEnd[t]   = e;
                    nbk   = e > b ? (e - 1) / kBlockSize - b / kBlockSize + 1 : 0;
                }
                local[q] = nbk;
                sum += nbk;
            }
            int totalBlocks;
            int run = warpExclusive(sum, lane, &totalBlocks);
#pragma unroll
            for (int q = 0; q < kLeafCap / kWarp; ++q)
            {
                int t = lane * (kLeafCap / kWarp) + q;
                if (t < numLeaves) { blkPre[t] = run; }
                run += local[q];
            }
            __syncwarp();

            for (int base = 0; base < totalBlocks; base += kWarp)
            {
                int t     = base + lane;
                bool keep = false;
                int ps = 0, plen = 0;
                if (t < totalBlocks)
                {
                    int rr = findSlot(blkPre, numLeaves, t);
                    int b = leafFirst[rr], e = leafEnd[rr];
                    int c = b / kBlockSize + (t - blkPre[rr]);
                    ps    = max(c * kBlockSize, b);
                    plen  = min(c * kBlockSize + kBlockSize, e) - ps;
                    float4 lo = __ldg(tv.blockLo + c);
                    float4 hb = __ldg(tv.blockHi + c);
                    float bl[3] = {lo.x, lo.y, lo.z};
                    float bh[3] = {hb.x, hb.y, hb.z};
                    keep = plen > 0;
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                    {
                        float d = 0.5f * (bl[k] + bh[k]) - gcb[k];
                        if (box.periodic[k]) { d -= lenf[k] * rintf(d * ilenf[k]); }
                        keep = keep && fabsf(d) <= gsb[k] + 0.5f * (bh[k] - bl[k]) + 1e-6f * lenf[k];
                    }
                }
                unsigned m = __ballot_sync(0xffffffffu, keep);
                int totalCand;
                int before = warpExclusive(keep ? plen : 0, lane, &totalCand);
                if (keep)
                {
                    int pos     = __popc(m & ((1u << lane) - 1u));
                    pStart[pos] = ps;
                    pPre[pos]   = before;
                    for (int q = 0; q < plen; ++q)
                    {
                        sh.pieceOf[warp][before + q] = uint8_t(pos);
                    }
                }
                __syncwarp();
                for (int cbase = 0; cbase < totalCand; cbase += kWarp)
                {
                    int tc = cbase + lane;
                    if (tc < totalCand)
                    {
                        int rr = sh.pieceOf[warp][tc];
                        int j  = pStart[rr] + (tc - pPre[rr]);
                        if (j < 0 || size_t(j) >= n)
                        {
                            // a layout that points outside the particle arrays: report, stage a far-away point
                            atomicOr(status, 2u);
                            sh.cx[warp][lane] = INFINITY;
                            sh.cy[warp][lane] = INFINITY;
                            sh.cz[warp][lane] = INFINITY;
                            sh.cj[warp][lane] = -1;
                        }
                        else
                        {
                            sh.cx[warp][lane] =
                                float(minImage(x[j] - gc[0], box.len[0], box.ilen[0], box.periodic[0]));
                            sh.cy[warp][lane] =
                                float(minImage(y[j] - gc[1], box.len[1], box.ilen[1], box.periodic[1]));
                            sh.cz[warp][lane] =
                                float(minImage(z[j] - gc[2], box.len[2], box.ilen[2], box.periodic[2]));
                            sh.cj[warp][lane] = j;
                        }
                    }
                    else
                    {
                        // pad with points that no sphere reaches, so the test is branch-free
                        sh.cx[warp][lane] = INFINITY;
                        sh.cy[warp][lane] = INFINITY;
                        sh.cz[warp][lane] = INFINITY;
                        sh.cj[warp][lane] = -1;
                    }
                    __syncwarp();
                    testStaged(totalCand - cbase);
                    __syncwarp();
                }
            }
            numLeaves = 0;
        };

        // Depth-first traversal in SFC order, the lowest key on top of the stack: an entry is the first child of an internal
        // node or the complement of a leaf. Every round takes the top four entries, tests the children of the internal ones,
        // one per lane, and buffers the leaves that come before the first internal node; the rest goes back in order. With a node
        // a round, tested by eight lanes and its leaves looked up by one, the search of 81^3 Noh particles took 716 us, now 525.
        const int rootChild = tv.childOffsets[0];
        int sp              = 1;
        if (lane == 0) { stack[0] = rootChild ? rootChild : ~tv.nodeToLeaf[0]; }
        __syncwarp();
        while (sp > 0)
        {
            const int take = sp > kStackWide ? 1 : min(sp, kWarp / 8);
            int entry      = 0;
            bool ov        = false;
            if (lane / 8 < take)
            {
                entry = stack[sp - 1 - lane / 8];
                ov    = lane % 8 == 0;
                if (entry > 0)
                {
                    int c     = entry + lane % 8;
                    int child = tv.childOffsets[c];
                    int leaf  = tv.nodeToLeaf[c];
                    ov        = true;
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                    {
                        double d = tv.centers[3 * c + k] - gc[k];
                        if (box.periodic[k]) { d -= box.len[k] * rint(d * box.ilen[k]); }
                        ov = ov && fabs(d) <= gs[k] + tv.sizes[3 * c + k] * (1.0 + 1e-12) + tv.ext;
                    }
                    entry = child ? child : ~leaf;
                }
            }
            __syncwarp();
            sp -= take;
            unsigned found    = __ballot_sync(0xffffffffu, ov);
            unsigned internal = __ballot_sync(0xffffffffu, ov && entry > 0);
            unsigned ready    = internal ? found & ((internal & (0u - internal)) - 1u) : found;
            int numReady      = __popc(ready);
            if (numLeaves + numReady > kLeafCap) { flush(); }
            if ((ready >> lane) & 1u) { leafFirst[numLeaves + __popc(ready & ((1u << lane) - 1u))] = ~entry; }
            numLeaves += numReady;
            unsigned later = found & ~ready;
            int pushes     = __popc(later);
            if (sp + pushes > kStackCap)
            {
                overflow = true;
                break;
            }
            // in reverse, so that the lowest key is on top
            if ((later >> lane) & 1u) { stack[sp + __popc(later >> lane >> 1)] = entry; }
            sp += pushes;
            __syncwarp();
        }
        if (overflow) { break; }
        if (numLeaves > 0) { flush(); }
        // the last, partly filled chunk of the list (entries past the count, or past the capacity, are never read)
        if (active)
        {
            unsigned kept = min(count, listCap);
            if (kept % kNbChunk != 0 && piece == 0) { storeChunk(kept / kNbChunk); }
        }

        // smoothing-length iteration (skin rows: one pass at the given h)
        if (kSkin) { active = false; }
        if (active)
        {
            unsigned ncSph = count + 1;
            bool failing   = ngmin > ncSph || (ncSph - 1) > prm.ngmax;
            if (failing && updates < prm.maxIterations)
            {
                hi = updateH(prm.ng0, ncSph, hi);
                ++updates;
            }
            else { active = false; }
        }
    }

    if (overflow)
    {
        if (lane == 0) { atomicOr(status, 1u); }
        return;
    }
    if (valid && piece == 0)
    {
        if constexpr (kSkin)
        {
            ex.sl.count[i]  = count;
            ex.sl.radius[i] = __dmul_rn(2.0 * hi, ex.onePlusSkin);
        }
        else
        {
            ncOut[i] = count + 1;
            h[i]     = hi;
        }
    }
}

template<bool kBatched, int kKind, int kPer>
__global__ void __launch_bounds__(kNbThreads, residentBlocks<kPer, kKind == kSearchSkin>())
    findNeighborsKernel(const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
                        const double4* __restrict__ pos, double* h, size_t n, TreeView tree, DevBox box,
                        NeighborParams prm, uint32_t* __restrict__ nidx, unsigned* __restrict__ ncOut, unsigned* status,
                        const TreeView* __restrict__ views, const uint8_t* __restrict__ inst, SearchExtras ex)
{
    __shared__ NbShared<kPer, kKind == kSearchSkin> sh;
    if (ex.gate && !((ex.gateMask >> __ldg(ex.gate)) & 1u)) { return; }
    searchUnit<kBatched, kKind, kPer>(sh, size_t(blockIdx.x) * kNbWarps + threadIdx.x / kWarp, x, y, z, pos, h, n, tree,
                                      box, prm, nidx, ncOut, status, views, inst, ex);
}

//! the listed groups by as many blocks as stay resident: only the device knows how many they are
template<bool kBatched>
__global__ void __launch_bounds__(kNbThreads, residentBlocks<1, false>())
    findListedKernel(const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
                     const double4* __restrict__ pos, double* h, size_t n, TreeView tree, DevBox box, NeighborParams prm,
                     uint32_t* __restrict__ nidx, unsigned* __restrict__ ncOut, unsigned* status,
                     const TreeView* __restrict__ views, const uint8_t* __restrict__ inst, SearchExtras ex)
{
    __shared__ union
    {
        NbShared<1, false> one;
        NbShared<kManyLanes, false> many;
    } sh;
    const size_t listed = *ex.numListed;
    const size_t stride = size_t(gridDim.x) * kNbWarps;
    size_t unit         = size_t(blockIdx.x) * kNbWarps + threadIdx.x / kWarp;
    if (listed <= kManyLanesListed)
    {
        for (; unit < listed * kManyLanes; unit += stride)
        {
            searchUnit<kBatched, kSearchListed, kManyLanes>(sh.many, unit, x, y, z, pos, h, n, tree, box, prm, nidx, ncOut,
                                                            status, views, inst, ex);
            __syncwarp();
        }
        return;
    }
    for (; unit < listed; unit += stride)
    {
        searchUnit<kBatched, kSearchListed, 1>(sh.one, unit, x, y, z, pos, h, n, tree, box, prm, nidx, ncOut, status, views,
                                               inst, ex);
        __syncwarp();
    }
}

//! bounding box of each run of kBlockSize consecutive particles, relative to the box corner, rounded outwards
__global__ void blockBoxesKernel(const double* __restrict__ x, const double* __restrict__ y,
                                 const double* __restrict__ z, size_t n, DevBox box, float4* lo, float4* hi)
{
    size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    size_t b = c * kBlockSize;
    if (b >= n) { return; }
    size_t e  = min(b + kBlockSize, n);
    double l[3] = {INFINITY, INFINITY, INFINITY}, u[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (size_t j = b; j < e; ++j)
    {
        double p[3] = {x[j] - box.lo[0], y[j] - box.lo[1], z[j] - box.lo[2]};
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            l[k] = fmin(l[k], p[k]);
            u[k] = fmax(u[k], p[k]);
        }
    }
    lo[c] = make_float4(__double2float_rd(l[0]), __double2float_rd(l[1]), __double2float_rd(l[2]), 0.f);
    hi[c] = make_float4(__double2float_ru(u[0]), __double2float_ru(u[1]), __double2float_ru(u[2]), 0.f);
}

} // namespace

int computeBlockBoxes(const double* x, const double* y, const double* z, size_t n, const DevBox& box, float4* lo,
                      float4* hi, cudaStream_t stream)
{
    if (n == 0) { return kOk; }
    size_t blocks = (n + kBlockSize - 1) / kBlockSize;
    blockBoxesKernel<<<ceilDiv(blocks, 256), 256, 0, stream>>>(x, y, z, n, box, lo, hi);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

namespace
{
unsigned searchBlocks(size_t n, int per)
{
    size_t units = (n + kWarp - 1) / kWarp * size_t(per);
    return unsigned((units + kNbWarps - 1) / kNbWarps);
}

//! KERNEL<batched, kind, lanes per target> with one tree or the members' trees
#define SPHB_SEARCH(KIND, PER, BLOCKS, H, NIDX, NC)                                                                    \
    if (views)                                                                                                          \
    {                                                                                                                   \
        findNeighborsKernel<true, KIND, PER><<<BLOCKS, kNbThreads, 0, stream>>>(x, y, z, pos, H, n, tree, box, prm,     \
                                                                                NIDX, NC, status, views, inst, ex);     \
    }                                                                                                                   \
    else                                                                                                                \
    {                                                                                                                   \
        findNeighborsKernel<false, KIND, PER><<<BLOCKS, kNbThreads, 0, stream>>>(                                       \
            x, y, z, pos, H, n, tree, box, prm, NIDX, NC, status, nullptr, nullptr, ex);                                \
    }
} // namespace

int findNeighbors(const double* x, const double* y, const double* z, const double4* pos, double* h, size_t n,
                  const TreeView& tree, const DevBox& box, NeighborParams prm, uint32_t* nidx, unsigned* nc,
                  unsigned* status, cudaStream_t stream, const TreeView* views, const uint8_t* inst,
                  const unsigned* gate, unsigned gateMask)
{
    if (n == 0) { return kOk; }
    if ((views == nullptr) != (inst == nullptr)) { return kErrArg; }
    SearchExtras ex{};
    ex.gate     = gate;
    ex.gateMask = gateMask;
    if (n <= kManyLanesAll) { SPHB_SEARCH(kSearchAll, kManyLanes, searchBlocks(n, kManyLanes), h, nidx, nc) }
    else if (n <= kFewLanesAll) { SPHB_SEARCH(kSearchAll, kFewLanes, searchBlocks(n, kFewLanes), h, nidx, nc) }
    else { SPHB_SEARCH(kSearchAll, 1, searchBlocks(n, 1), h, nidx, nc) }
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int findNeighborsListed(const double* x, const double* y, const double* z, const double4* pos, double* h, size_t n,
                        const TreeView& tree, const DevBox& box, NeighborParams prm, uint32_t* nidx, unsigned* nc,
                        unsigned* status, const unsigned* groups, const unsigned* numListed, cudaStream_t stream,
                        const TreeView* views, const uint8_t* inst)
{
    if (n == 0) { return kOk; }
    if (!groups || !numListed || (views == nullptr) != (inst == nullptr)) { return kErrArg; }
    SearchExtras ex{};
    ex.groups    = groups;
    ex.numListed = numListed;
    unsigned blocks = std::min(searchBlocks(n, kManyLanes), unsigned(smCount() * residentBlocks<1, false>()));
    if (views)
    {
        findListedKernel<true><<<blocks, kNbThreads, 0, stream>>>(x, y, z, pos, h, n, tree, box, prm, nidx, nc, status,
                                                                  views, inst, ex);
    }
    else
    {
        findListedKernel<false><<<blocks, kNbThreads, 0, stream>>>(x, y, z, pos, h, n, tree, box, prm, nidx, nc, status,
                                                                   nullptr, nullptr, ex);
    }
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int buildSkinLists(const double* x, const double* y, const double* z, const double4* pos, const double* h, size_t n,
                   const TreeView& tree, const DevBox& box, NeighborParams prm, double skin, SkinLists sl,
                   unsigned* status, cudaStream_t stream, const TreeView* views, const uint8_t* inst,
                   const unsigned* gate, unsigned gateMask)
{
    if (n == 0) { return kOk; }
    if (!(skin > 0.0) || sl.cap == 0 || sl.cap % kNbChunk != 0 || (views == nullptr) != (inst == nullptr))
    {
        return kErrArg;
    }
    SearchExtras ex{};
    ex.sl          = sl;
    ex.onePlusSkin = 1.0 + skin;
    ex.gate        = gate;
    ex.gateMask    = gateMask;
    // the kernel writes h only in the iterating kinds, never in this one
    double* hRead = const_cast<double*>(h);
    if (n <= kManyLanesAll) { SPHB_SEARCH(kSearchSkin, kManyLanes, searchBlocks(n, kManyLanes), hRead, nullptr, nullptr) }
    else if (n <= kFewLanesAll) { SPHB_SEARCH(kSearchSkin, kFewLanes, searchBlocks(n, kFewLanes), hRead, nullptr, nullptr) }
    else { SPHB_SEARCH(kSearchSkin, 1, searchBlocks(n, 1), hRead, nullptr, nullptr) }
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

} // namespace sphb
