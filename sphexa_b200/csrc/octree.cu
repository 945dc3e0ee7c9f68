// Cornerstone trees on the GPU: leaf counts, csarray rebalance (global tree), focus-tree update at one rank,
// the linked octree (level-major node order) and node geometry.
//
// The O(n) work (binary searches over the particle keys) and all O(nodes) decisions run as kernels; the host only
// reads a few status words per update to drive the convergence loops, as the reference's loops do
// (cstone/domain/assignment.hpp:114-123, cstone/focus/octree_focus_mpi.hpp:582-599).
#include <algorithm>
#include <cstring>
#include <vector>

#include "octree.cuh"
#include "sfc.cuh"

namespace sphb
{

namespace
{

__device__ inline size_t lowerBound(const uint64_t* a, size_t n, uint64_t v)
{
    size_t lo = 0, hi = n;
    while (lo < hi)
    {
        size_t mid = (lo + hi) >> 1;
        if (a[mid] < v) { lo = mid + 1; }
        else { hi = mid; }
    }
    return lo;
}

//! level of the coarsest node that starts at key (number of leading octal digits up to the last non-zero one)
__host__ __device__ inline unsigned alignmentLevel(uint64_t key)
{
    if (key == 0) { return 0; }
#ifdef __CUDA_ARCH__
    unsigned tz = __ffsll((long long)key) - 1;
#else
    unsigned tz = __builtin_ctzll(key);
#endif
    return (63u - tz + 2u) / 3u;
}

__host__ __device__ inline unsigned octalDigitAt(uint64_t key, unsigned level)
{
    return unsigned(key >> (3u * (kMaxLevel - level))) & 7u;
}

// ---------------------------------------------------------------------------------------------------------------
// linked octree construction
// ---------------------------------------------------------------------------------------------------------------

// The node order is level-major, and within a level the nodes are in key order, which is the order of the leaves that
// start them: leaf i starts one node on every level from the coarsest aligned with its key to its own. The position
// of a node is therefore its level's first index plus the number of leaves before i that start a node of the level: a
// count per level and block of leaves, one scan, and the positions. This replaces a radix sort of the prefixes (eight
// passes and two host reads); with one scan launch per array and no scan for the layout, the sync takes 235 instead
// of 300 us at 4,096 particles, 510 instead of 630 at 27,000, 945 instead of 1,110 at 128^3.

constexpr int kLevels       = int(kMaxLevel) + 1;
constexpr int kLevelThreads = 256;
constexpr int kLevelWarps   = kLevelThreads / 32;

/*! the levels [a, b] of the nodes that leaf i starts (b: the leaf itself); a > b past the end and for a malformed
 *  leaf array */
__device__ __forceinline__ void startedLevels(const uint64_t* leaves, int numLeaves, int i, uint64_t* key, int* a, int* b)
{
    *a = 1;
    *b = 0;
    if (i >= numLeaves) { return; }
    *key = leaves[i];
    *b   = min(int(treeLevelOf(leaves[i + 1] - *key)), int(kMaxLevel));
    *a   = min(int(alignmentLevel(*key)), *b);
}

//! counts[l * gridDim.x + block] = nodes of level l started by the block's leaves
__global__ void __launch_bounds__(kLevelThreads) levelCountKernel(const uint64_t* leaves, int numLeaves, int* counts)
{
    __shared__ int sh[kLevels];
    if (threadIdx.x < kLevels) { sh[threadIdx.x] = 0; }
    __syncthreads();
    uint64_t key;
    int a, b;
    startedLevels(leaves, numLeaves, blockIdx.x * kLevelThreads + threadIdx.x, &key, &a, &b);
    for (int l = 0; l < kLevels; ++l)
    {
        unsigned m = __ballot_sync(0xffffffffu, l >= a && l <= b);
        if ((threadIdx.x & 31) == 0 && m) { atomicAdd(&sh[l], __popc(m)); }
    }
    __syncthreads();
    if (threadIdx.x < kLevels) { counts[threadIdx.x * gridDim.x + blockIdx.x] = sh[threadIdx.x]; }
}

//! counts -> first node index per level and block, and the level ranges (one block, one warp per level)
__global__ void __launch_bounds__(kLevels * 32) levelScanKernel(int* counts, int numBlocks, int numNodes, int* levelRange)
{
    __shared__ int total[kLevels];
    __shared__ int first[kLevels + 1];
    int l = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* row = counts + size_t(l) * numBlocks;
    int sum  = 0;
    for (int q = lane; q < numBlocks; q += 32)
    {
        sum += row[q];
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) { total[l] = sum; }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int run = 0;
        for (int k = 0; k < kLevels; ++k)
        {
            first[k] = run;
            run += total[k];
        }
        first[kLevels] = numNodes;
    }
    __syncthreads();
    if (threadIdx.x <= kLevels) { levelRange[threadIdx.x] = first[threadIdx.x]; }
    int carry = first[l];
    for (int base = 0; base < numBlocks; base += 32)
    {
        int q = base + lane;
        int v = q < numBlocks ? row[q] : 0;
        int incl = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
        {
            int t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) { incl += t; }
        }
        if (q < numBlocks) { row[q] = carry + incl - v; }
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
}

//! every node at its position (positions past the arrays, of a malformed leaf array, are dropped)
__global__ void __launch_bounds__(kLevelThreads) emitNodesKernel(const uint64_t* leaves, int numLeaves, int numNodes,
                                                                const int* firstOf, uint64_t* prefixes,
                                                                int* nodeToLeaf, int* leafToNode)
{
    __shared__ int before[kLevelWarps][kLevels];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * kLevelThreads + threadIdx.x;
    uint64_t key;
    int a, b;
    startedLevels(leaves, numLeaves, i, &key, &a, &b);
    for (int l = 0; l < kLevels; ++l)
    {
        unsigned m = __ballot_sync(0xffffffffu, l >= a && l <= b);
        if (lane == 0) { before[warp][l] = __popc(m); }
    }
    __syncthreads();
    if (threadIdx.x < kLevels)
    {
        int run = firstOf[threadIdx.x * gridDim.x + blockIdx.x];
        for (int w = 0; w < kLevelWarps; ++w)
        {
            int c                  = before[w][threadIdx.x];
            before[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int l = 0; l < kLevels; ++l)
    {
        bool mine  = l >= a && l <= b;
        unsigned m = __ballot_sync(0xffffffffu, mine);
        if (!mine) { continue; }
        int p = before[warp][l] + __popc(m & ((1u << lane) - 1u));
        if (p < numNodes)
        {
            prefixes[p]   = encodePrefix(key, unsigned(l));
            nodeToLeaf[p] = l == b ? i : -1;
        }
        if (l == b) { leafToNode[i] = min(p, numNodes - 1); }
    }
}

struct LevelRange
{
    int r[kMaxLevel + 2];
};

__global__ void linkKernel(const uint64_t* prefixes, const int* nodeToLeaf, int numNodes, const int* levelRange,
                           int* childOffsets, int* parents)
{
    __shared__ LevelRange lr;
    if (threadIdx.x < kMaxLevel + 2) { lr.r[threadIdx.x] = levelRange[threadIdx.x]; }
    __syncthreads();
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= numNodes) { return; }
    if (nodeToLeaf[p] >= 0)
    {
        childOffsets[p] = 0;
        return;
    }
    uint64_t prefix = prefixes[p];
    unsigned level  = prefixLevel(prefix);
    if (prefix == 0 || level >= kMaxLevel)
    {
        childOffsets[p] = 0; // malformed leaf array
        return;
    }
    uint64_t child  = encodePrefix(prefixStart(prefix), level + 1);
    int b           = lr.r[level + 1];
    int e           = lr.r[level + 2];
    int c = b + int(lowerBound(prefixes + b, size_t(e - b), child));
    if (c >= e || c + 8 > numNodes || prefixes[c] != child)
    {
        childOffsets[p] = 0; // malformed leaf array: leave the node childless rather than link out of range
        return;
    }
    childOffsets[p]      = c;
    parents[(c - 1) / 8] = p;
}

// ---------------------------------------------------------------------------------------------------------------
// counts and geometry
// ---------------------------------------------------------------------------------------------------------------

constexpr int kCountThreads = 256;

/*! Trees of at most this many leaves are updated by single blocks that do several of the steps below one after another: a
 *  step over a few thousand nodes takes about 3 us, most of it launch, and eleven launches become three. Sync of 16^3
 *  particles 157 -> 127 us, of 30^3 164 -> 137 us. Beyond 2,048 leaves a phase is several rounds of one SM. */
constexpr int kSmallTree    = 2048;
constexpr int kSmallThreads = 1024;

/*! data[0 .. n) -> its exclusive scan, in place, and the sum to data[n], by one block of kSmallThreads */
__device__ void blockScanInPlace(int* data, int n)
{
    __shared__ int warpSum[kSmallThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += kSmallThreads)
    {
        int i    = base + threadIdx.x;
        int v    = i < n ? data[i] : 0;
        int incl = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
        {
            int t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) { incl += t; }
        }
        if (lane == 31) { warpSum[warp] = incl; }
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < kSmallThreads / 32; ++w)
        {
            before += w < warp ? warpSum[w] : 0;
            all += warpSum[w];
        }
        if (i < n) { data[i] = carry + before + incl - v; }
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) { data[n] = carry; }
}

/*! counts[i] = keys in [leaves[i], leaves[i + 1]), the layout first[i] = keys below leaves[i] (i <= numLeaves; the
 *  exclusive scan of the counts, since the leaves start at key 0), and the largest count into *maxCount; first and
 *  maxCount may be null. One binary search per boundary: a leaf takes its end from the next thread. */
__global__ void __launch_bounds__(kCountThreads) leafCountsKernel(const uint64_t* leaves, int numLeaves,
                                                                 const uint64_t* keys, size_t n, unsigned* counts,
                                                                 int* first, unsigned* maxCount)
{
    __shared__ size_t bound[kCountThreads];
    int i = blockIdx.x * (kCountThreads - 1) + threadIdx.x;
    size_t b = i <= numLeaves ? lowerBound(keys, n, leaves[i]) : n;
    bound[threadIdx.x] = b;
    __syncthreads();
    unsigned c = 0;
    if (threadIdx.x < kCountThreads - 1 && i <= numLeaves)
    {
        if (first) { first[i] = int(b); }
        if (i < numLeaves)
        {
            c         = unsigned(bound[threadIdx.x + 1] - b);
            counts[i] = c;
        }
    }
    if (maxCount)
    {
        c = __reduce_max_sync(0xffffffffu, c);
        if ((threadIdx.x & 31) == 0 && c) { atomicMax(maxCount, c); }
    }
}

//! count of node p: a leaf's own, or the layout at the ends of the leaves an internal node covers
__device__ __forceinline__ void nodeCountOf(int p, const uint64_t* prefixes, const int* nodeToLeaf,
                                            const uint64_t* leaves, int numLeaves, const unsigned* leafCounts,
                                            const int* layout, unsigned* nodeCounts)
{
    int leaf = nodeToLeaf[p];
    if (leaf >= 0)
    {
        nodeCounts[p] = leafCounts[leaf];
        return;
    }
    uint64_t prefix = prefixes[p];
    unsigned level  = prefixLevel(prefix);
    uint64_t start  = prefixStart(prefix);
    uint64_t end    = start + nodeRangeAt(level);
    size_t b        = lowerBound(leaves, size_t(numLeaves) + 1, start);
    size_t e        = lowerBound(leaves, size_t(numLeaves) + 1, end);
    nodeCounts[p]   = unsigned(layout[e] - layout[b]);
}

__global__ void nodeCountsKernel(const uint64_t* prefixes, const int* nodeToLeaf, int numNodes, const uint64_t* leaves,
                                 int numLeaves, const unsigned* leafCounts, const int* layout, unsigned* nodeCounts)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < numNodes) { nodeCountOf(p, prefixes, nodeToLeaf, leaves, numLeaves, leafCounts, layout, nodeCounts); }
}

__device__ __forceinline__ void geoOf(int p, const uint64_t* prefixes, const DevBox& box, double* centers, double* sizes)
{
    uint64_t prefix = prefixes[p];
    unsigned level  = prefixLevel(prefix);
    unsigned ixyz[3];
    hilbertDecode(prefixStart(prefix), ixyz);
    unsigned edge = (1u << kMaxLevel) >> level;
    unsigned mask = ~(edge - 1u);
    for (int k = 0; k < 3; ++k)
    {
        unsigned lo     = ixyz[k] & mask;
        unsigned hi     = lo + edge;
        double halfUnit = 0.5 * (1.0 / double(1u << kMaxLevel)) * box.len[k];
        centers[3 * p + k] = box.lo[k] + double(hi + lo) * halfUnit;
        sizes[3 * p + k]   = double(hi - lo) * halfUnit;
    }
}

__global__ void geoKernel(const uint64_t* prefixes, int numNodes, DevBox box, double* centers, double* sizes)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < numNodes) { geoOf(p, prefixes, box, centers, sizes); }
}

/*! the number of keys below every leaf boundary into bound (shared, kSmallTree + 1 entries), and the leaves' counts, by one
 *  block; returns this thread's largest count */
__device__ unsigned blockLeafCounts(const uint64_t* leaves, int numLeaves, const uint64_t* keys, size_t n,
                                    unsigned* counts, unsigned* bound)
{
    for (int i = threadIdx.x; i <= numLeaves; i += kSmallThreads)
    {
        bound[i] = unsigned(lowerBound(keys, n, leaves[i]));
    }
    __syncthreads();
    unsigned largest = 0;
    for (int i = threadIdx.x; i < numLeaves; i += kSmallThreads)
    {
        unsigned c = bound[i + 1] - bound[i];
        counts[i]  = c;
        largest    = max(largest, c);
    }
    return largest;
}

//! leaf counts, layout, node counts and, if centers is set, the node geometry of a small tree
__global__ void __launch_bounds__(kSmallThreads) smallCountsKernel(const uint64_t* leaves, int numLeaves,
                                                                  const uint64_t* keys, size_t n, unsigned* counts,
                                                                  int* layout, const uint64_t* prefixes,
                                                                  const int* nodeToLeaf, int numNodes,
                                                                  unsigned* nodeCounts, DevBox box, double* centers,
                                                                  double* sizes)
{
    __shared__ unsigned bound[kSmallTree + 1];
    blockLeafCounts(leaves, numLeaves, keys, n, counts, bound);
    for (int i = threadIdx.x; i <= numLeaves; i += kSmallThreads)
    {
        layout[i] = int(bound[i]);
    }
    __syncthreads();
    for (int p = threadIdx.x; p < numNodes; p += kSmallThreads)
    {
        nodeCountOf(p, prefixes, nodeToLeaf, leaves, numLeaves, counts, layout, nodeCounts);
        if (centers) { geoOf(p, prefixes, box, centers, sizes); }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// global tree: csarray rebalance (cstone/tree/csarray.hpp:248-389)
// ---------------------------------------------------------------------------------------------------------------

__device__ __forceinline__ void csNodeOp(int i, const uint64_t* leaves, const unsigned* counts, int numLeaves,
                                         unsigned bucket, int* ops, unsigned* flags)
{
    if (i == numLeaves)
    {
        ops[i] = 0;
        return;
    }
    uint64_t key   = leaves[i];
    unsigned level = treeLevelOf(leaves[i + 1] - key);
    int op         = 1;
    bool decided   = false;
    if (level > 0)
    {
        int sib = int(octalDigitAt(key, level));
        // the 8 siblings are all leaves if the group spans exactly one parent node
        bool siblings = sib > 0 && leaves[i - sib + 8] == leaves[i - sib] + nodeRangeAt(level - 1);
        if (siblings)
        {
            const unsigned* g = counts + i - sib;
            size_t parentCount = 0;
            for (int k = 0; k < 8; ++k)
            {
                parentCount += g[k];
            }
            if (parentCount <= size_t(bucket))
            {
                op      = 0;
                decided = true;
            }
        }
    }
    if (!decided)
    {
        unsigned c = counts[i];
        if (c > bucket * 512u && level + 3 < kMaxLevel) { op = 4096; }
        else if (c > bucket * 64u && level + 2 < kMaxLevel) { op = 512; }
        else if (c > bucket * 8u && level + 1 < kMaxLevel) { op = 64; }
        else if (c > bucket && level < kMaxLevel) { op = 8; }
    }
    ops[i] = op;
    if (op != 1) { atomicOr(flags, 1u); }
}

__global__ void csNodeOpsKernel(const uint64_t* leaves, const unsigned* counts, int numLeaves, unsigned bucket,
                                int* ops, unsigned* flags)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= numLeaves) { csNodeOp(i, leaves, counts, numLeaves, bucket, ops, flags); }
}

//! globalTreeStep's ops, their scan and the counts of the current leaves for a small tree; flags cleared before
__global__ void __launch_bounds__(kSmallThreads) smallGlobalStepKernel(const uint64_t* leaves, unsigned* counts,
                                                                      int numLeaves, unsigned bucket, int* ops,
                                                                      unsigned* flags, const uint64_t* keys, size_t n)
{
    __shared__ unsigned bound[kSmallTree + 1];
    if (threadIdx.x < 4) { flags[threadIdx.x] = 0; }
    __syncthreads();
    for (int i = threadIdx.x; i <= numLeaves; i += kSmallThreads)
    {
        csNodeOp(i, leaves, counts, numLeaves, bucket, ops, flags);
    }
    __syncthreads();
    blockScanInPlace(ops, numLeaves + 1);
    unsigned largest = blockLeafCounts(leaves, numLeaves, keys, n, counts, bound);
    if (largest) { atomicMax(flags + 1, largest); }
}

//! new leaves from scanned ops (processNode, cstone/tree/csarray.hpp:340-366)
__global__ void rebalanceKernel(const uint64_t* leaves, int numLeaves, const int* scan, uint64_t* newLeaves)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > numLeaves) { return; }
    if (i == numLeaves)
    {
        newLeaves[scan[numLeaves]] = leaves[numLeaves];
        return;
    }
    uint64_t key   = leaves[i];
    unsigned level = treeLevelOf(leaves[i + 1] - key);
    int op         = scan[i + 1] - scan[i];
    int out        = scan[i];
    if (op == 1) { newLeaves[out] = key; }
    else if (op > 1)
    {
        unsigned levelDiff = op == 8 ? 1 : op == 64 ? 2 : op == 512 ? 3 : 4;
        uint64_t step      = nodeRangeAt(level + levelDiff);
        for (int s = 0; s < op; ++s)
        {
            newLeaves[out + s] = key + uint64_t(s) * step;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// focus tree update at one rank (cstone/focus/rebalance.hpp, octree_focus.hpp:61-129)
// ---------------------------------------------------------------------------------------------------------------

enum Resolution : unsigned
{
    kConverged   = 0,
    kCancelMerge = 1,
    kRebalance   = 2,
    kFailed      = 3,
};

/*! mergeCountAndMacOp (rebalance.hpp:31-75) with the whole key range in focus: every node is inside the focus and
 *  every sibling group is in the fringe, so the MAC never decides and only particle counts do. */
__device__ __forceinline__ void focusOp(int p, const uint64_t* prefixes, const int* childOffsets, const int* parents,
                                        const unsigned* counts, unsigned bucket, int* ops)
{
    if (p > 0)
    {
        int parent = parents[(p - 1) / 8];
        if (counts[parent] <= bucket)
        {
            ops[p] = 0;
            return;
        }
    }
    unsigned level = prefixLevel(prefixes[p]);
    int op         = 1;
    if (childOffsets[p] == 0)
    {
        unsigned c = counts[p];
        if (level + 3 < kMaxLevel && c > 4096u * bucket) { op = 4096; }
        else if (level + 2 < kMaxLevel && c > 512u * bucket) { op = 512; }
        else if (level + 1 < kMaxLevel && c > 64u * bucket) { op = 64; }
        else if (level < kMaxLevel && c > bucket) { op = 8; }
    }
    ops[p] = op;
}

__global__ void focusOpsKernel(const uint64_t* prefixes, const int* childOffsets, const int* parents,
                               const unsigned* counts, int numNodes, unsigned bucket, int* ops)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < numNodes) { focusOp(p, prefixes, childOffsets, parents, counts, bucket, ops); }
}

//! smallest existing node containing the node with placeholder-bit key `want` (octree.hpp:199-216)
__device__ int containingNodeOf(uint64_t want, const uint64_t* prefixes, const int* childOffsets)
{
    unsigned wantLevel = prefixLevel(want);
    uint64_t key       = prefixStart(want);
    int node           = 0;
    for (unsigned l = 1; l <= wantLevel; ++l)
    {
        if (childOffsets[node] == 0 || prefixes[node] == want) { break; }
        node = childOffsets[node] + int(octalDigitAt(key, l));
    }
    return node;
}

/*! enforceKeySingle (rebalance.hpp:161-212) for every mandatory key in parallel. Sibling resets only ever turn 0
 *  into 1 and splits take the maximum, so the final ops and the maximum status do not depend on key order. */
__device__ __forceinline__ void enforceKey(uint64_t key, const uint64_t* prefixes, const int* childOffsets,
                                           const int* parents, int* ops, unsigned* status)
{
    if (key == 0 || key == kRootRange) { return; }

    unsigned lastNz    = kMaxLevel - unsigned(__ffsll((long long)key) - 1) / 3u;
    uint64_t want      = encodePrefix(key, lastNz);
    int node           = containingNodeOf(want, prefixes, childOffsets);
    uint64_t have      = prefixes[node];
    unsigned haveLevel = prefixLevel(have);

    unsigned st     = kConverged;
    bool trySplit   = have != want && haveLevel < kMaxLevel;
    bool undoMerges = ops[node] == 0 || trySplit;
    if (undoMerges && node > 0)
    {
        st         = kCancelMerge;
        int parent = node;
        do
        {
            parent    = parents[(parent - 1) / 8];
            int first = childOffsets[parent];
            for (int s = first; s < first + 8; ++s)
            {
                atomicCAS(ops + s, 0, 1); // 0 -> 1 only; must not undo a concurrent split of the same node
            }
        } while (parent != 0);
    }
    if (trySplit)
    {
        int levelDiff = int(lastNz) - int(haveLevel);
        st            = levelDiff > 1 ? kFailed : kRebalance;
        atomicMax(ops + node, 8);
    }
    if (st != kConverged) { atomicMax(status, st); }
}

__global__ void enforceKeysKernel(const uint64_t* keys, int numKeys, const uint64_t* prefixes, const int* childOffsets,
                                  const int* parents, int* ops, unsigned* status)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < numKeys) { enforceKey(keys[t], prefixes, childOffsets, parents, ops, status); }
}

//! nzAncestorOp (rebalance.hpp:96-116): merged nodes are kept only as the left-most descendant of a kept ancestor
__device__ __forceinline__ void protectOp(int p, const uint64_t* prefixes, const int* parents, const int* opsIn,
                                          int* opsOut, unsigned* numChanges)
{
    int res;
    if (p == 0) { res = opsIn[0]; }
    else
    {
        int anc = p;
        while (opsIn[anc] == 0)
        {
            anc = parents[(anc - 1) / 8];
        }
        res = prefixStart(prefixes[p]) == prefixStart(prefixes[anc]) ? opsIn[anc] : 0;
    }
    opsOut[p] = res;
    if (res != 1) { atomicAdd(numChanges, 1u); }
}

__global__ void protectKernel(const uint64_t* prefixes, const int* parents, const int* opsIn, int numNodes,
                              int* opsOut, unsigned* numChanges)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < numNodes) { protectOp(p, prefixes, parents, opsIn, opsOut, numChanges); }
}

__device__ __forceinline__ void leafOp(int i, const int* nodeOps, const int* leafToNode, int numLeaves, int* leafOps,
                                       unsigned* numNotOne)
{
    if (i == numLeaves)
    {
        leafOps[i] = 0;
        return;
    }
    int op     = nodeOps[leafToNode[i]];
    leafOps[i] = op;
    if (op != 1) { atomicAdd(numNotOne, 1u); }
}

__global__ void leafOpsKernel(const int* nodeOps, const int* leafToNode, int numLeaves, int* leafOps,
                              unsigned* numNotOne)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= numLeaves) { leafOp(i, nodeOps, leafToNode, numLeaves, leafOps, numNotOne); }
}

//! focusUpdateTree's ops of nodes and leaves and their scan for a small tree; flags cleared before
__global__ void __launch_bounds__(kSmallThreads) smallFocusOpsKernel(const uint64_t* prefixes, const int* childOffsets,
                                                                    const int* parents, const unsigned* counts,
                                                                    int numNodes, unsigned bucket,
                                                                    const uint64_t* keys, int numKeys,
                                                                    const int* leafToNode, int numLeaves, int* ops,
                                                                    int* opsOut, unsigned* flags)
{
    if (threadIdx.x < 4) { flags[threadIdx.x] = 0; }
    for (int p = threadIdx.x; p < numNodes; p += kSmallThreads)
    {
        focusOp(p, prefixes, childOffsets, parents, counts, bucket, ops);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < numKeys; t += kSmallThreads)
    {
        enforceKey(keys[t], prefixes, childOffsets, parents, ops, flags);
    }
    __syncthreads();
    for (int p = threadIdx.x; p < numNodes; p += kSmallThreads)
    {
        protectOp(p, prefixes, parents, ops, opsOut, flags + 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= numLeaves; i += kSmallThreads)
    {
        leafOp(i, opsOut, leafToNode, numLeaves, ops, flags + 2);
    }
    __syncthreads();
    blockScanInPlace(ops, numLeaves + 1);
}

__global__ void setLeavesKernel(uint64_t* leaves, unsigned* counts, unsigned initialCount)
{
    leaves[0] = 0;
    leaves[1] = kRootRange;
    if (counts) { counts[0] = initialCount; }
}

//! the canonical cornerstone cover of [a, b): largest aligned nodes, greedy from a (host, used for key injection)
void spanRange(uint64_t a, uint64_t b, std::vector<uint64_t>& out)
{
    while (a < b)
    {
        unsigned level = alignmentLevel(a);
        while (a + nodeRangeAt(level) > b)
        {
            ++level;
        }
        out.push_back(a);
        a += nodeRangeAt(level);
    }
}

} // namespace

// -------------------------------------------------------------------------------------------------------------------

int buildLinkedOctree(const uint64_t* leaves, int numLeaves, LinkedOctree& t, TreeScratch& s, cudaStream_t stream)
{
    t.numLeaves   = numLeaves;
    t.numInternal = (numLeaves - 1) / 7;
    t.numNodes    = t.numLeaves + t.numInternal;
    int nn        = t.numNodes;

    SPHB_TRY(t.prefixes.reserve(nn));
    SPHB_TRY(t.childOffsets.reserve(nn + 1));
    SPHB_TRY(t.parents.reserve(std::max(1, (nn - 1) / 8)));
    SPHB_TRY(t.nodeToLeaf.reserve(nn));
    SPHB_TRY(t.leafToNode.reserve(numLeaves));
    SPHB_TRY(t.nodeCounts.reserve(nn));
    SPHB_TRY(t.centers.reserve(3 * size_t(nn)));
    SPHB_TRY(t.sizes.reserve(3 * size_t(nn)));
    unsigned nb = ceilDiv(numLeaves, kLevelThreads);
    SPHB_TRY(s.ints.reserve(size_t(kLevels) * nb));
    // the level ranges stay on the device: the link kernel reads them there (no host round trip per tree build)
    SPHB_TRY(t.levelRangeD.reserve(kMaxLevel + 2));
    levelCountKernel<<<nb, kLevelThreads, 0, stream>>>(leaves, numLeaves, s.ints.data());
    levelScanKernel<<<1, kLevels * 32, 0, stream>>>(s.ints.data(), int(nb), nn, t.levelRangeD.data());
    emitNodesKernel<<<nb, kLevelThreads, 0, stream>>>(leaves, numLeaves, nn, s.ints.data(), t.prefixes.data(),
                                                      t.nodeToLeaf.data(), t.leafToNode.data());
    countLaunch(3);
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_CUDA_TRY(cudaMemsetAsync(t.parents.data(), 0, sizeof(int) * std::max(1, (nn - 1) / 8), stream));
    linkKernel<<<ceilDiv(nn, 256), 256, 0, stream>>>(t.prefixes.data(), t.nodeToLeaf.data(), nn,
                                                     t.levelRangeD.data(), t.childOffsets.data(), t.parents.data());
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int computeLeafCounts(const uint64_t* leaves, int numLeaves, const uint64_t* keys, size_t n, unsigned* counts,
                      cudaStream_t stream, int* layout, unsigned* maxCount)
{
    unsigned nb = ceilDiv(numLeaves + 1, kCountThreads - 1);
    leafCountsKernel<<<nb, kCountThreads, 0, stream>>>(leaves, numLeaves, keys, n, counts, layout, maxCount);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int computeNodeCounts(const uint64_t* leaves, const unsigned* leafCounts, const int* layout, LinkedOctree& t,
                      cudaStream_t stream)
{
    nodeCountsKernel<<<ceilDiv(t.numNodes, 256), 256, 0, stream>>>(t.prefixes.data(), t.nodeToLeaf.data(), t.numNodes,
                                                                  leaves, t.numLeaves, leafCounts, layout,
                                                                  t.nodeCounts.data());
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int computeGeoCenters(LinkedOctree& t, const DevBox& box, cudaStream_t stream)
{
    geoKernel<<<ceilDiv(t.numNodes, 256), 256, 0, stream>>>(t.prefixes.data(), t.numNodes, box, t.centers.data(),
                                                           t.sizes.data());
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

// -------------------------------------------------------------------------------------------------------------------

int initGlobalTree(GlobalTree& g, unsigned bucket, cudaStream_t stream)
{
    // one root leaf with count bucket-1 (GlobalAssignment constructor, cstone/domain/assignment.hpp:57-74)
    g.bucket    = bucket;
    g.numLeaves = 1;
    g.firstCall = true;
    SPHB_TRY(g.leaves.reserve(2));
    SPHB_TRY(g.counts.reserve(1));
    setLeavesKernel<<<1, 1, 0, stream>>>(g.leaves.data(), g.counts.data(), bucket - 1);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int globalTreeStep(GlobalTree& g, const uint64_t* keys, size_t n, TreeScratch& s, cudaStream_t stream,
                   unsigned* maxCount)
{
    int L = g.numLeaves;
    SPHB_TRY(s.ints.reserve(L + 2));
    SPHB_TRY(s.scanTmp.reserve(scanTempInts(L + 1) + 1));
    SPHB_TRY(s.flags.reserve(4));
    // with the counts of the current leaves, before knowing whether they change: in the steady state nothing splits or
    // merges and one read back serves both decisions
    if (L <= kSmallTree && n <= UINT32_MAX)
    {
        smallGlobalStepKernel<<<1, kSmallThreads, 0, stream>>>(g.leaves.data(), g.counts.data(), L, g.bucket,
                                                               s.ints.data(), s.flags.data(), keys, n);
        countLaunch();
        SPHB_CUDA_TRY(cudaGetLastError());
    }
    else
    {
        SPHB_CUDA_TRY(cudaMemsetAsync(s.flags.data(), 0, 4 * sizeof(unsigned), stream));
        csNodeOpsKernel<<<ceilDiv(L + 1, 256), 256, 0, stream>>>(g.leaves.data(), g.counts.data(), L, g.bucket,
                                                                 s.ints.data(), s.flags.data());
        countLaunch();
        SPHB_TRY(exclusiveScan(s.ints.data(), s.ints.data(), L + 1, s.scanTmp.data(), stream));
        SPHB_TRY(computeLeafCounts(g.leaves.data(), L, keys, n, g.counts.data(), stream, nullptr, s.flags.data() + 1));
    }
    unsigned msg[3]; // new leaf count, any op, largest count
    SPHB_TRY(readBack(stream, {{msg, s.ints.data() + L, sizeof(int)}, {msg + 1, s.flags.data(), 2 * sizeof(unsigned)}}));
    int newL       = int(msg[0]);
    unsigned anyOp = msg[1];
    if (anyOp)
    {
        // every op 1 would give the same leaves: the rebalance runs only when a node splits or merges
        SPHB_TRY(g.leavesAlt.reserve(newL + 1));
        rebalanceKernel<<<ceilDiv(L + 1, 256), 256, 0, stream>>>(g.leaves.data(), L, s.ints.data(),
                                                                 g.leavesAlt.data());
        countLaunch();
        SPHB_CUDA_TRY(cudaGetLastError());
        g.leaves.swap(g.leavesAlt);
        g.numLeaves = newL;
        SPHB_TRY(g.counts.reserve(newL));
        SPHB_CUDA_TRY(cudaMemsetAsync(s.flags.data() + 1, 0, sizeof(unsigned), stream));
        SPHB_TRY(computeLeafCounts(g.leaves.data(), newL, keys, n, g.counts.data(), stream, nullptr,
                                   s.flags.data() + 1));
        SPHB_TRY(readBack(stream, {{msg + 2, s.flags.data() + 1, sizeof(unsigned)}}));
    }
    *maxCount = anyOp ? msg[2] : 0u;
    return kOk;
}

int updateGlobalTree(GlobalTree& g, const uint64_t* keys, size_t n, TreeScratch& s, cudaStream_t stream)
{
    unsigned maxCount = 0;
    SPHB_TRY(globalTreeStep(g, keys, n, s, stream, &maxCount));
    if (g.firstCall || maxCount >= 8 * g.bucket)
    {
        g.firstCall = false;
        int guard   = 0;
        do
        {
            SPHB_TRY(globalTreeStep(g, keys, n, s, stream, &maxCount));
            if (++guard > 64) { return kErrNotConverged; }
        } while (maxCount > g.bucket);
    }
    return kOk;
}

// -------------------------------------------------------------------------------------------------------------------

int initFocusTree(FocusTree& f, unsigned bucket, TreeScratch& s, cudaStream_t stream)
{
    // FocusedOctree constructor (octree_focus_mpi.hpp:63-88): root leaf, counts bucket+1
    f.bucket    = bucket;
    f.numLeaves = 1;
    f.firstCall = true;
    SPHB_TRY(f.leaves.reserve(2));
    SPHB_TRY(f.leafCounts.reserve(1));
    SPHB_TRY(f.layout.reserve(2));
    setLeavesKernel<<<1, 1, 0, stream>>>(f.leaves.data(), f.leafCounts.data(), bucket + 1);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_TRY(buildLinkedOctree(f.leaves.data(), 1, f.tree, s, stream));
    unsigned c = bucket + 1;
    SPHB_CUDA_TRY(cudaMemcpyAsync(f.tree.nodeCounts.data(), &c, sizeof(unsigned), cudaMemcpyHostToDevice, stream));
    SPHB_CUDA_TRY(cudaStreamSynchronize(stream));
    return kOk;
}

int focusUpdateTree(FocusTree& f, const GlobalTree& g, TreeScratch& s, cudaStream_t stream, bool* converged)
{
    LinkedOctree& t = f.tree;
    int nn          = t.numNodes;
    int L           = f.numLeaves;
    SPHB_TRY(s.ints.reserve(nn + L + 2));
    SPHB_TRY(s.ints2.reserve(nn + L + 2));
    SPHB_TRY(s.scanTmp.reserve(scanTempInts(L + 1) + 1));
    SPHB_TRY(s.flags.reserve(4));
    int* ops    = s.ints.data();
    int* opsOut = s.ints2.data();
    int* leafOps = ops; // node ops no longer needed
    // mandatory keys: the global leaves (the focus start 0 and end 2^63 are always converged)
    if (L <= kSmallTree && g.numLeaves <= kSmallTree)
    {
        smallFocusOpsKernel<<<1, kSmallThreads, 0, stream>>>(
            t.prefixes.data(), t.childOffsets.data(), t.parents.data(), t.nodeCounts.data(), nn, f.bucket,
            g.leaves.data(), g.numLeaves + 1, t.leafToNode.data(), L, ops, opsOut, s.flags.data());
        countLaunch();
        SPHB_CUDA_TRY(cudaGetLastError());
    }
    else
    {
        SPHB_CUDA_TRY(cudaMemsetAsync(s.flags.data(), 0, 4 * sizeof(unsigned), stream));
        focusOpsKernel<<<ceilDiv(nn, 256), 256, 0, stream>>>(t.prefixes.data(), t.childOffsets.data(),
                                                             t.parents.data(), t.nodeCounts.data(), nn, f.bucket, ops);
        enforceKeysKernel<<<ceilDiv(g.numLeaves + 1, 128), 128, 0, stream>>>(
            g.leaves.data(), g.numLeaves + 1, t.prefixes.data(), t.childOffsets.data(), t.parents.data(), ops,
            s.flags.data());
        protectKernel<<<ceilDiv(nn, 256), 256, 0, stream>>>(t.prefixes.data(), t.parents.data(), ops, nn, opsOut,
                                                            s.flags.data() + 1);
        leafOpsKernel<<<ceilDiv(L + 1, 256), 256, 0, stream>>>(opsOut, t.leafToNode.data(), L, leafOps,
                                                               s.flags.data() + 2);
        countLaunch(4);
        SPHB_CUDA_TRY(cudaGetLastError());
        SPHB_TRY(exclusiveScan(leafOps, leafOps, L + 1, s.scanTmp.data(), stream));
    }
    int newL = 0;
    unsigned flags[3];
    SPHB_TRY(readBack(stream, {{&newL, leafOps + L, sizeof(int)}, {flags, s.flags.data(), sizeof(flags)}}));
    unsigned status = flags[0];
    bool conv       = flags[1] == 0;
    if (status == kCancelMerge) { conv = flags[2] == 0; }
    else if (status == kRebalance) { conv = false; }
    if (status != kFailed && flags[2] == 0 && newL == L)
    {
        // every leaf keeps its op 1: the leaves, and so the linked octree, stay as they are
        *converged = conv;
        return kOk;
    }

    SPHB_TRY(f.leavesAlt.reserve(newL + 1));
    rebalanceKernel<<<ceilDiv(L + 1, 256), 256, 0, stream>>>(f.leaves.data(), L, leafOps, f.leavesAlt.data());
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    f.leaves.swap(f.leavesAlt);
    f.numLeaves = newL;

    if (status == kFailed)
    {
        // injectKeys (cstone/focus/inject.hpp): merge the spanning tree of the mandatory keys into the leaves
        conv = false;
        std::vector<uint64_t> leaves(newL + 1);
        std::vector<uint64_t> mand(g.numLeaves + 1);
        SPHB_CUDA_TRY(cudaMemcpyAsync(leaves.data(), f.leaves.data(), (newL + 1) * sizeof(uint64_t),
                                      cudaMemcpyDeviceToHost, stream));
        SPHB_CUDA_TRY(cudaMemcpyAsync(mand.data(), g.leaves.data(), (g.numLeaves + 1) * sizeof(uint64_t),
                                      cudaMemcpyDeviceToHost, stream));
        SPHB_CUDA_TRY(cudaStreamSynchronize(stream));
        mand.push_back(0);
        mand.push_back(kRootRange);
        std::sort(mand.begin(), mand.end());
        mand.erase(std::unique(mand.begin(), mand.end()), mand.end());
        std::vector<uint64_t> span;
        for (size_t k = 0; k + 1 < mand.size(); ++k)
        {
            spanRange(mand[k], mand[k + 1], span);
        }
        span.push_back(kRootRange);
        leaves.insert(leaves.end(), span.begin(), span.end());
        std::sort(leaves.begin(), leaves.end());
        leaves.erase(std::unique(leaves.begin(), leaves.end()), leaves.end());
        newL = int(leaves.size()) - 1;
        SPHB_TRY(f.leaves.reserve(newL + 1));
        SPHB_CUDA_TRY(cudaMemcpyAsync(f.leaves.data(), leaves.data(), leaves.size() * sizeof(uint64_t),
                                      cudaMemcpyHostToDevice, stream));
        SPHB_CUDA_TRY(cudaStreamSynchronize(stream));
        f.numLeaves = newL;
    }
    SPHB_TRY(buildLinkedOctree(f.leaves.data(), f.numLeaves, f.tree, s, stream));
    *converged = conv;
    return kOk;
}

int focusUpdateCounts(FocusTree& f, const uint64_t* keys, size_t n, cudaStream_t stream, const DevBox* box)
{
    int L = f.numLeaves;
    SPHB_TRY(f.leafCounts.reserve(L));
    SPHB_TRY(f.layout.reserve(L + 1));
    if (L <= kSmallTree && n <= UINT32_MAX)
    {
        LinkedOctree& t = f.tree;
        smallCountsKernel<<<1, kSmallThreads, 0, stream>>>(
            f.leaves.data(), L, keys, n, f.leafCounts.data(), f.layout.data(), t.prefixes.data(), t.nodeToLeaf.data(),
            t.numNodes, t.nodeCounts.data(), box ? *box : DevBox{}, box ? t.centers.data() : nullptr,
            box ? t.sizes.data() : nullptr);
        countLaunch();
        SPHB_CUDA_TRY(cudaGetLastError());
        return kOk;
    }
    SPHB_TRY(computeLeafCounts(f.leaves.data(), L, keys, n, f.leafCounts.data(), stream, f.layout.data()));
    SPHB_TRY(computeNodeCounts(f.leaves.data(), f.leafCounts.data(), f.layout.data(), f.tree, stream));
    return box ? computeGeoCenters(f.tree, *box, stream) : int(kOk);
}

} // namespace sphb

// ------------------------------------------------------------------------------------------------------------------
// The converged tree of sorted keys, directly
//
// The fixed point of the rebalance steps (split leaves with more than `bucket` keys above the deepest level, merge 8
// sibling leaves with at most `bucket` together) is unique: the internal nodes are the nodes above the deepest level
// with more than `bucket` keys. Let c_p be the deepest level of a node that holds the keys p - 1 and p, and E_p that of
// a node that holds the keys p .. p + bucket (at most one above the deepest). The deepest internal node that holds key
// p is then on level D_p = max(E_p, min(D_{p-1}, c_p)), and functions x -> max(e, min(x, c)) compose, so D is a scan. The
// leaf of key p is on level D_p + 1, it starts at p if c_p <= D_p, and the empty leaves between two keys' leaves are the
// children that the paths between them pass by. A second scan, of the leaves that each key opens, places them.
// Three sweeps over the keys, a search per leaf boundary for the counts and one host read, instead of a rebalance, a
// scan, a recount and a host read for every few levels, with buffers that grew in between: 150,000 leaves of 4,000,037
// clustered keys 2.6 -> 0.2 ms.
// ------------------------------------------------------------------------------------------------------------------
namespace sphb
{
namespace
{

constexpr int kConvThreads = 256;
constexpr int kConvItems   = 8;
constexpr int kConvTile    = kConvThreads * kConvItems;

//! x -> max(e, min(x, c)) on levels -1 .. 21
struct LevelClamp
{
    int e, c;
};

__device__ __forceinline__ LevelClamp clampIdentity() { return {-1, int(kMaxLevel)}; }

//! first f, then g
__device__ __forceinline__ LevelClamp clampThen(LevelClamp f, LevelClamp g)
{
    return {max(g.e, min(f.e, g.c)), min(f.c, g.c)};
}

//! deepest level of a node that holds both keys
__device__ __forceinline__ int commonLevel(uint64_t a, uint64_t b)
{
    return a == b ? int(kMaxLevel) : (int(__clzll((long long)(a ^ b))) - 1) / 3;
}

//! the keys below the removal key (the last leaf ends there)
__device__ inline size_t keptKeys(const uint64_t* keys, size_t n) { return lowerBound(keys, n, kRootRange); }

__device__ __forceinline__ LevelClamp clampOf(const uint64_t* __restrict__ keys, size_t n, unsigned bucket, size_t p)
{
    if (p >= n) { return clampIdentity(); }
    uint64_t k = __ldg(keys + p);
    int c      = p ? commonLevel(__ldg(keys + p - 1), k) : -1;
    int e      = -1;
    if (p + bucket < n) { e = min(commonLevel(k, __ldg(keys + p + bucket)), int(kMaxLevel) - 1); }
    return {e, c};
}

//! exclusive scan of one clamp per thread over the block; *total receives the composition of all
__device__ LevelClamp blockScanClamp(LevelClamp v, LevelClamp* total)
{
    __shared__ LevelClamp warpTotal[kConvThreads / 32 + 1];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    LevelClamp incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        LevelClamp o{__shfl_up_sync(0xffffffffu, incl.e, off), __shfl_up_sync(0xffffffffu, incl.c, off)};
        if (lane >= off) { incl = clampThen(o, incl); }
    }
    if (lane == 31) { warpTotal[warp] = incl; }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        LevelClamp run = clampIdentity();
        for (int w = 0; w < kConvThreads / 32; ++w)
        {
            LevelClamp t = warpTotal[w];
            warpTotal[w] = run;
            run          = clampThen(run, t);
        }
        warpTotal[kConvThreads / 32] = run;
    }
    __syncthreads();
    LevelClamp ex{__shfl_up_sync(0xffffffffu, incl.e, 1), __shfl_up_sync(0xffffffffu, incl.c, 1)};
    if (lane == 0) { ex = clampIdentity(); }
    ex     = clampThen(warpTotal[warp], ex);
    *total = warpTotal[kConvThreads / 32];
    __syncthreads();
    return ex;
}

__global__ void __launch_bounds__(kConvThreads) convTileKernel(const uint64_t* keys, size_t n, unsigned bucket, int2* tiles)
{
    __shared__ size_t kept;
    if (threadIdx.x == 0) { kept = keptKeys(keys, n); }
    __syncthreads();
    size_t base  = size_t(blockIdx.x) * kConvTile + size_t(threadIdx.x) * kConvItems;
    LevelClamp v = clampIdentity();
#pragma unroll
    for (int q = 0; q < kConvItems; ++q)
    {
        v = clampThen(v, clampOf(keys, kept, bucket, base + q));
    }
    LevelClamp total;
    blockScanClamp(v, &total);
    if (threadIdx.x == 0) { tiles[blockIdx.x] = make_int2(total.e, total.c); }
}

//! tiles[t].x = D of the key before tile t
__global__ void __launch_bounds__(kConvThreads) convScanKernel(int2* tiles, int numTiles)
{
    LevelClamp carry = clampIdentity();
    for (int base = 0; base < numTiles; base += kConvThreads)
    {
        int t        = base + threadIdx.x;
        LevelClamp v = t < numTiles ? LevelClamp{tiles[t].x, tiles[t].y} : clampIdentity();
        LevelClamp total;
        LevelClamp ex = clampThen(carry, blockScanClamp(v, &total));
        if (t < numTiles) { tiles[t].x = max(ex.e, min(-1, ex.c)); }
        carry = clampThen(carry, total);
    }
}

//! sum of the octal digits from level lo to level hi of the key, or of 7 minus the digit
__device__ __forceinline__ int digitSum(uint64_t key, int lo, int hi, bool complement)
{
    int sum = 0;
    for (int l = lo; l <= hi; ++l)
    {
        sum += int(octalDigitAt(key, unsigned(l)));
    }
    return complement ? 7 * max(0, hi - lo + 1) - sum : sum;
}

/*! leaves that key p opens: its own, if p is the first key in it, and the empty ones before it; for p == n the empty
 *  ones after the last key. dPrev = D_{p-1}, d = D_p. */
__device__ __forceinline__ int opened(const uint64_t* __restrict__ keys, size_t n, size_t p, int dPrev, int d)
{
    if (n == 0) { return p == 0 ? 1 : 0; } // the root
    if (p == n) { return digitSum(__ldg(keys + n - 1), 1, dPrev + 1, true); }
    uint64_t k = __ldg(keys + p);
    if (p == 0) { return digitSum(k, 1, d + 1, false) + 1; }
    uint64_t o = __ldg(keys + p - 1);
    int c      = commonLevel(o, k);
    if (c > d) { return 0; }
    return digitSum(o, c + 2, dPrev + 1, true) + int(octalDigitAt(k, unsigned(c + 1))) -
           int(octalDigitAt(o, unsigned(c + 1))) + digitSum(k, c + 2, d + 1, false);
}

/*! kEmit false: sums[tile] = leaves opened by the tile's keys. kEmit true: the leaves, from the scanned sums, if all
 *  numLeaves + 1 keys fit into capacity. */
template<bool kEmit>
__global__ void __launch_bounds__(kConvThreads) convLeavesKernel(const uint64_t* __restrict__ keys, size_t nAll,
                                                                unsigned bucket, const int2* __restrict__ tiles,
                                                                int* sums, uint64_t* leaves, size_t capacity,
                                                                const int* numLeaves)
{
    __shared__ size_t kept;
    __shared__ int warpSum[kConvThreads / 32];
    if (threadIdx.x == 0) { kept = keptKeys(keys, nAll); }
    __syncthreads();
    const size_t n    = kept;
    const size_t base = size_t(blockIdx.x) * kConvTile + size_t(threadIdx.x) * kConvItems;
    LevelClamp f[kConvItems];
    LevelClamp v = clampIdentity();
#pragma unroll
    for (int q = 0; q < kConvItems; ++q)
    {
        f[q] = clampOf(keys, n, bucket, base + q);
        v    = clampThen(v, f[q]);
    }
    LevelClamp total;
    LevelClamp ex = blockScanClamp(v, &total);
    int d         = max(ex.e, min(tiles[blockIdx.x].x, ex.c));
    int dPrev[kConvItems + 1];
    int w[kConvItems];
    int sum  = 0;
    dPrev[0] = d;
#pragma unroll
    for (int q = 0; q < kConvItems; ++q)
    {
        d            = max(f[q].e, min(d, f[q].c));
        dPrev[q + 1] = d;
        w[q]         = base + q <= n ? opened(keys, n, base + q, dPrev[q], d) : 0;
        sum += w[q];
    }
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        int t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) { incl += t; }
    }
    if (lane == 31) { warpSum[warp] = incl; }
    __syncthreads();
    int before = 0, all = 0;
    for (int q = 0; q < kConvThreads / 32; ++q)
    {
        before += q < warp ? warpSum[q] : 0;
        all += warpSum[q];
    }
    if constexpr (!kEmit)
    {
        if (threadIdx.x == 0) { sums[blockIdx.x] = all; }
        return;
    }
    const int num = *numLeaves;
    if (num < 1 || size_t(num) + 1 > capacity) { return; }
    auto put = [&](int pos, uint64_t key) {
        if (pos >= 0 && pos < num) { leaves[pos] = key; } // (keys out of order place leaves anywhere)
    };
    int pos = sums[blockIdx.x] + before + incl - sum;
    for (int q = 0; q < kConvItems; ++q)
    {
        size_t p = base + q;
        if (p > n || w[q] == 0) { continue; }
        int at = pos;
        pos += w[q];
        if (n == 0)
        {
            put(0, 0);
            continue;
        }
        // children right of the previous key's path, from its leaf upwards
        uint64_t o = p ? __ldg(keys + p - 1) : 0;
        uint64_t k = p < n ? __ldg(keys + p) : 0;
        int c      = p == 0 ? -1 : p == n ? -1 : commonLevel(o, k);
        if (p > 0)
        {
            for (int l = dPrev[q] + 1; l >= c + 2 - (p == n ? 1 : 0); --l)
            {
                if (l < 1) { break; }
                uint64_t range  = nodeRangeAt(unsigned(l));
                uint64_t parent = o & ~(8 * range - 1);
                for (unsigned dig = octalDigitAt(o, unsigned(l)) + 1; dig < 8; ++dig)
                {
                    put(at++, parent + dig * range);
                }
            }
        }
        if (p == n) { continue; }
        // children left of this key's path, from the first level on which the paths differ downwards
        for (int l = max(c + 1, 1); l <= dPrev[q + 1] + 1; ++l)
        {
            uint64_t range  = nodeRangeAt(unsigned(l));
            uint64_t parent = k & ~(8 * range - 1);
            unsigned first  = l == c + 1 && p > 0 ? octalDigitAt(o, unsigned(l)) + 1 : 0;
            for (unsigned dig = first; dig < octalDigitAt(k, unsigned(l)); ++dig)
            {
                put(at++, parent + dig * range);
            }
        }
        uint64_t leafRange = nodeRangeAt(unsigned(dPrev[q + 1] + 1));
        put(at, k & ~(leafRange - 1));
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) { leaves[num] = kRootRange; }
}

} // namespace
} // namespace sphb

extern "C" int sphb_compute_octree(const uint64_t* sorted_keys, size_t n, unsigned bucket, uint64_t* leaves,
                                   uint32_t* counts, size_t capacity, size_t* num_leaves, void* stream)
{
    using namespace sphb;
    if (!num_leaves || bucket == 0 || (n && !sorted_keys)) { return SPHB_ERR_ARG; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    size_t numTiles = (n + 1 + kConvTile - 1) / kConvTile;
    // per tile: the level clamp (two ints), the leaves opened, and the scan's scratch
    DeviceBuffer<int> tmp;
    SPHB_TRY(tmp.reserve(3 * numTiles + 2 + scanTempInts(numTiles) + 1));
    int2* tiles  = reinterpret_cast<int2*>(tmp.data());
    int* sums    = tmp.data() + 2 * numTiles;
    int* scanTmp = sums + numTiles + 1;
    size_t cap   = leaves && counts ? capacity : 0;
    convTileKernel<<<unsigned(numTiles), kConvThreads, 0, st>>>(sorted_keys, n, bucket, tiles);
    convScanKernel<<<1, kConvThreads, 0, st>>>(tiles, int(numTiles));
    convLeavesKernel<false><<<unsigned(numTiles), kConvThreads, 0, st>>>(sorted_keys, n, bucket, tiles, sums, nullptr, 0,
                                                                          nullptr);
    countLaunch(3);
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_TRY(exclusiveScan(sums, sums, numTiles, scanTmp, st));
    convLeavesKernel<true><<<unsigned(numTiles), kConvThreads, 0, st>>>(sorted_keys, n, bucket, tiles, sums, leaves, cap,
                                                                         sums + numTiles);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    int num = 0;
    SPHB_TRY(readBack(st, {{&num, sums + numTiles, sizeof(int)}}));
    if (num < 1) { return SPHB_ERR_ARG; } // keys out of order
    *num_leaves = size_t(num);
    if (size_t(num) + 1 <= cap)
    {
        SPHB_TRY(computeLeafCounts(leaves, num, sorted_keys, n, counts, st));
        SPHB_CUDA_TRY(cudaStreamSynchronize(st));
    }
    return size_t(num) + 1 <= capacity ? SPHB_OK : SPHB_ERR_CAPACITY;
}

// ------------------------------------------------------------------------------------------------------------------
// The linked octree in the reference's OctreeData layout (cstone/tree/octree.hpp:283-358)
// ------------------------------------------------------------------------------------------------------------------
namespace sphb
{
namespace
{

//! digitWeight of the reference's binary-radix to octree index map (cstone/sfc/common.hpp:318-322)
__device__ __forceinline__ int refDigitWeight(int digit)
{
    int fourGeqMask = -int(digit >= 4);
    return ((7 - digit) & fourGeqMask) - (digit & ~fourGeqMask);
}

/*! internalToLeaf / leafToInternal in the reference's unsorted-index convention (createUnsortedLayoutCpu,
 *  octree.hpp:77-99 and buildOctreeCpu, :170-196): the unsorted index of leaf l is numInternal + l, that of the
 *  internal node found at leaf boundary tid (common prefix a multiple of 3 bits) is
 *  (tid + binaryKeyWeight(key, level)) / 7; internalToLeaf[sorted] = unsorted - numInternal,
 *  leafToInternal[unsorted] = sorted. */
__global__ void refNodeMapKernel(const uint64_t* leaves, int numLeaves, int numInternal, const uint64_t* prefixes,
                                 int numNodes, const int* leafToNode, int* internalToLeaf, int* leafToInternal)
{
    int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= numLeaves) { return; }
    int sortedLeaf                       = leafToNode[tid];
    internalToLeaf[sortedLeaf]           = tid;
    leafToInternal[numInternal + tid]    = sortedLeaf;
    if (tid >= numLeaves - 1) { return; }
    uint64_t key     = leaves[tid];
    int prefixLength = int(__clzll(key ^ leaves[tid + 1])) - 1;
    if (prefixLength % 3 != 0) { return; }
    int level  = prefixLength / 3;
    int weight = 0;
    for (int l = 1; l <= level + 1; ++l)
    {
        weight += refDigitWeight(int((key >> (3 * (int(kMaxLevel) - l))) & 7u));
    }
    int octIndex    = (tid + weight) / 7;
    uint64_t prefix = (uint64_t(1) << prefixLength) | (key >> (3 * int(kMaxLevel) - prefixLength));
    // sorted position of this internal node: prefixes are unique and sorted
    int lo = 0, hi = numNodes;
    while (lo < hi)
    {
        int mid = (lo + hi) >> 1;
        if (prefixes[mid] < prefix) { lo = mid + 1; }
        else { hi = mid; }
    }
    internalToLeaf[lo]       = octIndex - numInternal;
    leafToInternal[octIndex] = lo;
}

} // namespace
} // namespace sphb

extern "C" int sphb_build_octree(const uint64_t* leaves, size_t num_leaves, uint64_t* prefixes, int* child_offsets,
                                 int* parents, int* level_range, int* internal_to_leaf, int* leaf_to_internal,
                                 void* stream)
{
    using namespace sphb;
    if (!leaves || num_leaves == 0 || num_leaves >= (size_t(1) << 30) || !prefixes || !child_offsets || !parents ||
        !level_range || !internal_to_leaf || !leaf_to_internal)
    {
        return SPHB_ERR_ARG;
    }
    auto st = static_cast<cudaStream_t>(stream);
    LinkedOctree t;
    TreeScratch sc;
    SPHB_TRY(buildLinkedOctree(leaves, int(num_leaves), t, sc, st));
    int nn = t.numNodes;
    SPHB_CUDA_TRY(cudaMemcpyAsync(prefixes, t.prefixes.data(), nn * sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
    SPHB_CUDA_TRY(cudaMemcpyAsync(child_offsets, t.childOffsets.data(), nn * sizeof(int), cudaMemcpyDeviceToDevice,
                                  st));
    SPHB_CUDA_TRY(cudaMemcpyAsync(parents, t.parents.data(), std::max(1, (nn - 1) / 8) * sizeof(int),
                                  cudaMemcpyDeviceToDevice, st));
    refNodeMapKernel<<<ceilDiv(num_leaves, 256), 256, 0, st>>>(leaves, t.numLeaves, t.numInternal, t.prefixes.data(),
                                                                 nn, t.leafToNode.data(), internal_to_leaf,
                                                                 leaf_to_internal);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_CUDA_TRY(cudaStreamSynchronize(st));
    SPHB_CUDA_TRY(
        cudaMemcpy(level_range, t.levelRangeD.data(), (kMaxLevel + 2) * sizeof(int), cudaMemcpyDeviceToHost));
    return SPHB_OK;
}

// ------------------------------------------------------------------------------------------------------------------
// One step of the multi-rank global tree: the caller sums the leaf counts of every rank between the steps
// (cstone::updateOctreeGlobal, cstone/tree/update_mpi.hpp:64-99)
// ------------------------------------------------------------------------------------------------------------------

extern "C" int sphb_leaf_counts(const uint64_t* leaves, size_t num_leaves, const uint64_t* sorted_keys, size_t n,
                                uint32_t* counts, void* stream)
{
    using namespace sphb;
    if (!leaves || !counts || num_leaves == 0 || num_leaves >= (size_t(1) << 30) || (n && !sorted_keys))
    {
        return SPHB_ERR_ARG;
    }
    return computeLeafCounts(leaves, int(num_leaves), sorted_keys, n, counts, static_cast<cudaStream_t>(stream));
}

extern "C" int sphb_rebalance_tree(const uint64_t* leaves, size_t num_leaves, const uint32_t* counts, unsigned bucket,
                                   uint64_t* new_leaves, size_t capacity, size_t* num_new, int* converged,
                                   void* stream)
{
    using namespace sphb;
    if (!leaves || !counts || !new_leaves || !num_new || !converged || bucket == 0 || num_leaves == 0 ||
        num_leaves >= (size_t(1) << 30) || new_leaves == leaves)
    {
        return SPHB_ERR_ARG;
    }
    auto st = static_cast<cudaStream_t>(stream);
    int L   = int(num_leaves);
    TreeScratch s;
    SPHB_TRY(s.ints.reserve(L + 2));
    SPHB_TRY(s.scanTmp.reserve(scanTempInts(L + 1) + 1));
    SPHB_TRY(s.flags.reserve(1));
    SPHB_CUDA_TRY(cudaMemsetAsync(s.flags.data(), 0, sizeof(unsigned), st));
    csNodeOpsKernel<<<ceilDiv(L + 1, 256), 256, 0, st>>>(leaves, counts, L, bucket, s.ints.data(), s.flags.data());
    countLaunch();
    SPHB_TRY(exclusiveScan(s.ints.data(), s.ints.data(), L + 1, s.scanTmp.data(), st));
    int newL       = 0;
    unsigned anyOp = 0;
    SPHB_TRY(readBack(st, {{&newL, s.ints.data() + L, sizeof(int)}, {&anyOp, s.flags.data(), sizeof(unsigned)}}));
    *num_new   = size_t(newL);
    *converged = anyOp ? 0 : 1;
    if (size_t(newL) + 1 > capacity) { return SPHB_ERR_CAPACITY; }
    rebalanceKernel<<<ceilDiv(L + 1, 256), 256, 0, st>>>(leaves, L, s.ints.data(), new_leaves);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_CUDA_TRY(cudaStreamSynchronize(st));
    return SPHB_OK;
}
