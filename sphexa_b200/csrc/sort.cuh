// Radix sort interface (see sort.cu).
#pragma once

#include "common.cuh"

namespace sphb
{

size_t sortScratchBytes(size_t n);

//! stable in-place sort of (key, value) pairs; values set to 0..n-1 first if initValues
int sortByKey(uint64_t* keys, uint32_t* values, size_t n, bool initValues, void* scratch, size_t scratchBytes,
              cudaStream_t stream);

/*! The same stable sort for keys that are nearly in order (the previous step's order of slowly moving particles):
 *  values are set to 0..n-1; if no adjacent pair is out of order, nothing moves and *identity is set; otherwise the
 *  tiles that hold inversions are sorted in shared memory (two overlapping tilings), and the full radix sort runs
 *  only if that left any inversion. The result equals sortByKey's. */
int sortNearlySorted(uint64_t* keys, uint32_t* values, size_t n, void* scratch, size_t scratchBytes, bool* identity,
                     cudaStream_t stream);

//! where sortByLeaves left the sorted keys
enum class LeafSort
{
    identity, // the keys were in order already
    inPlace,  // in keys
    keysOut   // in keysOut
};

//! entries of LeafSortScratch::first for so many buckets (the leaves and one for the keys past the last leaf)
size_t leafSortInts(size_t numBuckets);

//! device buffers of sortByLeaves
struct LeafSortScratch
{
    DeviceBuffer<uint2> slot;
    DeviceBuffer<int> first;
    DeviceBuffer<int> scanTmp;
};

/*! The same stable sort (values = 0..n-1 first) with the help of a cornerstone leaf array that held few keys per leaf
 *  for keys close to these, the tree of the previous step: every key finds its leaf, a scan of the leaf counts places
 *  the leaves, and one warp sorts each leaf, a block one of more than 128 keys. One host read, of whether anything is out
 *  of order and whether a leaf grew past 2,048 keys (then the radix sort runs, in place). It reads and writes the keys
 *  twice whatever the particles' motion is, where the radix sort takes four passes of that, eight if the keys crowd. */
int sortByLeaves(uint64_t* keys, uint64_t* keysOut, uint32_t* values, size_t n, const uint64_t* leaves, int numLeaves,
                 LeafSortScratch& ls, void* scratch, size_t scratchBytes, LeafSort* result, cudaStream_t stream);

/*! The same sort without any host synchronisation (stream-capturable): runs exactly the passes of passMask (bit p
 *  = byte p of the key, from the least significant) and ORs a look-back timeout into *errorOut (device) if set. */
int sortByKeyAsync(uint64_t* keys, uint32_t* values, size_t n, bool initValues, void* scratch, size_t scratchBytes,
                   unsigned passMask, uint32_t* errorOut, cudaStream_t stream, const uint32_t* gate = nullptr);

//! most keys of sortShortKeysAsync
constexpr size_t kSortShortMax = 16384;

/*! stable sort of up to kSortShortMax keys below 2^32 with their values by one block, without scratch: one launch instead
 *  of a histogram and a launch and two memsets per digit, each of them latency at this size. The time steps of the
 *  groups of a block time step: the rungs and the integration of 64^3 particles take 144 us per substep instead of 185. */
int sortShortKeysAsync(uint64_t* keys, uint32_t* values, size_t n, cudaStream_t stream);

//! one cornerstone leaf array among several: its leaves are the buckets bucket0 .. bucket0 + numLeaves - 1, and the
//! bucket after them takes the keys past the last leaf
struct LeafSet
{
    const uint64_t* leaves;
    int numLeaves;
    uint32_t bucket0;
};

/*! sortByLeaves for an array of contiguous segments (seg[i] ascending; sets[k] the leaves of segment k, numBuckets
 *  buckets over all segments), without any host synchronisation. values = 0..n-1, then the stable order by (segment,
 *  key) and the keys in it in keysOut; if a bucket grew past 2,048 keys, **overflow (device) is not 0 and only values =
 *  0..n-1 was written. The buffers of ls must be large enough beforehand (slot n, first leafSortInts(numBuckets), scanTmp
 *  scanTempInts(numBuckets) + 1). */
int sortSegmentsByLeavesAsync(const uint64_t* keys, uint64_t* keysOut, uint32_t* values, size_t n, const uint64_t* seg,
                              const LeafSet* sets, size_t numBuckets, LeafSortScratch& ls, void* scratch,
                              size_t scratchBytes, const unsigned** overflow, cudaStream_t stream);

} // namespace sphb
