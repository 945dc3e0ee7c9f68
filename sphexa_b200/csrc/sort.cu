// Stable LSD radix sort of (uint64 key, uint32 value) pairs: one histogram sweep for all digits, then one
// "onesweep" pass per 8-bit digit in which each tile ranks its keys, resolves its global digit offsets through a
// decoupled look-back over the preceding tiles, and scatters. Passes whose digit is identical for every key are
// skipped. Replaces the reference's CUB DeviceRadixSort::SortPairs (cstone/primitives/primitives_gpu.cu:308-339).
//
// Tile = 8 warps x 16 keys x 32 lanes = 4096 keys. Within a warp, key k of lane l is element warpBase + k*32 + l, and
// ranking walks k then l, so ranks follow input order (stability). The look-back status word per (tile, digit) is
// 32 bits: 2 flag bits (0 = empty, 1 = tile aggregate, 2 = inclusive prefix) and a 30-bit count, so n < 2^30.
// Every spin on a predecessor's status is bounded; on timeout the pass records an error word that the host reads.
#include <mutex>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "primitives.cuh"
#include "sort.cuh"

namespace sphb
{

namespace
{

constexpr int kRadixBits   = 8;
constexpr int kRadix       = 1 << kRadixBits;
constexpr int kSortWarps   = 8;
constexpr int kSortThreads = kSortWarps * kWarp;
constexpr int kItems       = 16;
constexpr int kTile        = kSortThreads * kItems;
constexpr int kPasses      = 8;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kValMask = (1u << 30) - 1;
constexpr long kSpinLimit   = 1L << 24;

struct SortScratch
{
    uint64_t* keysAlt;
    uint32_t* valsAlt;
    uint32_t* hist;       // [kPasses][kRadix] counts, then exclusive offsets
    uint32_t* status;     // [numTiles][kRadix], directly behind hist
    uint32_t* counters;   // [0] tile counter, [1] error word, [2] longRunsKernel's flag, [3] runs that sortRunsKernel listed
};

size_t alignUp(size_t x, size_t a) { return (x + a - 1) / a * a; }

size_t numTilesOf(size_t n) { return (n + kTile - 1) / kTile; }

SortScratch carve(void* base, size_t n)
{
    char* p = static_cast<char*>(base);
    SortScratch s;
    s.keysAlt = reinterpret_cast<uint64_t*>(p);
    p += alignUp(n * sizeof(uint64_t), 256);
    s.valsAlt = reinterpret_cast<uint32_t*>(p);
    p += alignUp(n * sizeof(uint32_t), 256);
    s.hist = reinterpret_cast<uint32_t*>(p);
    p += alignUp(kPasses * kRadix * sizeof(uint32_t), 256);
    s.status = reinterpret_cast<uint32_t*>(p);
    p += alignUp(numTilesOf(n) * kRadix * sizeof(uint32_t), 256);
    s.counters = reinterpret_cast<uint32_t*>(p);
    return s;
}

//! keys of equal upper bits that one thread puts in order, and those that a block sorts
constexpr int kRunCap      = 32;
constexpr int kRunBlockCap = 2048;

//! passes on the upper digits before the runs are looked at: 32 bits tell nearly all of 2^30 spread keys apart
constexpr int kUpperPasses = 4;

constexpr int kHistThreads = 1024;
constexpr int kSamples     = 4096;
constexpr int kSampleSlots = 2 * kSamples;

/*! *crowded = 1 if many keys probably lie in runs that no block sorts, else 0: counts the samples (spread evenly,
 *  up to kSamples) that agree in the upper digits with an earlier, different one. A hash table holds 8 bits of a fingerprint, the
 *  first sample and the count of each. A run of kRunBlockCap keys holds kRunBlockCap samples / n of them; three of spread
 *  keys hardly ever agree. Equal keys, which are in order, do not count. The upper digits are the kUpperPasses highest
 *  ones in which the samples differ. By one block of kHistThreads. */
__device__ void sampleRuns(const uint64_t* __restrict__ keys, size_t n, uint32_t* slots, uint32_t* crowded)
{
    __shared__ uint32_t differ; // the digits in which the samples differ
    if (threadIdx.x == 0) { differ = 0; }
    // one a thread serves few keys as well
    const size_t samples = min(min(n, size_t(kSamples)), max(n / 32, size_t(kHistThreads)));
    uint64_t key[kSamples / kHistThreads];
#pragma unroll
    for (int r = 0; r < kSamples / kHistThreads; ++r)
    {
        size_t q = threadIdx.x + size_t(r) * kHistThreads;
        key[r]   = __ldg(keys + (q < samples ? n * q / samples : 0));
    }
    for (int t = threadIdx.x; t < kSampleSlots; t += kHistThreads)
    {
        slots[t] = 0;
    }
    __syncthreads();
    uint64_t bits = 0;
#pragma unroll
    for (int r = 0; r < kSamples / kHistThreads; ++r)
    {
        bits |= key[r] ^ __ldg(keys);
    }
    uint32_t mine = 0;
#pragma unroll
    for (int p = 0; p < kPasses; ++p)
    {
        mine |= ((bits >> (p * kRadixBits)) & (kRadix - 1)) ? 1u << p : 0u;
    }
    mine = __reduce_or_sync(0xffffffffu, mine);
    if ((threadIdx.x & (kWarp - 1)) == 0) { atomicOr(&differ, mine); }
    __syncthreads();
    uint32_t upper = differ;
    while (__popc(upper) > kUpperPasses)
    {
        upper &= upper - 1;
    }
    const int shift    = upper ? (__ffs(upper) - 1) * kRadixBits : 0;
    const size_t limit = max(size_t(3), size_t(kRunBlockCap) * samples * 3 / (4 * n));
    unsigned most      = 0;
#pragma unroll
    for (int r = 0; r < kSamples / kHistThreads; ++r)
    {
        if (threadIdx.x + size_t(r) * kHistThreads >= samples) { continue; }
        uint64_t h = (key[r] >> shift) * 0x9E3779B97F4A7C15ull; // multiplicative hashing (golden ratio)
        h ^= h >> 29;
        const uint32_t self = threadIdx.x + r * kHistThreads;
        const uint32_t word = (uint32_t(h >> 32) & 0xff000000u) | (self << 12) | 1u;
        for (uint32_t at = uint32_t(h >> 40) % kSampleSlots;; at = (at + 1) % kSampleSlots)
        {
            uint32_t old = atomicCAS(&slots[at], 0u, word);
            if (old == 0) { break; }
            if ((old ^ word) >> 24) { continue; }
            // kSamples / 2 are enough for any limit, and no count reaches the sample's bits
            bool equal = __ldg(keys + n * ((old >> 12) & 0xfffu) / samples) == key[r];
            if (!equal && (old & 0xfffu) < kSamples / 2) { most = max(most, (atomicAdd(&slots[at], 1u) & 0xfffu) + 1u); }
            break;
        }
    }
    bool many = __syncthreads_or(most >= limit);
    if (threadIdx.x == 0) { *crowded = many ? 1u : 0u; }
}

//! digit histograms of all 8 byte positions in one sweep over the keys; with crowded set, the first block takes a sample
//! instead (sampleRuns), which costs nothing beside the sweep
__global__ void __launch_bounds__(kHistThreads) histogramKernel(const uint64_t* __restrict__ keys, size_t n,
                                                                uint32_t* __restrict__ hist, const uint32_t* gate,
                                                                uint32_t* crowded = nullptr)
{
    if (gate && *gate == 0) { return; }
    __shared__ uint32_t sh[kSampleSlots];
    const unsigned blocks = crowded ? gridDim.x - 1 : gridDim.x;
    const unsigned block  = crowded ? blockIdx.x - 1 : blockIdx.x;
    if (crowded && blockIdx.x == 0)
    {
        sampleRuns(keys, n, sh, crowded);
        return;
    }
    for (int t = threadIdx.x; t < kPasses * kRadix; t += kHistThreads)
    {
        sh[t] = 0;
    }
    __syncthreads();
    for (size_t i = block * size_t(kHistThreads) + threadIdx.x; i < n; i += size_t(blocks) * kHistThreads)
    {
        uint64_t k = keys[i];
#pragma unroll
        for (int p = 0; p < kPasses; ++p)
        {
            atomicAdd(&sh[p * kRadix + ((k >> (p * kRadixBits)) & (kRadix - 1))], 1u);
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kPasses * kRadix; t += kHistThreads)
    {
        uint32_t c = sh[t];
        if (c) { atomicAdd(hist + t, c); }
    }
}

unsigned histogramBlocks(size_t n) { return unsigned(std::min<size_t>(ceilDiv(n, 4 * kHistThreads), size_t(smCount()) * 2)); }

//! exclusive scan of each pass's 256 digit counts, in place (one block per pass)
__global__ void histScanKernel(uint32_t* hist, const uint32_t* gate)
{
    if (gate && *gate == 0) { return; }
    __shared__ uint32_t sh[kRadix];
    uint32_t* h = hist + blockIdx.x * kRadix;
    int t       = threadIdx.x;
    uint32_t v  = h[t];
    sh[t]       = v;
    __syncthreads();
    for (int off = 1; off < kRadix; off <<= 1)
    {
        uint32_t add = t >= off ? sh[t - off] : 0;
        __syncthreads();
        sh[t] += add;
        __syncthreads();
    }
    h[t] = sh[t] - v;
}

__global__ void iotaKernel(uint32_t* v, size_t n)
{
    size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i < n) { v[i] = uint32_t(i); }
}

//! *count += number of adjacent pairs with keys[i] > keys[i + 1] (one atomic per block)
__global__ void __launch_bounds__(256) inversionsKernel(const uint64_t* __restrict__ keys, size_t n,
                                                        uint32_t* count)
{
    uint32_t c = 0;
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i + 1 < n; i += size_t(gridDim.x) * blockDim.x)
    {
        c += keys[i] > keys[i + 1] ? 1u : 0u;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    __shared__ uint32_t warpSum[8];
    if ((threadIdx.x & 31) == 0) { warpSum[threadIdx.x >> 5] = c; }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        uint32_t s = 0;
        for (int w = 0; w < 8; ++w)
        {
            s += warpSum[w];
        }
        if (s) { atomicAdd(count, s); }
    }
}

constexpr int kRepairTile    = 2048;
constexpr int kRepairThreads = 256;

/*! Stable sort of one tile of (key, value) pairs in shared memory, tile t covering [offset + t T, offset + (t+1) T),
 *  skipped when the tile and its left neighbour pair are already in order. Bitonic network on (key, position in the
 *  tile), so equal keys keep their order; positions past n are padded with the largest key. */
__global__ void __launch_bounds__(kRepairThreads) repairTilesKernel(uint64_t* keys, uint32_t* vals, size_t n,
                                                                   size_t offset)
{
    __shared__ uint64_t sk[kRepairTile];
    __shared__ uint32_t sv[kRepairTile];
    __shared__ uint16_t sp[kRepairTile];
    size_t t0 = offset + size_t(blockIdx.x) * kRepairTile;
    if (t0 >= n) { return; }
    size_t len = min(size_t(kRepairTile), n - t0);
    bool d     = false;
    for (size_t q = threadIdx.x; q + 1 < len; q += kRepairThreads)
    {
        d = d || keys[t0 + q] > keys[t0 + q + 1];
    }
    if (__syncthreads_or(d) == 0) { return; }
    for (int q = threadIdx.x; q < kRepairTile; q += kRepairThreads)
    {
        bool in = size_t(q) < len;
        sk[q]   = in ? keys[t0 + q] : ~uint64_t(0);
        sv[q]   = in ? vals[t0 + q] : 0u;
        sp[q]   = uint16_t(q);
    }
    __syncthreads();
    for (int size = 2; size <= kRepairTile; size <<= 1)
    {
        for (int stride = size >> 1; stride > 0; stride >>= 1)
        {
            for (int q = threadIdx.x; q < kRepairTile; q += kRepairThreads)
            {
                int p = q ^ stride;
                if (p > q)
                {
                    bool up      = (q & size) == 0;
                    bool greater = sk[q] > sk[p] || (sk[q] == sk[p] && sp[q] > sp[p]);
                    if (greater == up)
                    {
                        uint64_t k = sk[q];
                        sk[q]      = sk[p];
                        sk[p]      = k;
                        uint32_t v = sv[q];
                        sv[q]      = sv[p];
                        sv[p]      = v;
                        uint16_t o = sp[q];
                        sp[q]      = sp[p];
                        sp[p]      = o;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (size_t q = threadIdx.x; q < len; q += kRepairThreads)
    {
        keys[t0 + q] = sk[q];
        vals[t0 + q] = sv[q];
    }
}

/*! One onesweep pass over bits [shift, shift+8).
 *
 * Shared memory: per-warp digit counters (8 x 256), the tile's exclusive digit prefix (256) and the tile index.
 */
__global__ void __launch_bounds__(kSortThreads) onesweepKernel(const uint64_t* __restrict__ keysIn,
                                                               const uint32_t* __restrict__ valsIn,
                                                               uint64_t* __restrict__ keysOut,
                                                               uint32_t* __restrict__ valsOut, size_t n, int shift,
                                                               const uint32_t* __restrict__ digitOffsets,
                                                               uint32_t* status, uint32_t* counters,
                                                               const uint32_t* gate)
{
    if (gate && *gate == 0) { return; } // the whole pass is skipped: no tile waits on another
    __shared__ uint32_t warpCount[kSortWarps][kRadix];
    __shared__ uint32_t tilePrefix[kRadix];
    __shared__ uint32_t tileIdxSh;

    const int lane = threadIdx.x & (kWarp - 1);
    const int warp = threadIdx.x / kWarp;

    if (threadIdx.x == 0) { tileIdxSh = atomicAdd(counters, 1u); }
    for (int t = threadIdx.x; t < kSortWarps * kRadix; t += kSortThreads)
    {
        (&warpCount[0][0])[t] = 0;
    }
    __syncthreads();
    const size_t tile     = tileIdxSh;
    const size_t tileBase = tile * kTile;
    const size_t warpBase = tileBase + size_t(warp) * kItems * kWarp;

    uint64_t key[kItems];
    uint32_t val[kItems];
    uint32_t rank[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k)
    {
        size_t idx = warpBase + size_t(k) * kWarp + lane;
        bool valid = idx < n;
        key[k]     = valid ? keysIn[idx] : ~uint64_t(0);
        val[k]     = valid ? valsIn[idx] : 0u;
    }

    // warp-local stable ranking: peers with equal digits are found with match.any
#pragma unroll
    for (int k = 0; k < kItems; ++k)
    {
        size_t idx      = warpBase + size_t(k) * kWarp + lane;
        bool valid      = idx < n;
        uint32_t digit  = uint32_t(key[k] >> shift) & (kRadix - 1);
        uint32_t active = __ballot_sync(0xffffffffu, valid);
        uint32_t peers  = __match_any_sync(0xffffffffu, valid ? digit : 0xffffffffu);
        peers &= active;
        uint32_t before = 0;
        if (valid)
        {
            before = warpCount[warp][digit];
        }
        __syncwarp();
        if (valid)
        {
            uint32_t lowerPeers = peers & ((1u << lane) - 1u);
            rank[k]             = before + __popc(lowerPeers);
            if (lowerPeers == 0) { warpCount[warp][digit] = before + __popc(peers); }
        }
        __syncwarp();
    }
    __syncthreads();

    // per digit: exclusive scan over warps, tile total, then look-back across tiles (thread t owns digit t)
    {
        const int d    = threadIdx.x;
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w)
        {
            uint32_t c     = warpCount[w][d];
            warpCount[w][d] = total;
            total += c;
        }
        uint32_t* myStatus = status + tile * kRadix + d;
        if (tile == 0) { atomicExch(myStatus, kFlagInc | total); }
        else { atomicExch(myStatus, kFlagAgg | total); }
        __threadfence();

        uint32_t exclusive = 0;
        if (tile > 0)
        {
            long pred = long(tile) - 1;
            long spins = 0;
            while (pred >= 0)
            {
                uint32_t s = *((volatile uint32_t*)(status + size_t(pred) * kRadix + d));
                uint32_t flag = s & ~kValMask;
                if (flag == 0)
                {
                    if (++spins > kSpinLimit)
                    {
                        atomicExch(counters + 1, 1u);
                        break;
                    }
                    __nanosleep(32);
                    continue;
                }
                exclusive += s & kValMask;
                if (flag == kFlagInc) { break; }
                --pred;
            }
            atomicExch(myStatus, kFlagInc | ((exclusive + total) & kValMask));
        }
        tilePrefix[d] = digitOffsets[d] + exclusive;
    }
    __syncthreads();

#pragma unroll
    for (int k = 0; k < kItems; ++k)
    {
        size_t idx = warpBase + size_t(k) * kWarp + lane;
        if (idx < n)
        {
            uint32_t digit = uint32_t(key[k] >> shift) & (kRadix - 1);
            uint32_t pos   = tilePrefix[digit] + warpCount[warp][digit] + rank[k];
            if (pos < n)
            {
                keysOut[pos] = key[k];
                valsOut[pos] = val[k];
            }
            else { atomicExch(counters + 1, 2u); } // inconsistent offsets: report instead of writing
        }
    }
}

} // namespace

size_t sortScratchBytes(size_t n)
{
    return alignUp(n * sizeof(uint64_t), 256) + alignUp(n * sizeof(uint32_t), 256) +
           alignUp(kPasses * kRadix * sizeof(uint32_t), 256) + alignUp(numTilesOf(n) * kRadix * sizeof(uint32_t), 256) +
           256;
}

namespace
{
int runPasses(uint64_t* keys, uint32_t* values, size_t n, const SortScratch& s, unsigned passMask,
              cudaStream_t stream, const uint32_t* gate = nullptr);

__global__ void orErrorKernel(const uint32_t* err, uint32_t* out)
{
    if (*err) { atomicOr(out, 1u); }
}
} // namespace

namespace
{

//! one past the last of the keys in [i, end) whose upper bits are those of key i
__device__ __forceinline__ size_t runEnd(const uint64_t* keys, size_t i, size_t end, int shift)
{
    uint64_t up = keys[i] >> shift;
    while (end - i > 1)
    {
        size_t mid = i + (end - i) / 2;
        if ((keys[mid] >> shift) == up) { i = mid; }
        else { end = mid; }
    }
    return end;
}

//! the first of the keys in [begin, i] whose upper bits are those of key i
__device__ __forceinline__ size_t runBegin(const uint64_t* keys, size_t begin, size_t i, int shift)
{
    uint64_t up = keys[i] >> shift;
    while (i > begin)
    {
        size_t mid = begin + (i - begin) / 2;
        if ((keys[mid] >> shift) == up) { i = mid; }
        else { begin = mid + 1; }
    }
    return i;
}

/*! After a stable sort by the bits from `shift` up, sets *flag if a run of more than kRunBlockCap keys of equal upper bits
 *  is out of order. */
__global__ void __launch_bounds__(256) longRunsKernel(const uint64_t* __restrict__ keys, size_t n, int shift,
                                                      uint32_t* flag)
{
    size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x + 1;
    if (i >= n || keys[i] >= keys[i - 1]) { return; }
    uint64_t up = keys[i] >> shift;
    bool back   = i >= size_t(kRunCap) && (keys[i - kRunCap] >> shift) == up;
    bool ahead  = i + kRunCap < n && (keys[i + kRunCap] >> shift) == up;
    if (!back && !ahead) { return; }
    size_t b = runBegin(keys, i > size_t(kRunBlockCap) ? i - kRunBlockCap : 0, i, shift);
    size_t e = runEnd(keys, i, min(n, i + kRunBlockCap + 1), shift);
    if (e - b > size_t(kRunBlockCap)) { *flag = 1u; }
}

/*! the thread of the first key of every run of equal upper bits sorts the run by insertion, stably, or lists it (counters
 *  [3], list) for runBlockKernel: after longRunsKernel, which leaves no larger one out of order (counters[2] clear) */
__global__ void __launch_bounds__(256) sortRunsKernel(uint64_t* keys, uint32_t* values, size_t n, int shift,
                                                      uint32_t* counters, uint32_t* list)
{
    size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i + 1 >= n || counters[2]) { return; }
    uint64_t up = keys[i] >> shift;
    if ((keys[i + 1] >> shift) != up || (i > 0 && (keys[i - 1] >> shift) == up)) { return; }
    if (i + kRunCap < n && (keys[i + kRunCap] >> shift) == up)
    {
        list[atomicAdd(counters + 3, 1u)] = uint32_t(i); // at most n / (kRunCap + 1) of them
        return;
    }
    for (size_t a = i + 1; a < n && a - i < size_t(kRunCap); ++a)
    {
        uint64_t k = keys[a];
        if ((k >> shift) != up) { return; }
        if (k >= keys[a - 1]) { continue; }
        uint32_t v = values[a];
        size_t b   = a;
        for (; b > i && keys[b - 1] > k; --b)
        {
            keys[b]   = keys[b - 1];
            values[b] = values[b - 1];
        }
        keys[b]   = k;
        values[b] = v;
    }
}

constexpr int kRunBlockThreads = 256;

//! bitonic network over elements 0 .. width - 1 (a power of two) by one block; exchange(q, p, up) puts the pair q < p in
//! ascending (up) or descending order
template<int kThreads, class F>
__device__ __forceinline__ void blockBitonic(int width, F&& exchange)
{
    for (int size = 2; size <= width; size <<= 1)
    {
        for (int stride = size >> 1; stride > 0; stride >>= 1)
        {
            // pair t of the stage: its lower element has a zero at the stride's bit
            for (int t = threadIdx.x; t < width / 2; t += kThreads)
            {
                int q = 2 * t - (t & (stride - 1));
                exchange(q, q + stride, (q & size) == 0);
            }
            __syncthreads();
        }
    }
}

/*! one block per listed run (longer ones than kRunBlockCap are in order): its open lower bits, at most 32, with the
 *  position behind them, so that equal keys keep their order */
__global__ void __launch_bounds__(kRunBlockThreads) runBlockKernel(uint64_t* keys, uint32_t* values, size_t n, int shift,
                                                                   const uint32_t* counters, const uint32_t* list)
{
    __shared__ uint64_t v[kRunBlockCap];
    if (counters[2]) { return; }
    const unsigned num      = counters[3];
    const uint64_t openBits = (uint64_t(1) << shift) - 1;
    for (unsigned l = blockIdx.x; l < num; l += gridDim.x)
    {
        const size_t b = list[l];
        const size_t e = runEnd(keys, b, min(n, b + kRunBlockCap + 1), shift);
        const int m    = int(e - b);
        if (m > kRunBlockCap) { continue; }
        const uint64_t up = keys[b] & ~openBits;
        int width         = 64;
        while (width < m)
        {
            width <<= 1;
        }
        for (int t = threadIdx.x; t < width; t += kRunBlockThreads)
        {
            v[t] = t < m ? ((keys[b + t] & openBits) << 11) | uint64_t(t) : ~uint64_t(0);
        }
        __syncthreads();
        bool disorder = false;
        for (int t = threadIdx.x; t + 1 < m; t += kRunBlockThreads)
        {
            disorder = disorder || v[t] > v[t + 1];
        }
        if (!__syncthreads_or(disorder)) { continue; }
        blockBitonic<kRunBlockThreads>(width, [&](int q, int p, bool ascending) {
            uint64_t x = v[q], y = v[p];
            if ((x > y) == ascending)
            {
                v[q] = y;
                v[p] = x;
            }
        });
        uint32_t val[kRunBlockCap / kRunBlockThreads];
#pragma unroll
        for (int r = 0; r < kRunBlockCap / kRunBlockThreads; ++r)
        {
            int t  = threadIdx.x + r * kRunBlockThreads;
            val[r] = t < m ? values[b + (v[t] & (kRunBlockCap - 1))] : 0u;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRunBlockCap / kRunBlockThreads; ++r)
        {
            int t = threadIdx.x + r * kRunBlockThreads;
            if (t < m)
            {
                keys[b + t]   = up | (v[t] >> 11);
                values[b + t] = val[r];
            }
        }
        __syncthreads();
    }
}

} // namespace

int sortByKey(uint64_t* keys, uint32_t* values, size_t n, bool initValues, void* scratch, size_t scratchBytes,
              cudaStream_t stream)
{
    if (n == 0) { return kOk; }
    if (n >= (size_t(1) << 30)) { return kErrArg; }
    if (!scratch || scratchBytes < sortScratchBytes(n)) { return kErrCapacity; }
    SortScratch s = carve(scratch, n);

    if (initValues)
    {
        iotaKernel<<<ceilDiv(n, 256), 256, 0, stream>>>(values, n);
        SPHB_CUDA_TRY(cudaGetLastError());
    }

    SPHB_CUDA_TRY(cudaMemsetAsync(s.hist, 0, kPasses * kRadix * sizeof(uint32_t), stream));
    unsigned histBlocks = histogramBlocks(n);
    const bool sample = n > size_t(kRunBlockCap);
    histogramKernel<<<histBlocks + (sample ? 1 : 0), kHistThreads, 0, stream>>>(keys, n, s.hist, nullptr,
                                                                                sample ? s.status : nullptr);
    SPHB_CUDA_TRY(cudaGetLastError());

    // decide on the host which passes are trivial (one digit holds every key); the word behind tells the sample's finding
    uint32_t h[kPasses * kRadix + 1];
    SPHB_CUDA_TRY(cudaMemcpyAsync(h, s.hist, sizeof(h), cudaMemcpyDeviceToHost, stream));
    SPHB_CUDA_TRY(cudaStreamSynchronize(stream));
    bool doPass[kPasses];
    for (int p = 0; p < kPasses; ++p)
    {
        doPass[p] = true;
        for (int d = 0; d < kRadix; ++d)
        {
            if (h[p * kRadix + d] == n) { doPass[p] = false; }
        }
    }

    unsigned mask = 0;
    for (int p = 0; p < kPasses; ++p)
    {
        mask |= doPass[p] ? (1u << p) : 0u;
    }
    // Space-filling-curve keys differ in all eight digits, but few agree in the upper four: half the passes and a sort of
    // the runs that do, by a thread (up to 32 keys) or a block (up to 2,048). Keys of which many lie in longer runs are
    // told by a sample beforehand and take all eight passes. Where the sample missed a long run that is out of order, they
    // follow the four; they are stable, as what came before, so the result is the same.
    // 4,000,037 keys, us, eight passes / this: spread 857 / 502, one run of 40 858 / 513, a tenth in runs of 40 845 / 604,
    // all in runs of 64 774 / 775 or of 1,000 748 / 750, half in one cell 793 / 792, half equal 687 / 423.
    unsigned upper = mask;
    while (!(sample && h[kPasses * kRadix]) && __builtin_popcount(upper) > kUpperPasses)
    {
        upper &= upper - 1;
    }
    // a plain read: this path serves sphb_sort_by_key_static, which must call no allocating routine (the pinned
    // block of readBack is allocated on its first use in a thread)
    uint32_t msg[2] = {0, 0};
    SPHB_TRY(runPasses(keys, values, n, s, upper, stream));
    SPHB_CUDA_TRY(cudaMemsetAsync(s.counters + 2, 0, 2 * sizeof(uint32_t), stream));
    if (upper != mask)
    {
        int shift = __builtin_ctz(upper) * kRadixBits;
        longRunsKernel<<<ceilDiv(n, 256), 256, 0, stream>>>(keys, n, shift, s.counters + 2);
        sortRunsKernel<<<ceilDiv(n, 256), 256, 0, stream>>>(keys, values, n, shift, s.counters, s.valsAlt);
        unsigned blocks = unsigned(std::min<size_t>(ceilDiv(n, kRunCap + 1), size_t(smCount()) * 8));
        runBlockKernel<<<blocks, kRunBlockThreads, 0, stream>>>(keys, values, n, shift, s.counters, s.valsAlt);
        SPHB_CUDA_TRY(cudaGetLastError());
    }
    SPHB_CUDA_TRY(cudaMemcpyAsync(msg, s.counters + 1, sizeof(msg), cudaMemcpyDeviceToHost, stream));
    SPHB_CUDA_TRY(cudaStreamSynchronize(stream));
    if (!msg[0] && msg[1])
    {
        SPHB_CUDA_TRY(cudaMemsetAsync(s.hist, 0, kPasses * kRadix * sizeof(uint32_t), stream));
        histogramKernel<<<histBlocks, kHistThreads, 0, stream>>>(keys, n, s.hist, nullptr);
        SPHB_CUDA_TRY(cudaGetLastError());
        SPHB_TRY(runPasses(keys, values, n, s, mask, stream));
        SPHB_CUDA_TRY(cudaMemcpyAsync(msg, s.counters + 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
        SPHB_CUDA_TRY(cudaStreamSynchronize(stream));
    }
    // 1: a look-back wait gave up; 2: offsets left inconsistent by such a wait (nothing else produces them)
    return msg[0] ? kErrTimeout : kOk;
}

int sortNearlySorted(uint64_t* keys, uint32_t* values, size_t n, void* scratch, size_t scratchBytes, bool* identity,
                     cudaStream_t stream)
{
    *identity = false;
    if (n == 0)
    {
        *identity = true;
        return kOk;
    }
    if (n >= (size_t(1) << 30)) { return kErrArg; }
    if (!scratch || scratchBytes < sortScratchBytes(n)) { return kErrCapacity; }
    SortScratch s = carve(scratch, n);
    iotaKernel<<<ceilDiv(n, 256), 256, 0, stream>>>(values, n);
    SPHB_CUDA_TRY(cudaGetLastError());
    unsigned blocks = unsigned(std::min<size_t>(ceilDiv(n, 256 * 8), size_t(smCount()) * 8));
    auto countInversions = [&](uint32_t* out) -> int {
        SPHB_CUDA_TRY(cudaMemsetAsync(s.counters, 0, sizeof(uint32_t), stream));
        inversionsKernel<<<blocks, 256, 0, stream>>>(keys, n, s.counters);
        SPHB_CUDA_TRY(cudaGetLastError());
        SPHB_TRY(readBack(stream, {{out, s.counters, sizeof(uint32_t)}}));
        return kOk;
    };
    uint32_t inv = 0;
    SPHB_TRY(countInversions(&inv));
    if (inv == 0)
    {
        *identity = true;
        return kOk;
    }
    // sparse, local disorder: stable sorts of the dirty tiles, then of the tiles shifted by half a tile
    size_t tiles = ceilDiv(n, size_t(kRepairTile));
    repairTilesKernel<<<unsigned(tiles), kRepairThreads, 0, stream>>>(keys, values, n, 0);
    repairTilesKernel<<<unsigned(ceilDiv(n, size_t(kRepairTile))), kRepairThreads, 0, stream>>>(keys, values, n,
                                                                                               kRepairTile / 2);
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_TRY(countInversions(&inv));
    if (inv == 0) { return kOk; }
    // otherwise the full radix sort; the repaired sequence kept equal keys in their original order, so a stable
    // sort of it is the stable sort of the original
    return sortByKey(keys, values, n, false, scratch, scratchBytes, stream);
}

namespace
{

constexpr int kBlockSortThreads = 1024;
constexpr int kBlockSortItems   = 16;
constexpr int kBlockSortWarps   = kBlockSortThreads / kWarp;
constexpr int kBlockSortMax     = kBlockSortThreads * kBlockSortItems;
static_assert(kBlockSortMax == int(kSortShortMax), "sort.cuh");

struct BlockSortShared
{
    uint32_t key[kBlockSortMax];
    uint32_t val[kBlockSortMax];
    uint16_t warpCount[kBlockSortWarps][kRadix]; // keys of a digit per warp, then those of the warps before it
    uint32_t digitBase[kRadix];
    uint32_t warpSum[kRadix / kWarp];
};

/*! stable LSD sort of up to kBlockSortMax keys of 32 bits by one block in shared memory, ranked as in onesweepKernel; a
 *  digit that all keys share is skipped */
__global__ void __launch_bounds__(kBlockSortThreads) blockSortKernel(uint64_t* keys, uint32_t* values, int n)
{
    extern __shared__ __align__(16) char raw[];
    BlockSortShared& sh = *reinterpret_cast<BlockSortShared*>(raw);
    const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
    const int base = warp * kBlockSortItems * kWarp + lane;

    for (int i = threadIdx.x; i < n; i += kBlockSortThreads)
    {
        sh.key[i] = uint32_t(keys[i]);
        sh.val[i] = values[i];
    }
    for (int shift = 0; shift < 32; shift += kRadixBits)
    {
        for (int t = threadIdx.x; t < kBlockSortWarps * kRadix; t += kBlockSortThreads)
        {
            (&sh.warpCount[0][0])[t] = 0;
        }
        __syncthreads();
        uint32_t key[kBlockSortItems], val[kBlockSortItems];
        uint16_t rank[kBlockSortItems];
#pragma unroll
        for (int k = 0; k < kBlockSortItems; ++k)
        {
            const int idx    = base + k * kWarp;
            const bool valid = idx < n;
            key[k]           = valid ? sh.key[idx] : 0u;
            val[k]           = valid ? sh.val[idx] : 0u;
            uint32_t digit   = (key[k] >> shift) & (kRadix - 1);
            uint32_t peers   = __match_any_sync(0xffffffffu, valid ? digit : 0xffffffffu);
            uint32_t before  = valid ? sh.warpCount[warp][digit] : 0u;
            uint32_t lower   = peers & ((1u << lane) - 1u);
            rank[k]          = uint16_t(before + __popc(lower));
            __syncwarp();
            if (valid && lower == 0) { sh.warpCount[warp][digit] = uint16_t(before + __popc(peers)); }
            __syncwarp();
        }
        __syncthreads();
        // per digit: the warps' counts, then the digits' first positions (thread d owns digit d)
        uint32_t total = 0, incl = 0;
        if (threadIdx.x < kRadix)
        {
            for (int w = 0; w < kBlockSortWarps; ++w)
            {
                uint32_t c                    = sh.warpCount[w][threadIdx.x];
                sh.warpCount[w][threadIdx.x] = uint16_t(total);
                total += c;
            }
            incl = total;
#pragma unroll
            for (int off = 1; off < kWarp; off <<= 1)
            {
                uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) { incl += t; }
            }
            if (lane == kWarp - 1) { sh.warpSum[warp] = incl; }
        }
        const bool shared = __syncthreads_or(threadIdx.x < kRadix && total == uint32_t(n));
        if (shared) { continue; }
        if (threadIdx.x < kRadix)
        {
            uint32_t before = 0;
            for (int w = 0; w < warp; ++w)
            {
                before += sh.warpSum[w];
            }
            sh.digitBase[threadIdx.x] = before + incl - total;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kBlockSortItems; ++k)
        {
            if (base + k * kWarp < n)
            {
                uint32_t digit = (key[k] >> shift) & (kRadix - 1);
                uint32_t pos   = sh.digitBase[digit] + sh.warpCount[warp][digit] + rank[k];
                sh.key[pos]    = key[k];
                sh.val[pos]    = val[k];
            }
        }
        __syncthreads();
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kBlockSortThreads)
    {
        keys[i]   = sh.key[i];
        values[i] = sh.val[i];
    }
}

} // namespace

int sortShortKeysAsync(uint64_t* keys, uint32_t* values, size_t n, cudaStream_t stream)
{
    if (n == 0) { return kOk; }
    if (n > kSortShortMax) { return kErrArg; }
    SPHB_CUDA_TRY(cudaFuncSetAttribute(blockSortKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(sizeof(BlockSortShared))));
    blockSortKernel<<<1, kBlockSortThreads, sizeof(BlockSortShared), stream>>>(keys, values, int(n));
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int sortByKeyAsync(uint64_t* keys, uint32_t* values, size_t n, bool initValues, void* scratch, size_t scratchBytes,
                   unsigned passMask, uint32_t* errorOut, cudaStream_t stream, const uint32_t* gate)
{
    if (n == 0) { return kOk; }
    if (n >= (size_t(1) << 30)) { return kErrArg; }
    if (!scratch || scratchBytes < sortScratchBytes(n)) { return kErrCapacity; }
    SortScratch s = carve(scratch, n);
    if (initValues)
    {
        iotaKernel<<<ceilDiv(n, 256), 256, 0, stream>>>(values, n);
        SPHB_CUDA_TRY(cudaGetLastError());
    }
    SPHB_CUDA_TRY(cudaMemsetAsync(s.hist, 0, kPasses * kRadix * sizeof(uint32_t), stream));
    unsigned histBlocks = histogramBlocks(n);
    histogramKernel<<<histBlocks, kHistThreads, 0, stream>>>(keys, n, s.hist, gate);
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_TRY(runPasses(keys, values, n, s, passMask, stream, gate));
    if (errorOut) { orErrorKernel<<<1, 1, 0, stream>>>(s.counters + 1, errorOut); }
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

namespace
{

//! keys/values from the alternate buffers, unless the gate is closed (the passes did not run)
__global__ void gatedCopyKernel(const uint64_t* kIn, const uint32_t* vIn, uint64_t* kOut, uint32_t* vOut, size_t n,
                                const uint32_t* gate)
{
    if (*gate == 0) { return; }
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    {
        kOut[i] = kIn[i];
        vOut[i] = vIn[i];
    }
}

//! scan the histograms and run the passes of passMask (bit p: digit p), leaving the result in keys/values; with a
//! gate, every kernel returns at once when *gate is 0 (device-side decision, capturable)
int runPasses(uint64_t* keys, uint32_t* values, size_t n, const SortScratch& s, unsigned passMask,
              cudaStream_t stream, const uint32_t* gate)
{
    histScanKernel<<<kPasses, kRadix, 0, stream>>>(s.hist, gate);
    SPHB_CUDA_TRY(cudaGetLastError());
    SPHB_CUDA_TRY(cudaMemsetAsync(s.counters + 1, 0, sizeof(uint32_t), stream));

    size_t tiles      = numTilesOf(n);
    uint64_t* kIn     = keys;
    uint32_t* vIn     = values;
    uint64_t* kOut    = s.keysAlt;
    uint32_t* vOut    = s.valsAlt;
    for (int p = 0; p < kPasses; ++p)
    {
        if (!(passMask & (1u << p))) { continue; }
        SPHB_CUDA_TRY(cudaMemsetAsync(s.status, 0, tiles * kRadix * sizeof(uint32_t), stream));
        SPHB_CUDA_TRY(cudaMemsetAsync(s.counters, 0, sizeof(uint32_t), stream));
        onesweepKernel<<<unsigned(tiles), kSortThreads, 0, stream>>>(kIn, vIn, kOut, vOut, n, p * kRadixBits,
                                                                      s.hist + p * kRadix, s.status, s.counters,
                                                                      gate);
        SPHB_CUDA_TRY(cudaGetLastError());
        std::swap(kIn, kOut);
        std::swap(vIn, vOut);
    }
    if (kIn != keys && gate)
    {
        unsigned blocks = unsigned(std::min<size_t>(ceilDiv(n, 256), size_t(smCount()) * 8));
        gatedCopyKernel<<<blocks, 256, 0, stream>>>(kIn, vIn, keys, values, n, gate);
        SPHB_CUDA_TRY(cudaGetLastError());
    }
    else if (kIn != keys)
    {
        SPHB_CUDA_TRY(cudaMemcpyAsync(keys, kIn, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, stream));
        SPHB_CUDA_TRY(cudaMemcpyAsync(values, vIn, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, stream));
    }
    return kOk;
}

} // namespace

// ---------------------------------------------------------------------------------------------------------------
// Sort of a step's particles by the leaves of the previous step's tree
//
// Bound by memory: 2 reads and 2 writes of the pairs plus the leaf searches, whatever moved. The repair of nearly sorted
// keys pays only while particles stay within a tile of 2,048; one that crosses an octant boundary of the curve far up
// moves by up to n, and then both repair passes (45 us each at 4,096 particles, 91 us at 128^3) were followed by the
// radix sort (eight passes of 18 to 38 us and an 8 KB host read). Sync of a step with such a motion: 16^3 235 -> 154 us,
// 30^3 510 -> 168 us, 81^3 (Noh) 663 -> 263 us, 128^3 0.95 -> 0.43 ms. A warp sorts a leaf in registers, at most
// 128 keys (four per lane): the tree splits leaves of more than 64, so only a sudden compression exceeds it, or trees
// that stay those of the last rebuild (an ensemble's; 663,000 particles in 16 members 0.69 -> 0.21 ms): a block sorts
// such a leaf, up to 2,048 keys. Beyond that the radix sort runs.
// ---------------------------------------------------------------------------------------------------------------

namespace
{

//! the largest leaf a warp sorts (four elements per lane), and the largest one a block sorts
constexpr int kLeafSortCap  = 128;
constexpr int kLeafBlockCap = 2048;

//! words before the bucket counts
enum LeafFlag
{
    kLeafInversions, // an adjacent pair is out of order (one tree only)
    kLeafOverflow,   // a bucket exceeds kLeafBlockCap: nothing is sorted
    kLeafLarge,      // a bucket exceeds kLeafSortCap
    kLeafListed,     // number of such buckets, listed by leafSortKernel
    kNumLeafFlags
};

//! largest l with leaves[l] <= key (leaves[0] = 0; l = numLeaves for keys past the last leaf)
__device__ __forceinline__ int leafOf(const uint64_t* __restrict__ leaves, int numLeaves, uint64_t key)
{
    int lo = 0, hi = numLeaves + 1;
    while (hi - lo > 1)
    {
        int mid = (lo + hi) >> 1;
        if (__ldg(leaves + mid) <= key) { lo = mid; }
        else { hi = mid; }
    }
    return lo;
}

//! the leaves that hold key i: one tree, or the tree of the key's segment
template<bool kSeg>
__device__ __forceinline__ LeafSet leafSetOf(const LeafSet& one, const LeafSet* __restrict__ many,
                                             const uint64_t* __restrict__ seg, size_t i)
{
    if constexpr (kSeg) { return many[seg[i]]; }
    else { return one; }
}

/*! values = 0..n-1; slot[i] = {bucket (leaf) of key i, its place among the bucket's keys in arrival order}, counts[l] =
 *  keys per bucket (zero on entry), and the flags (zero on entry). The lanes of a bucket (most of a warp: the keys are nearly in order) share one
 *  atomic. */
template<bool kSeg>
__global__ void __launch_bounds__(256) leafSlotKernel(const uint64_t* __restrict__ keys, size_t n, LeafSet one,
                                                      const LeafSet* __restrict__ many,
                                                      const uint64_t* __restrict__ seg, uint32_t* __restrict__ values,
                                                      uint2* __restrict__ slot, int* counts, unsigned* flags)
{
    size_t i   = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    bool valid = i < n;
    int bucket = -1;
    bool inv   = false;
    if (valid)
    {
        uint64_t k = keys[i];
        if constexpr (!kSeg) { inv = i + 1 < n && k > keys[i + 1]; }
        LeafSet t = leafSetOf<kSeg>(one, many, seg, i);
        bucket    = int(t.bucket0) + leafOf(t.leaves, t.numLeaves, k);
        values[i] = uint32_t(i);
    }
    unsigned lane  = threadIdx.x & (kWarp - 1);
    unsigned peers = __match_any_sync(0xffffffffu, bucket);
    int leader     = __ffs(peers) - 1;
    int base       = 0;
    if (int(lane) == leader && valid) { base = atomicAdd(counts + bucket, __popc(peers)); }
    base      = __shfl_sync(0xffffffffu, base, leader);
    int place = base + __popc(peers & ((1u << lane) - 1u));
    if (valid) { slot[i] = make_uint2(unsigned(bucket), unsigned(place)); }
    unsigned anyInv   = __ballot_sync(0xffffffffu, inv);
    unsigned anyLarge = __ballot_sync(0xffffffffu, valid && place >= kLeafSortCap);
    unsigned anyOver  = __ballot_sync(0xffffffffu, valid && place >= kLeafBlockCap);
    if (lane == 0 && anyInv) { flags[kLeafInversions] = 1u; }
    if (lane == 0 && anyLarge) { flags[kLeafLarge] = 1u; }
    if (lane == 0 && anyOver) { flags[kLeafOverflow] = 1u; }
}

/*! composite[first[bucket] + place] = (the upper 32 bits of the key within its leaf, index): what a warp sorts. A leaf
 *  of level L leaves 63 - 3 L bits of the key open. */
template<bool kSeg>
__global__ void __launch_bounds__(256) leafScatterKernel(const uint64_t* __restrict__ keys, size_t n, LeafSet one,
                                                         const LeafSet* __restrict__ many,
                                                         const uint64_t* __restrict__ seg,
                                                         const uint2* __restrict__ slot, const int* __restrict__ first,
                                                         uint64_t* __restrict__ composite, const unsigned* flags)
{
    size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i >= n || (kSeg && flags[kLeafOverflow] != 0)) { return; }
    uint2 s        = slot[i];
    LeafSet t      = leafSetOf<kSeg>(one, many, seg, i);
    int leaf       = int(s.x - t.bucket0);
    uint64_t start = __ldg(t.leaves + leaf);
    int shift      = 0;
    if (leaf < t.numLeaves) { shift = max(0, 31 - int(__clzll(__ldg(t.leaves + leaf + 1) - start))); }
    size_t dst = size_t(__ldg(first + s.x)) + s.y;
    if (dst < n) { composite[dst] = (((keys[i] - start) >> shift) << 32) | uint64_t(i); }
}

//! bitonic sort of 32 kPer values of a warp, value e in register e / 32 of lane e % 32
template<int kPer>
__device__ __forceinline__ void warpSort(uint64_t (&v)[kPer], int lane)
{
#pragma unroll
    for (int size = 2; size <= 32 * kPer; size <<= 1)
    {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1)
        {
            if (stride >= 32)
            {
#pragma unroll
                for (int r = 0; r < kPer; ++r)
                {
                    int q = r ^ (stride / 32);
                    if (q > r)
                    {
                        bool up = ((r * 32) & size) == 0;
                        if ((v[r] > v[q]) == up)
                        {
                            uint64_t t = v[r];
                            v[r]       = v[q];
                            v[q]       = t;
                        }
                    }
                }
            }
            else
            {
#pragma unroll
                for (int r = 0; r < kPer; ++r)
                {
                    uint64_t o = __shfl_xor_sync(0xffffffffu, v[r], stride);
                    bool up    = ((r * 32 + lane) & size) == 0;
                    bool low   = (lane & stride) == 0;
                    v[r]       = ((v[r] < o) == (up == low)) ? v[r] : o;
                }
            }
        }
    }
}

/*! One leaf: its composites sorted, then the keys and values in that order. Composites that agree in their upper half
 *  may belong to different keys (the open bits beyond 32): such a leaf is ranked by its full keys instead. */
template<int kPer>
__device__ __forceinline__ void sortLeaf(const uint64_t* composite, const uint64_t* __restrict__ keysIn, int first, int m,
                                         int lane, uint64_t* keysOut, uint32_t* values)
{
    uint64_t v[kPer];
#pragma unroll
    for (int r = 0; r < kPer; ++r)
    {
        int e = r * 32 + lane;
        v[r]  = e < m ? composite[first + e] : ~uint64_t(0);
    }
    warpSort<kPer>(v, lane);
    uint64_t key[kPer];
    bool tie = false;
#pragma unroll
    for (int r = 0; r < kPer; ++r)
    {
        int e         = r * 32 + lane;
        key[r]        = e < m ? __ldg(keysIn + uint32_t(v[r])) : ~uint64_t(0);
        uint64_t next = __shfl_down_sync(0xffffffffu, v[r], 1);
        if (r + 1 < kPer)
        {
            uint64_t wrap = __shfl_sync(0xffffffffu, v[r + 1 < kPer ? r + 1 : r], 0);
            if (lane == 31) { next = wrap; }
        }
        tie = tie || (e + 1 < m && (lane < 31 || r + 1 < kPer) && (v[r] >> 32) == (next >> 32));
    }
    int place[kPer];
#pragma unroll
    for (int r = 0; r < kPer; ++r)
    {
        place[r] = r * 32 + lane;
    }
    if (__any_sync(0xffffffffu, tie))
    {
#pragma unroll
        for (int r = 0; r < kPer; ++r)
        {
            place[r] = 0;
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q)
        {
            for (int src = 0; src < 32; ++src)
            {
                if (q * 32 + src >= m) { break; }
                uint64_t ko = __shfl_sync(0xffffffffu, key[q], src);
                uint32_t io = __shfl_sync(0xffffffffu, uint32_t(v[q]), src);
#pragma unroll
                for (int r = 0; r < kPer; ++r)
                {
                    place[r] += (ko < key[r] || (ko == key[r] && io < uint32_t(v[r]))) ? 1 : 0;
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kPer; ++r)
    {
        if (r * 32 + lane < m)
        {
            keysOut[first + place[r]] = key[r];
            values[first + place[r]]  = uint32_t(v[r]);
        }
    }
}

//! one warp per bucket; larger ones are listed for leafBlockKernel (flags zero in kLeafListed on entry)
__global__ void __launch_bounds__(256) leafSortKernel(const uint64_t* __restrict__ composite,
                                                      const uint64_t* __restrict__ keysIn, int numBuckets,
                                                      const int* __restrict__ first, uint64_t* __restrict__ keysOut,
                                                      uint32_t* __restrict__ values, unsigned* flags, uint32_t* large)
{
    int bucket = int((blockIdx.x * size_t(blockDim.x) + threadIdx.x) / kWarp);
    int lane   = threadIdx.x & (kWarp - 1);
    if (bucket >= numBuckets || flags[kLeafOverflow] != 0) { return; }
    int b = first[bucket], m = first[bucket + 1] - b;
    if (m <= 0) { return; }
    if (m <= 32) { sortLeaf<1>(composite, keysIn, b, m, lane, keysOut, values); }
    else if (m <= 64) { sortLeaf<2>(composite, keysIn, b, m, lane, keysOut, values); }
    else if (m <= kLeafSortCap) { sortLeaf<4>(composite, keysIn, b, m, lane, keysOut, values); }
    else if (lane == 0) { large[atomicAdd(flags + kLeafListed, 1u)] = uint32_t(bucket); }
}

constexpr int kLeafBlockThreads = 512;

/*! One block per listed bucket: bitonic network on (key, index) in shared memory. An ensemble's trees stay those of the
 *  last rebuild, and a contracting member outgrows the warps for the rest of a run; the radix sort of all slots that took
 *  over before cost 140 us a step for 512,000 of them (sync 315 us, with this kernel 185, 176 before the leaf grew). */
__global__ void __launch_bounds__(kLeafBlockThreads) leafBlockKernel(const uint64_t* __restrict__ composite,
                                                                     const uint64_t* __restrict__ keysIn,
                                                                     const int* __restrict__ first,
                                                                     uint64_t* __restrict__ keysOut,
                                                                     uint32_t* __restrict__ values,
                                                                     const unsigned* flags, const uint32_t* large)
{
    __shared__ uint64_t key[kLeafBlockCap];
    __shared__ uint32_t val[kLeafBlockCap];
    if (flags[kLeafOverflow] != 0) { return; }
    const unsigned num = flags[kLeafListed];
    for (unsigned l = blockIdx.x; l < num; l += gridDim.x)
    {
        const int b = first[large[l]];
        const int m = min(first[large[l] + 1] - b, kLeafBlockCap);
        int width   = 2 * kLeafSortCap;
        while (width < m)
        {
            width <<= 1;
        }
        for (int e = threadIdx.x; e < width; e += kLeafBlockThreads)
        {
            val[e] = e < m ? uint32_t(composite[b + e]) : 0xffffffffu;
            key[e] = e < m ? __ldg(keysIn + val[e]) : ~uint64_t(0);
        }
        __syncthreads();
        blockBitonic<kLeafBlockThreads>(width, [&](int q, int p, bool up) {
            if ((key[q] > key[p] || (key[q] == key[p] && val[q] > val[p])) == up)
            {
                uint64_t k = key[q];
                key[q]     = key[p];
                key[p]     = k;
                uint32_t v = val[q];
                val[q]     = val[p];
                val[p]     = v;
            }
        });
        for (int e = threadIdx.x; e < m; e += kLeafBlockThreads)
        {
            keysOut[b + e] = key[e];
            values[b + e]  = val[e];
        }
        __syncthreads();
    }
}

//! blocks of leafBlockKernel: every one may find a bucket, none has many
unsigned leafBlocks(size_t n) { return unsigned(std::min<size_t>(ceilDiv(n, kLeafSortCap), size_t(smCount()) * 2)); }

} // namespace

size_t leafSortInts(size_t numBuckets) { return kNumLeafFlags + numBuckets + 1; }

int sortByLeaves(uint64_t* keys, uint64_t* keysOut, uint32_t* values, size_t n, const uint64_t* leaves, int numLeaves,
                 LeafSortScratch& ls, void* scratch, size_t scratchBytes, LeafSort* result, cudaStream_t stream)
{
    *result = LeafSort::inPlace;
    if (n == 0)
    {
        *result = LeafSort::identity;
        return kOk;
    }
    if (n >= (size_t(1) << 30) || numLeaves < 1) { return kErrArg; }
    if (!scratch || scratchBytes < sortScratchBytes(n)) { return kErrCapacity; }
    size_t buckets = size_t(numLeaves) + 1;
    SPHB_TRY(ls.slot.reserve(n));
    SPHB_TRY(ls.first.reserve(leafSortInts(buckets)));
    SPHB_TRY(ls.scanTmp.reserve(scanTempInts(buckets) + 1));
    int* counts     = ls.first.data() + kNumLeafFlags;
    unsigned* flags = reinterpret_cast<unsigned*>(ls.first.data());
    SPHB_CUDA_TRY(cudaMemsetAsync(ls.first.data(), 0, (kNumLeafFlags + buckets) * sizeof(int), stream));
    LeafSet one{leaves, numLeaves, 0};
    leafSlotKernel<false><<<ceilDiv(n, 256), 256, 0, stream>>>(keys, n, one, nullptr, nullptr, values, ls.slot.data(),
                                                               counts, flags);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    unsigned msg[kLeafLarge + 1];
    SPHB_TRY(readBack(stream, {{msg, flags, sizeof(msg)}}));
    if (!msg[kLeafInversions])
    {
        *result = LeafSort::identity;
        return kOk;
    }
    if (msg[kLeafOverflow]) { return sortByKey(keys, values, n, false, scratch, scratchBytes, stream); }
    uint64_t* composite = carve(scratch, n).keysAlt;
    uint32_t* large     = carve(scratch, n).valsAlt;
    SPHB_TRY(exclusiveScan(counts, counts, buckets, ls.scanTmp.data(), stream));
    leafScatterKernel<false><<<ceilDiv(n, 256), 256, 0, stream>>>(keys, n, one, nullptr, nullptr, ls.slot.data(), counts,
                                                                  composite, nullptr);
    leafSortKernel<<<ceilDiv(buckets * kWarp, 256), 256, 0, stream>>>(composite, keys, int(buckets), counts, keysOut,
                                                                      values, flags, large);
    countLaunch(2);
    if (msg[kLeafLarge])
    {
        leafBlockKernel<<<leafBlocks(n), kLeafBlockThreads, 0, stream>>>(composite, keys, counts, keysOut, values, flags,
                                                                         large);
        countLaunch();
    }
    SPHB_CUDA_TRY(cudaGetLastError());
    *result = LeafSort::keysOut;
    return kOk;
}

int sortSegmentsByLeavesAsync(const uint64_t* keys, uint64_t* keysOut, uint32_t* values, size_t n, const uint64_t* seg,
                              const LeafSet* sets, size_t numBuckets, LeafSortScratch& ls, void* scratch,
                              size_t scratchBytes, const unsigned** overflow, cudaStream_t stream)
{
    if (!scratch || scratchBytes < sortScratchBytes(n) || ls.slot.capacity() < n ||
        ls.first.capacity() < leafSortInts(numBuckets) || ls.scanTmp.capacity() < scanTempInts(numBuckets) + 1)
    {
        return kErrCapacity;
    }
    int* counts     = ls.first.data() + kNumLeafFlags;
    unsigned* flags = reinterpret_cast<unsigned*>(ls.first.data());
    *overflow       = flags + kLeafOverflow;
    SPHB_CUDA_TRY(cudaMemsetAsync(ls.first.data(), 0, (kNumLeafFlags + numBuckets) * sizeof(int), stream));
    if (n == 0) { return kOk; }
    uint64_t* composite = carve(scratch, n).keysAlt;
    uint32_t* large     = carve(scratch, n).valsAlt;
    LeafSet none{nullptr, 0, 0};
    leafSlotKernel<true><<<ceilDiv(n, 256), 256, 0, stream>>>(keys, n, none, sets, seg, values, ls.slot.data(), counts,
                                                              flags);
    countLaunch();
    SPHB_TRY(exclusiveScan(counts, counts, numBuckets, ls.scanTmp.data(), stream));
    leafScatterKernel<true><<<ceilDiv(n, 256), 256, 0, stream>>>(keys, n, none, sets, seg, ls.slot.data(), counts,
                                                                 composite, flags);
    leafSortKernel<<<ceilDiv(numBuckets * kWarp, 256), 256, 0, stream>>>(composite, keys, int(numBuckets), counts,
                                                                         keysOut, values, flags, large);
    leafBlockKernel<<<leafBlocks(n), kLeafBlockThreads, 0, stream>>>(composite, keys, counts, keysOut, values, flags,
                                                                     large);
    countLaunch(3);
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

// ---------------------------------------------------------------------------------------------------------------
// Allocation-free variant: the scratch lives in a fixed device array of this library (see sphb_sort_by_key_static)
// ---------------------------------------------------------------------------------------------------------------

//! largest n accepted by the allocation-free sort
constexpr size_t kStaticSortMaxN = size_t(1) << 20;

constexpr size_t alignUpC(size_t x, size_t a) { return (x + a - 1) / a * a; }

constexpr size_t kStaticSortBytes = alignUpC(kStaticSortMaxN * sizeof(uint64_t), 256) +
                                    alignUpC(kStaticSortMaxN * sizeof(uint32_t), 256) +
                                    alignUpC(kPasses * kRadix * sizeof(uint32_t), 256) +
                                    alignUpC((kStaticSortMaxN + kTile - 1) / kTile * kRadix * sizeof(uint32_t), 256) +
                                    256;

/*! Scratch of the allocation-free sort: ~12.6 MB of device memory that every GPU which loads this library holds until
 *  the process exits. Host code must not use the symbol itself as a device address; it asks the runtime for the
 *  device address of this array once per device (staticSortScratch below). */
static __device__ __align__(256) unsigned char gStaticSortScratch[kStaticSortBytes];

namespace
{

//! one looked-up address per CUDA context: a context created after cudaDeviceReset gets its own entry
struct StaticScratchEntry
{
    CUcontext ctx;
    void* addr;
};
constexpr int kMaxContexts = 64;
std::mutex gStaticScratchMutex;
StaticScratchEntry gStaticScratch[kMaxContexts] = {};
int gStaticScratchNext                          = 0;
PFN_cuCtxGetCurrent_v4000 gCtxGetCurrent        = nullptr;

/*! Device address of gStaticSortScratch in the current context, looked up with the context's device current on the
 *  first call in that context. The driver's cuCtxGetCurrent is reached through the runtime's entry-point query, so
 *  this library does not link libcuda. */
int staticSortScratch(void** ptr)
{
    std::lock_guard<std::mutex> lock(gStaticScratchMutex);
    if (!gCtxGetCurrent)
    {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        SPHB_CUDA_TRY(cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !fn) { return kErrCuda; }
        gCtxGetCurrent = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(fn);
    }
    CUcontext ctx = nullptr;
    if (gCtxGetCurrent(&ctx) != CUDA_SUCCESS) { return kErrCuda; }
    if (!ctx)
    {
        // no context is current on this thread yet: make the current device's primary context current
        int dev = 0;
        SPHB_CUDA_TRY(cudaGetDevice(&dev));
        SPHB_CUDA_TRY(cudaSetDevice(dev));
        if (gCtxGetCurrent(&ctx) != CUDA_SUCCESS || !ctx) { return kErrCuda; }
    }
    for (const StaticScratchEntry& e : gStaticScratch)
    {
        if (e.ctx == ctx && e.addr)
        {
            *ptr = e.addr;
            return kOk;
        }
    }
    void* p = nullptr;
    SPHB_CUDA_TRY(cudaGetSymbolAddress(&p, gStaticSortScratch));
    gStaticScratch[gStaticScratchNext] = {ctx, p};
    gStaticScratchNext                 = (gStaticScratchNext + 1) % kMaxContexts;
    *ptr                               = p;
    return kOk;
}

} // namespace

} // namespace sphb

extern "C" size_t sphb_sort_by_key_static_max(void) { return sphb::kStaticSortMaxN; }

extern "C" int sphb_sort_by_key_static(uint64_t* keys, uint32_t* values, size_t n, int init_values, void* stream)
{
    if (n && (!keys || !values)) { return SPHB_ERR_ARG; }
    if (n > sphb::kStaticSortMaxN)
    {
        std::fprintf(stderr, "sphb_sort_by_key_static: n = %zu exceeds the fixed scratch capacity of %zu pairs\n", n,
                     sphb::kStaticSortMaxN);
        return SPHB_ERR_CAPACITY;
    }
    void* scratch = nullptr;
    int rc        = sphb::staticSortScratch(&scratch);
    if (rc != SPHB_OK) { return rc; }
    return sphb::sortByKey(keys, values, n, init_values != 0, scratch, sphb::kStaticSortBytes,
                           static_cast<cudaStream_t>(stream));
}

extern "C" size_t sphb_sort_by_key_scratch_bytes(size_t n) { return sphb::sortScratchBytes(n); }

extern "C" int sphb_sort_by_key(uint64_t* keys, uint32_t* values, size_t n, int init_values, void* scratch,
                                size_t scratch_bytes, void* stream)
{
    if (n && (!keys || !values)) { return SPHB_ERR_ARG; }
    return sphb::sortByKey(keys, values, n, init_values != 0, scratch, scratch_bytes,
                           static_cast<cudaStream_t>(stream));
}

extern "C" int sphb_sort_by_key_nearly_sorted(uint64_t* keys, uint32_t* values, size_t n, void* scratch,
                                              size_t scratch_bytes, int* identity, void* stream)
{
    if (!identity || (n && (!keys || !values))) { return SPHB_ERR_ARG; }
    bool id = false;
    int rc  = sphb::sortNearlySorted(keys, values, n, scratch, scratch_bytes, &id, static_cast<cudaStream_t>(stream));
    *identity = id ? 1 : 0;
    return rc;
}
