// Device helpers shared by the SPH-VE J-loops (hydro_ve.cu) and their adjoints (adjoint.cu): neighbour-sum
// accumulators, kernel evaluation, pair separations per precision, packed record loads and the chunked list reads.
#pragma once

#include "hydro.cuh"
#include "neighbors.cuh"

namespace sphb
{
namespace chain
{

constexpr int kChainThreads = 128;

//! compile-time variants of the J-loop kernels: write the adjoint's tape, or run over a batched ensemble
constexpr int kModeTape    = 1;
constexpr int kModeBatch   = 2;
constexpr int kModeAvClean = 4;
constexpr int kModeList    = 8; // block time steps: only the groups of a device-side list
constexpr int kModeFullAv  = 16; // AV switches on AVFullRec records

/*! Neighbour-sum accumulator. Terms are summed plainly within one list chunk of 8 neighbours, in list order, and the
 *  chunk sums are added in chunk order: FP64 plainly, FP32 with Kahan compensation (explicit round-to-nearest
 *  intrinsics keep the compiler from fusing or reordering it). A chunk may be summed by another lane (foldChunks), so
 *  the result does not depend on how many lanes share a target. */
template<class T>
struct BlockSum;

template<>
struct BlockSum<double>
{
    double s, part;
    __device__ explicit BlockSum(double v = 0.0)
        : s(v)
        , part(0.0)
    {
    }
    __device__ void add(double v) { part += v; }
    __device__ void addChunk(double v) { s += v; }
    __device__ double get() const { return s; }
};

template<>
struct BlockSum<float>
{
    float s, comp, part;
    __device__ explicit BlockSum(float v = 0.f)
        : s(v)
        , comp(0.f)
        , part(0.f)
    {
    }
    __device__ void add(float v) { part += v; }
    __device__ void addChunk(float v)
    {
        float y = __fsub_rn(v, comp);
        float t = __fadd_rn(s, y);
        comp    = __fsub_rn(__fsub_rn(t, s), y);
        s       = t;
    }
    __device__ float get() const { return s; }
};

/*! Add the chunk sums of one round to the accumulators and clear them: this lane's own (kSplit = 1), or those of the
 *  kSplit lanes that share a target, in chunk order (chunks first .. first + kSplit - 1 of numChunks); every lane of
 *  the warp calls it, and the lanes of a target end with equal sums. */
template<int kSplit, class... S>
__device__ __forceinline__ void foldChunks(unsigned first, unsigned numChunks, S&... acc)
{
    if constexpr (kSplit == 1) { (acc.addChunk(acc.part), ...); }
    else
    {
#pragma unroll
        for (int s = 0; s < kSplit; ++s)
        {
            auto one = [&](auto& a) {
                auto v = __shfl_sync(0xffffffffu, a.part, s, kSplit);
                if (first + s < numChunks) { a.addChunk(v); }
            };
            (one(acc), ...);
        }
    }
    ((acc.part = 0), ...);
}

//! the largest value over the lanes that share a target
template<int kSplit, class T>
__device__ __forceinline__ T maxOverSplit(T v)
{
#pragma unroll
    for (int off = 1; off < kSplit; off <<= 1)
    {
        T o = __shfl_xor_sync(0xffffffffu, v, off);
        v   = o > v ? o : v;
    }
    return v;
}

//! a / b: IEEE division in FP64 (the reference's rounding), the fast 2-ulp reciprocal-multiply in FP32
__device__ __forceinline__ double fdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }

// Sums of products with the rounding written out. Left to the compiler, which product of a sum becomes the FMA's differs
// between the instances of a kernel (one lane or several per target, a single simulation or an ensemble), and with it the
// last bit of their results. A last bit counts: the AV switches jump where divv changes its sign, by the full range of
// alpha for such a particle. So every FP32 sum keeps the order that the one-lane instances had when the compiler chose
// it, and where that is not the order of these functions the sum is written with fma; tests/test_gpu_mixed_bits.py holds
// the results to it.

//! a . b: y first, then x, then z
template<class T>
__device__ __forceinline__ T dot3(T ax, T ay, T az, T bx, T by, T bz)
{
    return fma(az, bz, fma(ax, bx, ay * by));
}

//! a b + c d
template<class T>
__device__ __forceinline__ T prodSum(T a, T b, T c, T d)
{
    return fma(a, b, c * d);
}

//! a b - c d
template<class T>
__device__ __forceinline__ T prodDiff(T a, T b, T c, T d)
{
    return fma(a, b, -(c * d));
}

//! linear interpolation in a 20000-entry table on [0, 2] (sph/include/sph/table_lookup.hpp:14-26)
template<class T>
__device__ __forceinline__ T tableLookup(const T* __restrict__ table, T v)
{
    if constexpr (sizeof(T) == 8)
    {
        // FP64: the interval and the position in it from one addition of 1.5 * 2^52 (its low word is the rounded
        // integer), instead of two conversions between FP64 and integers, which run at a quarter of the FP64 rate
        constexpr double kMagic = 6755399441055744.0;
        double u = v * (0.5 * (kTableSize - 1));
        if (!(u < double(kTableSize - 1))) { return 0.0; } // v >= 2, or not a number (coincident particles)
        double t  = (u - 0.5) + kMagic;
        int idx   = __double2loint(t);
        double t0 = __ldg(table + idx);
        double t1 = __ldg(table + idx + 1);
        return t0 + (t1 - t0) * (u - (t - kMagic));
    }
    constexpr int numIntervals = kTableSize - 1;
    constexpr T dx             = T(2.0) / numIntervals;
    constexpr T invDx          = T(1) / dx;
    int idx                    = int(v * invDx);
    if (idx >= numIntervals) { return T(0); }
    T t0 = __ldg(table + idx);
    T t1 = __ldg(table + idx + 1);
    T derivative = (t1 - t0) * invDx;
    return t0 + derivative * (v - T(idx) * dx);
}

//! Horner evaluation of the FP32 kernel polynomial at t = v^2/2 - 1
__device__ __forceinline__ float polyEvalT(const float (&c)[kPolyTerms], float t)
{
    float acc = c[kPolyTerms - 1];
#pragma unroll
    for (int p = kPolyTerms - 2; p >= 0; --p)
    {
        acc = fmaf(acc, t, c[p]);
    }
    return acc;
}

//! Horner evaluation of the FP32 kernel polynomial in t = v^2/2 - 1
__device__ __forceinline__ float polyEval(const float (&c)[kPolyTerms], float v)
{
    float t   = fmaf(0.5f * v, v, -1.0f);
    float acc = c[kPolyTerms - 1];
#pragma unroll
    for (int p = kPolyTerms - 2; p >= 0; --p)
    {
        acc = fmaf(acc, t, c[p]);
    }
    return acc;
}

//! the smoothing kernel W(v), zero from v = 2 on: FP64 by table lookup (as the reference), FP32 by polynomial
template<class T>
__device__ __forceinline__ T kernelW(const T* __restrict__ table, const HydroConsts<T>& k, T v)
{
    if constexpr (sizeof(T) == 4)
    {
        if (k.usePoly) { return v < T(2) ? polyEval(k.wpoly, v) : T(0); }
    }
    return tableLookup(table, v);
}

/*! W of a pair from its squared separation r2, for a target with hInv = 1/h and hh = hInv^2 / 2. FP32 with the
 *  polynomial: t = v^2/2 - 1 = r2 hh - 1 directly, zero from t = 1 (v = 2) on, without the square root. Otherwise
 *  (FP64, or an FP32 simulation whose polynomial fit failed) the table at v = sqrt(r2) hInv, the expression of the
 *  reference's order. */
template<class T>
__device__ __forceinline__ T kernelWr2(const T* __restrict__ table, const HydroConsts<T>& k, T r2, T hInv, T hh)
{
    if constexpr (sizeof(T) == 4)
    {
        if (k.usePoly)
        {
            float t = fmaf(r2, hh, -1.0f);
            return t < 1.0f ? polyEvalT(k.wpoly, t) : 0.0f;
        }
    }
    return tableLookup(table, T(sqrt(r2)) * hInv);
}

//! dW/dv, zero from v = 2 on
template<class T>
__device__ __forceinline__ T kernelDW(const T* __restrict__ table, const HydroConsts<T>& k, T v)
{
    if constexpr (sizeof(T) == 4)
    {
        if (k.usePoly) { return v < T(2) ? v * polyEval(k.dwpoly, v) : T(0); }
    }
    return tableLookup(table, v);
}

//! periodic shift of a pair separation by one box length if it exceeds r (cstone/sfc/box.hpp applyPBC, legacy form)
__device__ __forceinline__ void shiftPbc(double& rx, double& ry, double& rz, double r, const DevBox& box)
{
    if (box.periodic[0])
    {
        if (rx > r) { rx -= box.len[0]; }
        else if (rx < -r) { rx += box.len[0]; }
    }
    if (box.periodic[1])
    {
        if (ry > r) { ry -= box.len[1]; }
        else if (ry < -r) { ry += box.len[1]; }
    }
    if (box.periodic[2])
    {
        if (rz > r) { rz -= box.len[2]; }
        else if (rz < -r) { rz += box.len[2]; }
    }
}

//! one 32-byte (256-bit) read-only vector load of 8 floats; p must be 32-byte aligned
__device__ __forceinline__ void ldg256(const void* p, float (&v)[8])
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
}

//! 32-byte read-only load as two 16-byte vector loads (one sector)
__device__ __forceinline__ double4 ldg4(const double4* p)
{
    double4 v;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}

// ---------------------------------------------------------------------------------------------------------------
// positions and pair separations per precision
// ---------------------------------------------------------------------------------------------------------------

template<class T>
struct Pos;

template<>
struct Pos<double>
{
    double x, y, z, m;
};

template<>
struct Pos<float>
{
    int x, y, z;
    float m;
};

__device__ __forceinline__ Pos<double> posOf(const ChainArrays<double>& a, size_t j)
{
    double4 v = ldg4(a.pos + j);
    return {v.x, v.y, v.z, v.w};
}

__device__ __forceinline__ Pos<float> posOf(const ChainArrays<float>& a, size_t j)
{
    int4 v = __ldg(a.posq + j);
    return {v.x, v.y, v.z, __int_as_float(v.w)};
}

template<class T>
struct Sep
{
    T rx, ry, rz;
};

//! x_i - x_j with the reference's periodic shift (threshold r = 2 h_i), FP64
__device__ __forceinline__ Sep<double> separation(const Pos<double>& pi, const Pos<double>& pj, double r,
                                                  const DevBox& box, const HydroConsts<double>&)
{
    double rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
    // the high words order as the magnitudes do, so a component can exceed r only if its high word reaches that of r:
    // the six FP64 comparisons of the shift run only for such pairs (across the box, or at the edge of the sphere)
    int top = max(max(__double2hiint(rx) & 0x7fffffff, __double2hiint(ry) & 0x7fffffff),
                  __double2hiint(rz) & 0x7fffffff);
    if (top >= __double2hiint(r)) { shiftPbc(rx, ry, rz, r, box); }
    return {rx, ry, rz};
}

//! x_i - x_j from fixed-point coordinates: an exact integer difference, wrapped to the nearest image on periodic
//! axes, rounded once to FP32
__device__ __forceinline__ Sep<float> separation(const Pos<float>& pi, const Pos<float>& pj, double,
                                                 const DevBox&, const HydroConsts<float>& k)
{
    int dx = int(unsigned(pi.x) - unsigned(pj.x));
    int dy = int(unsigned(pi.y) - unsigned(pj.y));
    int dz = int(unsigned(pi.z) - unsigned(pj.z));
    return {float(dx) * k.qscale[0], float(dy) * k.qscale[1], float(dz) * k.qscale[2]};
}

template<class T>
__device__ __forceinline__ HydroRec<T> loadHydro(const HydroRec<T>* p)
{
    HydroRec<T> r;
    if constexpr (sizeof(T) == 8)
    {
        const double4* q = reinterpret_cast<const double4*>(p);
        double4 a = ldg4(q), b = ldg4(q + 1);
        r = {T(a.x), T(a.y), T(a.z), T(a.w), T(b.x), T(b.y), T(b.z), T(b.w)};
    }
    else
    {
        float v[8];
        ldg256(p, v);
        r = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
    }
    return r;
}

template<class T>
__device__ __forceinline__ GradRec<T> loadGrad(const GradRec<T>* p)
{
    GradRec<T> r;
    if constexpr (sizeof(T) == 8)
    {
        const double4* q = reinterpret_cast<const double4*>(p);
        double4 a = ldg4(q), b = ldg4(q + 1);
        r = {T(a.x), T(a.y), T(a.z), T(a.w), T(b.x), T(b.y), T(b.z), T(b.w)};
    }
    else
    {
        float v[8];
        ldg256(p, v);
        r = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
    }
    return r;
}

struct Target
{
    size_t i;
    size_t group;
    unsigned lane;
    unsigned count;
    unsigned ngPad;
    unsigned sub{0};       // which of the lanes that share the target
    unsigned numChunks{0}; // list chunks of the target
    unsigned rounds{0};    // turns of the chunk loop: the target's own, or the warp's most where lanes share targets
};

//! the rest of a target's description once its particle is known; without a particle (valid false) an empty list
template<int kSplit>
__device__ __forceinline__ void fillTarget(Target& t, bool valid, const unsigned* nc, unsigned ngmax)
{
    if (!valid) { t.i = 0; }
    t.group     = t.i >> 5;
    t.lane      = unsigned(t.i & 31);
    t.count     = valid ? min(nc[t.i] - 1u, ngmax) : 0u;
    t.ngPad     = paddedNgmax(ngmax);
    t.numChunks = (t.count + kNbChunk - 1) / kNbChunk;
    t.rounds    = t.numChunks;
    if constexpr (kSplit > 1)
    {
        t.rounds = __reduce_max_sync(0xffffffffu, (t.numChunks + kSplit - 1) / kSplit);
    }
}

template<int kSplit = 1>
__device__ __forceinline__ bool targetOf(size_t n, const unsigned* nc, unsigned ngmax, Target& t,
                                         const uint8_t* inst = nullptr)
{
    size_t thread = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    t.i           = thread / kSplit;
    t.sub         = unsigned(thread % kSplit);
    bool valid    = t.i < n && !(inst && inst[t.i] == kGhost);
    if (kSplit == 1 && !valid) { return false; }
    fillTarget<kSplit>(t, valid, nc, ngmax);
    return valid;
}

/*! The target of this thread: thread i of the launch, or in list mode lane i % 32 of group groupList[i / 32], whose
 *  particles are [groupBounds[g], groupBounds[g + 1]) (GroupView slices of sph/include/sph/groups.hpp:96-103; a group
 *  is at most 32 particles). kSplit threads share a target; with kSplit > 1 every thread gets a usable target, with an
 *  empty list where there is no particle (false is returned). */
template<int kMode, int kSplit = 1, class T>
__device__ __forceinline__ bool chainTarget(const ChainArrays<T>& a, unsigned ngmax, Target& t)
{
    if constexpr (kMode & kModeList)
    {
        size_t thread = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) / kSplit;
        size_t slot   = thread >> 5;
        t.sub         = threadIdx.x % kSplit;
        bool valid    = slot < a.numListed;
        if (kSplit == 1 && !valid) { return false; }
        if (valid)
        {
            uint32_t g = __ldg(a.groupList + slot);
            t.i        = size_t(__ldg(a.groupBounds + g)) + (thread & 31);
            valid      = t.i < __ldg(a.groupBounds + g + 1);
        }
        if (kSplit == 1 && !valid) { return false; }
        fillTarget<kSplit>(t, valid, a.nc, ngmax);
        return valid;
    }
    else { return targetOf<kSplit>(a.n, a.nc, ngmax, t, (kMode & kModeBatch) ? a.batch.inst : nullptr); }
}

/*! Run term(j) over this lane's chunk of a round (chunk round * kSplit + sub): every neighbour of a full chunk in an
 *  unrolled body, or one neighbour per iteration (kRolled). */
template<int kSplit, bool kRolled, class F>
__device__ __forceinline__ void overChunk(const uint32_t* nidx, const Target& t, unsigned round, F&& term);

template<class T>
__device__ __forceinline__ AVFullRec<T> loadAV(const AVFullRec<T>* p)
{
    AVFullRec<T> r;
    if constexpr (sizeof(T) == 8)
    {
        const double4* q = reinterpret_cast<const double4*>(p);
        double4 a = ldg4(q), b = ldg4(q + 1);
        r = {a.x, a.y, a.z, a.w, b.x, b.y, T(0), T(0)};
    }
    else
    {
        float v[8];
        ldg256(p, v);
        r = {v[0], v[1], v[2], v[3], v[4], v[5], 0.f, 0.f};
    }
    return r;
}

__device__ __forceinline__ AVRec<float> loadAV(const AVRec<float>* p)
{
    float2 v = __ldg(reinterpret_cast<const float2*>(p));
    return {v.x, v.y};
}

__device__ __forceinline__ AVRec<double> loadAV(const AVRec<double>* p)
{
    double2 v = __ldg(reinterpret_cast<const double2*>(p));
    return {v.x, v.y};
}

template<class T>
__device__ __forceinline__ void loadDV(const DVRec<T>* p, T (&g)[6])
{
    if constexpr (sizeof(T) == 8)
    {
        const double2* q = reinterpret_cast<const double2*>(p);
        double2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
        g[0] = a.x, g[1] = a.y, g[2] = b.x, g[3] = b.y, g[4] = c.x, g[5] = c.y;
    }
    else
    {
        const float4* q = reinterpret_cast<const float4*>(p);
        float4 a = __ldg(q);
        float2 b = __ldg(reinterpret_cast<const float2*>(q + 1));
        g[0] = a.x, g[1] = a.y, g[2] = a.z, g[3] = a.w, g[4] = b.x, g[5] = b.y;
    }
}

/*! Additive AV-cleaning correction of rv = r . v_ij (momentum_energy_kern.hpp:43-63): the quadratic forms of both
 *  particles' symmetrised velocity gradients along r, damped by how far min(v_i, v_j) falls below eta_crit. */
template<class T>
__device__ __forceinline__ T avRvCorrection(T rx, T ry, T rz, T etaAb, T etaCrit, const T (&gi)[6], const T (&gj)[6])
{
    T dmy1 = dot3(rx, ry, rz, dot3(gi[0], gi[1], gi[2], rx, ry, rz), prodSum(gi[3], ry, gi[4], rz), gi[5] * rz);
    T dmy2 = dot3(rx, ry, rz, dot3(gj[0], gj[1], gj[2], rx, ry, rz), prodSum(gj[3], ry, gj[4], rz), gj[5] * rz);
    T dmy3 = T(1);
    if (etaAb < etaCrit)
    {
        T etaDiff = T(5) * (etaAb - etaCrit);
        dmy3      = exp(-etaDiff * etaDiff);
    }
    T aAb   = (dmy2 != T(0)) ? dmy1 / dmy2 : T(0);
    T aAbp1 = T(1) + aAb;
    T q     = T(4) * aAb / (aAbp1 * aAbp1);
    q       = q < T(1) ? q : T(1);
    q       = q > T(0) ? q : T(0);
    T phiAb = T(0.5) * dmy3 * q;
    return -phiAb * (dmy1 + dmy2);
}

//! the 8 neighbour indices of list chunk q0 / 8 of the target (two 16-byte loads of one sector)
__device__ __forceinline__ void loadChunk(const uint32_t* nidx, const Target& t, unsigned ngPad, unsigned q0,
                                          uint32_t (&js)[kNbChunk])
{
    const uint32_t* p = nidx + nidxAt(t.group, ngPad, q0, t.lane);
    // one 256-bit load of the chunk's sector; the lists are read once per kernel, so the streaming (evict-first)
    // hint keeps them from evicting the neighbour records in L2
    asm("ld.global.cs.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(js[0]), "=r"(js[1]), "=r"(js[2]), "=r"(js[3]), "=r"(js[4]), "=r"(js[5]), "=r"(js[6]), "=r"(js[7])
        : "l"(p));
}

/*! The next neighbour index of a list chunk: returns js[0] and shifts the rest down. Every index stays static, so
 *  the chunk stays in registers while a pair loop runs one pair per iteration instead of fully unrolled (the largest
 *  FP32 J-loop's unrolled 8-pair body overflowed the instruction cache). */
__device__ __forceinline__ uint32_t popChunk(uint32_t (&js)[kNbChunk])
{
    uint32_t j = js[0];
#pragma unroll
    for (unsigned r = 0; r + 1 < kNbChunk; ++r)
    {
        js[r] = js[r + 1];
    }
    return j;
}

template<int kSplit, bool kRolled, class F>
__device__ __forceinline__ void overChunk(const uint32_t* nidx, const Target& t, unsigned round, F&& term)
{
    unsigned q0 = (round * kSplit + t.sub) * kNbChunk;
    if (kSplit > 1 && q0 >= t.count) { return; }
    uint32_t js[kNbChunk];
    loadChunk(nidx, t, t.ngPad, q0, js);
    unsigned qn = min(kNbChunk, t.count - q0);
    if constexpr (kRolled)
    {
#pragma unroll 1
        for (unsigned q = 0; q < qn; ++q)
        {
            term(popChunk(js));
        }
    }
    else
    {
#pragma unroll
        for (unsigned q = 0; q < kNbChunk; ++q)
        {
            if (q >= qn) { break; }
            term(js[q]);
        }
    }
}

/*! Maximum (kMax) or minimum of one double per thread, published as ordered bits with one atomic per block on
 *  *single (one simulation), or one atomic per warp on the warp's instance slot batch.reduce[2 q + slot] (an ensemble:
 *  a warp never spans two instances). Every thread of the block must call it. */
template<bool kMax, bool kBatched>
__device__ __forceinline__ void reduceOrdered(double v, size_t n, unsigned long long* single, const BatchView& batch,
                                              int slot)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
    {
        double o = __shfl_xor_sync(0xffffffffu, v, off);
        v        = kMax ? fmax(v, o) : fmin(v, o);
    }
    if constexpr (kBatched)
    {
        size_t first = blockIdx.x * size_t(blockDim.x) + (threadIdx.x & ~31u);
        if ((threadIdx.x & 31) == 0 && first < n)
        {
            uint8_t q = batch.inst[first];
            if (q != kGhost)
            {
                if (kMax) { atomicMax(batch.reduce + 2 * q + slot, orderedBits(v)); }
                else { atomicMin(batch.reduce + 2 * q + slot, orderedBits(v)); }
            }
        }
        return;
    }
    __shared__ double warpVal[kChainMaxThreads / 32];
    if ((threadIdx.x & 31) == 0) { warpVal[threadIdx.x >> 5] = v; }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double m = warpVal[0];
        for (int w = 1; w < int(blockDim.x >> 5); ++w)
        {
            m = kMax ? fmax(m, warpVal[w]) : fmin(m, warpVal[w]);
        }
        if (kMax) { atomicMax(single, orderedBits(m)); }
        else { atomicMin(single, orderedBits(m)); }
    }
}

} // namespace chain
} // namespace sphb
