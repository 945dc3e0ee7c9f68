// SPH-VE kernel chain on sm_100a: XMass, VeDefGradh (+ ideal-gas EOS), IAD + divv/curlv, AV switches,
// momentum-energy. One thread per target particle; a warp is a group of 32 consecutive SFC-ordered particles whose
// neighbour lists are read slot-major (one coalesced line per slot). Each J-loop walks the list in stored (ascending)
// order, like the reference CPU loops, and reads neighbour data through the packed records of hydro.cuh.
//
// T = double: the plain FP64 drop-in. Positions are FP64 and the periodic shift is the reference's. Sums run over blocks of
// 8 neighbours in list order, whose partial sums are added in list order. The pair terms are the reference's up to
// algebra that keeps FP64 rounding (a reciprocal for a division, a constant factor taken out of a sum), so results differ
// from the reference CPU by rounding, 1e-15 of a force.
//
// T = float: the mixed form. Pair separations come from 32-bit fixed-point coordinates (exact integer differences,
// periodic wrap by overflow; one unit = L / 2^32), all pair arithmetic is FP32, the kernel W is a degree-12
// polynomial instead of a table, and every neighbour sum is block-compensated: plain FP32 partial sums over blocks of
// 8 neighbours, each added to a Kahan-compensated FP32 accumulator.
#include "chain_detail.cuh"
#include "hydro.cuh"
#include "neighbors.cuh"
#include "primitives.cuh"

namespace sphb
{

namespace
{

using namespace chain;

constexpr int kSplitThreads = 128; // block size of the launches whose lanes share targets
// launches of at most so many targets take eight or four lanes per target (chainSplit)
constexpr size_t kEightLaneTargets = 16384;
constexpr size_t kFourLaneTargets  = 65536;


// ---------------------------------------------------------------------------------------------------------------
// XMass: rho0_i = (m_i + sum_j W_ij m_j) K / h_i^3, xm_i = m_i / rho0_i (sph/include/sph/hydro_ve/xmass_kern.hpp:50-79)
// ---------------------------------------------------------------------------------------------------------------
// FP32: at most 32 registers, eight 256-thread blocks per SM: more gathers in flight (0.348 -> 0.325 ms at 128^3)
template<class T, int kMode, int kSplit>
__global__ void __launch_bounds__(kChainMaxThreads, sizeof(T) == 4 && kSplit == 1 ? 8 : 0)
    xmassKernel(ChainArrays<T> a, HydroConsts<T> k, DevBox box)
{
    Target t;
    const bool valid = chainTarget<kMode, kSplit>(a, k.ngmax, t);
    if (kSplit == 1 && !valid) { return; }
    Pos<T> pi  = posOf(a, t.i);
    double hiD = a.h[t.i];
    T hi       = T(hiD);
    T mi       = T(pi.m);
    T hInv     = T(1.0) / hi;
    T h3Inv    = hInv * hInv * hInv;
    T hh       = T(0.5) * hInv * hInv;

    BlockSum<T> rho0(mi);
    for (unsigned round = 0; round < t.rounds; ++round)
    {
        overChunk<kSplit, false>(a.nidx, t, round, [&](uint32_t j) {
            Pos<T> pj  = posOf(a, j);
            Sep<T> r   = separation(pi, pj, 2.0 * hiD, box, k);
            T r2       = dot3(r.rx, r.ry, r.rz, r.rx, r.ry, r.rz);
            rho0.add(kernelWr2(a.wh, k, r2, hInv, hh) * T(pj.m));
        });
        foldChunks<kSplit>(round * kSplit, t.numChunks, rho0);
    }
    if (kSplit > 1 && (!valid || t.sub != 0)) { return; }
    a.xm[t.i] = mi / (rho0.get() * k.K * h3Inv);
}

// ---------------------------------------------------------------------------------------------------------------
// VeDefGradh (sph/include/sph/hydro_ve/ve_def_gradh_kern.hpp:43-90) + ideal-gas EOS (hydro_ve/eos.hpp:52-94,
// sph/include/sph/eos.hpp:19-50); writes kx, gradh, prho, c and the hydro record of the particle.
// ---------------------------------------------------------------------------------------------------------------
// FP32: at most 40 registers, six 256-thread blocks per SM, for the gathers' latency (0.625 -> 0.566 ms at 128^3,
// though it spills a little; 48 registers gave 0.588, 32 gave 0.582)
template<class T, int kMode, int kSplit>
__global__ void __launch_bounds__(kChainMaxThreads, sizeof(T) == 4 && kSplit == 1 ? 6 : 0)
    veDefGradhEosKernel(ChainArrays<T> a, HydroConsts<T> k, DevBox box)
{
    Target t;
    const bool valid = chainTarget<kMode, kSplit>(a, k.ngmax, t);
    if (kSplit == 1 && !valid) { return; }
    Pos<T> pi  = posOf(a, t.i);
    double hiD = a.h[t.i];
    T hi       = T(hiD);
    T mi       = T(pi.m);
    T xmassi   = a.xm[t.i];
    T hInv     = T(1) / hi;
    T h3Inv    = hInv * hInv * hInv;
    [[maybe_unused]] float hhV = 0.5f * float(hInv) * float(hInv);

    BlockSum<T> kxS(xmassi), whomegaS(-T(3) * xmassi), wrho0S(-T(3) * mi);
    for (unsigned round = 0; round < t.rounds; ++round)
    {
        overChunk<kSplit, false>(a.nidx, t, round, [&](uint32_t j) {
            Pos<T> pj  = posOf(a, j);
            Sep<T> r   = separation(pi, pj, 2.0 * hiD, box, k);
            T r2       = dot3(r.rx, r.ry, r.rz, r.rx, r.ry, r.rz);
            T w, dterh;
            if constexpr (sizeof(T) == 4)
            {
                if (k.usePoly)
                {
                    // t = v^2/2 - 1 from r2 (no square root); W and dW's polynomial side by side in packed FP32
                    // (sm_100 FFMA2); v dW = v^2 P'(t) = 2 (t + 1) P'(t) (0.638 -> 0.624 ms at 128^3)
                    float tt   = fmaf(r2, hhV, -1.0f);
                    float2 acc = make_float2(k.wpoly[kPolyTerms - 1], k.dwpoly[kPolyTerms - 1]);
#pragma unroll
                    for (int p = kPolyTerms - 2; p >= 0; --p)
                    {
                        acc = __ffma2_rn(acc, make_float2(tt, tt), make_float2(k.wpoly[p], k.dwpoly[p]));
                    }
                    bool in = tt < 1.0f;
                    w       = in ? acc.x : 0.0f;
                    dterh   = in ? -prodSum(3.0f, acc.x, 2.0f * (tt + 1.0f), acc.y) : 0.0f;
                }
                else
                {
                    T vloc = T(r2 * rsqrtf(float(r2))) * hInv;
                    w      = kernelW(a.wh, k, vloc);
                    dterh  = -prodSum(T(3), w, vloc, kernelDW(a.whd, k, vloc));
                }
            }
            else
            {
                T vloc = T(sqrt(r2)) * hInv;
                w      = kernelW(a.wh, k, vloc);
                T dw   = kernelDW(a.whd, k, vloc);
                dterh  = -prodSum(T(3), w, vloc, dw);
            }
            T xmassj   = __ldg(a.xm + j);
            kxS.add(w * xmassj);
            whomegaS.add(dterh * xmassj);
            wrho0S.add(dterh * T(pj.m));
        });
        foldChunks<kSplit>(round * kSplit, t.numChunks, kxS, whomegaS, wrho0S);
    }
    if (kSplit > 1 && (!valid || t.sub != 0)) { return; }
    T kxi      = kxS.get() * (k.K * h3Inv);
    T whomegai = whomegaS.get() * (k.K * h3Inv * hInv);
    T wrho0i   = wrho0S.get() * (k.K * h3Inv * hInv);
    if constexpr (kMode & kModeTape)
    {
        a.tape.whomega[t.i] = whomegai;
        a.tape.wrho0[t.i]   = wrho0i;
    }
    whomegai   = fma(fma(-(k.K * xmassi), h3Inv, kxi), wrho0i, whomegai * mi / xmassi);
    T rhoi     = kxi * mi / xmassi;
    T dhdrho   = -hi / (rhoi * T(3));
    T gradhi   = fma(-dhdrho, whomegai, T(1));

    // EOS in FP64 (per particle): rho = kx m / xm, p = rho u (gamma - 1), c = sqrt(gamma u (gamma - 1))
    double gamma = k.gamma, cv = k.cv;
    if constexpr (kMode & kModeBatch)
    {
        uint8_t q = a.batch.inst[t.i];
        gamma     = a.batch.gamma[q];
        cv        = a.batch.cv[q];
    }
    double rho  = double(kxi) * double(mi) / double(xmassi);
    double u    = cv * a.temp[t.i];
    double tmp  = u * (gamma - 1.0);
    double p    = rho * tmp;
    double c    = sqrt(gamma * tmp);
    double prho = p / (double(kxi) * double(mi) * double(mi) * double(gradhi));

    a.kx[t.i]    = kxi;
    a.gradh[t.i] = gradhi;
    a.prho[t.i]  = T(prho);
    a.c[t.i]     = T(c);
    if (a.recordNoVelocity)
    {
        a.hrec[t.i] = HydroRec<T>{T(0), T(0), T(0), T(1) / hi, xmassi, xmassi / kxi, T(c), T(prho)};
    }
    else
    {
        a.hrec[t.i] = HydroRec<T>{T(a.vx[t.i]), T(a.vy[t.i]), T(a.vz[t.i]), T(1) / hi, xmassi, xmassi / kxi, T(c),
                                  T(prho)};
    }
}

//! the velocity part of the hydro record, the same values VeDefGradh writes there otherwise
template<class T>
__global__ void packVelocityKernel(size_t n, const double* __restrict__ vx, const double* __restrict__ vy,
                                   const double* __restrict__ vz, HydroRec<T>* __restrict__ hrec)
{
    size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i >= n) { return; }
    hrec[i].vx = T(vx[i]);
    hrec[i].vy = T(vy[i]);
    hrec[i].vz = T(vz[i]);
}

template<class T>
__device__ __forceinline__ int expOf(T v)
{
    return v == T(0) ? 0 : ilogb(v);
}

/*! IAD + divv/curlv (sph/include/sph/hydro_ve/iad_kern.hpp:43-110, then divv_curlv_kern.hpp:43-123 with the
 *  particle's own c_ij) in one pass over the list; also the running max of divv for the rho time step. The divv/curlv loop of the reference sums, per pair,
 *  f_a tA_b with f = (v_j - v_i) xm_j and tA = -(C_i r) W, i.e. dV_ab = -sum_c C_bc M_ac with
 *  M_ac = sum_j f_a r_c W: M is accumulated in the same pass as tau, and C_i, known only after the pass, is applied
 *  to the nine sums at the end. Same quantities, one gather of each neighbour instead of two. */
// FP32: at most 80 registers (three 256-thread blocks per SM), as MomentumEnergy: measured 1.04 -> 0.95 ms at 128^3
// against 87 registers. FP64 ran the two list passes of the reference before, bound by its FP64 pipe and the second
// gather: 2.10 -> 1.16 ms at 101^3.
template<class T, int kMode, int kSplit>
__global__ void __launch_bounds__(kChainMaxThreads, sizeof(T) == 4 && kSplit == 1 ? 3 : 0)
    iadDivvCurlvFusedKernel(ChainArrays<T> a, HydroConsts<T> k, DevBox box)
{
    Target t;
    const bool valid = chainTarget<kMode, kSplit>(a, k.ngmax, t);
    double divvOut   = -INFINITY;
    BlockSum<T> s11, s12, s13, s22, s23, s33;
    BlockSum<T> mxx, mxy, mxz, myx, myy, myz, mzx, mzy, mzz;
    T vsigI = T(0);
    [[maybe_unused]] int vsigJ = -1;
    if (kSplit > 1 || valid)
    {
        Pos<T> pi      = posOf(a, t.i);
        double hiD     = a.h[t.i];
        T hi           = T(hiD);
        T hiInv        = T(1) / hi;
        T hh           = T(0.5) * hiInv * hiInv;
        HydroRec<T> hr = a.hrec[t.i];
        vsigI          = T(1.e-40) * hr.c;
        for (unsigned round = 0; round < t.rounds; ++round)
        {
            overChunk<kSplit, false>(a.nidx, t, round, [&](uint32_t j) {
                Pos<T> pj      = posOf(a, j);
                HydroRec<T> hj = loadHydro(a.hrec + j);
                Sep<T> r       = separation(pi, pj, 2.0 * hiD, box, k);
                T r2           = dot3(r.rx, r.ry, r.rz, r.rx, r.ry, r.rz);
                T dvx = hj.vx - hr.vx, dvy = hj.vy - hr.vy, dvz = hj.vz - hr.vz;
                T rv  = dot3(r.rx, r.ry, r.rz, dvx, dvy, dvz);
                T rinv, w;
                if constexpr (sizeof(T) == 4)
                {
                    rinv = rsqrtf(r2);
                    w    = kernelWr2(a.wh, k, r2, hiInv, hh);
                }
                else
                {
                    rinv = rsqrt(r2);
                    w    = kernelW(a.wh, k, r2 * rinv * hiInv);
                }
                // the AV switches' signal velocity c_i + c_j - 3 r.v_ij / r over approaching pairs
                T vsig = rv > T(0) ? fma(T(3) * rv, rinv, hr.c + hj.c) : T(0);
                if constexpr (kMode & kModeTape)
                {
                    if (!(vsigI > vsig)) { vsigJ = int(j); }
                }
                vsigI   = vsigI > vsig ? vsigI : vsig;
                T voljW = hj.vol * w;
                s11.add(r.rx * r.rx * voljW);
                s12.add(r.rx * r.ry * voljW);
                s13.add(r.rx * r.rz * voljW);
                s22.add(r.ry * r.ry * voljW);
                s23.add(r.ry * r.rz * voljW);
                s33.add(r.rz * r.rz * voljW);
                T xw = hj.xm * w;
                T fx = dvx * xw;
                T fy = dvy * xw;
                T fz = dvz * xw;
                mxx.add(fx * r.rx);
                mxy.add(fx * r.ry);
                mxz.add(fx * r.rz);
                myx.add(fy * r.rx);
                myy.add(fy * r.ry);
                myz.add(fy * r.rz);
                mzx.add(fz * r.rx);
                mzy.add(fz * r.ry);
                mzz.add(fz * r.rz);
            });
            foldChunks<kSplit>(round * kSplit, t.numChunks, s11, s12, s13, s22, s23, s33, mxx, mxy, mxz, myx, myy, myz,
                               mzx, mzy, mzz);
        }
        vsigI = maxOverSplit<kSplit>(vsigI);
    }
    if (valid && t.sub == 0)
    {
        T hi           = T(a.h[t.i]);
        T hiInv        = T(1) / hi;
        HydroRec<T> hr = a.hrec[t.i];
        T tau11 = s11.get(), tau12 = s12.get(), tau13 = s13.get();
        T tau22 = s22.get(), tau23 = s23.get(), tau33 = s33.get();
        int expSum = expOf(tau11) + expOf(tau12) + expOf(tau13) + expOf(tau22) + expOf(tau23) + expOf(tau33);
        T norm     = ldexp(T(1), -expSum / 6);
        tau11 *= norm;
        tau12 *= norm;
        tau13 *= norm;
        tau22 *= norm;
        tau23 *= norm;
        tau33 *= norm;
        T det = prodSum(tau11 * tau22, tau33, T(2) * tau12 * tau23, tau13);
        det   = fma(-(tau11 * tau23), tau23, det);
        det   = fma(-(tau22 * tau13), tau13, det);
        det   = fma(-(tau33 * tau12), tau12, det);
        T factor = norm * (hi * hi * hi) / (det * k.K);
        if (isnan(factor) && t.count == 0) { factor = T(0); }
        T c11i = prodDiff(tau22, tau33, tau23, tau23) * factor;
        T c12i = prodDiff(tau13, tau23, tau33, tau12) * factor;
        T c13i = prodDiff(tau12, tau23, tau22, tau13) * factor;
        T c22i = prodDiff(tau11, tau33, tau13, tau13) * factor;
        T c23i = prodDiff(tau13, tau12, tau11, tau23) * factor;
        T c33i = fma(-tau12, tau12, tau11 * tau22) * factor;

        // dV_ab = -sum_c C_bc M_ac
        T M[3][3] = {{mxx.get(), mxy.get(), mxz.get()}, {myx.get(), myy.get(), myz.get()},
                     {mzx.get(), mzy.get(), mzz.get()}};
        T C[3][3] = {{c11i, c12i, c13i}, {c12i, c22i, c23i}, {c13i, c23i, c33i}};
        T dV[3][3];
#pragma unroll
        for (int p = 0; p < 3; ++p)
        {
#pragma unroll
            for (int q = 0; q < 3; ++q)
            {
                dV[p][q] = -dot3(C[q][0], C[q][1], C[q][2], M[p][0], M[p][1], M[p][2]);
            }
        }
        T hiInv3 = hiInv * hiInv * hiInv;
        T normKx = k.K * hiInv3 / a.kx[t.i];
        T divv   = normKx * (dV[0][0] + dV[1][1] + dV[2][2]);
        T cx     = dV[2][1] - dV[1][2];
        T cy     = dV[0][2] - dV[2][0];
        T cz     = dV[1][0] - dV[0][1];
        T curlv  = normKx * sqrt(dot3(cx, cy, cz, cx, cy, cz));
        if constexpr (kMode & kModeAvClean)
        {
            DVRec<T> g{{normKx * dV[0][0], normKx * (dV[0][1] + dV[1][0]), normKx * (dV[0][2] + dV[2][0]),
                        normKx * dV[1][1], normKx * (dV[1][2] + dV[2][1]), normKx * dV[2][2]},
                       T(0),
                       T(0)};
            a.dvrec[t.i] = g;
#pragma unroll
            for (int q = 0; q < 6; ++q)
            {
                a.dv[q][t.i] = g.dv[q];
            }
        }

        a.cij[0][t.i] = c11i;
        a.cij[1][t.i] = c12i;
        a.cij[2][t.i] = c13i;
        a.cij[3][t.i] = c22i;
        a.cij[4][t.i] = c23i;
        a.cij[5][t.i] = c33i;
        a.divv[t.i]   = divv;
        a.curlv[t.i]  = curlv;
        a.grec[t.i]   = GradRec<T>{c11i, c12i, c13i, c22i, c23i, c33i, divv, T(a.alpha[t.i])};
        a.avrec[t.i]  = AVRec<T>{hr.vol, divv};
        a.vsig[t.i]   = vsigI;
        if constexpr (kMode & kModeTape) { a.tape.vsigJ[t.i] = vsigJ; }
        divvOut       = double(divv);
    }
    reduceOrdered<true, (kMode & kModeBatch) != 0>(divvOut, a.n, a.reduce + 0, a.batch, 0);
}

// ---------------------------------------------------------------------------------------------------------------
// AV switches (sph/include/sph/hydro_ve/av_switches_kern.hpp:43-137)
// ---------------------------------------------------------------------------------------------------------------
// The signal velocity comes from IAD's loop, so a neighbour costs a 16-byte position and an 8-byte record here instead of
// a 32-byte one with velocity and sound speed (the loop was bound by its gathers, at 90 % of the L1's throughput): FP32
// 0.760 -> 0.476 ms at 128^3 for 0.142 ms more in IAD, FP64 1.24 -> 0.70 ms at 101^3 for 0.02.
// FP32: up to 384 threads, run in 384-thread blocks (12 consecutive groups sharing their neighbours in L1); at most 56
// registers for three such blocks per SM. FP64 keeps the common bound with no block minimum.
template<class T, int kMode, int kSplit>
__global__ void __launch_bounds__(sizeof(T) == 4 ? kAvMaxThreads : kChainMaxThreads, sizeof(T) == 4 && kSplit == 1 ? 3 : 0)
    avSwitchesKernel(ChainArrays<T> a, HydroConsts<T> k, DevBox box, double dt)
{
    Target t;
    const bool valid = chainTarget<kMode, kSplit>(a, k.ngmax, t);
    if (kSplit == 1 && !valid) { return; }
    Pos<T> pi      = posOf(a, t.i);
    double hiD     = a.h[t.i];
    HydroRec<T> hr = a.hrec[t.i];
    GradRec<T> gr  = a.grec[t.i];
    T hi           = T(hiD);
    T ci           = hr.c;
    T vijsignalI   = (kMode & kModeFullAv) ? T(1.e-40) * ci : a.vsig[t.i];
    T hiInv        = T(1) / hi;
    T hiInv3       = hiInv * hiInv * hiInv;
    T KhiInv3      = k.K * hiInv3;
    T hh           = T(0.5) * hiInv * hiInv;
    T divvI        = gr.divv;

    BlockSum<T> gx, gy, gz;
    for (unsigned round = 0; round < t.rounds; ++round)
    {
        overChunk<kSplit, false>(a.nidx, t, round, [&](uint32_t j) {
            Pos<T> pj = posOf(a, j);
            T volJ, divvJ;
            Sep<T> r  = separation(pi, pj, 2.0 * hiD, box, k);
            T r2      = dot3(r.rx, r.ry, r.rz, r.rx, r.ry, r.rz);
            if constexpr (kMode & kModeFullAv)
            {
                AVFullRec<T> hj = loadAV(a.avfull + j);
                volJ            = hj.vol;
                divvJ           = hj.divv;
                T rv            = dot3(r.rx, r.ry, r.rz, hj.vx - hr.vx, hj.vy - hr.vy, hj.vz - hr.vz);
                T rinv;
                if constexpr (sizeof(T) == 4) { rinv = rsqrtf(r2); }
                else { rinv = rsqrt(r2); }
                T vsig     = rv > T(0) ? fma(T(3) * rv, rinv, ci + hj.c) : T(0);
                vijsignalI = vijsignalI > vsig ? vijsignalI : vsig;
            }
            else
            {
                AVRec<T> hj = loadAV(a.avrec + j);
                volJ        = hj.vol;
                divvJ       = hj.divv;
            }
            T W = kernelWr2(a.wh, k, r2, hiInv, hh);
            // sum fac W r and apply -C_i once after the loop (the same vector, 9 FMAs less per pair)
            T sw = volJ * (divvI - divvJ) * (KhiInv3 * W);
            gx.add(sw * r.rx);
            gy.add(sw * r.ry);
            gz.add(sw * r.rz);
        });
        foldChunks<kSplit>(round * kSplit, t.numChunks, gx, gy, gz);
    }
    if constexpr (kMode & kModeFullAv) { vijsignalI = maxOverSplit<kSplit>(vijsignalI); }
    if (kSplit > 1 && (!valid || t.sub != 0)) { return; }
    T gdx = gx.get(), gdy = gy.get(), gdz = gz.get();
    {
        T sx = gdx, sy = gdy, sz = gdz;
        gdx  = -fma(gr.c13, sz, fma(gr.c12, sy, gr.c11 * sx));
        gdy  = -fma(gr.c23, sz, fma(gr.c22, sy, gr.c12 * sx));
        gdz  = -fma(gr.c33, sz, fma(gr.c23, sy, gr.c13 * sx));
    }
    T graddivv = sqrt(dot3(gdx, gdy, gdz, gdx, gdy, gdz));
    if constexpr (kMode & kModeTape)
    {
        a.tape.gx[t.i]    = gdx;
        a.tape.gy[t.i]    = gdy;
        a.tape.gz[t.i]    = gdz;
        a.tape.vsig[t.i]  = vijsignalI;
    }
    T alphaI   = T(a.alpha[t.i]);
    T alphaloc = T(0);
    if (divvI < T(0))
    {
        T aConst = hi * hi * graddivv;
        alphaloc = k.alphamax * aConst / fma(T(0.05), ci, fma(hi, fabs(divvI), aConst));
    }
    if (alphaloc >= alphaI) { alphaI = alphaloc; }
    else
    {
        T decay    = hi / (k.decay * vijsignalI);
        T alphadot = alphaloc >= k.alphamin ? (alphaloc - alphaI) / decay : (k.alphamin - alphaI) / decay;
        double dtq = dt;
        if constexpr (kMode & kModeBatch) { dtq = a.batch.dt[a.batch.inst[t.i]]; }
        alphaI = fma(alphadot, T(dtq), alphaI);
    }
    a.alpha[t.i]      = double(alphaI);
    a.grec[t.i].alpha = alphaI; // the alpha slot of the record is not read by this kernel
}

// ---------------------------------------------------------------------------------------------------------------
// Momentum and energy (sph/include/sph/hydro_ve/momentum_energy_kern.hpp:65-222, avClean = false;
// artificial_viscosity sph/include/sph/kernels.hpp:71-85) with the Courant time step per particle
// (tsKCourant, kernels.hpp:10-17) reduced to the minimum.
// ---------------------------------------------------------------------------------------------------------------
// FP64 is bound by its FP64 pipe. It ran five divisions and a square root per pair (and four powers on the Atwood
// ramp); with one rsqrt, the densities compared as |rho_i vol_j - m_j| and the loop rolled it takes 2.12 instead of
// 3.98 ms at 101^3, the result unchanged to 4e-15.
// FP32 without AV cleaning: at most 80 registers (three 256-thread blocks per SM) keeps more warps resident for the
// gathers; measured 2.11 -> 2.05 ms at 128^3 against 96 registers (the AV-cleaning form would spill)
template<class T, int kMode, int kSplit>
__global__ void __launch_bounds__(kChainMaxThreads, (sizeof(T) == 4 && kSplit == 1 && !(kMode & kModeAvClean)) ? 3 : 1)
    momentumEnergyKernel(ChainArrays<T> a, HydroConsts<T> k, DevBox box)
{
    Target t;
    const bool valid = chainTarget<kMode, kSplit>(a, k.ngmax, t);
    double dtMin     = INFINITY;
    if (kSplit > 1 || valid)
    {
        Pos<T> pi      = posOf(a, t.i);
        double hiD     = a.h[t.i];
        HydroRec<T> hr = a.hrec[t.i];
        GradRec<T> gr  = a.grec[t.i];
        T hi          = T(hiD);
        T mi          = T(pi.m);
        T ci          = hr.c;
        T kxi         = a.kx[t.i];
        T alphaI      = gr.alpha;
        T xmassi      = hr.xm;
        // FP32: log2 xm_i for the Atwood ramp's xm_i^(2-s) xm_j^s = exp2((2-s) log2 xm_i + s log2 xm_j)
        T lxi         = sizeof(T) == 4 ? T(log2f(float(xmassi))) : T(0);
        T rhoi        = kxi * mi / xmassi;
        T invRhoi     = T(1) / rhoi;
        T prhoi       = hr.prho;
        T hiInv       = T(1) / hi;
        T hiInv3      = hiInv * hiInv * hiInv;
        T maxvsignalI = T(0);
        BlockSum<T> momX, momY, momZ, energyS, aViscE;
        [[maybe_unused]] T gradVi[6];
        [[maybe_unused]] T etaCrit = T(0);
        if constexpr (kMode & kModeAvClean)
        {
            loadDV(a.dvrec + t.i, gradVi);
            etaCrit = T(cbrt(32.0 * M_PI / 3.0 / double(t.count + 1)));
        }

        // the term of one neighbour j, added to the five sums
        auto pairTerm = [&](uint32_t j) {
            if constexpr (sizeof(T) == 4 && !(kMode & kModeAvClean))
            {
                // FP32: the i and j halves of the pair side by side in packed FP32 (sm_100 FFMA2/FMUL2): the IAD
                // gradients tA = -(C r) W, their products with v_ij and the momentum coefficients. The viscous
                // term joins the momentum sums as (m_j prho_i a_mom + aVisc/2) tA_i + (m_j prho_j b_mom + bVisc/2)
                // tA_j (1.54 -> 1.48 ms at 128^3; the errors against FP64 unchanged). The ensemble's batch form
                // takes the same body, so that its members stay bit-identical to single simulations (it spills a
                // little there: 4.97 ms per step for 64 members, against 4.84 with the scalar body)
                Pos<T> pj      = posOf(a, j);
                HydroRec<T> hj = loadHydro(a.hrec + j);
                GradRec<T> gj  = loadGrad(a.grec + j);
                Sep<T> r       = separation(pi, pj, 2.0 * hiD, box, k);
                float r2       = dot3(r.rx, r.ry, r.rz, r.rx, r.ry, r.rz);
                float rinv     = rsqrtf(r2);
                float dist     = r2 * rinv;
                float vxij     = hr.vx - hj.vx;
                float vyij     = hr.vy - hj.vy;
                float vzij     = hr.vz - hj.vz;

                float v1 = dist * hiInv, v2 = dist * hj.hInv;
                float hjInv3 = hj.hInv * hj.hInv * hj.hInv;
                float2 W = make_float2(-hiInv3 * kernelW(a.wh, k, v1), -hjInv3 * kernelW(a.wh, k, v2));

                // tA = -(C r) W of i and j side by side
                float2 RX  = make_float2(r.rx, r.rx), RY = make_float2(r.ry, r.ry), RZ = make_float2(r.rz, r.rz);
                float2 tA1 = __ffma2_rn(make_float2(gr.c13, gj.c13), RZ,
                                        __ffma2_rn(make_float2(gr.c12, gj.c12), RY,
                                                   __fmul2_rn(make_float2(gr.c11, gj.c11), RX)));
                float2 tA2 = __ffma2_rn(make_float2(gr.c23, gj.c23), RZ,
                                        __ffma2_rn(make_float2(gr.c22, gj.c22), RY,
                                                   __fmul2_rn(make_float2(gr.c12, gj.c12), RX)));
                float2 tA3 = __ffma2_rn(make_float2(gr.c33, gj.c33), RZ,
                                        __ffma2_rn(make_float2(gr.c23, gj.c23), RY,
                                                   __fmul2_rn(make_float2(gr.c13, gj.c13), RX)));
                tA1 = __fmul2_rn(tA1, W);
                tA2 = __fmul2_rn(tA2, W);
                tA3 = __fmul2_rn(tA3, W);

                float mj     = float(pj.m);
                float cj     = hj.c;
                float xmassj = hj.xm;
                float rhoj   = fdiv(mj, hj.vol);
                float rv     = dot3(r.rx, r.ry, r.rz, vxij, vyij, vzij);
                float wij    = rv * rinv;
                float visc   = 0.0f;
                if (wij < 0.0f)
                {
                    float vijSignal = fmaf((alphaI + gj.alpha) * 0.25f, ci + cj, -2.0f * wij);
                    visc            = -vijSignal * wij;
                }
                float vijsignal = 0.5f * (ci + cj) - 2.0f * wij;
                maxvsignalI     = vijsignal > maxvsignalI ? vijsignal : maxvsignalI;

                float aMom, bMom;
                float dRho = fabsf(rhoi - rhoj), sRho = rhoi + rhoj;
                if (dRho < k.Atmin * sRho)
                {
                    aMom = xmassi * xmassi;
                    bMom = xmassj * xmassj;
                }
                else if (dRho > k.Atmax * sRho)
                {
                    aMom = xmassi * xmassj;
                    bMom = aMom;
                }
                else
                {
                    float sigma = k.ramp * (fdiv(dRho, sRho) - k.Atmin);
                    float lxj   = log2f(xmassj);
                    aMom        = exp2f(prodSum(sigma, lxj, 2.0f - sigma, lxi));
                    bMom        = exp2f(prodSum(sigma, lxi, 2.0f - sigma, lxj));
                }
                float aVisc = mj * invRhoi * visc;
                float bVisc = hj.vol * visc;
                // (tA_i . v_ij, tA_j . v_ij)
                float2 dv = __ffma2_rn(tA3, make_float2(vzij, vzij),
                                       __ffma2_rn(tA2, make_float2(vyij, vyij),
                                                  __fmul2_rn(tA1, make_float2(vxij, vxij))));
                aViscE.add(0.5f * prodSum(aVisc, dv.x, bVisc, dv.y));
                energyS.add(mj * aMom * dv.x);
                float cI = prodSum(0.5f, aVisc, mj * prhoi, aMom);
                float cJ = prodSum(0.5f, bVisc, mj * hj.prho, bMom);
                momX.add(prodSum(cI, tA1.x, cJ, tA1.y));
                momY.add(prodSum(cI, tA2.x, cJ, tA2.y));
                momZ.add(prodSum(cI, tA3.x, cJ, tA3.y));
            }
            else
            {
                Pos<T> pj      = posOf(a, j);
                HydroRec<T> hj = loadHydro(a.hrec + j);
                GradRec<T> gj  = loadGrad(a.grec + j);
                Sep<T> r       = separation(pi, pj, 2.0 * hiD, box, k);
                T r2           = dot3(r.rx, r.ry, r.rz, r.rx, r.ry, r.rz);
                // 1/r from one rsqrt (r and w_ij = r.v / r without a square root or a division), m_j / rho_j as
                // vol_j, and the Atwood thresholds compared without a division (FP32: 1.68 -> 1.58 ms at 128^3; the
                // errors against FP64 unchanged)
                T rinv;
                if constexpr (sizeof(T) == 4) { rinv = rsqrtf(r2); }
                else { rinv = rsqrt(r2); }
                T dist         = r2 * rinv;
                T vxij         = hr.vx - hj.vx;
                T vyij         = hr.vy - hj.vy;
                T vzij         = hr.vz - hj.vz;
                T v1           = dist * hiInv;
                T v2           = dist * hj.hInv;
                T hjInv3       = hj.hInv * hj.hInv * hj.hInv;
                T Wi           = hiInv3 * kernelW(a.wh, k, v1);
                T Wj           = hjInv3 * kernelW(a.wh, k, v2);

                T tA1i = -dot3(gr.c11, gr.c12, gr.c13, r.rx, r.ry, r.rz) * Wi;
                T tA2i = -dot3(gr.c12, gr.c22, gr.c23, r.rx, r.ry, r.rz) * Wi;
                T tA3i = -dot3(gr.c13, gr.c23, gr.c33, r.rx, r.ry, r.rz) * Wi;
                T tA1j = -dot3(gj.c11, gj.c12, gj.c13, r.rx, r.ry, r.rz) * Wj;
                T tA2j = -dot3(gj.c12, gj.c22, gj.c23, r.rx, r.ry, r.rz) * Wj;
                T tA3j = -dot3(gj.c13, gj.c23, gj.c33, r.rx, r.ry, r.rz) * Wj;

                T mj     = T(pj.m);
                T cj     = hj.c;
                T xmassj = hj.xm;

                T rv   = dot3(r.rx, r.ry, r.rz, vxij, vyij, vzij);
                if constexpr (kMode & kModeAvClean)
                {
                    T gradVj[6];
                    loadDV(a.dvrec + j, gradVj);
                    rv += avRvCorrection(r.rx, r.ry, r.rz, v1 < v2 ? v1 : v2, etaCrit, gradVi, gradVj);
                }
                T wij  = rv * rinv;
                T visc = T(0);
                if (wij < T(0))
                {
                    T vijSignal = fma((alphaI + gj.alpha) * T(0.25), ci + cj, T(-2) * wij);
                    visc        = -vijSignal * wij;
                }
                T vijsignal = T(0.5) * (ci + cj) - T(2) * wij;
                maxvsignalI = vijsignal > maxvsignalI ? vijsignal : maxvsignalI;

                // |rho_i - rho_j| against A (rho_i + rho_j); FP64: both times vol_j = m_j / rho_j, without a division
                T aMom, bMom;
                T dRho, sRho;
                if constexpr (sizeof(T) == 4)
                {
                    T rhoj = fdiv(mj, hj.vol);
                    dRho   = fabs(rhoi - rhoj);
                    sRho   = rhoi + rhoj;
                }
                else
                {
                    T rhoiVol = rhoi * hj.vol;
                    dRho      = fabs(rhoiVol - mj);
                    sRho      = rhoiVol + mj;
                }
                if (dRho < k.Atmin * sRho)
                {
                    aMom = xmassi * xmassi;
                    bMom = xmassj * xmassj;
                }
                else if (dRho > k.Atmax * sRho)
                {
                    aMom = xmassi * xmassj;
                    bMom = aMom;
                }
                else
                {
                    T sigma = k.ramp * (fdiv(dRho, sRho) - k.Atmin);
                    if constexpr (sizeof(T) == 4)
                    {
                        T lxj = log2f(xmassj);
                        aMom  = exp2f(prodSum(sigma, lxj, T(2) - sigma, lxi));
                        bMom  = exp2f(prodSum(sigma, lxi, T(2) - sigma, lxj));
                    }
                    else
                    {
                        // xm_i^(2-s) xm_j^s = xm_i^2 q and xm_j^(2-s) xm_i^s = xm_j^2 / q with q = (xm_j / xm_i)^s:
                        // one logarithm and one exponential instead of four powers
                        T q  = exp(sigma * log(xmassj / xmassi));
                        aMom = xmassi * xmassi * q;
                        bMom = xmassj * xmassj / q;
                    }
                }

                T aVisc  = mj * invRhoi * visc;
                T bVisc  = hj.vol * visc;
                T viscX = prodSum(aVisc, tA1i, bVisc, tA1j);
                T viscY = prodSum(aVisc, tA2i, bVisc, tA2j);
                T viscZ = prodSum(aVisc, tA3i, bVisc, tA3j);
                aViscE.add(dot3(T(0.5) * viscX, T(0.5) * viscY, T(0.5) * viscZ, vxij, vyij, vzij));
                energyS.add(mj * aMom * dot3(vxij, vyij, vzij, tA1i, tA2i, tA3i));
                T momI = mj * prhoi * aMom;
                T momJ = mj * hj.prho * bMom;
                momX.add(fma(T(0.5), viscX, prodSum(momI, tA1i, momJ, tA1j)));
                momY.add(fma(T(0.5), viscY, prodSum(momI, tA2i, momJ, tA2j)));
                momZ.add(fma(T(0.5), viscZ, prodSum(momI, tA3i, momJ, tA3j)));
            }
        };
        // one pair per iteration: the unrolled 8-pair body overflowed the instruction cache (FP32 2.04 -> 1.71 ms at
        // 128^3; unrolled by 2 or 4 it ran slower too, 1.59 against 1.48 ms; FP64 2.23 -> 2.12 ms at 101^3)
        for (unsigned round = 0; round < t.rounds; ++round)
        {
            overChunk<kSplit, true>(a.nidx, t, round, pairTerm);
            foldChunks<kSplit>(round * kSplit, t.numChunks, momX, momY, momZ, energyS, aViscE);
        }
        maxvsignalI = maxOverSplit<kSplit>(maxvsignalI);
        if (valid && t.sub == 0)
        {
            if constexpr (kMode & kModeTape)
            {
                a.tape.energy[t.i] = energyS.get();
                a.tape.avisc[t.i]  = aViscE.get();
            }
            T aViscEnergy = aViscE.get() > T(0) ? aViscE.get() : T(0);
            a.du[t.i] = double(k.K * prodSum(prhoi, energyS.get(), T(0.5), aViscEnergy));
            a.ax[t.i] = -k.K * momX.get();
            a.ay[t.i] = -k.K * momY.get();
            a.az[t.i] = -k.K * momZ.get();

            double v = maxvsignalI > T(0) ? double(maxvsignalI) : double(ci);
            // FP32: h read again here rather than kept in two registers across the pair loop (1.478 -> 1.465 ms)
            double hEnd = sizeof(T) == 4 ? a.h[t.i] : hiD;
            dtMin       = hEnd > 0.0 ? k.Kcour * hEnd / v : INFINITY;
        }
    }
    if constexpr (kMode & kModeList)
    {
        // the group's Courant step lowers its block time step (momentum_energy_gpu.cu:96-103); rounding to float is
        // monotonic, so min(float, double) stored as float equals the min of the float values
        unsigned w  = unsigned((blockIdx.x * size_t(blockDim.x) + threadIdx.x) / (32 * kSplit));
        double gmin = dtMin;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
        {
            gmin = fmin(gmin, __shfl_xor_sync(0xffffffffu, gmin, off));
        }
        if ((threadIdx.x & 31) == 0 && w < a.numListed)
        {
            // a group's targets span kSplit warps; time steps are positive, so their bits order as integers
            if constexpr (kSplit == 1) { a.groupDt[w] = fminf(a.groupDt[w], float(gmin)); }
            else { atomicMin(reinterpret_cast<int*>(a.groupDt + w), __float_as_int(float(gmin))); }
        }
    }
    reduceOrdered<false, (kMode & kModeBatch) != 0>(dtMin, a.n, a.reduce + 1, a.batch, 1);
}

template<class T>
size_t chainTargets(const ChainArrays<T>& a)
{
    return a.groupList ? size_t(a.numListed) * 32 : a.n;
}

/*! Lanes that share a target. A launch of few targets leaves most of the GPU idle while each thread walks its ~100
 *  neighbours alone; several lanes take a chunk of eight neighbours each. The sums are the same bit for bit.
 *  Measured (us for the five loops, one lane / four / eight): 4,096 targets FP32 215 / 89 / 73, 9,261 targets FP64
 *  409 / 164 / 147, 24,000 targets FP32 (AV cleaning) 245 / 147 / 165, 27,000 targets FP64 420 / 266 / 297, 125,000
 *  targets FP32 475 / 491 / 610. */
template<class T>
int chainSplit(const ChainArrays<T>& a)
{
    size_t targets = chainTargets(a);
    return targets <= kEightLaneTargets ? 8 : targets <= kFourLaneTargets ? 4 : 1;
}

template<class T>
unsigned chainBlocks(const ChainArrays<T>& a)
{
    return ceilDiv(chainTargets(a), size_t(a.threads));
}

//! blocks of kSplitThreads threads for `lanes` lanes per target
template<class T>
unsigned splitBlocks(const ChainArrays<T>& a, int lanes)
{
    return ceilDiv(chainTargets(a) * lanes, size_t(kSplitThreads));
}

} // namespace

//! kernel variant: kModeTape when the adjoint's tape pointers are set, kModeBatch for an ensemble
template<class T>
int chainMode(const ChainArrays<T>& a)
{
    int mode = (a.tape.energy ? kModeTape : 0) | (a.batch.inst ? kModeBatch : 0);
    if (a.groupList) { return mode == 0 ? kModeList : -1; } // block time steps: no tape, no ensemble
    return mode == (kModeTape | kModeBatch) ? -1 : mode;
}

//! the mode of the two kernels that AV cleaning changes (IAD writes the gradients, MomentumEnergy reads them)
template<class T>
int chainModeAv(const ChainArrays<T>& a)
{
    int mode = chainMode(a);
    if (mode < 0 || !a.dvrec) { return mode; }
    return (mode & kModeTape) ? -1 : (mode | kModeAvClean); // the adjoint has no AV-cleaning variant
}

#define SPHB_LAUNCH(KERNEL, MODE, ...) KERNEL<T, (MODE), 1><<<chainBlocks(a), a.threads, 0, s>>>(__VA_ARGS__)
#define SPHB_LAUNCH_SPLIT(KERNEL, MODE, ...)                                                                           \
    switch (chainSplit(a))                                                                                              \
    {                                                                                                                   \
    case 8: KERNEL<T, (MODE), 8><<<splitBlocks(a, 8), kSplitThreads, 0, s>>>(__VA_ARGS__); break;                      \
    case 4: KERNEL<T, (MODE), 4><<<splitBlocks(a, 4), kSplitThreads, 0, s>>>(__VA_ARGS__); break;                      \
    default: SPHB_LAUNCH(KERNEL, MODE, __VA_ARGS__); break;                                                             \
    }

// the taped form keeps one lane per target (it records which neighbour sets the signal velocity), the ensemble's batch
// form as well (its launches cover every member)
#define SPHB_DISPATCH_AV(KERNEL, ...)                                                                                   \
    switch (chainModeAv(a))                                                                                             \
    {                                                                                                                   \
    case 0: SPHB_LAUNCH_SPLIT(KERNEL, 0, __VA_ARGS__) break;                                                            \
    case kModeTape: SPHB_LAUNCH(KERNEL, kModeTape, __VA_ARGS__); break;                                                 \
    case kModeBatch: SPHB_LAUNCH(KERNEL, kModeBatch, __VA_ARGS__); break;                                               \
    case kModeAvClean: SPHB_LAUNCH_SPLIT(KERNEL, kModeAvClean, __VA_ARGS__) break;                                      \
    case kModeList: SPHB_LAUNCH_SPLIT(KERNEL, kModeList, __VA_ARGS__) break;                                            \
    case kModeAvClean | kModeList: SPHB_LAUNCH_SPLIT(KERNEL, kModeAvClean | kModeList, __VA_ARGS__) break;              \
    case kModeAvClean | kModeBatch: SPHB_LAUNCH(KERNEL, kModeAvClean | kModeBatch, __VA_ARGS__); break;                 \
    default: return kErrArg;                                                                                            \
    }

#define SPHB_DISPATCH(KERNEL, ...)                                                                                      \
    switch (chainMode(a))                                                                                               \
    {                                                                                                                   \
    case 0: SPHB_LAUNCH_SPLIT(KERNEL, 0, __VA_ARGS__) break;                                                            \
    case kModeTape: SPHB_LAUNCH(KERNEL, kModeTape, __VA_ARGS__); break;                                                 \
    case kModeBatch: SPHB_LAUNCH(KERNEL, kModeBatch, __VA_ARGS__); break;                                               \
    case kModeList: SPHB_LAUNCH_SPLIT(KERNEL, kModeList, __VA_ARGS__) break;                                            \
    default: return kErrArg;                                                                                            \
    }

template<class T>
int launchXMass(const ChainArrays<T>& a, const HydroConsts<T>& k, const DevBox& box, cudaStream_t s)
{
    if (a.n == 0 || (a.groupList && a.numListed == 0)) { return kOk; }
    SPHB_DISPATCH(xmassKernel, a, k, box)
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

template<class T>
int launchVeDefGradhEos(const ChainArrays<T>& a, const HydroConsts<T>& k, const DevBox& box, cudaStream_t s)
{
    if (a.n == 0 || (a.groupList && a.numListed == 0)) { return kOk; }
    SPHB_DISPATCH(veDefGradhEosKernel, a, k, box)
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

template<class T>
int launchPackVelocity(const ChainArrays<T>& a, cudaStream_t s)
{
    if (a.n == 0) { return kOk; }
    packVelocityKernel<T><<<ceilDiv(a.n, 256), 256, 0, s>>>(a.n, a.vx, a.vy, a.vz, a.hrec);
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

template<class T>
int launchIadDivvCurlv(const ChainArrays<T>& a, const HydroConsts<T>& k, const DevBox& box, cudaStream_t s)
{
    if (a.n == 0 || (a.groupList && a.numListed == 0)) { return kOk; }
    SPHB_DISPATCH_AV(iadDivvCurlvFusedKernel, a, k, box)
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

template<class T>
int launchAVswitches(const ChainArrays<T>& a, const HydroConsts<T>& k, const DevBox& box, double dt, cudaStream_t s)
{
    if (a.n == 0 || (a.groupList && a.numListed == 0)) { return kOk; }
    if (a.avfull)
    {
        if (chainMode(a) != 0) { return kErrArg; }
        SPHB_LAUNCH_SPLIT(avSwitchesKernel, kModeFullAv, a, k, box, dt)
    }
    else { SPHB_DISPATCH(avSwitchesKernel, a, k, box, dt) }
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

template<class T>
int launchMomentumEnergy(const ChainArrays<T>& a, const HydroConsts<T>& k, const DevBox& box, cudaStream_t s)
{
    if (a.n == 0 || (a.groupList && a.numListed == 0)) { return kOk; }
    SPHB_DISPATCH_AV(momentumEnergyKernel, a, k, box)
    countLaunch();
    SPHB_CUDA_TRY(cudaGetLastError());
    return kOk;
}

#define SPHB_INSTANTIATE(T)                                                                                            \
    template int launchXMass<T>(const ChainArrays<T>&, const HydroConsts<T>&, const DevBox&, cudaStream_t);          \
    template int launchVeDefGradhEos<T>(const ChainArrays<T>&, const HydroConsts<T>&, const DevBox&, cudaStream_t);  \
    template int launchPackVelocity<T>(const ChainArrays<T>&, cudaStream_t);                                           \
    template int launchIadDivvCurlv<T>(const ChainArrays<T>&, const HydroConsts<T>&, const DevBox&, cudaStream_t);   \
    template int launchAVswitches<T>(const ChainArrays<T>&, const HydroConsts<T>&, const DevBox&, double,            \
                                     cudaStream_t);                                                                  \
    template int launchMomentumEnergy<T>(const ChainArrays<T>&, const HydroConsts<T>&, const DevBox&, cudaStream_t);

SPHB_INSTANTIATE(double)
SPHB_INSTANTIATE(float)

} // namespace sphb
