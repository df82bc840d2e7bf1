// Device helpers shared by the pass kernels (included by kernels.cu, linep.cuh and line2.cuh).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "kdesc.h"
#include "kernels.h"

namespace srwg {

// programmatic dependent launch: the next kernel in the stream may be set up from here on; this one
// waits until the kernel before it has completed and its writes are visible.  (Both do nothing in an
// ordinary launch.)
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// complex add / subtract as one packed FP32x2 instruction each (sm_100); b * (-1) + a is exactly a - b
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
// multiply by -i (forward, DIR=+1) or +i (inverse, DIR=-1)
template <int DIR> __device__ __forceinline__ float2 mul_mi(float2 a)
{
    return DIR > 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}

// exp(i*ph): Cody-Waite reduction of the FP64 argument by 2*pi (two-term constant) to [-pi, pi],
// then the FP32 hardware sine/cosine (absolute error ~4e-7 on that interval, the same order as
// the reference's own polynomial CosAndSin, sroptelm.h:856).
__device__ __forceinline__ float2 expi(double ph)
{
    const double inv2pi = 0.15915494309189533577;
    const double twopi_hi = 6.283185307179586232;      // nearest double to 2*pi
    const double twopi_lo = 2.4492935982947064e-16;    // 2*pi - twopi_hi
    double k = rint(ph * inv2pi);
    double r = fma(-k, twopi_hi, ph);
    r = fma(-k, twopi_lo, r);
    float s, c;
    __sincosf((float)r, &s, &c);
    return make_float2(c, s);
}

// ------------------------------------------------------------------------------------------------
// small DFTs of the pass of 16384 points (DIR=+1: exp(-2 pi i nk/R) like FFTW_FORWARD; DIR=-1: exp(+...) like FFTW_BACKWARD)
// ------------------------------------------------------------------------------------------------
template <int DIR> __device__ __forceinline__ void dft4(float2& v0, float2& v1, float2& v2, float2& v3)
{
    float2 a0 = cadd(v0, v2), a1 = csub(v0, v2), a2 = cadd(v1, v3), a3 = mul_mi<DIR>(csub(v1, v3));
    v0 = cadd(a0, a2);
    v2 = csub(a0, a2);
    v1 = cadd(a1, a3);
    v3 = csub(a1, a3);
}
template <int DIR> __device__ __forceinline__ void dft4(float2* v) { dft4<DIR>(v[0], v[1], v[2], v[3]); }

template <int DIR> __device__ __forceinline__ void dft16(float2* v)
{
    // n = 4 n1 + n2, k = k1 + 4 k2
    float2 y[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
        float2 a0 = v[n2], a1 = v[4 + n2], a2 = v[8 + n2], a3 = v[12 + n2];
        dft4<DIR>(a0, a1, a2, a3);
        y[n2][0] = a0; y[n2][1] = a1; y[n2][2] = a2; y[n2][3] = a3;
    }
    // twiddles W16^(n2 k1)
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
    const float sg = DIR > 0 ? -1.f : 1.f;
    const float2 w1 = make_float2(c1, sg * s1), w2 = make_float2(h, sg * h), w3 = make_float2(s1, sg * c1);
    y[1][1] = cmul(y[1][1], w1); y[1][2] = cmul(y[1][2], w2); y[1][3] = cmul(y[1][3], w3);
    y[2][1] = cmul(y[2][1], w2); y[2][2] = mul_mi<DIR>(y[2][2]);
    y[2][3] = cmul(y[2][3], make_float2(-h, sg * h));
    y[3][1] = cmul(y[3][1], w3); y[3][2] = cmul(y[3][2], make_float2(-h, sg * h));
    y[3][3] = cmul(y[3][3], make_float2(-c1, -sg * s1));
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
        float2 a0 = y[0][k1], a1 = y[1][k1], a2 = y[2][k1], a3 = y[3][k1];
        dft4<DIR>(a0, a1, a2, a3);
        v[k1] = a0; v[k1 + 4] = a1; v[k1 + 8] = a2; v[k1 + 12] = a3;
    }
}

template <int R, int DIR> __device__ __forceinline__ void dftR(float2* v)
{
    static_assert(R == 4 || R == 16, "stages of 16384 points");
    if constexpr (R == 4) dft4<DIR>(v);
    else dft16<DIR>(v);
}

// ------------------------------------------------------------------------------------------------
// point-wise operators
// ------------------------------------------------------------------------------------------------
// exact (non-contracted) FP64 coordinate arithmetic, as the reference's x87/SSE code evaluates it
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }

// RadPointModifier_PropToWaistBeyondParax (sroptdrf.h:712-754): exp(i k L (sqrt(1 + X) - 1)), or with
// k L sqrt(1 + X) on the path-length option, X = -lambda^2 (qx^2 + qz^2); the square root for
// |X| > 0.01, else the reference's binomial series; FP64, then reduced by 2 pi.  Out of line: rare,
// and it keeps the passes that may evaluate it small.
static __device__ __noinline__ float2 bpx_factor(const PwOps& e, int i, int j)
{
    const double qx = e.bqx0 + (double)i * e.bdqx, qz = e.bqz0 + (double)j * e.bdqz;
    const double lx = e.blam * qx, lz = e.blam * qz;
    const double X = -(lx * lx + lz * lz);
    double r;
    if (fabs(X) > 0.01) {
        r = sqrt(1. + X);
        if (!e.btreat) r -= 1.;
    } else {
        r = X * (0.5 + X * (-0.125 + X * (0.0625 + X * (-0.0390625 + X * (0.02734375 + X * (-0.0205078125 +
                                                                                  X * 0.01611328125))))));
        if (e.btreat) r += 1.;
    }
    return expi(e.bkL * r);
}

// srTGenTransmission::RadPointModifier (sroptgtr.h:163-310), one photon energy: amplitude
// transmission and optical path difference bilinear in the table (FP64, its index rules: the
// 1e-5 step snap, clamping to the last cell), the phase 2 pi / lambda * OPD; zero outside the table
// (within 1e-3 of a step) when the element says so.  Returns false to zero the point.
static __device__ __noinline__ bool tr_factor(const PwOps& e, int i, int j, const float2* tabs, float2& f)
{
    const double xRel = dadd(e.tr_x0, dmul((double)i, e.tr_dx)), zRel = dadd(e.tr_z0, dmul((double)j, e.tr_dz));
    const int Nx = e.tr_nx, Nz = e.tr_nz;
    const double xs = e.tr_xs, zs = e.tr_zs, xst = e.tr_xstep, zst = e.tr_zstep;
    if (e.tr_outer == 1) {
        const double xEnd = xs + (Nx - 1) * xst, zEnd = zs + (Nz - 1) * zst;
        const double tx = xst * 0.001, tz = zst * 0.001;
        if ((xRel < xs - tx) || (xRel > xEnd + tx) || (zRel < zs - tz) || (zRel > zEnd + tz)) return false;
    }
    double xr = 0., zr = 0.;
    long long ix = (long long)((xRel - xs) / xst);
    if (fabs(xRel - ((ix + 1) * xst + xs)) < 1.E-05 * xst) ix++;
    if (ix < 0) ix = 0;
    else if (ix > Nx - 2) { ix = Nx - 2; xr = 1.; }
    else xr = (xRel - (ix * xst + xs)) / xst;
    long long iz = (long long)((zRel - zs) / zst);
    if (fabs(zRel - ((iz + 1) * zst + zs)) < 1.E-05 * zst) iz++;
    if (iz < 0) iz = 0;
    else if (iz > Nz - 2) { iz = Nz - 2; zr = 1.; }
    else zr = (zRel - (iz * zst + zs)) / zst;
    const double xrzr = xr * zr;
    const double* d = reinterpret_cast<const double*>(tabs + e.tr_off);
    const long long zPer = (long long)Nx << 1;
    const double* p00 = d + (iz * zPer + (ix << 1));
    const double *p10 = p00 + 2, *p01 = p00 + zPer, *p11 = p01 + 2;
    const double Axz = p00[0] - p01[0] - p10[0] + p11[0], Bxz = p00[1] - p01[1] - p10[1] + p11[1];
    const double Ax = p10[0] - p00[0], Bx = p10[1] - p00[1];
    const double Az = p01[0] - p00[0], Bz = p01[1] - p00[1];
    const double T = Axz * xrzr + Ax * xr + Az * zr + p00[0];
    const double Ph = (Bxz * xrzr + Bx * xr + Bz * zr + p00[1]) * e.tr_k;
    const float2 c = expi(Ph);
    f = cmul(f, make_float2((float)(T * c.x), (float)(T * c.y)));
    return true;
}

// non-separable point-wise work: circular masks, rectangular obstacles, the quartic remainder of
// the angular transfer function, the beyond-paraxial propagator (everything separable is in the
// plan's tables)
__device__ __forceinline__ void extra_eval(const PwOps& e, int i, int j, float2& f, bool& zero, const float2* tabs)
{
    if (e.has_ang) {
        float qx = (float)(e.qx0 + (double)i * e.dqx), qz = (float)(e.qz0 + (double)j * e.dqz);
        float q2 = qx * qx + qz * qz;
        float c1q2 = (float)e.c1 * q2;
        float ph = (float)e.c0 * q2 * c1q2 * (1.f + 2.f * c1q2);
        float sn, cs;
        __sincosf(ph, &sn, &cs);
        f = cmul(f, make_float2(cs, sn));
    }
    if (e.has_bpx) f = cmul(f, bpx_factor(e, i, j));
    if (e.has_tr && !tr_factor(e, i, j, tabs, f)) zero = true;
    for (int m = 0; m < e.nmask; m++) {
        const PwMask& k = e.mask[m];
        double x = dadd(k.x0, dmul((double)i, k.dx));
        double z = dadd(k.z0, dmul((double)j, k.dz));
        double xr = dsub(x, k.cx), zr = dsub(z, k.cz);
        bool outside;
        if (k.type == 1) outside = (xr < -k.hx) || (xr > k.hx) || (zr < -k.hz) || (zr > k.hz);
        else outside = dadd(dmul(xr, xr), dmul(zr, zr)) > k.r2;
        zero |= k.obstacle ? !outside : outside;
    }
}

// chain with its along-line factors in a table: W[k] = tab[k] * extra(k ^ xi, line) * V[k ^ xs].  For
// power-of-two lines the centring rotation and the mirror are XOR masks: (k + N/2) mod N = k ^ N/2,
// N - 1 - k = k ^ (N - 1).  The chain's per-line factor is not part of it: the line factors of all
// chains of a pass are multiplied once per line and applied at the store (a per-line constant
// commutes with the FFT along the line).
struct Chain2 {
    int xs;                  // source index mask: rotation (rs2), mirror, rotation (rs1)
    int xi;                  // evaluation index mask of the non-separable work (rs2, mirror)
    int xinv;                // output chains: destination of transform output q is q ^ xinv
    int tab;                 // offset of the along-line factors in the plan's tables, or -1
    int extra;               // the pass's non-separable work applies to this chain
};

// v <- factor(k) v; `tabs` are the plan's tables, `ex` the pass's non-separable work
template <bool EXTRA>
__device__ __forceinline__ float2 chain2_apply(const Chain2& c, int k, int line, float2 v, const float2* tabs,
                                               const PwOps* ex, int axis)
{
    if (c.tab >= 0) v = cmul(__ldg(&tabs[c.tab + k]), v);
    if (EXTRA && c.extra) {
        const int i = k ^ c.xi;
        bool zero = false;
        float2 f = make_float2(1.f, 0.f);
        extra_eval(*ex, axis == 0 ? i : line, axis == 0 ? line : i, f, zero, tabs);
        v = zero ? make_float2(0.f, 0.f) : cmul(f, v);
    }
    return v;
}

__device__ __forceinline__ Chain2 make_chain2(const ChainTab& t, int rs1, int mir, int rs2, int extra, int N)
{
    Chain2 c;
    const int h = N >> 1;
    c.xi = (rs2 ? h : 0) ^ (mir ? N - 1 : 0);
    c.xs = c.xi ^ (rs1 ? h : 0);
    c.xinv = (rs1 ? h : 0) ^ (mir ? N - 1 : 0);
    c.tab = t.tab >= 0 ? (int)t.tab : -1;
    c.extra = extra;
    return c;
}

// element i of a line pass's output line: row-major (offset i * str) or, for a row pass feeding a
// column pass, column-blocked: blocks of 2^lg columns stored contiguously per row, offset
// (i >> lg) * bstr + (i & mask)
struct OutMap {
    int str, lg, bstr;
    __device__ __forceinline__ int at(int i) const { return lg < 0 ? i * str : ((i >> lg) * bstr + (i & ((1 << lg) - 1))); }
};

}  // namespace srwg
