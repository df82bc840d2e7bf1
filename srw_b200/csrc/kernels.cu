// sm_100a kernels for SRW's Fourier-optics propagation path.
//
// All passes are HBM-bandwidth bound (a complex FP32 point is read and written once per pass,
// ~1-4 flop/B), so they are plain SIMT kernels organised around full-line shared-memory tiles;
// no tensor cores.  Phase arguments are formed and reduced modulo 2*pi in FP64 and evaluated
// with an FP32 sincosf, as the reference forms them in double before its float CosAndSin
// (sroptelm.h:856-871).
#include <algorithm>
#include <mutex>
#include <set>

#include "common.cuh"

namespace srwg {

// CUDA function attributes (here: the dynamic shared-memory limit) belong to a device's context,
// so they are set once per device and kernel group, before that group's first launch there
static bool attrs_needed(int group)
{
    static std::mutex m;
    static std::set<long long> done;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return true;
    std::lock_guard<std::mutex> lk(m);
    return done.insert(((long long)dev << 8) | group).second;
}

// ------------------------------------------------------------------------------------------------
// RESIZE pass (RadResizeCore, sroptelm.cpp:3038-3337; OnlyLargerRange :4231)
// ------------------------------------------------------------------------------------------------
// sqrt(FI / app), the amplitude correction of ImproveReAndIm, from two reciprocal square roots (no
// division, and FI * app cannot overflow); within a few ulp of the correctly rounded value; FI >= 0,
// app > 0
__device__ __forceinline__ float amp_ratio(float FI, float app)
{
    return FI > 0.f ? FI * rsqrtf(FI) * rsqrtf(app) : 0.f;
}

__device__ __forceinline__ void lagrange4(float t, float* w)
{
    // cubic through nodes -1, 0, 1, 2 (the reference's SetupInterpolAux02 polynomial)
    float tm1 = t - 1.f, tm2 = t - 2.f, tp1 = t + 1.f;
    w[0] = -t * tm1 * tm2 * (1.f / 6.f);
    w[1] = tp1 * tm1 * tm2 * 0.5f;
    w[2] = -tp1 * t * tm2 * 0.5f;
    w[3] = tp1 * t * tm1 * (1.f / 6.f);
}

__device__ __forceinline__ ResizeAxis load_axis(const float2* tabs, long long off, int i)
{
    ResizeAxis a;
    float4 v = __ldg(reinterpret_cast<const float4*>(tabs + off) + i);
    a.st = __float_as_int(v.x);
    a.ir = __float_as_int(v.y);
    a.rel = v.z;
    a.pad = v.w;
    return a;
}

// one new point of one component: bicubic of Re, Im and |E|^2 over the 4x4 old stencil, the
// reference's bilinear fallback when any of the 32 values is exactly zero, and the amplitude
// correction by the interpolated intensity (ImproveReAndIm)
__device__ __forceinline__ float2 pre_factor(const ResizeDesc& d, const float2* tabs, int ix, int iz);

__device__ __forceinline__ float2 resize_point(const float2* __restrict__ o, int nxo, const float* wx, const float* wz,
                                               float xr, float zr, int irx, int irz, const ResizeDesc* pre = nullptr,
                                               const float2* tabs = nullptr, int gx = 0, int gz = 0)
{
    float2 f[4][4];
    bool low = false;
#pragma unroll
    for (int dz = 0; dz < 4; dz++)
#pragma unroll
        for (int dx = 0; dx < 4; dx++) {
            float2 v = __ldg(&o[(size_t)dz * nxo + dx]);
            if (pre) v = cmul(pre_factor(*pre, tabs, gx + dx, gz + dz), v);
            f[dz][dx] = v;
            low |= (v.x == 0.f) || (v.y == 0.f);
        }
    float2 F;
    float FI;
    if (!low) {
        F = make_float2(0.f, 0.f);
        FI = 0.f;
#pragma unroll
        for (int dz = 0; dz < 4; dz++) {
            float2 rowF = make_float2(0.f, 0.f);
            float rowI = 0.f;
#pragma unroll
            for (int dx = 0; dx < 4; dx++) {
                float2 v = f[dz][dx];
                rowF.x = fmaf(wx[dx], v.x, rowF.x);
                rowF.y = fmaf(wx[dx], v.y, rowF.y);
                rowI = fmaf(wx[dx], v.x * v.x + v.y * v.y, rowI);
            }
            F.x = fmaf(wz[dz], rowF.x, F.x);
            F.y = fmaf(wz[dz], rowF.y, F.y);
            FI = fmaf(wz[dz], rowI, FI);
        }
    } else {
        // bilinear on the 2x2 sub-cell (irx, irz) evaluated at (xr, zr): CheckForLowOrderInterp
        float2 f00 = f[irz][irx], f10 = f[irz][irx + 1], f01 = f[irz + 1][irx], f11 = f[irz + 1][irx + 1];
        float xz = xr * zr;
        F.x = f00.x + (f10.x - f00.x) * xr + (f01.x - f00.x) * zr + (f00.x - f01.x - f10.x + f11.x) * xz;
        F.y = f00.y + (f10.y - f00.y) * xr + (f01.y - f00.y) * zr + (f00.y - f01.y - f10.y + f11.y) * xz;
        float i00 = f00.x * f00.x + f00.y * f00.y, i10 = f10.x * f10.x + f10.y * f10.y;
        float i01 = f01.x * f01.x + f01.y * f01.y, i11 = f11.x * f11.x + f11.y * f11.y;
        FI = i00 + (i10 - i00) * xr + (i01 - i00) * zr + (i00 - i01 - i10 + i11) * xz;
    }
    FI = FI > 0.f ? FI : 0.f;
    float app = F.x * F.x + F.y * F.y;          // ImproveReAndIm
    if (app != 0.f) {
        float fac = amp_ratio(FI, app);
        F.x *= fac; F.y *= fac;
    }
    return F;
}

// interpolation of one point from its 4x4 stencil already in registers (see resize_point)
__device__ __forceinline__ float2 interp_stencil(const float2 (&f)[4][4], const float* wx, const float* wz, float xr,
                                                 float zr, int irx, int irz)
{
    bool low = false;
#pragma unroll
    for (int dz = 0; dz < 4; dz++)
#pragma unroll
        for (int dx = 0; dx < 4; dx++) low |= (f[dz][dx].x == 0.f) || (f[dz][dx].y == 0.f);
    float2 F;
    float FI;
    if (!low) {
        F = make_float2(0.f, 0.f);
        FI = 0.f;
#pragma unroll
        for (int dz = 0; dz < 4; dz++) {
            float2 rowF = make_float2(0.f, 0.f);
            float rowI = 0.f;
#pragma unroll
            for (int dx = 0; dx < 4; dx++) {
                float2 v = f[dz][dx];
                rowF.x = fmaf(wx[dx], v.x, rowF.x);
                rowF.y = fmaf(wx[dx], v.y, rowF.y);
                rowI = fmaf(wx[dx], v.x * v.x + v.y * v.y, rowI);
            }
            F.x = fmaf(wz[dz], rowF.x, F.x);
            F.y = fmaf(wz[dz], rowF.y, F.y);
            FI = fmaf(wz[dz], rowI, FI);
        }
    } else {
        float2 f00 = f[0][0], f10 = f[0][1], f01 = f[1][0], f11 = f[1][1];
        // select the 2x2 sub-cell (irx, irz) without dynamic register indexing
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int c = 0; c < 3; c++)
                if (a == irz && c == irx) { f00 = f[a][c]; f10 = f[a][c + 1]; f01 = f[a + 1][c]; f11 = f[a + 1][c + 1]; }
        float xz = xr * zr;
        F.x = f00.x + (f10.x - f00.x) * xr + (f01.x - f00.x) * zr + (f00.x - f01.x - f10.x + f11.x) * xz;
        F.y = f00.y + (f10.y - f00.y) * xr + (f01.y - f00.y) * zr + (f00.y - f01.y - f10.y + f11.y) * xz;
        float i00 = f00.x * f00.x + f00.y * f00.y, i10 = f10.x * f10.x + f10.y * f10.y;
        float i01 = f01.x * f01.x + f01.y * f01.y, i11 = f11.x * f11.x + f11.y * f11.y;
        FI = i00 + (i10 - i00) * xr + (i01 - i00) * zr + (i00 - i01 - i10 + i11) * xz;
    }
    FI = FI > 0.f ? FI : 0.f;
    float app = F.x * F.x + F.y * F.y;          // ImproveReAndIm
    if (app != 0.f) {
        float fac = amp_ratio(FI, app);
        F.x *= fac; F.y *= fac;
    }
    return F;
}

__device__ __forceinline__ float2 pick3(const float2* c, int o, int dx)
{   // c[o + dx] for o in {0, 1, 2} with compile-time register indices
    return o == 0 ? c[dx] : (o == 1 ? c[dx + 1] : c[dx + 2]);
}

__device__ __forceinline__ float2 resize_factor(const ResizeDesc& d, const float2* tabs, int ix, int iz)
{
    float2 e = make_float2(1.f, 0.f);
    if (d.t.tab >= 0) e = __ldg(&tabs[d.t.tab + ix]);
    if (d.t.ltab >= 0) e = cmul(e, __ldg(&tabs[d.t.ltab + iz]));
    bool zero = false;
    if (d.has_extra) extra_eval(d.extra, ix, iz, e, zero, tabs);
    return zero ? make_float2(0.f, 0.f) : e;
}

// RESIZE pass (RadResizeCore, sroptelm.cpp:3038-3337; OnlyLargerRange :4231).  The index
// arithmetic is tabulated per axis by the host (exact reference formulas); this kernel gathers,
// interpolates, applies the new-mesh point-wise factors and writes every new point (zero outside
// the window).  A thread produces two horizontally adjacent points: when their stencils start at
// most one old node apart, each stencil row is read once as three aligned float4 (6 complex).
__global__ void __launch_bounds__(256) resize_kernel(const ResizeLaunch p)
{
    const ResizeDesc& d = *reinterpret_cast<const ResizeDesc*>(reinterpret_cast<const char*>(p.gd) + blockIdx.z * p.bDesc);
    const float2* S[2] = {p.src[0] + blockIdx.z * p.bSrc, p.src[1] + blockIdx.z * p.bSrc};
    float2* D[2] = {p.dst[0] + blockIdx.z * p.bDst, p.dst[1] + blockIdx.z * p.bDst};
    const float2* tabs = p.tabs + blockIdx.z * p.bTab;
    const int ix0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int iz = blockIdx.y * blockDim.y + threadIdx.y;
    if (ix0 >= d.nxn || iz >= d.nzn) return;
    const bool two = ix0 + 1 < d.nxn;
    float2 out[2][2] = {{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}};
    const bool zin = (iz >= d.izStart) && (iz <= d.izEnd);
    const bool in0 = zin && (ix0 >= d.ixStart) && (ix0 <= d.ixEnd);
    const bool in1 = two && zin && (ix0 + 1 >= d.ixStart) && (ix0 + 1 <= d.ixEnd);
    if (in0 || in1) {
        const ResizeAxis az = load_axis(tabs, d.axz, iz);
        const ResizeAxis a0 = load_axis(tabs, d.axx, ix0);
        const ResizeAxis a1 = two ? load_axis(tabs, d.axx, ix0 + 1) : a0;
        if (d.only_larger) {
#pragma unroll
            for (int c = 0; c < 2; c++) {
                if (in0) out[0][c] = __ldg(&S[c][(size_t)az.st * d.nxo + a0.st]);
                if (in1) out[1][c] = __ldg(&S[c][(size_t)az.st * d.nxo + a1.st]);
            }
        } else {
            float wz[4], wx0[4], wx1[4];
            lagrange4(az.rel, wz);
            lagrange4(a0.rel, wx0);
            lagrange4(a1.rel, wx1);
            const int base = a0.st & ~1;
            const int o0 = a0.st - base, o1 = a1.st - base;
            const bool vec = p.vec_ok && in0 && in1 && (o1 >= o0) && (o1 <= 2) && (base + 6 <= d.nxo) && !d.has_pre;
            if (vec) {
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const float2* __restrict__ o = S[c] + (size_t)az.st * d.nxo + base;
                    float2 f0[4][4], f1[4][4];
#pragma unroll
                    for (int dz = 0; dz < 4; dz++) {
                        const float4* r4 = reinterpret_cast<const float4*>(o + (size_t)dz * d.nxo);
                        float4 q0 = __ldg(r4), q1 = __ldg(r4 + 1), q2 = __ldg(r4 + 2);
                        float2 cc[6] = {make_float2(q0.x, q0.y), make_float2(q0.z, q0.w), make_float2(q1.x, q1.y),
                                        make_float2(q1.z, q1.w), make_float2(q2.x, q2.y), make_float2(q2.z, q2.w)};
#pragma unroll
                        for (int dx = 0; dx < 4; dx++) {
                            f0[dz][dx] = pick3(cc, o0, dx);
                            f1[dz][dx] = pick3(cc, o1, dx);
                        }
                    }
                    out[0][c] = interp_stencil(f0, wx0, wz, a0.rel, az.rel, a0.ir, az.ir);
                    out[1][c] = interp_stencil(f1, wx1, wz, a1.rel, az.rel, a1.ir, az.ir);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const ResizeDesc* pre = d.has_pre ? &d : nullptr;
                    if (in0) out[0][c] = resize_point(S[c] + (size_t)az.st * d.nxo + a0.st, d.nxo, wx0, wz, a0.rel,
                                                      az.rel, a0.ir, az.ir, pre, tabs, a0.st, az.st);
                    if (in1) out[1][c] = resize_point(S[c] + (size_t)az.st * d.nxo + a1.st, d.nxo, wx1, wz, a1.rel,
                                                      az.rel, a1.ir, az.ir, pre, tabs, a1.st, az.st);
                }
            }
        }
        if (d.has_pw) {
            if (in0) {
                float2 e = resize_factor(d, tabs, ix0, iz);
                out[0][0] = cmul(out[0][0], e);
                out[0][1] = cmul(out[0][1], e);
            }
            if (in1) {
                float2 e = resize_factor(d, tabs, ix0 + 1, iz);
                out[1][0] = cmul(out[1][0], e);
                out[1][1] = cmul(out[1][1], e);
            }
        }
    }
    const size_t o = (size_t)iz * d.nxn + ix0;
#pragma unroll
    for (int c = 0; c < 2; c++) {
        if (p.vec_ok && two && ((o & 1) == 0)) {
            __stcs(reinterpret_cast<float4*>(D[c] + o), make_float4(out[0][c].x, out[0][c].y, out[1][c].x, out[1][c].y));
        } else {
            __stcs(&D[c][o], out[0][c]);
            if (two) __stcs(&D[c][o + 1], out[1][c]);
        }
    }
}

// point-wise work folded in from a preceding element-wise pass, at old index (ix, iz); the same
// operations in the same order as pw_kernel
__device__ __forceinline__ float2 pre_factor(const ResizeDesc& d, const float2* tabs, int ix, int iz)
{
    float2 e = make_float2(1.f, 0.f);
    if (d.tp.tab >= 0) e = __ldg(&tabs[d.tp.tab + ix]);
    if (d.tp.ltab >= 0) e = cmul(e, __ldg(&tabs[d.tp.ltab + iz]));
    bool zero = false;
    if (d.has_pre_extra) extra_eval(d.pre_extra, ix, iz, e, zero, tabs);
    return zero ? make_float2(0.f, 0.f) : e;
}

// Tiled RESIZE pass: a CTA makes a TZ x TX tile of new points.  The old points under the tile's
// stencils are staged once in shared memory (with the folded point-wise work applied); the 4x4
// interpolation is separable, so the x interpolation of Re, Im and |E|^2 is done once per (old
// row, new column) and each new point combines four of those rows.  The operation order per new
// point is that of resize_kernel (x first, then z; same FMAs), so both kernels give identical
// results.  Points outside the window are written as zeros.
__global__ void __launch_bounds__(256) resize2_kernel(const ResizeLaunch p)
{
    const ResizeDesc& d = *reinterpret_cast<const ResizeDesc*>(reinterpret_cast<const char*>(p.gd) + blockIdx.z * p.bDesc);
    const float2* S[2] = {p.src[0] + blockIdx.z * p.bSrc, p.src[1] + blockIdx.z * p.bSrc};
    float2* D[2] = {p.dst[0] + blockIdx.z * p.bDst, p.dst[1] + blockIdx.z * p.bDst};
    const float2* tabs = p.tabs + blockIdx.z * p.bTab;
    constexpr int TX = SRWG_RESIZE_TX, TZ = SRWG_RESIZE_TZ;
    extern __shared__ float4 rsm[];
    const int OR = d.tile_or, OC = d.tile_oc;
    float4* wxs = rsm;                    // x weights per tile column
    float4* axs = wxs + TX;               // (st, ir, rel) per tile column
    float4* wzs = axs + TX;               // z weights per tile row
    float4* azs = wzs + TZ;
    float4* H = azs + TZ;                 // [comp][old row][tile column]: (Re, Im, |E|^2, any zero)
    float2* old = reinterpret_cast<float2*>(H + 2 * OR * TX);   // [comp][old row][old column]
    __shared__ int ext[4];
    const int tid = threadIdx.x;
    // a resize that writes only its window starts at this wavefront's first tile of it
    const int x0 = (blockIdx.x + (d.skip_zero ? max(0, (int)d.ixStart) / TX : 0)) * TX;
    const int z0 = (blockIdx.y + (d.skip_zero ? max(0, (int)d.izStart) / TZ : 0)) * TZ;
    const int xa = max(x0, (int)d.ixStart), xb = min(min(x0 + TX, d.nxn) - 1, (int)d.ixEnd);
    const int za = max(z0, (int)d.izStart), zb = min(min(z0 + TZ, d.nzn) - 1, (int)d.izEnd);
    if (xa > xb || za > zb) {
        if (d.skip_zero) return;
        for (int e = tid; e < TZ * TX; e += 256) {
            const int gi = x0 + (e & (TX - 1)), gj = z0 + e / TX;
            if (gi < d.nxn && gj < d.nzn) {
                const size_t o = (size_t)gj * d.nxn + gi;
                __stcs(&D[0][o], make_float2(0.f, 0.f));
                __stcs(&D[1][o], make_float2(0.f, 0.f));
            }
        }
        return;
    }
    if (tid == 0) { ext[0] = 1 << 30; ext[1] = -1; ext[2] = 1 << 30; ext[3] = -1; }
    __syncthreads();
    if (tid < TX) {
        const int i = x0 + tid;
        if (i >= xa && i <= xb) {
            const ResizeAxis a = load_axis(tabs, d.axx, i);
            float w[4];
            lagrange4(a.rel, w);
            wxs[tid] = make_float4(w[0], w[1], w[2], w[3]);
            axs[tid] = make_float4(__int_as_float(a.st), __int_as_float(a.ir), a.rel, 0.f);
            atomicMin(&ext[0], a.st);
            atomicMax(&ext[1], a.st);
        }
    } else if (tid >= 128 && tid < 128 + TZ) {
        const int j = z0 + tid - 128;
        if (j >= za && j <= zb) {
            const ResizeAxis a = load_axis(tabs, d.axz, j);
            float w[4];
            lagrange4(a.rel, w);
            wzs[tid - 128] = make_float4(w[0], w[1], w[2], w[3]);
            azs[tid - 128] = make_float4(__int_as_float(a.st), __int_as_float(a.ir), a.rel, 0.f);
            atomicMin(&ext[2], a.st);
            atomicMax(&ext[3], a.st);
        }
    }
    __syncthreads();
    const int ox0 = ext[0], oz0 = ext[2];
    const int nc = ext[1] - ox0 + 4, nr = ext[3] - oz0 + 4;     // <= OC, OR (host-computed maxima)
    // old tile of both components, with the folded point-wise work
    for (int e = tid; e < nr * nc; e += 256) {
        const int r = e / nc, c = e - r * nc;
        const int gx = ox0 + c, gz = oz0 + r;
        const size_t go = (size_t)gz * d.nxo + gx;
        float2 v0 = __ldg(&S[0][go]), v1 = __ldg(&S[1][go]);
        if (d.has_pre) {
            const float2 f = pre_factor(d, tabs, gx, gz);
            v0 = cmul(f, v0);
            v1 = cmul(f, v1);
        }
        old[r * OC + c] = v0;
        old[OR * OC + r * OC + c] = v1;
    }
    __syncthreads();
    // x interpolation per (old row, tile column)
    for (int e = tid; e < 2 * nr * TX; e += 256) {
        const int comp = e >= nr * TX;
        const int e2 = e - comp * nr * TX;
        const int r = e2 / TX, i = e2 & (TX - 1);
        const int gi = x0 + i;
        if (gi < xa || gi > xb) continue;
        const float4 w4 = wxs[i];
        const float w[4] = {w4.x, w4.y, w4.z, w4.w};
        const float2* row = old + comp * OR * OC + r * OC + (__float_as_int(axs[i].x) - ox0);
        float rx = 0.f, ry = 0.f, ri = 0.f;
        bool low = false;
#pragma unroll
        for (int dx = 0; dx < 4; dx++) {
            const float2 v = row[dx];
            low |= (v.x == 0.f) || (v.y == 0.f);
            rx = fmaf(w[dx], v.x, rx);
            ry = fmaf(w[dx], v.y, ry);
            ri = fmaf(w[dx], v.x * v.x + v.y * v.y, ri);
        }
        H[comp * OR * TX + r * TX + i] = make_float4(rx, ry, ri, low ? 1.f : 0.f);
    }
    __syncthreads();
    // new points: z interpolation, low-order fallback, amplitude correction, new-mesh factors
    for (int e = tid; e < TZ * TX; e += 256) {
        const int jj = e / TX, i = e & (TX - 1);
        const int gi = x0 + i, gj = z0 + jj;
        if (gi >= d.nxn || gj >= d.nzn) continue;
        float2 out[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const bool inw = gi >= xa && gi <= xb && gj >= za && gj <= zb;
        if (!inw && d.skip_zero) continue;
        if (inw) {
            const float4 wz4 = wzs[jj], az = azs[jj], ax = axs[i];
            const float wz[4] = {wz4.x, wz4.y, wz4.z, wz4.w};
            const int r0 = __float_as_int(az.x) - oz0;
#pragma unroll
            for (int comp = 0; comp < 2; comp++) {
                const float4* h = H + comp * OR * TX + r0 * TX + i;
                float2 F = make_float2(0.f, 0.f);
                float FI = 0.f;
                bool low = false;
#pragma unroll
                for (int dz = 0; dz < 4; dz++) {
                    const float4 q = h[dz * TX];
                    low |= q.w != 0.f;
                    F.x = fmaf(wz[dz], q.x, F.x);
                    F.y = fmaf(wz[dz], q.y, F.y);
                    FI = fmaf(wz[dz], q.z, FI);
                }
                if (low) {
                    // bilinear on the 2x2 sub-cell (ir_x, ir_z) of the stencil (CheckForLowOrderInterp)
                    const int irx = __float_as_int(ax.y), irz = __float_as_int(az.y);
                    const float xr = ax.z, zr = az.z;
                    const float2* c0 = old + comp * OR * OC + (r0 + irz) * OC + (__float_as_int(ax.x) - ox0) + irx;
                    const float2 f00 = c0[0], f10 = c0[1], f01 = c0[OC], f11 = c0[OC + 1];
                    const float xz = xr * zr;
                    F.x = f00.x + (f10.x - f00.x) * xr + (f01.x - f00.x) * zr + (f00.x - f01.x - f10.x + f11.x) * xz;
                    F.y = f00.y + (f10.y - f00.y) * xr + (f01.y - f00.y) * zr + (f00.y - f01.y - f10.y + f11.y) * xz;
                    const float i00 = f00.x * f00.x + f00.y * f00.y, i10 = f10.x * f10.x + f10.y * f10.y;
                    const float i01 = f01.x * f01.x + f01.y * f01.y, i11 = f11.x * f11.x + f11.y * f11.y;
                    FI = i00 + (i10 - i00) * xr + (i01 - i00) * zr + (i00 - i01 - i10 + i11) * xz;
                }
                FI = FI > 0.f ? FI : 0.f;
                const float app = F.x * F.x + F.y * F.y;      // ImproveReAndIm
                if (app != 0.f) {
                    const float fac = amp_ratio(FI, app);
                    F.x *= fac;
                    F.y *= fac;
                }
                out[comp] = F;
            }
            if (d.has_pw) {
                const float2 f = resize_factor(d, tabs, gi, gj);
                out[0] = cmul(out[0], f);
                out[1] = cmul(out[1], f);
            }
        }
        const size_t o = d.cp ? (size_t)(gj - d.cz0) * d.cp + (gi - d.cx0) : (size_t)gj * d.nxn + gi;
        __stcs(&D[0][o], out[0]);
        __stcs(&D[1][o], out[1]);
    }
}

// ------------------------------------------------------------------------------------------------
// element-wise PW pass
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) pw_kernel(const PwLaunch p)
{
    const PwDesc& d = *reinterpret_cast<const PwDesc*>(reinterpret_cast<const char*>(p.gd) + blockIdx.z * p.bDesc);
    const float2* S[2] = {p.src[0] + blockIdx.z * p.bSrc, p.src[1] + blockIdx.z * p.bSrc};
    float2* D[2] = {p.dst[0] + blockIdx.z * p.bDst, p.dst[1] + blockIdx.z * p.bDst};
    const float2* tabs = p.tabs + blockIdx.z * p.bTab;
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iz = blockIdx.y;
    if (ix >= d.nx) return;
    float2 e = make_float2(1.f, 0.f);
    if (d.t.tab >= 0) e = __ldg(&tabs[d.t.tab + ix]);
    if (d.t.ltab >= 0) e = cmul(e, __ldg(&tabs[d.t.ltab + iz]));
    bool zero = false;
    if (d.has_extra) extra_eval(d.extra, ix, iz, e, zero, tabs);
    if (zero) e = make_float2(0.f, 0.f);
    const int ox = d.mirror_x ? d.nx - 1 - ix : ix;
    const int oz = d.mirror_z ? d.nz - 1 - iz : iz;
    const size_t i = (size_t)iz * d.nx + ix, o = (size_t)oz * d.nx + ox;
#pragma unroll
    for (int c = 0; c < 2; c++) __stcs(&D[c][o], cmul(e, __ldcs(&S[c][i])));
}

// ------------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------------
// the line pass of N points: the fixed schedule where the length has one
static LineFn line_fn(int N, bool cols, int mode, int extra)
{
    switch (N) {
#define SRWG_LINEF_CASE(M, A, B, C, D, T) case M: return linef_get_##M(cols, mode, extra);
    SRWG_LINEF_LENGTHS(SRWG_LINEF_CASE)
#undef SRWG_LINEF_CASE
    default: break;
    }
    switch (mode + (cols ? 3 : 0)) {
    case 0: return linep_get_0_0(extra);
    case 1: return linep_get_0_1(extra);
    case 2: return linep_get_0_2(extra);
    case 3: return linep_get_1_0(extra);
    case 4: return linep_get_1_1(extra);
    default: return linep_get_1_2(extra);
    }
}

// launches f; pdl: as a programmatic dependent of the kernel before it in the stream
template <class A>
static cudaError_t launch_one(void (*f)(const A), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl, const A& a)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, f, a);
}

cudaError_t launch_line(const LineLaunch& pin, cudaStream_t st, bool pdl)
{
    LineArgs p = pin;
    const LineDesc& d = pin.d;
    dim3 grid((p.nlines + p.L - 1) / p.L, 2, p.nb > 1 ? p.nb : 1);
    if (p.nblk > 0) grid.x = std::min((int)grid.x, p.nblk);      // only the window's line blocks
    if (attrs_needed(0)) {
        const int dirs[8][2] = {{1, 1}, {1, -1}, {-1, 1}, {-1, -1}, {1, 0}, {-1, 0}, {0, 1}, {0, -1}};
        for (int e = 0; e < 2; e++) {
            for (int m = 0; m < 8; m++) {
                cudaFuncSetAttribute(line2_get_14(e, dirs[m][0], dirs[m][1]),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, SRWG_LINE_SMEM_MAX);
                cudaFuncSetAttribute(line2e_get_14(e, dirs[m][0], dirs[m][1]),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, SRWG_LINE_SMEM_MAX);
            }
            const int modes[6][2] = {{0, 0}, {0, 2}, {1, 0}, {1, 1}, {1, 2}, {2, 0}};
            for (const auto& m : modes) {
                cudaFuncSetAttribute(line_fn(0, e, m[0], m[1]), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SRWG_LINE_SMEM_MAX);
#define SRWG_LINEF_ATTR(M, A, B, C, D, T)                                                                   \
                cudaFuncSetAttribute(line_fn(M, e, m[0], m[1]), cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     SRWG_LINE_SMEM_MAX);
                SRWG_LINEF_LENGTHS(SRWG_LINEF_ATTR)
#undef SRWG_LINEF_ATTR
            }
        }
    }
    if (p.v2 == 0) {
        const bool inten = d.out_int != 0;
        if (inten && (d.has_extra || (d.f1 && d.f2))) return cudaErrorInvalidValue;
        size_t smem = (size_t)p.G * p.P * sizeof(float4);
        // a windowed tile that is one block of its input (the pass before it wrote blocks of this width):
        // the window by bulk copies into shared memory behind the slots, where that leaves the CTAs per SM
        // (two of 256 threads at 128 registers, more of fewer) room.  The largest window of the launch
        // is the host's; an electron's larger one loads directly.
        p.bulk = 0;
        if (d.zwin && d.blk_in == p.L && d.za0 <= d.za1 && ((((uintptr_t)p.src[0]) | ((uintptr_t)p.src[1])) & 15) == 0 &&
            (p.bSrc & 1) == 0 && (p.L & 1) == 0) {
            const size_t pts = (size_t)(std::min(p.N, d.za1 - d.za0 + 9)) * p.L;
            const size_t stg = pts * sizeof(float2) * (inten ? 2 : 1);
            const int ctas = std::min(4, std::max(1, 512 / (p.T * p.G)));
            if ((smem + stg + 1024) * ctas <= SRWG_LINE_SMEM_MAX) {
                p.bulk = (int)pts;
                smem += stg;
            }
        }
        if (p.T * p.G > 512 || smem > SRWG_LINE_SMEM_MAX || (!inten && (p.nlines & 1))) return cudaErrorInvalidValue;
        p.alignIn = ((((uintptr_t)p.src[0]) | ((uintptr_t)p.src[1])) & 15) == 0 && (p.bSrc & 1) == 0;
        p.alignOut = ((((uintptr_t)p.dst[0]) | ((uintptr_t)p.dst[1])) & 15) == 0 && (p.bDst & 1) == 0;
        if (inten) grid.y = 1;                  // a pair holds both components
        LineFn f = line_fn(p.N, d.axis != 0, inten ? 2 : (d.f1 && d.f2) ? 1 : 0, d.has_extra ? 2 : d.ang ? 1 : 0);
        if (f == nullptr) return cudaErrorInvalidValue;
        return launch_one(f, grid, dim3(p.T * p.G), smem, st, pdl, p);
    } else {
        const size_t smem = (size_t)p.L * p.P * sizeof(float2);
        if (d.out_int || p.N != 16384 || smem > SRWG_LINE_SMEM_MAX) return cudaErrorInvalidValue;
        LineFn f = d.has_extra ? line2e_get_14(d.axis != 0, d.f1, d.f2) : line2_get_14(d.axis != 0, d.f1, d.f2);
        if (f == nullptr) return cudaErrorInvalidValue;
        f<<<grid, p.T * p.L, smem, st>>>(p);
    }
    return cudaGetLastError();
}

static SampleFn sample_fn(int N)
{
    switch (N) {
#define SRWG_LINEF_CASE(M, A, B, C, D, T) case M: return lines_get_##M();
    SRWG_LINEF_LENGTHS(SRWG_LINEF_CASE)
#undef SRWG_LINEF_CASE
    default: return lines_get();
    }
}

// two pairs' slots, two intensity rows, the detector row's sums
static size_t sample_smem(const LineLaunch& p, int anx)
{
    return (size_t)2 * p.P * sizeof(float4) + (size_t)(2 * p.N + (p.N & 1) * 2) * sizeof(float) + (size_t)anx * sizeof(double);
}
bool sample_fits(const LineLaunch& p, int anx)
{
    return p.v2 == 0 && 2 * p.T <= 512 && sample_smem(p, anx) <= SRWG_LINE_SMEM_MAX;
}

// A block per electron.  The column pass before the sampled pass then writes those rows only: at 1536 x 1600
// on 512 detector rows 640 of 1600, at 4096^2 1024 of 4096.  There the column pass of 16 electrons, bound by
// its writes, went from 383 to 308 us; at 1536 x 1600 it is bound by its instructions (410 us of 64 electrons
// either way).  The mask itself takes 2 us.
__global__ void __launch_bounds__(256) row_mask_kernel(const LineArgs p, const SampleArgs q, unsigned* mask, int words)
{
    __shared__ unsigned m[256];                          // (columns of at most 8192 points)
    const int b = blockIdx.x;
    const LineRun& d = reinterpret_cast<const LineDesc*>(reinterpret_cast<const char*>(p.gd) + b * p.bDesc)->run;
    const ElecParams& e = q.ep[b];
    m[threadIdx.x] = 0;
    __syncthreads();
    for (int j = threadIdx.x; j < q.anz; j += 256) {
        const int iy0 = sample_row(q, e, j);
        if (iy0 < 0 || iy0 >= e.onz - 1) continue;
        for (int g = 0; g < 2; g++) {
            const int line = d.mirror_lines ? p.nlines - 1 - (iy0 + g) : iy0 + g, k = line - d.in_l0;
            if (k >= 0 && (k >> 5) < words) atomicOr(&m[k >> 5], 1u << (k & 31));
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < words) mask[(size_t)b * words + threadIdx.x] = m[threadIdx.x];
}
cudaError_t launch_row_mask(const LineLaunch& p, const SampleArgs& q, unsigned* mask, int words, cudaStream_t st)
{
    if (words < 1 || words > 256) return cudaErrorInvalidValue;
    row_mask_kernel<<<q.nb, 256, 0, st>>>(p, q, mask, words);
    return cudaGetLastError();
}
cudaError_t launch_line_sample(const LineLaunch& p, const SampleArgs& q, cudaStream_t st, bool pdl)
{
    if (!sample_fits(p, q.anx) || p.d.axis != 0 || p.d.has_extra || p.d.ang || (p.d.f1 && p.d.f2) || q.per < 1)
        return cudaErrorInvalidValue;
    if (attrs_needed(2)) {
#define SRWG_LINEF_ATTR(M, A, B, C, D, T)                                                                   \
        cudaFuncSetAttribute(lines_get_##M(), cudaFuncAttributeMaxDynamicSharedMemorySize, SRWG_LINE_SMEM_MAX);
        SRWG_LINEF_LENGTHS(SRWG_LINEF_ATTR)
#undef SRWG_LINEF_ATTR
        cudaFuncSetAttribute(lines_get(), cudaFuncAttributeMaxDynamicSharedMemorySize, SRWG_LINE_SMEM_MAX);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(q.anz, (q.nb + q.per - 1) / q.per);
    cfg.blockDim = dim3(2 * p.T);
    cfg.dynamicSmemBytes = sample_smem(p, q.anx);
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, sample_fn(p.N), (const LineArgs&)p, q);
}

cudaError_t launch_resize(const ResizeLaunch& q, cudaStream_t st)
{
    ResizeLaunch p = q;
    p.vec_ok = ((q.d.nxo & 1) == 0) && ((q.d.nxn & 1) == 0) && ((q.bSrc & 1) == 0) && ((q.bDst & 1) == 0);
    for (int c = 0; c < 2; c++)
        p.vec_ok = p.vec_ok && ((((uintptr_t)q.src[c]) & 15) == 0) && ((((uintptr_t)q.dst[c]) & 15) == 0);
    if (p.d.tile_or > 0 && p.d.tile_oc > 0 && p.d.tile_or <= SRWG_RESIZE_OR_MAX && p.d.tile_oc <= SRWG_RESIZE_OC_MAX) {
        const size_t smem = (size_t)(2 * SRWG_RESIZE_TX + 2 * SRWG_RESIZE_TZ) * sizeof(float4) +
                            (size_t)2 * p.d.tile_or * SRWG_RESIZE_TX * sizeof(float4) +
                            (size_t)2 * p.d.tile_or * p.d.tile_oc * sizeof(float2);
        if (attrs_needed(1))
            cudaFuncSetAttribute(resize2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SRWG_LINE_SMEM_MAX);
        dim3 grid((p.d.nxn + SRWG_RESIZE_TX - 1) / SRWG_RESIZE_TX, (p.d.nzn + SRWG_RESIZE_TZ - 1) / SRWG_RESIZE_TZ,
                  p.nb > 1 ? p.nb : 1);
        ResizeLaunch q = p;
        if (p.ntx > 0 && p.ntz > 0) {            // only the window's tiles
            grid.x = std::min((int)grid.x, p.ntx);
            grid.y = std::min((int)grid.y, p.ntz);
        }
        resize2_kernel<<<grid, 256, smem, st>>>(q);
        return cudaGetLastError();
    }
    dim3 blk(64, 4);
    const int nxh = (p.d.nxn + 1) / 2;
    dim3 grid((nxh + blk.x - 1) / blk.x, (p.d.nzn + blk.y - 1) / blk.y, p.nb > 1 ? p.nb : 1);
    resize_kernel<<<grid, blk, 0, st>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_pw(const PwLaunch& p, cudaStream_t st)
{
    dim3 blk(256);
    dim3 grid((p.d.nx + 255) / 256, p.d.nz, p.nb > 1 ? p.nb : 1);
    pw_kernel<<<grid, blk, 0, st>>>(p);
    return cudaGetLastError();
}

}  // namespace srwg
