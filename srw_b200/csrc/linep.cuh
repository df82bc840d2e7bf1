// Line pass: whole rows (axis 0) or tiles of whole columns (axis 1) through one or two 1D transforms
// with the point-wise chains before, between and after them.  One family for every length
// N = 2^a 3^b 5^c 7^d 11^e 13^f up to 8192 (line2.cuh serves 16384).
//
// Packed pairs.  A thread transforms TWO lines at once (neighbouring rows or columns; in an intensity
// pass the two components of one line): a value is the pair of real parts and the pair of imaginary
// parts, so that every complex addition is two packed FP32x2 instructions for both lines, a
// multiplication by -i is a renaming, and indices, addresses, twiddles and table factors are formed
// once for two points.  The one-line form of this pass was bound by instruction issue (116
// instructions per point at 4096, complex numbers in (re, im) registers).
//
// In-place decimation in frequency.  N = R1 R2 ... Rn, L_s = N / (R1 ... R_s).  Stage s transforms
// digit k_s of the position k1 L1 + k2 L2 + ... + kn in place (each butterfly reads and writes its own
// places, so one barrier per stage is enough) and multiplies by W_(L_(s-1))^(j k_s), j < L_s the
// position below the digit.  The first stage reads global memory (butterflies over j: neighbouring
// threads read neighbouring points), the last one writes it: butterfly u = k1 + R1 k2 + ... holds the
// outputs u + (N / Rn) k_n, so neighbouring threads write neighbouring points.  The output index of a
// first transform is thus spread over its last stage exactly as the input of a second one with the
// digits in reverse order: the two stages run in registers with the middle chain between them, and
// the second transform goes back through the digits (twiddle W_(R1..Rs)^(u_low q), u_low the natural
// index of the digits below s), its last stage over k1 writing global memory.  Two transforms cost
// 2n - 1 stages and 2n - 2 barriers.
// Shared memory: 16 bytes per position (both lines); blocks of k1 have an odd pitch, which makes
// the last stage's reads (neighbouring k1) and everyone's consecutive accesses free of conflicts.
// Inverse transforms conjugate at the ends (conj DFT(conj x)).
#pragma once
#include "common.cuh"
#include "linep_shape.h"

namespace srwg {

// ------------------------------------------------------------------------------------------------
// bulk async copies into shared memory, completion through an mbarrier (one per CTA, phase 0)
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, unsigned bytes)
{
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(smem_addr(bar)),
                 "r"(bytes) : "memory");
}
// global -> shared, `bytes` a multiple of 16, both addresses 16-byte aligned
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
// non-blocking test of the phase of parity `phase` (try_wait would suspend the thread for a
// hardware-defined time, which would make an iteration limit meaningless)
__device__ __forceinline__ bool mbar_try(uint64_t* bar, unsigned phase)
{
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(smem_addr(bar)), "r"(phase) : "memory");
    return ok != 0;
}
// waits for the phase of parity `phase` at most `limit` tries (32 ns apart); on giving up it counts
// the event in *status and waits (at most 2^24 more tries, about a second) for the copies still in
// flight, so that none lands after the CTA has left.
// Returns false when any thread of the CTA gave up (the CTA then skips its work as a whole).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned phase, long long limit, int* status)
{
    long long it = 0;
    bool done = mbar_try(bar, phase);
    while (!done && ++it < limit) {
        __nanosleep(32);
        done = mbar_try(bar, phase);
    }
    const bool gave_up = !done;
    if (gave_up) {
        if (status) atomicAdd(status, 1);
        long long k = 0;
        while (!mbar_try(bar, phase) && ++k < (1ll << 24)) __nanosleep(64);
    }
    return !__syncthreads_or(gave_up);
}

struct P2 {
    float2 re, im;          // (line 0, line 1)
};

// loads of the field: once, past the L1 cache (the tables stay in it)
__device__ __forceinline__ float2 ldfield(const float2* p)
{
    float2 v;
    asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ldfield4(const float2* p)
{
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
// the same where `on`, else v stays (one predicated instruction: no branch, so that a butterfly's loads
// are in flight together)
__device__ __forceinline__ void ldfield_if(bool on, const float2* p, float& x, float& y)
{
    asm volatile("{ .reg .pred q; setp.ne.b32 q, %3, 0; @q ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2]; }"
                 : "+f"(x), "+f"(y) : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ldfield4_if(bool on, const float2* p, float4& v)
{
    asm volatile("{ .reg .pred q; setp.ne.b32 q, %5, 0; @q ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4]; }"
                 : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : "l"(p), "r"((int)on));
}
__device__ __forceinline__ float2 f2sub(float2 a, float2 b)
{
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ P2 padd(const P2& a, const P2& b) { return {__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)}; }
__device__ __forceinline__ P2 psub(const P2& a, const P2& b) { return {f2sub(a.re, b.re), f2sub(a.im, b.im)}; }
// a - i b and a + i b
__device__ __forceinline__ P2 pami(const P2& a, const P2& b) { return {__fadd2_rn(a.re, b.im), f2sub(a.im, b.re)}; }
__device__ __forceinline__ P2 papi(const P2& a, const P2& b) { return {f2sub(a.re, b.im), __fadd2_rn(a.im, b.re)}; }
// Additions are packed; multiplications by one factor for both lines are scalar: they take the same
// time in the FMA pipe, and a packed one needs its factor twice in neighbouring registers first.
__device__ __forceinline__ P2 pscale(const P2& a, float s)
{
    return {make_float2(a.re.x * s, a.re.y * s), make_float2(a.im.x * s, a.im.y * s)};
}
// a + s b (real s)
__device__ __forceinline__ P2 paxpy(const P2& a, const P2& b, float s)
{
    return {make_float2(fmaf(b.re.x, s, a.re.x), fmaf(b.re.y, s, a.re.y)),
            make_float2(fmaf(b.im.x, s, a.im.x), fmaf(b.im.y, s, a.im.y))};
}
// both lines times one complex factor
__device__ __forceinline__ P2 pmul(const P2& a, float2 w)
{
    return {make_float2(fmaf(-a.im.x, w.y, a.re.x * w.x), fmaf(-a.im.y, w.y, a.re.y * w.x)),
            make_float2(fmaf(a.im.x, w.x, a.re.x * w.y), fmaf(a.im.y, w.x, a.re.y * w.y))};
}
// each line times its own complex factor (fr, fi: the factors' real and imaginary pairs)
__device__ __forceinline__ P2 pmul2(const P2& a, float2 fr, float2 fi)
{
    return {f2sub(__fmul2_rn(a.re, fr), __fmul2_rn(a.im, fi)), __ffma2_rn(a.im, fr, __fmul2_rn(a.re, fi))};
}

// ------------------------------------------------------------------------------------------------
// small forward DFTs (exp(-2 pi i n k / R)) on pairs, in place, natural order in and out
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void pd2(P2& a, P2& b)
{
    const P2 t = a;
    a = padd(t, b);
    b = psub(t, b);
}
__device__ __forceinline__ void pd3(P2& a, P2& b, P2& c)
{
    const float s = 0.86602540378443864676f;
    const P2 t1 = padd(b, c), t2 = paxpy(a, t1, -0.5f), t3 = pscale(psub(b, c), s);
    a = padd(a, t1);
    b = pami(t2, t3);
    c = papi(t2, t3);
}
__device__ __forceinline__ void pd4(P2& a, P2& b, P2& c, P2& d)
{
    const P2 s0 = padd(a, c), s1 = psub(a, c), s2 = padd(b, d), s3 = psub(b, d);
    a = padd(s0, s2);
    c = psub(s0, s2);
    b = pami(s1, s3);
    d = papi(s1, s3);
}
__device__ __forceinline__ void pd5(P2& a, P2& b, P2& c, P2& d, P2& e)
{
    const float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;
    const float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;
    const P2 t1 = padd(b, e), t2 = padd(c, d), t3 = psub(b, e), t4 = psub(c, d);
    const P2 a1 = paxpy(paxpy(a, t1, c1), t2, c2), a2 = paxpy(paxpy(a, t1, c2), t2, c1);
    const P2 b1 = paxpy(pscale(t3, s1), t4, s2), b2 = paxpy(pscale(t3, s2), t4, -s1);
    a = padd(a, padd(t1, t2));
    b = pami(a1, b1);
    e = papi(a1, b1);
    c = pami(a2, b2);
    d = papi(a2, b2);
}
// odd prime R from the symmetric pairs v_k +- v_(R-k): the real parts of the roots weigh the sums,
// the imaginary ones the differences
template <int R> __device__ __forceinline__ constexpr float odd_cos(int h)
{
    if constexpr (R == 7) {
        return h == 1 ? 0.62348980185873359f : h == 2 ? -0.22252093395631434f : -0.90096886790241903f;
    }
    if constexpr (R == 11) {
        return h == 1 ? 0.84125353283118121f : h == 2 ? 0.41541501300188644f : h == 3 ? -0.14231483827328500f : 
               h == 4 ? -0.65486073394528499f : -0.95949297361449737f;
    }
    if constexpr (R == 13) {
        return h == 1 ? 0.88545602565320991f : h == 2 ? 0.56806474673115592f : h == 3 ? 0.12053668025532301f : 
               h == 4 ? -0.35460488704253545f : h == 5 ? -0.74851074817110119f : -0.97094181742605201f;
    }
    return 0.f;
}
template <int R> __device__ __forceinline__ constexpr float odd_sin(int h)
{
    if constexpr (R == 7) {
        return h == 1 ? 0.78183148246802980f : h == 2 ? 0.97492791218182362f : 0.43388373911755823f;
    }
    if constexpr (R == 11) {
        return h == 1 ? 0.54064081745559756f : h == 2 ? 0.90963199535451833f : h == 3 ? 0.98982144188093280f : 
               h == 4 ? 0.75574957435425827f : 0.28173255684142967f;
    }
    if constexpr (R == 13) {
        return h == 1 ? 0.46472317204376851f : h == 2 ? 0.82298386589365635f : h == 3 ? 0.99270887409805397f : 
               h == 4 ? 0.93501624268541483f : h == 5 ? 0.66312265824079519f : 0.23931566428755768f;
    }
    return 0.f;
}
template <int R> __device__ __forceinline__ void pdodd(P2* v)
{
    constexpr int H = R / 2;
    P2 a[H + 1], b[H + 1], sum = v[0];
#pragma unroll
    for (int k = 1; k <= H; k++) {
        a[k] = padd(v[k], v[R - k]);
        b[k] = psub(v[k], v[R - k]);
        sum = padd(sum, a[k]);
    }
    const P2 v0 = v[0];
    v[0] = sum;
#pragma unroll
    for (int m = 1; m <= H; m++) {
        P2 x = v0, y;
#pragma unroll
        for (int k = 1; k <= H; k++) {
            const int q = (m * k) % R, h = q <= H ? q : R - q;
            const float c = odd_cos<R>(h), s = q <= H ? odd_sin<R>(h) : -odd_sin<R>(h);
            x = paxpy(x, a[k], c);
            y = k == 1 ? pscale(b[k], s) : paxpy(y, b[k], s);
        }
        v[m] = pami(x, y);
        v[R - m] = papi(x, y);
    }
}

template <int R> __device__ __forceinline__ void pdft(P2* v);

// R = A B, A and B coprime (Good 1958, Thomas 1963): inputs B n1 + A n2, outputs k with k mod A, k mod B:
// no twiddles between the two
template <int A, int B> __device__ __forceinline__ void pdpfa(P2* v)
{
    constexpr int R = A * B;
    P2 y[A][B];
#pragma unroll
    for (int n2 = 0; n2 < B; n2++) {
        P2 t[A];
#pragma unroll
        for (int n1 = 0; n1 < A; n1++) t[n1] = v[(B * n1 + A * n2) % R];
        pdft<A>(t);
#pragma unroll
        for (int k1 = 0; k1 < A; k1++) y[k1][n2] = t[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) pdft<B>(y[k1]);
#pragma unroll
    for (int k = 0; k < R; k++) v[k] = y[k % A][k % B];
}

// v times exp(-i pi m / 4) for m = 1 (1 - i)/sqrt 2 and m = 3 (-1 - i)/sqrt 2
__device__ __forceinline__ P2 pw8(const P2& v)
{
    const float h = 0.70710678118654752440f;
    return pscale({__fadd2_rn(v.re, v.im), f2sub(v.im, v.re)}, h);
}
__device__ __forceinline__ P2 pw83(const P2& v)
{
    const float h = 0.70710678118654752440f;
    const float2 a = f2sub(v.im, v.re), b = __fadd2_rn(v.re, v.im);
    return {make_float2(a.x * h, a.y * h), make_float2(b.x * -h, b.y * -h)};
}

__device__ __forceinline__ void pd8(P2* v)
{
    pd4(v[0], v[2], v[4], v[6]);
    pd4(v[1], v[3], v[5], v[7]);
    const P2 o0 = v[1], o1 = pw8(v[3]), o2 = v[5], o3 = pw83(v[7]);
    const P2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = padd(e0, o0);
    v[4] = psub(e0, o0);
    v[1] = padd(e1, o1);
    v[5] = psub(e1, o1);
    v[2] = pami(e2, o2);
    v[6] = papi(e2, o2);
    v[3] = padd(e3, o3);
    v[7] = psub(e3, o3);
}

__device__ __forceinline__ void pd9(P2* v)
{
    const float2 w1 = make_float2(0.76604444311897803520f, -0.64278760968653932632f);
    const float2 w2 = make_float2(0.17364817766693034885f, -0.98480775301220805937f);
    const float2 w4 = make_float2(-0.93969262078590838405f, -0.34202014332566873304f);
#pragma unroll
    for (int n = 0; n < 3; n++) pd3(v[n], v[n + 3], v[n + 6]);      // v[n + 3 k1]
    v[4] = pmul(v[4], w1);
    v[5] = pmul(v[5], w2);
    v[7] = pmul(v[7], w2);
    v[8] = pmul(v[8], w4);
#pragma unroll
    for (int k = 0; k < 3; k++) pd3(v[3 * k], v[3 * k + 1], v[3 * k + 2]);   // k1 + 3 k2 at 3 k1 + k2
    P2 t;
    t = v[1]; v[1] = v[3]; v[3] = t;
    t = v[2]; v[2] = v[6]; v[6] = t;
    t = v[5]; v[5] = v[7]; v[7] = t;
}

__device__ __forceinline__ void pd16(P2* v)
{
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
    // n = 4 n1 + n2: columns of four, then twiddles W16^(n2 k1), then rows (k = k1 + 4 k2)
#pragma unroll
    for (int n = 0; n < 4; n++) pd4(v[n], v[n + 4], v[n + 8], v[n + 12]);
    v[5] = pmul(v[5], make_float2(c1, -s1));
    v[9] = pw8(v[9]);
    v[13] = pmul(v[13], make_float2(s1, -c1));
    v[6] = pw8(v[6]);
    v[14] = pw83(v[14]);
    v[7] = pmul(v[7], make_float2(s1, -c1));
    v[11] = pw83(v[11]);
    v[15] = pmul(v[15], make_float2(-c1, s1));
    // W16^4 = -i at (n2 = 2, k1 = 2): folded into that row's first additions
    {
        const P2 a = v[8], b = v[9], c = v[10], d = v[11];
        const P2 p0 = pami(a, c), p1 = papi(a, c), p2 = padd(b, d), p3 = psub(b, d);
        v[8] = padd(p0, p2);
        v[10] = psub(p0, p2);
        v[9] = pami(p1, p3);
        v[11] = papi(p1, p3);
    }
    pd4(v[0], v[1], v[2], v[3]);
    pd4(v[4], v[5], v[6], v[7]);
    pd4(v[12], v[13], v[14], v[15]);
    // output k1 + 4 k2 stands at 4 k1 + k2: transpose the 4 x 4 registers
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = a + 1; b < 4; b++) {
            const P2 t = v[4 * a + b];
            v[4 * a + b] = v[4 * b + a];
            v[4 * b + a] = t;
        }
}

template <int R> __device__ __forceinline__ void pdft(P2* v)
{
    if constexpr (R == 2) pd2(v[0], v[1]);
    else if constexpr (R == 3) pd3(v[0], v[1], v[2]);
    else if constexpr (R == 4) pd4(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 5) pd5(v[0], v[1], v[2], v[3], v[4]);
    else if constexpr (R == 6) pdpfa<2, 3>(v);
    else if constexpr (R == 8) pd8(v);
    else if constexpr (R == 9) pd9(v);
    else if constexpr (R == 10) pdpfa<2, 5>(v);
    else if constexpr (R == 12) pdpfa<4, 3>(v);
    else if constexpr (R == 14) pdpfa<2, 7>(v);
    else if constexpr (R == 15) pdpfa<3, 5>(v);
    else if constexpr (R == 16) pd16(v);
    else pdodd<R>(v);
}

// twiddles of a stage: v_k *= w^k from its table (entry m of each of its rows of `pitch` entries), loaded before the
// butterfly's inputs.  A product of two table entries has their roundings and its own: with products of up to
// four entries (1, 2, 4, 8) at every radix, propagations between drifts at 64^2, 256^2, 512^2 and 2048^2 were
// 4.0, 4.8, 3.8 and 4.9e-7 off in 64 bits, with the rows of tw_power 2.9, 3.1, 2.5 and 4.2e-7, for 0 to 2 %
// of the time (512^2 30.5 us either way, 2048^2 211 to 213, 2240 x 1536, where registers are short, 212 to
// 215).  A sixth row for radix 16 (power 3) gives 3.9e-7 at 2048^2 and takes 221 us.
template <int R> struct TwP {
    float2 w[tw_rows(R)];
};
template <int R> __device__ __forceinline__ TwP<R> ptwload(const float2* __restrict__ tw, int m, int pitch)
{
    TwP<R> p;
#pragma unroll
    for (int e = 0; e < tw_rows(R); e++) p.w[e] = __ldg(&tw[m + e * pitch]);
    return p;
}
template <int R> __device__ __forceinline__ void ptwiddle(P2* v, const TwP<R>& p)
{
#pragma unroll
    for (int r = 1; r < R; r++) {
        float2 w;
        if constexpr (R <= 8) {
            w = p.w[r - 1];
        } else if constexpr (R == 16) {
            const float2 lo = r % 4 == 3 ? cmul(p.w[0], p.w[1]) : p.w[r % 4 == 2];
            const float2 hi = r / 4 == 3 ? p.w[4] : p.w[r / 4 == 2 ? 3 : 2];
            w = r < 4 ? lo : r % 4 == 0 ? hi : cmul(lo, hi);
        } else {
            bool first = true;
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (r & (1 << e)) { w = first ? p.w[e] : cmul(w, p.w[e]); first = false; }
        }
        v[r] = pmul(v[r], w);
    }
}

// a thread's view of its pair of lines: uniform base pointers and 32-bit element offsets
struct PLine {
    const float2* g0;       // input: point q of line 0 at g0[ioff + q gstr], of line 1 at g1[...]
    const float2* g1;
    const float2 *sg0, *sg1;  // bulk-copied input: point q of line 0 at sg0[(q - za0) gstr], of line 1 at sg1[...]
    unsigned ioff;
    bool full;              // every point of both lines has input
    int gstr, vin;          // vin: the two values are one aligned 16-byte load at g0
    bool in0, in1;          // the line has input (else zeros)
    int za0;                // input points outside [za0, za0 + zn] are zero
    unsigned zn;
    float2* o0;             // output: point k of line 0 at o0[ooff + place(k)], of line 1 at o1[...]
    float2* o1;
    unsigned ooff;
    int ostr, lg, bstr;     // place(k) = k ostr, or (lg >= 0) (k >> lg) bstr + (k & (2^lg - 1))
    int vout;
    bool st0, st1;          // the line is stored
    const float2* tabs;
    const PwOps* ex;
    int line0, line1;
    float* si;              // intensity line in shared memory
    const unsigned* mask;   // columns: a bit per output point that is read (NULL: all of them are)
    bool has_lf;
    float2 lfr, lfi;        // line factors
    const float* qtab;      // quartic angular term (EXTRA 1): q^2 along the line, of the two lines, coefficients
    float2 ql;
    float qc0, qc1;
    bool qsmall;
    __device__ __forceinline__ int place(int k) const
    {
        return lg < 0 ? k * ostr : (k >> lg) * bstr + (k & ((1 << lg) - 1));
    }
};

// a chain: destination p takes source index s(p) = rot_out(mirror(rot_in(p))) times tab[p] (and the
// non-separable work at index mirror(rot_in(p)))
struct PChain {
    int rot_in, mir, rot_out;
    int tab, extra;
};
__device__ __forceinline__ int prot(int p, int N, int on)
{
    const int q = p + (on ? (N >> 1) : 0);
    return q >= N ? q - N : q;
}
__device__ __forceinline__ int pindex(const PChain& c, int p, int N)
{
    const int m = prot(p, N, c.rot_in);
    return c.mir ? N - 1 - m : m;
}

// non-separable factors of both lines at index i, out of line (rare, and costly at every point)
template <bool COLS> __device__ __noinline__ float4 linep_extra(const PwOps* ex, int i, int l0, int l1, const float2* tabs)
{
    float2 f[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        bool zero = false;
        f[k] = make_float2(1.f, 0.f);
        const int l = k ? l1 : l0;
        extra_eval(*ex, COLS ? l : i, COLS ? i : l, f[k], zero, tabs);
        if (zero) f[k] = make_float2(0.f, 0.f);
    }
    return make_float4(f[0].x, f[1].x, f[0].y, f[1].y);
}
template <bool COLS> __device__ __forceinline__ P2 pextra(const P2& v, const PLine& x, int i)
{
    const float4 f = linep_extra<COLS>(x.ex, i, x.line0, x.line1, x.tabs);
    return pmul2(v, make_float2(f.x, f.y), make_float2(f.z, f.w));
}
// cos and sin of a phase pair: series for |phase| < 0.0375 (next terms: sine 6e-10, cosine 4e-12), else the hardware's
__device__ __forceinline__ P2 pcis(float2 ph, bool small)
{
    P2 f;
    if (small) {
        const float2 p2 = __fmul2_rn(ph, ph);
        f.re = make_float2(fmaf(p2.x, fmaf(p2.x, 1.f / 24.f, -0.5f), 1.f), fmaf(p2.y, fmaf(p2.y, 1.f / 24.f, -0.5f), 1.f));
        f.im = make_float2(fmaf(ph.x * p2.x, -1.f / 6.f, ph.x), fmaf(ph.y * p2.y, -1.f / 6.f, ph.y));
    } else {
        __sincosf(ph.x, &f.im.x, &f.re.x);
        __sincosf(ph.y, &f.im.y, &f.re.y);
    }
    return f;
}
template <int R> __device__ __forceinline__ void pconj(P2 (&v)[R])
{
#pragma unroll
    for (int r = 0; r < R; r++) v[r].im = __fmul2_rn(v[r].im, make_float2(-1.f, -1.f));
}

// the R inputs p = j + r L1 of butterfly j from global memory through the input chain.  R is even, so
// the centring rotation is +N/2 for the lower half of r and -N/2 for the upper one, and a source
// index is a base plus r steps.
template <int R, bool COLS, int EXTRA, bool VEC>
__device__ __forceinline__ void pload(P2 (&v)[R], const PLine& x, const PChain& c, int j, int L1, int N, float cj)
{
    static_assert(R % 2 == 0, "first radix");
    const int h = (c.rot_in != c.rot_out) ? (N >> 1) : 0;
    float4 a[R];
    if (x.full && !c.mir) {
        // no window, no mirror: unconditional loads at a pointer per half (row-major rows: constant distances)
        // (the upper half's base may lie before the field: signed distances)
        if (VEC && x.vin) {
            const int gs = x.gstr;
            const float2 *pA = x.g0 + ((long long)x.ioff + (j + h) * gs), *pB = x.g0 + ((long long)x.ioff + (j - h) * gs);
#pragma unroll
            for (int r = 0; r < R; r++)
                a[r] = ldfield4((r < R / 2 ? pA : pB) + r * L1 * gs);
        } else {
            const int gs = COLS ? x.gstr : 1;
            const long long eA = (long long)x.ioff + (j + h) * gs, eB = (long long)x.ioff + (j - h) * gs;
            const float2 *pA = x.g0 + eA, *pB = x.g0 + eB, *qA = x.g1 + eA, *qB = x.g1 + eB;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float2 t0 = ldfield((r < R / 2 ? pA : pB) + r * L1 * gs);
                const float2 t1 = ldfield((r < R / 2 ? qA : qB) + r * L1 * gs);
                a[r] = make_float4(t0.x, t0.y, t1.x, t1.y);
            }
        }
    } else {
        const int q0 = c.mir ? N - 1 - j : j, hs = c.mir ? -h : h, qs = c.mir ? -L1 : L1;
        const int gs = x.gstr;
        const unsigned oA = x.ioff + (unsigned)((q0 + hs) * gs), oB = x.ioff + (unsigned)((q0 - hs) * gs);
        const unsigned os = (unsigned)(qs * gs);
        const int wA = q0 + hs - x.za0, wB = q0 - hs - x.za0;
        auto in = [&](int r) { return (unsigned)((r < R / 2 ? wA : wB) + r * qs) <= x.zn; };
        auto at = [&](int r) { return (r < R / 2 ? oA : oB) + (unsigned)r * os; };
#pragma unroll
        for (int r = 0; r < R; r++) a[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (x.sg0 != nullptr) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int e = ((r < R / 2 ? wA : wB) + r * qs) * gs;
                if (in(r)) {
                    const float2 t0 = x.sg0[e], t1 = x.sg1[e];
                    a[r] = make_float4(t0.x, t0.y, t1.x, t1.y);
                }
            }
        } else if (VEC && x.vin) {
#pragma unroll
            for (int r = 0; r < R; r++) ldfield4_if(in(r), x.g0 + at(r), a[r]);
        } else {
#pragma unroll
            for (int r = 0; r < R; r++) {
                ldfield_if(in(r) && x.in0, x.g0 + at(r), a[r].x, a[r].y);
                ldfield_if(in(r) && x.in1, x.g1 + at(r), a[r].z, a[r].w);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        v[r].re = make_float2(a[r].x, a[r].z);
        v[r].im = make_float2(a[r].y, a[r].w);
    }
    if (!(x.in0 && x.in1) && !x.full) {              // a pair at the edge of the window: one line is zero
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r].re = make_float2(x.in0 ? v[r].re.x : 0.f, x.in1 ? v[r].re.y : 0.f);
            v[r].im = make_float2(x.in0 ? v[r].im.x : 0.f, x.in1 ? v[r].im.y : 0.f);
        }
    }
    if (c.tab >= 0) {
        const float2* tb = x.tabs + c.tab + j;
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = pmul(v[r], __ldg(tb + r * L1));
    }
    if (EXTRA == 2 && c.extra) {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = pextra<COLS>(v[r], x, pindex(c, j + r * L1, N));
    }
    if (cj < 0.f) pconj(v);
}

// one output of both lines to p0 and p1; OUTI: the intensity of the pair (both components) as one float
template <bool COLS, int OUTI>
__device__ __forceinline__ void pput(const P2& o, const PLine& x, void* p0, float2* p1, float iscale, bool on = true)
{
    if (OUTI) {
        const float2 I = __ffma2_rn(o.im, o.im, __fmul2_rn(o.re, o.re));
        if (x.st0) __stcs(reinterpret_cast<float*>(p0), (I.x + I.y) * iscale);
    } else if (COLS && x.vout) {
        if (x.st0 && on) __stcs(reinterpret_cast<float4*>(p0), make_float4(o.re.x, o.im.x, o.re.y, o.im.y));
    } else {
        if (x.st0 && on) __stcs(reinterpret_cast<float2*>(p0), make_float2(o.re.x, o.im.x));
        if (x.st1 && on) __stcs(p1, make_float2(o.re.y, o.im.y));
    }
}

// the output chain's factors on the R outputs with destinations kk(r): the table's values are loaded
// together (a load per output between its stores waited for each in turn)
template <int R, bool COLS, int EXTRA, class KK>
__device__ __forceinline__ void pfactors(P2 (&v)[R], const PLine& x, const PChain& c, int N, const KK& kk)
{
    if (c.tab >= 0) {
        const float2* tb = x.tabs + c.tab;
        constexpr int H = R > 8 ? (R + 1) / 2 : R;       // (more at once does not fit the registers)
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += H) {
            float2 f[H];
#pragma unroll
            for (int r = 0; r < H; r++)
                if (r0 + r < R) f[r] = __ldg(tb + kk(r0 + r));
#pragma unroll
            for (int r = 0; r < H; r++)
                if (r0 + r < R) v[r0 + r] = pmul(v[r0 + r], f[r]);
        }
    }
    if (EXTRA == 2 && c.extra) {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = pextra<COLS>(v[r], x, pindex(c, kk(r), N));
    }
    if (x.has_lf) {
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = pmul2(v[r], x.lfr, x.lfi);
    }
}

// the R outputs u + r M of a line's last stage through the output chain: OUTI 0 the fields, 1 the intensity
// of the pair (both components) to global memory, 2 that intensity to shared memory
template <int R, bool COLS, int EXTRA, int OUTI>
__device__ __forceinline__ void pstore(P2 (&v)[R], const PLine& x, const PChain& c, int u, int M, int N, float cj,
                                       float iscale)
{
    if (cj < 0.f) pconj(v);
    if constexpr (OUTI == 2) {
        // the intensity of the pair, in shared memory
        auto kk = [&](int r) {
            const int k = prot(u + r * M, N, c.rot_out);
            return c.mir ? N - 1 - k : k;
        };
        pfactors<R, COLS, EXTRA>(v, x, c, N, kk);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float2 I = __ffma2_rn(v[r].im, v[r].im, __fmul2_rn(v[r].re, v[r].re));
            x.si[kk(r)] = (I.x + I.y) * iscale;
        }
        return;
    }
    constexpr int EB = OUTI ? 4 : 8;                     // bytes of an output element
    auto wanted = [&](auto&& kk) {                       // bit r: point kk(r) is read
        unsigned on = ~0u;
        if (COLS && OUTI == 0 && x.mask != nullptr) {
            on = 0;
#pragma unroll
            for (int r = 0; r < R; r++) on |= ((__ldg(x.mask + (kk(r) >> 5)) >> (kk(r) & 31)) & 1u) << r;
        }
        return on;
    };
    const int h = c.rot_out ? (N >> 1) : 0;
    char* b0 = reinterpret_cast<char*>(x.o0);
    char* b1 = reinterpret_cast<char*>(x.o1);
    if (!COLS && x.lg < 0 && !c.mir && (R % 2 == 0 || h == 0)) {
        // rows, row-major, no mirror: constant distances from a pointer per half
        // (the upper half's base may lie before the field: signed distances)
        const long long eA = ((long long)x.ooff + (u + h)) * EB, eB = ((long long)x.ooff + (u - h)) * EB;
        char *pA = b0 + eA, *pB = b0 + eB, *qA = b1 + eA, *qB = b1 + eB;
        pfactors<R, COLS, EXTRA>(v, x, c, N, [&](int r) { return (r < R / 2 ? u + h : u - h) + r * M; });
#pragma unroll
        for (int r = 0; r < R; r++)
            pput<COLS, OUTI>(v[r], x, (r < R / 2 ? pA : pB) + r * M * EB,
                             reinterpret_cast<float2*>((r < R / 2 ? qA : qB) + r * M * EB), iscale);
    } else if ((R % 2 == 0 || h == 0) && (x.lg < 0 || (M & ((1 << x.lg) - 1)) == 0)) {
        // destinations and their places are a base (per half of r) plus r steps
        const int kA = c.mir ? N - 1 - (u + h) : u + h, kB = c.mir ? N - 1 - (u - h) : u - h, ks = c.mir ? -M : M;
        const unsigned pA = x.ooff + (unsigned)x.place(kA), pB = x.ooff + (unsigned)x.place(kB);
        const unsigned ps = (unsigned)(x.lg < 0 ? ks * x.ostr : (ks >> x.lg) * x.bstr);
        const unsigned on = wanted([&](int r) { return (r < R / 2 ? kA : kB) + r * ks; });
        pfactors<R, COLS, EXTRA>(v, x, c, N, [&](int r) { return (r < R / 2 ? kA : kB) + r * ks; });
#pragma unroll
        for (int r = 0; r < R; r++) {
            const unsigned o = (r < R / 2 ? pA : pB) + (unsigned)r * ps;
            pput<COLS, OUTI>(v[r], x, b0 + (size_t)o * EB, reinterpret_cast<float2*>(b1 + (size_t)o * EB), iscale,
                             (on >> r) & 1u);
        }
    } else {
        auto kk = [&](int r) {
            const int k = prot(u + r * M, N, c.rot_out);
            return c.mir ? N - 1 - k : k;
        };
        const unsigned on = wanted(kk);
        pfactors<R, COLS, EXTRA>(v, x, c, N, kk);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const unsigned o = x.ooff + (unsigned)x.place(kk(r));
            pput<COLS, OUTI>(v[r], x, b0 + (size_t)o * EB, reinterpret_cast<float2*>(b1 + (size_t)o * EB), iscale,
                             (on >> r) & 1u);
        }
    }
}

__device__ __forceinline__ P2 lds2(const float4* s)
{
    const float4 a = *s;
    return {make_float2(a.x, a.y), make_float2(a.z, a.w)};
}
__device__ __forceinline__ void sts2(float4* s, const P2& v) { *s = make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }

#define LINEP_EVEN(X) X(2) X(4) X(6) X(8) X(10) X(12) X(14) X(16)
#define LINEP_ALL(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

// ------------------------------------------------------------------------------------------------
// stages
// ------------------------------------------------------------------------------------------------
template <int R, class Z, bool COLS, int EXTRA, bool VEC>
__device__ __forceinline__ void run_first(const Z& z, float4* s, const PLine& x, const PChain& c, float cj,
                                          const float2* __restrict__ tw, int t)
{
    const int L1 = z.L(1);
#pragma unroll 1
    for (int j = t; j < L1; j += z.T()) {
        const TwP<R> wp = ptwload<R>(tw + z.tw1(0), j, L1);
        P2 v[R];
        pload<R, COLS, EXTRA, VEC>(v, x, c, j, L1, z.N(), cj);
        pdft<R>(v);
        ptwiddle<R>(v, wp);
#pragma unroll
        for (int k = 0; k < R; k++) sts2(s + k * z.pitch() + j, v[k]);
    }
}

// FWD: twiddles of the first transform (position below the digit), else of the second (digits below)
template <int R, class Z, bool FWD>
__device__ __forceinline__ void run_mid(const Z& z, int st, float4* s, const float2* __restrict__ tw, int t)
{
    const int nb = z.N() / R, Ls = z.L(st + 1);
    const float2* tb = tw + (FWD ? z.tw1(st) : z.tw2(st));
    const int tp = FWD ? Ls : z.N() / z.L(st);
#pragma unroll 1
    for (int b = t; b < nb; b += z.T()) {
        int w, o;
        float4* a = s + place_mid(z, st, b, w, o);
        const TwP<R> wp = ptwload<R>(tb, FWD ? o : low_index(z, st, w), tp);
        P2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = lds2(a + r * Ls);
        pdft<R>(v);
        ptwiddle<R>(v, wp);
#pragma unroll
        for (int r = 0; r < R; r++) sts2(a + r * Ls, v[r]);
    }
}

template <int R, class Z, bool COLS, int EXTRA, int OUTI>
__device__ __forceinline__ void run_last(const Z& z, float4* s, const PLine& x, const PChain& c, float cj,
                                         float iscale, int t)
{
    const int M = z.N() / R;
#pragma unroll 1
    for (int u = t; u < M; u += z.T()) {
        const float4* a = s + place_last(z, u);
        P2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = lds2(a + r);
        pdft<R>(v);
        pstore<R, COLS, EXTRA, OUTI>(v, x, c, u, M, z.N(), cj, iscale);
    }
}

// last stage of the first transform, middle chain, first stage of the second transform
template <int R, class Z, bool COLS, int EXTRA>
__device__ __forceinline__ void run_turn(const Z& z, float4* s, const PLine& x, const PChain& c, float cj1,
                                         float cj2, const float2* __restrict__ tw, int t)
{
    const int M = z.N() / R;
#pragma unroll 1
    for (int u = t; u < M; u += z.T()) {
        float4* a = s + place_last(z, u);
        const TwP<R> wp = ptwload<R>(tw + z.tw2(z.n() - 1), u, M);
        P2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = lds2(a + r);
        pdft<R>(v);
        if (cj1 < 0.f) pconj(v);
        if (c.tab >= 0) {
            const float2* tb = x.tabs + c.tab + u;
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = pmul(v[r], __ldg(tb + r * M));
        }
        if (EXTRA == 1) {
            // quartic part of the angular transfer function, from the tables of q^2
            const float* qt = x.qtab + u;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float q = __ldg(qt + r * M);
                const float2 q2 = __fadd2_rn(make_float2(q, q), x.ql);
                const float2 k = make_float2(x.qc1 * q2.x, x.qc1 * q2.y);
                const float2 ph = make_float2(x.qc0 * q2.x * k.x * fmaf(2.f, k.x, 1.f), x.qc0 * q2.y * k.y * fmaf(2.f, k.y, 1.f));
                const P2 f = pcis(ph, x.qsmall);
                v[r] = pmul2(v[r], f.re, f.im);
            }
        }
        if (EXTRA == 2 && c.extra) {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = pextra<COLS>(v[r], x, pindex(c, u + r * M, z.N()));
        }
        if (cj2 < 0.f) pconj(v);
        pdft<R>(v);
        ptwiddle<R>(v, wp);
#pragma unroll
        for (int r = 0; r < R; r++) sts2(a + r, v[r]);
    }
}

// last stage of the second transform, over k1
template <int R, class Z, bool COLS, int EXTRA>
__device__ __forceinline__ void run_back(const Z& z, float4* s, const PLine& x, const PChain& c, float cj, int t)
{
    const int M = z.L(1);
#pragma unroll 1
    for (int b = t; b < M; b += z.T()) {
        const float4* a = s + place_back(z, b);
        P2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = lds2(a + r * z.pitch());
        pdft<R>(v);
        pstore<R, COLS, EXTRA, false>(v, x, c, b, M, z.N(), cj, 1.f);
    }
}

// MODE 0: one transform, 1: two transforms, 2: one transform and the intensity of both components.
// Z: the length's schedule, fixed at compile time (FShape) or from the launch (PShape)
template <class Z, bool COLS, int MODE, int EXTRA>
__global__ void __launch_bounds__(Z::bound, 1) linep_kernel(const LineArgs p)
{
    constexpr bool INT = MODE == 2;
    constexpr int LPP = INT ? 1 : 2;                     // lines per pair
    extern __shared__ float4 smp[];
    pdl_launch();
    Z z;
    if constexpr (!Z::fixed) {
        z.N_ = p.N; z.n_ = p.nst; z.T_ = p.T; z.pitch_ = p.pitch;
        z.R_ = p.radix; z.L_ = p.len; z.dL = p.dL; z.dR = p.dR; z.dB = p.dB; z.t1 = p.tw1; z.t2 = p.tw2;
    }
    const LineDesc* gd = reinterpret_cast<const LineDesc*>(reinterpret_cast<const char*>(p.gd) + blockIdx.z * p.bDesc);
    LineRun d;
    if (p.byValue) d = p.run;
    else d = gd->run;
    const int comp = INT ? 0 : blockIdx.y;
    const float2* src = p.src[comp] + blockIdx.z * p.bSrc;
    float2* dst = p.dst[comp] + blockIdx.z * p.bDst;
    const int N = z.N(), nl = p.nlines, Lp = p.G, tid = threadIdx.x;
    const int g = COLS ? tid % Lp : tid / z.T();
    const int t = COLS ? tid / Lp : tid - g * z.T();
    // a pass that writes only its window's lines starts at this wavefront's first block of them
    const int bx = blockIdx.x + (d.zwin && d.zskip ? d.zl0 / p.L : 0);
    PLine x;
    int line0 = (bx * Lp + g) * LPP;
    const bool valid = line0 < nl;
    if (!valid) line0 = nl - LPP;                        // surplus threads compute a copy, store nothing
    x.line0 = line0;
    x.line1 = INT ? line0 : line0 + 1;                   // (pairs: an even number of lines)
    x.st0 = x.st1 = valid;
    float4* s = smp + g * p.P;
    // input: row-major, or blocks of blk_in lines stored together; only the window where it is stored alone
    const int ip = d.in_p;
    x.gstr = COLS ? ip : 1;
    x.ioff = COLS ? (unsigned)(line0 - d.in_l0 - d.in_q0 * ip) : (unsigned)((line0 - d.in_l0) * ip - d.in_q0);
    x.g0 = src;
    x.g1 = src + (COLS || d.blk_in > 0 ? 1 : ip);
    bool pairIn = COLS || d.blk_in > 0;
    if (d.blk_in > 0) {
        x.gstr = d.blk_in;
        x.ioff = (unsigned)((line0 / d.blk_in * ip - d.in_q0) * d.blk_in + line0 % d.blk_in);
    }
    if (INT) {
        x.g1 = p.src[1] + blockIdx.z * p.bSrc;
        pairIn = false;
    }
    x.vin = pairIn && p.alignIn;
    const int o0 = d.mirror_lines ? nl - 1 - line0 : line0, od = d.mirror_lines ? -1 : 1;
    const int op = d.out_p;
    x.ooff = COLS ? (unsigned)(o0 - d.out_l0) : (unsigned)((o0 - d.out_l0) * op);
    x.ostr = COLS ? op : 1;
    x.lg = -1;
    x.bstr = 0;
    x.o0 = dst;
    x.o1 = dst + (COLS ? od : od * op);
    x.vout = COLS && p.alignOut && od == 1;
    if (!INT && d.blk_out > 0) {
        x.lg = 31 - __clz(d.blk_out);
        x.bstr = op * d.blk_out;
        x.ooff = (unsigned)((o0 - d.out_l0) * d.blk_out);
        x.o1 = dst + od * d.blk_out;
        x.vout = 0;
    }
    if (COLS && INT && d.blk_out > 0) {
        x.ostr = d.blk_out;
        x.ooff = (unsigned)(o0 / d.blk_out) * (unsigned)(N * d.blk_out) + (unsigned)(o0 % d.blk_out);
    }
    if (INT) x.o0 = reinterpret_cast<float2*>(reinterpret_cast<float*>(p.dst[0]) + blockIdx.z * p.bDst);
    x.za0 = 0;
    x.zn = N - 1;
    x.in0 = x.in1 = true;
    x.full = COLS || d.blk_in == 0 || x.vin;             // (rows' plain path: distance 1 between points)
    if (d.zwin) {
        const int l0 = bx * p.L, l1 = min(l0 + p.L, nl) - 1;
        if (l1 < d.zl0 || l0 > d.zl1) {
            pdl_wait();
            // every line of the tile is zero, and so is its transform
            if (INT || !d.zskip)
                for (int k = t; k < N; k += z.T()) {
                    const unsigned o = x.ooff + (unsigned)x.place(k);
                    if (INT) {
                        if (x.st0) __stcs(reinterpret_cast<float*>(x.o0) + o, 0.f);
                    } else {
                        if (x.st0) __stcs(x.o0 + o, make_float2(0.f, 0.f));
                        if (x.st1) __stcs(x.o1 + o, make_float2(0.f, 0.f));
                    }
                }
            return;
        }
        x.in0 = line0 >= d.zl0 && line0 <= d.zl1 && d.za0 <= d.za1;
        x.in1 = x.line1 >= d.zl0 && x.line1 <= d.zl1 && d.za0 <= d.za1;
        if (d.zskip && !INT) {                           // zero lines that nothing reads
            x.st0 = x.st0 && line0 >= d.zl0 && line0 <= d.zl1;
            x.st1 = x.st1 && x.line1 >= d.zl0 && x.line1 <= d.zl1;
        }
        x.full = false;
        x.za0 = d.za0;
        x.zn = (unsigned)max(d.za1 - d.za0, 0);
        if (!(x.in0 || x.in1)) x.vin = 0;
    }
    if (x.st0 != x.st1) x.vout = 0;
    x.sg0 = x.sg1 = nullptr;
    __shared__ uint64_t bar;
    pdl_wait();
    if (p.bulk && d.zwin && d.blk_in == p.L && d.za0 <= d.za1) {
        // the tile is one block of lines: its nonzero points lie together and arrive in shared memory,
        // behind the slots, by one bulk copy per component while the chains are set up
        float2* stg = reinterpret_cast<float2*>(smp + Lp * p.P);
        const int pts = (d.za1 - d.za0 + 1) * p.L;
        if (pts <= p.bulk) {
            const size_t o = ((size_t)bx * ip + (d.za0 - d.in_q0)) * p.L;
            if (tid == 0) {
                mbar_init(&bar);
                mbar_expect(&bar, (unsigned)(pts * sizeof(float2)) * (INT ? 2 : 1));
                bulk_load(stg, src + o, (unsigned)(pts * sizeof(float2)), &bar);
                if (INT) bulk_load(stg + p.bulk, x.g1 + o, (unsigned)(pts * sizeof(float2)), &bar);
            }
            x.sg0 = stg + g * LPP;
            x.sg1 = INT ? x.sg0 + p.bulk : x.sg0 + 1;
            x.vin = 0;
        }
    }
    x.mask = COLS && p.mask != nullptr ? p.mask + blockIdx.z * p.maskWords : nullptr;
    x.tabs = p.tabs + blockIdx.z * p.bTab;
    x.ex = EXTRA == 2 ? &gd->extra : nullptr;
    PChain pre, mid, fin;
    pre.rot_in = d.pre_rot; pre.mir = 0; pre.rot_out = 0; pre.tab = d.pre_tab; pre.extra = 0;
    mid.rot_in = d.mid_in; mid.mir = d.mid_mir; mid.rot_out = d.mid_out; mid.tab = d.mid_tab;
    mid.extra = EXTRA == 2 ? d.extra : 0;
    fin.rot_in = 0; fin.mir = 0; fin.rot_out = d.fin_rot; fin.tab = d.fin_tab; fin.extra = 0;
    float iscale = 1.f;
    x.has_lf = d.lt[0] >= 0;
    const bool one = MODE != 1 && d.dir1 != 0;           // the single transform is the first one
    if (INT && d.int_flat) {
        // the output factors have one magnitude: the intensity is scaled instead
        if (one) mid.tab = -1;
        else fin.tab = -1;
        x.has_lf = false;
        iscale = d.int_scale;
    }
    if (EXTRA == 1) {
        x.qtab = reinterpret_cast<const float*>(x.tabs + d.qtab);
        const float* ql = reinterpret_cast<const float*>(x.tabs + d.qline);
        x.ql = make_float2(__ldg(ql + line0), __ldg(ql + x.line1));
        x.qc0 = d.qc0;
        x.qc1 = d.qc1;
        x.qsmall = d.ang == 1;
    }
    // line factors: loaded before the last barrier, multiplied after it
    float2 fa[3], fb[3];
    auto load_factors = [&]() {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            fa[k] = fb[k] = make_float2(1.f, 0.f);
            if (x.has_lf && d.lt[k] >= 0) {
                fa[k] = __ldg(&x.tabs[d.lt[k] + line0]);
                fb[k] = __ldg(&x.tabs[d.lt[k] + x.line1]);
            }
        }
    };
    auto line_factors = [&]() {
        const float2 a = cmul(cmul(fa[0], fa[1]), fa[2]), b = cmul(cmul(fb[0], fb[1]), fb[2]);
        x.lfr = make_float2(a.x, b.x);
        x.lfi = make_float2(a.y, b.y);
    };
    if (x.sg0 != nullptr) {
        __syncthreads();                                 // (the barrier's initialisation)
        if (!mbar_wait_bounded(&bar, 0, p.spin > 0 ? p.spin : (1ll << 22), p.status)) return;
    }
    const float2* tw = p.tw;
    const float c1 = d.dir1 < 0 ? -1.f : 1.f, c2 = d.dir2 < 0 ? -1.f : 1.f;
    const PChain& cin = (MODE == 1 || one) ? pre : mid;
    const PChain& cout = one ? mid : fin;
    const float cjin = (MODE == 1 || one) ? c1 : c2;
    if constexpr (Z::fixed) {
        constexpr int n = Z::n(), RA = Z::R(0), RB = Z::R(1), RC = Z::R(2), RL = Z::R(Z::n() - 1);
        run_first<RA, Z, COLS, EXTRA, !INT>(z, s, x, cin, cjin, tw, t);
        if constexpr (n >= 3) { __syncthreads(); run_mid<RB, Z, true>(z, 1, s, tw, t); }
        if constexpr (n >= 4) { __syncthreads(); run_mid<RC, Z, true>(z, 2, s, tw, t); }
        if constexpr (MODE != 1) {
            load_factors();
            __syncthreads();
            line_factors();
            run_last<RL, Z, COLS, EXTRA, INT ? 1 : 0>(z, s, x, cout, cjin, iscale, t);
        } else {
            __syncthreads();
            run_turn<RL, Z, COLS, EXTRA>(z, s, x, mid, c1, c2, tw, t);
            if constexpr (n >= 4) { __syncthreads(); run_mid<RC, Z, false>(z, 2, s, tw, t); }
            if constexpr (n >= 3) { __syncthreads(); run_mid<RB, Z, false>(z, 1, s, tw, t); }
            load_factors();
            __syncthreads();
            line_factors();
            run_back<RA, Z, COLS, EXTRA>(z, s, x, fin, c2, t);
        }
    } else {
#define LINEP_FIRST(R_) case R_: run_first<R_, Z, COLS, EXTRA, !INT>(z, s, x, cin, cjin, tw, t); break;
        switch (z.R(0)) { LINEP_EVEN(LINEP_FIRST) default: break; }
        for (int st = 1; st + 1 < z.n(); st++) {
            __syncthreads();
#define LINEP_MID(R_) case R_: run_mid<R_, Z, true>(z, st, s, tw, t); break;
            switch (z.R(st)) { LINEP_ALL(LINEP_MID) default: break; }
        }
        if constexpr (MODE != 1) {
            load_factors();
            __syncthreads();
            line_factors();
#define LINEP_LAST(R_) case R_: run_last<R_, Z, COLS, EXTRA, INT ? 1 : 0>(z, s, x, cout, cjin, iscale, t); break;
            switch (z.R(z.n() - 1)) { LINEP_ALL(LINEP_LAST) default: break; }
        } else {
            __syncthreads();
#define LINEP_TURN(R_) case R_: run_turn<R_, Z, COLS, EXTRA>(z, s, x, mid, c1, c2, tw, t); break;
            switch (z.R(z.n() - 1)) { LINEP_ALL(LINEP_TURN) default: break; }
            for (int st = z.n() - 2; st >= 1; st--) {
                __syncthreads();
#define LINEP_MID2(R_) case R_: run_mid<R_, Z, false>(z, st, s, tw, t); break;
                switch (z.R(st)) { LINEP_ALL(LINEP_MID2) default: break; }
            }
            load_factors();
            __syncthreads();
            line_factors();
#define LINEP_BACK(R_) case R_: run_back<R_, Z, COLS, EXTRA>(z, s, x, fin, c2, t); break;
            switch (z.R(0)) { LINEP_EVEN(LINEP_BACK) default: break; }
        }
    }
}

// Last pass of a multi-electron batch along the rows, fused with the accumulation: only the rows the
// detector samples are transformed.  A CTA makes one detector row for several electrons in turn: the
// two output rows around it (one pair of both components per row), their intensities in shared
// memory, bilinear interpolation onto the detector row (avg_update_interp, order 1: nothing outside an
// electron's mesh) in FP64, summed over the CTA's electrons in their order; the groups' sums are added
// by accum_parts_kernel.  At 1536 x 1600 on 512^2 (a detector row per 5 output rows) it transforms 640 of
// the 1600 rows and writes no intensities.
template <class Z>
__global__ void __launch_bounds__(Z::bound, 1) linep_sample_kernel(const LineArgs p, const SampleArgs q)
{
    extern __shared__ float4 smp[];
    Z z;
    if constexpr (!Z::fixed) {
        z.N_ = p.N; z.n_ = p.nst; z.T_ = p.T; z.pitch_ = p.pitch;
        z.R_ = p.radix; z.L_ = p.len; z.dL = p.dL; z.dR = p.dR; z.dB = p.dB; z.t1 = p.tw1; z.t2 = p.tw2;
    }
    const int N = z.N(), nl = p.nlines, tid = threadIdx.x;
    const int g = tid / z.T(), t = tid - g * z.T();      // g: the output row below / above the detector row
    const int j = blockIdx.x, b1 = min(q.nb, (int)(blockIdx.y + 1) * q.per);
    float4* s = smp + g * p.P;
    float* I0 = reinterpret_cast<float*>(smp + 2 * p.P);
    float* I1 = I0 + N;
    double* acc = reinterpret_cast<double*>(I0 + 2 * N + (N & 1) * 2);
    for (int i = tid; i < q.anx; i += blockDim.x) acc[i] = 0.;
    PLine x;
    x.g0 = x.g1 = nullptr;
    x.sg0 = x.sg1 = nullptr;
    x.o0 = x.o1 = nullptr;
    x.ooff = 0;
    x.ostr = 1; x.lg = -1; x.bstr = 0;
    x.st0 = x.st1 = true;
    x.vin = x.vout = 0;
    x.ex = nullptr;
    x.si = g ? I1 : I0;
    const float2* tw = p.tw;
    pdl_wait();
    for (int b = blockIdx.y * q.per; b < b1; b++) {
        const ElecParams& e = q.ep[b];
        const double y = sample_y(q, j);
        const int iy0 = sample_row(q, e, j);
        if (iy0 < 0 || iy0 >= e.onz - 1) continue;
        const LineRun d = reinterpret_cast<const LineDesc*>(reinterpret_cast<const char*>(p.gd) + b * p.bDesc)->run;
        const int row = iy0 + g, line = d.mirror_lines ? nl - 1 - row : row;
        x.line0 = x.line1 = line;
        x.g0 = p.src[0] + b * p.bSrc;
        x.g1 = p.src[1] + b * p.bSrc;
        x.gstr = d.blk_in > 0 ? d.blk_in : 1;
        x.ioff = d.blk_in > 0 ? (unsigned)((line / d.blk_in * d.in_p - d.in_q0) * d.blk_in + line % d.blk_in)
                              : (unsigned)((line - d.in_l0) * d.in_p - d.in_q0);
        x.za0 = 0;
        x.zn = N - 1;
        x.in0 = true;
        x.full = d.blk_in == 0;
        if (d.zwin) {
            x.full = false;
            x.in0 = line >= d.zl0 && line <= d.zl1 && d.za0 <= d.za1;
            x.za0 = d.za0;
            x.zn = (unsigned)max(d.za1 - d.za0, 0);
        }
        x.in1 = x.in0;
        x.tabs = p.tabs + b * p.bTab;
        PChain pre, mid, fin;
        pre.rot_in = d.pre_rot; pre.mir = 0; pre.rot_out = 0; pre.tab = d.pre_tab; pre.extra = 0;
        mid.rot_in = d.mid_in; mid.mir = d.mid_mir; mid.rot_out = d.mid_out; mid.tab = d.mid_tab; mid.extra = 0;
        fin.rot_in = 0; fin.mir = 0; fin.rot_out = d.fin_rot; fin.tab = d.fin_tab; fin.extra = 0;
        const bool one = d.dir1 != 0;
        x.has_lf = d.lt[0] >= 0;
        float iscale = 1.f;
        if (d.int_flat) {
            if (one) mid.tab = -1;
            else fin.tab = -1;
            x.has_lf = false;
            iscale = d.int_scale;
        }
        x.lfr = make_float2(1.f, 1.f);
        x.lfi = make_float2(0.f, 0.f);
        if (x.has_lf) {
            float2 a = make_float2(1.f, 0.f);
#pragma unroll
            for (int k = 0; k < 3; k++)
                if (d.lt[k] >= 0) a = cmul(a, __ldg(&x.tabs[d.lt[k] + line]));
            x.lfr = make_float2(a.x, a.x);
            x.lfi = make_float2(a.y, a.y);
        }
        const PChain cin = one ? pre : mid, cout = one ? mid : fin;
        const float cj = (one ? d.dir1 : d.dir2) < 0 ? -1.f : 1.f;
        if constexpr (Z::fixed) {
            constexpr int n = Z::n(), RA = Z::R(0), RB = Z::R(1), RC = Z::R(2), RL = Z::R(Z::n() - 1);
            run_first<RA, Z, false, 0, false>(z, s, x, cin, cj, tw, t);
            if constexpr (n >= 3) { __syncthreads(); run_mid<RB, Z, true>(z, 1, s, tw, t); }
            if constexpr (n >= 4) { __syncthreads(); run_mid<RC, Z, true>(z, 2, s, tw, t); }
            __syncthreads();
            run_last<RL, Z, false, 0, 2>(z, s, x, cout, cj, iscale, t);
        } else {
#define LINEP_SFIRST(R_) case R_: run_first<R_, Z, false, 0, false>(z, s, x, cin, cj, tw, t); break;
            switch (z.R(0)) { LINEP_EVEN(LINEP_SFIRST) default: break; }
            for (int st = 1; st + 1 < z.n(); st++) {
                __syncthreads();
#define LINEP_SMID(R_) case R_: run_mid<R_, Z, true>(z, st, s, tw, t); break;
                switch (z.R(st)) { LINEP_ALL(LINEP_SMID) default: break; }
            }
            __syncthreads();
#define LINEP_SLAST(R_) case R_: run_last<R_, Z, false, 0, 2>(z, s, x, cout, cj, iscale, t); break;
            switch (z.R(z.n() - 1)) { LINEP_ALL(LINEP_SLAST) default: break; }
        }
        __syncthreads();
        // (the next electron's first barrier comes before its intensities)
        const double ty = (y - (e.ozStart + e.ozStep * iy0)) * e.ozInv;
        for (int i = tid; i < q.anx; i += blockDim.x) {
            const double xx = q.axStart + (double)i * q.axStep;
            const int ix0 = (int)trunc((xx - e.oxStart) * e.oxInv + 1.e-09);
            if (ix0 < 0 || ix0 >= e.onx - 1) continue;
            const double tx = (xx - (e.oxStart + e.oxStep * ix0)) * e.oxInv;
            const double a00 = I0[ix0], f10 = I0[ix0 + 1], f01 = I1[ix0], f11 = I1[ix0 + 1];
            const double a10 = f10 - a00, a01 = f01 - a00, a11 = a00 - f01 - f10 + f11;
            acc[i] += a00 + tx * (a10 + ty * a11) + ty * a01;
        }
    }
    double* part = q.part + ((size_t)blockIdx.y * q.anz + j) * q.anx;
    for (int i = tid; i < q.anx; i += blockDim.x) part[i] = acc[i];
}

}  // namespace srwg
