// Stage schedules and places of the line passes on pairs (linep.cuh): the host's schedule of a length
// and the index arithmetic the kernels share with it.
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>
#include "kdesc.h"
#include "linep_lengths.h"

#ifdef __CUDACC__
#define SRWG_HD __host__ __device__ __forceinline__
#else
#define SRWG_HD inline
#endif

namespace srwg {

// quotient by a launch constant d: mul = floor(2^32 / d) + 1 (exact for u d < 2^32), 0 for d = 1
SRWG_HD int qdiv(int u, unsigned mul)
{
#ifdef __CUDA_ARCH__
    return mul ? (int)__umulhi((unsigned)u, mul) : u;
#else
    return mul ? (int)(((unsigned long long)(unsigned)u * mul) >> 32) : u;
#endif
}

// a length's schedule as the kernels see it: run-time (PShape) or fixed at compile time (FShape)
struct PShape {
    int N_, n_, T_, pitch_;           // points, stages, threads per pair, pitch of the k1 blocks
    const int* R_;                    // radices
    const int* L_;                    // L[s] = N / (R[0] .. R[s - 1])
    const unsigned* dL;               // reciprocals of L[s], of R[s], of R[1] .. R[s - 1]
    const unsigned* dR;
    const unsigned* dB;
    const int* t1;                    // offsets of the stages' twiddle tables (first, second transform)
    const int* t2;
    static constexpr bool fixed = false;
    static constexpr int bound = 512; // (see FShape)
    SRWG_HD int tw1(int s) const { return t1[s]; }
    SRWG_HD int tw2(int s) const { return t2[s]; }
    SRWG_HD int N() const { return N_; }
    SRWG_HD int n() const { return n_; }
    SRWG_HD int T() const { return T_; }
    SRWG_HD int pitch() const { return pitch_; }
    SRWG_HD int R(int s) const { return R_[s]; }
    SRWG_HD int L(int s) const { return L_[s]; }
    SRWG_HD int divR(int u, int s) const { return qdiv(u, dR[s]); }
    SRWG_HD int divL(int u, int s) const { return qdiv(u, dL[s]); }
    SRWG_HD int divB(int u, int s) const { return qdiv(u, dB[s]); }
};

// rows of a stage's twiddle table: every power below the radix up to radix 8; 1, 2, 4, 8 above it (the others are
// products), and 12 for radix 16
SRWG_HD constexpr int tw_rows(int R) { return R == 16 ? 5 : R > 8 ? 4 : R - 1; }
SRWG_HD constexpr int tw_power(int R, int row) { return R <= 8 ? row + 1 : row < 4 ? 1 << row : 12; }

template <int R0, int R1, int R2, int R3, int TT> struct FShape {
    static constexpr bool fixed = true;
    // the twiddle tables one after the other: first transform's stages 0 .. n - 2 (L[s + 1] entries per
    // row), second transform's n - 1 .. 1 (R[0] .. R[s - 1] entries)
    SRWG_HD static constexpr int tw1(int s)
    {
        int o = 0;
        for (int i = 0; i < s; i++) o += tw_rows(R(i)) * L(i + 1);
        return o;
    }
    SRWG_HD static constexpr int tw2(int s)
    {
        int o = tw1(n() - 1);
        for (int i = n() - 1; i > s; i--) o += tw_rows(R(i)) * (N() / L(i));
        return o;
    }
    SRWG_HD static constexpr int n() { return R2 == 1 ? 2 : R3 == 1 ? 3 : 4; }
    SRWG_HD static constexpr int N() { return R0 * R1 * R2 * R3; }
    SRWG_HD static constexpr int T() { return TT; }
    SRWG_HD static constexpr int R(int s) { return s == 0 ? R0 : s == 1 ? R1 : s == 2 ? R2 : R3; }
    SRWG_HD static constexpr int L(int s)
    {
        return s == 0 ? R0 * R1 * R2 * R3 : s == 1 ? R1 * R2 * R3 : s == 2 ? R2 * R3 : s == 3 ? R3 : 1;
    }
    SRWG_HD static constexpr int pitch() { return L(1) | 1; }
    // threads the kernels' registers are bounded for: 640 (96 registers) where that puts more CTAs on an SM,
    // 512 (128 registers) where it only spills.  Warps per SM are 21 instead of 16: CTAs of a power of two
    // threads gain nothing (two of 256 either way), others do (2240 x 1536, drifts: 239 to 216 us; quadratic
    // drifts at 4096^2 would go from 935 to 1000), and so do short radix-8 lines (512: 32.7 to 30.8; 16 x 8 x 8
    // at 1024 would go from 65 to 69, 8 x 8 x 4 at 256 on 32 threads from 43 to 47 for a batch of 8).
    static constexpr bool pow2T = (TT & (TT - 1)) == 0;
    static constexpr int maxR = R0 > R1 ? (R0 > R2 ? R0 : R2) : (R1 > R2 ? R1 : R2);
    static constexpr int bound = TT < 64 ? 512 : !pow2T || maxR <= 8 ? 640 : 512;
    SRWG_HD static constexpr int divR(int u, int s) { return (int)((unsigned)u / (unsigned)R(s)); }
    SRWG_HD static constexpr int divL(int u, int s) { return (int)((unsigned)u / (unsigned)L(s)); }
    SRWG_HD static constexpr int divB(int u, int s)
    {
        return (int)((unsigned)u / (unsigned)(s <= 1 ? 1 : s == 2 ? R1 : R1 * R2));
    }
};

// place of the last stage's butterfly u = k1 + R1 k2 + ...
template <class Z> SRWG_HD int place_last(const Z& z, int u)
{
    int k = z.divR(u, 0);
    int base = (u - k * z.R(0)) * z.pitch();
    u = k;
    for (int s = 1; s + 1 < z.n(); s++) {
        k = z.divR(u, s);
        base += (u - k * z.R(s)) * z.L(s + 1);
        u = k;
    }
    return base;
}

// butterfly b of stage s (from 0; neither the first nor the last): block w of L[s] places, offset
// o < L[s + 1] in it
template <class Z> SRWG_HD int place_mid(const Z& z, int s, int b, int& w, int& o)
{
    w = z.divL(b, s + 1);
    o = b - w * z.L(s + 1);
    const int k1 = z.divB(w, s);
    return w * z.L(s) + k1 * (z.pitch() - z.L(1)) + o;
}

// place of the back transform's last butterfly b = q_n + R_n q_(n-1) + ... (over k1)
template <class Z> SRWG_HD int place_back(const Z& z, int b)
{
    int place = 0;
    for (int i = z.n() - 1; i >= 2; i--) {
        const int q = z.divR(b, i);
        place += (b - q * z.R(i)) * z.L(i + 1);
        b = q;
    }
    return place + b * z.L(2);
}

// natural index k1 + R1 k2 + ... of the digits below stage s, from the block number w = k1 (R2 .. R_s)
// + ... + k_s
template <class Z> SRWG_HD int low_index(const Z& z, int s, int w)
{
    if (s == 1) return w;
    int idx = 0, weight = 1;
    for (int i = 0; i + 1 < s; i++) weight *= z.R(i);
    for (int i = s - 1; i >= 1; i--) {
        const int q = z.divR(w, i);
        idx += (w - q * z.R(i)) * weight;
        w = q;
        weight = i >= 2 ? z.divR(weight, i - 1) : 1;
    }
    return idx + w;
}

// ------------------------------------------------------------------------------------------------
// host: the schedule of a length
// ------------------------------------------------------------------------------------------------
struct PairShape {
    int n = 0, T = 0, pitch = 0, slot = 0;      // stages, threads per pair, k1 block pitch, float4 per pair
    int tw1[SRWG_MAX_STAGES], tw2[SRWG_MAX_STAGES], twLen = 0;   // twiddle tables: offsets, float2 in all
    int R[SRWG_MAX_STAGES], len[SRWG_MAX_STAGES + 1];
    unsigned dL[SRWG_MAX_STAGES + 1], dR[SRWG_MAX_STAGES], dB[SRWG_MAX_STAGES];
};

// real operations per point of a radix-R butterfly (linep.cuh)
inline double radix_cost(int R)
{
    switch (R) {
    case 2: return 2.;
    case 3: return 5.3;
    case 4: return 4.;
    case 5: return 8.;
    case 6: return 7.3;
    case 8: return 6.8;
    case 9: return 12.;
    case 10: return 10.;
    case 12: return 9.3;
    case 14: return 16.;
    case 15: return 13.3;
    case 16: return 10.5;
    default: return 2. * (R - 1);               // 7, 11, 13
    }
}
const double STAGE_COST = 14.;           // twiddles and the exchange, per point

// The schedule of least cost: radices, and threads per pair.  A stage takes its rounds (butterflies per
// thread) times a butterfly's instructions, and a constant for the barrier and its loads; a pair's threads
// weigh by T^alpha.  Long lines fill the chip and the work counts (alpha = 1: no idle threads); short ones
// are a chain of single warps that run every instruction once (at 216 x 200 ncu shows 8 of 13 cycles per
// instruction waiting for code), so butterflies are small and threads many.  Propagations between drifts,
// the work alone (radices 16 first, about 16 points per thread) and this rule: 100 x 90 55 and 45 us,
// 216 x 200 57 and 45, 360 x 350 96 and 55, 500 x 504 64 and 59, 1000 x 1080 120 and 111, 1400 x 1470 222
// and 206; 720 x 700 84 and 88; above 1600 points the work alone: 2000 x 1980 380, with alpha 0.7 403.
inline void best_schedule(int N, int most, std::vector<int>& cur, std::vector<int>& best, int& bestT, double& bestCost)
{
    int m = N;
    for (int R : cur) m /= R;
    if (m == 1) {
        if (cur.size() < 2) return;
        // the first radix is even and, where there is one, at least 8 (neighbouring k1 then fill the banks)
        size_t f = 0;
        while (f < cur.size() && (cur[f] & 1)) f++;
        if (f == cur.size()) return;
        const double al = N <= 400 ? 0.3 : N <= 1600 ? 0.7 : 1., sy = N <= 400 ? 60. : 20.;
        for (int T = std::max(1, N / 32); T <= std::min(512, std::max(1, N / 2)); T++) {
            double w = 0.;
            for (int R : cur) w += (double)((N / R + T - 1) / T) * (radix_cost(R) + STAGE_COST) * R + sy;
            const double q = w * std::pow((double)T, al);
            if (q < bestCost) {
                bestCost = q;
                bestT = T;
                best = cur;
                std::rotate(best.begin(), best.begin() + f, best.begin() + f + 1);
            }
        }
        return;
    }
    for (int R = std::min(most, 16); R >= 2; R--) {
        if (m % R || (int)cur.size() + 1 > SRWG_MAX_STAGES) continue;
        cur.push_back(R);
        best_schedule(N, R, cur, best, bestT, bestCost);
        cur.pop_back();
    }
}

inline unsigned recip(int d) { return d <= 1 ? 0u : (unsigned)(0x100000000ull / (unsigned)d) + 1u; }

inline bool make_pair_shape(int N, PairShape& z)
{
    if (N < 4 || N > 8192 || (N & 1)) return false;
    int m = N;
    for (int p : {2, 3, 5, 7, 11, 13})
        while (m % p == 0) m /= p;
    if (m != 1) return false;
    std::vector<int> cur, r;
    z.T = 0;
#define SRWG_LINEF_SHAPE(M, A, B, C, D, TT)                             \
    if (N == M) {                                                       \
        r = {A, B};                                                     \
        if (C > 1) r.push_back(C);                                      \
        if (D > 1) r.push_back(D);                                      \
        z.T = TT;                                                       \
    }
    SRWG_LINEF_LENGTHS(SRWG_LINEF_SHAPE)
#undef SRWG_LINEF_SHAPE
    if (r.empty()) {
        double c = 1e300;
        best_schedule(N, 16, cur, r, z.T, c);
        if (r.empty()) return false;
    }
    z.n = (int)r.size();
    z.len[0] = N;
    for (int s = 0; s < z.n; s++) {
        z.R[s] = r[s];
        z.len[s + 1] = z.len[s] / r[s];
        z.dR[s] = recip(r[s]);
    }
    for (int s = 0; s <= z.n; s++) z.dL[s] = recip(z.len[s]);
    int blk = 1;                                 // R2 .. R_s: blocks of a stage per block of k1
    for (int s = 0; s < z.n; s++) {
        z.dB[s] = recip(blk);
        if (s + 1 < z.n && s >= 1) blk *= z.R[s];
    }
    z.pitch = z.len[1] | 1;
    z.slot = z.R[0] * z.pitch;
    int o = 0;
    for (int s = 0; s + 1 < z.n; s++) { z.tw1[s] = o; o += tw_rows(z.R[s]) * z.len[s + 1]; }
    for (int s = z.n - 1; s >= 1; s--) { z.tw2[s] = o; o += tw_rows(z.R[s]) * (N / z.len[s]); }
    z.tw1[z.n - 1] = z.tw2[0] = o;              // (not used)
    z.twLen = o;
    return true;
}

// the twiddle tables of a schedule: for stage s of the first transform W_(L[s])^(o e), o < L[s + 1], for digit s
// of the second one W_(R[0] .. R[s])^(u e), u < R[0] .. R[s - 1]; a row per power e (tw_power).  (FP64, rounded)
template <class F2> inline void fill_twiddles(const PairShape& z, std::vector<F2>& h)
{
    h.resize(z.twLen);
    auto put = [&](int off, int R, int n, int period) {
        for (int e = 0; e < tw_rows(R); e++)
            for (int k = 0; k < n; k++) {
                const double a = -2. * M_PI * (double)((long long)k * tw_power(R, e) % period) / (double)period;
                F2& v = h[off + e * n + k];
                v.x = (float)cos(a);
                v.y = (float)sin(a);
            }
    };
    const int N = z.len[0];
    for (int s = 0; s + 1 < z.n; s++) put(z.tw1[s], z.R[s], z.len[s + 1], z.len[s]);
    for (int s = z.n - 1; s >= 1; s--) put(z.tw2[s], z.R[s], N / z.len[s], N / z.len[s + 1]);
}

}  // namespace srwg
