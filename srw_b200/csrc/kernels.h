// Launch parameters of the sm_100a kernels (kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <vector>
#include "kdesc.h"
#include "linen_lengths.h"
#include "linep_lengths.h"

namespace srwg {

// dynamic shared memory of a line pass (leaves room for the static descriptor copy)
#define SRWG_LINE_SMEM_MAX (220 * 1024)

// shared-memory pitch of a line of N points in the pass of 16384 (line2.cuh): one pad point per 16 (conflict-free
// Stockham exchanges), a multiple of 16 bytes; with L lines as the tuning entry points' bound on entries (a
// column tile's lines 32 / L banks apart)
inline size_t line_pitch(int N, int L = 1, bool cols = false)
{
    const size_t P = (size_t)N + N / 16;
    const size_t r = (cols && L >= 2) ? (L >= 16 ? 1 : 16 / L) : 4;
    return P + ((r + 16 - P % 16) % 16);
}

// what a line pass kernel takes (its descriptor stays in device memory)
struct LineArgs {
    const float2* src[2];
    float2* dst[2];
    const float2* tw;        // the length's twiddle tables (line_twiddles)
    int N, nlines;           // line length, number of lines
    int T, L, P, G;          // threads per line (pair), lines per CTA, shared memory of one (float2; pairs:
                             //   float4), lines (pairs) per CTA
    int nst;                 // stages, their radices and (pairs, linep.cuh) lengths and reciprocals
    int radix[SRWG_MAX_STAGES];
    int len[SRWG_MAX_STAGES + 1];
    unsigned dL[SRWG_MAX_STAGES + 1], dR[SRWG_MAX_STAGES], dB[SRWG_MAX_STAGES];
    int tw1[SRWG_MAX_STAGES], tw2[SRWG_MAX_STAGES];
    int pitch;               // pairs: pitch of the first digit's blocks
    int alignIn, alignOut;   // pairs: 16-byte aligned fields (two lines at once)
    int v2;                  // 0: pairs of lines (linep_kernel), 1: one line (line2_kernel, 16384 points)
    const float2* tabs;      // the plan's separable point-wise tables
    const LineDesc* gd;      // this pass's descriptor in device memory
    int byValue;             // pairs: one descriptor for the whole launch, in `run` (else gd's)
    LineRun run;
    int nb;                  // wavefronts in the launch (grid z; 0 or 1: one)
    long long bDesc, bTab;   // per wavefront: descriptor stride (bytes), table stride (float2)
    long long bSrc, bDst;    // per wavefront: source / destination field stride (float2)
    int bulk;                // points of staging per component behind the slots (0: no bulk copies)
    int* status;             // device counter of waits that gave up (NULL: not recorded)
    long long spin;          // iteration limit of the bulk-copy wait
    const unsigned* mask;    // columns before a sampled pass: a bit per output row that it reads (NULL: all are)
    int maskWords;           // words of it per wavefront
    int nblk;                // line blocks launched, from the window's first one (0: all)
};
struct LineLaunch : LineArgs {
    LineDesc d;              // host copy (launch shapes)
};

// per-electron parameters of a multi-electron batch in device memory
struct ElecParams {
    double kx, kz;                       // kick: phase kx x + kz z on the base mesh (fused by the planner)
    double dx, dz;                       // mesh shift of the electron's wavefront
    double oxStart, oxStep, ozStart, ozStep;   // output mesh (steps as (Fin - Start)/(n - 1))
    double oxInv, ozInv;                       // 1 / step: the accumulation multiplies (no FP64 divisions)
    int onx, onz;
    int pad[2];
};

// the sampled last pass of a multi-electron batch (linep_sample_kernel): detector mesh, electrons per
// CTA, and the groups' sums [groups][anz][anx]
struct SampleArgs {
    const ElecParams* ep;
    double* part;
    int nb, per, anx, anz;
    double axStart, axStep, azStart, azStep;
};
#ifdef __CUDACC__
// detector row j and the output row below it on an electron's mesh (its operations written out: the pass
// and the mask of the rows it reads agree)
__device__ __forceinline__ double sample_y(const SampleArgs& q, int j) { return __fma_rn((double)j, q.azStep, q.azStart); }
__device__ __forceinline__ int sample_row(const SampleArgs& q, const ElecParams& e, int j)
{
    return (int)trunc(__fma_rn(__dadd_rn(sample_y(q, j), -e.ozStart), e.ozInv, 1.e-09));
}
#endif

// tiled resize: a CTA makes TZ x TX new points from an old tile of at most OR_MAX x OC_MAX points
#define SRWG_RESIZE_TX 64
#define SRWG_RESIZE_TZ 16
#define SRWG_RESIZE_OR_MAX 40
#define SRWG_RESIZE_OC_MAX 80

struct ResizeLaunch {
    ResizeDesc d;
    const float2* src[2];
    float2* dst[2];
    const float2* tabs;
    const ResizeDesc* gd;
    int vec_ok;              // even row lengths and 16-byte aligned buffers: float4 paths allowed
    double xStepInvO, zStepInvO;
    int nb;                  // wavefronts in the launch (grid z; 0 or 1: one)
    long long bDesc, bTab;   // per wavefront: descriptor stride (bytes), table stride (float2)
    long long bSrc, bDst;    // per wavefront: source / destination field stride (float2)
    int ntx, ntz;            // tiled kernel: tiles launched per axis, from the window's first ones (0: all)
};

struct PwLaunch {
    PwDesc d;
    const float2* src[2];
    float2* dst[2];
    const float2* tabs;
    const PwDesc* gd;
    int nb;                  // wavefronts in the launch (grid z; 0 or 1: one)
    long long bDesc, bTab;   // per wavefront: descriptor stride (bytes), table stride (float2)
    long long bSrc, bDst;    // per wavefront: source / destination field stride (float2)
};

// MOM pass (moments.cu): reduction of one field into the 22 sums of ComputeRadMoments.  For nb
// wavefronts the passes run one wavefront after the other (scratch reused in stream order).
struct MomLaunch {
    MomDesc d;                 // host copy (launch shapes); the kernels read gd
    const float2* src[2];
    const float2* tabs;
    const MomDesc* gd;
    double* scratch;           // mom_scratch_doubles(nx, nz) doubles
    double* out;               // result slot of wavefront 0 (SRWG_MOM_SLOT doubles)
    int nb;
    long long bDesc, bTab;     // per wavefront: descriptor stride (bytes), table stride (float2)
    long long bSrc, bOut;      // per wavefront: field stride (float2), result stride (doubles)
};
size_t mom_scratch_doubles(int nx, int nz);
cudaError_t launch_moments(const MomLaunch& p, cudaStream_t st);

// intensity extraction from a field with the operators still pending on it (d: host copy, gd: the
// device copy the kernel reads); writes nx * nz values (float, or double for the phase) to out
cudaError_t launch_extract(const MomDesc& d, const MomDesc* gd, const float2* s0, const float2* s1,
                           const float2* tabs, char* out, cudaStream_t st);

// pdl: the kernel may start while the one before it in the stream (a line pass or resize of the same run)
// ends; it waits for it before it touches a field
cudaError_t launch_line(const LineLaunch& p, cudaStream_t st, bool pdl = false);
// the sampled row pass of a batch; its shape (threads, shared memory) must fit: sample_fits
// the rows a sampled pass of descriptors p.gd reads, a bit each: words per electron, into mask
cudaError_t launch_row_mask(const LineLaunch& p, const SampleArgs& q, unsigned* mask, int words, cudaStream_t st);
cudaError_t launch_line_sample(const LineLaunch& p, const SampleArgs& q, cudaStream_t st, bool pdl);
bool sample_fits(const LineLaunch& p, int anx);
void fill_line_run(LineDesc& d);      // d.run from the rest of d (planner.cpp)

// line pass kernels: pairs of lines (linep.cu, one unit per axis and mode), 16384 points (line2_14.cu)
typedef void (*LineFn)(const LineArgs);
typedef void (*SampleFn)(const LineArgs, const SampleArgs);
SampleFn lines_get();
#define SRWG_LINEP_DECL(C, M) LineFn linep_get_##C##_##M(int extra);
SRWG_LINEP_DECL(0, 0) SRWG_LINEP_DECL(0, 1) SRWG_LINEP_DECL(0, 2)
SRWG_LINEP_DECL(1, 0) SRWG_LINEP_DECL(1, 1) SRWG_LINEP_DECL(1, 2)
#undef SRWG_LINEP_DECL
#define SRWG_LINEF_DECL(N, A, B, C, D, T) LineFn linef_get_##N(bool cols, int mode, int extra); SampleFn lines_get_##N();
SRWG_LINEF_LENGTHS(SRWG_LINEF_DECL)
#undef SRWG_LINEF_DECL
LineFn line2_get_14(bool cols, int f1, int f2);
LineFn line2e_get_14(bool cols, int f1, int f2);
inline bool line2_supported(int N) { return N >= 64 && N <= 16384 && (N & (N - 1)) == 0; }
// general lengths with launch shapes of their own in the tuning table
inline bool linen_supported(int N)
{
#define SRWG_LINEN_IS(M) if (N == M) return true;
    SRWG_LINEN_LENGTHS(SRWG_LINEN_IS)
#undef SRWG_LINEN_IS
    return false;
}
inline bool linen_pow2(int N)
{
#define SRWG_LINEN_IS(M) if (N == M) return true;
    SRWG_LINEN_POW2(SRWG_LINEN_IS)
#undef SRWG_LINEN_IS
    return false;
}
// lengths of the passes on pairs of lines: every even 2^a 3^b 5^c 7^d 11^e 13^f from 4 to
// 8192 (they take zero windows and column blocks, and write intensities)
bool pair_supported(int N);
// the twiddle tables of a line pass of N points, as its kernel reads them
void line_twiddles(int N, std::vector<float2>& h);
// columns that a column pass of N points transforms per CTA on a grid of nl columns: the width of
// the column blocks the row pass before it writes (0: the pass is not one on pairs, or nl has no such blocks)
int pair_block(int N, int nl);
// classes of tuned lengths (the tuning entry points' families)
enum { FAM_POW2 = 1, FAM_SPEC = 3 };
// whether the tuning entry points take L lines per CTA for length N of class fam
inline bool fixed_lines_valid(int axis, int N, int L, int fam)
{
    if (L < 1 || (size_t)L * line_pitch(N, L, axis == 1) * 8 > SRWG_LINE_SMEM_MAX) return false;
    if (axis == 1 && (L > 32 || (L & (L - 1)) != 0)) return false;      // column blocks: a power of two
    if (fam == FAM_POW2 && line2_supported(N)) return (N / 16) * L <= 1024;
    if (fam == FAM_SPEC && (linen_supported(N) || linen_pow2(N))) return ((N + 15) / 16) * L <= 512;
    return false;
}
// class of a tuned length, and the lines per CTA its passes are launched with (whole pairs; fewer where a launch has
// few lines, as many as its blocks where it reads blocks of lines; 0 for other lengths)
int fixed_family(int axis, int N);
int fixed_lines_per_cta(int axis, int N);
cudaError_t launch_resize(const ResizeLaunch& p, cudaStream_t st);
cudaError_t launch_pw(const PwLaunch& p, cudaStream_t st);

}  // namespace srwg
