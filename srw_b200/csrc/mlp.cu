// Kernels of the learned resize-factor predictor: a small FP32 MLP (GEMM, bias + GELU, their
// gradients, mean-squared-error loss, Adam) and the wavefront features it reads (intensity
// downsampled to 64 x 64, fitted phase-curvature radii).  The network is small (a few 10^6
// multiply-adds per wavefront), so these are plain SIMT kernels with shared-memory tiling; the
// training loop and the memory they run on are driven from the host (srw_b200/learned.py).
// Nothing here has a counterpart in the reference: it chooses the resize factors that the
// reference's users set by hand in the propagation parameters (pp[5..8]).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <string>

#include "../../include/srwl_b200.h"
#include "errors.h"
#include "exec.h"

namespace cg = cooperative_groups;

namespace srwg {

__device__ __forceinline__ float gelu(float z)
{   // tanh form of GELU (Hendrycks & Gimpel 2016)
    const float c = 0.7978845608028654f;
    return 0.5f * z * (1.f + tanhf(c * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float gelu_grad(float z)
{
    const float c = 0.7978845608028654f;
    const float u = c * (z + 0.044715f * z * z * z);
    const float t = tanhf(u);
    return 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * c * (1.f + 3.f * 0.044715f * z * z);
}

// What follows a product in its kernel: Z = alpha op(A) op(B) + beta C + bias (row broadcast) to C; with
// act, Y = GELU(Z) beside it (act 0: Y = Z); with zgrad, Z *= GELU'(zgrad) (same layout as C); with
// bsum, the column sums of op(B) (the bias gradients that go with a weight gradient)
struct GemmTail {
    const float* bias;
    float* Y;
    int act;
    const float* zgrad;
    float* bsum;
};

// op(A) is M x K (A row-major, lda; transposed when TA), op(B) is K x N.  A CTA makes a GM x 64 tile over one of
// gridDim.z pieces of K (steps of 32, the next step's operands loaded while this one is multiplied); the pieces
// are the CTAs of a cluster, which then add their tiles through distributed shared memory in piece order (no
// workspace, no atomics: the sum does not depend on scheduling); one piece writes its tile from registers.
// The network's products are small and long: 128 x 256 with K = 4109 is 8 tiles of 64 x 64, whose 257
// serial steps took 385 us; 16 tiles of 32 x 64 in 8 pieces occupy 128 SMs with 17 steps each (37 us).  Large
// ones take tiles of 64 rows: 2048^3 506 us, with 32 rows 780, 655 before the pieces; 4096^2 with K = 16 28 us,
// with full steps and scalar stores 56, before the pieces 32.
#define GN 64
#define GK 32
template <int GM, bool TA, bool TB>
__global__ void __launch_bounds__(256) gemm_kernel(int M, int N, int K, int kc, const float* __restrict__ A, int lda,
                                                   const float* __restrict__ B, int ldb, float* __restrict__ C, int ldc,
                                                   float alpha, float beta, const GemmTail t)
{
    __shared__ float As[2][GK][GM + 1];
    __shared__ __align__(16) float Bs[2][GK][GN + 4];
    __shared__ float cs[GN];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.x * GM, n0 = blockIdx.y * GN;
    const int ka = blockIdx.z * kc, kb = min(K, ka + kc), nt = ka < kb ? (kb - ka + GK - 1) / GK : 0;
    const bool sums = t.bsum != nullptr && blockIdx.x == 0;
    constexpr int GR = GM / 16;                  // rows of a thread
    float acc[GR][4] = {{0.f}}, bs = 0.f;
    float ra[GM / 8], rb[8];
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < GM / 8; i++) {
            const int e = tid + 256 * i;
            const int kk = TA ? e / GM : e % GK, mm = TA ? e % GM : e / GK;
            const int gm = m0 + mm, gk = k0 + kk;
            ra[i] = (gm < M && gk < kb) ? __ldg(&A[TA ? (size_t)gk * lda + gm : (size_t)gm * lda + gk]) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int e = tid + 256 * i;
            const int kk = TB ? e % GK : e / GN, nn = TB ? e / GK : e % GN;
            const int gn = n0 + nn, gk = k0 + kk;
            rb[i] = (gn < N && gk < kb) ? __ldg(&B[TB ? (size_t)gn * ldb + gk : (size_t)gk * ldb + gn]) : 0.f;
        }
    };
    auto put = [&](int u) {
#pragma unroll
        for (int i = 0; i < GM / 8; i++) {
            const int e = tid + 256 * i;
            As[u][TA ? e / GM : e % GK][TA ? e % GM : e / GK] = ra[i];
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int e = tid + 256 * i;
            Bs[u][TB ? e % GK : e / GN][TB ? e / GK : e % GN] = rb[i];
        }
    };
    if (nt > 0) {
        load(ka);
        put(0);
    }
    __syncthreads();
    for (int s = 0; s < nt; s++) {
        const int u = s & 1;
        if (s + 1 < nt) load(ka + (s + 1) * GK);
        const int ke = kb - ka - s * GK;                 // (the last step: eight at a time)
#pragma unroll
        for (int k8 = 0; k8 < GK; k8 += 8) {
            if (k8 >= ke) break;
#pragma unroll
            for (int kk = k8; kk < k8 + 8; kk++) {
                const float4 b = *reinterpret_cast<const float4*>(&Bs[u][kk][tx * 4]);
#pragma unroll
                for (int i = 0; i < GR; i++) {
                    const float a = As[u][kk][ty * GR + i];
                    acc[i][0] = fmaf(a, b.x, acc[i][0]); acc[i][1] = fmaf(a, b.y, acc[i][1]);
                    acc[i][2] = fmaf(a, b.z, acc[i][2]); acc[i][3] = fmaf(a, b.w, acc[i][3]);
                }
            }
        }
        if (sums && tid < GN)
            for (int kk = 0; kk < GK; kk++) bs += Bs[u][kk][tid];
        if (s + 1 < nt) put(u ^ 1);
        __syncthreads();
    }
    auto out = [&](int gm, int gn, float v) {
        if (gm >= M || gn >= N) return;
        const size_t o = (size_t)gm * ldc + gn;
        float z = alpha * v + (beta != 0.f ? beta * C[o] : 0.f);
        if (t.bias) z += __ldg(&t.bias[gn]);
        if (t.zgrad) z *= gelu_grad(__ldg(&t.zgrad[o]));
        C[o] = z;
        if (t.Y) t.Y[o] = t.act ? gelu(z) : z;
    };
    if (gridDim.z == 1) {                        // one piece: no tiles to add
        const bool four = !t.bias && !t.zgrad && !t.Y && n0 + tx * 4 + 4 <= N && ldc % 4 == 0 && (reinterpret_cast<size_t>(C) & 15) == 0;
#pragma unroll
        for (int i = 0; i < GR; i++) {
            const int gm = m0 + ty * GR + i;
            if (four && beta == 0.f) {
                if (gm < M)
                    *reinterpret_cast<float4*>(&C[(size_t)gm * ldc + n0 + tx * 4]) =
                        make_float4(alpha * acc[i][0], alpha * acc[i][1], alpha * acc[i][2], alpha * acc[i][3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) out(gm, n0 + tx * 4 + j, acc[i][j]);
            }
        }
        if (sums && tid < GN && n0 + tid < N) t.bsum[n0 + tid] = bs;
        return;
    }
    // the piece's tile in shared memory (the operands are done with), then the sum over the cluster
    float* red = &Bs[0][0][0];
#pragma unroll
    for (int i = 0; i < GR; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) red[(ty * GR + i) * GN + tx * 4 + j] = acc[i][j];
    if (sums && tid < GN) cs[tid] = bs;
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    const int S = (int)cl.num_blocks(), r = (int)cl.block_rank();
    for (int e = r * 256 + tid; e < GM * GN; e += S * 256) {
        float v = 0.f;
        for (int q = 0; q < S; q++) v += *cl.map_shared_rank(red + e, q);
        out(m0 + e / GN, n0 + e % GN, v);
    }
    if (sums && r == 0 && tid < GN && n0 + tid < N) {
        float v = 0.f;
        for (int q = 0; q < S; q++) v += *cl.map_shared_rank(cs + tid, q);
        t.bsum[n0 + tid] = v;
    }
    cl.sync();                    // no CTA leaves while another reads its tile
}

// Z[M x N] += bias (row broadcast); Y = act(Z) with act 0 = identity, 1 = GELU
__global__ void bias_act_kernel(float* __restrict__ Z, const float* __restrict__ bias, float* __restrict__ Y, int M,
                                int N, int act)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)M * N) return;
    const float z = Z[i] + bias[i % N];
    Z[i] = z;
    Y[i] = act ? gelu(z) : z;
}

// dY <- dY * act'(Z)
__global__ void act_backward_kernel(const float* __restrict__ Z, float* __restrict__ dY, size_t n, int act)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !act) return;
    dY[i] *= gelu_grad(Z[i]);
}

// db[N] = sum over rows of dZ[M x N]: 32 columns per CTA, 8 partial sums each, added in order
__global__ void __launch_bounds__(256) colsum_kernel(const float* __restrict__ dZ, float* __restrict__ db, int M, int N)
{
    __shared__ float part[8][33];
    const int c = threadIdx.x & 31, g = threadIdx.x >> 5, j = blockIdx.x * 32 + c;
    float s = 0.f;
    if (j < N)
        for (int i = g; i < M; i += 8) s += dZ[(size_t)i * N + j];
    part[g][c] = s;
    __syncthreads();
    if (g == 0 && j < N) {
        for (int k = 1; k < 8; k++) s += part[k][c];
        db[j] = s;
    }
}

// mean squared error over M x N: loss (one value, summed in FP64 per block then atomically) and
// dOut = 2 (out - target) / (M N)
__global__ void mse_kernel(const float* __restrict__ out, const float* __restrict__ target, float* __restrict__ dout,
                           double* __restrict__ loss, int n)
{
    __shared__ double red[256];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.;
    if (i < n) {
        const float d = out[i] - target[i];
        dout[i] = 2.f * d / (float)n;
        l = (double)d * d / n;
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0]);
}

// Adam (Kingma & Ba 2015) with bias correction, step t >= 1
__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, size_t n, float lr, float b1, float b2, float eps, float c1, float c2)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// the same for several parameter arrays in one launch (element i of array k at index off[k] + i)
#define ADAM_MOST 16
struct AdamArrays {
    float* w[ADAM_MOST];
    const float* g[ADAM_MOST];
    float* m[ADAM_MOST];
    float* v[ADAM_MOST];
    long long off[ADAM_MOST + 1];
    int n;
};
__global__ void __launch_bounds__(256) adam_many_kernel(const AdamArrays a, float lr, float b1, float b2, float eps,
                                                        float c1, float c2)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.off[a.n]) return;
    int k = 0;
    while (i >= a.off[k + 1]) k++;
    const long long j = i - a.off[k];
    const float gi = a.g[k][j];
    const float mi = b1 * a.m[k][j] + (1.f - b1) * gi;
    const float vi = b2 * a.v[k][j] + (1.f - b2) * gi * gi;
    a.m[k][j] = mi;
    a.v[k][j] = vi;
    a.w[k][j] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// features of one wavefront: total intensity averaged over 64 x 64 cells of the mesh (cell (cy, cx)
// covers rows [cy ny / 64, (cy + 1) ny / 64) and the same for columns), written to feat[64 * 64]
__global__ void downsample_kernel(const float2* __restrict__ ex, const float2* __restrict__ ey, int nx, int ny,
                                  float* __restrict__ feat)
{
    const int cx = blockIdx.x, cy = blockIdx.y;
    const int x0 = (int)((long long)cx * nx / 64), x1 = (int)((long long)(cx + 1) * nx / 64);
    const int y0 = (int)((long long)cy * ny / 64), y1 = (int)((long long)(cy + 1) * ny / 64);
    __shared__ double red[128];
    double s = 0.;
    const int w = x1 - x0, h = y1 - y0;
    for (int e = threadIdx.x; e < w * h; e += blockDim.x) {
        const int y = y0 + e / w, x = x0 + e % w;
        const float2 u = ex[(size_t)y * nx + x], v = ey[(size_t)y * nx + x];
        s += (double)u.x * u.x + (double)u.y * u.y + (double)v.x * v.x + (double)v.y * v.y;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int k = 64; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) feat[cy * 64 + cx] = (w * h > 0) ? (float)(red[0] / (w * h)) : 0.f;
}

// phase-curvature fit: for neighbouring points along x (and along z) the phase difference
// arg(E(p+1) conj(E(p))) ~ k x dx / R.  The known part 1/R0 (the wavefront's own radius, whose
// quadratic phase the mesh need not resolve) is taken out first, the rest wrapped to [-pi, pi];
// sums for the intensity-weighted least squares 1/R - 1/R0 = sum(w x dphi) / (k dx sum(w x^2))
// (w = |E(p)| |E(p+1)|): sums[0] = sum w x dphi, sums[1] = sum w x^2 (x), sums[2], sums[3] along z
__global__ void curvature_kernel(const float2* __restrict__ ex, int nx, int ny, double xStart, double xStep,
                                 double zStart, double zStep, double k, double invRx0, double invRz0,
                                 double* __restrict__ sums)
{
    const double twoPi = 6.283185307179586;
    __shared__ double red[4][256];
    double a0 = 0., a1 = 0., a2 = 0., a3 = 0.;
    const size_t n = (size_t)nx * ny;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int y = (int)(i / nx), x = (int)(i % nx);
        const float2 e = ex[i];
        if (x + 1 < nx) {
            const float2 f = ex[i + 1];
            const double re = (double)f.x * e.x + (double)f.y * e.y, im = (double)f.y * e.x - (double)f.x * e.y;
            const double w = sqrt(re * re + im * im);
            const double xm = xStart + (x + 0.5) * xStep;
            double d = atan2(im, re) - k * xm * xStep * invRx0;
            d -= twoPi * rint(d / twoPi);
            a0 += w * xm * d;
            a1 += w * xm * xm;
        }
        if (y + 1 < ny) {
            const float2 f = ex[i + nx];
            const double re = (double)f.x * e.x + (double)f.y * e.y, im = (double)f.y * e.x - (double)f.x * e.y;
            const double w = sqrt(re * re + im * im);
            const double zm = zStart + (y + 0.5) * zStep;
            double d = atan2(im, re) - k * zm * zStep * invRz0;
            d -= twoPi * rint(d / twoPi);
            a2 += w * zm * d;
            a3 += w * zm * zm;
        }
    }
    red[0][threadIdx.x] = a0; red[1][threadIdx.x] = a1; red[2][threadIdx.x] = a2; red[3][threadIdx.x] = a3;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (threadIdx.x < k)
            for (int c = 0; c < 4; c++) red[c][threadIdx.x] += red[c][threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 4; c++) atomicAdd(&sums[c], red[c][0]);
}

}  // namespace srwg

using namespace srwg;

static int launch_status(cudaError_t e)
{
    if (e == cudaSuccess) return 0;
    set_last_detail(std::string("kernel launch: ") + cudaGetErrorString(e));
    return SRWG_ERR_CUDA;
}

static int gemm(int M, int N, int K, const float* A, int lda, int transA, const float* B, int ldb, int transB, float* C,
                int ldc, float alpha, float beta, const GemmTail& t, cudaStream_t st)
{
    const int most = 65535 * GN;                 // columns of one launch
    if (N > most) {
        auto at = [](auto* q, int n) { return q ? q + n : q; };
        for (int n = 0; n < N; n += most) {
            const GemmTail u{at(t.bias, n), at(t.Y, n), t.act, at(t.zgrad, n), at(t.bsum, n)};
            const int r = gemm(M, N - n < most ? N - n : most, K, A, lda, transA, transB ? B + (size_t)n * ldb : B + n, ldb,
                               transB, C + n, ldc, alpha, beta, u, st);
            if (r) return r;
        }
        return 0;
    }
    const int tn = (N + GN - 1) / GN;
    // tiles of 64 rows (half the loads of B per multiplication) where they are many enough to fill the chip with
    // pieces of K: 512 x 512, K = 512 (64 tiles) 21 us with 32 rows, 17 with 64; 256 x 256, K = 4109 (16 tiles)
    // 37 and 46; 2000 x 64, K = 64 (32 tiles) 6 and 8.5
    const int gm = (long long)((M + 63) / 64) * tn >= 64 ? 64 : 32;
    const int tm = (M + gm - 1) / gm;
    // pieces of K: as many CTAs as two per SM, at least 64 steps of K each
    int S = 8;
    while (S > 1 && ((long long)tm * tn * S > 2 * 148 || K / S < 64)) S /= 2;
    const int kc = (((K + S - 1) / S + GK - 1) / GK) * GK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tm, tn, S);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = at.val.clusterDim.y = 1;
    at.val.clusterDim.z = S;
    cfg.attrs = &at;
    cfg.numAttrs = S > 1 ? 1 : 0;
    auto run = [&](auto k) { return cudaLaunchKernelEx(&cfg, k, M, N, K, kc, A, lda, B, ldb, C, ldc, alpha, beta, t); };
    const cudaError_t e = gm == 64 ? (transA ? (transB ? run(gemm_kernel<64, true, true>) : run(gemm_kernel<64, true, false>))
                                             : (transB ? run(gemm_kernel<64, false, true>) : run(gemm_kernel<64, false, false>)))
                                   : (transA ? (transB ? run(gemm_kernel<32, true, true>) : run(gemm_kernel<32, true, false>))
                                             : (transB ? run(gemm_kernel<32, false, true>) : run(gemm_kernel<32, false, false>)));
    return launch_status(e);
}

extern "C" SRWG_API int srwgMlpGemm(int M, int N, int K, const float* A, int lda, int transA, const float* B, int ldb,
                                    int transB, float* C, int ldc, float alpha, float beta, void* stream)
{
    if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C) return SRWG_ERR_BAD_ARG;
    return gemm(M, N, K, A, lda, transA, B, ldb, transB, C, ldc, alpha, beta, GemmTail{nullptr, nullptr, 0, nullptr, nullptr},
                (cudaStream_t)stream);
}

extern "C" SRWG_API int srwgMlpLinear(int M, int N, int K, const float* X, const float* W, const float* bias, float* Z,
                                      float* Y, int act, void* stream)
{
    if (M <= 0 || N <= 0 || K <= 0 || !X || !W || !bias || !Z || !Y) return SRWG_ERR_BAD_ARG;
    return gemm(M, N, K, X, K, 0, W, N, 0, Z, N, 1.f, 0.f, GemmTail{bias, Y, act, nullptr, nullptr}, (cudaStream_t)stream);
}

extern "C" SRWG_API int srwgMlpLinearBackward(int M, int N, int K, const float* X, const float* W, const float* dZ,
                                              float* dW, float* db, float* dX, const float* Zprev, void* stream)
{
    if (M <= 0 || N <= 0 || K <= 0 || !X || !dZ || !dW || !db || (dX && !W)) return SRWG_ERR_BAD_ARG;
    int r = gemm(K, N, M, X, K, 1, dZ, N, 0, dW, N, 1.f, 0.f, GemmTail{nullptr, nullptr, 0, nullptr, db}, (cudaStream_t)stream);
    if (r == 0 && dX)
        r = gemm(M, K, N, dZ, N, 0, W, N, 1, dX, K, 1.f, 0.f, GemmTail{nullptr, nullptr, 0, Zprev, nullptr},
                 (cudaStream_t)stream);
    return r;
}

extern "C" SRWG_API int srwgMlpBiasAct(float* Z, const float* bias, float* Y, int M, int N, int act, void* stream)
{
    if (M <= 0 || N <= 0 || !Z || !bias || !Y) return SRWG_ERR_BAD_ARG;
    const size_t n = (size_t)M * N;
    bias_act_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(Z, bias, Y, M, N, act);
    return launch_status(cudaGetLastError());
}

extern "C" SRWG_API int srwgMlpActBackward(const float* Z, float* dY, long long n, int act, void* stream)
{
    if (n <= 0 || !Z || !dY) return SRWG_ERR_BAD_ARG;
    act_backward_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(Z, dY, (size_t)n, act);
    return launch_status(cudaGetLastError());
}

extern "C" SRWG_API int srwgMlpColSum(const float* dZ, float* db, int M, int N, void* stream)
{
    if (M <= 0 || N <= 0 || !dZ || !db) return SRWG_ERR_BAD_ARG;
    colsum_kernel<<<(N + 31) / 32, 256, 0, (cudaStream_t)stream>>>(dZ, db, M, N);
    return launch_status(cudaGetLastError());
}

extern "C" SRWG_API int srwgMlpMse(const float* out, const float* target, float* dout, double* loss, int n, void* stream)
{
    if (n <= 0 || !out || !target || !dout || !loss) return SRWG_ERR_BAD_ARG;
    mse_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(out, target, dout, loss, n);
    return launch_status(cudaGetLastError());
}

extern "C" SRWG_API int srwgMlpAdam(float* w, const float* g, float* m, float* v, long long n, float lr, float b1,
                                    float b2, float eps, int t, void* stream)
{
    if (n <= 0 || !w || !g || !m || !v || t < 1) return SRWG_ERR_BAD_ARG;
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, (size_t)n, lr, b1, b2, eps, c1,
                                                                              c2);
    return launch_status(cudaGetLastError());
}

extern "C" SRWG_API int srwgMlpAdamMany(int n, float* const* w, const float* const* g, float* const* m, float* const* v,
                                        const long long* len, float lr, float b1, float b2, float eps, int t, void* stream)
{
    if (n <= 0 || !w || !g || !m || !v || !len || t < 1) return SRWG_ERR_BAD_ARG;
    for (int i = 0; i < n; i++)
        if (len[i] <= 0 || !w[i] || !g[i] || !m[i] || !v[i]) return SRWG_ERR_BAD_ARG;
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    for (int i0 = 0; i0 < n; i0 += ADAM_MOST) {
        AdamArrays a;
        a.n = n - i0 < ADAM_MOST ? n - i0 : ADAM_MOST;
        a.off[0] = 0;
        for (int i = 0; i < a.n; i++) {
            a.w[i] = w[i0 + i]; a.g[i] = g[i0 + i]; a.m[i] = m[i0 + i]; a.v[i] = v[i0 + i];
            a.off[i + 1] = a.off[i] + len[i0 + i];
        }
        adam_many_kernel<<<(unsigned)((a.off[a.n] + 255) / 256), 256, 0, (cudaStream_t)stream>>>(a, lr, b1, b2, eps, c1, c2);
    }
    return launch_status(cudaGetLastError());
}

extern "C" SRWG_API int srwgWfrFeatures(const float* dEx, const float* dEy, int nx, int ny, double xStart, double xStep,
                                        double zStart, double zStep, double k, double invRx0, double invRz0,
                                        float* dFeat, double* dSums, void* stream)
{
    if (!dEx || !dEy || nx < 64 || ny < 64 || !dFeat || !dSums) return SRWG_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    downsample_kernel<<<dim3(64, 64), 128, 0, st>>>((const float2*)dEx, (const float2*)dEy, nx, ny, dFeat);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemsetAsync(dSums, 0, 4 * sizeof(double), st);
    if (e == cudaSuccess) {
        curvature_kernel<<<296, 256, 0, st>>>((const float2*)dEx, nx, ny, xStart, xStep, zStart, zStep, k, invRx0,
                                              invRz0, dSums);
        e = cudaGetLastError();
    }
    return launch_status(e);
}
