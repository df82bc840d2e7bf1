// C-ABI of the library: the reference's srwlPropagElecField / srwlUtiSetWfrModifFunc /
// srwlUtiSetAllocArrayFunc / srwlUtiGetErrText (cpp/src/lib/srwlib.h:542, 549, 574, 821) and the srwgPlan* extensions, plus the
// executor that runs a plan's passes on a CUDA stream.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/srwl_b200.h"
#include "errors.h"
#include "kernels.h"
#include "exec.h"
#include "linep_shape.h"
#include "planner.h"

namespace srwg {

static std::string g_lastDetail;                          // detail text of the last error
void set_last_detail(const std::string& s) { g_lastDetail = s; }
const std::string& last_detail() { return g_lastDetail; }
static int (*g_modifFunc)(int, SRWLWfr*, char) = nullptr;  // client re-allocation callback
static char* (*g_allocArrayFunc)(char, long long) = nullptr; // client array allocation (extracted intensities)
static std::mutex g_mutex;
std::mutex& library_mutex() { return g_mutex; }

static std::map<int, DeviceCtx*> g_ctx;
static long long g_waitLimit = 0;                           // 0: the kernels' own default
long long wait_limit() { return g_waitLimit; }

#define CUDA_TRY(x)                                                                     \
    do {                                                                                \
        cudaError_t e__ = (x);                                                          \
        if (e__ != cudaSuccess) {                                                       \
            g_lastDetail = std::string(#x) + ": " + cudaGetErrorString(e__);            \
            return SRWG_ERR_CUDA;                                                       \
        }                                                                               \
    } while (0)

int device_ctx(int dev, DeviceCtx** out)
{
    auto it = g_ctx.find(dev);
    if (it != g_ctx.end()) {
        CUDA_TRY(cudaSetDevice(dev));
        *out = it->second;
        return 0;
    }
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) {
        g_lastDetail = "no CUDA device available";
        return SRWG_ERR_NO_DEVICE;
    }
    if (dev < 0 || dev >= n) {
        g_lastDetail = "device index out of range";
        return SRWG_ERR_NO_DEVICE;
    }
    CUDA_TRY(cudaSetDevice(dev));
    DeviceCtx* c = new DeviceCtx();
    c->dev = dev;
    CUDA_TRY(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
    CUDA_TRY(cudaMalloc(&c->status, sizeof(int)));
    CUDA_TRY(cudaMemset(c->status, 0, sizeof(int)));
    g_ctx[dev] = c;
    *out = c;
    return 0;
}

static std::mutex g_shapeMutex;
static std::map<int, PairShape> g_shapes;
static const PairShape* pair_shape(int N)
{
    std::lock_guard<std::mutex> lk(g_shapeMutex);
    auto it = g_shapes.find(N);
    if (it == g_shapes.end()) {
        PairShape z;
        if (!make_pair_shape(N, z)) z.n = 0;
        it = g_shapes.emplace(N, z).first;
    }
    return it->second.n ? &it->second : nullptr;
}

bool pair_supported(int N) { return pair_shape(N) != nullptr; }

// passes on pairs: the stages' tables (linep_shape.h); 16384 points: exp(-2 pi i k / N)
void line_twiddles(int N, std::vector<float2>& h)
{
    const PairShape* z = pair_shape(N);
    if (z != nullptr) {
        fill_twiddles(*z, h);
        return;
    }
    h.resize(N);
    for (int k = 0; k < N; k++) {
        const double a = -2. * M_PI * (double)k / (double)N;
        h[k] = make_float2((float)cos(a), (float)sin(a));
    }
}

int device_twiddles(DeviceCtx& c, int N, const float2** out)
{
    auto it = c.tw.find(N);
    if (it != c.tw.end()) { *out = it->second; return 0; }
    std::vector<float2> h;
    line_twiddles(N, h);
    float2* d = nullptr;
    CUDA_TRY(cudaMalloc(&d, sizeof(float2) * h.size()));
    CUDA_TRY(cudaMemcpy(d, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice));
    c.tw[N] = d;
    *out = d;
    return 0;
}

// ------------------------------------------------------------------------------------------------
// autotuned launch shapes: lines per CTA per (axis, N), measured by srw_b200.tune and stored as lines
// "rows|cols N L [spec]" in models/line_tuning.txt next to the library (or the file named by SRWG_TUNING);
// srwgTuneSetLines changes entries at run time.  The class of a length (power of two, or "spec": general) bounds
// the lines an entry may have (fixed_lines_valid) and chooses no kernel.
// ------------------------------------------------------------------------------------------------
static std::mutex g_tuneMutex;
struct TuneEntry {
    int fam = 0;       // 0: the length's own class
    int lines = 0;     // 0: the built-in choice
};
static std::map<std::pair<int, int>, TuneEntry> g_tune;
static bool g_tuneLoaded = false;

static int default_family(int N)
{
    return line2_supported(N) ? FAM_POW2 : linen_supported(N) ? FAM_SPEC : 0;
}

static int tune_load_file(const char* path, int* nOut)
{
    FILE* f = fopen(path, "r");
    if (!f) return -1;
    char line[256];
    int n = 0;
    while (fgets(line, sizeof(line), f)) {
        char ax[16], fam[16] = {0};
        int N = 0, L = 0;
        if (line[0] == '#') continue;
        const int got = sscanf(line, "%15s %d %d %15s", ax, &N, &L, fam);
        if (got < 3) continue;
        const int axis = strcmp(ax, "rows") == 0 ? 0 : strcmp(ax, "cols") == 0 ? 1 : -1;
        const int f = (got == 4 && strcmp(fam, "spec") == 0) ? FAM_SPEC : default_family(N);
        if (axis < 0 || !fixed_lines_valid(axis, N, L, f)) continue;
        TuneEntry e;
        e.fam = f;
        e.lines = L;
        g_tune[std::make_pair(axis, N)] = e;
        n++;
    }
    fclose(f);
    if (nOut) *nOut = n;
    return 0;
}

static void tune_ensure_loaded()
{
    if (g_tuneLoaded) return;
    g_tuneLoaded = true;
    const char* env = getenv("SRWG_TUNING");
    if (env != nullptr) {
        if (*env) tune_load_file(env, nullptr);           // SRWG_TUNING="" : defaults only
        return;
    }
    Dl_info info;
    if (dladdr((void*)&tune_load_file, &info) && info.dli_fname) {
        std::string so(info.dli_fname);
        const size_t cut = so.find_last_of('/');
        const std::string dir = cut == std::string::npos ? std::string(".") : so.substr(0, cut);
        tune_load_file((dir + "/../models/line_tuning.txt").c_str(), nullptr);
    }
}

static TuneEntry tuned(int axis, int N)
{
    std::lock_guard<std::mutex> lk(g_tuneMutex);
    tune_ensure_loaded();
    auto it = g_tune.find(std::make_pair(axis, N));
    return it != g_tune.end() ? it->second : TuneEntry();
}

int fixed_family(int axis, int N)
{
    const TuneEntry e = tuned(axis, N);
    return e.fam ? e.fam : default_family(N);
}

// pairs of lines per CTA: the tuned lines halved, else about 256 threads (columns: at least two pairs,
// 32-byte pieces of a row, a power of two)
static int pairs_per_cta(int axis, int N, const PairShape& z)
{
    const int lines = tuned(axis, N).lines;
    int G = lines > 0 ? lines / 2 : 256 / z.T;
    if (axis == 1 && lines == 0 && G < 2) G = 2;
    if (G < 1) G = 1;
    if (axis == 1) {
        if (G > 16) G = 16;
        while (G & (G - 1)) G &= G - 1;
    }
    while (G > 1 && (G * z.T > 512 || (size_t)G * (z.slot + 8) * 16 > SRWG_LINE_SMEM_MAX)) G = axis == 1 ? G / 2 : G - 1;
    return G;
}

int fixed_lines_per_cta(int axis, int N)
{
    if (default_family(N) == 0) return 0;
    const PairShape* z = pair_shape(N);
    return z ? 2 * pairs_per_cta(axis, N, *z) : 1;
}

int pair_block(int N, int nl)
{
    const PairShape* z = pair_shape(N);
    if (z == nullptr) return 0;
    int w = 2 * pairs_per_cta(1, N, *z);
    if (w < 4) w = 4;                        // whole 32-byte sectors for the row pass
    return nl % w == 0 ? w : 0;
}

int line_config(const LineDesc& d, LineLaunch& p)
{
    p.d = d;
    const int N = d.axis == 0 ? d.nx : d.nz;
    p.N = N;
    p.nlines = d.axis == 0 ? d.nz : d.nx;
    const PairShape* z = pair_shape(N);
    if (z != nullptr) {
        p.v2 = 0;
        p.T = z->T;
        p.G = pairs_per_cta(d.axis, N, *z);
        p.nst = z->n;
        for (int s = 0; s < z->n; s++) { p.radix[s] = z->R[s]; p.dR[s] = z->dR[s]; p.dB[s] = z->dB[s]; p.tw1[s] = z->tw1[s]; p.tw2[s] = z->tw2[s]; }
        for (int s = 0; s <= z->n; s++) { p.len[s] = z->len[s]; p.dL[s] = z->dL[s]; }
        p.pitch = z->pitch;
        // a windowed row pass on blocks of rows takes whole blocks where they are small
        if (d.axis == 0 && d.zwin && d.blk_in > 0) {
            const int G = d.blk_in / 2;
            if (!d.out_int && G * z->T <= 256) p.G = G;
        }
        if (d.axis == 0 && d.out_int) p.G = std::max(1, 128 / z->T);
        // few lines: rather more CTAs than pairs sharing one
        if (d.axis == 0)
            while (p.G > 1 && (long long)p.nlines * std::max(1, p.nb) < 148LL * 2 * p.G) p.G = (p.G + 1) / 2;
        p.L = (d.out_int ? 1 : 2) * p.G;
        // slots of a column tile start 8 / G places apart (their pairs read neighbouring lines together)
        p.P = z->slot;
        if (d.axis == 1 && p.G >= 2) {
            const int r = p.G >= 8 ? 1 : 8 / p.G;
            p.P += (r + 8 - p.P % 8) % 8;
        }
        return 0;
    }
    if (N == 16384) {
        // 16 points of one line per thread, radix-16 stages (line2.cuh)
        p.v2 = 1;
        p.T = N / 16;
        p.L = p.G = 1;
        p.P = (int)line_pitch(N, 1, d.axis == 1);
        return 0;
    }
    g_lastDetail = N > 8192 ? "FFT length above 8192" : "FFT length is not 2^a 3^b 5^c 7^d 11^e 13^f";
    return SRWG_ERR_UNSUPPORTED;
}

// device copy of a plan's constant data: its point-wise tables, then (256-byte aligned) its pass
// descriptors; returns the byte offset of the descriptors
static size_t const_bytes(const Planner& pl, size_t* descOff)
{
    size_t tb = pl.tables.size() * sizeof(float2);
    size_t off = (tb + 255) & ~(size_t)255;
    *descOff = off;
    return off + pl.kernels.size() * sizeof(KernelDesc);
}

static int upload_tables(const Planner& pl, float2** buf, size_t* capElems, cudaStream_t st)
{
    size_t descOff;
    size_t bytes = const_bytes(pl, &descOff);
    size_t n = (bytes + sizeof(float2) - 1) / sizeof(float2);
    if (*capElems < n || *buf == nullptr) {
        if (*buf) cudaFree(*buf);
        *buf = nullptr;
        *capElems = 0;
        CUDA_TRY(cudaMalloc(buf, n * sizeof(float2)));
        *capElems = n;
    }
    if (!pl.tables.empty())
        CUDA_TRY(cudaMemcpyAsync(*buf, pl.tables.data(), pl.tables.size() * sizeof(float2), cudaMemcpyHostToDevice, st));
    if (!pl.kernels.empty())
        CUDA_TRY(cudaMemcpyAsync((char*)*buf + descOff, pl.kernels.data(), pl.kernels.size() * sizeof(KernelDesc),
                                 cudaMemcpyHostToDevice, st));
    return 0;
}

// a pass whose lines outside its window are zero and read by nothing (zskip) launches only the window's
// line blocks; `d` holds the widest window of the launch (its wavefronts' windows start where each
// one's descriptor says, so that a batch of shifted ones launches no blocks outside them)
void line_window(const LineDesc& d, LineLaunch& p)
{
    if (d.zwin && d.zskip && d.zl0 <= d.zl1 && p.L > 0) p.nblk = (d.zl1 - d.zl0 + p.L - 1) / p.L + 1;
}

// a tiled resize that writes only its window launches only the window's tiles
void resize_window(const ResizeDesc& r, ResizeLaunch& p)
{
    if (!r.skip_zero || r.tile_or <= 0 || r.ixStart > r.ixEnd || r.izStart > r.izEnd) return;
    p.ntx = (int)((r.ixEnd - r.ixStart + SRWG_RESIZE_TX - 1) / SRWG_RESIZE_TX) + 1;
    p.ntz = (int)((r.izEnd - r.izStart + SRWG_RESIZE_TZ - 1) / SRWG_RESIZE_TZ) + 1;
}

// runs a pass list on nb wavefronts at once: buffer 0 = input (wavefront b at inX + b * inStride), 1/2 =
// work buffers (layout [buffer][component][wavefront][workElems]); the last pass writes the output
// (outX + b * outStride).  dconst holds per wavefront (stride constStride bytes) the tables and, at
// descOff, the pass descriptors; all wavefronts have passes of the same kinds and sizes.
int execute_passes(const std::vector<KernelDesc>& ks, DeviceCtx& c, int nb, const float2* inX, const float2* inY,
                   long long inStride, float2* outX, float2* outY, long long outStride, float2* work, size_t workElems,
                   const char* dconst, long long constStride, size_t descOff, cudaStream_t st, cudaEvent_t* ev,
                   const std::vector<KernelDesc>* hostMax, double* momScratch, double* momSlots, int nSlots,
                   char* intOut, size_t nRun, const unsigned* mask, int maskWords)
{
    const size_t nk = ks.size();
    const size_t W = (size_t)nb * workElems;
    float2* wb[3][2] = {{nullptr, nullptr}, {work, work + W}, {work + 2 * W, work + 3 * W}};
    const float2* tabs = (const float2*)dconst;
    const KernelDesc* gk = (const KernelDesc*)(dconst + descOff);
    const long long tabStride = constStride / (long long)sizeof(float2);
    // the last pass that writes a field writes the output; MOM passes after it read the output
    size_t lastField = nk;
    for (size_t i = nk; i-- > 0;)
        if (!reads_only(ks[i].kind)) { lastField = i; break; }

    for (size_t i = 0; i < nk && i < nRun; i++) {
        const KernelDesc& k = hostMax ? (*hostMax)[i] : ks[i];
        if (ev) CUDA_TRY(cudaEventRecord(ev[2 * i], st));
        const bool fromOut = reads_only(k.kind) && k.src != 0 && i > lastField && k.src == ks[lastField].dst;
        const bool fromIn = k.src == 0, toOut = i == lastField;
        const float2* s0 = fromOut ? outX : fromIn ? inX : wb[k.src][0];
        const float2* s1 = fromOut ? outY : fromIn ? inY : wb[k.src][1];
        float2* d0 = toOut ? outX : wb[k.dst][0];
        float2* d1 = toOut ? outY : wb[k.dst][1];
        const long long bSrc = fromOut ? outStride : fromIn ? inStride : (long long)workElems;
        const long long bDst = toOut ? outStride : (long long)workElems;
        // line passes may be set up while the pass before them ends (not between timing events)
        const bool pdlOk = i > 0 && ev == nullptr;
        cudaError_t e = cudaSuccess;
        if (k.kind == K_MOM) {
            if (momScratch == nullptr || momSlots == nullptr || k.mom.slot < 0 || k.mom.slot >= nSlots) {
                g_lastDetail = "moment pass without result buffers";
                return SRWG_ERR_BAD_ARG;
            }
            MomLaunch p;
            memset(&p, 0, sizeof(p));
            p.d = k.mom;
            p.src[0] = s0;
            p.src[1] = s1;
            p.tabs = tabs;
            p.gd = &gk[i].mom;
            p.scratch = momScratch;
            p.out = momSlots + (size_t)k.mom.slot * SRWG_MOM_SLOT;
            p.nb = nb; p.bDesc = constStride; p.bTab = tabStride;
            p.bSrc = bSrc;
            p.bOut = (long long)nSlots * SRWG_MOM_SLOT;
            e = launch_moments(p, st);
        } else if (k.kind == K_INT) {
            if (intOut == nullptr || nb != 1) {
                g_lastDetail = "intensity extraction pass without its buffer";
                return SRWG_ERR_BAD_ARG;
            }
            e = launch_extract(k.mom, &gk[i].mom, s0, s1, tabs, intOut + k.mom.ioff, st);
        } else if (k.kind == K_LINE) {
            LineLaunch p;
            memset(&p, 0, sizeof(p));
            p.nb = nb;
            int r = line_config(k.line, p);
            if (r) return r;
            r = device_twiddles(c, p.N, &p.tw);
            if (r) return r;
            p.src[0] = s0; p.src[1] = s1; p.dst[0] = d0; p.dst[1] = d1;
            p.tabs = tabs;
            p.gd = &gk[i].line;
            p.nb = nb; p.bDesc = constStride; p.bTab = tabStride; p.bSrc = bSrc; p.bDst = bDst;
            p.status = c.status;
            p.spin = g_waitLimit;
            p.byValue = hostMax == nullptr;
            p.run = k.line.run;
            line_window(k.line, p);
            if (mask != nullptr && i + 1 == std::min(nRun, nk)) {
                p.mask = mask;
                p.maskWords = maskWords;
            }
            e = launch_line(p, st, pdlOk);
        } else if (k.kind == K_RESIZE) {
            ResizeLaunch p;
            memset(&p, 0, sizeof(p));
            p.d = k.rs;
            p.src[0] = s0; p.src[1] = s1; p.dst[0] = d0; p.dst[1] = d1;
            p.xStepInvO = 1. / k.rs.xStepO;
            p.zStepInvO = 1. / k.rs.zStepO;
            resize_window(k.rs, p);
            p.tabs = tabs;
            p.gd = &gk[i].rs;
            p.nb = nb; p.bDesc = constStride; p.bTab = tabStride; p.bSrc = bSrc; p.bDst = bDst;
            e = launch_resize(p, st);
        } else {
            PwLaunch p;
            memset(&p, 0, sizeof(p));
            p.d = k.pwk;
            p.src[0] = s0; p.src[1] = s1; p.dst[0] = d0; p.dst[1] = d1;
            p.tabs = tabs;
            p.gd = &gk[i].pwk;
            p.nb = nb; p.bDesc = constStride; p.bTab = tabStride; p.bSrc = bSrc; p.bDst = bDst;
            e = launch_pw(p, st);
        }
        if (e != cudaSuccess) {
            g_lastDetail = std::string("kernel launch: ") + cudaGetErrorString(e);
            return SRWG_ERR_CUDA;
        }
        if (ev) CUDA_TRY(cudaEventRecord(ev[2 * i + 1], st));
    }
    return 0;
}

// doubles of the scratch of the plan's largest moment pass (0: no moment pass)
static size_t mom_scratch_for(const Planner& pl)
{
    size_t m = 0;
    for (const KernelDesc& k : pl.kernels)
        if (k.kind == K_MOM) m = std::max(m, mom_scratch_doubles(k.mom.nx, k.mom.nz));
    return m;
}

static int ensure_doubles(double** buf, size_t* cap, size_t n)
{
    if (*buf && *cap >= n) return 0;
    if (*buf) { cudaFree(*buf); *buf = nullptr; *cap = 0; }
    CUDA_TRY(cudaMalloc(buf, n * sizeof(double)));
    *cap = n;
    return 0;
}

// runs the plan's passes on one wavefront (or nb wavefronts with the same plan); moment passes
// write their sums to momSlots (nMomSlots * SRWG_MOM_SLOT doubles per wavefront)
// All plans of a device share its work buffers, on whatever streams they run.  While one stream uses them its order
// is enough; from the second one on an execution waits on its stream for the one queued before it, which recorded
// the event when it was queued (0.35 us of host time on the default stream; the checks 0.1 us; a propagation at
// 64 x 64 takes 20).  The library's own stream (calls on host memory) has finished when its call returns: it
// waits for the others and nobody for it.  A stream under capture takes no part: its graph's replays are
// ordered by who launches them.
static int work_begin(DeviceCtx& c, cudaStream_t st, bool* record)
{
    *record = false;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone ||
        (c.workDone == nullptr && cudaStreamGetId(st, &id) != cudaSuccess)) {
        cudaGetLastError();
        return 0;
    }
    const bool own = st == c.stream;
    if (c.workDone != nullptr) {
        CUDA_TRY(cudaStreamWaitEvent(st, c.workDone, 0));
        *record = true;
        return 0;
    }
    if (c.workStream != 0 && c.workStream != id) {
        // the first stream's executions recorded nothing (and it may be gone): wait for the device once
        // (refused while some stream is under capture)
        if (cudaDeviceSynchronize() != cudaSuccess) cudaGetLastError();
        if (!own) {
            CUDA_TRY(cudaEventCreateWithFlags(&c.workDone, cudaEventDisableTiming));
            *record = true;
        }
    }
    c.workStream = own ? 0 : id;
    return 0;
}

static int execute(Planner& pl, DeviceCtx& c, const float2* inX, const float2* inY, float2* outX, float2* outY,
                   float2* work, size_t workElems, const float2* dtab, cudaStream_t st, cudaEvent_t* ev = nullptr,
                   int nb = 1, long long inStride = 0, long long outStride = 0, double* momSlots = nullptr,
                   double* momScratch = nullptr, char* intOut = nullptr)
{
    const size_t nOut = (size_t)pl.w.nx * pl.w.nz;
    bool anyField = false;
    for (const KernelDesc& k : pl.kernels) anyField |= !reads_only(k.kind);
    if (!anyField) {          // the output is the input (moment passes, if any, read the input)
        for (int b = 0; b < nb; b++) {
            CUDA_TRY(cudaMemcpyAsync(outX + b * outStride, inX + b * inStride, nOut * sizeof(float2),
                                     cudaMemcpyDeviceToDevice, st));
            CUDA_TRY(cudaMemcpyAsync(outY + b * outStride, inY + b * inStride, nOut * sizeof(float2),
                                     cudaMemcpyDeviceToDevice, st));
        }
        if (pl.kernels.empty()) return 0;
    }
    size_t descOff;
    const_bytes(pl, &descOff);
    bool record;
    int r = work_begin(c, st, &record);
    if (r) return r;
    r = execute_passes(pl.kernels, c, nb, inX, inY, inStride, outX, outY, outStride, work, workElems,
                       (const char*)dtab, 0, descOff, st, ev, nullptr, momScratch, momSlots, pl.nMomSlots, intOut);
    if (record) CUDA_TRY(cudaEventRecord(c.workDone, st));
    return r;
}

static int ensure_work(DeviceCtx& c, size_t elems)
{
    elems += elems & 1;                          // 16-byte aligned fields
    if (c.workElems >= elems && c.work) return 0;
    if (c.work) { cudaFree(c.work); c.work = nullptr; c.workElems = 0; }
    CUDA_TRY(cudaMalloc(&c.work, 4 * elems * sizeof(float2)));
    c.workElems = elems;
    return 0;
}

static int ensure_io(DeviceCtx& c, size_t elems)
{
    if (c.ioElems >= elems && c.io) return 0;
    if (c.io) { cudaFree(c.io); c.io = nullptr; c.ioElems = 0; }
    CUDA_TRY(cudaMalloc(&c.io, 4 * elems * sizeof(float2)));
    c.ioElems = elems;
    return 0;
}

static void out_wfr(const Planner& pl, SRWLWfr* p)
{   // OutSRWRadPtrs (srradstr.cpp:687): mesh and scalars
    const WfrState& w = pl.w;
    p->mesh.eStart = w.eStart;
    p->mesh.eFin = w.eStart;
    p->mesh.xStart = w.xStart;
    p->mesh.xFin = w.xStart + w.xStep * (w.nx - 1);
    p->mesh.yStart = w.zStart;
    p->mesh.yFin = w.zStart + w.zStep * (w.nz - 1);
    p->mesh.ne = 1;
    p->mesh.nx = w.nx;
    p->mesh.ny = w.nz;
    p->Rx = w.RobsX; p->Ry = w.RobsZ;
    p->dRx = w.RobsXAbsErr; p->dRy = w.RobsZAbsErr;
    p->xc = w.xc; p->yc = w.zc;
    p->presCA = (char)w.Pres;
    p->avgPhotEn = w.avgPhotEn;
    if (p->arElecPropMatr != nullptr && w.havePropM)
        for (int i = 0; i < 20; i++) p->arElecPropMatr[i] = w.propM[i];
}

// output moments: the plan-time ones, or (with moment passes) the replayed bookkeeping with the
// passes' result slots of one wavefront
static void out_moments(const Planner& pl, SRWLWfr* p, const double* slots = nullptr)
{
    double mx[11], mz[11];
    if (pl.nMomSlots > 0 && slots != nullptr) pl.replay_moments(slots, mx, mz);
    else for (int i = 0; i < 11; i++) { mx[i] = pl.w.momX[i]; mz[i] = pl.w.momZ[i]; }
    if (p->arMomX) for (int i = 0; i < 11; i++) p->arMomX[i] = mx[i];
    if (p->arMomY) for (int i = 0; i < 11; i++) p->arMomY[i] = mz[i];
}

}  // namespace srwg

using namespace srwg;

struct srwgPlan {
    Planner pl;
    int device = 0;
    DeviceCtx* ctx = nullptr;   // bound at the first execution
    float2* dtab = nullptr;     // the plan's point-wise tables on that device
    size_t dtabElems = 0;
    bool tabReady = false;
    double* dmom = nullptr;     // moment passes: result slots of every wavefront | scratch
    size_t dmomDoubles = 0;
    int lastN = 0;              // wavefronts of the last execution
    cudaEvent_t momEv = nullptr;  // recorded after the last execution
    ~srwgPlan()
    {
        if (dtab) cudaFree(dtab);
        if (dmom) cudaFree(dmom);
        if (momEv) cudaEventDestroy(momEv);
    }
};

// moment buffers of a plan for n wavefronts; slots of wavefront b at dmom + b * nMomSlots * SLOT
static int plan_moments(srwgPlan* plan, int n, double** slots, double** scratch)
{
    *slots = *scratch = nullptr;
    if (plan->pl.nMomSlots == 0) return 0;
    const size_t per = (size_t)plan->pl.nMomSlots * SRWG_MOM_SLOT;
    int r = ensure_doubles(&plan->dmom, &plan->dmomDoubles, per * (size_t)n + mom_scratch_for(plan->pl));
    if (r) return r;
    if (plan->momEv == nullptr) CUDA_TRY(cudaEventCreateWithFlags(&plan->momEv, cudaEventDisableTiming));
    *slots = plan->dmom;
    *scratch = plan->dmom + per * (size_t)n;
    return 0;
}

// result slots of wavefront b of the last execution (host copy); false when there are none
static bool plan_slots(const srwgPlan* plan, int b, std::vector<double>& hs)
{
    if (plan->pl.nMomSlots == 0 || plan->lastN <= b || plan->dmom == nullptr || plan->momEv == nullptr) return false;
    const size_t per = (size_t)plan->pl.nMomSlots * SRWG_MOM_SLOT;
    hs.resize(per);
    if (cudaSetDevice(plan->device) != cudaSuccess || cudaEventSynchronize(plan->momEv) != cudaSuccess ||
        cudaMemcpy(hs.data(), plan->dmom + per * (size_t)b, per * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
        return false;
    return true;
}

static int plan_bind(srwgPlan* plan, cudaStream_t st)
{
    int r = device_ctx(plan->device, &plan->ctx);
    if (r) return r;
    if (!plan->tabReady) {
        r = upload_tables(plan->pl, &plan->dtab, &plan->dtabElems, st);
        if (r) return r;
        CUDA_TRY(cudaStreamSynchronize(st));
        plan->tabReady = true;
    }
    return ensure_work(*plan->ctx, (size_t)plan->pl.maxElems);
}

extern "C" {

void srwlUtiSetWfrModifFunc(int (*pExtFunc)(int action, SRWLWfr* pWfrIn, char pol))
{
    std::lock_guard<std::mutex> lk(g_mutex);
    g_modifFunc = pExtFunc;
}

void srwlUtiSetAllocArrayFunc(char* (*pExtFunc)(char type, long long len))
{
    std::lock_guard<std::mutex> lk(g_mutex);
    g_allocArrayFunc = pExtFunc;
}

int srwlUtiGetErrText(char* t, int erNo)
{
    if (t == nullptr) return 0;
    const char* s = nullptr;
    switch (erNo) {
    case 0: s = ""; break;
    case MEMORY_ALLOCATION_FAILURE: s = "Memory allocation failure."; break;
    case UNKNOWN_OPTICAL_ELEMENT: s = "Unknown optical element or incorrect optical element definition."; break;
    case ERROR_IN_FFT: s = "Error in FFT."; break;
    case CAN_NOT_PROPAGATE_1D_RAD: s = "Propagation needs more than one point in both the horizontal and the vertical direction."; break;
    case PHOT_EN_SHOULD_BE_POSITIVE: s = "Photon energy should be positive."; break;
    case SRWL_INCORRECT_PARAM_FOR_GAUS_BEAM_COMP: s = "Incorrect or insufficient parameters for Gaussian beam calculation."; break;
    case SRWL_INCORRECT_PARAM_FOR_INT_EXTR: s = "Incorrect or insufficient parameters for intensity extraction."; break;
    case SRWL_WFR_EXT_MODIF_FAILED: s = "The wavefront modification (re-allocation) callback failed."; break;
    case SRWL_INCORRECT_PARAM_FOR_WFR_PROP: s = "Incorrect or insufficient parameters for wavefront propagation."; break;
    case SRWL_WFR_EXT_FUNC_NOT_DEFINED: s = "No wavefront modification (re-allocation) callback is registered."; break;
    case SRWL_EXT_ARRAY_ALLOC_FAILED: s = "Failed to allocate array in front-end / client environment."; break;
    case SRWG_ERR_UNSUPPORTED: s = "Not supported on the GPU propagation path"; break;
    case SRWG_ERR_CUDA: s = "CUDA error"; break;
    case SRWG_ERR_NO_DEVICE: s = "No usable CUDA device"; break;
    case SRWG_ERR_BAD_ARG: s = "Invalid argument"; break;
    case SRWG_ERR_STATIC_LIMIT: s = "Propagation too large for the allocation-free entry point"; break;
    default: s = "Unknown error or warning number."; break;
    }
    std::string txt(s);
    if ((erNo >= SRWG_ERR_UNSUPPORTED && erNo <= SRWG_ERR_STATIC_LIMIT) && !g_lastDetail.empty()) txt += ": " + g_lastDetail;
    strncpy(t, txt.c_str(), 2047);
    t[2047] = 0;
    return 0;
}

// the caller's field components into (dX, dY), zeros for one that is absent
static int field_to_device(DeviceCtx& c, const SRWLWfr* w, size_t n, float2* dX, float2* dY, cudaStream_t st)
{
    CopySeg seg[2];
    int k = 0;
    if (w->arEx) seg[k++] = {w->arEx, dX, n * sizeof(float2)};
    else CUDA_TRY(cudaMemsetAsync(dX, 0, n * sizeof(float2), st));
    if (w->arEy) seg[k++] = {w->arEy, dY, n * sizeof(float2)};
    else CUDA_TRY(cudaMemsetAsync(dY, 0, n * sizeof(float2), st));
    CUDA_TRY(copy_segments(c.ring, c.dev, seg, k, true, st));
    return 0;
}

// (dX, dY) into the caller's arrays, those that are there; the stream has finished on return
static int field_to_host(DeviceCtx& c, char* hX, char* hY, size_t n, float2* dX, float2* dY, cudaStream_t st)
{
    CopySeg seg[2];
    int k = 0;
    if (hX) seg[k++] = {hX, dX, n * sizeof(float2)};
    if (hY) seg[k++] = {hY, dY, n * sizeof(float2)};
    CUDA_TRY(copy_segments(c.ring, c.dev, seg, k, false, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    return 0;
}

// the intensity extractions of a stage that ran: each into the caller's array (allocated through the
// registered allocation function when the caller passed none, AllocExtIntArray srradstr.cpp:799),
// with its mesh (GetIntMesh, srradstr.cpp:4140: the wavefront's x and y mesh, eStart kept)
static int deliver_extractions(const Planner& pl, const char* dev, cudaStream_t st, char** arI, SRWLRadMesh* arIM)
{
    for (const IntOut& o : pl.intOuts) {
        char*& dst = arI[o.index];
        if (dst == nullptr) {
            if (g_allocArrayFunc != nullptr) dst = (*g_allocArrayFunc)(o.arType, (long long)o.nx * o.nz);
            if (dst == nullptr) return SRWL_EXT_ARRAY_ALLOC_FAILED;
        }
        CUDA_TRY(cudaMemcpyAsync(dst, dev + o.off, (size_t)o.bytes, cudaMemcpyDeviceToHost, st));
        if (arIM != nullptr) {
            SRWLRadMesh& m = arIM[o.index];
            m.ne = 1;
            m.nx = o.nx;
            m.xStart = o.xStart;
            m.xFin = o.xStart + o.xStep * (o.nx - 1);
            m.ny = o.nz;
            m.yStart = o.zStart;
            m.yFin = o.zStart + o.zStep * (o.nz - 1);
        }
    }
    CUDA_TRY(cudaStreamSynchronize(st));
    return 0;
}

// srwlPropagElecField for a plan with stage boundaries (an element planned on moments measured from
// the field) or intensity extractions: each stage runs from the previous stage's output into a stage
// buffer, its moment results and extractions come back to the host, and planning resumes; the last
// stage's output is the result.  pr: the planning status (SRWG_NEED_STAGE or 0 for a single stage)
static int propagate_staged(Planner& pl, SRWLWfr* pWfr, int dev, int pr, char** arI, SRWLRadMesh* arIM)
{
    DeviceCtx* c = nullptr;
    int r = device_ctx(dev, &c);
    if (r) return r;
    cudaStream_t st = c->stream;
    const size_t nIn = (size_t)pl.in.nx * pl.in.nz;
    r = ensure_io(*c, nIn);
    if (r) return r;
    r = field_to_device(*c, pWfr, nIn, c->io, c->io + c->ioElems, st);
    if (r) return r;
    const float2* curX = c->io;
    const float2* curY = c->io + c->ioElems;
    float2 *oX = nullptr, *oY = nullptr;
    std::vector<double> slots, tmp;
    for (int k = 0;; k++) {
        const bool last = (pr == 0);
        const size_t nSt = (size_t)pl.w.nx * pl.w.nz;
        float2*& sb = c->stg[k & 1];
        size_t& se = c->stgElems[k & 1];
        if (sb == nullptr || se < nSt) {
            if (sb) cudaFree(sb);
            sb = nullptr; se = 0;
            CUDA_TRY(cudaMalloc(&sb, 2 * nSt * sizeof(float2)));
            se = nSt;
        }
        oX = sb; oY = sb + se;
        r = ensure_work(*c, (size_t)std::max<long long>(pl.maxElems, 1));
        if (r) return r;
        r = upload_tables(pl, &c->tab, &c->tabElems, st);
        if (r) return r;
        const size_t nSlotD = (size_t)pl.nMomSlots * SRWG_MOM_SLOT;
        if (nSlotD) {
            r = ensure_doubles(&c->mom, &c->momDoubles, nSlotD + mom_scratch_for(pl));
            if (r) return r;
        }
        if (pl.intBytes > 0 && (c->genBuf == nullptr || c->genBytes < (size_t)pl.intBytes)) {
            if (c->genBuf) cudaFree(c->genBuf);
            c->genBuf = nullptr; c->genBytes = 0;
            CUDA_TRY(cudaMalloc(&c->genBuf, (size_t)pl.intBytes));
            c->genBytes = (size_t)pl.intBytes;
        }
        r = execute(pl, *c, curX, curY, oX, oY, c->work, c->workElems, c->tab, st, nullptr, 1, 0, 0,
                    nSlotD ? c->mom : nullptr, nSlotD ? c->mom + nSlotD : nullptr,
                    pl.intBytes > 0 ? (char*)c->genBuf : nullptr);
        if (r) return r;
        if (!pl.intOuts.empty()) {
            r = deliver_extractions(pl, (const char*)c->genBuf, st, arI, arIM);
            if (r) return r;
        }
        tmp.assign(nSlotD, 0.);
        if (nSlotD) CUDA_TRY(cudaMemcpyAsync(tmp.data(), c->mom, nSlotD * sizeof(double), cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaStreamSynchronize(st));
        slots.resize(nSlotD, 0.);
        for (const KernelDesc& kd : pl.kernels)          // the slots this stage's passes wrote
            if (kd.kind == K_MOM)
                std::copy(tmp.begin() + (size_t)kd.mom.slot * SRWG_MOM_SLOT,
                          tmp.begin() + (size_t)(kd.mom.slot + 1) * SRWG_MOM_SLOT,
                          slots.begin() + (size_t)kd.mom.slot * SRWG_MOM_SLOT);
        if (last) break;
        pr = pl.resume(slots.data());
        if (pr && pr != SRWG_NEED_STAGE) { g_lastDetail = pl.err; return pr; }
        curX = oX; curY = oY;
    }
    const size_t nOut = (size_t)pl.w.nx * pl.w.nz;
    bool hadX = pWfr->arEx != nullptr, hadY = pWfr->arEy != nullptr;
    bool resized = (pl.w.nx != pl.in.nx) || (pl.w.nz != pl.in.nz);
    out_wfr(pl, pWfr);
    if (resized) {
        if (g_modifFunc == nullptr) return SRWL_WFR_EXT_FUNC_NOT_DEFINED;
        if ((*g_modifFunc)(2, pWfr, 0)) return SRWL_WFR_EXT_MODIF_FAILED;
        out_wfr(pl, pWfr);
    }
    r = field_to_host(*c, hadX ? pWfr->arEx : nullptr, hadY ? pWfr->arEy : nullptr, nOut, oX, oY, st);
    if (r) return r;
    out_moments(pl, pWfr, slots.empty() ? nullptr : slots.data());
    return 0;
}

int srwlPropagElecField(SRWLWfr* pWfr, SRWLOptC* pOpt, int nInt, char** arID, SRWLRadMesh* arIM, char** arI,
                        double* arParGPU)
{
    std::lock_guard<std::mutex> lk(g_mutex);
    g_lastDetail.clear();
    if (pWfr == nullptr || pOpt == nullptr) return SRWL_INCORRECT_PARAM_FOR_WFR_PROP;
    int dev = 0;
    if (arParGPU != nullptr && arParGPU[0] >= 1. && arParGPU[1] >= 1.) dev = (int)arParGPU[1] - 1;
    if (pWfr->arEx == nullptr && pWfr->arEy == nullptr) return SRWL_INCORRECT_PARAM_FOR_WFR_PROP;

    Planner pl;
    pl.allowStages = true;
    // intensity extractions after elements (PropagateRadiationGuided, sroptcnt.cpp:268, and
    // ExtractPropagatedIntensity :429): arID[0..4][i] = element number (1-based), polarisation,
    // intensity type, dependence, representation; negative values (and arIM[i].ne < 0) of the
    // later requests take the first request's
    const bool wantInt = nInt > 0 && arID != nullptr && arI != nullptr;
    if (wantInt) {
        for (int j = 0; j < 5; j++)
            if (arID[j] == nullptr) return SRWL_INCORRECT_PARAM_FOR_WFR_PROP;
        for (int i = 0; i < nInt; i++) {
            IntReq q;
            q.index = i;
            q.elem = (int)arID[0][i] - 1;
            q.pol = arID[1][i]; q.type = arID[2][i]; q.dep = arID[3][i]; q.pres = arID[4][i];
            if (nInt > 1 && i > 0) {
                if (q.pol < 0) q.pol = arID[1][0];
                if (q.type < 0) q.type = arID[2][0];
                if (q.dep < 0) q.dep = arID[3][0];
                if (q.pres < 0) q.pres = arID[4][0];
                if (arIM != nullptr && arIM[i].ne < 0) arIM[i] = arIM[0];
            }
            pl.intReqs.push_back(q);
        }
    }
    int r = pl.plan(pWfr, pOpt);
    if (r == SRWG_NEED_STAGE || (r == 0 && wantInt))
        return propagate_staged(pl, pWfr, dev, r, wantInt ? arI : nullptr, wantInt ? arIM : nullptr);
    if (r) { g_lastDetail = pl.err; return r; }
    DeviceCtx* c = nullptr;
    r = device_ctx(dev, &c);
    if (r) return r;
    const size_t nIn = (size_t)pl.in.nx * pl.in.nz, nOut = (size_t)pl.w.nx * pl.w.nz;
    r = ensure_io(*c, nIn > nOut ? nIn : nOut);
    if (r) return r;
    r = ensure_work(*c, (size_t)pl.maxElems);
    if (r) return r;
    float2* inX = c->io;
    float2* inY = c->io + c->ioElems;
    float2* outX = c->io + 2 * c->ioElems;
    float2* outY = c->io + 3 * c->ioElems;
    cudaStream_t st = c->stream;
    r = field_to_device(*c, pWfr, nIn, inX, inY, st);
    if (r) return r;
    r = upload_tables(pl, &c->tab, &c->tabElems, st);
    if (r) return r;
    const size_t nSlotD = (size_t)pl.nMomSlots * SRWG_MOM_SLOT;
    if (nSlotD) {
        r = ensure_doubles(&c->mom, &c->momDoubles, nSlotD + mom_scratch_for(pl));
        if (r) return r;
    }
    r = execute(pl, *c, inX, inY, outX, outY, c->work, c->workElems, c->tab, st, nullptr, 1, 0, 0,
                nSlotD ? c->mom : nullptr, nSlotD ? c->mom + nSlotD : nullptr);
    if (r) return r;
    std::vector<double> hs(nSlotD);
    if (nSlotD) CUDA_TRY(cudaMemcpyAsync(hs.data(), c->mom, nSlotD * sizeof(double), cudaMemcpyDeviceToHost, st));
    bool hadX = pWfr->arEx != nullptr, hadY = pWfr->arEy != nullptr;
    bool resized = (pl.w.nx != pl.in.nx) || (pl.w.nz != pl.in.nz);
    out_wfr(pl, pWfr);
    if (resized) {
        CUDA_TRY(cudaStreamSynchronize(st));
        if (g_modifFunc == nullptr) return SRWL_WFR_EXT_FUNC_NOT_DEFINED;
        if ((*g_modifFunc)(2, pWfr, 0)) return SRWL_WFR_EXT_MODIF_FAILED;
        out_wfr(pl, pWfr);
    }
    r = field_to_host(*c, hadX ? pWfr->arEx : nullptr, hadY ? pWfr->arEy : nullptr, nOut, outX, outY, st);
    if (r) return r;
    out_moments(pl, pWfr, nSlotD ? hs.data() : nullptr);
    return 0;
}

int srwgPlanCreate(const SRWLWfr* pWfr, const SRWLOptC* pOpt, int device, srwgPlan** ppPlan)
{
    if (ppPlan == nullptr) return SRWG_ERR_BAD_ARG;
    *ppPlan = nullptr;
    // the planner is host bookkeeping without shared state: plans are made outside the library lock,
    // so that threads can plan concurrently
    srwgPlan* p = new srwgPlan();
    int r = p->pl.plan(pWfr, pOpt);
    std::lock_guard<std::mutex> lk(g_mutex);
    g_lastDetail.clear();
    if (r) { g_lastDetail = p->pl.err; delete p; return r; }
    p->device = device;
    // validate every pass configuration up front
    for (const KernelDesc& k : p->pl.kernels) {
        if (k.kind == K_LINE) {
            LineLaunch l;
            memset(&l, 0, sizeof(l));
            r = line_config(k.line, l);
            if (r) { delete p; return r; }
        }
    }
    *ppPlan = p;
    return 0;
}

int srwgPlanGetOutput(const srwgPlan* plan, SRWLWfr* pWfrOut)
{
    if (plan == nullptr || pWfrOut == nullptr) return SRWG_ERR_BAD_ARG;
    out_wfr(plan->pl, pWfrOut);
    std::vector<double> hs;
    const bool have = plan_slots(plan, 0, hs);
    out_moments(plan->pl, pWfrOut, have ? hs.data() : nullptr);
    return 0;
}

int srwgPlanGetMoments(const srwgPlan* plan, int index, double* momX, double* momY)
{
    if (plan == nullptr || index < 0) return SRWG_ERR_BAD_ARG;
    double mx[11], mz[11];
    if (plan->pl.nMomSlots == 0) {
        for (int i = 0; i < 11; i++) { mx[i] = plan->pl.w.momX[i]; mz[i] = plan->pl.w.momZ[i]; }
    } else {
        std::vector<double> hs;
        if (!plan_slots(plan, index, hs)) {
            g_lastDetail = "no executed wavefront with this index";
            return SRWG_ERR_BAD_ARG;
        }
        plan->pl.replay_moments(hs.data(), mx, mz);
    }
    if (momX) for (int i = 0; i < 11; i++) momX[i] = mx[i];
    if (momY) for (int i = 0; i < 11; i++) momY[i] = mz[i];
    return 0;
}

int srwgPlanInfo(const srwgPlan* plan, long* nxIn, long* nyIn, long* nxOut, long* nyOut, int* nKernels, long long* workBytes)
{
    if (plan == nullptr) return SRWG_ERR_BAD_ARG;
    if (nxIn) *nxIn = plan->pl.in.nx;
    if (nyIn) *nyIn = plan->pl.in.nz;
    if (nxOut) *nxOut = plan->pl.w.nx;
    if (nyOut) *nyOut = plan->pl.w.nz;
    if (nKernels) *nKernels = (int)plan->pl.kernels.size();
    if (workBytes) *workBytes = 4LL * plan->pl.maxElems * (long long)sizeof(float2);
    return 0;
}

int srwgPlanExecute(srwgPlan* plan, const float* dExIn, const float* dEyIn, float* dExOut, float* dEyOut, void* stream)
{
    return srwgPlanExecuteBatch(plan, 1, dExIn, dEyIn, 0, dExOut, dEyOut, 0, stream);
}

int srwgPlanExecuteBatch(srwgPlan* plan, int n, const float* dExIn, const float* dEyIn, long long strideIn,
                         float* dExOut, float* dEyOut, long long strideOut, void* stream)
{
    std::lock_guard<std::mutex> lk(g_mutex);
    g_lastDetail.clear();
    if (plan == nullptr || dExIn == nullptr || dEyIn == nullptr || dExOut == nullptr || dEyOut == nullptr || n < 1)
        return SRWG_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    int r = plan_bind(plan, st);
    if (r) return r;
    DeviceCtx& c = *plan->ctx;
    if ((strideIn & 1) || (strideOut & 1)) return SRWG_ERR_BAD_ARG;     // whole complex points
    // one launch per pass for the whole batch (grid z = wavefront) when the work buffers hold it
    const size_t per = ((size_t)plan->pl.maxElems + 1) & ~(size_t)1;     // 16-byte aligned fields
    int chunk = n;
    const size_t budget = (size_t)1 << 30;                               // work elements (8 GiB)
    while (chunk > 1 && 4 * (size_t)chunk * per > budget) chunk = (chunk + 1) / 2;
    r = ensure_work(c, (size_t)chunk * per);
    if (r) return r;
    double *slots, *scratch;
    r = plan_moments(plan, n, &slots, &scratch);
    if (r) return r;
    const size_t perSlots = (size_t)plan->pl.nMomSlots * SRWG_MOM_SLOT;
    for (int b0 = 0; b0 < n; b0 += chunk) {
        const int nb = std::min(chunk, n - b0);
        r = execute(plan->pl, c, (const float2*)(dExIn + b0 * strideIn), (const float2*)(dEyIn + b0 * strideIn),
                    (float2*)(dExOut + b0 * strideOut), (float2*)(dEyOut + b0 * strideOut), c.work, per, plan->dtab,
                    st, nullptr, nb, strideIn / 2, strideOut / 2, slots ? slots + perSlots * b0 : nullptr, scratch);
        if (r) return r;
    }
    if (slots) {
        CUDA_TRY(cudaEventRecord(plan->momEv, st));
        plan->lastN = n;
    }
    return 0;
}

int srwgPlanExecuteTimed(srwgPlan* plan, const float* dExIn, const float* dEyIn, float* dExOut, float* dEyOut,
                         void* stream, float* kernelMs, int maxKernels, int* nTimed)
{
    std::lock_guard<std::mutex> lk(g_mutex);
    g_lastDetail.clear();
    if (plan == nullptr || dExIn == nullptr || dEyIn == nullptr || dExOut == nullptr || dEyOut == nullptr)
        return SRWG_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    int r = plan_bind(plan, st);
    if (r) return r;
    DeviceCtx& c = *plan->ctx;
    const size_t nk = plan->pl.kernels.size();
    std::vector<cudaEvent_t> ev(2 * nk);
    for (auto& e : ev) CUDA_TRY(cudaEventCreate(&e));
    double *slots, *scratch;
    r = plan_moments(plan, 1, &slots, &scratch);
    if (r == 0)
        r = execute(plan->pl, c, (const float2*)dExIn, (const float2*)dEyIn, (float2*)dExOut, (float2*)dEyOut, c.work,
                    c.workElems, plan->dtab, st, nk ? ev.data() : nullptr, 1, 0, 0, slots, scratch);
    if (r == 0 && slots) {
        if (cudaEventRecord(plan->momEv, st) != cudaSuccess) r = SRWG_ERR_CUDA;
        else plan->lastN = 1;
    }
    if (r == 0) {
        CUDA_TRY(cudaStreamSynchronize(st));
        for (size_t i = 0; i < nk && (int)i < maxKernels; i++) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev[2 * i], ev[2 * i + 1]);
            if (kernelMs) kernelMs[i] = ms;
        }
        if (nTimed) *nTimed = (int)nk;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    return r;
}

int srwgPlanDestroy(srwgPlan* plan)
{
    delete plan;
    return 0;
}

int srwgSetWaitLimit(long long iterations)
{
    std::lock_guard<std::mutex> lk(g_mutex);
    if (iterations < 0) return SRWG_ERR_BAD_ARG;
    g_waitLimit = iterations;
    return 0;
}

int srwgGetWaitStatus(int device, int* count, int reset)
{
    std::lock_guard<std::mutex> lk(g_mutex);
    if (count == nullptr) return SRWG_ERR_BAD_ARG;
    DeviceCtx* c = nullptr;
    int r = device_ctx(device, &c);
    if (r) return r;
    CUDA_TRY(cudaMemcpy(count, c->status, sizeof(int), cudaMemcpyDeviceToHost));
    if (reset) CUDA_TRY(cudaMemset(c->status, 0, sizeof(int)));
    return 0;
}

long srwgNextFftNumber(long n)
{
    return srwg::next_correct_number_for_fft(n);
}

int srwgTuneSetFamily(int axis, int N, int family)
{
    std::lock_guard<std::mutex> lk(g_tuneMutex);
    tune_ensure_loaded();
    if ((axis != 0 && axis != 1) || !default_family(N)) return SRWG_ERR_BAD_ARG;
    const int f = family == 0 ? default_family(N) : family;
    if (!(f == FAM_POW2 && line2_supported(N)) && !(f == FAM_SPEC && (linen_supported(N) || linen_pow2(N)))) {
        g_lastDetail = "no kernel of this family for this line length";
        return SRWG_ERR_BAD_ARG;
    }
    TuneEntry& e = g_tune[std::make_pair(axis, N)];
    e.fam = f;
    if (e.lines && !fixed_lines_valid(axis, N, e.lines, f)) e.lines = 0;
    return 0;
}

int srwgTuneSetLines(int axis, int N, int lines)
{
    std::lock_guard<std::mutex> lk(g_tuneMutex);
    tune_ensure_loaded();
    if (axis != 0 && axis != 1) return SRWG_ERR_BAD_ARG;
    auto key = std::make_pair(axis, N);
    auto it = g_tune.find(key);
    const int fam = (it != g_tune.end() && it->second.fam) ? it->second.fam : default_family(N);
    if (lines == 0) {
        if (it != g_tune.end()) g_tune.erase(it);
        return 0;
    }
    if (!fixed_lines_valid(axis, N, lines, fam)) {
        g_lastDetail = "not a valid launch shape for this line length";
        return SRWG_ERR_BAD_ARG;
    }
    g_tune[key].fam = fam;
    g_tune[key].lines = lines;
    return 0;
}

int srwgTuneGetLines(int axis, int N, int* lines)
{
    if (lines == nullptr || (axis != 0 && axis != 1)) return SRWG_ERR_BAD_ARG;
    *lines = fixed_lines_per_cta(axis, N);
    return 0;
}

int srwgTuneGetFamily(int axis, int N, int* family)
{
    if (family == nullptr || (axis != 0 && axis != 1)) return SRWG_ERR_BAD_ARG;
    *family = fixed_family(axis, N);
    return 0;
}

int srwgTuneLoad(const char* path, int* nEntries)
{
    std::lock_guard<std::mutex> lk(g_tuneMutex);
    g_tuneLoaded = true;
    g_tune.clear();
    if (path == nullptr || !*path) { if (nEntries) *nEntries = 0; return 0; }
    if (tune_load_file(path, nEntries) != 0) {
        g_lastDetail = std::string("cannot read ") + path;
        return SRWG_ERR_BAD_ARG;
    }
    return 0;
}

int srwgPlanDescribe(const srwgPlan* plan, char* buf, int bufLen)
{
    if (plan == nullptr || buf == nullptr || bufLen <= 0) return SRWG_ERR_BAD_ARG;
    std::string s = plan->pl.describe();
    strncpy(buf, s.c_str(), bufLen - 1);
    buf[bufLen - 1] = 0;
    return 0;
}

}  // extern "C"
