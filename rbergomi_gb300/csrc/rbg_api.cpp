// rbg_api.cpp -- host side of librbergomi_gb300: device contexts, cached
// buffers and tables, the drop-in C ABI and the extended rbg_* API.
//
// The drop-in functions keep the reference's observable behaviour
// (rBergLib/cinterface.cpp): same argument meaning and output layout, the
// same stderr message + exit(17) on out_size != par_size * op_size and
// exit(21) on num_threads < 1.  GPU failures, which the reference cannot
// have, exit with status 70 after a message.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <iostream>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "rbg_fp64x.hpp"
#include "rbg_internal.hpp"
#include "rbg_mixed.hpp"

namespace rbg {

static std::atomic<uint64_t> g_launches{0};
void count_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }

static thread_local std::string g_err;
// ------------------------------------------------------------- profiling
// When enabled, CUDA events are recorded on the launching stream around each
// stage; durations are folded in after the call's final synchronisation.
enum { kStageNormals = 0, kStagePathFp64 = 1, kStageMixed = 2, kStagePayoff = 3, kStageReduce = 4, kStages = 5 };
struct Prof {
    std::mutex mu;
    bool on = false;
    double ms[kStages] = {0};
    uint64_t n[kStages] = {0};
    const char* path = "";  // kernels of the last profiled FP64 path pass
    std::vector<cudaEvent_t> pool;
    std::vector<std::tuple<int, cudaEvent_t, cudaEvent_t, int>> pending;
};
static Prof g_prof;

struct ProfScope {
    int stage, count;
    cudaStream_t st;
    cudaEvent_t a = nullptr, b = nullptr;
    ProfScope(int stage_, cudaStream_t st_, int count_ = 1) : stage(stage_), count(count_), st(st_)
    {
        std::lock_guard<std::mutex> lk(g_prof.mu);
        if (!g_prof.on) return;
        for (cudaEvent_t* e : {&a, &b}) {
            if (!g_prof.pool.empty()) { *e = g_prof.pool.back(); g_prof.pool.pop_back(); }
            else cudaEventCreate(e);
        }
        cudaEventRecord(a, st);
    }
    ~ProfScope()
    {
        if (!a) return;
        cudaEventRecord(b, st);
        std::lock_guard<std::mutex> lk(g_prof.mu);
        g_prof.pending.emplace_back(stage, a, b, count);
    }
};

// Names the kernels of the FP64 form's path pass, while profiling is on.
static void prof_path(const char* kernels)
{
    std::lock_guard<std::mutex> lk(g_prof.mu);
    if (g_prof.on) g_prof.path = kernels;
}

// called after the stream that carried the pending events has synchronised
static void prof_collect()
{
    std::lock_guard<std::mutex> lk(g_prof.mu);
    for (auto& t : g_prof.pending) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, std::get<1>(t), std::get<2>(t)) == cudaSuccess) {
            g_prof.ms[std::get<0>(t)] += ms;
            g_prof.n[std::get<0>(t)] += (uint64_t)std::get<3>(t);
        }
        cudaGetLastError();
        g_prof.pool.push_back(std::get<1>(t));
        g_prof.pool.push_back(std::get<2>(t));
    }
    g_prof.pending.clear();
}

// bytes moved between host and device by the last completed call
static thread_local uint64_t g_h2d = 0, g_d2h = 0;


static void host_neumaier_add(double& s, double& c, double x)
{
    const double t = s + x;
    if (std::fabs(s) >= std::fabs(x)) c += (s - t) + x;
    else c += (x - t) + s;
    s = t;
}

static int fail(int code, const std::string& msg)
{
    g_err = msg;
    return code;
}

#define RBG_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess) {                                                                \
            cudaGetLastError();                                                                 \
            return fail(RBG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));      \
        }                                                                                       \
    } while (0)

// Grow-only device buffer.
struct DevBuf {
    void* p = nullptr;
    size_t n = 0;
    int ensure(size_t bytes)
    {
        if (bytes <= n) return 0;
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        size_t want = std::max(bytes, (size_t)256);
        if (cudaMalloc(&p, want) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        n = want;
        return 0;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    template <class T>
    T* as() const { return (T*)p; }
};

// Grow-only pinned host buffer (results read back after a call's one wait).
struct PinBuf {
    void* p = nullptr;
    size_t n = 0;
    int ensure(size_t bytes)
    {
        if (bytes <= n) return 0;
        release();
        const size_t want = std::max(bytes, (size_t)4096);
        if (cudaMallocHost(&p, want) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            return -1;
        }
        n = want;
        return 0;
    }
    void release()
    {
        if (p) cudaFreeHost(p);
        p = nullptr;
        n = 0;
    }
};

// Device views of the FP64 tables of one call (pointers into Ctx::tabs).
struct TableSet {
    Fp64Tables t{};
    const double* Tvals = nullptr;
    const X64Vol* xvols = nullptr;  // fixed-point path pass only
    const X64Group* xgrps = nullptr;
    const uint64_t* xcomp = nullptr;
    const int64_t* xgam = nullptr;
};

struct Ctx {
    int dev = -1;
    cudaStream_t stream = nullptr;
    std::mutex mu;
    DevBuf z, ivb, ivp, part, acc, tabs, res, pay, mixed_ws, cv, sobol, sobol32;
    // fixed-point FP64 path pass: digits of W1, X, and the Toeplitz panels of the tables in `tabs`
    DevBuf xdig, xbuf, xpan;
    PinBuf pin;
    cudaEvent_t digits_done = nullptr;  // the caller's normals of a batch are in xdig (payoffs_quadrature)
    bool xpan_ready = false;
    // host images of what `tabs`, `mixed_ws` and `sobol` hold, so that a call
    // with the same tables (a calibration loop, a benchmark) uploads nothing
    std::vector<unsigned char> tabs_img, mixed_img;
    std::vector<unsigned long long> sobol_img;
    std::vector<unsigned int> sobol32_img;
    // changes whenever tabs_img or mixed_img (what the device holds) changes
    uint64_t img_gen = 0;
    // The last plain mixed call (rbg_price_rt / rbg_price_mc): its inputs but
    // the seed, path offset and stream, and what they produced -- plan, job,
    // table pointers.  A call with the same inputs (another seed, another
    // shard) skips planning, table building and image comparison while the
    // device images are the ones it set up (img_gen).
    struct MixedCache {
        std::vector<unsigned char> key;
        Plan plan;
        MixedJob job;
        TableSet ts;
        uint64_t gen = ~0ull;
    } mcache;
    ~Ctx() {}
};

// One context per (device, caller stream): its own buffers, device tables,
// plan cache and lock, so calls on different streams run concurrently and
// only calls on one stream (which that stream orders anyway) wait for each
// other.  A NULL stream maps to a context with the library's own
// non-blocking stream.  Contexts live until the process exits.
static std::mutex g_ctx_mu;
static std::map<std::pair<int, void*>, std::unique_ptr<Ctx>> g_ctx;

static int get_ctx(Ctx** out, void* stream = nullptr)
{
    int dev = 0;
    RBG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_ctx_mu);
    auto& slot = g_ctx[{dev, stream}];
    if (!slot) {
        std::unique_ptr<Ctx> c(new Ctx());
        c->dev = dev;
        if (stream)
            c->stream = (cudaStream_t)stream;
        else
            RBG_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
        slot = std::move(c);
    }
    *out = slot.get();
    return RBG_OK;
}

// Every context of the current device (rbg_synchronize, rbg_release).
static int device_ctxs(std::vector<Ctx*>& out)
{
    int dev = 0;
    RBG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_ctx_mu);
    for (auto& kv : g_ctx)
        if (kv.first.first == dev) out.push_back(kv.second.get());
    return RBG_OK;
}

// The buffers only the digit convolution uses.  (cudaFree waits for work in flight.)
static void release_fixed(Ctx& c)
{
    for (DevBuf* b : {&c.xdig, &c.xbuf, &c.xpan}) b->release();
    c.xpan_ready = false;
}

// Grows one of the context's buffers.  The digit convolution's buffers, which an
// earlier call on the stream may have left, make room where there is none; a call
// therefore asks for what it cannot do without before it asks for those.
static int ensure(Ctx& c, DevBuf& b, size_t bytes, const char* what)
{
    if (!b.ensure(bytes)) return RBG_OK;
    release_fixed(c);
    if (b.ensure(bytes)) return fail(RBG_ERR_NOMEM, std::string("device allocation failed: ") + what);
    return RBG_OK;
}

// The digit convolution's buffers: digits, X (or sums), panels.  Without room for
// them the call goes on with the FP64 kernels, which need none of them.
static bool ensure_fixed(Ctx& c, size_t digits, size_t paths, size_t panels)
{
    if (c.xpan.n < panels) c.xpan_ready = false;
    if (!c.xdig.ensure(digits) && !c.xbuf.ensure(paths) && !c.xpan.ensure(panels)) return true;
    release_fixed(c);
    return false;
}

// ---------------------------------------------------------------- tables
static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// The FP64 form's Volterra backend for N steps: logL > 0 selects the FFT
// convolution (AUTO: from kFp64FftMinN steps), 0 the direct sum.
static int fp64_conv_log2(int conv, int N, int* logL)
{
    *logL = 0;
    if (conv == RBG_CONV_GEMM) return fail(RBG_ERR_UNSUPPORTED, "the FP64 form has no GEMM backend");
    if (conv == RBG_CONV_DIRECT) return RBG_OK;
    const int l = fp64_fft_log2_len(N);
    if (conv == RBG_CONV_FFT) {
        if (!l) return fail(RBG_ERR_UNSUPPORTED, "the FP64 FFT convolution needs 2 <= N <= 2048");
        *logL = l;
    } else if (N >= kFp64FftMinN) {
        *logL = l;
    }
    return RBG_OK;
}

// logL > 0: also the FP64 FFT convolution's spectra (one per distinct H) and
// twiddles; xt: also the fixed-point path pass's tables (fixed_panels builds their
// Toeplitz panels)
// fp64: the FP64 path kernels' Gamma and compensators too (the other path
// passes bring their own).
static int upload_tables(Ctx& c, const Plan& plan, cudaStream_t st, TableSet& ts, int logL = 0,
                         const X64Tables* xt = nullptr, bool fp64 = true)
{
    const int nv = (int)plan.vols.size(), ng = (int)plan.vgs.size(), no = (int)plan.outs.size(), N = plan.N;
    std::vector<VolDev> vols(nv);
    for (int v = 0; v < nv; ++v) vols[v] = VolDev{plan.vols[v].a1, plan.vols[v].a2, plan.vols[v].vg_begin, plan.vols[v].vg_end};
    std::vector<VGDev> vgs(ng);
    for (int g = 0; g < ng; ++g) {
        const VGroup& G = plan.vgs[g];
        vgs[g] = VGDev{G.scale, G.eta, G.dt, G.sdt, G.xi, G.nsteps, G.vol};
    }
    std::vector<OutDev> outs(no);
    std::vector<double> Tv(no);
    for (int i = 0; i < no; ++i) {
        outs[i] = OutDev{plan.outs[i].rho, plan.outs[i].K, plan.outs[i].vg, 0};
        Tv[i] = plan.outs[i].T;
    }
    size_t off_vols = 0;
    size_t off_vgs = align_up(off_vols + sizeof(VolDev) * nv, 256);
    size_t off_outs = align_up(off_vgs + sizeof(VGDev) * ng, 256);
    size_t off_T = align_up(off_outs + sizeof(OutDev) * no, 256);
    size_t off_gamma = align_up(off_T + sizeof(double) * no, 256);
    size_t off_comp = align_up(off_gamma + (fp64 ? sizeof(double) * plan.gamma.size() : 0), 256);
    const size_t L = logL > 0 ? (size_t)1 << logL : 0;
    size_t off_spec = align_up(off_comp + (fp64 ? sizeof(double) * plan.comp.size() : 0), 256);
    size_t off_tw = align_up(off_spec + 2 * sizeof(double) * L * nv, 256);
    size_t off_xvols = align_up(off_tw + 2 * sizeof(double) * L, 256);
    size_t off_xgrps = align_up(off_xvols + (xt ? sizeof(X64Vol) * nv : 0), 256);
    size_t off_xgam = align_up(off_xgrps + (xt ? sizeof(X64Group) * ng : 0), 256);
    size_t off_xcomp = align_up(off_xgam + (xt ? 8 * (size_t)nv * N : 0), 256);
    size_t total = align_up(off_xcomp + (xt ? 8 * (size_t)ng * N : 0), 256);
    std::vector<unsigned char> host(total, 0);
    if (xt) {
        std::memcpy(host.data() + off_xvols, xt->vols.data(), sizeof(X64Vol) * nv);
        std::memcpy(host.data() + off_xgrps, xt->grps.data(), sizeof(X64Group) * ng);
        std::memcpy(host.data() + off_xgam, xt->gam.data(), 8 * xt->gam.size());
        std::memcpy(host.data() + off_xcomp, xt->comp.data(), 8 * xt->comp.size());
    }
    if (logL > 0)
        fp64_fft_tables(plan.gamma.data(), nv, N, logL, (double*)(host.data() + off_spec),
                        (double*)(host.data() + off_tw));
    std::memcpy(host.data() + off_vols, vols.data(), sizeof(VolDev) * nv);
    std::memcpy(host.data() + off_vgs, vgs.data(), sizeof(VGDev) * ng);
    std::memcpy(host.data() + off_outs, outs.data(), sizeof(OutDev) * no);
    std::memcpy(host.data() + off_T, Tv.data(), sizeof(double) * no);
    if (fp64) {
        std::memcpy(host.data() + off_gamma, plan.gamma.data(), sizeof(double) * plan.gamma.size());
        std::memcpy(host.data() + off_comp, plan.comp.data(), sizeof(double) * plan.comp.size());
    }
    if (!(c.tabs.p && c.tabs_img == host)) {
        c.tabs_img.clear();
        c.xpan_ready = false;
        ++c.img_gen;
        int rc = ensure(c, c.tabs, total, "tables");
        if (rc) return rc;
        // a pageable source is staged before the call returns, so `host` may die
        RBG_CUDA(cudaMemcpyAsync(c.tabs.p, host.data(), total, cudaMemcpyHostToDevice, st));
        g_h2d += total;
        c.tabs_img.swap(host);
    }
    unsigned char* base = (unsigned char*)c.tabs.p;
    ts.t.vols = (const VolDev*)(base + off_vols);
    ts.t.vgs = (const VGDev*)(base + off_vgs);
    ts.t.outs = (const OutDev*)(base + off_outs);
    ts.t.gamma = fp64 ? (const double*)(base + off_gamma) : nullptr;
    ts.t.comp = fp64 ? (const double*)(base + off_comp) : nullptr;
    ts.t.spec = logL > 0 ? (const double2*)(base + off_spec) : nullptr;
    ts.t.tw = logL > 0 ? (const double2*)(base + off_tw) : nullptr;
    ts.t.logL = logL;
    ts.t.n_vol = nv;
    ts.t.n_vg = ng;
    ts.t.n_out = no;
    ts.t.N = N;
    ts.t.xi = plan.xi;
    ts.Tvals = (const double*)(base + off_T);
    if (xt) {
        ts.xvols = (const X64Vol*)(base + off_xvols);
        ts.xgrps = (const X64Group*)(base + off_xgrps);
        ts.xcomp = (const uint64_t*)(base + off_xcomp);
        ts.xgam = (const int64_t*)(base + off_xgam);
    }
    return RBG_OK;
}

// What the digit convolution holds beside the FP64 kernels' buffers: digits of a batch
// (16 bytes a path-step, within 2 GiB by the batch's size), X or the fused sums of vstep
// passes and their panels, each within 2 GiB.
constexpr int64_t kFixedBytes = (int64_t)1 << 31;
struct FixedPlan {
    int vstep = 1;       // passes a convolution launch
    size_t paths = 0;    // bytes of X or sums of vstep passes
    size_t panels = 0;   // bytes of panels: of every pass where that fits, else of vstep
    bool keep = false;   // every pass's panels, kept with the tables
};
// per: bytes of X or sums of one pass
static FixedPlan fixed_plan(int nv, int N, size_t per)
{
    const int64_t pan = (int64_t)x64_panel_bytes(N);
    FixedPlan f;
    f.keep = pan * nv <= kFixedBytes;
    f.vstep = (int)std::max<int64_t>(1, std::min({(int64_t)nv, kFixedBytes / (int64_t)per, kFixedBytes / pan}));
    f.paths = (size_t)f.vstep * per;
    f.panels = (size_t)(pan * (f.keep ? nv : f.vstep));
    return f;
}

// Panels of the passes v0 .. v0 + k - 1 of the tables in c.tabs, in c.xpan.
static const unsigned char* fixed_panels(Ctx& c, const TableSet& ts, const FixedPlan& f, int v0, int k, cudaStream_t st)
{
    unsigned char* at = c.xpan.as<unsigned char>();
    const int N = ts.t.N;
    if (!f.keep) {
        c.xpan_ready = false;
        launch_panels(ts.xgam + (size_t)v0 * N, k, N, at, st);
        return at;
    }
    if (!c.xpan_ready) launch_panels(ts.xgam, ts.t.n_vol, N, at, st);
    c.xpan_ready = true;
    return at + (size_t)v0 * x64_panel_bytes(N);
}

// ------------------------------------------------------------ FP64 form
uint64_t fold_seed(const uint64_t* seed, int seed_size)
{
    if (!seed || seed_size <= 0) return 0;
    uint64_t h = seed[0];
    for (int i = 1; i < seed_size; ++i) {
        uint64_t x = h + seed[i];
        x += 0x9E3779B97F4A7C15ull;
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        h = x ^ (x >> 31);
    }
    return h;
}

// SMs per device, looked up once per ordinal (the attribute query is cheap,
// but this runs on every call)
int device_sms()
{
    static std::mutex mu;
    static std::map<int, int> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(dev);
    if (it != cache.end()) return it->second;
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = 1;
    }
    cache[dev] = n;
    return n;
}

static int64_t fp64_batch(const Plan& plan, int64_t M, int ns = 2)
{
    // normals (8 ns N B/path) within 2 GiB, variance-path sums within 1 GiB
    int64_t by_z = ((int64_t)1 << 31) / (8 * ns * (int64_t)plan.N);
    int64_t by_iv = ((int64_t)1 << 30) / (8 * ns * (int64_t)std::max<size_t>(1, plan.vgs.size()));
    int64_t B = std::min(by_z, by_iv);
    B = std::max<int64_t>(256, B / 256 * 256);
    return std::min(B, M);
}

// The call's results (5 n_out doubles at c.res) and its kernel error word (err,
// or null) through pinned memory, with one wait; `what` names the kernels whose
// bounded waits the word reports.
static int read_back(Ctx& c, int no, const unsigned int* err, const char* what, cudaStream_t st, double* host_res)
{
    const size_t bytes = sizeof(double) * 5 * (size_t)no;
    if (c.pin.ensure(bytes + sizeof(double))) return fail(RBG_ERR_NOMEM, "pinned result buffer");
    unsigned int* word = (unsigned int*)c.pin.p;
    double* res = (double*)c.pin.p + 1;
    *word = 0;
    if (err) RBG_CUDA(cudaMemcpyAsync(word, err, sizeof *word, cudaMemcpyDeviceToHost, st));
    RBG_CUDA(cudaMemcpyAsync(res, c.res.p, bytes, cudaMemcpyDeviceToHost, st));
    RBG_CUDA(cudaStreamSynchronize(st));
    if (*word)
        return fail(RBG_ERR_TIMEOUT,
                    std::string(what) + ": a bounded pipeline wait expired (site " + std::to_string(*word) + ")");
    std::memcpy(host_res, res, bytes);
    g_d2h += bytes + (err ? sizeof *word : 0);
    prof_collect();
    return RBG_OK;
}

// mc: the plain Monte Carlo estimator (third normal stream Wperp, payoff
// max(S_T - K, 0)) instead of the Romano-Touzi conditional price.
// sobol_vt: Sobol' quasi-Monte Carlo normals (device direction table
// [kSobolBits][2N], path m takes point path_offset + m + 1; br: Brownian
// bridge or nullptr) instead of the Philox stream.  RT only.
static int price_fp64(Ctx& c, const Plan& plan, const rbg_options& o, int64_t M, cudaStream_t st,
                      double* host_res, bool mc, const unsigned long long* sobol_vt = nullptr,
                      const SobolBridge* br = nullptr)
{
    TableSet ts;
    int logL = 0;
    // Philox normals, no backend asked for: the exact tensor-core convolution and
    // fixed-point functions wherever the plan's numbers fit their ranges
    X64Tables xt;
    bool fixed = o.conv == RBG_CONV_AUTO && !sobol_vt && x64_prepare(plan, xt);
    int rc = fixed ? RBG_OK : fp64_conv_log2(o.conv, plan.N, &logL);
    if (rc) return rc;
    const int no = (int)plan.outs.size(), N = plan.N, ns = mc ? 3 : 2, nv = (int)plan.vols.size();
    const int64_t B = fp64_batch(plan, M, ns);
    if ((rc = ensure(c, c.z, sizeof(double) * ns * N * (size_t)B, "normals"))) return rc;
    if ((rc = ensure(c, c.ivb, sizeof(double) * 2 * plan.vgs.size() * (size_t)B, "variance sums"))) return rc;
    if (mc && (rc = ensure(c, c.ivp, sizeof(double) * plan.vgs.size() * (size_t)B, "variance sums"))) return rc;
    double* ivp = mc ? c.ivp.as<double>() : nullptr;
    // The variance pass inside the convolution's read-out for up to x64_fuse_groups
    // variance groups a pass, where its sums (one value per group, path and 32 steps)
    // stay within X's limit of 2 GiB for one pass.
    const size_t sums = (size_t)std::max(xt.max_groups, 1) * x64_slot_bytes(B, N, ns);
    const bool fused = xt.u53 && xt.max_groups <= x64_fuse_groups(ns) && sums <= ((size_t)1 << 31);
    const FixedPlan fp = fixed_plan(nv, N, fused ? sums : 8 * (size_t)N * (size_t)B);
    const int vstep = fp.vstep;
    const int G = payoff_paths_per_thread(B, device_sms());
    const int64_t max_chunks = (B + 256 * (int64_t)G - 1) / (256 * (int64_t)G);
    if ((rc = ensure(c, c.part, sizeof(double) * 4 * no * (size_t)max_chunks, "partials"))) return rc;
    // the kernel error word follows the accumulators
    if ((rc = ensure(c, c.acc, sizeof(double) * (4 * no + 1), "accumulators"))) return rc;
    if ((rc = ensure(c, c.res, sizeof(double) * 5 * no, "results"))) return rc;
    // what both forms need is there; without room for the rest of the digit
    // convolution's the FP64 kernels take the call
    if (fixed) {
        rc = upload_tables(c, plan, st, ts, 0, &xt, false);
        if (rc && rc != RBG_ERR_NOMEM) return rc;
        fixed = !rc && ensure_fixed(c, x64_digit_bytes(B, N), fp.paths, fp.panels);
    }
    if (!fixed) {
        if ((rc = fp64_conv_log2(o.conv, N, &logL))) return rc;
        if ((rc = upload_tables(c, plan, st, ts, logL))) return rc;
    }
    prof_path(!fixed ? (logL > 0 ? "k_path_fp64_fft" : "k_path_fp64")
                     : (fused ? "k_volterra_exact + k_slot_sums" : "k_volterra_exact + k_variance_fixed"));
    unsigned int* err = (unsigned int*)(c.acc.as<double>() + 4 * no);
    if (fixed) RBG_CUDA(cudaMemsetAsync(err, 0, sizeof(unsigned int), st));
    bool wide = true;
    const MergeFinal fin{ts.t.outs, ts.Tvals, c.res.as<double>(), M, o.compute_iv};
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        {
            ProfScope ps(kStageNormals, st);
            if (sobol_vt) {
                if (launch_sobol_normals(sobol_vt, N, (uint64_t)(o.path_offset + m0 + 1), b, br, c.z.as<double>(), st))
                    return fail(RBG_ERR_UNSUPPORTED, "Brownian bridge shared memory not available for this N");
            } else if (launch_normals_fixed(o.seed, o.path_offset + m0, b, N, o.normals == RBG_NORMALS_F32,
                                            c.z.as<double>(), fixed ? c.xdig.as<unsigned char>() : nullptr,
                                            !fixed ? 0 : (fused ? kFixAll : kFixW1perp), ns, st)) {
                return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
            }
        }
        if (fixed && m0 == 0) wide = x64_wide(xt, N);
        {
            ProfScope ps(kStagePathFp64, st, fixed ? 2 * ((nv + vstep - 1) / vstep) : 1);
            if (!fixed) launch_path_fp64(ts.t, c.z.as<double>(), b, c.ivb.as<double>(), st, ivp);
            for (int v0 = 0; fixed && v0 < nv; v0 += vstep) {
                const int k = std::min(vstep, nv - v0);
                const unsigned char* pan = fixed_panels(c, ts, fp, v0, k, st);
                if (fused) {
                    const int g0 = plan.vols[v0].vg_begin, ng = plan.vols[v0 + k - 1].vg_end - g0;
                    if (launch_volterra_variance(c.xdig.as<unsigned char>(), pan, ts.xvols + v0, ts.xgrps, ts.xcomp,
                                                 c.z.as<double>(), k, g0, ng, ns, wide, N, b, c.xbuf.as<double>(),
                                                 c.ivb.as<double>(), ivp, err, st))
                        return fail(RBG_ERR_CUDA, "FP64 path kernels could not be configured");
                } else if (launch_volterra_exact(c.xdig.as<unsigned char>(), pan, ts.xvols + v0, k, N, b, false, wide,
                                                 c.xbuf.as<uint64_t>(), err, st) ||
                           launch_variance_fixed(ts.xvols + v0, ts.xgrps, ts.xcomp, c.z.as<double>(),
                                                 c.xbuf.as<uint64_t>(), k, xt.max_groups, xt.u53, false, ns, N, b,
                                                 c.ivb.as<double>(), ivp, st)) {
                    return fail(RBG_ERR_CUDA, "FP64 path kernels could not be configured");
                }
            }
        }
        const int nchunks = (int)((b + 256 * (int64_t)G - 1) / (256 * (int64_t)G));
        {
            ProfScope ps(kStagePayoff, st);
            if (launch_payoff_sums(ts.t, c.ivb.as<double>(), b, b, G, c.part.as<double>(), nchunks, st, ivp))
                return fail(RBG_ERR_CUDA, "FP64 payoff kernel could not be configured");
        }
        {
            ProfScope ps(kStageReduce, st);
            if (launch_merge(c.part.as<double>(), nchunks, no, c.acc.as<double>(), m0 == 0, st,
                             m0 + B >= M ? &fin : nullptr))
                return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
        }
        RBG_CUDA(cudaGetLastError());
    }
    return read_back(c, no, fixed ? err : nullptr, "FP64 convolution", st, host_res);
}

// Sobol' normals materialized per batch on the device and read by the mixed
// path kernel as caller normals (quadrature layout): the mixed form's QMC
// where its GEMM producer cannot draw the points itself -- the Brownian
// bridge (each bridged step needs the whole point), the FFT backend, and
// more than 1024 steps (multi-pass tiles redraw earlier chunks).
struct SobolZ {
    const unsigned long long* vt;  // FP64 direction table [62][2N] on the device
    const SobolBridge* br;         // null: no bridge; FP32 quantile (the GEMM producer's normals), FP32 bridge
    int64_t path_offset;
};

// Setup of a mixed call: the FP64 tables and the job's workspace image on
// the device, every buffer the run needs.
static int mixed_setup(Ctx& c, const Plan& plan, const rbg_options& o, int64_t M, cudaStream_t st, bool mc,
                       const unsigned int* sob, const SobolZ* sz, TableSet& ts, MixedJob& job)
{
    int rc = upload_tables(c, plan, st, ts, 0, nullptr, false);
    if (rc) return rc;
    const int no = (int)plan.outs.size();
    // materialized normals: 2 N doubles per path, at most 2 GiB per batch
    const int64_t zcap = sz ? std::max<int64_t>(256, ((int64_t)1 << 31) / (16 * (int64_t)plan.N)) : 0;
    if ((rc = mixed_prepare(plan, o, M, job, g_err, zcap, mc))) return rc;
    job.sob = sob;
    if (sob && (job.backend != RBG_CONV_GEMM || plan.N > 1024))
        return fail(RBG_ERR_UNSUPPORTED, "Sobol' normals in the mixed form need the GEMM backend and N <= 1024");
    const int64_t B = job.batch;
    if (sz && (rc = ensure(c, c.z, sizeof(double) * 2 * plan.N * (size_t)B, "normals"))) return rc;
    if ((rc = ensure(c, c.mixed_ws, job.workspace_bytes, "mixed workspace"))) return rc;
    const int G = payoff_paths_per_thread(B, job.sms);
    const int64_t max_chunks = job.fused ? mixed_part_rows(job, B) : (B + 256 * (int64_t)G - 1) / (256 * (int64_t)G);
    if (!job.fused && (rc = ensure(c, c.ivb, sizeof(float) * 2 * plan.vgs.size() * (size_t)B, "variance sums")))
        return rc;
    if (mc && (rc = ensure(c, c.ivp, sizeof(float) * plan.vgs.size() * (size_t)B, "variance sums"))) return rc;
    if ((rc = ensure(c, c.part, sizeof(double) * 4 * no * (size_t)max_chunks, "partials"))) return rc;
    if ((rc = ensure(c, c.acc, sizeof(double) * 4 * no, "accumulators"))) return rc;
    if ((rc = ensure(c, c.res, sizeof(double) * 5 * no, "results"))) return rc;
    if (c.mixed_img != job.host_ws) {
        c.mixed_img.clear();
        ++c.img_gen;
        if ((rc = mixed_upload(job, c.mixed_ws.p, st, g_err))) return rc;
        g_h2d += job.host_ws.size();
        c.mixed_img = job.host_ws;
    }
    return RBG_OK;
}

// Run of a prepared mixed call: path kernels, payoff sums, merges, finalize.
static int mixed_run(Ctx& c, const Plan& plan, const TableSet& ts, const MixedJob& job, const rbg_options& o,
                     int64_t M, cudaStream_t st, double* host_res, bool mc, const SobolZ* sz)
{
    int rc = RBG_OK;
    const int no = (int)plan.outs.size();
    const int64_t B = job.batch;
    const int G = payoff_paths_per_thread(B, job.sms);
    const double* zext = sz ? c.z.as<double>() : nullptr;
    float* ivq = mc ? c.ivp.as<float>() : nullptr;
    RBG_CUDA(cudaMemsetAsync((unsigned char*)c.mixed_ws.p + job.off_err, 0, 4, st));  // the kernel error word
    const MergeFinal fin{ts.t.outs, ts.Tvals, c.res.as<double>(), M, o.compute_iv};
    auto merge = [&](int rows, int64_t m0) {
        return launch_merge(c.part.as<double>(), rows, no, c.acc.as<double>(), m0 == 0, st, m0 + B >= M ? &fin : nullptr)
                   ? fail(RBG_ERR_CUDA, "fixed-point tables not found on the device")
                   : RBG_OK;
    };
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        if (sz) {
            ProfScope ps(kStageNormals, st);
            if (launch_sobol_normals(sz->vt, plan.N, (uint64_t)(sz->path_offset + m0 + 1), b, sz->br, c.z.as<double>(),
                                     st, 1))
                return fail(RBG_ERR_UNSUPPORTED, "Brownian bridge shared memory not available for this N");
        }
        if (job.fused) {
            // payoffs summed inside the path kernel: one partial row per CTA
            const int rows = mixed_part_rows(job, b);
            RBG_CUDA(cudaMemsetAsync(c.part.p, 0, sizeof(double) * 4 * no * (size_t)rows, st));
            {
                ProfScope ps(kStageMixed, st, (int)job.launches.size());
                if ((rc = mixed_launch(job, c.mixed_ws.p, o.seed, o.path_offset + m0, b, nullptr, st, g_err, nullptr,
                                       nullptr, c.part.as<double>(), nullptr, nullptr, zext)))
                    return rc;
            }
            ProfScope ps(kStageReduce, st);
            if ((rc = merge(rows, m0))) return rc;
        } else {
            {
                ProfScope ps(kStageMixed, st, (int)job.launches.size());
                if ((rc = mixed_launch(job, c.mixed_ws.p, o.seed, o.path_offset + m0, b, c.ivb.p, st, g_err, nullptr,
                                       nullptr, nullptr, nullptr, ivq, zext)))
                    return rc;
            }
            const int nchunks = (int)((b + 256 * (int64_t)G - 1) / (256 * (int64_t)G));
            {
                ProfScope ps(kStagePayoff, st);
                launch_payoff_sums_f32(ts.t.outs, no, c.ivb.p, b, G, c.part.as<double>(), nchunks, st, ivq);
            }
            {
                ProfScope ps(kStageReduce, st);
                if ((rc = merge(nchunks, m0))) return rc;
            }
        }
        RBG_CUDA(cudaGetLastError());
    }
    // one wait for the whole call: the kernel error word is read with the results
    // (finalizing the sums of a launch that gave up is harmless; its results are
    // discarded)
    return read_back(c, no, (const unsigned int*)((unsigned char*)c.mixed_ws.p + job.off_err), "mixed kernel", st, host_res);
}

// Mixed form: tcgen05 fused path kernel writes FP32 (Ivdt, IsvdW) per
// (variance group, path); the FP64 payoff/sum kernels finish.
// sob: Sobol' normals (device table [32][2N], bits 30..61 of the direction
// integers; GEMM backend, RT) instead of the Philox stream; sz: Sobol'
// normals materialized per batch instead.
static int price_mixed(Ctx& c, const Plan& plan, const rbg_options& o, int64_t M, cudaStream_t st,
                       double* host_res, bool mc = false, const unsigned int* sob = nullptr,
                       const SobolZ* sz = nullptr)
{
    TableSet ts;
    MixedJob job;
    int rc = mixed_setup(c, plan, o, M, st, mc, sob, sz, ts, job);
    if (rc) return rc;
    return mixed_run(c, plan, ts, job, o, M, st, host_res, mc, sz);
}

static int price_plan(const Plan& plan, int64_t M, const rbg_options* o, std::vector<double>& res, bool mc = false)
{
    Ctx* c = nullptr;
    int rc = get_ctx(&c, o->stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = o->stream ? (cudaStream_t)o->stream : c->stream;
    res.assign(5 * plan.outs.size(), 0.0);
    if (o->precision == RBG_FP64) return price_fp64(*c, plan, *o, M, st, res.data(), mc);
    if (o->precision == RBG_MIXED) return price_mixed(*c, plan, *o, M, st, res.data(), mc);
    return fail(RBG_ERR_ARG, "unknown precision");
}

// The inputs of a plain mixed call that its plan and job depend on: all but
// the seed, the path offset and the stream.
static std::vector<unsigned char> mixed_key(const rbg_params& p, const rbg_options& o, bool mc)
{
    std::vector<unsigned char> k;
    auto put = [&k](const void* x, size_t n) {
        const unsigned char* b = (const unsigned char*)x;
        k.insert(k.end(), b, b + n);
    };
    const int hdr[7] = {p.par_size, p.op_size, p.N, o.precision, o.conv, o.split, (o.compute_iv ? 1 : 0) | (mc ? 2 : 0)};
    put(hdr, sizeof hdr);
    put(&p.xi, sizeof p.xi);
    put(&p.M, sizeof p.M);
    if (p.par_size > 0 && p.H && p.eta && p.rho) {
        put(p.H, sizeof(double) * p.par_size);
        put(p.eta, sizeof(double) * p.par_size);
        put(p.rho, sizeof(double) * p.par_size);
    }
    if (p.op_size > 0 && p.T && p.K) {
        put(p.T, sizeof(double) * p.op_size);
        put(p.K, sizeof(double) * p.op_size);
    }
    return k;
}

// A plain mixed call (Philox normals), through the per-context cache.
static int price_mixed_cached(const rbg_params& p, const rbg_options& o, std::vector<double>& res, bool mc)
{
    Ctx* c = nullptr;
    int rc = get_ctx(&c, o.stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = o.stream ? (cudaStream_t)o.stream : c->stream;
    std::vector<unsigned char> key = mixed_key(p, o, mc);
    Ctx::MixedCache& mcache = c->mcache;
    if (mcache.gen == c->img_gen && mcache.key == key) {
        res.assign(5 * mcache.plan.outs.size(), 0.0);
        return mixed_run(*c, mcache.plan, mcache.ts, mcache.job, o, p.M, st, res.data(), mc, nullptr);
    }
    mcache.gen = ~0ull;
    Plan plan;
    std::string err;
    if (!build_plan(p, plan, err, mc)) return fail(RBG_ERR_ARG, err);
    TableSet ts;
    MixedJob job;
    if ((rc = mixed_setup(*c, plan, o, p.M, st, mc, nullptr, nullptr, ts, job))) return rc;
    res.assign(5 * plan.outs.size(), 0.0);
    mcache.key.swap(key);
    mcache.plan = std::move(plan);
    mcache.job = std::move(job);
    mcache.ts = ts;
    mcache.gen = c->img_gen;
    return mixed_run(*c, mcache.plan, mcache.ts, mcache.job, o, p.M, st, res.data(), mc, nullptr);
}

static int price_any(const rbg_params* p, const rbg_options* o, std::vector<double>& res, bool mc = false)
{
    if (!p || !o) return fail(RBG_ERR_ARG, "null params/options");
    g_h2d = g_d2h = 0;
    if (o->precision == RBG_MIXED) return price_mixed_cached(*p, *o, res, mc);
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err, mc)) return fail(RBG_ERR_ARG, err);
    return price_plan(plan, p->M, o, res, mc);
}

// Control-variate Romano-Touzi estimator (ML_console_ST), FP64.  Zc / Z: host
// normals, or null for the Philox stream (pilot paths 2^62 + path_offset + m).
static const int64_t kCvPilotPath0 = (int64_t)1 << 62;

static int price_cv(Ctx& c, const Plan& plan, const rbg_cv_params& p, const rbg_options& o, const double* Zc,
                    const double* Z, cudaStream_t st, double* host_res)
{
    TableSet ts;
    int logL = 0;
    int rc = fp64_conv_log2(o.conv, plan.N, &logL);
    if (rc) return rc;
    if ((rc = upload_tables(c, plan, st, ts, logL))) return rc;
    const int no = (int)plan.outs.size(), N = plan.N, ng = (int)plan.vgs.size();
    const int64_t Mc = p.M_control, M = p.M;
    const int64_t B = fp64_batch(plan, M, 4);  // normals plus two (Ivdt, IsvdW) sets per path
    if (Mc > fp64_batch(plan, Mc, 2)) return fail(RBG_ERR_ARG, "M_control too large for one pilot batch");
    const int64_t zpaths = std::max(B, Mc);
    if ((rc = ensure(c, c.z, sizeof(double) * 2 * N * (size_t)zpaths, "normals"))) return rc;
    if ((rc = ensure(c, c.ivb, sizeof(double) * 2 * ng * (size_t)zpaths, "variance sums"))) return rc;
    if ((rc = ensure(c, c.ivp, sizeof(double) * 2 * ng * (size_t)B, "antithetic sums"))) return rc;
    const size_t cv_bytes = sizeof(double) * (size_t)no * (2 * (size_t)Mc + 2) + sizeof(unsigned long long) * no;
    if ((rc = ensure(c, c.cv, cv_bytes, "control-variate scratch"))) return rc;
    double* alpha = c.cv.as<double>();
    double* Q = alpha + no;
    unsigned long long* count = (unsigned long long*)(Q + no);
    double* xy = (double*)(count + no);
    const int G = payoff_paths_per_thread(B, device_sms());
    const int64_t max_chunks = (B + 256 * (int64_t)G - 1) / (256 * (int64_t)G);
    if ((rc = ensure(c, c.part, sizeof(double) * 4 * no * (size_t)max_chunks, "partials"))) return rc;
    if ((rc = ensure(c, c.acc, sizeof(double) * 4 * no, "accumulators"))) return rc;
    if ((rc = ensure(c, c.res, sizeof(double) * 5 * no, "results"))) return rc;
    // pilot: one batch of Mc paths
    if (Zc) {
        RBG_CUDA(cudaMemcpyAsync(c.z.p, Zc, sizeof(double) * 2 * N * Mc, cudaMemcpyHostToDevice, st));
    } else {
        if (launch_normals_fixed(o.seed, kCvPilotPath0 + o.path_offset, Mc, N, o.normals == RBG_NORMALS_F32,
                                 c.z.as<double>(), nullptr, 0, 2, st))
            return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
    }
    launch_path_fp64(ts.t, c.z.as<double>(), Mc, c.ivb.as<double>(), st);
    launch_cv_pilot(ts.t, c.ivb.as<double>(), Mc, xy, alpha, Q, st);
    RBG_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned long long) * no, st));
    // main paths, antithetic pairs
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        if (Z) {
            RBG_CUDA(cudaMemcpyAsync(c.z.p, Z + (size_t)m0 * 2 * N, sizeof(double) * 2 * N * b, cudaMemcpyHostToDevice,
                                     st));
        } else {
            if (launch_normals_fixed(o.seed, o.path_offset + m0, b, N, o.normals == RBG_NORMALS_F32, c.z.as<double>(),
                                     nullptr, 0, 2, st))
                return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
        }
        launch_path_fp64(ts.t, c.z.as<double>(), b, c.ivb.as<double>(), st, nullptr, c.ivp.as<double>());
        const int nchunks = (int)((b + 256 * (int64_t)G - 1) / (256 * (int64_t)G));
        launch_payoff_sums_cv(ts.t, c.ivb.as<double>(), c.ivp.as<double>(), b, alpha, Q, p.Q_max, G,
                              c.part.as<double>(), count, nchunks, st);
        if (launch_merge(c.part.as<double>(), nchunks, no, c.acc.as<double>(), m0 == 0, st))
            return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
        RBG_CUDA(cudaGetLastError());
    }
    if (launch_finalize_cv(c.acc.as<double>(), no, M, ts.t.outs, ts.Tvals, alpha, Q, count, p.Q_max, o.compute_iv,
                           c.res.as<double>(), st))
        return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
    RBG_CUDA(cudaGetLastError());
    RBG_CUDA(cudaMemcpyAsync(host_res, c.res.p, sizeof(double) * 5 * no, cudaMemcpyDeviceToHost, st));
    RBG_CUDA(cudaStreamSynchronize(st));
    return RBG_OK;
}

// Control-variate estimator in the mixed form: the pilot in FP64 on the
// mixed form's FP32 normals (the same alpha and Q as the FP64 form with
// RBG_NORMALS_F32), the main paths through the tensor-core path kernel twice
// per batch -- as is, then with the variance exponent's coefficient negated,
// which prices the antithetic paths -W exactly -- with xi = 0 in the kernel's
// final sums, since each tuple carries its own xi (added back per group by the
// FP32 control-variate payoff kernel).
static int price_cv_mixed(Ctx& c, const Plan& plan, const rbg_cv_params& p, const rbg_options& o, cudaStream_t st,
                          double* host_res)
{
    TableSet ts;
    int logL = 0;
    int rc = fp64_conv_log2(RBG_CONV_AUTO, plan.N, &logL);
    if (rc) return rc;
    if ((rc = upload_tables(c, plan, st, ts, logL))) return rc;
    const int no = (int)plan.outs.size(), N = plan.N, ng = (int)plan.vgs.size();
    const int64_t Mc = p.M_control, M = p.M;
    if (Mc > fp64_batch(plan, Mc, 2)) return fail(RBG_ERR_ARG, "M_control too large for one pilot batch");
    MixedJob job;
    if ((rc = mixed_prepare(plan, o, M, job, g_err, 0, false))) return rc;
    if (job.fused) return fail(RBG_ERR_UNSUPPORTED, "the control-variate estimator needs the unfused path kernel");
    const int64_t B = job.batch;
    const int G = payoff_paths_per_thread(B, job.sms);
    const int64_t max_chunks = (B + 256 * (int64_t)G - 1) / (256 * (int64_t)G);
    if ((rc = ensure(c, c.z, sizeof(double) * 2 * N * (size_t)Mc, "pilot normals"))) return rc;
    if ((rc = ensure(c, c.ivp, sizeof(double) * 2 * ng * (size_t)Mc, "pilot sums"))) return rc;
    if ((rc = ensure(c, c.ivb, sizeof(float) * 4 * ng * (size_t)B, "variance sums"))) return rc;
    const size_t cv_bytes = sizeof(double) * (size_t)no * (2 * (size_t)Mc + 2) + sizeof(unsigned long long) * no;
    if ((rc = ensure(c, c.cv, cv_bytes, "control-variate scratch"))) return rc;
    if ((rc = ensure(c, c.mixed_ws, job.workspace_bytes, "mixed workspace"))) return rc;
    if ((rc = ensure(c, c.part, sizeof(double) * 4 * no * (size_t)max_chunks, "partials"))) return rc;
    if ((rc = ensure(c, c.acc, sizeof(double) * 4 * no, "accumulators"))) return rc;
    if ((rc = ensure(c, c.res, sizeof(double) * 5 * no, "results"))) return rc;
    double* alpha = c.cv.as<double>();
    double* Q = alpha + no;
    unsigned long long* count = (unsigned long long*)(Q + no);
    double* xy = (double*)(count + no);
    // pilot: one FP64 batch of Mc paths on FP32 normals
    if (launch_normals_fixed(o.seed, kCvPilotPath0 + o.path_offset, Mc, N, 1, c.z.as<double>(), nullptr, 0, 2, st))
        return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
    launch_path_fp64(ts.t, c.z.as<double>(), Mc, c.ivp.as<double>(), st);
    launch_cv_pilot(ts.t, c.ivp.as<double>(), Mc, xy, alpha, Q, st);
    RBG_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned long long) * no, st));
    // main paths: the job as is and its antithetic twin, both with xi = 0 in the final sums
    for (MixedLaunch& L : job.launches) L.args.xi = L.args.sqrt_xi = 0.f;
    MixedJob anti = job;
    for (MixedLaunch& L : anti.launches)
        for (int g = 0; g < L.args.n_g; ++g) L.args.alpha[g] = -L.args.alpha[g];
    if (c.mixed_img != job.host_ws) {
        c.mixed_img.clear();
        ++c.img_gen;
        if ((rc = mixed_upload(job, c.mixed_ws.p, st, g_err))) return rc;
        c.mixed_img = job.host_ws;
    } else {
        RBG_CUDA(cudaMemsetAsync((unsigned char*)c.mixed_ws.p + job.off_err, 0, 4, st));
    }
    float2* ivb = c.ivb.as<float2>();
    float2* ivn = ivb + (size_t)ng * B;
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        {
            ProfScope ps(kStageMixed, st, 2 * (int)job.launches.size());
            if ((rc = mixed_launch(job, c.mixed_ws.p, o.seed, o.path_offset + m0, b, ivb, st, g_err))) return rc;
            if ((rc = mixed_launch(anti, c.mixed_ws.p, o.seed, o.path_offset + m0, b, ivn, st, g_err))) return rc;
        }
        const int nchunks = (int)((b + 256 * (int64_t)G - 1) / (256 * (int64_t)G));
        {
            ProfScope ps(kStagePayoff, st);
            launch_payoff_sums_cv_f32(ts.t.outs, ts.t.vgs, no, ivb, ivn, b, G, o.seed, o.path_offset + m0, alpha, Q,
                                      p.Q_max, c.part.as<double>(), count, nchunks, st);
        }
        {
            ProfScope ps(kStageReduce, st);
            if (launch_merge(c.part.as<double>(), nchunks, no, c.acc.as<double>(), m0 == 0, st))
                return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
        }
        RBG_CUDA(cudaGetLastError());
    }
    if (launch_finalize_cv(c.acc.as<double>(), no, M, ts.t.outs, ts.Tvals, alpha, Q, count, p.Q_max, o.compute_iv,
                           c.res.as<double>(), st))
        return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
    RBG_CUDA(cudaGetLastError());
    if ((rc = mixed_check(job, c.mixed_ws.p, st, g_err))) return rc;
    RBG_CUDA(cudaMemcpyAsync(host_res, c.res.p, sizeof(double) * 5 * no, cudaMemcpyDeviceToHost, st));
    RBG_CUDA(cudaStreamSynchronize(st));
    prof_collect();
    return RBG_OK;
}

static int price_cv_any(const rbg_cv_params* p, const rbg_options* o, const double* Zc, const double* Z,
                        std::vector<double>& res)
{
    if (!p || !o) return fail(RBG_ERR_ARG, "null params/options");
    if (!p->xi) return fail(RBG_ERR_ARG, "null xi array");
    if (p->M_control < 2) return fail(RBG_ERR_ARG, "M_control must be >= 2");
    if (o->precision != RBG_FP64 && o->precision != RBG_MIXED) return fail(RBG_ERR_ARG, "unknown precision");
    if (o->precision == RBG_MIXED && (Zc || Z))
        return fail(RBG_ERR_UNSUPPORTED, "the control-variate estimator on caller normals runs in FP64");
    g_h2d = g_d2h = 0;
    rbg_unordered u{p->xi[0], p->H, p->eta, p->rho, p->T, p->K, p->size, p->N, p->M};
    Plan plan;
    std::string err;
    if (p->size > 0 && !build_plan_unordered(u, plan, err, p->xi, 1)) return fail(RBG_ERR_ARG, err);
    if (p->size <= 0) return fail(RBG_ERR_ARG, "size must be positive");
    Ctx* c = nullptr;
    int rc = get_ctx(&c, o->stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = o->stream ? (cudaStream_t)o->stream : c->stream;
    res.assign(5 * plan.outs.size(), 0.0);
    if (o->precision == RBG_MIXED) return price_cv_mixed(*c, plan, *p, *o, st, res.data());
    return price_cv(*c, plan, *p, *o, Zc, Z, st, res.data());
}

// Whether a quadrature call of M paths goes through the digit convolution, by the two
// forms' times in microseconds beyond what they share, fitted to 478 calls on device
// pointers (1 to 4096 steps, 1 to 16000 paths, 1 to 1000 H, 1 to 8 groups each; the choice costs
// 0.4 % of the better form on average, at most 20 %).
// FP64 kernel: one launch.  The paths the chip holds at once take the time of one, half the
// steps (direct sum, steps rounded to 32) or a transform (FFT of L points, L / 2 steps) a
// pass and step; the FP64 pipe, 6.1e11 operations a second, takes the rest.
// Digits: four launches, then for each pass the blocks of 128 steps of a path group
// one after the other, with 64 and with 256 paths at full weight.
// Digits against FP64 kernel: 64 steps, 2000 paths 84 / 64 us, 8000 paths 87 / 120; 100
// steps, 1000 paths 98 / 68, 4000 paths 101 / 151; 512 steps, 256 paths 203 / 146, 1000 paths
// 202 / 239; 2048 steps, 1 path 301 / 508; 4096 steps, 1 path 530 / 10900; 100 H of
// 100 steps, 64 paths 1670 / 3070.
static bool quadrature_by_digits(const Plan& plan, int64_t M, int ns, int logL)
{
    const double N = plan.N, nv = (double)plan.vols.size(), ng = (double)plan.vgs.size(), m = (double)M;
    const double up = (plan.N + 31) / 32 * 32, group = ns == 3 ? 60.0 : 44.0;
    double one, rest;
    if (logL > 0) {
        const double s = (double)(1 << (logL - 1));
        one = s * (0.05 + 0.15 * nv + 0.02 * ng);
        rest = std::max(0.0, m - 200.0) * s * (24.0 + 50.0 * nv + group * ng);
    } else {
        one = nv * (2.0 + 0.0011 * up * up) + 0.075 * ng * up;
        rest = std::max(0.0, m - 1216.0) * up * (nv * (0.5 * N + 32.0) + group * ng);
    }
    const double a = std::min(1.0, m / 64.0), b = std::min(1.0, m / 256.0);
    const double digits = 34.0 + N * (0.05 + 0.03 * a) + nv * (2.0 + 3.0 * a + N * (0.04 + 0.09 * a + 0.05 * b)) + (ng - nv) +
                          m * N * (2.3e-5 * nv + 4e-6 * ng);
    return digits < one + rest / 6.1e5;
}

static int payoffs_quadrature(const rbg_params* p, const double* Z, double* payoff, int device_ptrs,
                              cudaStream_t user_stream, bool mc = false, int conv = RBG_CONV_AUTO)
{
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err, mc)) return fail(RBG_ERR_ARG, err);
    if (!Z || !payoff) return fail(RBG_ERR_ARG, "null Z/payoff");
    Ctx* c = nullptr;
    int rc = get_ctx(&c, user_stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = user_stream ? user_stream : c->stream;
    TableSet ts;
    int logL = 0;
    // no backend asked for, and paths enough: the exact tensor-core convolution and
    // fixed-point functions; a batch with normals outside their range takes the FP64 kernels
    X64Tables xt;
    if ((rc = fp64_conv_log2(conv, plan.N, &logL))) return rc;
    const int no = (int)plan.outs.size(), N = plan.N, ns = mc ? 3 : 2, nv = (int)plan.vols.size();
    const int64_t M = p->M;
    bool fixed = conv == RBG_CONV_AUTO && quadrature_by_digits(plan, M, ns, logL) && x64_prepare(plan, xt, true);
    int64_t B = fp64_batch(plan, M, ns);
    // payoffs of a batch within 1 GiB too
    B = std::min<int64_t>(B, std::max<int64_t>(256, ((int64_t)1 << 30) / (8 * (int64_t)no)));
    const FixedPlan fp = fixed_plan(nv, N, 8 * (size_t)N * (size_t)B);
    const int vstep = fp.vstep;
    if ((rc = ensure(*c, c->ivb, sizeof(double) * 2 * plan.vgs.size() * (size_t)B, "variance sums"))) return rc;
    if (mc && (rc = ensure(*c, c->ivp, sizeof(double) * plan.vgs.size() * (size_t)B, "variance sums"))) return rc;
    double* ivp = mc ? c->ivp.as<double>() : nullptr;
    if (!device_ptrs) {
        if ((rc = ensure(*c, c->z, sizeof(double) * ns * N * (size_t)B, "normals"))) return rc;
        if ((rc = ensure(*c, c->pay, sizeof(double) * no * (size_t)B, "payoffs"))) return rc;
    }
    // device words: kernel error, normals out of range; read through pinned memory
    if ((rc = ensure(*c, c->acc, 2 * sizeof(unsigned int), "accumulators"))) return rc;
    // without room for the digit convolution's buffers the FP64 kernels take the call;
    // beside it their own tables wait for a batch that needs them
    if (fixed) {
        rc = upload_tables(*c, plan, st, ts, 0, &xt, false);
        if (rc && rc != RBG_ERR_NOMEM) return rc;
        fixed = !rc && ensure_fixed(*c, x64_digit_bytes(B, N), fp.paths, fp.panels);
    }
    if (!fixed && (rc = upload_tables(*c, plan, st, ts, logL))) return rc;
    bool fp64_tables = !fixed;
    unsigned int* words = c->acc.as<unsigned int>();
    volatile unsigned int* seen = nullptr;
    if (fixed) {
        if (c->pin.ensure(2 * sizeof(unsigned int))) return fail(RBG_ERR_NOMEM, "pinned result buffer");
        seen = (unsigned int*)c->pin.p;
        if (!c->digits_done) RBG_CUDA(cudaEventCreateWithFlags(&c->digits_done, cudaEventDisableTiming));
        RBG_CUDA(cudaMemsetAsync(words, 0, 2 * sizeof(unsigned int), st));
    }
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        const double* Zd;
        double* Pd;
        if (device_ptrs) {
            Zd = Z + m0 * ns * N;
            Pd = payoff + m0 * no;
        } else {
            RBG_CUDA(cudaMemcpyAsync(c->z.p, Z + m0 * ns * N, sizeof(double) * ns * N * b, cudaMemcpyHostToDevice,
                                     st));
            Zd = c->z.as<double>();
            Pd = c->pay.as<double>();
        }
        if (fixed) {
            if (m0) RBG_CUDA(cudaMemsetAsync(words + 1, 0, sizeof(unsigned int), st));
            launch_digits(Zd, b, N, ns, c->xdig.as<unsigned char>(), words + 1, st);
            RBG_CUDA(cudaMemcpyAsync((void*)(seen + 1), words + 1, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
            RBG_CUDA(cudaEventRecord(c->digits_done, st));
            for (int v0 = 0; v0 < nv; v0 += vstep) {
                const int k = std::min(vstep, nv - v0);
                if (launch_volterra_exact(c->xdig.as<unsigned char>(), fixed_panels(*c, ts, fp, v0, k, st), ts.xvols + v0, k,
                                          N, b, true, true, c->xbuf.as<uint64_t>(), words, st) ||
                    launch_variance_fixed(ts.xvols + v0, ts.xgrps, ts.xcomp, Zd, c->xbuf.as<uint64_t>(), k, xt.max_groups,
                                          xt.u53, true, ns, N, b, c->ivb.as<double>(), ivp, st))
                    return fail(RBG_ERR_CUDA, "FP64 path kernels could not be configured");
            }
        }
        // whether the batch's normals were in range is known once the digits are, while
        // the kernels queued behind them run
        bool out_of_range = false;
        if (fixed) {
            RBG_CUDA(cudaEventSynchronize(c->digits_done));
            out_of_range = seen[1] != 0;
        }
        if (out_of_range && !fp64_tables) {
            // (growing the tables may have taken the digit convolution's buffers)
            if ((rc = upload_tables(*c, plan, st, ts, logL, &xt, true))) return rc;
            fp64_tables = true;
            fixed = c->xdig.p && c->xbuf.p && c->xpan.p;
        }
        if (!fixed || out_of_range) launch_path_fp64(ts.t, Zd, b, c->ivb.as<double>(), st, ivp);
        if (launch_payoff_store(ts.t, c->ivb.as<double>(), b, b, Pd, st, ivp))
            return fail(RBG_ERR_CUDA, "FP64 payoff kernel could not be configured");
        RBG_CUDA(cudaGetLastError());
        if (!device_ptrs)
            RBG_CUDA(cudaMemcpyAsync(payoff + m0 * no, Pd, sizeof(double) * no * b, cudaMemcpyDeviceToHost, st));
    }
    if (seen) RBG_CUDA(cudaMemcpyAsync((void*)seen, words, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
    RBG_CUDA(cudaStreamSynchronize(st));
    if (seen && seen[0])
        return fail(RBG_ERR_TIMEOUT,
                    "FP64 convolution: a bounded pipeline wait expired (site " + std::to_string(seen[0]) + ")");
    return RBG_OK;
}

// Mixed form of the quadrature entry points: the caller's normals run through
// the tensor-core path kernel (FP32 path state; a.ext instead of the Philox
// stream) and the FP32 payoff per path is written as double.
static int payoffs_quadrature_mixed(const rbg_params* p, const rbg_options& o, const double* Z, double* payoff,
                                    int device_ptrs, bool mc)
{
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err, mc)) return fail(RBG_ERR_ARG, err);
    if (!Z || !payoff) return fail(RBG_ERR_ARG, "null Z/payoff");
    Ctx* c = nullptr;
    int rc = get_ctx(&c, o.stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = o.stream ? (cudaStream_t)o.stream : c->stream;
    TableSet ts;
    if ((rc = upload_tables(*c, plan, st, ts, 0, nullptr, false))) return rc;
    const int no = (int)plan.outs.size(), N = plan.N, ns = mc ? 3 : 2;
    const int64_t M = p->M;
    MixedJob job;
    if ((rc = mixed_prepare(plan, o, M, job, g_err, 0, mc))) return rc;
    int64_t B = job.batch;
    B = std::min<int64_t>(B, std::max<int64_t>(256, ((int64_t)1 << 30) / (8 * (int64_t)no)));  // payoffs <= 1 GiB
    if (!device_ptrs)  // staged normals <= 2 GiB
        B = std::min<int64_t>(B, std::max<int64_t>(256, ((int64_t)1 << 31) / (8 * (int64_t)ns * N)));
    if ((rc = ensure(*c, c->mixed_ws, job.workspace_bytes, "mixed workspace"))) return rc;
    if ((rc = ensure(*c, c->ivb, sizeof(float) * 2 * plan.vgs.size() * (size_t)B, "variance sums"))) return rc;
    if (mc && (rc = ensure(*c, c->ivp, sizeof(float) * plan.vgs.size() * (size_t)B, "variance sums"))) return rc;
    float* ivq = mc ? c->ivp.as<float>() : nullptr;
    if (!device_ptrs) {
        if ((rc = ensure(*c, c->z, sizeof(double) * ns * N * (size_t)B, "normals"))) return rc;
        if ((rc = ensure(*c, c->pay, sizeof(double) * no * (size_t)B, "payoffs"))) return rc;
    }
    if (c->mixed_img != job.host_ws) {
        c->mixed_img.clear();
        ++c->img_gen;
        if ((rc = mixed_upload(job, c->mixed_ws.p, st, g_err))) return rc;
        c->mixed_img = job.host_ws;
    } else {
        RBG_CUDA(cudaMemsetAsync((unsigned char*)c->mixed_ws.p + job.off_err, 0, 4, st));
    }
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        const double* Zd;
        double* Pd;
        if (device_ptrs) {
            Zd = Z + m0 * ns * N;
            Pd = payoff + m0 * no;
        } else {
            RBG_CUDA(cudaMemcpyAsync(c->z.p, Z + m0 * ns * N, sizeof(double) * ns * N * b, cudaMemcpyHostToDevice,
                                     st));
            Zd = c->z.as<double>();
            Pd = c->pay.as<double>();
        }
        if ((rc = mixed_launch(job, c->mixed_ws.p, o.seed, 0, b, c->ivb.p, st, g_err, nullptr, nullptr, nullptr,
                               nullptr, ivq, Zd)))
            return rc;
        launch_payoff_store_f32(ts.t.outs, no, c->ivb.p, ivq, b, Pd, st);
        RBG_CUDA(cudaGetLastError());
        if (!device_ptrs)
            RBG_CUDA(cudaMemcpyAsync(payoff + m0 * no, Pd, sizeof(double) * no * b, cudaMemcpyDeviceToHost, st));
    }
    if ((rc = mixed_check(job, c->mixed_ws.p, st, g_err))) return rc;
    RBG_CUDA(cudaStreamSynchronize(st));
    return RBG_OK;
}

}  // namespace rbg

using namespace rbg;

// ===================================================================== ABI
extern "C" {

void rbg_default_options(rbg_options* o)
{
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->precision = RBG_FP64;
    o->conv = RBG_CONV_AUTO;
    o->normals = RBG_NORMALS_F64;
    o->split = RBG_SPLIT_BF16X3;
    o->compute_iv = 1;
}

const char* rbg_last_error(void) { return g_err.c_str(); }

uint64_t rbg_launch_count(void) { return g_launches.load(); }

int rbg_price_rt(const rbg_params* p, const rbg_options* o, double* price, double* stat, double* iv)
{
    std::vector<double> res;
    int rc = price_any(p, o, res);
    if (rc) return rc;
    const size_t no = res.size() / 5;
    if (price) std::memcpy(price, res.data(), no * sizeof(double));
    if (stat) std::memcpy(stat, res.data() + no, no * sizeof(double));
    if (iv) std::memcpy(iv, res.data() + 2 * no, no * sizeof(double));
    return RBG_OK;
}

int rbg_price_rt_unordered(const rbg_unordered* u, const rbg_options* o, double* price, double* stat, double* iv)
{
    if (!u || !o) return fail(RBG_ERR_ARG, "null params/options");
    g_h2d = g_d2h = 0;
    Plan plan;
    std::string err;
    if (!build_plan_unordered(*u, plan, err)) return fail(RBG_ERR_ARG, err);
    std::vector<double> res;
    int rc = price_plan(plan, u->M, o, res);
    if (rc) return rc;
    const size_t no = res.size() / 5;
    if (price) std::memcpy(price, res.data(), no * sizeof(double));
    if (stat) std::memcpy(stat, res.data() + no, no * sizeof(double));
    if (iv) std::memcpy(iv, res.data() + 2 * no, no * sizeof(double));
    return RBG_OK;
}

int rbg_price_rt_cv(const rbg_cv_params* p, const rbg_options* o, double* price, double* stat, double* iv)
{
    std::vector<double> res;
    int rc = price_cv_any(p, o, nullptr, nullptr, res);
    if (rc) return rc;
    const size_t no = res.size() / 5;
    if (price) std::memcpy(price, res.data(), no * sizeof(double));
    if (stat) std::memcpy(stat, res.data() + no, no * sizeof(double));
    if (iv) std::memcpy(iv, res.data() + 2 * no, no * sizeof(double));
    return RBG_OK;
}

int rbg_price_rt_cv_normals(const rbg_cv_params* p, const double* Zc, const double* Z, double* price, double* stat,
                            double* iv)
{
    if (!Zc || !Z) return fail(RBG_ERR_ARG, "null normals");
    rbg_options o;
    rbg_default_options(&o);
    std::vector<double> res;
    int rc = price_cv_any(p, &o, Zc, Z, res);
    if (rc) return rc;
    const size_t no = res.size() / 5;
    if (price) std::memcpy(price, res.data(), no * sizeof(double));
    if (stat) std::memcpy(stat, res.data() + no, no * sizeof(double));
    if (iv) std::memcpy(iv, res.data() + 2 * no, no * sizeof(double));
    return RBG_OK;
}

int rbg_price_rt_sums(const rbg_params* p, const rbg_options* o, double* sum, double* sum2)
{
    std::vector<double> res;
    int rc = price_any(p, o, res);
    if (rc) return rc;
    const size_t no = res.size() / 5;
    if (sum) std::memcpy(sum, res.data() + 3 * no, no * sizeof(double));
    if (sum2) std::memcpy(sum2, res.data() + 4 * no, no * sizeof(double));
    return RBG_OK;
}

int rbg_merge_sums(int n_shards, int n, const double* sum, const double* sum2, int64_t M, double* price,
                   double* stat)
{
    if (n_shards < 1 || n < 0 || M < 1 || (n > 0 && (!sum || !sum2 || !price || !stat)))
        return fail(RBG_ERR_ARG, "rbg_merge_sums: need n_shards >= 1, n >= 0, M >= 1 and non-null arrays");
    const double invM = 1.0 / (double)M, isq = 1.0 / std::sqrt((double)M);
    for (int i = 0; i < n; ++i) {
        // shard order, Neumaier-compensated: the merge does not depend on how
        // the caller's collective ordered its additions
        double S = 0, C = 0, S2 = 0, C2 = 0;
        for (int k = 0; k < n_shards; ++k) {
            host_neumaier_add(S, C, sum[(size_t)k * n + i]);
            host_neumaier_add(S2, C2, sum2[(size_t)k * n + i]);
        }
        S += C;
        S2 += C2;
        // rBergLib/rBergomiMT.cpp:404-409
        const double pr = S * invM;
        const double var = std::fma(-pr, pr, S2 * invM);
        price[i] = pr;
        stat[i] = std::sqrt(var > 0.0 ? var : 0.0) * isq;
    }
    return RBG_OK;
}

int rbg_payoffs_rt(const rbg_params* p, const rbg_options* o, const double* Z, double* payoff, int device_ptrs)
{
    if (!p) return fail(RBG_ERR_ARG, "null params");
    if (o && o->precision == RBG_MIXED) return payoffs_quadrature_mixed(p, *o, Z, payoff, device_ptrs, false);
    if (o && o->precision != RBG_FP64) return fail(RBG_ERR_ARG, "unknown precision");
    return payoffs_quadrature(p, Z, payoff, device_ptrs, o ? (cudaStream_t)o->stream : nullptr, false,
                              o ? o->conv : RBG_CONV_AUTO);
}

int rbg_generate_normals_streams(uint64_t seed, int64_t path_offset, int64_t M, int N, int precision, int streams,
                                 double* Z)
{
    if (M < 1 || N < 1 || !Z) return fail(RBG_ERR_ARG, "bad sizes");
    if (streams != 2 && streams != 3) return fail(RBG_ERR_ARG, "streams must be 2 or 3");
    Ctx* c = nullptr;
    int rc = get_ctx(&c);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    const int ns = streams;
    const int64_t B = std::max<int64_t>(1, std::min<int64_t>(M, ((int64_t)1 << 30) / (8 * ns * (int64_t)N)));
    if ((rc = ensure(*c, c->z, sizeof(double) * ns * N * (size_t)B, "normals"))) return rc;
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        if (launch_normals_fixed(seed, path_offset + m0, b, N, precision == RBG_MIXED, c->z.as<double>(), nullptr, 0, ns,
                                 c->stream, true))
            return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
        RBG_CUDA(cudaGetLastError());
        RBG_CUDA(cudaMemcpyAsync(Z + m0 * ns * N, c->z.p, sizeof(double) * ns * N * b, cudaMemcpyDeviceToHost,
                                 c->stream));
    }
    RBG_CUDA(cudaStreamSynchronize(c->stream));
    return RBG_OK;
}

int rbg_generate_normals(uint64_t seed, int64_t path_offset, int64_t M, int N, int precision, double* Z)
{
    return rbg_generate_normals_streams(seed, path_offset, M, N, precision, 2, Z);
}

// ------------------------------------------------------ Sobol' QMC normals
// Checks the request and puts the first 2N coordinates of the caller's
// direction table on the device, transposed to [kSobolBits][2N] (kept, so a
// repeated table uploads nothing).  bridge: the hierarchical map's
// coefficients, computed as rBergomi/aux.h:106-125 does (exp2 of halves).
static int sobol_setup(Ctx& c, const uint64_t* dirs, int dims, int N, int bridge, int64_t path_offset, int64_t M,
                       cudaStream_t st, SobolBridge& br)
{
    if (!dirs) return fail(RBG_ERR_ARG, "null Sobol' direction table");
    if (N < 1 || M < 1 || path_offset < 0) return fail(RBG_ERR_ARG, "bad sizes");
    if (dims < 2 * N) return fail(RBG_ERR_ARG, "the Sobol' direction table has fewer than 2N dimensions");
    if ((uint64_t)path_offset + (uint64_t)M >= ((uint64_t)1 << kSobolBits) - 1)
        return fail(RBG_ERR_ARG, "Sobol' point index beyond 2^62");
    if (bridge) {
        int m = 0;
        while ((1 << m) < N) ++m;
        if ((1 << m) != N) return fail(RBG_ERR_ARG, "the Brownian bridge needs N a power of two");
        if (m > kMaxBridgeLevels) return fail(RBG_ERR_UNSUPPORTED, "the Brownian bridge supports N <= 8192");
        br.m = m;
        br.c[0] = std::exp2(-0.5 * m);
        for (int n = 1; n <= m; ++n) br.c[n] = std::exp2(0.5 * (n - m - 1));
    }
    const int D = 2 * N;
    std::vector<unsigned long long> img((size_t)kSobolBits * D);
    for (int k = 0; k < kSobolBits; ++k)
        for (int d = 0; d < D; ++d) img[(size_t)k * D + d] = dirs[(size_t)d * kSobolBits + k];
    if (img != c.sobol_img) {
        int rc = ensure(c, c.sobol, sizeof(unsigned long long) * img.size(), "Sobol' table");
        if (rc) return rc;
        c.sobol_img.clear();
        RBG_CUDA(cudaMemcpyAsync(c.sobol.p, img.data(), sizeof(unsigned long long) * img.size(),
                                 cudaMemcpyHostToDevice, st));
        RBG_CUDA(cudaStreamSynchronize(st));
        g_h2d += sizeof(unsigned long long) * img.size();
        c.sobol_img.swap(img);
    }
    return RBG_OK;
}

int rbg_sobol_normals(const uint64_t* directions, int dims, int N, int64_t M, int64_t path_offset, int bridge,
                      int precision, double* Z)
{
    if (!Z) return fail(RBG_ERR_ARG, "null output");
    if (precision != RBG_FP64 && precision != RBG_MIXED) return fail(RBG_ERR_ARG, "unknown precision");
    if (precision == RBG_MIXED && bridge)
        return fail(RBG_ERR_UNSUPPORTED, "the Brownian bridge runs in the FP64 form only");
    if (precision == RBG_MIXED && (uint64_t)path_offset + (uint64_t)M + 128 >= ((uint64_t)1 << 32))
        return fail(RBG_ERR_ARG, "Sobol' point index beyond 2^32 in the mixed form");
    Ctx* c = nullptr;
    int rc = get_ctx(&c);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    SobolBridge br{};
    if ((rc = sobol_setup(*c, directions, dims, N, bridge, path_offset, M, c->stream, br))) return rc;
    const int64_t B = std::max<int64_t>(1, std::min<int64_t>(M, ((int64_t)1 << 30) / (16 * (int64_t)N)));
    if ((rc = ensure(*c, c->z, sizeof(double) * 2 * N * (size_t)B, "normals"))) return rc;
    for (int64_t m0 = 0; m0 < M; m0 += B) {
        const int64_t b = std::min(B, M - m0);
        if (launch_sobol_normals(c->sobol.as<unsigned long long>(), N, (uint64_t)(path_offset + m0 + 1), b,
                                 bridge ? &br : nullptr, c->z.as<double>(), c->stream, precision == RBG_MIXED))
            return fail(RBG_ERR_UNSUPPORTED, "Brownian bridge shared memory not available for this N");
        RBG_CUDA(cudaGetLastError());
        RBG_CUDA(cudaMemcpyAsync(Z + m0 * 2 * N, c->z.p, sizeof(double) * 2 * N * b, cudaMemcpyDeviceToHost,
                                 c->stream));
    }
    RBG_CUDA(cudaStreamSynchronize(c->stream));
    return RBG_OK;
}

// Mixed form: the table's bits 30..61 as uint32 [32][2N] (points below 2^32),
// kept on the device like the FP64 table.
static int sobol32_setup(Ctx& c, const uint64_t* dirs, int dims, int N, int64_t path_offset, int64_t M,
                         cudaStream_t st)
{
    if (!dirs) return fail(RBG_ERR_ARG, "null Sobol' direction table");
    if (N < 1 || M < 1 || path_offset < 0) return fail(RBG_ERR_ARG, "bad sizes");
    if (dims < 2 * N) return fail(RBG_ERR_ARG, "the Sobol' direction table has fewer than 2N dimensions");
    if ((uint64_t)path_offset + (uint64_t)M + 128 >= ((uint64_t)1 << 32))
        return fail(RBG_ERR_ARG, "Sobol' point index beyond 2^32 in the mixed form");
    const int D = 2 * N;
    std::vector<unsigned int> img((size_t)32 * D);
    for (int k = 0; k < 32; ++k)
        for (int d = 0; d < D; ++d) img[(size_t)k * D + d] = (unsigned int)(dirs[(size_t)d * kSobolBits + k] >> 30);
    if (img != c.sobol32_img) {
        int rc = ensure(c, c.sobol32, sizeof(unsigned int) * img.size(), "Sobol' table");
        if (rc) return rc;
        c.sobol32_img.clear();
        RBG_CUDA(cudaMemcpyAsync(c.sobol32.p, img.data(), sizeof(unsigned int) * img.size(), cudaMemcpyHostToDevice,
                                 st));
        RBG_CUDA(cudaStreamSynchronize(st));
        g_h2d += sizeof(unsigned int) * img.size();
        c.sobol32_img.swap(img);
    }
    return RBG_OK;
}

int rbg_price_rt_sobol(const rbg_params* p, const rbg_options* o, const uint64_t* directions, int dims, int bridge,
                       double* price, double* stat, double* iv)
{
    if (!p || !o) return fail(RBG_ERR_ARG, "null params/options");
    if (o->precision != RBG_FP64 && o->precision != RBG_MIXED) return fail(RBG_ERR_ARG, "unknown precision");
    g_h2d = g_d2h = 0;
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err, false)) return fail(RBG_ERR_ARG, err);
    Ctx* c = nullptr;
    int rc = get_ctx(&c, o->stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = o->stream ? (cudaStream_t)o->stream : c->stream;
    std::vector<double> res(5 * plan.outs.size(), 0.0);
    // the mixed form's GEMM producer draws the points itself (N <= 1024, point
    // indices below 2^32, no bridge); otherwise the normals are materialized
    const bool producer = !bridge && o->conv != RBG_CONV_FFT && plan.N <= 1024 &&
                          (uint64_t)o->path_offset + (uint64_t)p->M + 128 < ((uint64_t)1 << 32);
    if (o->precision == RBG_MIXED && producer) {
        if ((rc = sobol32_setup(*c, directions, dims, plan.N, o->path_offset, p->M, st))) return rc;
        if ((rc = price_mixed(*c, plan, *o, p->M, st, res.data(), false, c->sobol32.as<unsigned int>()))) return rc;
    } else if (o->precision == RBG_MIXED) {
        SobolBridge br{};
        if ((rc = sobol_setup(*c, directions, dims, plan.N, bridge, o->path_offset, p->M, st, br))) return rc;
        const SobolZ sz{c->sobol.as<unsigned long long>(), bridge ? &br : nullptr, o->path_offset};
        if ((rc = price_mixed(*c, plan, *o, p->M, st, res.data(), false, nullptr, &sz))) return rc;
    } else {
        SobolBridge br{};
        if ((rc = sobol_setup(*c, directions, dims, plan.N, bridge, o->path_offset, p->M, st, br))) return rc;
        if ((rc = price_fp64(*c, plan, *o, p->M, st, res.data(), false, c->sobol.as<unsigned long long>(),
                             bridge ? &br : nullptr)))
            return rc;
    }
    const size_t no = plan.outs.size();
    if (price) std::memcpy(price, res.data(), no * sizeof(double));
    if (stat) std::memcpy(stat, res.data() + no, no * sizeof(double));
    if (iv) std::memcpy(iv, res.data() + 2 * no, no * sizeof(double));
    return RBG_OK;
}

int rbg_price_mc(const rbg_params* p, const rbg_options* o, double* price, double* stat, double* iv)
{
    std::vector<double> res;
    int rc = price_any(p, o, res, true);
    if (rc) return rc;
    const size_t no = res.size() / 5;
    if (price) std::memcpy(price, res.data(), no * sizeof(double));
    if (stat) std::memcpy(stat, res.data() + no, no * sizeof(double));
    if (iv) std::memcpy(iv, res.data() + 2 * no, no * sizeof(double));
    return RBG_OK;
}

int rbg_payoffs_mc(const rbg_params* p, const rbg_options* o, const double* Z, double* payoff, int device_ptrs)
{
    if (!p) return fail(RBG_ERR_ARG, "null params");
    if (o && o->precision == RBG_MIXED) return payoffs_quadrature_mixed(p, *o, Z, payoff, device_ptrs, true);
    if (o && o->precision != RBG_FP64) return fail(RBG_ERR_ARG, "unknown precision");
    return payoffs_quadrature(p, Z, payoff, device_ptrs, o ? (cudaStream_t)o->stream : nullptr, true,
                              o ? o->conv : RBG_CONV_AUTO);
}

int rbg_implied_vol(int n, const double* price, const double* K, const double* T, double* iv)
{
    if (n < 0 || (n > 0 && (!price || !K || !T || !iv))) return fail(RBG_ERR_ARG, "bad arguments");
    if (n == 0) return RBG_OK;
    Ctx* c = nullptr;
    int rc = get_ctx(&c);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    if ((rc = ensure(*c, c->res, sizeof(double) * 4 * (size_t)n, "iv buffers"))) return rc;
    double* d = c->res.as<double>();
    RBG_CUDA(cudaMemcpyAsync(d, price, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    RBG_CUDA(cudaMemcpyAsync(d + n, K, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    RBG_CUDA(cudaMemcpyAsync(d + 2 * n, T, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    if (launch_implied_vol(n, d, d + n, d + 2 * n, d + 3 * n, c->stream))
        return fail(RBG_ERR_CUDA, "fixed-point tables not found on the device");
    RBG_CUDA(cudaGetLastError());
    RBG_CUDA(cudaMemcpyAsync(iv, d + 3 * n, sizeof(double) * n, cudaMemcpyDeviceToHost, c->stream));
    RBG_CUDA(cudaStreamSynchronize(c->stream));
    return RBG_OK;
}

int rbg_synchronize(void)
{
    Ctx* c = nullptr;
    int rc = get_ctx(&c);
    if (rc) return rc;
    RBG_CUDA(cudaStreamSynchronize(c->stream));
    return RBG_OK;
}

int rbg_release(void)
{
    Ctx* c0 = nullptr;
    int rc = get_ctx(&c0);
    if (rc) return rc;
    std::vector<Ctx*> all;
    if ((rc = device_ctxs(all))) return rc;
    // caller streams may be gone by now: wait for the device, not for each stream
    std::vector<std::unique_lock<std::mutex>> locks;
    for (Ctx* c : all) locks.emplace_back(c->mu);
    RBG_CUDA(cudaDeviceSynchronize());
    for (Ctx* c : all) {
        for (DevBuf* b : {&c->z, &c->ivb, &c->ivp, &c->part, &c->acc, &c->tabs, &c->res, &c->pay, &c->mixed_ws,
                          &c->cv, &c->sobol, &c->sobol32, &c->xdig, &c->xbuf, &c->xpan})
            b->release();
        c->pin.release();
        c->xpan_ready = false;
        c->tabs_img.clear();
        c->mixed_img.clear();
        c->sobol_img.clear();
        c->sobol32_img.clear();
        ++c->img_gen;
    }
    return RBG_OK;
}

int rbg_debug_mixed_paths(const rbg_params* p, const rbg_options* o, float* normals, float* x, float* ivb)
{
    if (!p || !o) return fail(RBG_ERR_ARG, "null params/options");
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err)) return fail(RBG_ERR_ARG, err);
    if (p->M > (1 << 20)) return fail(RBG_ERR_ARG, "diagnostic runs are limited to 2^20 paths");
    Ctx* c = nullptr;
    int rc = get_ctx(&c, o->stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = o->stream ? (cudaStream_t)o->stream : c->stream;
    MixedJob job;
    if ((rc = mixed_prepare(plan, *o, p->M, job, g_err))) return rc;
    if (job.batch < p->M) return fail(RBG_ERR_ARG, "diagnostic run does not fit one batch");
    const int Np = (plan.N + 31) / 32 * 32;
    const size_t M = (size_t)p->M, nvg = plan.vgs.size();
    if ((rc = ensure(*c, c->mixed_ws, job.workspace_bytes, "mixed workspace"))) return rc;
    DevBuf dbg;
    if (dbg.ensure(sizeof(float) * (M * 2 * Np + M * Np + 2 * nvg * M))) return fail(RBG_ERR_NOMEM, "debug buffers");
    float* dw = dbg.as<float>();
    float* dx = dw + M * 2 * Np;
    float* div = dx + M * Np;
    c->mixed_img.clear();
    ++c->img_gen;
    if ((rc = mixed_upload(job, c->mixed_ws.p, st, g_err))) { dbg.release(); return rc; }
    rc = mixed_launch(job, c->mixed_ws.p, o->seed, o->path_offset, p->M, div, st, g_err, dw, dx);
    if (!rc) rc = mixed_check(job, c->mixed_ws.p, st, g_err);
    if (!rc) {
        cudaError_t e = cudaSuccess;
        if (normals) e = cudaMemcpy(normals, dw, sizeof(float) * M * 2 * Np, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && x) e = cudaMemcpy(x, dx, sizeof(float) * M * Np, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && ivb) e = cudaMemcpy(ivb, div, sizeof(float) * 2 * nvg * M, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            cudaGetLastError();
            rc = fail(RBG_ERR_CUDA, std::string("debug copy: ") + cudaGetErrorString(e));
        }
    }
    dbg.release();
    return rc;
}

void rbg_profile_enable(int on)
{
    std::lock_guard<std::mutex> lk(g_prof.mu);
    g_prof.on = on != 0;
}

void rbg_profile_reset(void)
{
    std::lock_guard<std::mutex> lk(g_prof.mu);
    for (int i = 0; i < kStages; ++i) { g_prof.ms[i] = 0; g_prof.n[i] = 0; }
}

const char* rbg_profile_path(void)
{
    std::lock_guard<std::mutex> lk(g_prof.mu);
    return g_prof.path;
}

int rbg_profile_read(int stage, double* total_ms, uint64_t* launches)
{
    if (stage < 0 || stage >= kStages) return fail(RBG_ERR_ARG, "bad stage");
    std::lock_guard<std::mutex> lk(g_prof.mu);
    if (total_ms) *total_ms = g_prof.ms[stage];
    if (launches) *launches = g_prof.n[stage];
    return RBG_OK;
}

void rbg_last_transfer_bytes(uint64_t* h2d, uint64_t* d2h)
{
    if (h2d) *h2d = g_h2d;
    if (d2h) *d2h = g_d2h;
}

int rbg_debug_wait_timeout(unsigned int* site)
{
    Ctx* c = nullptr;
    int rc = get_ctx(&c);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    DevBuf word;
    if (word.ensure(sizeof(unsigned int))) return fail(RBG_ERR_NOMEM, "error word");
    unsigned int host = 0;
    cudaError_t e = cudaMemsetAsync(word.p, 0, sizeof(unsigned int), c->stream);
    const unsigned int kSite = 99;
    if (e == cudaSuccess && launch_wait_probe(word.as<unsigned int>(), kSite, c->stream))
        e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&host, word.p, sizeof(host), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    word.release();
    if (e != cudaSuccess) return fail(RBG_ERR_CUDA, std::string("wait probe: ") + cudaGetErrorString(e));
    if (site) *site = host;
    if (host != 0) return fail(RBG_ERR_TIMEOUT, "bounded wait expired (site " + std::to_string(host) + ")");
    return fail(RBG_ERR_CUDA, "wait probe returned without expiring");
}

int rbg_debug_mixed_profile(const rbg_params* p, const rbg_options* o, uint64_t* cycles, int n)
{
    if (!p || !o || !cycles || n < 32) return fail(RBG_ERR_ARG, "need params, options and 32 counters");
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err)) return fail(RBG_ERR_ARG, err);
    Ctx* c = nullptr;
    int rc = get_ctx(&c, o->stream);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(c->mu);
    cudaStream_t st = o->stream ? (cudaStream_t)o->stream : c->stream;
    MixedJob job;
    if ((rc = mixed_prepare(plan, *o, p->M, job, g_err))) return rc;
    if (job.batch < p->M) return fail(RBG_ERR_ARG, "diagnostic run does not fit one batch");
    const int no = (int)plan.outs.size();
    if ((rc = ensure(*c, c->mixed_ws, job.workspace_bytes, "mixed workspace"))) return rc;
    DevBuf dbg;
    const size_t ivb_bytes = job.fused ? 0 : sizeof(float) * 2 * plan.vgs.size() * (size_t)p->M;
    const size_t part_bytes = sizeof(double) * 4 * no * (size_t)std::max(1, mixed_part_rows(job, p->M));
    if (dbg.ensure(256 + ivb_bytes + part_bytes)) return fail(RBG_ERR_NOMEM, "debug buffers");
    unsigned long long* prof = dbg.as<unsigned long long>();
    unsigned char* ivb = (unsigned char*)dbg.p + 256;
    double* part = (double*)(ivb + ivb_bytes);
    c->mixed_img.clear();
    ++c->img_gen;
    if ((rc = mixed_upload(job, c->mixed_ws.p, st, g_err))) { dbg.release(); return rc; }
    cudaMemsetAsync(dbg.p, 0, 256 + ivb_bytes + part_bytes, st);
    rc = mixed_launch(job, c->mixed_ws.p, o->seed, o->path_offset, p->M, job.fused ? nullptr : (void*)ivb, st, g_err,
                      nullptr, nullptr, job.fused ? part : nullptr, prof);
    if (!rc) rc = mixed_check(job, c->mixed_ws.p, st, g_err);
    std::vector<unsigned long long> h(32, 0);
    if (!rc && cudaMemcpy(h.data(), prof, 256, cudaMemcpyDeviceToHost) != cudaSuccess) {
        cudaGetLastError();
        rc = fail(RBG_ERR_CUDA, "debug copy failed");
    }
    for (int i = 0; i < 32; ++i) cycles[i] = h[i];
    dbg.release();
    return rc;
}

int rbg_plan_info(const rbg_params* p, int* n_vol, int* n_vgroups, int* n_out, int* vgroup_of_output)
{
    if (!p) return fail(RBG_ERR_ARG, "null params");
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err)) return fail(RBG_ERR_ARG, err);
    if (n_vol) *n_vol = (int)plan.vols.size();
    if (n_vgroups) *n_vgroups = (int)plan.vgs.size();
    if (n_out) *n_out = (int)plan.outs.size();
    if (vgroup_of_output)
        for (size_t i = 0; i < plan.outs.size(); ++i) vgroup_of_output[i] = plan.outs[i].vg;
    return RBG_OK;
}

int rbg_plan_info_mc(const rbg_params* p, int* n_vol, int* n_vgroups, int* vgroup_of_output, double* rho_of_output)
{
    if (!p) return fail(RBG_ERR_ARG, "null params");
    Plan plan;
    std::string err;
    if (!build_plan(*p, plan, err, true)) return fail(RBG_ERR_ARG, err);
    if (n_vol) *n_vol = (int)plan.vols.size();
    if (n_vgroups) *n_vgroups = (int)plan.vgs.size();
    for (size_t i = 0; i < plan.outs.size(); ++i) {
        if (vgroup_of_output) vgroup_of_output[i] = plan.outs[i].vg;
        if (rho_of_output) rho_of_output[i] = plan.outs[i].rho;
    }
    return RBG_OK;
}

int rbg_plan_info_unordered(const rbg_unordered* u, int* n_vol, int* n_vgroups, int* vgroup_of_output)
{
    if (!u) return fail(RBG_ERR_ARG, "null list");
    Plan plan;
    std::string err;
    if (!build_plan_unordered(*u, plan, err)) return fail(RBG_ERR_ARG, err);
    if (n_vol) *n_vol = (int)plan.vols.size();
    if (n_vgroups) *n_vgroups = (int)plan.vgs.size();
    if (vgroup_of_output)
        for (size_t i = 0; i < plan.outs.size(); ++i) vgroup_of_output[i] = plan.outs[i].vg;
    return RBG_OK;
}

// ------------------------------------------------------------- drop-in
static void die_on(int rc)
{
    if (rc == RBG_OK) return;
    std::cerr << "rbergomi_gb300: " << rbg_last_error() << "\n";
    std::exit(70);
}

static void fill_tot(double* H, double* eta, double* rho, int par_size, double* T, double* K, int op_size,
                     double* H_tot, double* eta_tot, double* rho_tot, double* T_tot, double* K_tot)
{
    const long out = (long)par_size * op_size;
    for (long i = 0; i < out; ++i) {
        H_tot[i] = H[i / op_size];
        eta_tot[i] = eta[i / op_size];
        rho_tot[i] = rho[i / op_size];
        T_tot[i] = T[i % op_size];
        K_tot[i] = K[i % op_size];
    }
}


static void check_dropin_sizes(int par_size, int op_size, int num_threads, int out_size)
{
    if (out_size != par_size * op_size) {
        std::cerr << "Output arrays have wrong size:\n"
                  << "par_size * op_size = " << par_size * op_size << " != out_size.\n";
        std::exit(17);
    }
    if (num_threads < 1) {
        std::cerr << "Number of threads has to be a positive integer,\n"
                  << "obtained num_threads = " << num_threads << ".\n";
        std::exit(21);
    }
}

// Plain Monte Carlo (rBergLib/cinterface.cpp:10-46): FP64 form, third normal
// stream, payoff max(S_T - K, 0).  The reference hands rho_tot and eta_tot to
// Result2Array in swapped order (cinterface.cpp:45), so eta_tot receives the
// rho values and rho_tot the eta values; kept for drop-in compatibility.
void computeIV_tensor(double xi, double* H, double* eta, double* rho, int par_size, double* T, double* K,
                      int op_size, int N, long M, uint64_t* seed, int seed_size, int num_threads, double* price,
                      double* iv, double* stat, double* H_tot, double* eta_tot, double* rho_tot, double* T_tot,
                      double* K_tot, int out_size)
{
    check_dropin_sizes(par_size, op_size, num_threads, out_size);
    if (out_size == 0) return;  // an empty grid: the reference's loops run zero times
    rbg_params p{xi, H, eta, rho, par_size, T, K, op_size, N, (int64_t)M};
    rbg_options o;
    rbg_default_options(&o);
    const char* prec = std::getenv("RBG_PRECISION");
    if (prec && std::strcmp(prec, "mixed") == 0) o.precision = RBG_MIXED;
    o.seed = rbg::fold_seed(seed, seed_size);
    die_on(rbg_price_mc(&p, &o, price, stat, iv));
    fill_tot(H, eta, rho, par_size, T, K, op_size, H_tot, rho_tot, eta_tot, T_tot, K_tot);
}

void computeIVRT_tensor(double xi, double* H, double* eta, double* rho, int par_size, double* T, double* K,
                        int op_size, int N, long M, uint64_t* seed, int seed_size, int num_threads, double* price,
                        double* iv, double* stat, double* H_tot, double* eta_tot, double* rho_tot, double* T_tot,
                        double* K_tot, int out_size)
{
    check_dropin_sizes(par_size, op_size, num_threads, out_size);
    if (out_size == 0) return;  // an empty grid: the reference's loops run zero times
    rbg_params p{xi, H, eta, rho, par_size, T, K, op_size, N, (int64_t)M};
    rbg_options o;
    rbg_default_options(&o);
    const char* prec = std::getenv("RBG_PRECISION");
    if (prec && std::strcmp(prec, "mixed") == 0) o.precision = RBG_MIXED;
    o.seed = rbg::fold_seed(seed, seed_size);
    die_on(rbg_price_rt(&p, &o, price, stat, iv));
    fill_tot(H, eta, rho, par_size, T, K, op_size, H_tot, eta_tot, rho_tot, T_tot, K_tot);
}

void computeIVRT_tensor_quadrature(double xi, double* H, double* eta, double* rho, int par_size, double* T,
                                   double* K, int op_size, int N, long M, double* Z, int num_threads,
                                   double* payoff)
{
    (void)num_threads;
    if (M <= 0 || (long)par_size * op_size == 0) return;  // nothing to price: no payoffs written
    rbg_params p{xi, H, eta, rho, par_size, T, K, op_size, N, (int64_t)M};
    rbg_options o;
    rbg_default_options(&o);
    const char* prec = std::getenv("RBG_PRECISION");
    if (prec && std::strcmp(prec, "mixed") == 0) o.precision = RBG_MIXED;
    die_on(rbg_payoffs_rt(&p, &o, Z, payoff, 0));
}

}  // extern "C"
