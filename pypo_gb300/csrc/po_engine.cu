// po_engine.cu -- host orchestration of one propagation on device buffers.
//
// Mixed precision (precision 0):
//   frame -> pack sources and targets -> main N-body kernel over a (target
//   block, source chunk) grid -> near-tangent pairs -> FP64 epilogue summing
//   the chunks.
// Plain FP64 (precision 1):
//   pack sources (double) -> FP64 direct sum over a (target block, source
//   chunk) grid -> epilogue.
// Scratch is stream-ordered on the caller's stream, from the library's own
// memory pool (scratch_alloc / scratch_free); nothing here synchronises the
// device.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "po_internal.h"
#include "po_kernels.cuh"

namespace po {

namespace {

thread_local std::string t_err;
thread_local int t_launches = 0;

struct DeviceInfo {
    bool ready = false;
    int sms = 0;
    bool cluster = false;           // the device can hold the frame's cluster
    cudaMemPool_t pool = nullptr;   // the library's own scratch pool
    int occ2[3][2][2] = {};  // near-field and scalar kernels, [kind][t>0][has_m]
    int occ_ff[2][2] = {};   // far-field tile kernels, [t>0][has_m]
    std::map<void *, int> occ_adj;   // adjoint and FP64 kernels: resident CTAs, attribute set
};

std::mutex g_mu;
DeviceInfo g_dev[64];
constexpr uint64_t kPoolKeep = 16ull << 30;   // freed scratch a device's pool keeps (bytes)

// Timing ring: CUDA event pairs recorded around each main-kernel launch.
struct Timing {
    bool on = false;
    std::vector<cudaEvent_t> ev;   // 2 per slot
    int used = 0;
};
Timing g_timing;

const char *err_str(cudaError_t e) { return cudaGetErrorString(e); }

}  // namespace

int fail(int code, const std::string &msg)
{
    t_err = msg;
    return code;
}

void clear_error()
{
    t_err.clear();
    t_launches = 0;
}

void note_launches(int n) { t_launches += n; }

const char *last_error() { return t_err.c_str(); }
int last_launches() { return t_launches; }

int n_out(int mode)
{
    static const int n[6] = {12, 12, 24, 15, 12, 2};
    return (mode >= 0 && mode < 6) ? n[mode] : -1;
}

// Record a CUDA failure in rc (once) and carry on to the caller's cleanup.
#define PO_CK_RC(expr)                                                                      \
    do {                                                                                    \
        if (!rc) {                                                                          \
            cudaError_t e_ = (expr);                                                        \
            if (e_ != cudaSuccess) rc = fail(2, std::string(#expr) + ": " + err_str(e_));   \
        }                                                                                   \
    } while (0)

#define PO_CK(expr)                                                                         \
    do {                                                                                    \
        cudaError_t e_ = (expr);                                                            \
        if (e_ != cudaSuccess) return fail(2, std::string(#expr) + ": " + err_str(e_));     \
    } while (0)

// Whether the frame's cluster can run on the current device or the share of it
// that this context has (a cluster's CTAs need their SMs in one GPC).
static bool frame_cluster_fits()
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(kFrameCtas);
    c.blockDim = dim3(kFrameThreads);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kFrameCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    int n = 0;
    const bool ok = cudaFuncSetAttribute(frame_kernel(), cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, frame_kernel(), &c) == cudaSuccess && n > 0;
    if (!ok) (void)cudaGetLastError();
    return ok;
}

static int device_info(DeviceInfo *&out)
{
    int dev = 0;
    PO_CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(2, "device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_mu);
    DeviceInfo &di = g_dev[dev];
    if (!di.ready) {
        PO_CK(cudaDeviceGetAttribute(&di.sms, cudaDevAttrMultiProcessorCount, dev));
        for (int kind = 0; kind < 3; ++kind)
            for (int ts = 0; ts < 2; ++ts)
                for (int hm = 0; hm < 2; ++hm) {
                    if (kind == kKindFF || (kind == kKindScalar && hm)) continue;   // FF: occ_ff below
                    void *fn = pk_kernel(kind, ts ? 1 : -1, hm != 0, false);
                    const int smem = pk_smem_bytes(kind, hm != 0);
                    PO_CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
                    PO_CK(cudaFuncSetAttribute(pk_kernel(kind, ts ? 1 : -1, hm != 0, true),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
                    int nb = 0;
                    PO_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, kThreads, smem));
                    di.occ2[kind][ts][hm] = std::max(nb, 1);
                }
        for (int ts = 0; ts < 2; ++ts)
            for (int hm = 0; hm < 2; ++hm) {
                void *fn = ff_kernel(ts ? 1 : -1, hm != 0, false);
                const int smem = ff_smem_bytes(hm != 0);
                PO_CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
                PO_CK(cudaFuncSetAttribute(ff_kernel(ts ? 1 : -1, hm != 0, true),
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
                int nb = 0;
                PO_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, kThreads, smem));
                di.occ_ff[ts][hm] = std::max(nb, 1);
            }
        di.cluster = frame_cluster_fits();
        di.ready = true;
    }
    out = &di;
    return 0;
}

// load_split's costs: near-field and scalar forward, scalar adjoint; far-field
// forward (its tiles differ more in cost: narrow, wide, lit); near-field
// adjoint, at 2 to 4 CTAs an SM; the FP64 kernels, whose pipe two CTAs fill.
constexpr LoadCost kLoadNF = {8, 1.0, 0.2}, kLoadFF = {8, 3.0, 0.2}, kLoadAdj = {4, 0.2, 0.15}, kLoad64 = {2, 0.0, 0.03};

// Resident CTAs per SM of a kernel (and its shared-memory attribute), looked
// up once per device and kernel.
static int kernel_occupancy(DeviceInfo *di, void *fk, int threads, int smem, int &occ)
{
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = di->occ_adj.find(fk);
    if (it != di->occ_adj.end()) {
        occ = it->second;
        return 0;
    }
    int nb = 0;
    if (smem > 0) PO_CK(cudaFuncSetAttribute(fk, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    PO_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fk, threads, smem));
    occ = di->occ_adj[fk] = std::max(nb, 1);
    return 0;
}

// The far field's adjoint: waves of resident CTAs, with 0.3 of a stage for a
// CTA's start, 0.3 of a chunk for the last wave's idle share and 0.1 of a stage
// for a chunk's partials. Fitted to every split of 14 sizes (45^2 to 169^2
// points a side): 1.8 % slower than the best on average and 6 % at most (3 %
// and 11 % with 0.002 to 0.05 for the partials and no idle share).
long choose_split(long nb, long ns, long slots, long max_chunks, long tile)
{
    const long tiles = std::max(1L, (ns + tile - 1) / tile);
    long best = 1;
    double best_cost = 1e300;
    for (long s = 1; s <= std::min(tiles, std::min(std::max(1L, max_chunks), 1024L)); ++s) {
        const long chunk = (tiles + s - 1) / s;
        const long real = (tiles + chunk - 1) / chunk;
        if (real != s) continue;
        const long waves = (nb * real + slots - 1) / slots;
        const double cost = waves * (chunk + 0.3) + 0.3 * chunk + 0.1 * real;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = real;
        }
    }
    return best;
}

// The other kernels: the load of the fullest SM. With `busy` CTAs or more to
// hide latencies an SM works at one rate whatever their number, so the cost is
// its CTAs times their tiles; where they are not all resident at once (occ) the
// last ones run with fewer beside them, which costs about `tail` chunks; a
// CTA's start and partials cost `start` tiles. Fitted to every split of 134
// sizes (40^2 to 301^2 points a side): the forwards and the scalar adjoint are
// 0.2 to 0.9 % slower than the best split on average and 3 % at most, where
// counting waves of resident CTAs was 1 to 3 % and 14 % (4,422 x 4,356 with M
// 146.8 us, best 128.4); the near field's adjoint 1.1 % and 5 % (2.3 % and
// 18 %). FP64, 9,999 sources -> 1,763 targets, forward and adjoint 13.45 -> 12.79 ms.
long load_split(long nb, long ns, long sms, long occ, long max_chunks, long tile, LoadCost k)
{
    const long tiles = std::max(1L, (ns + tile - 1) / tile);
    long best = 1;
    double best_cost = 1e300;
    for (long s = 1; s <= std::min(tiles, std::min(std::max(1L, max_chunks), 1024L)); ++s) {
        const long chunk = (tiles + s - 1) / s;
        const long real = (tiles + chunk - 1) / chunk;
        if (real != s) continue;
        const long ctas = nb * real;
        const double load = (double)std::max((ctas + sms - 1) / sms, k.busy) + (ctas > sms * occ ? k.tail : 0.0);
        const double cost = chunk * load + k.start * ctas / sms;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = real;
        }
    }
    return best;
}

// Partial buffers of the chunked kernels are capped near 1 GiB.
static long partial_cap(long n, int nacc) { return std::max(1L, (1L << 30) / std::max(1L, n * nacc * 8)); }

int scratch_alloc(void **p, size_t bytes, cudaStream_t s)
{
    DeviceInfo *di = nullptr;
    if (int rc = device_info(di)) return rc;
    cudaMemPool_t pool = nullptr;
    {
        // Scratch comes from a stream-ordered pool of the library's own, made
        // on first use, so the device's default pool (shared with every
        // other user in the process) keeps its settings. A pool hands freed
        // memory back to the driver at every synchronisation unless told
        // otherwise, so each host-buffer call (which synchronises) would map
        // its scratch afresh; this one keeps up to kPoolKeep bytes of freed
        // scratch.
        std::lock_guard<std::mutex> lk(g_mu);
        if (!di->pool) {
            int dev = 0;
            PO_CK(cudaGetDevice(&dev));
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cudaMemPool_t np = nullptr;
            PO_CK(cudaMemPoolCreate(&np, &props));
            uint64_t keep = kPoolKeep;
            PO_CK(cudaMemPoolSetAttribute(np, cudaMemPoolAttrReleaseThreshold, &keep));
            di->pool = np;
        }
        pool = di->pool;
    }
    cudaError_t e = cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 16), pool, s);
    if (e != cudaSuccess) return fail(3, std::string("device scratch allocation failed: ") + err_str(e));
    return 0;
}

void scratch_free(void *p, cudaStream_t s)
{
    if (p) cudaFreeAsync(p, s);
}

int scratch_used(unsigned long long *bytes)
{
    *bytes = 0;
    int dev = 0;
    PO_CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(2, "device ordinal out of range");
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        pool = g_dev[dev].pool;
    }
    if (!pool) return 0;
    uint64_t used = 0;
    PO_CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
    *bytes = used;
    return 0;
}

// Stream-ordered scratch from the library's pool: one allocation per call
// (each costs the stream about 2 us), carved up at commit() and freed (in
// stream order) when the call's work is queued.
class PoolScratch : public Scratch {
public:
    explicit PoolScratch(cudaStream_t s) : s_(s) {}
    ~PoolScratch() override { scratch_free(base_, s_); }
    int take(void **p, size_t bytes) override
    {
        want_.push_back({p, used_});
        used_ += (std::max<size_t>(bytes, 16) + 255) / 256 * 256;
        return 0;
    }
    int commit() override
    {
        if (int rc = scratch_alloc(&base_, used_, s_)) return rc;
        for (const auto &w : want_) *w.first = static_cast<char *>(base_) + w.second;
        return 0;
    }
    size_t room() const override { return ~(size_t)0; }

private:
    cudaStream_t s_;
    void *base_ = nullptr;
    size_t used_ = 0;
    std::vector<std::pair<void **, size_t>> want_;
};

// For a kernel that begins with pdl_wait(): it may start while the kernel
// before it in the stream ends (programmatic stream serialisation; a chain
// of small kernels takes 1.5 instead of 2.1 us a launch).
static int launch_pdl(void *fn, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t s)
{
    if (grid.x == 0 || grid.y == 0) return 0;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = 1;
    PO_CK(cudaLaunchKernelExC(&c, fn, args));
    note_launches(1);
    return 0;
}

static int launch(void *fn, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t s)
{
    if (grid.x == 0 || grid.y == 0) return 0;
    PO_CK(cudaLaunchKernel(fn, grid, block, args, smem, s));
    note_launches(1);
    return 0;
}

static void timing_mark(cudaStream_t s, bool begin)
{
    if (!g_timing.on) return;
    std::lock_guard<std::mutex> lk(g_mu);
    const int slots = (int)g_timing.ev.size() / 2;
    if (slots == 0) return;
    if (begin) {
        if (g_timing.used >= slots) return;
        cudaEventRecord(g_timing.ev[2 * g_timing.used], s);
    } else {
        if (g_timing.used >= slots) return;
        cudaEventRecord(g_timing.ev[2 * g_timing.used + 1], s);
        ++g_timing.used;
    }
}

int timing_enable(int slots)
{
    std::lock_guard<std::mutex> lk(g_mu);
    for (cudaEvent_t e : g_timing.ev) cudaEventDestroy(e);
    g_timing.ev.clear();
    g_timing.used = 0;
    g_timing.on = slots > 0;
    for (int i = 0; i < 2 * std::max(slots, 0); ++i) {
        cudaEvent_t e;
        PO_CK(cudaEventCreate(&e));
        g_timing.ev.push_back(e);
    }
    return 0;
}

int timing_collect(float *ms, int max)
{
    std::lock_guard<std::mutex> lk(g_mu);
    int n = std::min(g_timing.used, max);
    for (int i = 0; i < n; ++i) {
        PO_CK(cudaEventSynchronize(g_timing.ev[2 * i + 1]));
        PO_CK(cudaEventElapsedTime(&ms[i], g_timing.ev[2 * i], g_timing.ev[2 * i + 1]));
    }
    g_timing.used = 0;
    return n;
}

// Persistent per-device error word, written by kernels that give up a wait.
static int *g_words[64] = {};

static int *error_word_impl(bool create)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_words[dev] && create) {
        if (cudaMalloc(&g_words[dev], sizeof(int)) != cudaSuccess) return nullptr;
        if (cudaMemset(g_words[dev], 0, sizeof(int)) != cudaSuccess) return nullptr;
    }
    return g_words[dev];
}

int *error_word() { return error_word_impl(true); }

int read_device_error(cudaStream_t s, int *code, int *words)
{
    // Both words: the allocating paths' (if it exists yet) and the
    // allocation-free entry's (if it has set up on this device). Nothing is
    // allocated here, on the device or page-locked, so callers of the
    // allocation-free entry can use it. They are read into the caller's
    // page-locked `words` (a copy into pageable memory waits for the stream and
    // costs 10 us more) or the stack, and cleared only where one is set.
    int local[2];
    int *got = words ? words : local;
    int *w[2] = {error_word_impl(false), static_status_word()};
    got[0] = got[1] = 0;
    for (int i = 0; i < 2; ++i)
        if (w[i]) PO_CK(cudaMemcpyAsync(&got[i], w[i], sizeof(int), cudaMemcpyDeviceToHost, s));
    PO_CK(cudaStreamSynchronize(s));
    *code = got[0] ? got[0] : got[1];
    bool cleared = false;
    for (int i = 0; i < 2; ++i)
        if (w[i] && got[i]) {
            PO_CK(cudaMemsetAsync(w[i], 0, sizeof(int), s));
            cleared = true;
        }
    if (cleared) PO_CK(cudaStreamSynchronize(s));
    return 0;
}

int validate(const RunArgs &a)
{
    if (a.mode < 0 || a.mode > 5) return fail(1, "mode must be 0..5 (JM EH JMEH EHP FF scalar)");
    if (a.ns < 0 || a.nt < 0) return fail(1, "negative size");
    if (a.ns > INT_MAX || a.nt > INT_MAX)
        return fail(1, "at most 2^31 - 1 sources and targets per call (indices are 32-bit on the device)");
    if (a.ns > 0 && a.gmode >= 0 && (a.ncx < 1 || a.ncy < 1)) return fail(1, "bad source grid shape");
    if (a.ns > 0 && a.gmode >= 0 && (long)a.ncx * a.ncy != a.ns)
        return fail(1, "ncx * ncy must equal the number of source points");
    if (!(a.t_dir == 1.0 || a.t_dir == -1.0)) return fail(1, "t_direction must be -1 (fwd) or +1 (bwd)");
    if (!(a.k > 0.0) || !std::isfinite(a.k)) return fail(1, "wavenumber k must be positive and finite");
    if (a.precision != 0 && a.precision != 1) return fail(1, "precision must be 0 (mixed) or 1 (fp64)");
    if (a.nt > 0 && ((a.ns > 0 && (!a.src7 || !a.cur)) || !a.tgt7 || !a.out)) return fail(1, "null buffer");
    return 0;
}

// The epilogue of nsplit chunks: one thread a target, eight from eight chunks
// on, and more where few targets (fewer blocks than SMs, each bound by its
// SM's FP64 additions) have many chunks: 25 targets, 630 chunks: 30 us with
// 32 threads, 18 us with 64.
static int launch_epilogue(long sms, int mode, int nacc, int nsplit, long nt, const double *part, const double *tgt7,
                           double t, double zeta_inv, double *out, cudaStream_t s)
{
    int groups = nsplit < 8 ? 1 : 8;
    if (nsplit >= 32 && nt <= sms * (kEpiThreads / 32)) groups = 32;
    if (nsplit >= 64 && nt <= sms * (kEpiThreads / 64)) groups = 64;
    const long per = kEpiThreads / groups;
    void *args[] = {&mode, &nacc, &nsplit, &nt, &part, &tgt7, &t, &zeta_inv, &out};
    return launch_pdl(epilogue_kernel(groups), dim3((unsigned)((nt + per - 1) / per)), dim3(kEpiThreads), args, 0, s);
}

int run_device(const RunArgs &a)
{
    if (int rc = validate(a)) return rc;
    if (a.nt == 0) return 0;
    cudaStream_t s = a.stream;
    if (a.precision == 0) {
        int *err = error_word();
        if (!err) return fail(2, "could not allocate the device error word");
        PoolScratch pool(s);
        return run_mixed(a, pool, err);
    }

    // ---- plain FP64
    const int kind = a.mode == kFF ? kKindFF : (a.mode == kScalar ? kKindScalar : kKindNF);
    const int nacc = kind == kKindScalar ? 2 : kAcc;
    const double pif = (double)3.14159265359f;   // the reference's float-literal pi
    const double pref = a.k * a.k / (4.0 * pif);
    const double c_l = (double)2.99792458e8f, mu0 = (double)1.2566370614e-6f;
    const double eps = a.epsilon * (1.0 / (mu0 * c_l * c_l));
    double zeta_inv = 1.0 / std::sqrt(mu0 / eps);
    // complex factor folded into each source's weighted current
    double fac_re = pref, fac_im = 0.0;
    if (kind == kKindFF) { fac_re = 0.0; fac_im = -pref; }
    if (kind == kKindScalar) fac_re = -pref;
    int rc = 0;
    const unsigned nblk_s = (unsigned)((a.ns + 255) / 256);
    long nt = a.nt, ns = a.ns;
    int mode = a.mode, gmode = a.gmode, ncx = a.ncx, ncy = a.ncy;
    double t = a.t_dir, k = a.k;
    const int scalar = kind == kKindScalar;
    const double *src7 = a.src7, *cur = a.cur, *tgt7 = a.tgt7;
    double *out = a.out;
    const bool has_m = !scalar && !a.m_zero;
    int rec = fp64_rec(kind, has_m);
    void *fk = fp64_kernel(kind, has_m);
    DeviceInfo *di = nullptr;
    int occ = 1;
    if ((rc = device_info(di)) || (rc = kernel_occupancy(di, fk, kThreadsD, 0, occ))) return rc;
    const long ntb = (nt + kThreadsD - 1) / kThreadsD;
    const long nsplit = load_split(ntb, ns, di->sms, occ, partial_cap(nt, nacc), kChunkD, kLoad64);
    const long tiles = std::max(1L, (ns + kChunkD - 1) / kChunkD);
    long chunk = (tiles + nsplit - 1) / nsplit * kChunkD;
    double *srcd = nullptr, *part = nullptr;
    PoolScratch sc(s);
    sc.get(&srcd, (size_t)std::max(ns, 1L) * rec);
    sc.get(&part, (size_t)nsplit * nacc * nt);
    if ((rc = sc.commit())) return rc;
    Wave64 w = wave64(k, t);
    void *pargs[] = {&ns, &src7, &cur, &gmode, &ncx, &ncy, &fac_re, &fac_im, (void *)&scalar, &rec, &srcd};
    if (ns > 0) rc = launch(pack_src_d_kernel(), dim3(nblk_s), dim3(256), pargs, 0, s);
    void *fargs[] = {&srcd, &ns, &chunk, &tgt7, &nt, &w, &part};
    timing_mark(s, true);
    if (!rc) rc = launch(fk, dim3((unsigned)ntb, (unsigned)nsplit), dim3(kThreadsD), fargs, 0, s);
    timing_mark(s, false);
    int nspl = (int)nsplit;
    if (!rc) rc = launch_epilogue(di->sms, mode, nacc, nspl, nt, part, tgt7, t, zeta_inv, out, s);
    return rc;
}

// CTAs of the box kernel for n points, or 0 where the frame comes from its cluster.
static int box_ctas(const DeviceInfo *di, long n)
{
    if (di->cluster && n <= kFrameClusterMax) return 0;
    return (int)std::max(1L, std::min((long)di->sms, (n + kFrameThreads - 1) / kFrameThreads));
}

// The frame of the sources' and nb targets' box (po_prep.cu), `zero` cleared.
// boxes: 48 bytes for each of the nbox CTAs, free until the frame is written.
static int launch_frame(const double *src7, long ns, const double *tgt7, long nb, double kappa, int centred, Frame *frame,
                        unsigned *zero, int nbox, long long *boxes, cudaStream_t s)
{
    if (nbox == 0) {
        void *args[] = {&src7, &ns, &tgt7, &nb, &kappa, &centred, &frame, &zero};
        return launch(frame_kernel(), dim3(kFrameCtas), dim3(kFrameThreads), args, 0, s);
    }
    void *bargs[] = {&src7, &ns, &tgt7, &nb, &boxes};
    if (int rc = launch(box_kernel(), dim3((unsigned)nbox), dim3(kFrameThreads), bargs, 0, s)) return rc;
    void *fargs[] = {&boxes, &nbox, &kappa, &centred, &frame, &zero};
    return launch_pdl(box_frame_kernel(), dim3(1), dim3(192), fargs, 0, s);
}

int mixed_prepare(const RunArgs &a, Scratch &sc, MixedPlan &p)
{
    DeviceInfo *di = nullptr;
    if (int rc = device_info(di)) return rc;
    p.kind = a.mode == kFF ? kKindFF : (a.mode == kScalar ? kKindScalar : kKindNF);
    p.nacc = p.kind == kKindScalar ? 2 : kAcc;
    const double pif = (double)3.14159265359f;   // the reference's float-literal pi
    const double pref = a.k * a.k / (4.0 * pif);
    p.kappa = a.k / (2.0 * 3.14159265358979323846);
    const double c_l = (double)2.99792458e8f, mu0 = (double)1.2566370614e-6f;
    const double eps = a.epsilon * (1.0 / (mu0 * c_l * c_l));
    p.zeta_inv = 1.0 / std::sqrt(mu0 / eps);
    p.ts = a.t_dir > 0 ? 1 : -1;
    // complex factor folded into each source's weighted current
    p.fac_re = pref;
    p.fac_im = 0.0;
    if (p.kind == kKindFF) { p.fac_re = 0.0; p.fac_im = -pref; }
    if (p.kind == kKindScalar) p.fac_re = -pref * p.kappa;
    const bool scalar = p.kind == kKindScalar;
    p.far = p.kind == kKindFF;
    p.has_m = !scalar && !a.m_zero;
    if (p.far && !p.has_m) p.nacc = 6;   // S_J alone
    const long ns = a.ns, nt = a.nt;
    p.tiles = std::max(1L, (ns + kTile - 1) / kTile);
    int rc = 0;
    if ((rc = sc.get(&p.frame, 1)) || (rc = sc.get(&p.tgtpk, (size_t)nt * 2))) return rc;
    if (!scalar) {
        p.band.cap = sc.band_cap(ns, nt);
        if ((rc = sc.get(&p.band.pairs, p.band.cap)) || (rc = sc.get(&p.band.count, 1))) return rc;
    }
    if (p.far) {
        // the far field's tiles along the sources' Hilbert order
        const long n1 = std::max(ns, 1L);
        cudaError_t e = ff_sort(nullptr, &p.sort_bytes, nullptr, nullptr, nullptr, nullptr, n1, a.stream);
        if (e != cudaSuccess) return fail(2, std::string("sort size query: ") + err_str(e));
        if ((rc = sc.get(&p.srcpk, (size_t)p.tiles * ff_tile4(p.has_m))) || (rc = sc.get(&p.keys, 2 * (size_t)n1)) ||
            (rc = sc.get(&p.order, 2 * (size_t)n1)) || (rc = sc.take(&p.sort_tmp, p.sort_bytes)))
            return rc;
    } else {
        // 11 float4 (scalar: 4) per two sources: no less than either layout's tiles take
        const size_t src_f4 = (size_t)((std::max(ns, 1L) + 1) / 2) * (scalar ? 4 : 11);
        if ((rc = sc.get(&p.srcpk, src_f4))) return rc;
    }
    // source chunks: balance waves over the SMs; the partials must fit the scratch left
    const long per_block = p.far ? 2L * kThreads : kThreads;   // targets per CTA
    p.ntb = (nt + per_block - 1) / per_block;
    const int occ = p.far ? di->occ_ff[p.ts > 0][p.has_m ? 1 : 0] : di->occ2[p.kind][p.ts > 0][p.has_m ? 1 : 0];
    const size_t room = std::min(sc.room(), (size_t)1 << 30);
    const long max_chunks = std::max(1L, (long)(room / ((size_t)p.nacc * nt * sizeof(double))));
    p.nsplit = load_split(p.ntb, ns, di->sms, occ, max_chunks, kTile, p.far ? kLoadFF : kLoadNF);
    p.sms = di->sms;
    p.few = p.ntb * p.nsplit <= 2L * di->sms;
    const long chunk_tiles = (p.tiles + p.nsplit - 1) / p.nsplit;
    p.chunk = chunk_tiles * (p.far ? 1 : kTile);   // tiles (far field) or sources per chunk
    if ((rc = sc.get(&p.part, (size_t)p.nsplit * p.nacc * nt)) || (rc = sc.commit())) return rc;
    // the boxes where the pack kernel writes the more numerous points' records (16 bytes a point and more)
    p.nbox = box_ctas(di, p.far ? ns : ns + nt);
    p.boxes = reinterpret_cast<long long *>(p.far || ns >= nt ? p.srcpk : p.tgtpk);
    return 0;
}

// Indices of the sources in the order of their keys, into i_out (k_in, i_in:
// ff_key_kernel's).
static int ff_order(long ns, unsigned long long *k_in, unsigned long long *k_out, int *i_in, int *i_out, void *tmp,
                    size_t tmp_bytes, cudaStream_t s)
{
    if (ns <= kFFRankMax) {
        int n = (int)ns;
        void *args[] = {&n, &k_in, &i_out};
        return launch_pdl(ff_rank_kernel(), dim3((unsigned)((n + 31) / 32)), dim3(256), args, 0, s);
    }
    const cudaError_t e = ff_sort(tmp, &tmp_bytes, k_in, k_out, i_in, i_out, ns, s);
    if (e != cudaSuccess) return fail(2, std::string("source sort: ") + err_str(e));
    note_launches(1);
    return 0;
}

int mixed_launch(const RunArgs &a, MixedPlan &p, int *err)
{
    cudaStream_t s = a.stream;
    long nt = a.nt, ns = a.ns;
    int mode = a.mode, gmode = a.gmode, ncx = a.ncx, ncy = a.ncy;
    double t = a.t_dir;
    const int scalar = p.kind == kKindScalar;
    const double *src7 = a.src7, *cur = a.cur, *tgt7 = a.tgt7;
    double *out = a.out;
    const unsigned nblk_s = (unsigned)((ns + 255) / 256);
    int rc = 0;
    // ---- frame: the box covers the sources, plus the targets in the near
    // field; the far field keeps the coordinate origin (its phase reference)
    long nb = p.far ? 0 : nt;
    int centred = p.far ? 0 : 1, farflag = p.far ? 1 : 0;
    rc = launch_frame(src7, ns, tgt7, nb, p.kappa, centred, p.frame, p.band.count, p.nbox, p.boxes, s);
    int boxes = !scalar && !p.has_m && ns > 0;   // the lit-tile proof serves the M = 0 kernels
    // ---- sources (near field, scalar) and targets
    long stiles = p.far || ns == 0 ? 0 : p.tiles;
    void *pkargs[] = {&ns, &src7, &cur, &gmode, &ncx, &ncy, &p.frame, &p.fac_re, &p.fac_im, &stiles,
                      &p.srcpk, &nt, &tgt7, &farflag, &p.tgtpk};
    if (!rc) rc = launch_pdl(pack_kernel(scalar, p.has_m), dim3((unsigned)(stiles + (nt + kTile - 1) / kTile)), dim3(kTile),
                             pkargs, 0, s);
    if (p.far && ns > 0) {
        // far-field sources in Hilbert order, packed tile by tile with their centres
        unsigned long long *k_in = p.keys, *k_out = p.keys + ns;
        int *i_in = p.order, *i_out = p.order + ns;
        void *kargs[] = {&ns, &src7, &p.frame, &k_in, &i_in};
        if (!rc) rc = launch_pdl(ff_key_kernel(), dim3(nblk_s), dim3(256), kargs, 0, s);
        if (!rc) rc = ff_order(ns, k_in, k_out, i_in, i_out, p.sort_tmp, p.sort_bytes, s);
        const int *ord = i_out;
        void *pargs[] = {&ns, &ord, &src7, &cur, &gmode, &ncx, &ncy, &p.frame, &p.fac_re, &p.fac_im, &p.srcpk};
        if (!rc) rc = launch_pdl(ff_pack_kernel(p.has_m), dim3((unsigned)p.tiles), dim3(kTile), pargs, 0, s);
    }
    const float4 *srcc = p.srcpk, *tgtc = p.tgtpk;
    long ntiles = ns > 0 ? p.tiles : 0;
    const int *sorted = p.order ? p.order + std::max(ns, 1L) : nullptr;   // far field: curve position -> source
    void *margs[] = {&srcc, p.far ? (void *)&ntiles : (void *)&ns, &p.chunk, &tgtc, &nt, &p.part, &err, &boxes,
                     &p.band, &ns, &sorted};
    timing_mark(s, true);
    if (!rc) {
        if (p.far)
            rc = launch_pdl(ff_kernel(p.ts, p.has_m, p.few), dim3((unsigned)p.ntb, (unsigned)p.nsplit),
                        dim3(kThreads), margs, ff_smem_bytes(p.has_m), s);
        else
            rc = launch_pdl(pk_kernel(p.kind, p.ts, p.has_m, p.few), dim3((unsigned)p.ntb, (unsigned)p.nsplit),
                        dim3(kThreads), margs, pk_smem_bytes(p.kind, p.has_m), s);
    }
    timing_mark(s, false);
    if (!rc && p.band.count && ns > 0) {
        // the near-tangent pairs, decided and summed in FP64 into chunk 0
        Wave64 w = wave64(a.k, t);
        void *xargs[] = {&p.band, &ns, &src7, &cur, &gmode, &ncx, &ncy, &p.fac_re, &p.fac_im, &nt, &tgt7, &w,
                         &p.part, &err};
        rc = launch_pdl(band_fixup_kernel(p.kind, p.has_m), dim3(kFixupBlocks), dim3(256), xargs, 0, s);
    }
    int nspl = (int)p.nsplit;
    if (!rc) rc = launch_epilogue(p.sms, mode, p.nacc, nspl, nt, p.part, tgt7, t, p.zeta_inv, out, s);
    if (!rc && a.extent_host) PO_CK_RC(cudaMemcpyAsync(a.extent_host, &p.frame->m, sizeof(double),
                                                       cudaMemcpyDeviceToHost, s));
    if (!rc && a.band_host && p.band.count)
        PO_CK_RC(cudaMemcpyAsync(a.band_host, p.band.count, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    return rc;
}

int run_mixed(const RunArgs &a, Scratch &sc, int *err)
{
    if (a.nt == 0) return 0;
    MixedPlan p;
    if (int rc = mixed_prepare(a, sc, p)) return rc;
    return mixed_launch(a, p, err);
}


// ---------------------------------------------------------------- adjoint

int run_adjoint(const AdjArgs &a)
{
    if (int rc = validate(a)) return rc;
    if (a.mode == kFF && a.grad_dt) return fail(1, "far-field targets are directions: no target displacement");
    if (a.nt > 0 && !a.cot) return fail(1, "null cotangent buffer");
    if (a.ns == 0) {
        // no sources: the target gradient is zero (the source gradients are empty)
        if (a.grad_dt && a.nt > 0) PO_CK(cudaMemsetAsync(a.grad_dt, 0, sizeof(double) * a.nt, a.stream));
        return 0;
    }
    if (a.nt == 0) {
        // no targets: every gradient is zero
        if (a.grad_cur)
            PO_CK(cudaMemsetAsync(a.grad_cur, 0, sizeof(double) * (a.mode == kScalar ? 2 : 12) * a.ns, a.stream));
        if (a.grad_ds) PO_CK(cudaMemsetAsync(a.grad_ds, 0, sizeof(double) * a.ns, a.stream));
        return 0;
    }
    DeviceInfo *di = nullptr;
    if (int rc = device_info(di)) return rc;
    int *err = error_word();
    if (!err) return fail(2, "could not allocate the device error word");

    const int kind = a.mode == kFF ? kKindFF : (a.mode == kScalar ? kKindScalar : kKindNF);
    const double pif = (double)3.14159265359f;
    const double pref = a.k * a.k / (4.0 * pif);
    const double kappa = a.k / (2.0 * 3.14159265358979323846);
    double fac_re = pref, fac_im = 0.0;
    if (kind == kKindFF) { fac_re = 0.0; fac_im = -pref; }
    if (kind == kKindScalar) fac_re = -pref * (a.precision == 0 ? kappa : 1.0);
    const int ts = a.t_dir > 0 ? 1 : -1;
    const bool far = kind == kKindFF;
    const bool has_m = kind != kKindScalar && !a.m_zero;
    const bool want_d = a.grad_ds != nullptr;
    cudaStream_t s = a.stream;
    long ns = a.ns, nt = a.nt;
    int mode = a.mode, gmode = a.gmode, ncx = a.ncx, ncy = a.ncy;
    double t = a.t_dir, k = a.k;
    const double *src7 = a.src7, *cur = a.cur, *tgt7 = a.tgt7, *cot = a.cot;
    double *grad_cur = a.grad_cur, *grad_ds = a.grad_ds, *grad_dt = a.grad_dt;
    const unsigned nblk_s = (unsigned)((ns + 255) / 256), nblk_t = (unsigned)((nt + 255) / 256);
    const bool want_c = grad_cur != nullptr, want_t = grad_dt != nullptr, fp64 = a.precision == 1;
    const int rows = adj_rows(kind, want_c, want_d);   // of the source-side partials
    // scalar sources: 2-row currents, S' in the record's J.x slot
    const int scalar = kind == kKindScalar ? 1 : 0;

    // ---- launch shape and scratch (one allocation)
    // FP64: a source per thread, targets streamed. Mixed near field and scalar:
    // the same on pairs of targets. Mixed far field: two sources per thread,
    // stages of kFFDirs directions. All fused: currents and displacements in
    // one pass.
    void *fk = fp64 ? adj_fp64_kernel(kind, has_m, want_c, want_d, want_t)
                    : (far ? ff_adj_kernel(ts, has_m, want_c, want_d)
                           : adj_pk_kernel(kind, ts, has_m, want_c, want_d, want_t));
    const int smem = fp64 ? 0 : (far ? ff_adj_smem_bytes(want_c, want_d)
                                     : adj_pk_smem_bytes(kind, has_m, want_c, want_d, want_t));
    const int threads = fp64 ? kThreadsD : (far ? ff_adj_threads() : kThreadsA);
    const int per_block = !fp64 && far ? kTile : threads;   // sources per block
    const long tile_t = fp64 ? kChunkD : (far ? kFFDirs : 2L * adj_pk_pairs_per_tile());
    int occ = 1, rc = 0;
    if ((rc = kernel_occupancy(di, fk, threads, smem, occ))) return rc;
    const long nsb = (ns + per_block - 1) / per_block;
    // FP64 target sums, a row of nt a source block: as many blocks a launch as
    // partial_cap has rows for (all of them but for the largest calls)
    const long nsb_l = fp64 && want_t ? std::min(nsb, partial_cap(nt, 1)) : nsb;
    const long cap = partial_cap(ns, std::max(rows, 1));
    const LoadCost load = fp64 ? kLoad64 : (kind == kKindScalar ? kLoadNF : kLoadAdj);
    const long split = !far || fp64
                           ? load_split(nsb_l, nt, di->sms, occ, cap, tile_t, load)
                           : choose_split(nsb, nt, (long)di->sms * occ, cap, tile_t);
    const long tiles_t = std::max(1L, (nt + tile_t - 1) / tile_t);
    const long per_chunk = (tiles_t + split - 1) / split;
    long chunk = !fp64 && far ? per_chunk : per_chunk * tile_t;   // stages (mixed far field) or targets

    PoolScratch sc(s);
    double *gam = nullptr, *eh = nullptr, *part = nullptr, *gt = nullptr, *srcd = nullptr, *trecd = nullptr;
    double *tsum = nullptr;
    Frame *frame = nullptr;
    float4 *srcpk = nullptr;
    float *trec = nullptr;
    unsigned long long *keys = nullptr;
    int *ord = nullptr;
    void *sort_tmp = nullptr;
    size_t sort_bytes = 0;
    BandList band{nullptr, nullptr, 0};   // near-tangent pairs (mixed, not the scalar kind)
    const long npair = (nt + 1) / 2, ntile_s = (ns + kTile - 1) / kTile;
    long nstage = (nt + kFFDirs - 1) / kFFDirs;
    int rec = fp64_rec(kind, has_m), rec4 = far ? 0 : adj_pk_rec4(has_m, want_t);
    sc.get(&gam, (size_t)12 * nt);
    if (a.mode == kEHP) sc.get(&eh, (size_t)12 * nt);
    sc.get(&part, (size_t)split * rows * ns);
    if (want_t) sc.get(&gt, (size_t)nt);
    if (fp64) {
        sc.get(&srcd, (size_t)ns * rec);
        sc.get(&trecd, (size_t)nt * adj64_rec(kind));
        if (want_t) sc.get(&tsum, (size_t)nsb_l * nt);
    } else {
        sc.get(&frame, 1);
        if (kind != kKindScalar) {
            band.cap = band_cap_for(ns, nt);
            sc.get(&band.pairs, band.cap);
            sc.get(&band.count, 1);
        }
        if (far) {
            cudaError_t e = ff_sort(nullptr, &sort_bytes, nullptr, nullptr, nullptr, nullptr, ns, s);
            if (e != cudaSuccess) return fail(2, std::string("sort size query: ") + err_str(e));
            sc.get(&keys, 2 * (size_t)ns);
            sc.get(&ord, 2 * (size_t)ns);
            sc.take(&sort_tmp, sort_bytes);
            sc.get(&srcpk, (size_t)ntile_s * ff_tile4(has_m));
            sc.get(&trec, (size_t)nstage * ff_adj_stage4() * 4);
        } else {
            sc.get(&srcpk, (size_t)nsb * threads * kRec);
            sc.get(&trec, (size_t)npair * rec4 * 4);
        }
    }
    if ((rc = sc.commit())) return rc;

    if (a.mode == kEHP) {
        // EHP is nonlinear in the target's fields: the EH forward at the same
        // inputs and precision, then the EHP map's vector-Jacobian product
        // there (po_adj_ehp_cot_kernel) gives the EH adjoint's cotangents
        RunArgs fa = a;
        fa.mode = kEH;
        fa.out = eh;
        fa.extent_host = nullptr;
        fa.band_host = nullptr;
        rc = run_device(fa);
        const double c_l = (double)2.99792458e8f, mu0 = (double)1.2566370614e-6f;
        double zi = 1.0 / std::sqrt(mu0 / (a.epsilon * (1.0 / (mu0 * c_l * c_l))));
        void *eargs[] = {&nt, &cot, &eh, &tgt7, &zi, &gam};
        if (!rc) rc = launch(adj_ehp_cot_kernel(), dim3((unsigned)((nt + 127) / 128)), dim3(128), eargs, 0, s);
        mode = kEH;
        cot = gam;
    }
    int nspl = (int)split;
    double dsc = 1.0, tsc = 1.0;   // gradient per mm from the kernels' units
    const int *curve = nullptr;   // far field: curve position -> source

    if (fp64) {
        dsc = far ? 1.0 : -1.0;
        if (a.mode != kEHP) {
            void *cargs[] = {&mode, &nt, &cot, &tgt7, &t, &gam};
            if (!rc) rc = launch(adj_cot_kernel(), dim3(nblk_t), dim3(256), cargs, 0, s);
        }
        Wave64 w = wave64(k, t);
        void *pargs[] = {&ns, &src7, &cur, &gmode, &ncx, &ncy, &fac_re, &fac_im, (void *)&scalar, &rec, &srcd};
        if (!rc) rc = launch(pack_src_d_kernel(), dim3(nblk_s), dim3(256), pargs, 0, s);
        void *tpargs[] = {&nt, &tgt7, &gam, &trecd};
        if (!rc) rc = launch(adj_pack_tgt_d_kernel(kind), dim3(nblk_t), dim3(256), tpargs, 0, s);
        for (long first = 0; first < nsb && !rc; first += nsb_l) {
            long blocks = std::min(nsb_l, nsb - first);
            void *sargs[] = {&srcd, &ns, &first, &trecd, &nt, &chunk, &w, &part, &tsum};
            timing_mark(s, true);
            rc = launch(fk, dim3((unsigned)blocks, (unsigned)split), dim3((unsigned)threads), sargs, 0, s);
            timing_mark(s, false);
            int add = first > 0;
            void *gargs[] = {&blocks, &nt, &tsum, &add, &gt};
            if (!rc && want_t)
                rc = launch_pdl(adj_tsum_kernel(), dim3((unsigned)((nt + 31) / 32)), dim3(256), gargs, 0, s);
        }
    } else {
        dsc = far ? kappa : -kappa;
        tsc = kappa;
        long nb = far ? 0 : nt;
        // the boxes where the pack kernels write the more numerous points' records
        long long *boxes = reinterpret_cast<long long *>(far || ns >= nt ? (void *)srcpk : (void *)trec);
        if (!rc) rc = launch_frame(src7, ns, tgt7, nb, kappa, far ? 0 : 1, frame, band.count, box_ctas(di, ns + nb), boxes, s);
        if (far) {
            // sources in Hilbert order, in the forward's tile records: one adjoint
            // CTA per tile, whose centre's phase goes into the cotangents
            void *p2args[] = {&nt, &tgt7, &cot, &t, &gam, &trec};
            if (!rc) rc = launch_pdl(ff_pack_cot_kernel(), dim3((unsigned)nstage), dim3(kFFDirs), p2args, 0, s);
            unsigned long long *k_in = keys, *k_out = keys + ns;
            int *i_in = ord, *i_out = ord + ns;
            void *kargs[] = {&ns, &src7, &frame, &k_in, &i_in};
            if (!rc) rc = launch_pdl(ff_key_kernel(), dim3(nblk_s), dim3(256), kargs, 0, s);
            if (!rc) rc = ff_order(ns, k_in, k_out, i_in, i_out, sort_tmp, sort_bytes, s);
            curve = i_out;
            void *fpargs[] = {&ns, &curve, &src7, &cur, &gmode, &ncx, &ncy, &frame, &fac_re, &fac_im, &srcpk};
            if (!rc) rc = launch_pdl(ff_pack_kernel(has_m), dim3((unsigned)ntile_s), dim3(kTile), fpargs, 0, s);
        } else {
            long sblk = nsb;
            double *gam_out = a.mode == kEHP ? nullptr : gam;   // EHP: the cotangents are gam already
            void *pargs[] = {&ns, &src7, &cur, &gmode, &ncx, &ncy, &frame, &fac_re, &fac_im, (void *)&scalar, &sblk,
                             &srcpk, &mode, &nt, &tgt7, &cot, &t, &gam_out, &rec4, &trec, &gt};
            if (!rc) rc = launch_pdl(adj_pack_kernel(), dim3((unsigned)(sblk + (2 * npair + 127) / 128)), dim3(128),
                                     pargs, 0, s);
        }
        const float4 *srcc = srcpk, *trc = reinterpret_cast<const float4 *>(trec);
        void *nfargs[] = {&srcc, &ns, &trc, &nt, &chunk, &part, &gt, &err, &band};
        void *ffargs[] = {&srcc, &ns, &trc, &nstage, &chunk, &nt, &part, &err, &band, &curve};
        timing_mark(s, true);
        if (!rc) rc = launch_pdl(fk, dim3((unsigned)nsb, (unsigned)split), dim3((unsigned)threads),
                                 far ? ffargs : nfargs, smem, s);
        timing_mark(s, false);
        if (!rc && band.count) {
            // the near-tangent pairs, decided and summed in FP64 into chunk 0 (and gt)
            double inv_kappa = 1.0 / kappa;
            Wave64 w = wave64(k, t);
            int wc = want_c, wd = want_d;
            void *xargs[] = {&band, &ns, &src7, &cur, &gmode, &ncx, &ncy, &fac_re, &fac_im, &nt, &tgt7, &gam, &w,
                             &inv_kappa, &wc, &wd, &part, &gt, &err};
            rc = launch_pdl(adj_band_fixup_kernel(kind, want_t), dim3(kFixupBlocks), dim3(256), xargs, 0, s);
        }
    }
    long nt_e = want_t ? nt : 0;
    const int groups = nspl >= 8 && ns <= (long)di->sms * kEpiThreads ? 8 : 1;   // fewer blocks than SMs: share the chunks
    const long per = kEpiThreads / groups;
    long nblk_e = rows > 0 ? (ns + per - 1) / per : 0;
    void *eargs[] = {(void *)&kind, &nspl, &ns, &part, &src7, &gmode, &ncx, &ncy, &fac_re, &fac_im, &dsc,
                     &grad_cur, &grad_ds, &nblk_e, &nt_e, &gt, &tsc, &grad_dt};
    if (!rc) rc = launch_pdl(adj_epilogue_kernel(groups, rows),
                             dim3((unsigned)(nblk_e + (nt_e + kEpiThreads - 1) / kEpiThreads)), dim3(kEpiThreads),
                             eargs, 0, s);
    if (!rc && a.extent_host && frame) PO_CK_RC(cudaMemcpyAsync(a.extent_host, &frame->m, sizeof(double),
                                                                cudaMemcpyDeviceToHost, s));
    if (!rc && a.band_host && band.count)
        PO_CK_RC(cudaMemcpyAsync(a.band_host, band.count, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    return rc;
}

}  // namespace po
