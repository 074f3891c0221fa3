// A CUDA runtime of the test's own and stand-ins for the library's kernel
// launchers, linked with the library's host code (api.cpp, plan.cpp): nothing
// runs, every copy and launch only records which memory it reads and writes,
// on which stream.  Streams, events and host waits carry vector clocks, so two
// accesses to the same bytes, one of them a write, with nothing that orders one
// before the other, are found whatever the timing would have been.
//
// As the runtime documents it: streams do not wait for each other or for the
// default stream (the library's are non-blocking), cudaMemcpy from pageable
// memory may return before its device write, cudaMemset always may, cudaFree
// waits for the device.
//
// usage: call_order <scenario> [call [call ...]]   prints the conflicts found
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include "sarbp_internal.h"

// ------------------------------------------------------------ vector clocks
namespace {
using Clock = std::map<int, long>;
void join(Clock &a, const Clock &b) {
    for (auto &kv : b) a[kv.first] = std::max(a[kv.first], kv.second);
}
struct Access {
    const char *lo, *hi;
    bool write;
    int stream;
    long time;
    const char *what;
};
Clock g_host;
std::map<int, Clock> g_streams;
std::map<int, Clock> g_events;
std::map<char *, size_t> g_device;
std::vector<Access> g_log;
int g_ids = 0, g_conflicts = 0;
bool g_fail_bp = false;
std::vector<size_t> g_uploads;  // bytes of each host-to-device copy
int g_frees = 0;

int id_of(const void *h) { return (int)(intptr_t)h; }  // stream and event handles are small integers
int begin_op(int stream) {
    Clock &c = g_streams[stream];
    join(c, g_host);
    ++c[stream];
    return stream;
}
void access(int stream, const char *what, const void *p, size_t bytes, bool write) {
    if (!p || !bytes) return;
    const char *lo = static_cast<const char *>(p), *hi = lo + bytes;
    const Clock &c = g_streams[stream];
    for (const Access &a : g_log) {
        if (a.hi <= lo || hi <= a.lo || !(a.write || write)) continue;
        auto it = c.find(a.stream);
        if (it != c.end() && it->second >= a.time) continue;
        ++g_conflicts;
        std::printf("conflict: %s (%s) on stream %d with %s (%s) on stream %d\n", what, write ? "writes" : "reads",
                    stream, a.what, a.write ? "writes" : "reads", a.stream);
    }
    g_log.push_back({lo, hi, write, stream, c.at(stream), what});
}
void host_waits(int stream) { join(g_host, g_streams[stream]); }
bool on_device(const void *p) {
    auto it = g_device.upper_bound((char *)p);
    if (it == g_device.begin()) return false;
    --it;
    return (char *)p < it->first + it->second;
}
struct Op {
    int s;
    const char *what;
    Op(cudaStream_t stream, const char *w) : s(begin_op(id_of(stream))), what(w) {}
    void r(const void *p, size_t n) { access(s, what, p, n, false); }
    void w(const void *p, size_t n) { access(s, what, p, n, true); }
};
}  // namespace

// -------------------------------------------------------------- the runtime
extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)(intptr_t)++g_ids; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)(intptr_t)++g_ids; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    begin_op(id_of(s));
    g_events[id_of(e)] = g_streams[id_of(s)];
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { join(g_host, g_events[id_of(e)]); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    begin_op(id_of(s));
    join(g_streams[id_of(s)], g_events[id_of(e)]);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { host_waits(id_of(s)); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
    for (auto &kv : g_streams) join(g_host, kv.second);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = std::malloc(n);
    if (!*p) return cudaErrorMemoryAllocation;
    g_device[(char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    ++g_frees;
    cudaDeviceSynchronize();
    auto it = g_device.find((char *)p);
    if (it == g_device.end()) return cudaErrorInvalidValue;
    std::vector<Access> keep;  // the address may come back as another buffer
    for (const Access &a : g_log)
        if (a.hi <= it->first || a.lo >= it->first + it->second) keep.push_back(a);
    g_log.swap(keep);
    g_device.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::memset(a, 0, sizeof *a);
    a->type = on_device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    Op op(s, "copy");
    if (on_device(src)) op.r(src, n);
    if (on_device(d)) op.w(d, n);
    if (on_device(d) && !on_device(src)) g_uploads.push_back(n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *src, size_t n, cudaMemcpyKind k) {
    cudaMemcpyAsync(d, src, n, k, nullptr);
    if (k == cudaMemcpyDeviceToHost) host_waits(0);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int, size_t n, cudaStream_t s) {
    Op(s, "memset").w(d, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
}

// ------------------------------------------------------------- the launchers
namespace sarbp {
static size_t esize(int storage) { return storage == SARBP_STORE_C64 ? 8 : 4; }
bool rc_size_supported(int n) { return n >= 2 && n <= 32768; }
cudaError_t prepare_rc_kernels(const RcPlan &) { return cudaSuccess; }
cudaError_t launch_rc_forward(const RcPlan &p, const float2 *echo, const float2 *filt, const float2 *etab, float2 *spec,
                              float *scale, cudaStream_t s) {
    Op op(s, "forward transform");
    op.r(echo, 8ull * p.np * p.ns);
    op.r(filt, 8ull * p.nfft);
    op.r(etab, 8ull * rc_etab_size(p.L, p.nfft));
    op.w(spec, 8ull * p.np * p.nfft);
    if (p.nfft == 32768) op.w(p.bound2, 8ull * p.np);
    else op.w(scale, 4ull * p.np);
    return cudaSuccess;
}
cudaError_t launch_rc_inverse(const RcPlan &p, const float2 *spec, const float2 *etab, const float *scale, void *out,
                              cudaStream_t s) {
    Op op(s, "inverse transform");
    op.r(spec, 8ull * p.np * p.nfft);
    op.r(etab, 8ull * rc_etab_size(p.L, p.nfft));
    if (p.nfft == 32768) op.r(p.bound2, 8ull * p.np);
    op.w(scale, 4ull * p.np);
    op.w(out, esize(p.storage) * p.np * p.nbins);
    return cudaSuccess;
}
static void read_pulses(Op &op, const BpPlan &p) {
    op.r(p.rc, esize(p.storage) * p.np * p.nbins);
    op.r(p.scale, 4ull * p.np);
    op.r(p.apc, 24ull * p.np);
    op.r(p.drange, 8ull * p.np);
    op.r(p.dphase, 8ull * p.np);
    op.w(p.pref, 32ull * p.np);
}
cudaError_t launch_bp(const BpPlan &p, cudaStream_t s, int *) {
    Op op(s, "back-projection");
    read_pulses(op, p);
    if (g_fail_bp) return cudaErrorLaunchOutOfResources;  // with the references queued
    const size_t npix = (size_t)p.g.nx * p.g.ny;
    if (p.segments > 1) op.w(p.partial, 8 * npix * p.segments);
    op.w(p.image, 8 * npix);
    return cudaSuccess;
}
size_t bp_tiles(const BpPlan &p) { return (size_t)((p.g.nx + 31) / 32) * ((p.g.ny + 8 * p.pix - 1) / (8 * p.pix)); }
cudaError_t bp_occupancy(const BpPlan &, int *n) { *n = 2; return cudaSuccess; }
cudaError_t launch_project(const BpPlan &p, double2 *out, cudaStream_t s, int *) {
    Op op(s, "projection");
    read_pulses(op, p);
    op.r(p.weight, 8ull * p.g.nx * p.g.ny);
    op.w(p.proj, 8 * bp_tiles(p) * p.np);
    op.w(out, 16ull * p.np);
    return cudaSuccess;
}
void bp_extremes_state_init(unsigned long long (&state)[6]) { std::memset(state, 0, sizeof state); }
cudaError_t launch_bp_extremes(const double *apc, int np, const sarbp_grid &, unsigned long long *state,
                               unsigned long long *result, unsigned long long seq, cudaStream_t s) {
    Op op(s, "planning extremes");
    op.r(apc, 24ull * np);
    op.w(state, 48);
    const double v[4] = {25e6, 26e6, 0.1, 0.1};  // squared ranges, cosines
    std::memcpy(result, v, sizeof v);
    result[4] = 0;
    result[5] = seq;
    host_waits(op.s);  // the library polls `result`, which the kernel writes last
    return cudaSuccess;
}
void bp_tile_dims(int pix, int *tx, int *ty) { *tx = 32; *ty = 8 * pix; }
size_t bp_smem_bytes(int storage, int win, int chunk) { return (size_t)chunk * win * (32 + 3 * esize(storage)) + 8192; }
int bp_max_chunk() { return 16; }
int sharpness_blocks(size_t) { return 8; }
cudaError_t launch_sharpness_weight(const float2 *img, size_t n, float2 *w, double *partial, cudaStream_t s) {
    Op op(s, "sharpness");
    op.r(img, 8 * n);
    op.w(w, 8 * n);
    op.w(partial, 64);
    return cudaSuccess;
}
bool dft_size_supported(int n) { return n >= 1 && n <= 8192; }
int dft_bluestein_size(int n) {
    if ((n & (n - 1)) == 0) return 0;
    int m = 1;
    while (m < 2 * n - 1) m *= 2;
    return m;
}
static void read_dft(Op &op, const DftPlan &p) {
    op.r(p.etab, 8ull * rc_etab_size(1, p.m ? p.m : p.n));
    if (p.m) {
        op.r(p.chirp, 8ull * p.n);
        op.r(p.kfwd, 8ull * p.m);
        op.r(p.kinv, 8ull * p.m);
    }
}
cudaError_t launch_dft_rows(const DftPlan &p, float2 *d, int rows, long long ld, bool, float, cudaStream_t s,
                            const DftIo &io) {
    Op op(s, "row transforms");
    read_dft(op, p);
    op.r(io.src, 8ull * rows * io.src_cols);
    op.r(io.rowmul, 8ull * rows);
    op.w(d, 8ull * rows * ld);
    return cudaSuccess;
}
bool dft_cols_supported(const DftPlan &p) { return p.m == 0 && p.n >= 512 && p.n <= 4096; }
cudaError_t launch_dft_cols(const DftPlan &p, const float2 *in, float2 *out, int ncols, bool, float, cudaStream_t s) {
    Op op(s, "column transforms");
    read_dft(op, p);
    op.r(in, 8ull * p.n * ncols);
    op.w(out, 8ull * p.n * ncols);
    return cudaSuccess;
}
cudaError_t launch_transpose(const float2 *in, float2 *out, int rows, int cols, cudaStream_t s) {
    Op op(s, "transpose");
    op.r(in, 8ull * rows * cols);
    op.w(out, 8ull * rows * cols);
    return cudaSuccess;
}
cudaError_t launch_wk_pad(const float2 *echo, int na, int nr, const float2 *rowmul, int, int, int NA, int NR,
                          float2 *out, cudaStream_t s) {
    Op op(s, "padding");
    op.r(echo, 8ull * na * nr);
    op.r(rowmul, 8ull * NA);
    op.w(out, 8ull * NA * NR);
    return cudaSuccess;
}
size_t wk_stolt_smem(int NR) { return 12ull * NR; }
cudaError_t launch_wk_stolt_ff(const float2 *in, float2 *out, int NA, int NR, const float *c, const float2 *ip,
                               const float2 *q, double, double, int, cudaStream_t s) {
    Op op(s, "Stolt mapping");
    op.r(c, 4ull * NR);
    op.r(ip, 8ull * NR);
    op.r(q, 8ull * NA);
    op.r(in, 8ull * NA * NR);
    op.w(out, 8ull * NA * NR);
    return cudaSuccess;
}
cudaError_t launch_wk_stolt(const float2 *in, float2 *out, int NA, int NR, const double *f2, const double *, const double *,
                            const double *, double, double, double, int, cudaStream_t s) {
    Op op(s, "Stolt mapping");
    op.r(f2, 8ull * (3 * NR + NA));
    op.r(in, 8ull * NA * NR);
    op.w(out, 8ull * NA * NR);
    return cudaSuccess;
}
cudaError_t launch_ceos_decode(const unsigned char *raw, const CeosGeom &g, const CeosGains &, float2 *echo, short *agc,
                               cudaStream_t s) {
    Op op(s, "CEOS decode");
    op.r(raw, (size_t)g.nlines * g.line_bytes);
    op.w(echo, 8ull * g.nlines * g.ncells);
    op.w(agc, 2ull * g.nlines);
    return cudaSuccess;
}
cudaError_t launch_echo_synth(const double *apc, int np, int ns, const sarbp_target *tg, int nt, double, double, double,
                              double, double, double, double, float2 *echo, double *power, cudaStream_t s) {
    Op op(s, "echo synthesis");
    op.r(apc, 24ull * np);
    op.r(tg, sizeof(sarbp_target) * nt);
    op.w(echo, 8ull * np * ns);
    op.w(power, 8);
    return cudaSuccess;
}
cudaError_t launch_echo_noise(float2 *echo, int64_t n, const double *power, double, uint64_t, cudaStream_t s) {
    Op op(s, "echo noise");
    op.w(echo, 8 * n);
    op.r(power, 8);
    return cudaSuccess;
}
cudaError_t launch_ref_echo(float2 *, const float *, const float *, const float *, const sarbp_ref_params &, int, int,
                            cudaStream_t) { return cudaSuccess; }
cudaError_t run_issue_probe(int, double *, double *, cudaStream_t) { return cudaSuccess; }
}  // namespace sarbp

// ------------------------------------------------------------------ the calls
namespace {
template <class T>
T *device(size_t n) {  // a caller's buffer
    void *p = nullptr;
    cudaMalloc(&p, n * sizeof(T));
    return static_cast<T *>(p);
}
sarbp_radar radar(double kr = 1e13, int upsample = 8) {
    sarbp_radar r{};
    r.c = 3e8; r.fc = 5.3e9; r.fs = 120e6; r.kr = kr; r.tp = 10e-6; r.tc = 5e-6; r.t_rec0 = 3e-5;
    r.upsample = upsample;
    return r;
}
sarbp_grid grid(int n) {
    sarbp_grid g{};
    g.origin[1] = 5000.0;
    g.ux[1] = g.uy[0] = 0.25;
    g.nx = g.ny = n;
    return g;
}
constexpr int kNp = 600, kNs = 800, kN = 96;
sarbp_rc_view view(const sarbp_radar &r, const void *data, const float *scale) {
    sarbp_rc_layout lay;
    sarbp_rc_layout_get(&r, kNs, &lay);
    sarbp_rc_view v{};
    v.data = data;
    v.scale = scale;
    v.storage = scale ? SARBP_STORE_C32H : SARBP_STORE_C64;
    v.np = kNp;
    v.nbins = lay.nbins;
    v.t0_bins = lay.t0_bins;
    v.bin_rate = lay.bin_rate;
    return v;
}
sarbp_wk_params wk_params(double r0 = 988647.462) {
    sarbp_wk_params w{};
    w.fr = 32317000.0; w.prf = 1256.98; w.f0 = 5.3e9; w.r0 = r0; w.kr = -721350000000.0; w.c = 299790000.0;
    w.vr = 7062.0; w.f_nc = -6900.0; w.taps = 6;
    return w;
}

// Every call kind by name, with buffers of its own; host kinds pass host memory.
// `other`: other parameters than the default ones.
using Call = std::function<sarbp_status(sarbp_ctx *, cudaStream_t, bool other)>;
template <class T>
T *host(size_t n) { return static_cast<T *>(std::calloc(n, sizeof(T))); }

sarbp_status range_compress(sarbp_ctx *c, cudaStream_t s, bool other, int storage, bool host_echo, int np, int ns,
                            int upsample = 8) {
    const sarbp_radar r = radar(other ? 9e12 : 1e13, upsample);
    const size_t out = (size_t)np * upsample * ns;
    auto *echo = host_echo ? host<sarbp_complex64>((size_t)np * ns) : device<sarbp_complex64>((size_t)np * ns);
    float *scale = storage == SARBP_STORE_C32H ? device<float>(np) : nullptr;
    return sarbp_range_compress(c, &r, echo, np, ns, storage, device<char>(out * 8), scale, s);
}
sarbp_status backproject(sarbp_ctx *c, cudaStream_t s, bool fp16, bool host_side) {
    const sarbp_radar r = radar();
    const size_t bytes = (size_t)kNp * 8 * kNs * (fp16 ? 4 : 8);
    const void *rows = host_side ? host<char>(bytes) : device<char>(bytes);
    float *scale = !fp16 ? nullptr : host_side ? host<float>(kNp) : device<float>(kNp);
    const sarbp_rc_view v = view(r, rows, scale);
    const sarbp_grid g = grid(kN);
    const double *apc = host_side ? host<double>(3 * kNp) : device<double>(3 * kNp);
    const sarbp_pulse_corr corr{host_side ? host<double>(kNp) : device<double>(kNp), nullptr};
    auto *img = host_side ? host<sarbp_complex64>(kN * kN) : device<sarbp_complex64>(kN * kN);
    return sarbp_backproject_ex(c, &r, &v, apc, &g, fp16 ? SARBP_MODE_FP16STORE : SARBP_MODE_SPLIT, &corr, img, 0, s);
}
sarbp_status project(sarbp_ctx *c, cudaStream_t s, bool host_side) {
    const sarbp_radar r = radar();
    const sarbp_rc_view v = view(r, device<char>((size_t)kNp * 8 * kNs * 8), nullptr);
    const sarbp_grid g = grid(kN);
    auto *w = host_side ? host<sarbp_complex64>(kN * kN) : device<sarbp_complex64>(kN * kN);
    double *out = host_side ? host<double>(2 * kNp) : device<double>(2 * kNp);
    return sarbp_project_weighted(c, &r, &v, device<double>(3 * kNp), &g, SARBP_MODE_SPLIT, nullptr, w, out, s);
}
sarbp_status image(sarbp_ctx *c, cudaStream_t s, bool other, int mode, bool host_side, int np = kNp) {
    const sarbp_radar r = radar(other ? 9e12 : 1e13);
    const sarbp_grid g = grid(kN);
    auto *echo = host_side ? host<sarbp_complex64>((size_t)np * kNs) : device<sarbp_complex64>((size_t)np * kNs);
    const double *apc = host_side ? host<double>(3 * np) : device<double>(3 * np);
    auto *img = host_side ? host<sarbp_complex64>(kN * kN) : device<sarbp_complex64>(kN * kN);
    return sarbp_image(c, &r, echo, np, kNs, apc, &g, mode, img, s);
}
sarbp_status ceos(sarbp_ctx *c, cudaStream_t s, bool other, bool host_side) {
    sarbp_ceos_layout l{};
    l.file_header = 0; l.header = 12; l.aux = 50; l.cells = 300; l.replica = 100; l.lines_per_block = 8;
    l.replica_line = 1; l.agc_byte = 7; l.gain = other ? 2.0f : 1.5f;
    const uint64_t bytes = 4 * (100 + 8 * 662);
    auto *raw = host_side ? host<uint8_t>(bytes) : device<uint8_t>(bytes);
    auto *echo = host_side ? host<sarbp_complex64>(32 * 300) : device<sarbp_complex64>(32 * 300);
    return sarbp_ceos_decode(c, raw, bytes, &l, 0, 32, 0, 300, 1, echo, nullptr, s);
}
sarbp_status synth(sarbp_ctx *c, cudaStream_t s, bool host_side) {
    const sarbp_radar r = radar();
    const double *apc = host_side ? host<double>(3 * kNp) : device<double>(3 * kNp);
    auto *tg = host_side ? host<sarbp_target>(4) : device<sarbp_target>(4);
    auto *echo = host_side ? host<sarbp_complex64>(kNp * kNs) : device<sarbp_complex64>(kNp * kNs);
    return sarbp_synthesize_echo(c, &r, apc, kNp, kNs, tg, 4, 20.0, 1, echo, s);
}

const std::map<std::string, Call> kCalls = {
    {"rc", [](sarbp_ctx *c, cudaStream_t s, bool o) { return range_compress(c, s, o, SARBP_STORE_C64, false, kNp, kNs); }},
    {"rc_fp16", [](sarbp_ctx *c, cudaStream_t s, bool o) { return range_compress(c, s, o, SARBP_STORE_C32H, false, kNp, kNs); }},
    {"rc_32768", [](sarbp_ctx *c, cudaStream_t s, bool o) { return range_compress(c, s, o, SARBP_STORE_C32H, false, 3, 20000, 2); }},
    {"rc_host", [](sarbp_ctx *c, cudaStream_t s, bool o) { return range_compress(c, s, o, SARBP_STORE_C64, true, 3000, kNs); }},
    {"bp", [](sarbp_ctx *c, cudaStream_t s, bool) { return backproject(c, s, false, false); }},
    {"bp_fp16", [](sarbp_ctx *c, cudaStream_t s, bool) { return backproject(c, s, true, false); }},
    {"bp_host", [](sarbp_ctx *c, cudaStream_t s, bool) { return backproject(c, s, true, true); }},
    {"project", [](sarbp_ctx *c, cudaStream_t s, bool) { return project(c, s, false); }},
    {"project_host", [](sarbp_ctx *c, cudaStream_t s, bool) { return project(c, s, true); }},
    {"autofocus", [](sarbp_ctx *c, cudaStream_t s, bool) {
         const sarbp_radar r = radar();
         const sarbp_rc_view v = view(r, device<char>((size_t)kNp * 8 * kNs * 8), nullptr);
         const sarbp_grid g = grid(kN);
         return sarbp_autofocus(c, &r, &v, device<double>(3 * kNp), &g, SARBP_MODE_SPLIT, 1, nullptr, host<double>(kNp),
                                host<sarbp_complex64>(kN * kN), nullptr, s);
     }},
    {"image", [](sarbp_ctx *c, cudaStream_t s, bool o) { return image(c, s, o, SARBP_MODE_SPLIT, false); }},
    {"image_fp16", [](sarbp_ctx *c, cudaStream_t s, bool o) { return image(c, s, o, SARBP_MODE_FP16STORE, false); }},
    {"image_host", [](sarbp_ctx *c, cudaStream_t s, bool o) { return image(c, s, o, SARBP_MODE_FP16STORE, true); }},
    {"plan", [](sarbp_ctx *c, cudaStream_t, bool) {
         const sarbp_radar r = radar();
         const sarbp_rc_view v = view(r, nullptr, nullptr);
         const sarbp_grid g = grid(kN);
         sarbp_bp_plan_info info;
         return sarbp_bp_plan(c, &r, &v, host<double>(3 * kNp), &g, SARBP_MODE_SPLIT, 0, &info);
     }},
    {"dft", [](sarbp_ctx *c, cudaStream_t s, bool o) { return sarbp_dft(c, device<sarbp_complex64>(20 * 999), 20, o ? 999 : 512, 0, s); }},
    {"dft_host", [](sarbp_ctx *c, cudaStream_t s, bool o) { return sarbp_dft(c, host<sarbp_complex64>(20 * 999), 20, o ? 999 : 512, 0, s); }},
    {"dft2d", [](sarbp_ctx *c, cudaStream_t s, bool o) { return sarbp_dft2d(c, device<sarbp_complex64>(70 * 100), o ? 66 : 70, 100, 0, s); }},
    {"wk", [](sarbp_ctx *c, cudaStream_t s, bool o) {
         const sarbp_wk_params w = wk_params(o ? 9e5 : 988647.462);
         int32_t na, nr;
         sarbp_wk_padded_size(48, 60, &na, &nr);
         return sarbp_wk_image(c, &w, device<sarbp_complex64>(48 * 60), 48, 60, device<sarbp_complex64>(na * nr), s);
     }},
    {"wk_preprocess", [](sarbp_ctx *c, cudaStream_t s, bool o) {
         const sarbp_wk_params w = wk_params(o ? 9e5 : 988647.462);
         int32_t na, nr;
         sarbp_wk_padded_size(48, 60, &na, &nr);
         return sarbp_wk_preprocess(c, &w, host<sarbp_complex64>(48 * 60), 48, 60, host<sarbp_complex64>(na * nr), s);
     }},
    {"wk_focus", [](sarbp_ctx *c, cudaStream_t s, bool o) {
         const sarbp_wk_params w = wk_params(o ? 9e5 : 988647.462);
         return sarbp_wk_focus(c, &w, host<sarbp_complex64>(64 * 100), 64, 100, host<sarbp_complex64>(64 * 100), s);
     }},
    {"ceos", [](sarbp_ctx *c, cudaStream_t s, bool o) { return ceos(c, s, o, false); }},
    {"ceos_host", [](sarbp_ctx *c, cudaStream_t s, bool o) { return ceos(c, s, o, true); }},
    {"synth", [](sarbp_ctx *c, cudaStream_t s, bool) { return synth(c, s, false); }},
    {"synth_host", [](sarbp_ctx *c, cudaStream_t s, bool) { return synth(c, s, true); }},
};

cudaStream_t stream() {
    cudaStream_t s;
    cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    return s;
}
sarbp_ctx *context() {
    sarbp_ctx *c = nullptr;
    if (sarbp_create(&c, 0) != SARBP_OK) std::exit(3);
    return c;
}
int call(const std::string &name, sarbp_ctx *c, cudaStream_t s, bool other, sarbp_status want = SARBP_OK) {
    const sarbp_status st = kCalls.at(name)(c, s, other);
    if (st == want) return 0;
    std::printf("%s: status %d, %s\n", name.c_str(), (int)st, sarbp_last_error(c));
    return 1;
}
}  // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    int bad = 0;
    if (what == "list") {
        for (auto &kv : kCalls) std::printf("%s\n", kv.first.c_str());
        return 0;
    }
    if (what == "detector") {  // one buffer written on two streams, then again with an event between them
        float *p = device<float>(4);
        cudaStream_t a = stream(), b = stream();
        cudaEvent_t e;
        cudaEventCreate(&e);
        cudaMemsetAsync(p, 0, 16, a);
        cudaMemsetAsync(p, 0, 16, b);
        const int without = g_conflicts;
        cudaDeviceSynchronize();
        cudaMemsetAsync(p, 0, 16, a);
        cudaEventRecord(e, a);
        cudaStreamWaitEvent(b, e, 0);
        cudaMemsetAsync(p, 0, 16, b);
        return without == 1 && g_conflicts == 1 ? 0 : 1;
    }
    sarbp_ctx *c = context();
    if (what == "first") {  // a call right after sarbp_create
        bad += call(argv[2], c, stream(), false);
    } else if (what == "streams") {  // argv[2] with every other call behind it, each on a stream of its own
        const std::string name = argv[2];
        for (auto &kv : kCalls) {
            cudaDeviceSynchronize();
            g_log.clear();
            const int before = g_conflicts;
            bad += call(name, c, stream(), false) + call(kv.first, c, stream(), false) + call(name, c, stream(), false);
            if (g_conflicts != before) std::printf("  in %s, %s, %s\n", name.c_str(), kv.first.c_str(), name.c_str());
        }
    } else if (what == "tables") {  // argv[2] with two sets of parameters in turn, on one stream and on two
        for (int two = 0; two < 2; ++two) {
            cudaDeviceSynchronize();
            g_log.clear();
            cudaStream_t a = stream(), b = two ? stream() : a;
            for (int k = 0; k < 4; ++k) bad += call(argv[2], c, k & 1 ? b : a, k & 1);
        }
    } else if (what == "lengths") {  // more DFT lengths than the context keeps tables of
        cudaStream_t s[2] = {stream(), stream()};
        const int n[] = {64, 100, 128, 200, 256, 300, 64, 100};
        for (int k = 0; k < 8; ++k) bad += sarbp_dft(c, device<sarbp_complex64>(10 * n[k]), 10, n[k], 0, s[k & 1]) != SARBP_OK;
    } else if (what == "uploads") {  // pulses of each chunk of a host echo of argv[2] pulses, argv[3] samples, upsampled by argv[4]
        const int np = std::atoi(argv[2]), ns = std::atoi(argv[3]);
        g_uploads.clear();
        g_frees = 0;
        bad += range_compress(c, stream(), false, SARBP_STORE_C32H, true, np, ns, std::atoi(argv[4])) != SARBP_OK;
        for (size_t n : g_uploads)
            if (n % (8ull * ns) == 0) std::printf("%zu ", n / (8ull * ns));
        std::printf("\n%d buffers freed\n", g_frees);
    } else if (what == "failed") {  // a back-projection that fails behind its first launch
        g_fail_bp = true;
        bad += call("image", c, stream(), false, SARBP_ERR_CUDA);
        g_fail_bp = false;
        bad += call("image", c, stream(), false);
    } else {
        return 2;
    }
    std::printf("%d conflicts, %d unexpected statuses\n", g_conflicts, bad);
    return g_conflicts || bad ? 1 : 0;
}
