// bp.cu -- back-projection on sm_103a.
//
// Algorithm: code/SAR_BP/matlab/BPA_SAR.m:177-197 (per pixel and pulse: slant
// range, range bin, sample, phase compensation exp(+j 4 pi fc R / c), coherent
// sum), with linear interpolation on the upsampled bins instead of the script's
// nearest bin.  Kernel shape replaces backProjectionKernel
// (code/SAR_BP/CUDA/BPA_CUDA_kernels.cu:47-77: one thread per pixel, global
// loads, sqrtf + sincosf per pulse).
//
// Design (one CTA per TILE_X x TILE_Y pixel tile, optionally per pulse segment):
//  * Pulses are processed in chunks of CHUNK.  For each chunk one staging warp
//    computes, a lane per pulse, the tile-centre reference: range R_T, wrapped
//    carrier phase, the bin of the tile centre and the window of bins the tile
//    can touch; it then issues one TMA bulk copy (cp.async.bulk, local HBM ->
//    shared memory, completion on an mbarrier) per pulse for that window.  A
//    three-stage ring of raw windows lets chunk c+1 load while chunk c computes.
//  * A conversion pass turns each raw window (complex64, or complex16 times the
//    per-pulse scale) into interpolation-ready pairs (mid, diff) with
//    mid_i = (s_i + s_{i+1})/2, diff_i = s_{i+1} - s_i, so one 16-byte shared load
//    and two FMAs interpolate.  Converted windows are double-buffered: one
//    block barrier per chunk.
//  * Who stages (helper_warps).  The parameters are a float-float chain of some 400
//    instructions; run by every warp for two pulses each, and with every warp
//    converting, staging cost a quarter of the instructions and held the pixel
//    warps at the barrier.
//    - 16-pulse chunks of 32 x 64 tiles: two extra warps stage the next chunk
//      beside the pixel warps' loop.  20 warps per SM leave 96 registers, which
//      that loop needs.  Config 2 45.8 -> 42.5 ms, FP16 rows 3.63 -> 3.37 ms (the
//      pixel warps staging, the parameters in turn: 44.8 and 3.49 ms), weighted
//      projection 1.78 -> 1.71 ms.
//    - 8- and 4-pulse chunks (wide windows, short tiles) have less pixel work per
//      staged bin, and two warps cannot keep up with the conversion: one extra
//      warp computes the parameters, the pixel warps convert.  1024 pulses onto
//      1024^2 at 1.0 m, none / one / two helpers: 1.32 / 1.27 / 1.40 ms; 1.4 m
//      rotated by 45 degrees 3.06 / 2.65 / 3.84 (3.80 with every warp preparing
//      parameters); its projection 3.66 / 3.17; 2.2 m onto 512^2 1.50 / 1.27 /
//      2.08 (1.84); 1200 x 1000 at 0.75 m, rotated 1.61 / 1.56.  The helper holds
//      these to 96 registers as well, and the linear-term ones spill for it: 8 bytes
//      a thread in back-projection, 4 in the three-term projection.  The times above
//      include that; what the pixel warps no longer do is worth more.
//    - The linear-term back-projection with 16-pulse chunks needs more than 96
//      registers too, but its narrow windows leave a helper little to take over
//      (0.37 m: 0.91 ms without a helper, 0.96 with one).  The FP64 and FP32
//      comparators have no helper, and the checked kernels follow.  There the pixel
//      warps stage, each chunk's parameters by the next warp in turn.
//  * SPLIT arithmetic per pixel and pulse: with q the pixel offset from the tile
//    centre, n = 2 q.w + |q|^2 (w = tile centre - APC) and the differential
//    range dR = sqrt(R_T^2 + n) - R_T = n (c1 + n (c2 + n (c3 + n c4))) (series
//    of sqrt(1+e); the planner bounds the truncation error) -- all on the FMA
//    pipe; the phase fma(dR, k_hi, phi_T) + dR k_lo (compensated product); the
//    only MUFU work is one sin/cos pair.
//  * What bounds the pixel loop is the register file's read ports (57.6% of the issue
//    slots are used): a scheduler reads two 32-lane registers per clock, so an FMA of three distinct registers takes
//    1.3-1.5 clk and a packed FP32x2 FMA of three register pairs 3.1, not 2
//    (microbenchmark; 2.6 with one operand a scalar read as both halves, 2.0
//    with two).  So per-pulse constants enter the packed operations as scalars
//    (not as stored pairs, which also halves their shared loads); the
//    interpolation and the sums run packed over (re, im) of one pixel, on two
//    accumulators, sum s cos and sum s sin, combined at the end, so neither
//    the loaded pair nor the sample is repacked (3 instructions per update, 6
//    before); and the staging buffer's address is part of the per-pulse
//    rounding constant, so a pixel's shared address is one shift-add with an
//    immediate.  Config 2 (4096 pulses, 4096^2 pixels) 52.9 -> 45.8 ms, FP16
//    rows 9% and the linear-term form 8% faster, same phases bit for bit.
//  * Staging windows are sized so every bin a pixel can need lies inside
//    [1, win-3]; the producer checks this per (tile, pulse) and, should a pulse
//    fail the check, neutralises it (no data, bin 1) and raises an error bit,
//    so shared-memory indices stay in bounds without a per-update clamp.  The
//    CHECKED variant keeps a clamp and reports whether it ever fired.
//  * FP32 and FP64 modes use the same staging with plain absolute-range
//    arithmetic (the comparators) and always clamp.
#include "sarbp_internal.h"

#include <math_constants.h>

#include "ffloat.cuh"
#include "tma.cuh"

#include <cstddef>
#include <cstring>

namespace sarbp {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTileX = 32;  // pixels along x (columns); tile height is 8 * PIX rows
#ifndef SARBP_BP_CHUNK
#define SARBP_BP_CHUNK 16
#endif
#ifndef SARBP_BP_MINBLOCKS
#define SARBP_BP_MINBLOCKS 2
#endif
// Per-update phase: phi_T + dR k_hi (k_hi = float(4 pi fc / c)); the
// compensated form adds dR k_lo.  The omitted term is at most
// |dR| ulp(k)/2 (7e-5 rad at config 2's tile corners) and is of the size of the
// FP32 rounding of dR itself and of the sin/cos argument, so the image does
// not change measurably (-81.68 dB against FP64 either way) and the update is
// one packed FMA shorter.
#ifndef SARBP_BP_PHASE_COMPENSATED
#define SARBP_BP_PHASE_COMPENSATED 0
#endif
constexpr int kChunk = SARBP_BP_CHUNK;  // pulses per staged chunk (a multiple of 8)
// Warps of a CTA beside its kWarps pixel warps: 2 stage whole chunks; 1 computes the
// parameters and issues the copies, the pixel warps convert; 0: the pixel warps
// do both, the parameters in turn.
template <int MODE, bool CHECKED, int PIX, bool ADJ, int CHUNK, bool LIN>
__host__ __device__ constexpr int helper_warps() {
    if (CHECKED || (MODE != SARBP_MODE_SPLIT && MODE != SARBP_MODE_FP16STORE)) return 0;
    if (CHUNK) return PIX == 8 && (ADJ || !LIN) ? 2 : 0;
    return 1;
}
static_assert(kChunk <= 32, "one staging lane per pulse of a chunk");
constexpr int kStages = 3;  // raw-window ring depth
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
constexpr unsigned kMagicBitsShift4 = 0x4B400000u << 4;

struct __align__(16) Prm {
    // split arithmetic: each constant once, the packed operations read a scalar
    // as both halves
    float4 k0;     // c1, c2, c3, c4 (LIN: c1, d2, d3, d4)      FP32: apc x, y, z, bin offset
    float4 k1;     // bin', phT, A, B (LIN: A c1, B c1)          FP32: phase correction
    float2 k2;     // LIN: the phase increments per pixel step PX, PY
    double ax, ay, az;  // FP64: APC position
    double dr, dph;     // FP64: per-pulse range (m) and phase (rad) corrections
    int ws;        // first bin of the window
    int lo, hi;    // copied part of the window [lo, hi) relative to ws
    float scale;   // FP16 storage scale
    int need;      // bins [0, need) hold every bin a pixel of the tile reads: (M, d) pairs [0, need - 1)
    int unused[4]; // keeps the record at the 128 bytes that the planner's bounds count
};
// which windows the planner accepts depends on it through bp_smem_bytes
static_assert(sizeof(Prm) == 128, "Prm size");

__device__ __forceinline__ float4 lds128(unsigned addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr));
    return v;
}

// Packed FP32x2 arithmetic (sm_100+ f32x2 instructions): two IEEE FP32
// operations, each rounded to nearest, per issue slot.  A pair lives in a
// 64-bit register pair (lo, hi).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void upk2(f2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 ffma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 fadd2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fmul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// A scalar as both halves of a packed operand: read as one register, not two.
__device__ __forceinline__ f2 bc2(float v) { return pk2(v, v); }
// acc += a b.  The accumulator stays a float pair outside the instruction: as a
// 64-bit loop variable it cost one register move per instruction and pulse body.
__device__ __forceinline__ void ffma2_acc(float2 &acc, f2 a, f2 b) {
    asm("{\n\t.reg .b64 d;\n\tmov.b64 d, {%0, %1};\n\tfma.rn.f32x2 d, %2, %3, d;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "l"(a), "l"(b));
}
__device__ __forceinline__ f2 fsub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// 16-byte shared store and load of two packed pairs
__device__ __forceinline__ void sts2x2(void *p, f2 a, f2 b) {
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(smem_addr(p)), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void lds2x2_at(unsigned addr, f2 &a, f2 &b) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}

struct Smem {
    float4 *staged;      // [2][chunk][win]
    unsigned char *raw;  // [kStages][chunk][win] stored elements (8 or 4 bytes)
    Prm *prm;            // [kStages][kChunk] (chunk <= kChunk pulses used per stage)
    uint64_t *bar;       // [kStages]
    float2 *red;         // [2][kWarps][kChunk] per-warp pulse sums (weighted projection)
};

// Bytes of one stored range bin in the raw ring: complex64 rows 8, complex16 4.
__host__ __device__ constexpr int raw_esize(int storage) { return storage == SARBP_STORE_C64 ? 8 : 4; }

template <int STORE>
__device__ __forceinline__ Smem carve(unsigned char *base, int win, int chunk) {
    Smem s;
    s.staged = reinterpret_cast<float4 *>(base);
    s.raw = base + (size_t)2 * chunk * win * 16;
    s.prm = reinterpret_cast<Prm *>(s.raw + (size_t)kStages * chunk * win * raw_esize(STORE));
    s.bar = reinterpret_cast<uint64_t *>(s.prm + kStages * kChunk);
    s.red = reinterpret_cast<float2 *>(s.bar + kStages);
    return s;
}

struct TileGeo {
    double pcx, pcy, pcz;   // tile centre
    float qq_max;           // max |q|^2 over the tile
    float xT, yT;           // tile centre in pixel units from the grid origin (exact)
    float qqh, qql;         // |xT ux + yT uy|^2 as a float pair
};

// Per-pulse reference (FP64), relative to the grid origin O:
//   a0 = |O - apc|^2, a1 = 2 ux.(O - apc), a2 = 2 uy.(O - apc)
// stored as float pairs: pref[2p] = (a0h, a0l, a1h, a1l), pref[2p+1] = (a2h, a2l, 0, 0).
// With (xT, yT) a tile centre in pixel units, R_T^2 = a0 + xT a1 + yT a2 + |q_T|^2.
// Per-pulse references for the SPLIT path.  The optional corrections enter
// as a bin offset db = drange * (2 bin_rate / c) and a phase offset
// dph = 2 pi frac(drange * 2 fc / c) + dphase (wrapped to [-pi, pi]), applied to
// the tile-centre bin and phase, so they cost nothing per update.
__global__ void pulse_ref_kernel(const double *__restrict__ apc, int np, BpGeom g, const double *__restrict__ drange,
                                 const double *__restrict__ dphase, double bins_per_m, double cyc_per_m,
                                 float4 *__restrict__ pref) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const double dr = drange ? drange[p] : 0.0;
    const double cyc = dr * cyc_per_m;
    double dph = 2.0 * CUDART_PI * (cyc - rint(cyc)) + (dphase ? dphase[p] : 0.0);
    dph -= 2.0 * CUDART_PI * rint(dph * (0.5 / CUDART_PI));
    const double wx = g.origin[0] - apc[3 * p], wy = g.origin[1] - apc[3 * p + 1], wz = g.origin[2] - apc[3 * p + 2];
    const double a0 = fma(wx, wx, fma(wy, wy, wz * wz));
    const double a1 = 2.0 * (g.ux[0] * wx + g.ux[1] * wy + g.ux[2] * wz);
    const double a2 = 2.0 * (g.uy[0] * wx + g.uy[1] * wy + g.uy[2] * wz);
    const float a0h = (float)a0, a1h = (float)a1, a2h = (float)a2;
    pref[2 * p] = make_float4(a0h, (float)(a0 - (double)a0h), a1h, (float)(a1 - (double)a1h));
    pref[2 * p + 1] = make_float4(a2h, (float)(a2 - (double)a2h), (float)(dr * bins_per_m), (float)dph);
}

// After the wait for chunk c ran out: raise the timeout bit and let the copies
// still in flight land before the CTA's shared memory is released.  The staging
// warps have issued chunks c and (if it exists) c + 1 and waited for all before them,
// so those two phases are the outstanding ones: wait for each on its own
// parity (chunk k is phase k / kStages of ring stage k % kStages).  Out of line:
// inlined, this cold path moved the main loop's schedule (config 2: 54.1 ms
// against 53.1 ms per launch).
template <bool TESTF>
__device__ __noinline__ void drain_after_timeout(const BpPlan &P, uint64_t *bars, int c, int nchunks) {
    atomicOr(P.err, kErrWaitTimeout);
    for (int k = c; k <= c + 1 && k < nchunks; ++k) {
        const unsigned bar = smem_addr(&bars[k % kStages]);
        if (TESTF && k == P.fault_chunk) mbar_complete_tx(bar, kFaultBytes);
        const uint64_t lim = TESTF && P.wait_ns > kDrainWaitNs ? P.wait_ns : kDrainWaitNs;
        if (!mbar_wait_bounded(bar, (k / kStages) & 1, lim)) atomicOr(P.err, kErrDrainTimeout);
    }
}

// Per-(tile, pulse) geometry, window and TMA issue for the pulses of one chunk,
// by one warp (a lane per pulse), which arrives once on the stage's barrier.
// `fault` (tests only) arms the arrival with kFaultBytes that no copy delivers,
// so the phase cannot complete and the staging warps' bounded wait runs out.
template <int MODE, int STORE, int PIX, bool LIN>
__device__ __forceinline__ void produce(const BpPlan &P, const Smem &S, int stage, int p0, int count,
                                        const TileGeo &T, bool fault) {
    constexpr int kTileY = 8 * PIX;
    const int slot = threadIdx.x & 31;
    const int win = P.win;
    const int esize = STORE == SARBP_STORE_C64 ? 8 : 4;
    unsigned bytes = 0;
    const char *src = nullptr;
    unsigned dst = 0;
    if (slot < count) {
        const int p = p0 + slot;
        const float bpm = P.kb_h;  // bins per metre of range
        const float hx = 0.5f * (kTileX - 1), hy = 0.5f * (kTileY - 1);
        const int cen = win >> 1;  // staged index origin
        Prm &q = S.prm[stage * kChunk + slot];
        int ws;  // window start, clamped to +-1e9 bins: int arithmetic throughout
        int need = win;
        bool sane;
        if (MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE) {
            // R_T^2 = a0 + xT a1 + yT a2 + |q_T|^2 in float-float
            const float4 r0v = __ldg(&P.pref[2 * p]);
            const float4 r1v = __ldg(&P.pref[2 * p + 1]);
            const ff a0 = {r0v.x, r0v.y}, a1 = {r0v.z, r0v.w}, a2 = {r1v.x, r1v.y};
            const ff S2 = ff_add(ff_add(a0, ff_mul_f(a1, T.xT)), ff_add(ff_mul_f(a2, T.yT), ff{T.qqh, T.qql}));
            const float r = sqrtf(S2.h);
            const float corr = (fmaf(-r, r, S2.h) + S2.l) * (0.5f / r);  // R_T = r + corr
            // bin of the tile centre: (2 R_T / c - t0) * bin_rate
            const float kbh = P.kb_h, kbl = P.kb_l;
            float ph_ = r * kbh;
            float pl_ = fmaf(r, kbh, -ph_) + fmaf(r, kbl, corr * kbh);
            const ff bT = ff_add(ff_add(quick_two_sum(ph_, pl_), ff{-P.tb_h, -P.tb_l}), ff{r1v.z, 0.f});
            // carrier phase 2 pi frac(R_T * 2 fc / c)
            const float kch = P.kc_h, kcl = P.kc_l;
            const float cy = r * kch;
            const float cy_e = fmaf(r, kch, -cy) + fmaf(r, kcl, corr * kch);
            const float fr = (cy - rintf(cy)) + cy_e;
            const float phT = fmaf(fr, 6.28318530717958647692f, r1v.w);
            const float iR = 1.0f / r;
            const float A = r0v.z + 2.f * (T.xT * P.gf11 + T.yT * P.gf12);
            const float B = r1v.x + 2.f * (T.xT * P.gf12 + T.yT * P.gf22);
            const float half = bpm * (fabsf(A) * hx + fabsf(B) * hy + T.qq_max) * 0.5f * iR * 1.03f + 2.f;
            ws = (int)floorf(fminf(fmaxf(bT.h - half, -1.0e9f), 1.0e9f));
            ws &= ~3;
            const int need_end = (int)ceilf(fminf(fmaxf(bT.h + half, -1.0e9f), 1.0e9f)) + 2;
            sane = isfinite(r) && r > 0.f && isfinite(half) && isfinite(phT) && need_end - ws <= win;
            // the tile's bins lie in [bT - half, bT + half]: pair indices up to
            // need_end - ws - 2, so pairs [0, need - 1) cover every read (the
            // checked build flags any read past need - 2)
            if (sane) need = need_end - ws;
            const float i2 = iR * iR;
            if (sane) {
                const float c1 = 0.5f * iR, c2 = -0.125f * iR * i2, c3 = 0.0625f * iR * i2 * i2;
                const float c4 = -0.0390625f * iR * i2 * i2 * i2;
                const float bb = ((bT.h - (float)ws) + bT.l) - 0.5f - (float)cen;
                if constexpr (LIN) {
                    // the series in m = n / (2 R_T): dR = m + m^2 (d2 + m (d3 + m d4)), and
                    // the phase's linear part from the increments per pixel step, half of
                    // 4 pi / lambda (u.w) / R_T reduced modulo 2 pi (the pixel offsets are
                    // half-integers, 2 xc and 2 yc integers), in float-float:
                    // u.w = a1 / 2 + xT g11 + yT g12 (x), a2 / 2 + xT g12 + yT g22 (y),
                    // 1 / R_T from iR and one Newton correction
                    const float d2 = -0.5f * iR, d3 = 0.5f * i2, d4 = -0.625f * i2 * iR;
                    const ff g11 = {P.gf11, P.gf11l}, g12 = {P.gf12, P.gf12l}, g22 = {P.gf22, P.gf22l};
                    const ff uxw = ff_add(ff{0.5f * a1.h, 0.5f * a1.l}, ff_add(ff_mul_f(g11, T.xT), ff_mul_f(g12, T.yT)));
                    const ff uyw = ff_add(ff{0.5f * a2.h, 0.5f * a2.l}, ff_add(ff_mul_f(g12, T.xT), ff_mul_f(g22, T.yT)));
                    const ff invR = quick_two_sum(iR, iR * (fmaf(-r, iR, 1.f) - corr * iR));
                    const ff kh = {0.5f * P.kp_h, 0.5f * P.kp_l};  // 2 pi fc / c
                    const float pxr = ff_mod_2pi(ff_mul(ff_mul(kh, uxw), invR));
                    const float pyr = ff_mod_2pi(ff_mul(ff_mul(kh, uyw), invR));
                    q.k0 = make_float4(c1, d2, d3, d4);
                    q.k1 = make_float4(bb, phT, A * c1, B * c1);
                    q.k2 = make_float2(pxr, pyr);
                } else {
                    q.k0 = make_float4(c1, c2, c3, c4);
                    q.k1 = make_float4(bb, phT, A, B);
                }
            } else {  // inert pulse: every pixel reads the centre bin of an all-zero window
                q.k0 = q.k1 = make_float4(0.f, 0.f, 0.f, 0.f);
                q.k2 = make_float2(0.f, 0.f);
            }
        } else {
            const double ax = __ldg(&P.apc[3 * p]), ay = __ldg(&P.apc[3 * p + 1]), az = __ldg(&P.apc[3 * p + 2]);
            const double wx = T.pcx - ax, wy = T.pcy - ay, wz = T.pcz - az;
            const double dr = P.drange ? __ldg(&P.drange[p]) : 0.0;
            const double dph = P.dphase ? __ldg(&P.dphase[p]) : 0.0;
            const double R = sqrt(fma(wx, wx, fma(wy, wy, wz * wz))) + dr;
            const float iR = (float)(1.0 / R);
            const float wxf = (float)wx, wyf = (float)wy, wzf = (float)wz;
            const float A = 2.f * ((float)P.g.ux[0] * wxf + (float)P.g.ux[1] * wyf + (float)P.g.ux[2] * wzf);
            const float B = 2.f * ((float)P.g.uy[0] * wxf + (float)P.g.uy[1] * wyf + (float)P.g.uy[2] * wzf);
            const double bT = fma(R, 2.0 / P.c * P.bin_rate, -P.t0_bins * P.bin_rate);
            const float half = bpm * (fabsf(A) * hx + fabsf(B) * hy + T.qq_max) * 0.5f * iR * 1.03f + 2.f;
            const float bTf = (float)bT;
            ws = (int)floorf(fminf(fmaxf(bTf - half, -1.0e9f), 1.0e9f));
            ws &= ~3;
            const int need_end = (int)ceilf(fminf(fmaxf(bTf + half, -1.0e9f), 1.0e9f)) + 2;
            sane = isfinite(R) && R > 0.0 && isfinite(half) && need_end - ws <= win;
            if (MODE == SARBP_MODE_FP32) {
                const double kph_d = 4.0 * CUDART_PI * P.fc / P.c;
                q.k0 = make_float4((float)ax, (float)ay, (float)az,
                                   (float)(dr * (2.0 / P.c * P.bin_rate) - P.t0_bins * P.bin_rate - (double)ws - 0.5 -
                                           (double)cen));
                q.k1 = make_float4((float)(kph_d * dr + dph), 0.f, 0.f, 0.f);
            }
            q.dr = dr;
            q.dph = dph;
            q.ax = ax;
            q.ay = ay;
            q.az = az;
        }
        if (!sane) atomicOr(P.err, kErrWindow);
        const int lo = ws < 0 ? 0 : ws;
        int hi = ws + win > P.nbins ? P.nbins : ws + win;
        if (hi < lo || !sane) hi = lo;
        q.ws = ws;
        q.lo = lo - ws;
        q.hi = hi - ws;
        q.need = need;
        q.scale = STORE == SARBP_STORE_C32H ? __ldg(&P.scale[p]) : 1.f;
        if (hi > lo) {
            bytes = (unsigned)((hi - lo) * esize);
            src = reinterpret_cast<const char *>(P.rc) + ((size_t)p * P.nbins + (size_t)lo) * esize;
            dst = smem_addr(S.raw + ((size_t)stage * P.chunk + (size_t)slot) * win * esize + (size_t)(lo - ws) * esize);
        }
    }
    unsigned total = bytes;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const unsigned bar = smem_addr(&S.bar[stage]);
    if (fault) total += kFaultBytes;
    __syncwarp();  // the arrival below publishes every lane's parameters
    if (slot == 0) mbar_expect_tx_arrive(bar, total);
    __syncwarp();
    if (bytes) tma_bulk_g2s(dst, src, bytes, bar);
}

// raw window -> (mid, diff) pairs; bins outside [lo, hi) read as zero.  By the
// staging warps, flat over (pulse, bin), the whole window: the checked build
// and the FP32 / FP64 comparators clamp reads anywhere in it.
template <int MODE, int STORE>
__device__ __forceinline__ void convert_flat(const Smem &S, int stage, int sbuf, int count, int win, unsigned win_magic,
                                             int chunk, int stager, int stagers) {
    const int total = count * win;
    float4 *st = S.staged + (size_t)sbuf * chunk * win;
    for (int e = 32 * stager + (threadIdx.x & 31); e < total; e += 32 * stagers) {
        const int pl = (int)__umulhi((unsigned)e, win_magic);
        const int i = e - pl * win;
        const Prm &q = S.prm[stage * kChunk + pl];
        const int lo = q.lo, hi = q.hi;
        const unsigned char *rw = S.raw + ((size_t)stage * chunk + pl) * win * raw_esize(STORE);
        float2 a = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
        if (STORE == SARBP_STORE_C64) {
            const float2 *r = reinterpret_cast<const float2 *>(rw);
            if (i >= lo && i < hi) a = r[i];
            if (i + 1 >= lo && i + 1 < hi) b = r[i + 1];
        } else {
            const __half2 *r = reinterpret_cast<const __half2 *>(rw);
            const float sc = q.scale;
            if (i >= lo && i < hi) a = __half22float2(r[i]);
            if (i + 1 >= lo && i + 1 < hi) b = __half22float2(r[i + 1]);
            a.x *= sc; a.y *= sc; b.x *= sc; b.y *= sc;
        }
        const float dx = b.x - a.x, dy = b.y - a.y;
        // FP32 arithmetic: pairs centred on the window middle, so that s = M + b d
        // takes the centred position b directly; FP64 keeps (mid, diff).
        const float o = MODE == SARBP_MODE_FP64 ? 0.f : (float)(i - (win >> 1));
        st[e] = make_float4(fmaf(-o, dx, 0.5f * (a.x + b.x)), fmaf(-o, dy, 0.5f * (a.y + b.y)), dx, dy);
    }
}

// One stored bin as a packed (re, im) pair, FP16 rows times the pulse's scale.
template <int STORE>
__device__ __forceinline__ f2 raw_bin(const unsigned char *row, int i, f2 scale) {
    if constexpr (STORE == SARBP_STORE_C64) {
        return *reinterpret_cast<const f2 *>(row + 8 * i);
    } else {
        const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(row + 4 * i));
        return fmul2(pk2(v.x, v.y), scale);
    }
}

// The same pairs for the unchecked SPLIT / FP16STORE kernels: a staging warp
// per pulse, packed over (re, im), and only the pairs [0, need - 1) the tile
// reads (bins [0, need); the checked build flags any read past need - 2).
// Windows that lie inside the row, all but those at the swath edges, skip
// the bounds tests.
template <int STORE>
__device__ __forceinline__ void convert_pulses(const Smem &S, int stage, int sbuf, int count, int win, int chunk,
                                               int stager, int stagers) {
    const int lane = threadIdx.x & 31;
    for (int pl = stager; pl < count; pl += stagers) {
        const Prm &q = S.prm[stage * kChunk + pl];
        const int lo = q.lo, hi = q.hi, n = q.need - 1;
        const f2 scale = bc2(STORE == SARBP_STORE_C32H ? q.scale : 1.f);
        const unsigned char *row = S.raw + ((size_t)stage * chunk + pl) * win * raw_esize(STORE);
        float4 *st = S.staged + ((size_t)sbuf * chunk + pl) * win;
        float o = (float)((win >> 1) - lane);  // from the pair to the window middle
        auto store = [&](int i, f2 a, f2 b) {
            const f2 d = fsub2(b, a);
            sts2x2(st + i, ffma2(bc2(o), d, fmul2(bc2(0.5f), fadd2(a, b))), d);
        };
        if (lo == 0 && hi > n) {
#pragma unroll 1
            for (int i = lane; i < n; i += 32, o -= 32.f)
                store(i, raw_bin<STORE>(row, i, scale), raw_bin<STORE>(row, i + 1, scale));
        } else {
#pragma unroll 1
            for (int i = lane; i < n; i += 32, o -= 32.f)
                store(i, i >= lo && i < hi ? raw_bin<STORE>(row, i, scale) : 0ull,
                      i + 1 >= lo && i + 1 < hi ? raw_bin<STORE>(row, i + 1, scale) : 0ull);
        }
    }
}

// Sum of the warps' projections for the pulses of one chunk into
// proj[tile][pulse] (fixed order: deterministic).
__device__ __forceinline__ void flush_projection(const BpPlan &P, const Smem &S, int buf, int p0, int count, int t) {
    if (t < count) {
        float sr = 0.f, si = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float2 v = S.red[(buf * kWarps + w) * kChunk + t];
            sr += v.x;
            si += v.y;
        }
        P.proj[(size_t)blockIdx.x * P.np + p0 + t] = make_float2(sr, si);
    }
}

// One chunk of the weighted projection: per pulse, this thread's sum over its
// pixels of conj(w) * term, then the warp's sum into red[2 pulse + {re, im}].
// conj(w) e^{i phi} = |w| e^{i (phi - arg w)}: the weight's phase joins the
// packed phase (half an op per pixel) and its magnitude scales cos / sin, so
// the weighted accumulate costs 6.5 FP32 ops instead of 8.
// Pulses go in pairs through one shared butterfly: the xor-16 step splits the
// pair's two pulses between the half-warps and the xor-8 step splits re / im,
// so a pair costs 6 shuffles instead of 20 for two separate 32-lane sums.
// LIN: the linear-term phase (as the back-projection's LIN loop), the weight's
// phase added to it the same way.
template <int NTERMS, int PIX, bool LIN>
__device__ __forceinline__ void project_chunk(const Smem &S, int stage, int count, int win, unsigned stg, int cen,
                                              float xc, const f2 (&YC2)[PIX / 2], const f2 (&QQ2)[PIX / 2], f2 BPM2,
                                              f2 KH2, f2 KL2, const f2 (&TH2)[PIX / 2], const float (&wm)[PIX],
                                              const f2 (&Y2C2)[LIN ? PIX / 2 : 1], float *red) {
    const int lane = threadIdx.x & 31;
    const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
    const f2 XC2 = bc2(xc);
    float mp = kMagic + (float)(int)((stg >> 4) + cen);  // the window middle's 16-byte slot
    const float winf = (float)win;
#pragma unroll 1
    for (int pl = 0; pl < count; pl += 2) {
        float tr[2] = {0.f, 0.f}, ti[2] = {0.f, 0.f};
#pragma unroll
        for (int u2 = 0; u2 < 2; ++u2) {
            if (u2 == 1 && pl + 1 >= count) break;  // odd tail: pulse-uniform
            const Prm &q = S.prm[stage * kChunk + pl + u2];
            const float4 v0 = lds128(smem_addr(&q.k0)), v1 = lds128(smem_addr(&q.k1));
            const f2 C1 = bc2(v0.x), C2 = bc2(v0.y), C3 = bc2(v0.z), C4 = bc2(v0.w);  // LIN: C1, D2, D3, D4
            const f2 BT = bc2(v1.x), PHT = bc2(v1.y), AA = bc2(v1.z), BB = bc2(v1.w);
            f2 PHX = PHT, PY = PHT;
            if constexpr (LIN) {
                const float2 v2 = q.k2;
                PHX = bc2(fmaf(2.f * xc, v2.x, v1.y));
                PY = bc2(v2.y);
            }
#pragma unroll
            for (int h = 0; h < PIX / 2; ++h) {
                f2 b2, ph2;
                if constexpr (LIN) {
                    const f2 qc = fmul2(QQ2[h], C1);
                    const f2 m = ffma2(YC2[h], BB, ffma2(XC2, AA, qc));
                    const f2 m2 = fmul2(m, m);
                    const f2 poly = NTERMS == 4 ? ffma2(m, ffma2(m, C4, C3), C2) : ffma2(m, C3, C2);
                    b2 = ffma2(ffma2(m2, poly, m), BPM2, BT);
                    ph2 = fadd2(ffma2(ffma2(m2, poly, qc), KH2, ffma2(Y2C2[h], PY, PHX)), TH2[h]);
                } else {
                    const f2 n = ffma2(YC2[h], BB, ffma2(XC2, AA, QQ2[h]));
                    f2 poly = NTERMS == 4 ? ffma2(n, ffma2(n, C4, C3), C2) : ffma2(n, C3, C2);
                    poly = ffma2(n, poly, C1);
                    const f2 dR = fmul2(n, poly);
                    b2 = ffma2(dR, BPM2, BT);
#if SARBP_BP_PHASE_COMPENSATED
                    ph2 = fadd2(ffma2(dR, KL2, ffma2(dR, KH2, PHT)), TH2[h]);
#else
                    ph2 = fadd2(ffma2(dR, KH2, PHT), TH2[h]);
#endif
                }
                float bb[2], ph[2], tt[2];
                upk2(b2, bb[0], bb[1]);
                upk2(ph2, ph[0], ph[1]);
                upk2(fadd2(b2, bc2(mp)), tt[0], tt[1]);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int j = 2 * h + u;
                    f2 M, D;
                    lds2x2_at((__float_as_uint(tt[u]) << 4) - kMagicBitsShift4, M, D);
                    float sr, si, sn, cs;
                    upk2(ffma2(bc2(bb[u]), D, M), sr, si);
                    __sincosf(ph[u], &sn, &cs);
                    const float zr = wm[j] * cs, zi = wm[j] * sn;
                    tr[u2] = fmaf(sr, zr, fmaf(-si, zi, tr[u2]));
                    ti[u2] = fmaf(sr, zi, fmaf(si, zr, ti[u2]));
                }
            }
            mp += winf;
        }
        float k0 = hi16 ? tr[1] : tr[0], k1 = hi16 ? ti[1] : ti[0];
        k0 += __shfl_xor_sync(0xffffffffu, hi16 ? tr[0] : tr[1], 16);
        k1 += __shfl_xor_sync(0xffffffffu, hi16 ? ti[0] : ti[1], 16);
        float k = hi8 ? k1 : k0;
        k += __shfl_xor_sync(0xffffffffu, hi8 ? k0 : k1, 8);
        k += __shfl_xor_sync(0xffffffffu, k, 4);
        k += __shfl_xor_sync(0xffffffffu, k, 2);
        k += __shfl_xor_sync(0xffffffffu, k, 1);
        const int pp = pl + (hi16 ? 1 : 0);
        if ((lane & 7) == 0 && pp < count) red[2 * pp + (hi8 ? 1 : 0)] = k;
    }
}

// ADJ: weighted projection (the adjoint) instead of back-projection: every
// pixel's term of pulse p is multiplied by conj(weight[pixel]) and summed over
// the tile into proj[tile][p] (SPLIT / FP16STORE arithmetic).
// CHUNK: pulses per staged chunk fixed at compile time (the hot unchecked
// SPLIT / FP16STORE case at 16), or 0 to take the planner's P.chunk.
// TESTF: the waits take their limit from P.wait_ns and P.fault_chunk arms one
// chunk's barrier so that its wait runs out (tests of the timeout path, through
// sarbp_debug_set); production variants wait 2 s and carry no injector.
template <int MODE, int STORE, int NTERMS, bool CHECKED, int PIX, bool ADJ = false, int CHUNK = 0, bool TESTF = false,
          bool LIN = false>
__global__ void __launch_bounds__(kThreads + 32 * helper_warps<MODE, CHECKED, PIX, ADJ, CHUNK, LIN>(), SARBP_BP_MINBLOCKS)
    bp_kernel(const __grid_constant__ BpPlan P, int tiles_y, int pulses_per_seg, float qq_max) {
    static_assert(!ADJ || MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE, "projection: split arithmetic");
    static_assert(!LIN || MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE,
                  "linear-term phase: split arithmetic only");
    constexpr int kPix = PIX;  // pixels per thread, all in one column
    constexpr int kTileY = 8 * PIX;
    // pulses per loop body: series form with 16-pulse chunks 2 / 4 / 8 / 16: 43.7 / 43.5 /
    // 43.6 / 42.6 ms at config 2; the others 1 / 2 / 4 / 8: 1.69 / 1.67 / 1.64 / 1.71 ms for
    // the linear-term form at 0.75 m, 1.38 / 1.38 / 1.35 / 1.40 at 1 m
    constexpr int kPulseUnroll = CHUNK && !LIN ? CHUNK : 4;
    constexpr int kHelpers = helper_warps<MODE, CHECKED, PIX, ADJ, CHUNK, LIN>();
    constexpr bool kAhead = kHelpers == 2;  // the helpers stage chunk c + 1 while the pixel warps run chunk c
    constexpr int kStager0 = kAhead ? kWarps : 0, kStagers = kAhead ? kHelpers : kWarps;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int win = P.win;
    const int chunk = CHUNK ? CHUNK : P.chunk;  // pulses per staged chunk: 16, 8 or 4 (two CTAs per SM)
    const Smem S = carve<STORE>(smem_raw, win, chunk);
    const unsigned win_magic = (unsigned)((0xFFFFFFFFull + (unsigned long long)win) / (unsigned long long)win);

    const int tile = blockIdx.x;
    const int ty = tile % tiles_y;  // tiles sharing a range strip run together (L2 reuse)
    const int tx = tile / tiles_y;
    const int seg = blockIdx.y;
    const int p_begin = seg * pulses_per_seg;
    const int p_end = min(P.np, p_begin + pulses_per_seg);
    const int nchunks = p_end > p_begin ? (p_end - p_begin + chunk - 1) / chunk : 0;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lx = lane >> 2, ly = lane & 3;
    const int xl = (warp & 3) * 8 + lx;
    const float xc = (float)xl - 0.5f * (kTileX - 1);
    float yc[kPix], qq[kPix];
    const float g11 = P.gf11, g12 = P.gf12, g22 = P.gf22;
#pragma unroll
    for (int j = 0; j < kPix; ++j) {
        const int yl = ((warp >> 2) + 2 * j) * 4 + ly;
        yc[j] = (float)yl - 0.5f * (kTileY - 1);
        qq[j] = xc * xc * g11 + 2.f * xc * yc[j] * g12 + yc[j] * yc[j] * g22;
    }
    TileGeo T;
    {
        const double pcx_i = tx * kTileX + 0.5 * (kTileX - 1), pcy_i = ty * kTileY + 0.5 * (kTileY - 1);
        T.pcx = P.g.origin[0] + pcx_i * P.g.ux[0] + pcy_i * P.g.uy[0];
        T.pcy = P.g.origin[1] + pcx_i * P.g.ux[1] + pcy_i * P.g.uy[1];
        T.pcz = P.g.origin[2] + pcx_i * P.g.ux[2] + pcy_i * P.g.uy[2];
        T.qq_max = qq_max;
        T.xT = (float)pcx_i;
        T.yT = (float)pcy_i;
        T.qqh = T.qql = 0.f;
        if (warp >= kStager0) {  // staging warps only: FP64 once per CTA
            const double qq = pcx_i * pcx_i * P.g.g11 + 2.0 * pcx_i * pcy_i * P.g.g12 + pcy_i * pcy_i * P.g.g22;
            T.qqh = (float)qq;
            T.qql = (float)(qq - (double)T.qqh);
        }
    }
    const int cen = win >> 1;
    const float cenf = (float)cen;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(smem_addr(&S.bar[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    float acc_r[kPix], acc_i[kPix];
    double dacc_r[MODE == SARBP_MODE_FP64 ? kPix : 1], dacc_i[MODE == SARBP_MODE_FP64 ? kPix : 1];
#pragma unroll
    for (int j = 0; j < kPix; ++j) { acc_r[j] = 0.f; acc_i[j] = 0.f; }
#pragma unroll
    for (int j = 0; j < (MODE == SARBP_MODE_FP64 ? kPix : 1); ++j) { dacc_r[j] = 0.0; dacc_i[j] = 0.0; }

    // back-projection sums, split arithmetic: sum of s cos(phase) and of s sin(phase)
    constexpr bool kSplitBp = !ADJ && (MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE);
    float2 acc_c[kSplitBp ? kPix : 1], acc_s[kSplitBp ? kPix : 1];
#pragma unroll
    for (int j = 0; j < (kSplitBp ? kPix : 1); ++j) acc_c[j] = acc_s[j] = make_float2(0.f, 0.f);

    const float bpm = P.kb_h;
    const float kph_hi = P.kp_h, kph_lo = P.kp_l;  // 4 pi fc / c as a float pair
    const float wmax = (float)(win - 2);

    // weighted projection: |weight| and -arg(weight) of this thread's pixels
    // (zero outside the grid)
    float wm[ADJ ? kPix : 1], wth[ADJ ? kPix : 1];
    if constexpr (ADJ) {
#pragma unroll
        for (int j = 0; j < kPix; ++j) {
            const int x = tx * kTileX + xl, y = ty * kTileY + ((warp >> 2) + 2 * j) * 4 + ly;
            float2 w = make_float2(0.f, 0.f);
            if (x < P.g.nx && y < P.g.ny) w = __ldg(&P.weight[(size_t)y * P.g.nx + x]);
            wm[j] = hypotf(w.x, w.y);
            wth[j] = -atan2f(w.y, w.x);
        }
    }

    float fpy[kPix], fpz[kPix], fpxx[kPix];
    if (MODE == SARBP_MODE_FP32) {
#pragma unroll
        for (int j = 0; j < kPix; ++j) {
            const double xi = tx * kTileX + xl, yi = ty * kTileY + ((warp >> 2) + 2 * j) * 4 + ly;
            fpxx[j] = (float)(P.g.origin[0] + xi * P.g.ux[0] + yi * P.g.uy[0]);
            fpy[j] = (float)(P.g.origin[1] + xi * P.g.ux[1] + yi * P.g.uy[1]);
            fpz[j] = (float)(P.g.origin[2] + xi * P.g.ux[2] + yi * P.g.uy[2]);
        }
    }

    const f2 XC2 = bc2(xc);
    const f2 BPM2 = pk2(bpm, bpm), KH2 = pk2(kph_hi, kph_hi), KL2 = pk2(kph_lo, kph_lo);
    f2 YC2[kPix / 2], QQ2[kPix / 2], TH2[ADJ ? kPix / 2 : 1], Y2C2[LIN ? kPix / 2 : 1];
#pragma unroll
    for (int h = 0; h < kPix / 2; ++h) {
        YC2[h] = pk2(yc[2 * h], yc[2 * h + 1]);
        QQ2[h] = pk2(qq[2 * h], qq[2 * h + 1]);
        if constexpr (ADJ) TH2[h] = pk2(wth[2 * h], wth[2 * h + 1]);
        if constexpr (LIN) Y2C2[h] = pk2(2.f * yc[2 * h], 2.f * yc[2 * h + 1]);
    }

    // Staging of chunk k: one warp computes the parameters and issues the copies of
    // chunk k + 1, then the staging warps wait for chunk k's copies and convert
    // them.  False when the wait ran out.
    const bool helper = kHelpers && warp >= kWarps;
    auto produce_chunk = [&](int k) {
        const int p0 = p_begin + k * chunk;
        if (k < nchunks && warp == (kHelpers ? kWarps : k % kWarps))
            produce<MODE, STORE, PIX, LIN>(P, S, k % kStages, p0, min(chunk, p_end - p0), T,
                                                TESTF && P.fault_chunk == k);
    };
    auto stage_chunk = [&](int k) {
        produce_chunk(k + 1);
        if (!mbar_wait_bounded(smem_addr(&S.bar[k % kStages]), (k / kStages) & 1, TESTF ? P.wait_ns : kDefaultWaitNs))
            return false;
        const int count = min(chunk, p_end - p_begin - k * chunk);
        if constexpr (!CHECKED && (MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE))
            convert_pulses<STORE>(S, k % kStages, k & 1, count, win, chunk, warp - kStager0, kStagers);
        else
            convert_flat<MODE, STORE>(S, k % kStages, k & 1, count, win, win_magic, chunk, warp - kStager0, kStagers);
        return true;
    };

    bool failed = false;
    bool clamped = false;
    if (warp >= kStager0) {
        produce_chunk(0);
        if (kAhead && nchunks > 0) failed = !stage_chunk(0);
    }
    if (kAhead) failed = __syncthreads_or(failed);
    // One block barrier per chunk.  Two helpers stage chunk c + 1 beside the pixel
    // warps' chunk c and the barrier ends both; otherwise it follows chunk c's own
    // staging.  Either way, when chunk k's copies and parameters are
    // issued every warp is done with chunk k - 3 (the ring stage), and when its
    // pairs are written with chunk k - 2 (the buffer).  A wait that ran out ends
    // the loop for every warp.
    int c = 0;  // after a failed wait, the chunk it was for
#pragma unroll 1
    for (; c < nchunks && !failed; ++c) {
        const int stage = c % kStages;
        const int sbuf = c & 1;
        const int pc0 = p_begin + c * chunk;
        const int count = min(chunk, p_end - pc0);
        if constexpr (!kAhead) {
            bool staged = true;
            if (kHelpers == 1 && helper) produce_chunk(c + 1);
            else staged = stage_chunk(c);
            failed = __syncthreads_or(!staged);
            if (failed) break;
            if (kHelpers == 1 && helper) continue;
        }
        if constexpr (ADJ) {  // every pixel warp has finished chunk c - 1: combine its pulse sums
            if (c > 0 && warp == kStager0) flush_projection(P, S, (c - 1) & 1, pc0 - chunk, chunk, lane);
        }
        if (helper) {
            if (kAhead && c + 1 < nchunks) failed = !stage_chunk(c + 1);
        } else {
        const float4 *stg = S.staged + (size_t)sbuf * chunk * win;
        if constexpr (ADJ) {
            project_chunk<NTERMS, kPix, LIN>(S, stage, count, win, smem_addr(stg), cen, xc, YC2, QQ2, BPM2, KH2, KL2, TH2, wm,
                                             Y2C2, reinterpret_cast<float *>(S.red + ((c & 1) * kWarps + warp) * kChunk));
        } else if (LIN && (MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE)) {
            // linear-term form (large tiles): m = n / (2 R_T) centred offset, bin from
            // dR = m + m^2 poly(m), phase from the increments per pixel step (reduced
            // modulo 2 pi per pulse) plus 4 pi / lambda times the nonlinear remainder
            // qq c1 + m^2 poly(m), so no FP32 quantity of the size of the tile's
            // extent enters the phase
            float mp = kMagic + (float)(int)((smem_addr(stg) >> 4) + cen);  // the window middle's 16-byte slot
            const float winf = (float)win;
#pragma unroll kPulseUnroll
            for (int pl = 0; pl < count; ++pl) {
                const Prm &q = S.prm[stage * kChunk + pl];
                const float4 v0 = lds128(smem_addr(&q.k0)), v1 = lds128(smem_addr(&q.k1));
                const float2 v2 = q.k2;
                const f2 C1 = bc2(v0.x), D2 = bc2(v0.y), D3 = bc2(v0.z), D4 = bc2(v0.w);
                const f2 BT = bc2(v1.x), BP = bc2(v1.w), PY = bc2(v2.y);
                const f2 AP = bc2(v1.z);
                const f2 PHX = bc2(fmaf(2.f * xc, v2.x, v1.y));
#pragma unroll
                for (int h = 0; h < kPix / 2; ++h) {
                    const f2 qc = fmul2(QQ2[h], C1);
                    const f2 m = ffma2(YC2[h], BP, ffma2(XC2, AP, qc));
                    const f2 m2 = fmul2(m, m);
                    const f2 poly = NTERMS == 4 ? ffma2(m, ffma2(m, D4, D3), D2) : ffma2(m, D3, D2);
                    const f2 dR = ffma2(m2, poly, m);
                    f2 b2 = ffma2(dR, BPM2, BT);  // bin positions relative to the window middle
                    const f2 nl = ffma2(m2, poly, qc);
                    const f2 ph2 = ffma2(nl, KH2, ffma2(Y2C2[h], PY, PHX));
                    float bb[2], ph[2];
                    upk2(b2, bb[0], bb[1]);
                    upk2(ph2, ph[0], ph[1]);
                    if (CHECKED) {
                        const float needf = (float)(q.need - 2) - cenf;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const float bc = fminf(fmaxf(bb[u], -cenf), wmax - cenf);
                            clamped |= !(bc == bb[u]) || bb[u] > needf;
                            bb[u] = bc;
                        }
                        b2 = pk2(bb[0], bb[1]);
                    }
                    const f2 t2 = fadd2(b2, bc2(mp));
                    float tt[2];
                    upk2(t2, tt[0], tt[1]);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int j = 2 * h + u;
                        f2 M, D;
                        lds2x2_at((__float_as_uint(tt[u]) << 4) - kMagicBitsShift4, M, D);
                        const f2 sv = ffma2(bc2(bb[u]), D, M);
                        float sn, cs;
                        __sincosf(ph[u], &sn, &cs);
                        ffma2_acc(acc_c[j], sv, bc2(cs));
                        ffma2_acc(acc_s[j], sv, bc2(sn));
                    }
                }
                mp += winf;
            }
        } else if (MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE) {
            // geometry, bin and phase for pixel pairs (2j, 2j+1) in packed FP32x2;
            // interpolation and the complex accumulate per pixel
            float mp = kMagic + (float)(int)((smem_addr(stg) >> 4) + cen);  // the window middle's 16-byte slot
            const float winf = (float)win;
#pragma unroll kPulseUnroll
            for (int pl = 0; pl < count; ++pl) {
                const Prm &q = S.prm[stage * kChunk + pl];
                const float4 v0 = lds128(smem_addr(&q.k0)), v1 = lds128(smem_addr(&q.k1));
                const f2 C1 = bc2(v0.x), C2 = bc2(v0.y), C3 = bc2(v0.z), C4 = bc2(v0.w);
                const f2 BT = bc2(v1.x), PHT = bc2(v1.y), BB = bc2(v1.w);
                const f2 AA = bc2(v1.z);
#pragma unroll
                for (int h = 0; h < kPix / 2; ++h) {
                    // x A + |q|^2 in one rounding, as the projection's mul + add
                    // compiles: the phase of a pixel depends on it in the last bits
                    const f2 n = ffma2(YC2[h], BB, ffma2(XC2, AA, QQ2[h]));
                    f2 poly = NTERMS == 4 ? ffma2(n, ffma2(n, C4, C3), C2) : ffma2(n, C3, C2);
                    poly = ffma2(n, poly, C1);
                    const f2 dR = fmul2(n, poly);
                    f2 b2 = ffma2(dR, BPM2, BT);  // bin positions relative to the window middle
#if SARBP_BP_PHASE_COMPENSATED
                    const f2 ph2 = ffma2(dR, KL2, ffma2(dR, KH2, PHT));
#else
                    const f2 ph2 = ffma2(dR, KH2, PHT);
#endif
                    float bb[2], ph[2];
                    upk2(b2, bb[0], bb[1]);
                    upk2(ph2, ph[0], ph[1]);
                    if (CHECKED) {
                        // past the window, or past the pairs an unchecked kernel converts
                        const float needf = (float)(q.need - 2) - cenf;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const float bc = fminf(fmaxf(bb[u], -cenf), wmax - cenf);
                            clamped |= !(bc == bb[u]) || bb[u] > needf;
                            bb[u] = bc;
                        }
                        b2 = pk2(bb[0], bb[1]);
                    }
                    const f2 t2 = fadd2(b2, bc2(mp));
                    float tt[2];
                    upk2(t2, tt[0], tt[1]);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int j = 2 * h + u;
                        f2 M, D;
                        lds2x2_at((__float_as_uint(tt[u]) << 4) - kMagicBitsShift4, M, D);
                        const f2 sv = ffma2(bc2(bb[u]), D, M);
                        float sn, cs;
                        __sincosf(ph[u], &sn, &cs);
                        ffma2_acc(acc_c[j], sv, bc2(cs));
                        ffma2_acc(acc_s[j], sv, bc2(sn));
                    }
                }
                mp += winf;
            }
        } else if (MODE == SARBP_MODE_FP32) {
#pragma unroll 1
            for (int pl = 0; pl < count; ++pl) {
                const Prm &q = S.prm[stage * kChunk + pl];
                const float4 k0 = q.k0;
                const float phc = q.k1.x;  // per-pulse phase correction
                const float mp = kMagic + (float)(pl * win + cen);
                const float kph = kph_hi;
#pragma unroll
                for (int j = 0; j < kPix; ++j) {
                    const float dx = k0.x - fpxx[j], dy = k0.y - fpy[j], dz = k0.z - fpz[j];
                    const float R = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
                    float b = fmaf(R, bpm, k0.w);
                    b = fminf(fmaxf(b, -cenf), wmax - cenf);
                    const float t = b + mp;
                    const float4 v = lds128((__float_as_uint(t) << 4) + smem_addr(stg) - kMagicBitsShift4);
                    const float sr = fmaf(b, v.z, v.x);
                    const float si = fmaf(b, v.w, v.y);
                    float sn, cs;
                    sincosf(fmaf(kph, R, phc), &sn, &cs);
                    acc_r[j] = fmaf(sr, cs, fmaf(-si, sn, acc_r[j]));
                    acc_i[j] = fmaf(sr, sn, fmaf(si, cs, acc_i[j]));
                }
            }
        } else {  // FP64
            const double cyc_per_m = 2.0 * P.fc / P.c;
#pragma unroll 1
            for (int pl = 0; pl < count; ++pl) {
                const Prm &q = S.prm[stage * kChunk + pl];
                const double ax = q.ax, ay = q.ay, az = q.az, dr = q.dr, dph_pi = q.dph / CUDART_PI;
                const double boff = -P.t0_bins * P.bin_rate - (double)q.ws;
                const float4 *st = stg + pl * win;
#pragma unroll
                for (int j = 0; j < kPix; ++j) {
                    const double xi = tx * kTileX + xl, yi = ty * kTileY + ((warp >> 2) + 2 * j) * 4 + ly;
                    const double px = P.g.origin[0] + xi * P.g.ux[0] + yi * P.g.uy[0];
                    const double py = P.g.origin[1] + xi * P.g.ux[1] + yi * P.g.uy[1];
                    const double pz = P.g.origin[2] + xi * P.g.ux[2] + yi * P.g.uy[2];
                    const double dx = ax - px, dy = ay - py, dz = az - pz;
                    const double R = sqrt(dx * dx + dy * dy + dz * dz) + dr;
                    double b = fma(R, 2.0 / P.c * P.bin_rate, boff) - 0.5;
                    b = fmin(fmax(b, 0.0), (double)(win - 2));
                    const double r0 = rint(b);
                    const double f = b - r0;
                    const float4 v = st[(int)r0];
                    const double sr = fma(f, (double)v.z, (double)v.x);
                    const double si = fma(f, (double)v.w, (double)v.y);
                    const double cyc = cyc_per_m * R;
                    double sn, cs;
                    sincospi(2.0 * (cyc - rint(cyc)) + dph_pi, &sn, &cs);
                    dacc_r[j] = fma(sr, cs, fma(-si, sn, dacc_r[j]));
                    dacc_i[j] = fma(sr, sn, fma(si, cs, dacc_i[j]));
                }
            }
        }
        }
        if constexpr (kAhead) failed = __syncthreads_or(failed);
    }

    if (CHECKED && clamped) atomicOr(P.err, kErrIndexClamp);
    if (failed) {
        if (threadIdx.x == 0) drain_after_timeout<TESTF>(P, S.bar, c, nchunks);
        __syncthreads();
        return;
    }

    if constexpr (ADJ) {
        if (nchunks > 0) {
            if (!kAhead) __syncthreads();
            const int last = nchunks - 1;
            if (warp == kStager0)
                flush_projection(P, S, last & 1, p_begin + last * chunk, min(chunk, p_end - p_begin - last * chunk), lane);
        }
        return;
    }

    if (helper) return;
    if constexpr (kSplitBp) {  // s e^{j phase}: (s.x cos - s.y sin, s.y cos + s.x sin)
#pragma unroll
        for (int j = 0; j < kPix; ++j) {
            acc_r[j] = acc_c[j].x - acc_s[j].y;
            acc_i[j] = acc_c[j].y + acc_s[j].x;
        }
    }

    // write the tile
    float2 *dst = P.segments > 1 ? P.partial + (size_t)seg * P.g.nx * P.g.ny : P.image;
    const bool acc_mode = P.segments == 1 && P.accumulate;
    const int x = tx * kTileX + xl;
#pragma unroll
    for (int j = 0; j < kPix; ++j) {
        const int y = ty * kTileY + ((warp >> 2) + 2 * j) * 4 + ly;
        if (x < P.g.nx && y < P.g.ny) {
            float2 v = MODE == SARBP_MODE_FP64 ? make_float2((float)dacc_r[j], (float)dacc_i[j])
                                               : make_float2(acc_r[j], acc_i[j]);
            const size_t idx = (size_t)y * P.g.nx + x;
            if (acc_mode) {
                const float2 o = dst[idx];
                v.x += o.x;
                v.y += o.y;
            }
            dst[idx] = v;
        }
    }
}

// image (=|+=) sum over segments of the partial images, fixed order.
__global__ void reduce_segments_kernel(const float2 *__restrict__ partial, int segments, size_t count,
                                       float2 *__restrict__ image, int accumulate) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count;
         i += (size_t)gridDim.x * blockDim.x) {
        float2 s = accumulate ? image[i] : make_float2(0.f, 0.f);
        for (int k = 0; k < segments; ++k) {
            const float2 v = __ldg(&partial[(size_t)k * count + i]);
            s.x += v.x;
            s.y += v.y;
        }
        image[i] = s;
    }
}

// When set (bp_occupancy), the dispatch below reports the chosen variant's
// resident CTAs per SM there instead of launching it.
thread_local int *t_occupancy = nullptr;

template <int MODE, int STORE, int NTERMS, bool CHECKED, int PIX, bool ADJ = false, int CHUNK = 0, bool TESTF = false,
          bool LIN = false>
cudaError_t launch_variant(const BpPlan &p, cudaStream_t s, int tiles, int tiles_y, int pps, float qq_max) {
    if (CHUNK && p.chunk != CHUNK) return cudaErrorInvalidValue;
    constexpr int threads = kThreads + 32 * helper_warps<MODE, CHECKED, PIX, ADJ, CHUNK, LIN>();
    auto k = bp_kernel<MODE, STORE, NTERMS, CHECKED, PIX, ADJ, CHUNK, TESTF, LIN>;
    const size_t smem = bp_smem_bytes(STORE, p.win, p.chunk);
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(k));
    if (e != cudaSuccess) return e;
    if (t_occupancy) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(t_occupancy, k, threads, smem);
    dim3 grid(tiles, p.segments);
    k<<<grid, threads, smem, s>>>(p, tiles_y, pps, qq_max);
    return cudaGetLastError();
}

template <int MODE, int STORE, int PIX>
cudaError_t launch_split(const BpPlan &p, cudaStream_t s, int tiles, int tiles_y, int pps, float qq_max) {
    if (p.lin) {  // large tiles: the linear-term phase
        if (p.checked)
            return p.nterms == 3 ? launch_variant<MODE, STORE, 3, true, PIX, false, 0, false, true>(p, s, tiles, tiles_y, pps, qq_max)
                                 : launch_variant<MODE, STORE, 4, true, PIX, false, 0, false, true>(p, s, tiles, tiles_y, pps, qq_max);
        if (p.chunk == kChunk)
            return p.nterms == 3 ? launch_variant<MODE, STORE, 3, false, PIX, false, kChunk, false, true>(p, s, tiles, tiles_y, pps, qq_max)
                                 : launch_variant<MODE, STORE, 4, false, PIX, false, kChunk, false, true>(p, s, tiles, tiles_y, pps, qq_max);
        return p.nterms == 3 ? launch_variant<MODE, STORE, 3, false, PIX, false, 0, false, true>(p, s, tiles, tiles_y, pps, qq_max)
                             : launch_variant<MODE, STORE, 4, false, PIX, false, 0, false, true>(p, s, tiles, tiles_y, pps, qq_max);
    }
    if (p.checked)
        return p.nterms == 3 ? launch_variant<MODE, STORE, 3, true, PIX>(p, s, tiles, tiles_y, pps, qq_max)
                             : launch_variant<MODE, STORE, 4, true, PIX>(p, s, tiles, tiles_y, pps, qq_max);
    if (p.chunk == kChunk)
        return p.nterms == 3 ? launch_variant<MODE, STORE, 3, false, PIX, false, kChunk>(p, s, tiles, tiles_y, pps, qq_max)
                             : launch_variant<MODE, STORE, 4, false, PIX, false, kChunk>(p, s, tiles, tiles_y, pps, qq_max);
    return p.nterms == 3 ? launch_variant<MODE, STORE, 3, false, PIX>(p, s, tiles, tiles_y, pps, qq_max)
                         : launch_variant<MODE, STORE, 4, false, PIX>(p, s, tiles, tiles_y, pps, qq_max);
}

// A plan asks for the test variants when it carries a fault or a wait limit
// other than the default (sarbp_debug_set); they exist for 8-pixel columns, with
// the staging schemes of production (helper_warps): two helpers for 16-pulse
// chunks, one for smaller ones, none for FP64 and FP32.  Their phase is the series form.
bool bp_testing(const BpPlan &p) { return p.fault_chunk >= 0 || p.wait_ns != kDefaultWaitNs; }

template <int MODE, int STORE, bool ADJ>
cudaError_t launch_testf_mode(const BpPlan &p, cudaStream_t s, int tiles, int tiles_y, int pps, float qq_max) {
    if constexpr (MODE == SARBP_MODE_SPLIT || MODE == SARBP_MODE_FP16STORE) {
        if (p.chunk == kChunk)
            return p.nterms == 3 ? launch_variant<MODE, STORE, 3, false, 8, ADJ, kChunk, true>(p, s, tiles, tiles_y, pps, qq_max)
                                 : launch_variant<MODE, STORE, 4, false, 8, ADJ, kChunk, true>(p, s, tiles, tiles_y, pps, qq_max);
        return p.nterms == 3 ? launch_variant<MODE, STORE, 3, false, 8, ADJ, 0, true>(p, s, tiles, tiles_y, pps, qq_max)
                             : launch_variant<MODE, STORE, 4, false, 8, ADJ, 0, true>(p, s, tiles, tiles_y, pps, qq_max);
    } else
        return launch_variant<MODE, STORE, 4, false, 8, false, 0, true>(p, s, tiles, tiles_y, pps, qq_max);
}

template <bool ADJ>
cudaError_t launch_testf(const BpPlan &p, cudaStream_t s, int tiles, int tiles_y, int pps, float qq_max) {
    if (p.pix != 8) return cudaErrorNotSupported;
    const bool fp16 = p.storage == SARBP_STORE_C32H;
    if constexpr (ADJ)
        return fp16 ? launch_testf_mode<SARBP_MODE_SPLIT, SARBP_STORE_C32H, true>(p, s, tiles, tiles_y, pps, qq_max)
                    : launch_testf_mode<SARBP_MODE_SPLIT, SARBP_STORE_C64, true>(p, s, tiles, tiles_y, pps, qq_max);
    switch (p.mode) {
        case SARBP_MODE_FP64:
            return fp16 ? launch_testf_mode<SARBP_MODE_FP64, SARBP_STORE_C32H, false>(p, s, tiles, tiles_y, pps, qq_max)
                        : launch_testf_mode<SARBP_MODE_FP64, SARBP_STORE_C64, false>(p, s, tiles, tiles_y, pps, qq_max);
        case SARBP_MODE_FP32:
            return fp16 ? launch_testf_mode<SARBP_MODE_FP32, SARBP_STORE_C32H, false>(p, s, tiles, tiles_y, pps, qq_max)
                        : launch_testf_mode<SARBP_MODE_FP32, SARBP_STORE_C64, false>(p, s, tiles, tiles_y, pps, qq_max);
        default:
            return fp16 ? launch_testf_mode<SARBP_MODE_SPLIT, SARBP_STORE_C32H, false>(p, s, tiles, tiles_y, pps, qq_max)
                        : launch_testf_mode<SARBP_MODE_SPLIT, SARBP_STORE_C64, false>(p, s, tiles, tiles_y, pps, qq_max);
    }
}

template <int PIX>
cudaError_t launch_pix(const BpPlan &p, cudaStream_t s, int tiles, int tiles_y, int pps, float qq_max) {
    const bool fp16 = p.storage == SARBP_STORE_C32H;
    switch (p.mode) {
        case SARBP_MODE_FP64:
            return fp16 ? launch_variant<SARBP_MODE_FP64, SARBP_STORE_C32H, 4, false, PIX>(p, s, tiles, tiles_y, pps, qq_max)
                        : launch_variant<SARBP_MODE_FP64, SARBP_STORE_C64, 4, false, PIX>(p, s, tiles, tiles_y, pps, qq_max);
        case SARBP_MODE_FP32:
            return fp16 ? launch_variant<SARBP_MODE_FP32, SARBP_STORE_C32H, 4, false, PIX>(p, s, tiles, tiles_y, pps, qq_max)
                        : launch_variant<SARBP_MODE_FP32, SARBP_STORE_C64, 4, false, PIX>(p, s, tiles, tiles_y, pps, qq_max);
        default:
            return fp16 ? launch_split<SARBP_MODE_SPLIT, SARBP_STORE_C32H, PIX>(p, s, tiles, tiles_y, pps, qq_max)
                        : launch_split<SARBP_MODE_SPLIT, SARBP_STORE_C64, PIX>(p, s, tiles, tiles_y, pps, qq_max);
    }
}

// out[p] = sum over tiles of proj[tile][p] in FP64.  A CTA takes 32 pulses
// (one per lane, coalesced rows); its 16 warps take tiles w, w + 16, ... and
// their partial sums combine in warp order, so the order is fixed and the
// result deterministic.  (One thread per pulse walking every tile kept only
// np / 128 CTAs busy: 0.15 ms for 512 tiles x 4096 pulses.)
constexpr int kProjWarps = 16;
__global__ void __launch_bounds__(32 * kProjWarps)
    proj_reduce_kernel(const float2 *__restrict__ proj, int tiles, int np, double2 *__restrict__ out) {
    __shared__ double2 part[kProjWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    double sr = 0.0, si = 0.0;
    if (p < np) {
        for (int t = warp; t < tiles; t += kProjWarps) {
            const float2 v = __ldg(&proj[(size_t)t * np + p]);
            sr += v.x;
            si += v.y;
        }
    }
    part[warp][lane] = make_double2(sr, si);
    __syncthreads();
    if (warp == 0 && p < np) {
        double r = 0.0, i = 0.0;
#pragma unroll
        for (int w = 0; w < kProjWarps; ++w) {
            r += part[w][lane].x;
            i += part[w][lane].y;
        }
        out[p] = make_double2(r, i);
    }
}

template <int STORE, int PIX>
cudaError_t launch_proj_pix(const BpPlan &p, cudaStream_t s, int tiles, int tiles_y, int pps, float qq_max) {
    if (p.lin) {  // large tiles: the linear-term phase
        if constexpr (PIX == 8) {
            if (p.chunk == kChunk)
                return p.nterms == 3
                           ? launch_variant<SARBP_MODE_SPLIT, STORE, 3, false, PIX, true, kChunk, false, true>(p, s, tiles, tiles_y, pps, qq_max)
                           : launch_variant<SARBP_MODE_SPLIT, STORE, 4, false, PIX, true, kChunk, false, true>(p, s, tiles, tiles_y, pps, qq_max);
        }
        return p.nterms == 3 ? launch_variant<SARBP_MODE_SPLIT, STORE, 3, false, PIX, true, 0, false, true>(p, s, tiles, tiles_y, pps, qq_max)
                             : launch_variant<SARBP_MODE_SPLIT, STORE, 4, false, PIX, true, 0, false, true>(p, s, tiles, tiles_y, pps, qq_max);
    }
    if constexpr (PIX == 8) {  // the usual tile: pulse chunk fixed at compile time
        if (p.chunk == kChunk)
            return p.nterms == 3
                       ? launch_variant<SARBP_MODE_SPLIT, STORE, 3, false, PIX, true, kChunk>(p, s, tiles, tiles_y, pps, qq_max)
                       : launch_variant<SARBP_MODE_SPLIT, STORE, 4, false, PIX, true, kChunk>(p, s, tiles, tiles_y, pps, qq_max);
    }
    return p.nterms == 3 ? launch_variant<SARBP_MODE_SPLIT, STORE, 3, false, PIX, true>(p, s, tiles, tiles_y, pps, qq_max)
                         : launch_variant<SARBP_MODE_SPLIT, STORE, 4, false, PIX, true>(p, s, tiles, tiles_y, pps, qq_max);
}

void launch_geometry(const BpPlan &p, int *tiles, int *tiles_y, int *pps, float *qq_max) {
    const int tile_y = 8 * p.pix;
    const int tiles_x = (p.g.nx + kTileX - 1) / kTileX;
    *tiles_y = (p.g.ny + tile_y - 1) / tile_y;
    *tiles = tiles_x * *tiles_y;
    int n = (p.np + p.segments - 1) / p.segments;
    *pps = (n + kChunk - 1) / kChunk * kChunk;
    // |q|^2 bound over a tile (pixel offsets from the tile centre)
    const double hx = 0.5 * (kTileX - 1), hy = 0.5 * (tile_y - 1);
    *qq_max = (float)(hx * hx * p.g.g11 + 2.0 * hx * hy * fabs(p.g.g12) + hy * hy * p.g.g22);
}

cudaError_t launch_pulse_refs(const BpPlan &p, cudaStream_t s) {
    pulse_ref_kernel<<<(p.np + 127) / 128, 128, 0, s>>>(p.apc, p.np, p.g, p.drange, p.dphase,
                                                         2.0 / p.c * p.bin_rate, 2.0 * p.fc / p.c, p.pref);
    return cudaGetLastError();
}

}  // namespace

size_t bp_tiles(const BpPlan &p) {
    int tiles, tiles_y, pps;
    float qq;
    launch_geometry(p, &tiles, &tiles_y, &pps, &qq);
    return (size_t)tiles;
}

cudaError_t launch_project(const BpPlan &p, double2 *out, cudaStream_t s, int *launches) {
    if (p.np <= 0) return cudaSuccess;
    if (p.mode != SARBP_MODE_SPLIT && p.mode != SARBP_MODE_FP16STORE) return cudaErrorInvalidValue;
    if (p.pix != 8 && p.pix != 4 && p.pix != 2) return cudaErrorInvalidValue;
    if (!p.weight || !p.proj || !out) return cudaErrorInvalidValue;
    if (p.g.nx <= 0 || p.g.ny <= 0) return cudaMemsetAsync(out, 0, sizeof(double2) * p.np, s);
    int tiles, tiles_y, pps;
    float qq_max;
    launch_geometry(p, &tiles, &tiles_y, &pps, &qq_max);
    cudaError_t e = launch_pulse_refs(p, s);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
    const bool fp16 = p.storage == SARBP_STORE_C32H;
    if (bp_testing(p)) e = launch_testf<true>(p, s, tiles, tiles_y, pps, qq_max);
    else if (p.pix == 8) e = fp16 ? launch_proj_pix<SARBP_STORE_C32H, 8>(p, s, tiles, tiles_y, pps, qq_max)
                             : launch_proj_pix<SARBP_STORE_C64, 8>(p, s, tiles, tiles_y, pps, qq_max);
    else if (p.pix == 4) e = fp16 ? launch_proj_pix<SARBP_STORE_C32H, 4>(p, s, tiles, tiles_y, pps, qq_max)
                                  : launch_proj_pix<SARBP_STORE_C64, 4>(p, s, tiles, tiles_y, pps, qq_max);
    else e = fp16 ? launch_proj_pix<SARBP_STORE_C32H, 2>(p, s, tiles, tiles_y, pps, qq_max)
                  : launch_proj_pix<SARBP_STORE_C64, 2>(p, s, tiles, tiles_y, pps, qq_max);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
    proj_reduce_kernel<<<(p.np + 31) / 32, 32 * kProjWarps, 0, s>>>(p.proj, tiles, p.np, out);
    e = cudaGetLastError();
    if (launches) ++*launches;
    return e;
}

cudaError_t bp_occupancy(const BpPlan &p, int *ctas_per_sm) {
    *ctas_per_sm = 0;
    if (p.pix != 8 && p.pix != 4 && p.pix != 2) return cudaErrorInvalidValue;
    int tiles, tiles_y, pps;
    float qq_max;
    launch_geometry(p, &tiles, &tiles_y, &pps, &qq_max);
    t_occupancy = ctas_per_sm;
    cudaError_t e = p.pix == 8 ? launch_pix<8>(p, nullptr, tiles, tiles_y, pps, qq_max)
                  : p.pix == 4 ? launch_pix<4>(p, nullptr, tiles, tiles_y, pps, qq_max)
                               : launch_pix<2>(p, nullptr, tiles, tiles_y, pps, qq_max);
    t_occupancy = nullptr;
    return e;
}

void bp_tile_dims(int pix, int *tile_x, int *tile_y) {
    *tile_x = kTileX;
    *tile_y = 8 * pix;
}

int bp_max_chunk() { return kChunk; }

size_t bp_smem_bytes(int storage, int win, int chunk) {
    return (size_t)2 * chunk * win * 16 + (size_t)kStages * chunk * win * raw_esize(storage) +
           kStages * kChunk * sizeof(Prm) +
           kStages * sizeof(uint64_t) + 2 * kWarps * kChunk * sizeof(float2);
}

// ---------------------------------------------------------------- planning extremes
// One thread per (pulse, lattice row), nine points.  GB300 issues an FP64 warp
// instruction every 16 clocks per SM, so the cost is the FP64 work: a first pass
// in FP32 (coordinates as float pairs, so differences keep FP32 relative
// accuracy) finds the block's extremes, and only the points within the FP32
// error of one of them are evaluated in FP64, by the host's own expressions.
// The largest cosine is the smallest sine, |axis x w| / (|axis| R), which FP32
// separates to a microradian even where the cosines all round to 1 (a short
// aperture at broadside: half its points lie within FP32 rounding of the largest
// cosine, and evaluating them took 28 us at 256 pulses).  FP32 errors: squared
// range 11 ulp (7e-7 relative, kExtR2 is over 5 times that), sine 9e-7 absolute
// (kExtSin 4 times).  Points whose distance is not well above the rounding of
// the coordinates, or whose FP32 terms are not ordinary numbers, are always
// evaluated.  They go through a list in shared memory, so that the FP64 chain
// (about 70 instructions with a square root and a quotient) runs once for a
// block's few points side by side, not once per lattice column that holds one in
// some lane.  Min and max do not depend on the order, so the bits are the host's.
// The last block to finish hands the result to the host (mapped memory, `seq`
// last) and resets the state for the next call: one launch, no copy.  With the
// polled result (extremes_wait in api.cpp) a back-projection call of 256 pulses
// onto 128^2 pixels took 63 us instead of 129 before the list and before small
// images filled the chip (plan.cpp); with that 49.2, with the list 46.7 (64
// threads), 44.2 (128) and 42.7 (no reads of the state ahead of its atomics, one
// system fence).  Threads per block, same call: 32 49.7, 64 47, 96 46, 128 42.7,
// 192 42.9, 256 47, 288 43.7, 576 45.6.
constexpr int kExtThreads = 128;
constexpr float kExtR2 = 4e-6f, kExtSin = 4e-6f;
struct ExtAxes {
    double len[2];     // |ux|, |uy|
    float unit[2][3];  // ux / |ux|, uy / |uy| (0 for an axis of length 0)
};

__device__ __forceinline__ void ext_split(double v, float &h, float &l) {
    h = (float)v;
    l = (float)(v - (double)h);
}

__global__ void __launch_bounds__(kExtThreads)
    bp_extremes_kernel(const double *apc, int np, const sarbp_grid g, const ExtAxes ax, unsigned long long *state,
                       volatile unsigned long long *result, unsigned long long seq) {
    constexpr int kPts = kLattice * kLattice;
    __shared__ double P[kPts][3];
    __shared__ float Ph[kPts][3], Pl[kPts][3];
    __shared__ float red[4][kExtThreads / 32];
    __shared__ unsigned long long ext[5];
    __shared__ unsigned short list[kExtThreads * kLattice];  // points to evaluate: thread * 9 + column, cosines wanted
    __shared__ int count;
    __shared__ bool last;
    constexpr int kCosX = 1 << 14, kCosY = 1 << 15;
    static_assert(kExtThreads * kLattice <= kCosX, "list entry");
    const int t = threadIdx.x;
    const long long i = blockIdx.x * (long long)kExtThreads + t;
    const int p = (int)(i / kLattice), u = (int)(i - (long long)p * kLattice);
    bool live = i < (long long)np * kLattice;
    double a[3] = {0.0, 0.0, 0.0};  // loaded ahead of the lattice's FP64 work
    if (live)
        for (int d = 0; d < 3; ++d) a[d] = apc[3 * (size_t)p + d];
    for (int k = t; k < kPts; k += kExtThreads) {
        ext_lattice(g, k / kLattice, k % kLattice, P[k]);
        for (int d = 0; d < 3; ++d) ext_split(P[k][d], Ph[k][d], Pl[k][d]);
    }
    if (t == 0) count = 0;
    if (t < 5) ext[t] = t == 0 ? (unsigned long long)__double_as_longlong(1e300) : 0ull;
    __syncthreads();
    float ah[3], al[3], size = 0.f;
    if (live && (!isfinite(a[0]) || !isfinite(a[1]) || !isfinite(a[2]))) {
        live = false;
        ext[4] = 1ull;
    }
    for (int d = 0; d < 3; ++d) {
        ext_split(a[d], ah[d], al[d]);
        size = fmaxf(size, fabsf(ah[d]));
    }
    // |unit x w| / R: the sine of the angle to an axis
    auto sine = [](const float *e, const float *w, float inv) {
        const float a = e[1] * w[2] - e[2] * w[1], b = e[2] * w[0] - e[0] * w[2], c = e[0] * w[1] - e[1] * w[0];
        return sqrtf(fmaf(a, a, fmaf(b, b, c * c))) * inv;
    };
    auto terms = [&](int k, float &r2, float &sx, float &sy, float &always) {
        float w[3], s = size;
        for (int d = 0; d < 3; ++d) {
            w[d] = (Ph[k][d] - ah[d]) + (Pl[k][d] - al[d]);
            s = fmaxf(s, fabsf(Ph[k][d]));
        }
        r2 = fmaf(w[0], w[0], fmaf(w[1], w[1], w[2] * w[2]));
        const float inv = rsqrtf(r2);
        sx = sine(ax.unit[0], w, inv);
        sy = sine(ax.unit[1], w, inv);
        always = fmaxf(1e-30f, s * 2.4e-7f * (s * 2.4e-7f));
    };
    float m[4] = {0.f, 3.4e38f, 3.4e38f, 3.4e38f};  // max r2, min r2, min sines (fminf / fmaxf drop NaN)
    if (live) {
#pragma unroll 3
        for (int v = 0; v < kLattice; ++v) {
            float r2, sx, sy, always;
            terms(u * kLattice + v, r2, sx, sy, always);
            m[0] = fmaxf(m[0], r2);
            m[1] = fminf(m[1], r2);
            m[2] = fminf(m[2], sx);
            m[3] = fminf(m[3], sy);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m[0] = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], o));
#pragma unroll
        for (int k = 1; k < 4; ++k) m[k] = fminf(m[k], __shfl_xor_sync(0xffffffffu, m[k], o));
    }
    if ((t & 31) == 0)
        for (int k = 0; k < 4; ++k) red[k][t >> 5] = m[k];
    __syncthreads();
    for (int w = 0; w < kExtThreads / 32; ++w) {
        m[0] = fmaxf(m[0], red[0][w]);
        for (int k = 1; k < 4; ++k) m[k] = fminf(m[k], red[k][w]);
    }
    if (live) {
        const float hi = m[0] * (1.f - kExtR2), lo = m[1] * (1.f + kExtR2), ex = m[2] + kExtSin, ey = m[3] + kExtSin;
#pragma unroll
        for (int v = 0; v < kLattice; ++v) {
            float r2, sx, sy, always;
            terms(u * kLattice + v, r2, sx, sy, always);
            // false only for ordinary numbers clear of the extreme; a cosine's
            // quotient and square root only where it may be the largest
            const bool all = !(r2 > always);
            const bool range = all || !(r2 > lo) || !(r2 < hi);
            const bool cos_x = all || !(sx > ex), cos_y = all || !(sy > ey);
            if (range || cos_x || cos_y)
                list[atomicAdd(&count, 1)] = (unsigned short)((t * kLattice + v) | (cos_x ? kCosX : 0) | (cos_y ? kCosY : 0));
        }
    }
    __syncthreads();
    if (t < count) {
        ExtAcc acc;
        ext_acc_init(acc);
        for (int e = t; e < count; e += kExtThreads) {
            const int c = list[e], tv = c & (kCosX - 1), tt = tv / kLattice;
            const long long it = blockIdx.x * (long long)kExtThreads + tt;
            const long long pe = it / kLattice;
            const int k = (int)(it - pe * kLattice) * kLattice + tv - tt * kLattice;
            double ae[3], r2d, nx, ny;
            for (int d = 0; d < 3; ++d) ae[d] = apc[3 * (size_t)pe + d];
            ext_terms(g, P[k], ae, r2d, nx, ny);
            acc.r2min = fmin(acc.r2min, r2d);
            acc.r2max = fmax(acc.r2max, r2d);
            if (r2d > 0) {
                if ((c & kCosX) && ax.len[0] > 0) ext_cos(acc.cx, nx, r2d, ax.len[0]);
                if ((c & kCosY) && ax.len[1] > 0) ext_cos(acc.sy, ny, r2d, ax.len[1]);
            }
        }
        atomicMin(&ext[0], (unsigned long long)__double_as_longlong(acc.r2min));
        atomicMax(&ext[1], (unsigned long long)__double_as_longlong(acc.r2max));
        atomicMax(&ext[2], (unsigned long long)__double_as_longlong(acc.cx.best));
        atomicMax(&ext[3], (unsigned long long)__double_as_longlong(acc.sy.best));
    }
    __syncthreads();
    // all four quantities are >= 0, where the unsigned order of the bits is the
    // numeric order
    if (t == 0) {
        atomicMin(&state[0], ext[0]);
        for (int k = 1; k < 5; ++k)
            if (ext[k]) atomicMax(&state[k], ext[k]);
        __threadfence();
        last = atomicAdd(&state[5], 1ull) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && t < 5) {
        __threadfence();
        result[t] = atomicExch(&state[t], t == 0 ? (unsigned long long)__double_as_longlong(1e300) : 0ull);
        if (t == 0) state[5] = 0ull;
    }
    __syncthreads();
    if (last && t == 0) {
        __threadfence_system();  // covers what this block wrote before the barrier
        result[5] = seq;
    }
}

void bp_extremes_state_init(unsigned long long (&state)[6]) {
    const double none = 1e300;
    std::memcpy(&state[0], &none, sizeof none);
    for (int k = 1; k < 6; ++k) state[k] = 0ull;
}

cudaError_t launch_bp_extremes(const double *apc, int np, const sarbp_grid &g, unsigned long long *state,
                               unsigned long long *result, unsigned long long seq, cudaStream_t s) {
    if (np <= 0) return cudaErrorInvalidValue;
    ExtAxes ax;
    ext_axes(g, &ax.len[0], &ax.len[1]);
    for (int k = 0; k < 3; ++k) {
        ax.unit[0][k] = ax.len[0] > 0 ? (float)(g.ux[k] / ax.len[0]) : 0.f;
        ax.unit[1][k] = ax.len[1] > 0 ? (float)(g.uy[k] / ax.len[1]) : 0.f;
    }
    const long long total = (long long)np * kLattice;  // threads: (pulse, lattice row)
    bp_extremes_kernel<<<(unsigned)((total + kExtThreads - 1) / kExtThreads), kExtThreads, 0, s>>>(apc, np, g, ax, state,
                                                                                              result, seq);
    return cudaGetLastError();
}

cudaError_t launch_bp(const BpPlan &p, cudaStream_t s, int *launches) {
    if (p.np <= 0 || p.g.nx <= 0 || p.g.ny <= 0) return cudaSuccess;
    if (p.pix != 8 && p.pix != 4 && p.pix != 2) return cudaErrorInvalidValue;
    int tiles, tiles_y, pps;
    float qq_max;
    launch_geometry(p, &tiles, &tiles_y, &pps, &qq_max);
    cudaError_t e;
    if (p.mode == SARBP_MODE_SPLIT || p.mode == SARBP_MODE_FP16STORE) {
        e = launch_pulse_refs(p, s);
        if (e != cudaSuccess) return e;
        if (launches) ++*launches;
    }
    if (bp_testing(p)) e = launch_testf<false>(p, s, tiles, tiles_y, pps, qq_max);
    else if (p.pix == 8) e = launch_pix<8>(p, s, tiles, tiles_y, pps, qq_max);
    else if (p.pix == 4) e = launch_pix<4>(p, s, tiles, tiles_y, pps, qq_max);
    else e = launch_pix<2>(p, s, tiles, tiles_y, pps, qq_max);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
    if (p.segments > 1) {
        const size_t count = (size_t)p.g.nx * p.g.ny;
        const int blocks = (int)std::min<size_t>((count + 255) / 256, (size_t)current_sms() * 8);
        reduce_segments_kernel<<<blocks, 256, 0, s>>>(p.partial, p.segments, count, p.image, p.accumulate);
        e = cudaGetLastError();
        if (launches) ++*launches;
    }
    return e;
}

}  // namespace sarbp
