// po_adjoint_pk.cu -- pair-packed adjoint kernels (mixed precision).
//
// Near field: one fused kernel computes, for every (source, target) pair,
// both halves of the near-field adjoint of po_adjoint.cu:
//   source side  Jbar', Mbar' (12 accumulators) and n_s . grad_d phi (1);
//   target side  n_t . grad_d phi, summed over the sources.
// Both displacement terms share the pair's geometry, phase, coefficients and
// S = G (D1 alpha + D2 beta + D3 W.R_hat); only the normal differs
// (n . grad_d phi = (1/R) Re[(R_hat.n) S + C2 (grad(beta).n) + C3 (W.n)]).
//
// Layout: a thread owns one source (forward-packed record, registers) and
// streams PAIRS of targets through shared memory with TMA bulk copies; every
// packed FP32x2 operation works on the two targets of a pair (lane x: target
// 2p, lane y: target 2p + 1). Source-side sums stay per thread (float-float
// totals per tile). Target-side values are transposed through shared memory
// every kFlush target pairs, summed over the CTA's sources, and added into
// an FP64 accumulator per target with atomicAdd (the order of those adds
// varies from run to run: grad_dt is reproducible to ~1e-16, not bitwise).
//
// The three projections of W (on R_hat, n_s, n_t) come from one complex
// vector per pair, Z = b x J - a x M: W.v = -v.Z (scalar triple product).
// The far field's adjoint is in po_ff_adjoint.cu.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <cstdint>
#include <type_traits>

#include "po_device.cuh"
#include "po_kernels.cuh"

namespace po {

// Pair-packed cotangent record, float2 slots (target 2p, target 2p + 1):
//   0-2 hi position, 3-5 lo position (turns), 6-11 gE (re, im) x y z, 12-17 gH;
//   with the target displacement: 18-20 n_t, 21-22 a.n_t; with M as well:
//   23-24 b.n_t (a = conj(gE), b = conj(gH)). A padding target has zero
//   cotangent.
// The scalar kind has the near-field layout.
__host__ __device__ constexpr int adj2_rec(bool has_m, bool want_t) { return want_t ? (has_m ? 13 : 12) : 9; }

constexpr int kPairsA2 = PO_PAIRS_A;   // target pairs per shared-memory stage
#ifndef PO_FLUSH_A
#define PO_FLUSH_A 16
#endif
constexpr int kFlush = PO_FLUSH_A;   // target pairs per transpose of the target-side values
constexpr int kSegs = kThreadsA / kFlush;   // threads summing one target pair
static_assert(kThreadsA == 128 && (kFlush == 16 || kFlush == 32),
              "the transpose maps 128 threads onto 16 pairs x 8 segments or 32 pairs x 4");

// Per-thread constants of the thread's source (forward-packed record).
struct SrcC {
    float sh[3], sl[3], n[3];
    float J[6], M[6];            // (re, im) x y z
    float Jn[2], Mn[2];          // J.n_s, M.n_s
};

// The geometry of a target pair record against the thread's source, in the
// split representation: S0 = |d_hi|^2 (exact), S1 the rest of |d|^2, 1/R
// (approximate), R, d = t - s, and n_s . d. adj_nf_pair2 and
// adj_nf_band_scan both use these, so the scan's band decision is the pair
// loop's, bit for bit.
struct AdjGeo2 {
    float2 S0, S1, rinv0, Rh, dx, dy, dz, ndd;
};

__device__ __forceinline__ AdjGeo2 adj_geo2(const float2 *r, const SrcC &s)
{
    AdjGeo2 g;
    const float2 dhx = sub2(r[0], dup2(s.sh[0])), dhy = sub2(r[1], dup2(s.sh[1])), dhz = sub2(r[2], dup2(s.sh[2]));
    const float2 dlx = sub2(r[3], dup2(s.sl[0])), dly = sub2(r[4], dup2(s.sl[1])), dlz = sub2(r[5], dup2(s.sl[2]));
    const float2 two = dup2(2.0f);
    g.S0 = fma2(dhz, dhz, fma2(dhy, dhy, mul2(dhx, dhx)));
    g.S1 = fma2(dlz, fma2(two, dhz, dlz), fma2(dly, fma2(two, dhy, dly), mul2(dlx, fma2(two, dhx, dlx))));
    const float2 R2 = add2(g.S0, g.S1);
    g.rinv0 = make_float2(rsqrt_ftz(R2.x), rsqrt_ftz(R2.y));
    g.Rh = mul2(R2, g.rinv0);
    g.dx = add2(dhx, dlx);
    g.dy = add2(dhy, dly);
    g.dz = add2(dhz, dlz);
    g.ndd = fma2(dup2(s.n[2]), g.dz, fma2(dup2(s.n[1]), g.dy, mul2(dup2(s.n[0]), g.dx)));
    return g;
}

// One pair of targets against the thread's source. acc: 12 current
// accumulators + the source displacement term; vt: the two targets' terms.
// band: set when a pair lies inside the tangent band (left out here; the
// kernel lists it afterwards with adj_band_scan).
template <int T, bool HAS_M, bool WANT_C, bool WANT_D, bool WANT_T>
__device__ __forceinline__ void adj_nf_pair2(float2 *acc, float2 &vt, const float2 *r, const SrcC &s, bool &band)
{
    const AdjGeo2 g = adj_geo2(r, s);
    const float2 S0 = g.S0, S1 = g.S1, rinv0 = g.rinv0, Rh = g.Rh, dx = g.dx, dy = g.dy, dz = g.dz, ndd = g.ndd;
    float2 sn, cs, tq;
    phase_sincos2(S0, S1, Rh, rinv0, sn, cs, tq);
    cs = flip_parity(cs, tq);   // cos, sin of k R
    sn = flip_parity(sn, tq);
    const float2 bw = mul2(dup2(kTangentBand), Rh);
    band = band || (fabsf(ndd.x) < bw.x) || (fabsf(ndd.y) < bw.y);
    const float2 rinv = make_float2(ndd.x >= bw.x ? rinv0.x : 0.0f, ndd.y >= bw.y ? rinv0.y : 0.0f);
    const float2 ex = mul2(dx, rinv), ey = mul2(dy, rinv), ez = mul2(dz, rinv);
    const float2 u = mul2(rinv, dup2(0.159154943091895336f));
    // c1 = Gu (t u + j(u^2 - 1)), C2 = -3 c1 - 2 j Gu, C3 = Gu (-u + j t)
    const float2 gur = mul2(cs, u);
    const float2 gui = mul2(T > 0 ? sn : neg2(sn), u);
    const float2 tu = T > 0 ? u : neg2(u);
    const float2 b = fma2(u, u, dup2(-1.0f));
    const float2 c1r = fma2(gur, tu, mul2(neg2(gui), b));
    const float2 c1i = fma2(gur, b, mul2(gui, tu));
    const float2 C2r = fma2(dup2(-3.0f), c1r, add2(gui, gui));
    const float2 C2i = fma2(dup2(-3.0f), c1i, mul2(dup2(-2.0f), gur));
    const float2 C3r = T > 0 ? fma2(neg2(gur), u, neg2(gui)) : fma2(neg2(gur), u, gui);
    const float2 C3i = T > 0 ? fma2(neg2(gui), u, gur) : fma2(neg2(gui), u, neg2(gur));

    const float2 Exr = r[6], Exi = r[7], Eyr = r[8], Eyi = r[9], Ezr = r[10], Ezi = r[11];
    const float2 Hxr = r[12], Hxi = r[13], Hyr = r[14], Hyi = r[15], Hzr = r[16], Hzi = r[17];
    // gE.R_hat, gH.R_hat
    const float2 ger = fma2(Ezr, ez, fma2(Eyr, ey, mul2(Exr, ex))), gei = fma2(Ezi, ez, fma2(Eyi, ey, mul2(Exi, ex)));
    const float2 ghr = fma2(Hzr, ez, fma2(Hyr, ey, mul2(Hxr, ex))), ghi = fma2(Hzi, ez, fma2(Hyi, ey, mul2(Hxi, ex)));
    if (WANT_C) {
        // P = conj(C2) (gE.R_hat), Q = conj(C2) (gH.R_hat)
        const float2 Pr = fma2(C2r, ger, mul2(C2i, gei)), Pi = fma2(C2r, gei, mul2(neg2(C2i), ger));
        const float2 Qr = fma2(C2r, ghr, mul2(C2i, ghi)), Qi = fma2(C2r, ghi, mul2(neg2(C2i), ghr));
        // K = conj(C3) gH, L = conj(C3) gE
        const float2 Kxr = fma2(C3r, Hxr, mul2(C3i, Hxi)), Kxi = fma2(C3r, Hxi, mul2(neg2(C3i), Hxr));
        const float2 Kyr = fma2(C3r, Hyr, mul2(C3i, Hyi)), Kyi = fma2(C3r, Hyi, mul2(neg2(C3i), Hyr));
        const float2 Kzr = fma2(C3r, Hzr, mul2(C3i, Hzi)), Kzi = fma2(C3r, Hzi, mul2(neg2(C3i), Hzr));
        const float2 Lxr = fma2(C3r, Exr, mul2(C3i, Exi)), Lxi = fma2(C3r, Exi, mul2(neg2(C3i), Exr));
        const float2 Lyr = fma2(C3r, Eyr, mul2(C3i, Eyi)), Lyi = fma2(C3r, Eyi, mul2(neg2(C3i), Eyr));
        const float2 Lzr = fma2(C3r, Ezr, mul2(C3i, Ezi)), Lzi = fma2(C3r, Ezi, mul2(neg2(C3i), Ezr));
        // Jbar' += conj(c1) gE + P R_hat + K x R_hat
        acc[0] = fma2(c1r, Exr, fma2(c1i, Exi, fma2(Pr, ex, fma2(Kyr, ez, fma2(neg2(Kzr), ey, acc[0])))));
        acc[1] = fma2(c1r, Eyr, fma2(c1i, Eyi, fma2(Pr, ey, fma2(Kzr, ex, fma2(neg2(Kxr), ez, acc[1])))));
        acc[2] = fma2(c1r, Ezr, fma2(c1i, Ezi, fma2(Pr, ez, fma2(Kxr, ey, fma2(neg2(Kyr), ex, acc[2])))));
        acc[3] = fma2(c1r, Exi, fma2(neg2(c1i), Exr, fma2(Pi, ex, fma2(Kyi, ez, fma2(neg2(Kzi), ey, acc[3])))));
        acc[4] = fma2(c1r, Eyi, fma2(neg2(c1i), Eyr, fma2(Pi, ey, fma2(Kzi, ex, fma2(neg2(Kxi), ez, acc[4])))));
        acc[5] = fma2(c1r, Ezi, fma2(neg2(c1i), Ezr, fma2(Pi, ez, fma2(Kxi, ey, fma2(neg2(Kyi), ex, acc[5])))));
        // Mbar' += conj(c1) gH + Q R_hat - L x R_hat
        acc[6] = fma2(c1r, Hxr, fma2(c1i, Hxi, fma2(Qr, ex, fma2(neg2(Lyr), ez, fma2(Lzr, ey, acc[6])))));
        acc[7] = fma2(c1r, Hyr, fma2(c1i, Hyi, fma2(Qr, ey, fma2(neg2(Lzr), ex, fma2(Lxr, ez, acc[7])))));
        acc[8] = fma2(c1r, Hzr, fma2(c1i, Hzi, fma2(Qr, ez, fma2(neg2(Lxr), ey, fma2(Lyr, ex, acc[8])))));
        acc[9] = fma2(c1r, Hxi, fma2(neg2(c1i), Hxr, fma2(Qi, ex, fma2(neg2(Lyi), ez, fma2(Lzi, ey, acc[9])))));
        acc[10] = fma2(c1r, Hyi, fma2(neg2(c1i), Hyr, fma2(Qi, ey, fma2(neg2(Lzi), ex, fma2(Lxi, ez, acc[10])))));
        acc[11] = fma2(c1r, Hzi, fma2(neg2(c1i), Hzr, fma2(Qi, ez, fma2(neg2(Lxi), ey, fma2(Lyi, ex, acc[11])))));
    }
    if (!WANT_D && !WANT_T) return;

    // a = conj(gE), b = conj(gH): alpha = a.J (+ b.M), beta = (J.R_hat)(a.R_hat) (+ (M.R_hat)(b.R_hat)),
    // w = W.R_hat = -b.(J x R_hat) (+ a.(M x R_hat))
    const float2 Jxr = dup2(s.J[0]), Jxi = dup2(s.J[1]), Jyr = dup2(s.J[2]), Jyi = dup2(s.J[3]);
    const float2 Jzr = dup2(s.J[4]), Jzi = dup2(s.J[5]);
    float2 alr = fma2(Ezr, Jzr, fma2(Ezi, Jzi, fma2(Eyr, Jyr, fma2(Eyi, Jyi, fma2(Exr, Jxr, mul2(Exi, Jxi))))));
    float2 ali = fma2(Ezr, Jzi, fma2(neg2(Ezi), Jzr, fma2(Eyr, Jyi, fma2(neg2(Eyi), Jyr, fma2(Exr, Jxi,
                      mul2(neg2(Exi), Jxr))))));
    const float2 jer = fma2(Jzr, ez, fma2(Jyr, ey, mul2(Jxr, ex))), jei = fma2(Jzi, ez, fma2(Jyi, ey, mul2(Jxi, ex)));
    float2 ber = fma2(jer, ger, mul2(jei, gei)), bei = fma2(jei, ger, mul2(neg2(jer), gei));
    // Z = b x J (- a x M): by the scalar triple product, W.v = -b.(J x v)
    // (+ a.(M x v)) = -v.Z for each of v = R_hat, n_s and n_t.
    float2 zxr = fma2(Hyr, Jzr, fma2(Hyi, Jzi, fma2(neg2(Hzr), Jyr, mul2(neg2(Hzi), Jyi))));
    float2 zxi = fma2(Hyr, Jzi, fma2(neg2(Hyi), Jzr, fma2(neg2(Hzr), Jyi, mul2(Hzi, Jyr))));
    float2 zyr = fma2(Hzr, Jxr, fma2(Hzi, Jxi, fma2(neg2(Hxr), Jzr, mul2(neg2(Hxi), Jzi))));
    float2 zyi = fma2(Hzr, Jxi, fma2(neg2(Hzi), Jxr, fma2(neg2(Hxr), Jzi, mul2(Hxi, Jzr))));
    float2 zzr = fma2(Hxr, Jyr, fma2(Hxi, Jyi, fma2(neg2(Hyr), Jxr, mul2(neg2(Hyi), Jxi))));
    float2 zzi = fma2(Hxr, Jyi, fma2(neg2(Hxi), Jyr, fma2(neg2(Hyr), Jxi, mul2(Hyi, Jxr))));
    float2 mer = dup2(0.f), mei = dup2(0.f);
    if (HAS_M) {
        const float2 Mxr = dup2(s.M[0]), Mxi = dup2(s.M[1]), Myr = dup2(s.M[2]), Myi = dup2(s.M[3]);
        const float2 Mzr = dup2(s.M[4]), Mzi = dup2(s.M[5]);
        alr = fma2(Hzr, Mzr, fma2(Hzi, Mzi, fma2(Hyr, Myr, fma2(Hyi, Myi, fma2(Hxr, Mxr, fma2(Hxi, Mxi, alr))))));
        ali = fma2(Hzr, Mzi, fma2(neg2(Hzi), Mzr, fma2(Hyr, Myi, fma2(neg2(Hyi), Myr, fma2(Hxr, Mxi,
                   fma2(neg2(Hxi), Mxr, ali))))));
        mer = fma2(Mzr, ez, fma2(Myr, ey, mul2(Mxr, ex)));
        mei = fma2(Mzi, ez, fma2(Myi, ey, mul2(Mxi, ex)));
        ber = fma2(mer, ghr, fma2(mei, ghi, ber));
        bei = fma2(mei, ghr, fma2(neg2(mer), ghi, bei));
        // Z -= a x M
        zxr = fma2(neg2(Eyr), Mzr, fma2(neg2(Eyi), Mzi, fma2(Ezr, Myr, fma2(Ezi, Myi, zxr))));
        zxi = fma2(neg2(Eyr), Mzi, fma2(Eyi, Mzr, fma2(Ezr, Myi, fma2(neg2(Ezi), Myr, zxi))));
        zyr = fma2(neg2(Ezr), Mxr, fma2(neg2(Ezi), Mxi, fma2(Exr, Mzr, fma2(Exi, Mzi, zyr))));
        zyi = fma2(neg2(Ezr), Mxi, fma2(Ezi, Mxr, fma2(Exr, Mzi, fma2(neg2(Exi), Mzr, zyi))));
        zzr = fma2(neg2(Exr), Myr, fma2(neg2(Exi), Myi, fma2(Eyr, Mxr, fma2(Eyi, Mxi, zzr))));
        zzi = fma2(neg2(Exr), Myi, fma2(Exi, Myr, fma2(Eyr, Mxi, fma2(neg2(Eyi), Mxr, zzi))));
    }
    const float2 wr = neg2(fma2(ez, zzr, fma2(ey, zyr, mul2(ex, zxr))));
    const float2 wi = neg2(fma2(ez, zzi, fma2(ey, zyi, mul2(ex, zxi))));
    // Re S, S = G (D1 alpha + D2 beta + D3 w), G = (cs, t sn)
    const float2 u2 = mul2(u, u);
    const float2 p1 = fma2(dup2(-3.0f), u2, dup2(1.0f));
    const float2 d1r = T > 0 ? p1 : neg2(p1), d1i = mul2(u, fma2(dup2(-3.0f), u2, dup2(2.0f)));
    const float2 p2 = fma2(dup2(-15.0f), u2, dup2(1.0f));
    const float2 d2r = T > 0 ? neg2(p2) : p2, d2i = mul2(u, fma2(dup2(15.0f), u2, dup2(-6.0f)));
    const float2 d3r = neg2(p1), d3i = mul2(u, dup2(T > 0 ? -3.0f : 3.0f));
    const float2 xr = fma2(d3r, wr, fma2(neg2(d3i), wi, fma2(d2r, ber, fma2(neg2(d2i), bei, fma2(d1r, alr,
                           mul2(neg2(d1i), ali))))));
    const float2 xi = fma2(d3r, wi, fma2(d3i, wr, fma2(d2r, bei, fma2(d2i, ber, fma2(d1r, ali, mul2(d1i, alr))))));
    const float2 gi = T > 0 ? sn : neg2(sn);
    const float2 Sr = fma2(cs, xr, mul2(neg2(gi), xi));

    if (WANT_D) {
        // W.n_s = -n_s.Z; grad(beta).n_s = (a.R_hat)(J.n_s) + (J.R_hat)(a.n_s) (+ M terms)
        const float2 nsx = dup2(s.n[0]), nsy = dup2(s.n[1]), nsz = dup2(s.n[2]);
        const float2 wnr = neg2(fma2(nsz, zzr, fma2(nsy, zyr, mul2(nsx, zxr))));
        const float2 wni = neg2(fma2(nsz, zzi, fma2(nsy, zyi, mul2(nsx, zxi))));
        const float2 anr = fma2(Ezr, nsz, fma2(Eyr, nsy, mul2(Exr, nsx)));
        const float2 ani = neg2(fma2(Ezi, nsz, fma2(Eyi, nsy, mul2(Exi, nsx))));
        float2 gbr = fma2(ger, dup2(s.Jn[0]), fma2(gei, dup2(s.Jn[1]), fma2(jer, anr, mul2(neg2(jei), ani))));
        float2 gbi = fma2(ger, dup2(s.Jn[1]), fma2(neg2(gei), dup2(s.Jn[0]), fma2(jer, ani, mul2(jei, anr))));
        if (HAS_M) {
            const float2 bnr = fma2(Hzr, nsz, fma2(Hyr, nsy, mul2(Hxr, nsx)));
            const float2 bni = neg2(fma2(Hzi, nsz, fma2(Hyi, nsy, mul2(Hxi, nsx))));
            gbr = fma2(ghr, dup2(s.Mn[0]), fma2(ghi, dup2(s.Mn[1]), fma2(mer, bnr, fma2(neg2(mei), bni, gbr))));
            gbi = fma2(ghr, dup2(s.Mn[1]), fma2(neg2(ghi), dup2(s.Mn[0]), fma2(mer, bni, fma2(mei, bnr, gbi))));
        }
        const float2 en = mul2(ndd, rinv);   // R_hat . n_s
        const float2 inner = fma2(en, Sr, fma2(C2r, gbr, fma2(neg2(C2i), gbi, fma2(C3r, wnr,
                                  mul2(neg2(C3i), wni)))));
        acc[12] = fma2(rinv, inner, acc[12]);
    }
    if (WANT_T) {
        // W.n_t = -n_t.Z; grad(beta).n_t = (a.R_hat)(J.n_t) + (J.R_hat)(a.n_t) (+ M terms)
        const float2 ntx = r[18], nty = r[19], ntz = r[20];
        const float2 ent = fma2(ez, ntz, fma2(ey, nty, mul2(ex, ntx)));
        const float2 jnr = fma2(Jzr, ntz, fma2(Jyr, nty, mul2(Jxr, ntx)));
        const float2 jni = fma2(Jzi, ntz, fma2(Jyi, nty, mul2(Jxi, ntx)));
        float2 gbr = fma2(ger, jnr, fma2(gei, jni, fma2(jer, r[21], mul2(neg2(jei), r[22]))));
        float2 gbi = fma2(ger, jni, fma2(neg2(gei), jnr, fma2(jer, r[22], mul2(jei, r[21]))));
        const float2 wnr = neg2(fma2(ntz, zzr, fma2(nty, zyr, mul2(ntx, zxr))));
        const float2 wni = neg2(fma2(ntz, zzi, fma2(nty, zyi, mul2(ntx, zxi))));
        if (HAS_M) {
            const float2 Mxr = dup2(s.M[0]), Mxi = dup2(s.M[1]), Myr = dup2(s.M[2]), Myi = dup2(s.M[3]);
            const float2 Mzr = dup2(s.M[4]), Mzi = dup2(s.M[5]);
            const float2 mnr = fma2(Mzr, ntz, fma2(Myr, nty, mul2(Mxr, ntx)));
            const float2 mni = fma2(Mzi, ntz, fma2(Myi, nty, mul2(Mxi, ntx)));
            gbr = fma2(ghr, mnr, fma2(ghi, mni, fma2(mer, r[23], fma2(neg2(mei), r[24], gbr))));
            gbi = fma2(ghr, mni, fma2(neg2(ghi), mnr, fma2(mer, r[24], fma2(mei, r[23], gbi))));
        }
        const float2 inner = fma2(ent, Sr, fma2(C2r, gbr, fma2(neg2(C2i), gbi, fma2(C3r, wnr,
                                  mul2(neg2(C3i), wni)))));
        vt = mul2(rinv, inner);
    }
}

// Scalar pair of targets against the thread's source (S' in the J.x slot,
// the cotangent g in the gE.x slot): the forward term is S' c with
// c = e^{-t j k R} / R, so
//   Sbar' += conj(c) g,
//   n . grad_d phi = (dphi/dR) (n . d) / R with phi = Re[conj(g) S' c] and
//   dc/dR = c (-t j k - 1 / R)   (k = 2 pi in turns);
// no illumination test (the reference's scalar sum has none).
template <int T, bool WANT_C, bool WANT_D, bool WANT_T>
__device__ __forceinline__ void adj_sc_pair2(float2 *acc, float2 &vt, const float2 *r, const SrcC &s)
{
    const float2 dhx = sub2(r[0], dup2(s.sh[0])), dhy = sub2(r[1], dup2(s.sh[1])), dhz = sub2(r[2], dup2(s.sh[2]));
    const float2 dlx = sub2(r[3], dup2(s.sl[0])), dly = sub2(r[4], dup2(s.sl[1])), dlz = sub2(r[5], dup2(s.sl[2]));
    const float2 two = dup2(2.0f);
    const float2 S0 = fma2(dhz, dhz, fma2(dhy, dhy, mul2(dhx, dhx)));
    const float2 S1 = fma2(dlz, fma2(two, dhz, dlz), fma2(dly, fma2(two, dhy, dly), mul2(dlx, fma2(two, dhx, dlx))));
    const float2 R2 = add2(S0, S1);
    const float2 rinv = make_float2(rsqrt_ftz(R2.x), rsqrt_ftz(R2.y));
    const float2 Rh = mul2(R2, rinv);
    float2 sn, cs, tq;
    phase_sincos2(S0, S1, Rh, rinv, sn, cs, tq);
    // c = G / R, G = e^{-t j 2 pi R} = cos - t j sin
    const float2 rs = flip_parity(rinv, tq);
    const float2 cr = mul2(cs, rs), ci = mul2(T > 0 ? neg2(sn) : sn, rs);
    const float2 gr = r[6], gi = r[7];
    if (WANT_C) {
        acc[0] = fma2(cr, gr, fma2(ci, gi, acc[0]));
        acc[3] = fma2(cr, gi, fma2(neg2(ci), gr, acc[3]));
    }
    if (!WANT_D && !WANT_T) return;
    // X = conj(g) S', Y = X c, dphi/dR = Re[Y (-1/R - t j 2 pi)] = -Y.re / R + t 2 pi Y.im
    const float2 Sr = dup2(s.J[0]), Si = dup2(s.J[1]);
    const float2 xr = fma2(gr, Sr, mul2(gi, Si)), xi = fma2(gr, Si, mul2(neg2(gi), Sr));
    const float2 yr = fma2(xr, cr, mul2(neg2(xi), ci)), yi = fma2(xr, ci, mul2(xi, cr));
    const float2 dphi = fma2(neg2(yr), rinv, mul2(yi, dup2(T > 0 ? 6.28318530717958647f : -6.28318530717958647f)));
    const float2 dx = add2(dhx, dlx), dy = add2(dhy, dly), dz = add2(dhz, dlz);
    const float2 g = mul2(dphi, rinv);
    if (WANT_D) {
        const float2 ndd = fma2(dup2(s.n[2]), dz, fma2(dup2(s.n[1]), dy, mul2(dup2(s.n[0]), dx)));
        acc[12] = fma2(g, ndd, acc[12]);
    }
    if (WANT_T) vt = mul2(g, fma2(r[20], dz, fma2(r[19], dy, mul2(r[18], dx))));
}

// The rare path of a tile in which some pair fell inside the tangent band:
// the thread's source is tested again against the tile's targets, with the
// pair loop's operations, and each pair inside the band is listed for the
// FP64 fixup (an idle source or padding target is only left out). tile:
// cnt target pair records (RT float4 each), the first with target index
// 2 * pfirst.
template <int RT>
__device__ __forceinline__ void adj_band_scan(const float4 *tile, int cnt, long pfirst, const SrcC &s, long si,
                                              long ns, long nt, BandList bl)
{
    if (si >= ns) return;
#pragma unroll 1
    for (int p = 0; p < cnt; ++p) {
        float2 r[6];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float4 v = tile[p * RT + c];
            r[2 * c] = make_float2(v.x, v.y);
            r[2 * c + 1] = make_float2(v.z, v.w);
        }
        const AdjGeo2 g = adj_geo2(r, s);
        const float2 nd = g.ndd, bw = mul2(dup2(kTangentBand), g.Rh);
        const long t0 = 2 * (pfirst + p);
        if (fabsf(nd.x) < bw.x && t0 < nt) band_defer(bl, si, t0);
        if (fabsf(nd.y) < bw.y && t0 + 1 < nt) band_defer(bl, si, t0 + 1);
    }
}

// WANT_C: the currents' gradient. Without it (a fixed feed, the gradient with
// respect to a reflector's shape alone) the 12 current accumulators and the
// projections that only they use, a third of the pair's work, are left out,
// with their partials and epilogue rows; grad_dt alone has no partials. The
// scalar kind keeps its 2 current rows instead of 12. Measured, 40,000 sources
// x 20,000 targets, ms, with all accumulators / now: ds 6.58 / 3.86, dt 6.91 /
// 4.15, ds and dt 7.45 / 4.73; with M 8.12 / 5.61, 8.38 / 5.72, 9.37 / 6.61;
// scalar, all three gradients 1.69 / 1.49.
template <int KIND, int T, bool HAS_M, bool WANT_C, bool WANT_D, bool WANT_T>
__global__ void __launch_bounds__(kThreadsA, WANT_C ? (HAS_M ? kMinBlocksA2M : kMinBlocksA2)
                                                    : (HAS_M ? kMinBlocksA2MN : kMinBlocksA2N))
po_adj_pk_kernel(const float4 *srcpk, long ns, const float4 *trec, long nt, long chunk,
                 double *__restrict__ part, double *__restrict__ gt, int *__restrict__ err, BandList bl)
{
    constexpr int RT = adj2_rec(HAS_M, WANT_T);
    constexpr int NL = 2 * RT;                    // float2 slots read per pair
    extern __shared__ __align__(128) float4 stage[];   // kStages * kPairsA2 * RT, lo, transpose buffer
    __shared__ __align__(8) uint64_t full[kStages];
    pdl_wait();
    float *lo = reinterpret_cast<float *>(stage + (size_t)kStages * kPairsA2 * RT);
    constexpr int NROW = adj_rows(KIND, WANT_C, WANT_D);
    float2 *vbuf = reinterpret_cast<float2 *>(lo + NROW * kThreadsA);   // [kFlush][kThreadsA]

    SrcC s;
    const long si = (long)blockIdx.x * kThreadsA + threadIdx.x;
    {
        float4 q[kRec];
#pragma unroll
        for (int c = 0; c < kRec; ++c) q[c] = srcpk[(size_t)kRec * si + c];   // a record for each thread
        s.sh[0] = q[0].x; s.sh[1] = q[0].y; s.sh[2] = q[0].z;
        s.sl[0] = q[1].x; s.sl[1] = q[1].y; s.sl[2] = q[1].z;
        s.n[0] = q[0].w; s.n[1] = q[1].w; s.n[2] = q[5].x;
        const float jm[12] = {q[2].x, q[2].y, q[2].z, q[2].w, q[3].x, q[3].y, q[3].z, q[3].w, q[4].x, q[4].y, q[4].z,
                              q[4].w};
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            s.J[c] = jm[c];
            s.M[c] = jm[6 + c];
        }
    }
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const float *v = w == 0 ? s.J : s.M;
        float *dn = w == 0 ? s.Jn : s.Mn;
#pragma unroll
        for (int ri = 0; ri < 2; ++ri) dn[ri] = fmaf(v[4 + ri], s.n[2], fmaf(v[2 + ri], s.n[1], v[ri] * s.n[0]));
    }

    float hi[NROW > 0 ? NROW : 1];
#pragma unroll
    for (int a = 0; a < NROW; ++a) {
        hi[a] = 0.f;
        lo[a * kThreadsA + threadIdx.x] = 0.f;
    }

    const long t0 = (long)blockIdx.y * chunk;     // chunk: a multiple of 2 * kPairsA2 targets
    const long t1 = min(nt, t0 + chunk);
    const long p0 = t0 / 2, p1 = (t1 + 1) / 2;
    const int ntiles = p1 > p0 ? (int)((p1 - p0 + kPairsA2 - 1) / kPairsA2) : 0;
    if (threadIdx.x == 0) {
        for (int st = 0; st < kStages; ++st) mbar_init(&full[st], 1);
        mbar_fence_init();
    }
    __syncthreads();
    auto issue = [&](int it) {
        const long first = p0 + (long)it * kPairsA2;
        const long cnt = min((long)kPairsA2, p1 - first);
        const uint32_t bytes = (uint32_t)(cnt * RT * sizeof(float4));
        uint64_t *bar = &full[it % kStages];
        fence_proxy_async();
        mbar_expect_tx(bar, bytes);
        tma_load_1d(stage + (size_t)(it % kStages) * kPairsA2 * RT, trec + first * RT, bytes, bar);
    };
    if (threadIdx.x == 0)
        for (int it = 0; it < ntiles && it < kStages; ++it) issue(it);

    for (int it = 0; it < ntiles; ++it) {
        const bool ok = mbar_wait_bounded(&full[it % kStages], (uint32_t)((it / kStages) & 1));
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicExch(err, kErrWaitTimeout);
                for (int st = 0; st < kStages; ++st) (void)mbar_wait_bounded(&full[st], 0);
            }
            return;
        }
        const float4 *tile = stage + (size_t)(it % kStages) * kPairsA2 * RT;
        const long pfirst = p0 + (long)it * kPairsA2;
        const int cnt = (int)min((long)kPairsA2, p1 - pfirst);
        float2 acc[kAccAdj];
#pragma unroll
        for (int a = 0; a < kAccAdj; ++a) acc[a] = make_float2(0.f, 0.f);
        bool band = false;   // a pair of this tile fell inside the tangent band
        for (int fb = 0; fb < cnt; fb += kFlush) {
            const int fend = min(cnt, fb + kFlush);
#pragma unroll kUnrollA
            for (int p = fb; p < fend; ++p) {
                float2 rec[NL];
#pragma unroll
                for (int c = 0; c < RT; ++c) {
                    const float4 v = tile[p * RT + c];
                    rec[2 * c] = make_float2(v.x, v.y);
                    rec[2 * c + 1] = make_float2(v.z, v.w);
                }
                float2 vt = make_float2(0.f, 0.f);
                if (KIND == kKindNF)
                    adj_nf_pair2<T, HAS_M, WANT_C, WANT_D, WANT_T>(acc, vt, rec, s, band);
                else adj_sc_pair2<T, WANT_C, WANT_D, WANT_T>(acc, vt, rec, s);
                if (WANT_T) vbuf[(p - fb) * kThreadsA + threadIdx.x] = vt;
            }
            if (WANT_T) {
                // Sum the CTA's sources for each target pair of this flush: thread
                // (pl, k) adds kThreadsA / kSegs sources of pair pl (rotated reads:
                // the 8 threads of a shared-memory phase hit distinct banks), then
                // the kSegs segments combine by shuffles.
                __syncthreads();
                constexpr int kPer = kThreadsA / kSegs / 2;   // float4 (two sources each) per thread
                const int pl = threadIdx.x / kSegs, k = threadIdx.x % kSegs;
                const int rot = kSegs == 8 ? k : 4 * (pl & 1) + k;
                float2 sum = make_float2(0.f, 0.f);
                if (pl < fend - fb) {
                    const float4 *row = reinterpret_cast<const float4 *>(vbuf + pl * kThreadsA);
#pragma unroll
                    for (int j = 0; j < kPer; ++j) {
                        const float4 v = row[kPer * k + ((j + rot) & (kPer - 1))];
                        sum = add2(sum, add2(make_float2(v.x, v.y), make_float2(v.z, v.w)));
                    }
                }
#pragma unroll
                for (int m = 1; m < kSegs; m <<= 1) {
                    sum.x += __shfl_xor_sync(0xffffffffu, sum.x, m);
                    sum.y += __shfl_xor_sync(0xffffffffu, sum.y, m);
                }
                if (k == 0 && pl < fend - fb) {
                    const long tg = 2 * (pfirst + fb + pl);
                    if (tg < nt) atomicAdd(&gt[tg], (double)sum.x);
                    if (tg + 1 < nt) atomicAdd(&gt[tg + 1], (double)sum.y);
                }
                __syncthreads();
            }
        }
#pragma unroll
        for (int a = 0; a < kAccAdj; ++a) {
            const int r = adj_row(KIND, WANT_C, WANT_D, a);
            if (r < 0) continue;
            float sm, e;
            two_sum(hi[r], __fadd_rn(acc[a].x, acc[a].y), sm, e);
            hi[r] = sm;
            float &l = lo[r * kThreadsA + threadIdx.x];
            l = __fadd_rn(l, e);
        }
        if (KIND != kKindScalar && band) adj_band_scan<RT>(tile, cnt, pfirst, s, si, ns, nt, bl);
        __syncthreads();
        if (threadIdx.x == 0 && it + kStages < ntiles) issue(it + kStages);
    }
    pdl_trigger();
    if (si >= ns) return;
#pragma unroll
    for (int a = 0; a < NROW; ++a)
        part[((long)blockIdx.y * NROW + a) * ns + si] = (double)hi[a] + (double)lo[a * kThreadsA + threadIdx.x];
}

int adj_pk_smem_bytes(int kind, bool has_m, bool want_c, bool want_d, bool want_t)
{
    return kStages * kPairsA2 * adj2_rec(has_m, want_t) * 16 + adj_rows(kind, want_c, want_d) * kThreadsA * 4 +
           (want_t ? kFlush * kThreadsA * 8 : 0);
}

int adj_pk_pairs_per_tile() { return kPairsA2; }

int adj_pk_rec4(bool has_m, bool want_t) { return adj2_rec(has_m, want_t); }

template <int KIND, int T, bool HAS_M, bool WANT_C>
static void *adj_pk_sel(bool want_d, bool want_t)
{
    if (want_d) return want_t ? reinterpret_cast<void *>(&po_adj_pk_kernel<KIND, T, HAS_M, WANT_C, true, true>)
                              : reinterpret_cast<void *>(&po_adj_pk_kernel<KIND, T, HAS_M, WANT_C, true, false>);
    // at least one gradient is wanted
    if (want_t || !WANT_C) return reinterpret_cast<void *>(&po_adj_pk_kernel<KIND, T, HAS_M, WANT_C, false, true>);
    return reinterpret_cast<void *>(&po_adj_pk_kernel<KIND, T, HAS_M, true, false, false>);
}

template <int T>
static void *adj_pk_kind(int kind, bool has_m, bool want_c, bool want_d, bool want_t)
{
    if (kind == kKindScalar) return want_c ? adj_pk_sel<kKindScalar, T, false, true>(want_d, want_t)
                                           : adj_pk_sel<kKindScalar, T, false, false>(want_d, want_t);
    if (has_m) return want_c ? adj_pk_sel<kKindNF, T, true, true>(want_d, want_t)
                             : adj_pk_sel<kKindNF, T, true, false>(want_d, want_t);
    return want_c ? adj_pk_sel<kKindNF, T, false, true>(want_d, want_t)
                  : adj_pk_sel<kKindNF, T, false, false>(want_d, want_t);
}

void *adj_pk_kernel(int kind, int t_sign, bool has_m, bool want_c, bool want_d, bool want_t)
{
    return t_sign < 0 ? adj_pk_kind<-1>(kind, has_m, want_c, want_d, want_t)
                      : adj_pk_kind<1>(kind, has_m, want_c, want_d, want_t);
}

}  // namespace po
