// po_fp64.cu -- the plain FP64 sums: forward and adjoint of every kind, and
// the FP64 decision of the mixed path's near-tangent pairs.
//
// What bounds these kernels is the FP64 pipe (2 operations per clock and SM
// on GB300, 1/64 of the FP32 rate), so the count of FP64 instructions per
// pair is what is kept down, and every SM gets work:
//   * R and 1/R from one approximate rsqrt and a third-order (Householder)
//     correction, 9 operations, where the rounded square root and division cost
//     about 25; the correctly rounded pair is formed only for
//     a pair whose n . d is within 1e-12 R of zero, where the reference's
//     illumination decision needs its rounding;
//   * the phase k R, rounded as the reference rounds it (R^2 summed without
//     FMA, then R, then the product), reduced to quarter turns with 2/pi held
//     as hi + lo, sin and cos of the residual by near-minimax polynomials,
//     the quadrant and the direction of time on the integer pipe;
//   * kernels without magnetic terms where M == 0, unit-vector forms of the
//     coefficients, the adjoint's source and target sides fused (one
//     geometry, phase and coefficient set per pair, W.v through one vector
//     Z = b x J - a x M);
//   * a grid over (owning blocks, streamed chunks), so that a few thousand
//     points still fill the GPU; the epilogues add the chunks in order.
// Measured (one GB300): 101 x 99 sources -> 41 x 43 targets, EH, M = 0 (1.76e7
// pairs), forward and every gradient 12.6 ms (229 ms with one block per 128
// points, magnetic terms always and separate adjoint sides); 201 x 201 ->
// 101 x 101, JMEH with M (4.1e8 pairs), forward 115 ms (295 ms), about 165
// FP64 instructions a pair at 93 % of 2 per clock and SM.
#include <cuda_runtime.h>

#include <cstdint>

#include "po_device.cuh"
#include "po_kernels.cuh"

namespace po {

namespace {

// ------------------------------------------------------------ FP64 helpers

// a with its sign bit xor-ed by m (0 or 0x80000000): integer pipe.
__device__ __forceinline__ double flip64(double a, unsigned m)
{
    return __hiloint2double(__double2hiint(a) ^ (int)m, __double2loint(a));
}

// 1/sqrt(x) to about an ulp and sqrt(x) to half an ulp, x normal (R from
// 1.5e-154 to 1.3e154; NaN outside): y ~ 2^-22 from the
// hardware estimate, e = 1 - x y^2, y (1 + e/2 + 3 e^2/8), then one residual
// step for the root.
__device__ __forceinline__ void rsqrt64(double x, double &rinv, double &root)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    rinv = fma(fma(e, 0.375, 0.5), y * e, y);
    const double h = x * rinv;
    root = fma(fma(-h, h, x), 0.5 * rinv, h);
}

// cos and sin past sincos64's range: the general reduction.
__device__ __noinline__ double2 sincos64_far(double x)
{
    double s, c;
    sincos(x, &s, &c);
    return make_double2(c, s);
}

// cos and sin of the angle x. Past 2^51, infinite or NaN: the call above (one
// integer comparison a pair, whose cost does not show). Up to there: X = x 2/pi
// quarter turns, n = rint(X) from one fma against 1.5 2^52, y = X - n exact but
// for 2/pi's 2^-106; sin and cos of y pi/2, |y| <= 1/2, by polynomials in y^2
// (minimax fits by Remez exchange, errors 4e-18 and 4e-20 before rounding),
// placed by n mod 4.
__device__ __forceinline__ void sincos64(double x, double &cs, double &sn)
{
    if ((__double2hiint(x) & 0x7fffffff) >= 0x43200000) {
        const double2 f = sincos64_far(x);
        cs = f.x;
        sn = f.y;
        return;
    }
    const double magic = 6755399441055744.0;
    const double h = 0.6366197723675814, l = -3.935735335036497e-17;   // 2/pi
    const double t = fma(x, h, magic);
    const double q = t - magic;
    const double y = fma(x, l, fma(x, h, -q));
    const double z = y * y;
    double a = fma(z, 5.633604231088863e-08, -3.5986409469628637e-06);
    double c = fma(z, -6.3217635712021026e-09, 4.710614622760973e-07);
    a = fma(z, a, 0.00016044115008380884);
    c = fma(z, c, -2.5202036959231476e-05);
    a = fma(z, a, -0.004681754132257977);
    c = fma(z, c, 0.0009192602742201073);
    a = fma(z, a, 0.07969262624603828);
    c = fma(z, c, -0.020863480763315068);
    a = fma(z, a, -0.6459640975062442);
    c = fma(z, c, 0.2536695079010469);
    a = fma(z, a, 1.5707963267948966);
    c = fma(z, c, -1.2337005501361697);
    a *= y;
    c = fma(z, c, 1.0);
    const unsigned n = (unsigned)__double2loint(t);
    const bool swap = n & 1u;
    sn = flip64(swap ? c : a, (n << 30) & 0x80000000u);
    cs = flip64(swap ? a : c, ((n + 1u) << 30) & 0x80000000u);
}

// A pair of a near-field or scalar sum: d = t - s, R and 1/R.
struct Geo64 {
    double dx, dy, dz, R, rinv;
};

__device__ __forceinline__ Geo64 geo64(const double *t, const double *s)
{
    Geo64 g;
    g.dx = t[0] - s[0];
    g.dy = t[1] - s[1];
    g.dz = t[2] - s[2];
    rsqrt64(__dadd_rn(__dadd_rn(__dmul_rn(g.dx, g.dx), __dmul_rn(g.dy, g.dy)), __dmul_rn(g.dz, g.dz)), g.rinv, g.R);
    return g;
}

// The reference's illumination decision (lit_fp64) of a pair with n . d = nd:
// clear of zero by far more than any rounding, or decided with its rounding.
// Almost every pair is clear by its exponents alone (|nd| >= 2^(en - 1023) and
// R < 2^(er - 1022), so en >= er - 38 gives |nd| > 1e-12 R), which takes no FP64
// operation where the comparisons take three. For unit normals; n . d is off by
// some 1e-15 |n| R at most on either side, so lengths up to a thousand do as well.
__device__ __forceinline__ bool lit64(const double *n, const Geo64 &g, double nd)
{
    const int h = __double2hiint(nd), en = (h >> 20) & 0x7ff, er = (__double2hiint(g.R) >> 20) & 0x7ff;
    if (en > 0 && en < 0x7ff && er < 0x7ff && en + 38 >= er) return h >= 0;
    const double thr = 1e-12 * g.R;
    if (nd > thr) return true;
    if (nd < -thr) return false;
    const double R = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(g.dx, g.dx), __dmul_rn(g.dy, g.dy)),
                                          __dmul_rn(g.dz, g.dz)));
    return lit_fp64(n, g.dx, g.dy, g.dz, __ddiv_rn(1.0, R));
}

// The same for a far-field direction r (the reference: n . r < 0 unlit, the
// products summed left to right, no FMA).
__device__ __forceinline__ bool lit64_ff(const double *n, const double *r, double nd)
{
    // 2^-39 > 1e-12; not NaN or infinite
    const int h = __double2hiint(nd), en = (h >> 20) & 0x7ff;
    if (en >= 1023 - 39 && en < 0x7ff) return h >= 0;
    if (nd > 1e-12) return true;
    if (nd < -1e-12) return false;
    return !(__dadd_rn(__dadd_rn(__dmul_rn(n[0], r[0]), __dmul_rn(n[1], r[1])), __dmul_rn(n[2], r[2])) < 0.0);
}

// Near-field coefficients in unit-vector form, as in the mixed kernels:
// c1 = Gu (t u + j(u^2 - 1)), C2 = -3 c1 - 2 j Gu, C3 = Gu (-u + j t), with
// u = 1 / kR, G = cos kR + j t sin kR.
struct Coef64 {
    double u, cs, ts;   // u; G = (cs, ts)
    double c1r, c1i, c2r, c2i, c3r, c3i;
};

__device__ __forceinline__ Coef64 coef64(const Geo64 &g, const Wave64 &w)
{
    Coef64 c;
    double sn;
    sincos64(w.k * g.R, c.cs, sn);
    c.ts = flip64(sn, w.neg);
    c.u = g.rinv * w.inv_k;
    const double gr = c.cs * c.u, gi = c.ts * c.u;
    const double tu = flip64(c.u, w.neg), b = fma(c.u, c.u, -1.0);
    c.c1r = fma(gr, tu, -(gi * b));
    c.c1i = fma(gr, b, gi * tu);
    c.c2r = fma(-3.0, c.c1r, gi + gi);
    c.c2i = fma(-3.0, c.c1i, -(gr + gr));
    c.c3r = fma(-gr, c.u, -flip64(gi, w.neg));
    c.c3i = fma(-gi, c.u, flip64(gr, w.neg));
    return c;
}

// (re, im) of complex a . real e
__device__ __forceinline__ void dot_re(const double *a, const double *e, double &re, double &im)
{
    re = fma(a[4], e[2], fma(a[2], e[1], a[0] * e[0]));
    im = fma(a[5], e[2], fma(a[3], e[1], a[1] * e[0]));
}

// F += c1 v + C2 (v.e) e and G -= (C3 v) x e (sign -1) or G += (sign +1): the
// electric and magnetic halves of the dyadic kernel for one vector v ((re, im)
// x y z). fr/fi, gr/gi: re and im rows of the two fields.
template <int SIGN>
__device__ __forceinline__ void dyad64(const Coef64 &c, const double *v, const double *e, double *fr, double *fi,
                                       double *gr, double *gi)
{
    double der, dei;
    dot_re(v, e, der, dei);
    const double Pr = fma(c.c2r, der, -(c.c2i * dei)), Pi = fma(c.c2r, dei, c.c2i * der);
    double kr[3], ki[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        fr[a] = fma(Pr, e[a], fma(-c.c1i, v[2 * a + 1], fma(c.c1r, v[2 * a], fr[a])));
        fi[a] = fma(Pi, e[a], fma(c.c1i, v[2 * a], fma(c.c1r, v[2 * a + 1], fi[a])));
        kr[a] = fma(c.c3r, v[2 * a], -(c.c3i * v[2 * a + 1]));
        ki[a] = fma(c.c3r, v[2 * a + 1], c.c3i * v[2 * a]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, d = (a + 2) % 3;
        // (k x e)_a = k_b e_d - k_d e_b
        if (SIGN > 0) {
            gr[a] = fma(kr[b], e[d], fma(-kr[d], e[b], gr[a]));
            gi[a] = fma(ki[b], e[d], fma(-ki[d], e[b], gi[a]));
        } else {
            gr[a] = fma(kr[d], e[b], fma(-kr[b], e[d], gr[a]));
            gi[a] = fma(ki[d], e[b], fma(-ki[b], e[d], gi[a]));
        }
    }
}

// ------------------------------------------------------------------ forward

// One pair of the FP64 forward sum, added into acc (kAcc accumulators E.re,
// E.im, H.re, H.im, far field S_J and S_M likewise; 2 for the scalar kind):
// p the target point (mm) or direction, r the source's record.
template <int KIND, bool HAS_M>
__device__ __forceinline__ void fwd_pair64(const double *p, const double *r, const Wave64 &w, double *acc)
{
    if (KIND == kKindFF) {
        const double nd = fma(r[5], p[2], fma(r[4], p[1], r[3] * p[0]));
        if (!lit64_ff(r + 3, p, nd)) return;
        double cs, sn;
        sincos64(w.k * fma(r[2], p[2], fma(r[1], p[1], r[0] * p[0])), cs, sn);
        const double gs = flip64(sn, w.neg ^ 0x80000000u);   // G = e^{-t j k r.s}
#pragma unroll
        for (int c = 0; c < (HAS_M ? 6 : 3); ++c) {
            const double cr = r[6 + 2 * c], ci = r[7 + 2 * c];
            const int slot = c < 3 ? c : 6 + (c - 3);
            acc[slot] = fma(-gs, ci, fma(cs, cr, acc[slot]));
            acc[slot + 3] = fma(gs, cr, fma(cs, ci, acc[slot + 3]));
        }
        return;
    }
    const Geo64 g = geo64(p, r);
    if (KIND == kKindScalar) {
        double cs, sn;
        sincos64(w.k * g.R, cs, sn);
        const double gr = cs * g.rinv, gi = flip64(sn, w.neg ^ 0x80000000u) * g.rinv;
        acc[0] = fma(-gi, r[7], fma(gr, r[6], acc[0]));
        acc[1] = fma(gi, r[6], fma(gr, r[7], acc[1]));
        return;
    }
    const double nd = fma(r[5], g.dz, fma(r[4], g.dy, r[3] * g.dx));
    if (!lit64(r + 3, g, nd)) return;
    const Coef64 c = coef64(g, w);
    const double e[3] = {g.dx * g.rinv, g.dy * g.rinv, g.dz * g.rinv};
    dyad64<-1>(c, r + 6, e, acc, acc + 3, acc + 6, acc + 9);
    if (HAS_M) dyad64<1>(c, r + 12, e, acc + 6, acc + 9, acc, acc + 3);
}

}  // namespace

// Grid = (target blocks, source chunks of `chunk` sources). One target per
// thread; the chunk's records pass through shared memory.
template <int KIND, bool HAS_M>
__global__ void __launch_bounds__(kThreadsD)
po_fp64_kernel(const double *__restrict__ src, long ns, long chunk, const double *__restrict__ tgt7, long nt,
               Wave64 w, double *__restrict__ part)
{
    constexpr int REC = fp64_rec(KIND, HAS_M), NACC = KIND == kKindScalar ? 2 : kAcc;
    __shared__ double tile[kTileD * REC];
    const long ti = (long)blockIdx.x * blockDim.x + threadIdx.x;
    double p[3] = {0, 0, 0};
    if (ti < nt) {
        if constexpr (KIND == kKindFF) ff_direction_d(tgt7, nt, ti, p);
        else
            for (int c = 0; c < 3; ++c) p[c] = tgt7[c * nt + ti];
    }
    double acc[NACC];
#pragma unroll
    for (int a = 0; a < NACC; ++a) acc[a] = 0.0;
    const long s0 = (long)blockIdx.y * chunk, s1 = min(ns, s0 + chunk);
    for (long base = s0; base < s1; base += kTileD) {
        const int cnt = (int)min((long)kTileD, s1 - base);
        __syncthreads();
        for (int q = threadIdx.x; q < cnt * REC; q += blockDim.x) tile[q] = src[base * REC + q];
        __syncthreads();
        if (ti >= nt) continue;
#pragma unroll 1
        for (int s = 0; s < cnt; ++s) fwd_pair64<KIND, HAS_M>(p, tile + s * REC, w, acc);
    }
    if (ti >= nt) return;
#pragma unroll
    for (int a = 0; a < NACC; ++a) part[((long)blockIdx.y * NACC + a) * nt + ti] = acc[a];
}

// Source records of the FP64 kernels (src_record_d), rec doubles each.
__global__ void po_pack_src_d_kernel(long ns, const double *__restrict__ src7, const double *__restrict__ cur,
                                     int gmode, int ncx, int ncy, double fac_re, double fac_im, int scalar, int rec,
                                     double *__restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    src_record_d(i, ns, src7, cur, gmode, ncx, ncy, fac_re, fac_im, scalar, rec, out + (size_t)rec * i);
}

// The pairs a mixed kernel left out as inside the tangent band: each is
// decided by the reference's FP64 rounding and, if lit, its FP64 term is
// added into the first source chunk's partial sums (the epilogue adds the
// chunks afterwards). The order of those additions varies between runs for
// a target with several such pairs (last-bit differences there only).
template <int KIND, bool HAS_M>
__global__ void __launch_bounds__(256)
po_band_fixup_kernel(BandList bl, long ns, const double *__restrict__ src7, const double *__restrict__ cur,
                     int gmode, int ncx, int ncy, double fac_re, double fac_im, long nt,
                     const double *__restrict__ tgt7, Wave64 w, double *__restrict__ part, int *__restrict__ err)
{
    constexpr int REC = fp64_rec(KIND, HAS_M), NACC = KIND == kKindFF && !HAS_M ? 6 : kAcc;
    pdl_wait();
    const unsigned total = *bl.count;
    if (blockIdx.x == 0 && threadIdx.x == 0 && total > bl.cap) atomicExch(err, kErrBandOverflow);
    const unsigned n = min(total, bl.cap);
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int2 pr = bl.pairs[i];
        double rec[REC], p[3], acc[kAcc];
        src_record_d(pr.x, ns, src7, cur, gmode, ncx, ncy, fac_re, fac_im, 0, REC, rec);
        if constexpr (KIND == kKindFF) ff_direction_d(tgt7, nt, pr.y, p);
        else
            for (int c = 0; c < 3; ++c) p[c] = tgt7[c * nt + pr.y];
        for (int a = 0; a < kAcc; ++a) acc[a] = 0.0;
        fwd_pair64<KIND, HAS_M>(p, rec, w, acc);
        for (int a = 0; a < NACC; ++a)
            if (acc[a] != 0.0) atomicAdd(&part[(long)a * nt + pr.y], acc[a]);
    }
    pdl_trigger();
}

// ------------------------------------------------------------------ adjoint

namespace {

// Target records of the FP64 adjoint (adj64_rec doubles): near field point
// xyz, normal xyz, gE (re, im) x y z, gH likewise, a.n and b.n (a = conj gE,
// b = conj gH; (re, im) each); far field direction xyz, three unused, gS_J,
// gS_M; scalar point, normal, g (re, im).
template <int KIND>
__device__ __forceinline__ void adj_record64(long i, long nt, const double *tgt7, const double *gam, double *o)
{
    if constexpr (KIND == kKindFF) {
        ff_direction_d(tgt7, nt, i, o);
        o[3] = o[4] = o[5] = 0.0;
    } else {
        for (int c = 0; c < 6; ++c) o[c] = tgt7[c * nt + i];
    }
    if constexpr (KIND == kKindScalar) {
        o[6] = gam[i];
        o[7] = gam[3 * nt + i];
    } else {
        for (int g = 0; g < 2; ++g)
            for (int c = 0; c < 3; ++c) {
                o[6 + 6 * g + 2 * c] = gam[(6 * g + c) * nt + i];
                o[7 + 6 * g + 2 * c] = gam[(6 * g + 3 + c) * nt + i];
            }
    }
    if (KIND == kKindNF)
        for (int g = 0; g < 2; ++g) {
            const double *v = o + 6 + 6 * g, *n = o + 3;
            o[18 + 2 * g] = v[0] * n[0] + v[2] * n[1] + v[4] * n[2];
            o[19 + 2 * g] = -(v[1] * n[0] + v[3] * n[1] + v[5] * n[2]);
        }
}

// (re, im) of conj(g) . v, both complex ((re, im) x y z)
__device__ __forceinline__ void cdot64(const double *g, const double *v, double &re, double &im)
{
    re = fma(g[4], v[4], fma(g[5], v[5], fma(g[2], v[2], fma(g[3], v[3], fma(g[0], v[0], g[1] * v[1])))));
    im = fma(g[4], v[5], fma(-g[5], v[4], fma(g[2], v[3], fma(-g[3], v[2], fma(g[0], v[1], -(g[1] * v[0]))))));
}

// z += SIGN conj(g) x v, complex vectors
template <int SIGN>
__device__ __forceinline__ void ccross64(const double *g, const double *v, double *zr, double *zi)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, d = (a + 2) % 3;
        const double *p = SIGN > 0 ? g + 2 * b : g + 2 * d, *q = SIGN > 0 ? g + 2 * d : g + 2 * b;
        const double *vp = SIGN > 0 ? v + 2 * d : v + 2 * b, *vq = SIGN > 0 ? v + 2 * b : v + 2 * d;
        // conj(p) vp - conj(q) vq
        zr[a] = fma(p[0], vp[0], fma(p[1], vp[1], fma(-q[0], vq[0], fma(-q[1], vq[1], zr[a]))));
        zi[a] = fma(p[0], vp[1], fma(-p[1], vp[0], fma(-q[0], vq[1], fma(q[1], vq[0], zi[a]))));
    }
}

// Jbar' += conj(c1) g + conj(C2)(g.e) e + SIGN conj(C3)(h x e); ge: g . e
template <int SIGN>
__device__ __forceinline__ void vjp64(const Coef64 &c, const double *g, double ger, double gei, const double *h,
                                      const double *e, double *ar, double *ai)
{
    const double Pr = fma(c.c2r, ger, c.c2i * gei), Pi = fma(c.c2r, gei, -(c.c2i * ger));
    double kr[3], ki[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        ar[a] = fma(Pr, e[a], fma(c.c1i, g[2 * a + 1], fma(c.c1r, g[2 * a], ar[a])));
        ai[a] = fma(Pi, e[a], fma(-c.c1i, g[2 * a], fma(c.c1r, g[2 * a + 1], ai[a])));
        kr[a] = fma(c.c3r, h[2 * a], c.c3i * h[2 * a + 1]);
        ki[a] = fma(c.c3r, h[2 * a + 1], -(c.c3i * h[2 * a]));
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, d = (a + 2) % 3;
        if (SIGN > 0) {
            ar[a] = fma(kr[b], e[d], fma(-kr[d], e[b], ar[a]));
            ai[a] = fma(ki[b], e[d], fma(-ki[d], e[b], ai[a]));
        } else {
            ar[a] = fma(kr[d], e[b], fma(-kr[b], e[d], ar[a]));
            ai[a] = fma(ki[d], e[b], fma(-ki[b], e[d], ai[a]));
        }
    }
}

// v . z of a real v and a complex z in separate re, im
__device__ __forceinline__ double dot64(const double *v, const double *z)
{
    return fma(v[2], z[2], fma(v[1], z[1], v[0] * z[0]));
}

// One pair of the FP64 adjoint: the source's record s (kRecD or, without
// magnetic terms, 12 doubles) against the target record r. acc: the 12
// current accumulators (WANT_C) and n_s . grad_d phi (WANT_D); returns n_t . grad_d
// phi (WANT_T). Unlit pairs add nothing. The formulas are those of the mixed
// kernels (po_adjoint_pk.cu).
template <int KIND, bool HAS_M, bool WANT_C, bool WANT_D, bool WANT_T>
__device__ __forceinline__ double adj_pair64(const double *s, const double *r, const Wave64 &w, double *acc)
{
    if (KIND == kKindFF) {
        const double nd = fma(s[5], r[2], fma(s[4], r[1], s[3] * r[0]));
        if (!lit64_ff(s + 3, r, nd)) return 0.0;
        double cs, sn;
        sincos64(w.k * fma(s[2], r[2], fma(s[1], r[1], s[0] * r[0])), cs, sn);
        const double gs = flip64(sn, w.neg ^ 0x80000000u);   // G = (cs, gs)
#pragma unroll
        for (int c = 0; c < (WANT_C ? 6 : 0); ++c) {
            const double gr = r[6 + 2 * c], gi = r[7 + 2 * c];
            const int slot = c < 3 ? c : 6 + (c - 3);
            acc[slot] = fma(gs, gi, fma(cs, gr, acc[slot]));
            acc[slot + 3] = fma(-gs, gr, fma(cs, gi, acc[slot + 3]));
        }
        if (WANT_D) {
            double xr, xi;
            cdot64(r + 6, s + 6, xr, xi);
            if (HAS_M) {
                double yr, yi;
                cdot64(r + 12, s + 12, yr, yi);
                xr += yr;
                xi += yi;
            }
            // Re[-t j k G X] = t k Im(G X)
            acc[12] = fma(flip64(w.k, w.neg) * nd, fma(cs, xi, gs * xr), acc[12]);
        }
        return 0.0;
    }
    const Geo64 g = geo64(r, s);
    if (KIND == kKindScalar) {
        double cs, sn;
        sincos64(w.k * g.R, cs, sn);
        const double cr = cs * g.rinv, ci = flip64(sn, w.neg ^ 0x80000000u) * g.rinv;
        if (WANT_C) {
            acc[0] = fma(cr, r[6], fma(ci, r[7], acc[0]));
            acc[3] = fma(cr, r[7], fma(-ci, r[6], acc[3]));
        }
        if (!WANT_D && !WANT_T) return 0.0;
        const double xr = fma(r[6], s[6], r[7] * s[7]), xi = fma(r[6], s[7], -(r[7] * s[6]));
        const double yr = fma(xr, cr, -(xi * ci)), yi = fma(xr, ci, xi * cr);
        const double dphi = fma(-yr, g.rinv, flip64(w.k, w.neg) * yi) * g.rinv;
        const double d[3] = {g.dx, g.dy, g.dz};
        if (WANT_D) acc[12] = fma(dphi, dot64(s + 3, d), acc[12]);
        return WANT_T ? dphi * dot64(r + 3, d) : 0.0;
    }
    const double ndd = fma(s[5], g.dz, fma(s[4], g.dy, s[3] * g.dx));
    if (!lit64(s + 3, g, ndd)) return 0.0;
    const Coef64 c = coef64(g, w);
    const double e[3] = {g.dx * g.rinv, g.dy * g.rinv, g.dz * g.rinv};
    const double *E = r + 6, *H = r + 12;
    double ger, gei, ghr, ghi;
    dot_re(E, e, ger, gei);
    dot_re(H, e, ghr, ghi);
    if (WANT_C) {
        vjp64<1>(c, E, ger, gei, H, e, acc, acc + 3);
        vjp64<-1>(c, H, ghr, ghi, E, e, acc + 6, acc + 9);
    }
    if (!WANT_D && !WANT_T) return 0.0;

    // alpha = a.J + b.M, beta = (J.e)(a.e) + (M.e)(b.e), Z = b x J - a x M, W.v = -v.Z
    const double *J = s + 6, *M = s + 12;
    double alr, ali, jer, jei, mer = 0.0, mei = 0.0;
    cdot64(E, J, alr, ali);
    dot_re(J, e, jer, jei);
    double ber = fma(jer, ger, jei * gei), bei = fma(jei, ger, -(jer * gei));
    double zr[3] = {0.0, 0.0, 0.0}, zi[3] = {0.0, 0.0, 0.0};
    ccross64<1>(H, J, zr, zi);
    if (HAS_M) {
        double br, bi;
        cdot64(H, M, br, bi);
        alr += br;
        ali += bi;
        dot_re(M, e, mer, mei);
        ber = fma(mer, ghr, fma(mei, ghi, ber));
        bei = fma(mei, ghr, fma(-mer, ghi, bei));
        ccross64<-1>(E, M, zr, zi);
    }
    const double wr = -dot64(e, zr), wi = -dot64(e, zi);
    // Re S, S = G (D1 alpha + D2 beta + D3 w)
    const double u = c.u, u2 = u * u;
    const double p1 = fma(-3.0, u2, 1.0), p2 = fma(-15.0, u2, 1.0);
    const double d1r = flip64(p1, w.neg), d1i = u * fma(-3.0, u2, 2.0);
    const double d2r = flip64(p2, w.neg ^ 0x80000000u), d2i = u * fma(15.0, u2, -6.0);
    const double d3i = flip64(u * -3.0, w.neg);
    const double xr = fma(-p1, wr, fma(-d3i, wi, fma(d2r, ber, fma(-d2i, bei, fma(d1r, alr, -(d1i * ali))))));
    const double xi = fma(-p1, wi, fma(d3i, wr, fma(d2r, bei, fma(d2i, ber, fma(d1r, ali, d1i * alr)))));
    const double Sr = fma(c.cs, xr, -(c.ts * xi));

    // (1/R) Re[(e.n) S + C2 (grad(beta).n) + C3 (W.n)] for a normal n
    auto project = [&](double en, double gbr, double gbi, double wnr, double wni) {
        return g.rinv * fma(en, Sr, fma(c.c2r, gbr, fma(-c.c2i, gbi, fma(c.c3r, wnr, -(c.c3i * wni)))));
    };
    if (WANT_D) {
        const double *n = s + 3;
        double jnr, jni, anr, ani;
        dot_re(J, n, jnr, jni);   // J.n_s
        dot_re(E, n, anr, ani);   // a.n_s = (anr, -ani)
        double gbr = fma(ger, jnr, fma(gei, jni, fma(jer, anr, jei * ani)));
        double gbi = fma(ger, jni, fma(-gei, jnr, fma(-jer, ani, jei * anr)));
        if (HAS_M) {
            double mnr, mni, bnr, bni;
            dot_re(M, n, mnr, mni);
            dot_re(H, n, bnr, bni);
            gbr = fma(ghr, mnr, fma(ghi, mni, fma(mer, bnr, fma(mei, bni, gbr))));
            gbi = fma(ghr, mni, fma(-ghi, mnr, fma(-mer, bni, fma(mei, bnr, gbi))));
        }
        acc[12] += project(ndd * g.rinv, gbr, gbi, -dot64(n, zr), -dot64(n, zi));
    }
    if (!WANT_T) return 0.0;
    const double *n = r + 3;
    double jnr, jni;
    dot_re(J, n, jnr, jni);   // J.n_t
    double gbr = fma(ger, jnr, fma(gei, jni, fma(jer, r[18], -(jei * r[19]))));
    double gbi = fma(ger, jni, fma(-gei, jnr, fma(jer, r[19], jei * r[18])));
    if (HAS_M) {
        double mnr, mni;
        dot_re(M, n, mnr, mni);
        gbr = fma(ghr, mnr, fma(ghi, mni, fma(mer, r[20], fma(-mei, r[21], gbr))));
        gbi = fma(ghr, mni, fma(-ghi, mnr, fma(mer, r[21], fma(mei, r[20], gbi))));
    }
    return project(dot64(n, e), gbr, gbi, -dot64(n, zr), -dot64(n, zi));
}

constexpr int kFlushD = 16;   // targets per transpose of the target-side values

}  // namespace

template <int KIND>
__global__ void po_adj_pack_tgt_d_kernel(long nt, const double *__restrict__ tgt7, const double *__restrict__ gam,
                                         double *__restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nt) adj_record64<KIND>(i, nt, tgt7, gam, out + (size_t)adj64_rec(KIND) * i);
}

// Grid = (source blocks from `first` on, target chunks of `chunk` targets). One
// source per thread, its record in registers; the chunk's target records pass
// through shared memory kFlushD at a time. WANT_T: each target's values are
// summed over the CTA's sources through shared memory into the block's row of
// tsum, and po_adj_tsum_kernel adds the rows in order, so that grad_dt is the
// same bits each time, as the FP64 path is for comparisons (an atomicAdd a CTA
// and target, whose order varies: the same time). Only the accumulators of the
// gradients asked for are kept (8,000 sources x 8,000 targets, near field, ms:
// all three 33.0, the two displacements 22.2, the currents and grad_dt 29.7,
// grad_dt alone 19.4).
template <int KIND, bool HAS_M, bool WANT_C, bool WANT_D, bool WANT_T>
__global__ void __launch_bounds__(kThreadsD)
po_adj_fp64_kernel(const double *__restrict__ src, long ns, long first, const double *__restrict__ trec, long nt,
                   long chunk, Wave64 w, double *__restrict__ part, double *__restrict__ tsum)
{
    constexpr int SR = fp64_rec(KIND, HAS_M), TR = adj64_rec(KIND);
    __shared__ double tile[kFlushD * TR];
    __shared__ double vbuf[WANT_T ? kFlushD * (kThreadsD + 1) : 1];
    const long si = (first + blockIdx.x) * blockDim.x + threadIdx.x;
    double s[SR];
#pragma unroll
    for (int q = 0; q < SR; ++q) s[q] = si < ns ? src[(size_t)SR * si + q] : 0.0;
    double acc[kAccAdj];
#pragma unroll
    for (int a = 0; a < kAccAdj; ++a) acc[a] = 0.0;
    const long t0 = (long)blockIdx.y * chunk, t1 = min(nt, t0 + chunk);
    for (long base = t0; base < t1; base += kFlushD) {
        const int cnt = (int)min((long)kFlushD, t1 - base);
        __syncthreads();
        for (int q = threadIdx.x; q < cnt * TR; q += blockDim.x) tile[q] = trec[base * TR + q];
        __syncthreads();
        if (si < ns) {
#pragma unroll 1
            for (int q = 0; q < cnt; ++q) {
                const double v = adj_pair64<KIND, HAS_M, WANT_C, WANT_D, WANT_T>(s, tile + q * TR, w, acc);
                if (WANT_T) vbuf[q * (kThreadsD + 1) + threadIdx.x] = v;
            }
        } else if (WANT_T) {
            for (int q = 0; q < cnt; ++q) vbuf[q * (kThreadsD + 1) + threadIdx.x] = 0.0;
        }
        if (WANT_T) {
            // thread (q, g) adds the g-th eighth of target q's sources, then the eighths combine
            __syncthreads();
            constexpr int SEG = kThreadsD / kFlushD;   // threads per target
            const int q = threadIdx.x / SEG, g = threadIdx.x % SEG;
            double sum = 0.0;
            if (q < cnt)
#pragma unroll
                for (int j = 0; j < kFlushD; ++j) sum += vbuf[q * (kThreadsD + 1) + j * SEG + g];
#pragma unroll
            for (int m = 1; m < SEG; m <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
            if (g == 0 && q < cnt) tsum[blockIdx.x * nt + base + q] = sum;
        }
    }
    if (si >= ns) return;
#pragma unroll
    for (int a = 0; a < kAccAdj; ++a) {
        const int r = adj_row(KIND, WANT_C, WANT_D, a);
        if (r >= 0) part[((long)blockIdx.y * adj_rows(KIND, WANT_C, WANT_D) + r) * ns + si] = acc[a];
    }
}

// gt (with `add`, added to) = the sum of tsum's rows, in their order by eighths
// (row r in eighth r mod 8), then the eighths. A block has 32 targets.
__global__ void __launch_bounds__(256)
po_adj_tsum_kernel(long rows, long nt, const double *tsum, int add, double *__restrict__ gt)
{
    __shared__ double sh[8][32];
    pdl_wait();
    const int l = threadIdx.x & 31, g = threadIdx.x >> 5;
    const long j = (long)blockIdx.x * 32 + l;
    double v = 0.0;
    if (j < nt)
#pragma unroll 4
        for (long r = g; r < rows; r += 8) v += tsum[r * nt + j];
    sh[g][l] = v;
    __syncthreads();
    if (g > 0 || j >= nt) return;
    for (int q = 1; q < 8; ++q) v += sh[q][l];
    gt[j] = add ? gt[j] + v : v;
}

// The pairs the mixed adjoint left out as inside the tangent band: each is
// decided by the reference's FP64 rounding and, if lit, its FP64 terms go
// into the first source chunk's partials (currents; the source displacement
// and the target displacement in the mixed kernel's units, per turn:
// inv_kappa = 2 pi / k), before the epilogues. Order of the additions varies
// between runs for a point with several such pairs (last bits there only).
template <int KIND, bool WANT_T>
__global__ void __launch_bounds__(256)
po_adj_band_fixup_kernel(BandList bl, long ns, const double *__restrict__ src7, const double *__restrict__ cur,
                         int gmode, int ncx, int ncy, double fac_re, double fac_im, long nt,
                         const double *__restrict__ tgt7, const double *gam, Wave64 w,
                         double inv_kappa, int want_c, int want_d, double *__restrict__ part,
                         double *__restrict__ gt, int *__restrict__ err)
{
    pdl_wait();
    const unsigned total = *bl.count;
    if (blockIdx.x == 0 && threadIdx.x == 0 && total > bl.cap) atomicExch(err, kErrBandOverflow);
    const unsigned n = min(total, bl.cap);
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int2 pr = bl.pairs[i];
        double s[kRecD], r[adj64_rec(KIND)], acc[kAccAdj];
        src_record_d(pr.x, ns, src7, cur, gmode, ncx, ncy, fac_re, fac_im, 0, kRecD, s);
        adj_record64<KIND>(pr.y, nt, tgt7, gam, r);
        for (int a = 0; a < kAccAdj; ++a) acc[a] = 0.0;
        const double v = adj_pair64<KIND, true, true, true, WANT_T>(s, r, w, acc) * inv_kappa;
        for (int a = 0; a < kAccAdj; ++a) {
            const int row = adj_row(KIND, want_c, want_d, a);
            const double x = a < 12 ? acc[a] : acc[a] * inv_kappa;
            if (row >= 0 && x != 0.0) atomicAdd(&part[(long)row * ns + pr.x], x);
        }
        if (WANT_T && v != 0.0) atomicAdd(&gt[pr.y], v);
    }
    pdl_trigger();
}

// ---------------------------------------------------------------- host side

Wave64 wave64(double k, double t)
{
    Wave64 w;
    w.k = k;
    w.inv_k = 1.0 / k;
    w.neg = t < 0 ? 0x80000000u : 0u;
    return w;
}

void *pack_src_d_kernel() { return reinterpret_cast<void *>(&po_pack_src_d_kernel); }

void *fp64_kernel(int kind, bool has_m)
{
    if (kind == kKindScalar) return reinterpret_cast<void *>(&po_fp64_kernel<kKindScalar, false>);
    if (kind == kKindNF)
        return has_m ? reinterpret_cast<void *>(&po_fp64_kernel<kKindNF, true>)
                     : reinterpret_cast<void *>(&po_fp64_kernel<kKindNF, false>);
    return has_m ? reinterpret_cast<void *>(&po_fp64_kernel<kKindFF, true>)
                 : reinterpret_cast<void *>(&po_fp64_kernel<kKindFF, false>);
}

template <int KIND, bool HAS_M, bool WANT_C>
static void *adj_fp64_sel(bool want_d, bool want_t)
{
    if constexpr (KIND != kKindFF) {
        if (want_t && want_d) return reinterpret_cast<void *>(&po_adj_fp64_kernel<KIND, HAS_M, WANT_C, true, true>);
        if (want_t || (!WANT_C && !want_d))
            return reinterpret_cast<void *>(&po_adj_fp64_kernel<KIND, HAS_M, WANT_C, false, true>);
    }
    // at least one gradient is wanted
    if (want_d || !WANT_C) return reinterpret_cast<void *>(&po_adj_fp64_kernel<KIND, HAS_M, WANT_C, true, false>);
    return reinterpret_cast<void *>(&po_adj_fp64_kernel<KIND, HAS_M, true, false, false>);
}

template <int KIND, bool HAS_M>
static void *adj_fp64_c(bool want_c, bool want_d, bool want_t)
{
    return want_c ? adj_fp64_sel<KIND, HAS_M, true>(want_d, want_t) : adj_fp64_sel<KIND, HAS_M, false>(want_d, want_t);
}

void *adj_fp64_kernel(int kind, bool has_m, bool want_c, bool want_d, bool want_t)
{
    if (kind == kKindScalar) return adj_fp64_c<kKindScalar, false>(want_c, want_d, want_t);
    if (kind == kKindNF)
        return has_m ? adj_fp64_c<kKindNF, true>(want_c, want_d, want_t)
                     : adj_fp64_c<kKindNF, false>(want_c, want_d, want_t);
    return has_m ? adj_fp64_c<kKindFF, true>(want_c, want_d, want_t)
                 : adj_fp64_c<kKindFF, false>(want_c, want_d, want_t);
}

void *adj_tsum_kernel() { return reinterpret_cast<void *>(&po_adj_tsum_kernel); }

void *adj_pack_tgt_d_kernel(int kind)
{
    if (kind == kKindScalar) return reinterpret_cast<void *>(&po_adj_pack_tgt_d_kernel<kKindScalar>);
    return kind == kKindNF ? reinterpret_cast<void *>(&po_adj_pack_tgt_d_kernel<kKindNF>)
                           : reinterpret_cast<void *>(&po_adj_pack_tgt_d_kernel<kKindFF>);
}

template <bool HAS_M>
static void *band_fixup_sel(int kind)
{
    return kind == kKindFF ? reinterpret_cast<void *>(&po_band_fixup_kernel<kKindFF, HAS_M>)
                           : reinterpret_cast<void *>(&po_band_fixup_kernel<kKindNF, HAS_M>);
}

void *band_fixup_kernel(int kind, bool has_m) { return has_m ? band_fixup_sel<true>(kind) : band_fixup_sel<false>(kind); }

void *adj_band_fixup_kernel(int kind, bool want_t)
{
    if (kind == kKindFF) return reinterpret_cast<void *>(&po_adj_band_fixup_kernel<kKindFF, false>);
    return want_t ? reinterpret_cast<void *>(&po_adj_band_fixup_kernel<kKindNF, true>)
                  : reinterpret_cast<void *>(&po_adj_band_fixup_kernel<kKindNF, false>);
}

}  // namespace po
