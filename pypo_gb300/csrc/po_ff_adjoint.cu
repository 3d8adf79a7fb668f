// po_ff_adjoint.cu -- far-field adjoint (currents and source displacement) of
// the mixed path. Far-field targets are directions and do not move.
//
//   Jbar' += conj(G) gS_J, Mbar' += conj(G) gS_M   (G = e^{-t j k r.s}),
//   displacement: Re[-t j k G (conj(gS_J).J' + conj(gS_M).M')] (n_s . r).
//
// A CTA owns one tile of kTile sources in Hilbert order (the forward's tile
// records, po_farfield.cu), a thread two of them, the two lanes of every
// packed operation. e^{-t j k r.s} = e^{-t j k r.c} e^{-t j k r.(s - c)}: each
// stage of kFFDirs directions has its cotangents multiplied once by
// conj(e^{-t j k r.c}) for the CTA's centre c, and the pair loop takes only
// the offset's phase: FP32 for a narrow tile, split for a wide one.
//
// What bounds the pair loop is the register file: a packed operation reads
// one 64-bit operand a clock, so one with three distinct register pairs takes
// 3.2 clocks of the FP32 pipe instead of 2, and a factor that is one 32-bit
// register for both lanes counts half a read. With the two lanes on two
// sources, the direction and its twelve cotangent words are such factors, in
// most of the loop's operations, and a record serves two pairs a load where
// one source a thread took a record for each. 64 threads rotate the 64
// cotangents of a stage where one warp of four did, with the others waiting.
// The stage's even and odd directions are summed apart, first the even ones,
// then the odd, and added at the stage's end. Measured (one GB300), 251,001
// sources x 40,803 directions, M = 0: 18.4 -> 17.6 ms a call; 151 x 152 ->
// 71 x 70: 0.49 -> 0.44 ms; with M, 62,499 x 10,403: 1.95 -> 1.85 ms. Totals
// kept in FP64 instead of float-float pairs measured slower (18.7 ms): FP64
// additions are that slow here. Two pair records an iteration at 6 CTAs an
// SM; 7 and 8 measured 17.8, one record an iteration 18.2.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <cstdint>
#include <type_traits>

#include "po_device.cuh"
#include "po_kernels.cuh"

namespace po {

namespace {

// Stage of kFFDirs directions: a head of 2 float4 (lowest and highest r per
// axis, the lit-tile proof's box), then the records of the even directions,
// then those of the odd ones; 6 float4 a record: r xyz, gS_J (re, im) x y z,
// gS_M likewise, a spare word, r hi xyz (on 2^-11), r lo xyz, two spare words.
constexpr int kDirRec4 = 6, kDirHead = 2;
constexpr int kStage4 = kDirHead + kFFDirs * kDirRec4;
constexpr int kHalf = kFFDirs / 2;
constexpr int kThreadsFA = kTile / 2;

// Direction d of a stage: even ones first.
__host__ __device__ constexpr int dir_slot(int d) { return (d & 1) * kHalf + (d >> 1); }

}  // namespace

// One CTA per stage: the directions, and their cotangents mapped onto S_J and
// S_M (also written to gam for the near-tangent pairs). The last stage is
// filled up with copies of the last direction carrying no cotangent.
__global__ void __launch_bounds__(kFFDirs)
po_ff_pack_cot_kernel(long nt, const double *__restrict__ tgt7, const double *__restrict__ cot, double t,
                      double *__restrict__ gam, float4 *__restrict__ out)
{
    __shared__ __align__(16) float buf[kStage4 * 4];
    __shared__ float wbox[kFFDirs / 32][6];
    const long i = (long)blockIdx.x * kFFDirs + threadIdx.x;
    const long k = i < nt ? i : nt - 1;
    pdl_wait();
    double rd[3], gk[12];
    ff_direction_d(tgt7, nt, k, rd);
    cot_map(kFF, k, nt, cot, tgt7, rd, t, gk);
    if (i < nt)
        for (int q = 0; q < 12; ++q) gam[(long)q * nt + i] = gk[q];
    float *o = buf + (kDirHead + dir_slot(threadIdx.x) * kDirRec4) * 4;
    float v[6];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double hd = rint(rd[c] * 2048.0) / 2048.0;
        const float h = (float)hd, l = (float)(rd[c] - hd);
        o[c] = h + l;
        o[16 + c] = h;
        o[19 + c] = l;
        v[c] = v[3 + c] = o[c];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            o[3 + 6 * g + 2 * c] = i < nt ? (float)gk[6 * g + c] : 0.f;
            o[4 + 6 * g + 2 * c] = i < nt ? (float)gk[6 * g + 3 + c] : 0.f;
        }
    }
    o[15] = o[22] = o[23] = 0.f;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const float u = __shfl_xor_sync(0xffffffffu, v[q], s);
            v[q] = q < 3 ? fminf(v[q], u) : fmaxf(v[q], u);
        }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int q = 0; q < 6; ++q) wbox[threadIdx.x >> 5][q] = v[q];
    __syncthreads();
    if (threadIdx.x < kDirHead * 4) {
        const int q = threadIdx.x;
        float r = 0.f;
        if (q < 6) {
            r = wbox[0][q];
            for (int w = 1; w < kFFDirs / 32; ++w) r = q < 3 ? fminf(r, wbox[w][q]) : fmaxf(r, wbox[w][q]);
        }
        buf[q] = r;
    }
    __syncthreads();
    float4 *dst = out + (size_t)blockIdx.x * kStage4;
    for (int q = threadIdx.x; q < kStage4; q += kFFDirs) dst[q] = reinterpret_cast<const float4 *>(buf)[q];
    pdl_trigger();
}

namespace {

// The thread's two sources.
struct Src2 {
    float2 sh[3], sl[3], n[3], J[6], M[6];   // offset from the tile centre (hi, lo), normal, currents (re, im) x y z
};

__device__ __forceinline__ float2 ff_adj_ndr(const Src2 &s, const float *r)
{
    return fma2(s.n[2], dup2(r[2]), fma2(s.n[1], dup2(r[1]), mul2(s.n[0], dup2(r[0]))));
}

// One direction against the two sources. LIT: every pair of the stage is
// proven lit, so the mask is left out; the result is the same bits. band: set
// when a pair lies inside the tangent band (left out here; listed afterwards).
template <int T, bool HAS_M, bool WANT_C, bool WANT_D, bool LIT, bool WIDE>
__device__ __forceinline__ void ff_adj_pair(float2 *acc, const float *r, const Src2 &s, bool &band)
{
    float2 sn, cs, tq = dup2(0.0f);
    if (WIDE) {
        const float *h = r + 16, *l = r + 19;
        const float2 Ph = fma2(s.sh[2], dup2(h[2]), fma2(s.sh[1], dup2(h[1]), mul2(s.sh[0], dup2(h[0]))));
        const float2 Pl = fma2(s.sl[2], dup2(r[2]), fma2(s.sl[1], dup2(r[1]), fma2(s.sl[0], dup2(r[0]),
                          fma2(s.sh[2], dup2(l[2]), fma2(s.sh[1], dup2(l[1]), mul2(s.sh[0], dup2(l[0])))))));
        ff_phase_sincos2(Ph, Pl, sn, cs, tq);
    } else {
        const float2 magic = dup2(12582912.0f), twopi = dup2(6.28318530717958648f);
        const float2 P = fma2(s.sh[2], dup2(r[2]), fma2(s.sh[1], dup2(r[1]), mul2(s.sh[0], dup2(r[0]))));
        const float2 ang = mul2(sub2(P, sub2(add2(P, magic), magic)), twopi);
        __sincosf(ang.x, &sn.x, &cs.x);
        __sincosf(ang.y, &sn.y, &cs.y);
    }
    float2 ndr = dup2(0.f);
    if (!LIT || WANT_D) ndr = ff_adj_ndr(s, r);
    float2 gc, gs;   // G = (gc, gs)
    if (LIT) {
        gc = WIDE ? flip_parity(cs, tq) : cs;
        gs = WIDE ? flip_parity(T > 0 ? neg2(sn) : sn, tq) : (T > 0 ? neg2(sn) : sn);
    } else {
        const float2 one = WIDE ? flip_parity(dup2(1.0f), tq) : dup2(1.0f);
        band = band || (fabsf(ndr.x) < kTangentBand) || (fabsf(ndr.y) < kTangentBand);
        const float2 m = make_float2(ndr.x >= kTangentBand ? one.x : 0.0f, ndr.y >= kTangentBand ? one.y : 0.0f);
        gc = mul2(cs, m);
        gs = mul2(T > 0 ? neg2(sn) : sn, m);
    }
    // conj(G) g = (gc g.re + gs g.im, gc g.im - gs g.re)
    const float *gj = r + 3, *gm = r + 9;
#pragma unroll
    for (int c = 0; c < (WANT_C ? 3 : 0); ++c) {
        acc[c] = fma2(gs, dup2(gj[2 * c + 1]), fma2(gc, dup2(gj[2 * c]), acc[c]));
        acc[3 + c] = fma2(neg2(gs), dup2(gj[2 * c]), fma2(gc, dup2(gj[2 * c + 1]), acc[3 + c]));
        acc[6 + c] = fma2(gs, dup2(gm[2 * c + 1]), fma2(gc, dup2(gm[2 * c]), acc[6 + c]));
        acc[9 + c] = fma2(neg2(gs), dup2(gm[2 * c]), fma2(gc, dup2(gm[2 * c + 1]), acc[9 + c]));
    }
    if (WANT_D) {
        // X = conj(gS_J).J' (+ conj(gS_M).M'); Z = G X, Im Z = gc X.im + gs X.re
        float2 xr = dup2(0.f), xi = dup2(0.f);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 re = dup2(gj[2 * c]), im = dup2(gj[2 * c + 1]);
            xr = fma2(re, s.J[2 * c], fma2(im, s.J[2 * c + 1], xr));
            xi = fma2(re, s.J[2 * c + 1], fma2(neg2(im), s.J[2 * c], xi));
            if (HAS_M) {
                const float2 mre = dup2(gm[2 * c]), mim = dup2(gm[2 * c + 1]);
                xr = fma2(mre, s.M[2 * c], fma2(mim, s.M[2 * c + 1], xr));
                xi = fma2(mre, s.M[2 * c + 1], fma2(neg2(mim), s.M[2 * c], xi));
            }
        }
        const float2 zi = fma2(gc, xi, mul2(gs, xr));
        acc[12] = fma2(mul2(zi, ndr), dup2(T > 0 ? 6.28318530717958647f : -6.28318530717958647f), acc[12]);
    }
}

// One direction's record with its cotangents multiplied in place by
// conj(e^{-t j k r.c}) for the CTA's tile centre c (hi xyz, lo xyz, turns).
// With s = c + w, conj(G) g = conj(G_w) (conj(G_c) g). r.c in split form: hi
// products exact (r hi on 2^-11, c hi on the frame's quantum), the rest in
// one FP32 sum, reduced exactly to half turns, as the forward's tile phase.
template <int T>
__device__ __forceinline__ void ff_rotate_cot(float *r, const float *c)
{
    const float *h = r + 16, *l = r + 19;
    const float Ph = __fmaf_rn(c[2], h[2], __fmaf_rn(c[1], h[1], __fmul_rn(c[0], h[0])));
    const float Pl = __fmaf_rn(c[5], r[2], __fmaf_rn(c[4], r[1], __fmaf_rn(c[3], r[0],
                     __fmaf_rn(c[2], l[2], __fmaf_rn(c[1], l[1], __fmul_rn(c[0], l[0]))))));
    float2 sn2, cs2, tq;
    ff_phase_sincos2(dup2(Ph), dup2(Pl), sn2, cs2, tq);
    const float gc = flip_parity(cs2, tq).x, gs = flip_parity(T > 0 ? neg2(sn2) : sn2, tq).x;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const float re = r[3 + 2 * q], im = r[4 + 2 * q];
        r[3 + 2 * q] = __fmaf_rn(gc, re, __fmul_rn(gs, im));
        r[4 + 2 * q] = __fmaf_rn(gc, im, __fmul_rn(-gs, re));
    }
}

}  // namespace

// Grid = (source tiles, chunks of `chunk` stages). order: curve position ->
// source. boxes: the stages' direction boxes may prove a stage lit for the
// CTA's normals (M = 0 kernels). WANT_C, WANT_D: the gradients asked for; the
// other's accumulators are left out (40,000 sources x 20,000 directions, ms:
// both 1.61, the currents' alone 1.09, the displacement's alone 0.88).
template <int T, bool HAS_M, bool WANT_C, bool WANT_D>
__global__ void __launch_bounds__(kThreadsFA, HAS_M ? kMinBlocksFAM : kMinBlocksFA)
po_ff_adj_kernel(const float4 *tiles, long ns, const float4 *dirs, long nstage, long chunk,
                 long nt, double *__restrict__ part, int *__restrict__ err, BandList bl,
                 const int *order)
{
    constexpr int R4 = ff_rec4(HAS_M), T4 = ff_tile4(HAS_M);
    constexpr int NA = adj_rows(kKindFF, WANT_C, WANT_D);
    constexpr int A0 = WANT_C ? 0 : 12;   // first accumulator kept; row a holds accumulator A0 + a
    constexpr bool kLit = !HAS_M;
    extern __shared__ __align__(128) float4 stage[];   // kStagesFA stages, then per thread: totals' lo, the even sums
    __shared__ __align__(8) uint64_t full[kStagesFA];
    pdl_wait();
    float2 *keep = reinterpret_cast<float2 *>(stage + (size_t)kStagesFA * kStage4) + threadIdx.x;
    auto lo = [&](int a) -> float2 & { return keep[a * kThreadsFA]; };
    auto even = [&](int a) -> float2 & { return keep[(NA + a) * kThreadsFA]; };

    // the tile (po_ff_pack_kernel): centre, wide flag, and the thread's pair record
    const float4 *tile = tiles + (size_t)blockIdx.x * T4;
    const float *tf = reinterpret_cast<const float *>(tile);
    float cen[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) cen[c] = tf[c];
    const bool wide = tf[12] != 0.0f;
    Src2 s;
    {
        const float2 *rec = reinterpret_cast<const float2 *>(tile + kFFHead + (size_t)threadIdx.x * R4);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            s.sh[c] = rec[c];
            s.sl[c] = rec[12 + c];
            s.n[c] = rec[9 + c];
            s.J[2 * c] = rec[3 + c];
            s.J[2 * c + 1] = rec[6 + c];
            s.M[2 * c] = HAS_M ? rec[16 + c] : dup2(0.f);
            s.M[2 * c + 1] = HAS_M ? rec[19 + c] : dup2(0.f);
        }
    }
    const long pos = (long)blockIdx.x * kTile + 2 * threadIdx.x;   // curve position of the first source

    float2 hi[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) hi[a] = lo(a) = dup2(0.f);

    // The tile's box of normals (padding sources repeat the last one): the
    // CTA's side of the lit proof, min n.r >= 1e-5 over the two boxes, the
    // least of n.r being the sum of the least corner products per axis (the
    // per-pair test is lit when n.r >= 1e-6).
    float nbox[6];
    if (kLit) {
#pragma unroll
        for (int c = 0; c < 6; ++c) nbox[c] = tf[6 + c];
    }

    const long t0 = (long)blockIdx.y * chunk;
    const int nst = (int)max(0L, min(nstage, t0 + chunk) - t0);
    if (threadIdx.x == 0) {
        for (int q = 0; q < kStagesFA; ++q) mbar_init(&full[q], 1);
        mbar_fence_init();
    }
    __syncthreads();
    auto issue = [&](int it) {
        constexpr uint32_t bytes = (uint32_t)(kStage4 * sizeof(float4));
        uint64_t *bar = &full[it % kStagesFA];
        fence_proxy_async();
        mbar_expect_tx(bar, bytes);
        tma_load_1d(stage + (size_t)(it % kStagesFA) * kStage4, dirs + (t0 + it) * kStage4, bytes, bar);
    };
    if (threadIdx.x == 0)
        for (int it = 0; it < nst && it < kStagesFA; ++it) issue(it);

    for (int it = 0; it < nst; ++it) {
        const bool ok = mbar_wait_bounded(&full[it % kStagesFA], (uint32_t)((it / kStagesFA) & 1));
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicExch(err, kErrWaitTimeout);
                for (int q = 0; q < kStagesFA; ++q) (void)mbar_wait_bounded(&full[q], 0);
            }
            return;
        }
        float4 *st = stage + (size_t)(it % kStagesFA) * kStage4;
        const float *box = reinterpret_cast<const float *>(st);
        float *recs = reinterpret_cast<float *>(st + kDirHead);
        for (int d = threadIdx.x; d < kFFDirs; d += kThreadsFA) ff_rotate_cot<T>(recs + d * kDirRec4 * 4, cen);
        bool lit = false;   // block-uniform: the same boxes in every thread
        if (kLit) {
            float L = 0.0f;
#pragma unroll
            for (int c = 0; c < 3; ++c)
                L += fminf(fminf(nbox[c] * box[c], nbox[c] * box[3 + c]),
                           fminf(nbox[3 + c] * box[c], nbox[3 + c] * box[3 + c]));
            lit = L >= 1e-5f;
        }
        __syncthreads();
        bool band = false;
        auto half = [&](int h, auto lit_c, auto wide_c) {
            constexpr bool LIT = decltype(lit_c)::value, WIDE = decltype(wide_c)::value;
            constexpr int NL = WIDE ? 6 : 4;   // float4 read per record
            float2 acc[kAccAdj];
#pragma unroll
            for (int a = 0; a < kAccAdj; ++a) acc[a] = dup2(0.f);
            const float4 *rec4 = st + kDirHead + h * kHalf * kDirRec4;
#pragma unroll 2
            for (int p = 0; p < kHalf; ++p) {
                float r[4 * NL];
#pragma unroll
                for (int q = 0; q < NL; ++q) {
                    const float4 v = rec4[p * kDirRec4 + q];
                    r[4 * q] = v.x;
                    r[4 * q + 1] = v.y;
                    r[4 * q + 2] = v.z;
                    r[4 * q + 3] = v.w;
                }
                ff_adj_pair<T, HAS_M, WANT_C, WANT_D, LIT, WIDE>(acc, r, s, band);
            }
            if (h == 0) {
#pragma unroll
                for (int a = 0; a < NA; ++a) even(a) = acc[A0 + a];
            } else {
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    float2 sm, e;
                    two_sum2(hi[a], add2(even(a), acc[A0 + a]), sm, e);
                    hi[a] = sm;
                    lo(a) = add2(lo(a), e);
                }
            }
        };
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            if (wide)
                half(h, std::false_type{}, std::true_type{});
            else if (lit)
                half(h, std::bool_constant<kLit>{}, std::false_type{});
            else
                half(h, std::false_type{}, std::false_type{});
        }
        if (band) {
            // the rare path: the stage's pairs tested again, those inside the
            // band listed for the FP64 fixup (padding left out)
#pragma unroll 1
            for (int d = 0; d < kFFDirs; ++d) {
                const long ti = (t0 + it) * kFFDirs + d;
                if (ti >= nt) break;
                const float2 nd = ff_adj_ndr(s, recs + dir_slot(d) * kDirRec4 * 4);
                if (fabsf(nd.x) < kTangentBand && pos < ns) band_defer(bl, order[pos], ti);
                if (fabsf(nd.y) < kTangentBand && pos + 1 < ns) band_defer(bl, order[pos + 1], ti);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && it + kStagesFA < nst) issue(it + kStagesFA);
    }
    pdl_trigger();
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        if (pos + l >= ns) continue;
        const long si = order[pos + l];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const float2 e = lo(a);
            part[((long)blockIdx.y * NA + a) * ns + si] =
                l == 0 ? (double)hi[a].x + (double)e.x : (double)hi[a].y + (double)e.y;
        }
    }
}

// ------------------------------------------------------------------ host side

int ff_adj_smem_bytes(bool want_c, bool want_d)
{
    return kStagesFA * kStage4 * 16 + 2 * adj_rows(kKindFF, want_c, want_d) * kThreadsFA * 8;
}
int ff_adj_threads() { return kThreadsFA; }
int ff_adj_stage4() { return kStage4; }

template <int T, bool HAS_M>
static void *ff_adj_sel(bool want_c, bool want_d)
{
    if (!want_c) return reinterpret_cast<void *>(&po_ff_adj_kernel<T, HAS_M, false, true>);   // one of the two is wanted
    return want_d ? reinterpret_cast<void *>(&po_ff_adj_kernel<T, HAS_M, true, true>)
                  : reinterpret_cast<void *>(&po_ff_adj_kernel<T, HAS_M, true, false>);
}

void *ff_adj_kernel(int t_sign, bool has_m, bool want_c, bool want_d)
{
    if (t_sign < 0) return has_m ? ff_adj_sel<-1, true>(want_c, want_d) : ff_adj_sel<-1, false>(want_c, want_d);
    return has_m ? ff_adj_sel<1, true>(want_c, want_d) : ff_adj_sel<1, false>(want_c, want_d);
}

void *ff_pack_cot_kernel() { return reinterpret_cast<void *>(&po_ff_pack_cot_kernel); }

}  // namespace po
