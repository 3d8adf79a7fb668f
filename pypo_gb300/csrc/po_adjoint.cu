// po_adjoint.cu -- adjoint (vector-Jacobian) kernels of the PO integrator.
//
// The reference has no derivatives; these kernels are new. For a real loss
// L of the outputs with real cotangent rows y_bar, write gE = y_bar(E.re) +
// j y_bar(E.im) and gH likewise (after mapping the mode's epilogue back onto
// E and H). With d = r_t - r_s and the forward coefficients c1, c2' = G s2/R^2,
// c3' = G s3/R of the near-field kernel (E = c1 J + c2'(J.d)d + c3'(M x d),
// H = c1 M + c2'(M.d)d - c3'(J x d)):
//
//   currents      Jbar' = sum_t conj(c1) gE + conj(c2')(gE.d)d + conj(c3')(gH x d)
//                 Mbar' = sum_t conj(c1) gH + conj(c2')(gH.d)d - conj(c3')(gE x d)
//                 (primes: with respect to the folded currents; the epilogue
//                 multiplies by conj(prefactor * weight * area))
//   displacement  phi(d) = Re[a.F_E + b.F_H], a = conj(gE), b = conj(gH);
//                 grad_d phi = Re[sigma d + c2' grad(beta) + c3' W] with
//                 alpha = a.J + b.M, beta = (J.d)(a.d) + (M.d)(b.d),
//                 W = a x M - b x J, sigma = dc1 alpha + dc2 beta + dc3 (W.d),
//                 dc1 = G/R^2 [t(1-3u^2) + j(2u-3u^3)],
//                 dc2 = G/R^4 [-t(1-15u^2) + j(-6u+15u^3)],
//                 dc3 = G/R^3 [-(1-3u^2) - 3jtu]   (u = 1/kR)
//                 dL/d delta_s = -n_s . sum_t grad_d phi, dL/d delta_t = n_t . sum_s grad_d phi
//                 (normal-direction displacement with normals and areas frozen,
//                 the reference's surface-error convention).
//   far field     Jbar' = sum_t conj(G) gS_J, Mbar' = sum_t conj(G) gS_M with
//                 gS_J = P gE + t r x gH, gS_M = P gH - t r x gE (P = I - r r^T);
//                 dL/d delta_s = n_s . sum_t Re[-t j k G (conj(gS_J).J' + conj(gS_M).M')] r.
// The illumination mask is piecewise constant: its derivative is dropped.
//
// This file holds the formulas, the cotangent mapping and the epilogues. The
// mixed-precision kernels, pair-packed, are in po_adjoint_pk.cu, the plain
// FP64 ones in po_fp64.cu.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <cstdint>

#include "po_device.cuh"
#include "po_kernels.cuh"

namespace po {

// ------------------------------------------------------- cotangent mapping

// The mapping itself is cot_map (po_device.cuh); this kernel serves the FP64
// path, the mixed paths map while they pack (po_adj_pack_kernel below,
// po_ff_pack_cot_kernel).
__global__ void po_adj_cot_kernel(int mode, long nt, const double *__restrict__ cot, const double *__restrict__ tgt7,
                                  double t, double *__restrict__ gam)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nt) return;
    double g[12], r[3] = {0, 0, 0};
    if (mode == kFF) ff_direction_d(tgt7, nt, i, r);
    cot_map(mode, i, nt, cot, tgt7, r, t, g);
    for (int q = 0; q < 12; ++q) gam[(long)q * nt + i] = g[q];
}

// EHP: the outputs are a pointwise nonlinear function of the incident E, H at
// the target (ehp_reflect). Its vector-Jacobian product at the forward's
// fields, one forward-mode pass per input (E re xyz, E im, H re, H im):
// gam_k = sum_rows cot_row d(out_row)/d(in_k) is dL/d(in_k), i.e. gE and gH
// for the EH adjoint that follows. `eh` holds the EH forward's 12 rows.
__global__ void po_adj_ehp_cot_kernel(long nt, const double *__restrict__ cot, const double *__restrict__ eh,
                                      const double *__restrict__ tgt7, double zeta_inv, double *__restrict__ gam)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nt) return;
    const double n[3] = {tgt7[3 * nt + i], tgt7[4 * nt + i], tgt7[5 * nt + i]};
    double base[12];
    for (int q = 0; q < 12; ++q) base[q] = eh[(long)q * nt + i];
    for (int kq = 0; kq < 12; ++kq) {
        Dual in[12], out[15];
        for (int q = 0; q < 12; ++q) in[q] = Dual(base[q], q == kq ? 1.0 : 0.0);
        ehp_reflect(in, in + 3, in + 6, in + 9, n, zeta_inv, out);
        double g = 0.0;
        for (int r = 0; r < 15; ++r) g += cot[(long)r * nt + i] * out[r].d;
        gam[(long)kq * nt + i] = g;
    }
}

// ---------------------------------------------------------------- epilogues

// Sums the chunks of the source-side partials (N rows: adj_rows); unfolds the
// currents by conj(fac * weight * area); scales the displacement term to mm.
// G threads share a source (thread g adds chunks g, g + G, ..., then a tree),
// as in the forward's epilogue. The blocks past the nblk_s of the sources
// scale the target sums gt into grad_dt; where the call has no rows, nblk_s
// is 0 (of the N = 1 instance).
template <int G, int N>
__global__ void __launch_bounds__(kEpiThreads)
po_adj_epilogue_kernel(int kind, int nsplit, long ns, const double *part,
                       const double *__restrict__ src7, int gmode, int ncx, int ncy, double fac_re, double fac_im,
                       double dscale, double *__restrict__ grad_cur, double *__restrict__ grad_ds, long nblk_s, long nt,
                       const double *gt, double tscale, double *__restrict__ grad_dt)
{
    constexpr int SB = kEpiThreads / G;   // sources per block
    __shared__ double sh[G > 1 ? G / 2 : 1][G > 1 ? N : 1][G > 1 ? SB : 1];
    pdl_wait();
    if ((long)blockIdx.x >= nblk_s) {
        const long j = ((long)blockIdx.x - nblk_s) * kEpiThreads + threadIdx.x;
        if (j < nt) grad_dt[j] = tscale * gt[j];
        return;
    }
    const int sl = threadIdx.x % SB, g = threadIdx.x / SB;
    const long i = (long)blockIdx.x * SB + sl;
    double a[N];
#pragma unroll
    for (int q = 0; q < N; ++q) a[q] = 0.0;
    if (i < ns) {
#pragma unroll 2
        for (int s = g; s < nsplit; s += G)
#pragma unroll
            for (int q = 0; q < N; ++q) a[q] += part[((long)s * N + q) * ns + i];
    }
    if constexpr (G > 1) {
#pragma unroll
        for (int w = G / 2; w > 0; w >>= 1) {
            if (g >= w && g < 2 * w)
#pragma unroll
                for (int q = 0; q < N; ++q) sh[g - w][q][sl] = a[q];
            __syncthreads();
            if (g < w)
#pragma unroll
                for (int q = 0; q < N; ++q) a[q] += sh[g][q][sl];
            __syncthreads();
        }
        if (g > 0) return;
    }
    if (i >= ns) return;
    const double w = trap_weight(i, gmode, ncx, ncy) * src7[6 * ns + i];
    const double fr = fac_re * w, fi = fac_im * w;
    if (grad_cur && kind == kKindScalar) {
        // conj(f) * (re + j im), two rows
        grad_cur[i] = fr * a[0] + fi * a[N > 1 ? 1 : 0];
        grad_cur[ns + i] = fr * a[N > 1 ? 1 : 0] - fi * a[0];
    } else if (N >= 12 && grad_cur)
        for (int h = 0; h < 2; ++h)
            for (int c = 0; c < 3; ++c) {
                const double re = a[N >= 12 ? 6 * h + c : 0], im = a[N >= 12 ? 6 * h + 3 + c : 0];
                // conj(f) * (re + j im)
                grad_cur[(long)(6 * h + c) * ns + i] = fr * re + fi * im;
                grad_cur[(long)(6 * h + 3 + c) * ns + i] = fr * im - fi * re;
            }
    if (grad_ds) grad_ds[i] = dscale * a[N - 1];   // the last row
}

// -------------------------------------------------------------------- packing

// Set-up of the near-field and scalar adjoint. Blocks 0 .. sblk-1: one source
// a thread, as the one-source records of the pair kernel, 6 float4 (kRec):
//   r0 = (sh.x, sh.y, sh.z, n.x)     hi position (turns), normal x
//   r1 = (sl.x, sl.y, sl.z, n.y)     lo position (turns), normal y
//   r2 = (Jx.re, Jx.im, Jy.re, Jy.im)
//   r3 = (Jz.re, Jz.im, Mx.re, Mx.im)
//   r4 = (My.re, My.im, Mz.re, Mz.im)
//   r5 = (n.z, 0, 0, 0)
// (scalar: S' in the J.x slot, the rest zero); fac: complex factor folded into
// the currents (times weight * area). The last block's threads past the sources
// pack a record without normal and currents at 4096 quanta, where no target is
// (they reach to 1025), so that the pair kernel's thread for it adds zeros, not
// 0 / 0, to the target sums. The remaining blocks: a target each
// thread (an odd count's last pair padded with the last target carrying no
// cotangent): its cotangents mapped onto E and H, written to gam (unless null)
// for the near-tangent pairs and into the pair-packed records (layout in
// po_adjoint_pk.cu, rec4 float4 per pair); its sum gt cleared.
__global__ void __launch_bounds__(128)
po_adj_pack_kernel(long ns, const double *__restrict__ src7, const double *__restrict__ cur, int gmode, int ncx,
                   int ncy, const Frame *frp, double fac_re, double fac_im, int scalar, long sblk,
                   float4 *__restrict__ src, int mode, long nt, const double *__restrict__ tgt7,
                   const double *__restrict__ cot, double t, double *__restrict__ gam, int rec4,
                   float *__restrict__ tgt, double *__restrict__ gt)
{
    pdl_wait();
    const Frame fr = *frp;
    if ((long)blockIdx.x < sblk) {
        const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= ns) {
            float4 *o = src + (size_t)kRec * i;
            o[0] = make_float4(0.f, 0.f, (float)(4096.0 * fr.q), 0.f);
#pragma unroll
            for (int q = 1; q < kRec; ++q) o[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            pdl_trigger();
            return;
        }
        float h[3], l[3];
        for (int c = 0; c < 3; ++c) split_hi_lo((src7[c * ns + i] - fr.o[c]) * fr.kappa, fr, h[c], l[c]);
        const double w = trap_weight(i, gmode, ncx, ncy) * src7[6 * ns + i];
        const double fr_ = fac_re * w, fi_ = fac_im * w;
        float c[12];   // J.re/im x y z interleaved, then M
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const int grp = q / 3, ax = q % 3;
            if (scalar && q > 0) {
                c[2 * q] = c[2 * q + 1] = 0.f;
                continue;
            }
            const double re = cur[scalar ? i : (grp * 6 + ax) * ns + i];
            const double im = cur[scalar ? ns + i : (grp * 6 + 3 + ax) * ns + i];
            c[2 * q] = (float)(fr_ * re - fi_ * im);
            c[2 * q + 1] = (float)(fr_ * im + fi_ * re);
        }
        float4 *o = src + (size_t)kRec * i;
        o[0] = make_float4(h[0], h[1], h[2], (float)src7[3 * ns + i]);
        o[1] = make_float4(l[0], l[1], l[2], (float)src7[4 * ns + i]);
        o[2] = make_float4(c[0], c[1], c[2], c[3]);
        o[3] = make_float4(c[4], c[5], c[6], c[7]);
        o[4] = make_float4(c[8], c[9], c[10], c[11]);
        o[5] = make_float4((float)src7[5 * ns + i], 0.f, 0.f, 0.f);
        pdl_trigger();
        return;
    }
    const long i = ((long)blockIdx.x - sblk) * blockDim.x + threadIdx.x;
    if (i >= 2 * ((nt + 1) / 2)) return;
    const bool real = i < nt;
    const long k = real ? i : nt - 1;
    float v[26];
    for (int c = 0; c < 3; ++c) split_hi_lo((tgt7[c * nt + k] - fr.o[c]) * fr.kappa, fr, v[c], v[3 + c]);
    double g[12], n[3];   // gE re xyz, im xyz, gH likewise
    for (int q = 0; q < 12; ++q) g[q] = 0.0;
    for (int c = 0; c < 3; ++c) n[c] = 0.0;
    if (real) {
        cot_map(mode, k, nt, cot, tgt7, n, t, g);
        if (gam)
            for (int q = 0; q < 12; ++q) gam[(long)q * nt + k] = g[q];
        for (int c = 0; c < 3; ++c) n[c] = tgt7[(3 + c) * nt + k];
        if (gt) gt[k] = 0.0;
    }
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const double *gw = g + 6 * w;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[6 + 6 * w + 2 * c] = (float)gw[c];
            v[7 + 6 * w + 2 * c] = (float)gw[3 + c];
        }
        // a = conj(gE), b = conj(gH): a.n | b.n
        const double dr = gw[0] * n[0] + gw[1] * n[1] + gw[2] * n[2];
        const double di = -(gw[3] * n[0] + gw[4] * n[1] + gw[5] * n[2]);
        v[21 + 2 * w] = (float)dr;
        v[22 + 2 * w] = (float)di;
    }
    for (int c = 0; c < 3; ++c) v[18 + c] = (float)n[c];
    v[25] = 0.f;
    float *o = tgt + (i >> 1) * (long)(rec4 * 4) + (i & 1);
#pragma unroll
    for (int q = 0; q < 26; ++q)
        if (q < 2 * rec4) o[2 * q] = v[q];
    pdl_trigger();
}

// ----------------------------------------------------------- instantiations

void *adj_cot_kernel() { return reinterpret_cast<void *>(&po_adj_cot_kernel); }
void *adj_ehp_cot_kernel() { return reinterpret_cast<void *>(&po_adj_ehp_cot_kernel); }
void *adj_pack_kernel() { return reinterpret_cast<void *>(&po_adj_pack_kernel); }
template <int N>
static void *adj_epilogue_sel(int groups)
{
    return groups == 8 ? reinterpret_cast<void *>(&po_adj_epilogue_kernel<8, N>)
                       : reinterpret_cast<void *>(&po_adj_epilogue_kernel<1, N>);
}

void *adj_epilogue_kernel(int groups, int rows)
{
    switch (rows) {
    case 2: return adj_epilogue_sel<2>(groups);
    case 3: return adj_epilogue_sel<3>(groups);
    case 12: return adj_epilogue_sel<12>(groups);
    case 13: return adj_epilogue_sel<13>(groups);
    default: return adj_epilogue_sel<1>(groups);
    }
}

}  // namespace po
