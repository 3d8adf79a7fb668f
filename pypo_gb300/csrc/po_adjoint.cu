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

// Cotangents of the mode's output rows -> (gE, gH) per target (near field)
// or (gS_J, gS_M) (far field), as 12 double rows (re xyz, im xyz, ...).
__global__ void po_adj_cot_kernel(int mode, long nt, const double *__restrict__ cot, const double *__restrict__ tgt7,
                                  double t, double *__restrict__ gam)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nt) return;
    double ge[6] = {0, 0, 0, 0, 0, 0}, gh[6] = {0, 0, 0, 0, 0, 0};
    auto row = [&](int r) { return cot[(long)r * nt + i]; };
    if (mode == kEH || mode == kFF) {
        for (int c = 0; c < 6; ++c) {
            ge[c] = row(c);
            gh[c] = row(6 + c);
        }
    }
    if (mode == kScalar) {   // (re, im) of the one complex output, in the E.x slot
        ge[0] = row(0);
        ge[3] = row(1);
    }
    if (mode == kJMEH) {
        for (int c = 0; c < 6; ++c) {
            ge[c] = row(12 + c);
            gh[c] = row(18 + c);
        }
    }
    if (mode == kJM || mode == kJMEH) {
        // J = 2 n x H  ->  gH += 2 gJ x n
        const double n[3] = {tgt7[3 * nt + i], tgt7[4 * nt + i], tgt7[5 * nt + i]};
        for (int part_ = 0; part_ < 2; ++part_) {
            const double g[3] = {row(3 * part_ + 0), row(3 * part_ + 1), row(3 * part_ + 2)};
            gh[3 * part_ + 0] += 2.0 * (g[1] * n[2] - g[2] * n[1]);
            gh[3 * part_ + 1] += 2.0 * (g[2] * n[0] - g[0] * n[2]);
            gh[3 * part_ + 2] += 2.0 * (g[0] * n[1] - g[1] * n[0]);
        }
    }
    if (mode == kFF) {
        // gS_J = P gE + t r x gH ; gS_M = P gH - t r x gE
        const double th = tgt7[i], ph = tgt7[nt + i];
        const double r[3] = {cos(ph) * sin(th), sin(ph) * sin(th), cos(th)};
        double sj[6], sm[6];
        for (int part_ = 0; part_ < 2; ++part_) {
            const double *e = ge + 3 * part_, *h = gh + 3 * part_;
            const double ed = e[0] * r[0] + e[1] * r[1] + e[2] * r[2];
            const double hd = h[0] * r[0] + h[1] * r[1] + h[2] * r[2];
            const double rxh[3] = {r[1] * h[2] - r[2] * h[1], r[2] * h[0] - r[0] * h[2], r[0] * h[1] - r[1] * h[0]};
            const double rxe[3] = {r[1] * e[2] - r[2] * e[1], r[2] * e[0] - r[0] * e[2], r[0] * e[1] - r[1] * e[0]};
            for (int c = 0; c < 3; ++c) {
                sj[3 * part_ + c] = e[c] - ed * r[c] + t * rxh[c];
                sm[3 * part_ + c] = h[c] - hd * r[c] - t * rxe[c];
            }
        }
        for (int c = 0; c < 6; ++c) {
            ge[c] = sj[c];
            gh[c] = sm[c];
        }
    }
    for (int c = 0; c < 6; ++c) {
        gam[(long)c * nt + i] = ge[c];
        gam[(long)(6 + c) * nt + i] = gh[c];
    }
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

// Sums the chunks of the source-side partials; unfolds the currents by
// conj(fac * weight * area); scales the displacement term to mm.
__global__ void po_adj_src_epilogue_kernel(int kind, int nsplit, long ns, const double *__restrict__ part,
                                           const double *__restrict__ src7, int gmode, int ncx, int ncy,
                                           double fac_re, double fac_im, double dscale,
                                           double *__restrict__ grad_cur, double *__restrict__ grad_ds)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    double a[kAccAdj];
    for (int q = 0; q < kAccAdj; ++q) a[q] = 0.0;
    for (int s = 0; s < nsplit; ++s)
        for (int q = 0; q < kAccAdj; ++q) a[q] += part[((long)s * kAccAdj + q) * ns + i];
    double w = src7[6 * ns + i];
    if (gmode >= 0) {
        const long xu = i / ncy, yv = i - xu * ncy;
        if (xu == 0 || xu == ncx - 1) w *= 0.5;
        if (gmode != 1 && (yv == 0 || yv == ncy - 1)) w *= 0.5;
    }
    const double fr = fac_re * w, fi = fac_im * w;
    if (grad_cur && kind == kKindScalar) {
        // conj(f) * (re + j im), two rows
        grad_cur[i] = fr * a[0] + fi * a[3];
        grad_cur[ns + i] = fr * a[3] - fi * a[0];
    } else if (grad_cur)
        for (int g = 0; g < 2; ++g)
            for (int c = 0; c < 3; ++c) {
                const double re = a[6 * g + c], im = a[6 * g + 3 + c];
                // conj(f) * (re + j im)
                grad_cur[(long)(6 * g + c) * ns + i] = fr * re + fi * im;
                grad_cur[(long)(6 * g + 3 + c) * ns + i] = fr * im - fi * re;
            }
    if (grad_ds) grad_ds[i] = dscale * a[12];
}

__global__ void po_adj_tgt_epilogue_kernel(int nsplit, long nt, const double *__restrict__ part, double dscale,
                                           double *__restrict__ grad_dt)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nt) return;
    double s = 0.0;
    for (int c = 0; c < nsplit; ++c) s += part[(long)c * nt + i];
    grad_dt[i] = dscale * s;
}

// ----------------------------------------------------------- instantiations

void *adj_cot_kernel() { return reinterpret_cast<void *>(&po_adj_cot_kernel); }
void *adj_ehp_cot_kernel() { return reinterpret_cast<void *>(&po_adj_ehp_cot_kernel); }
void *adj_src_epilogue_kernel() { return reinterpret_cast<void *>(&po_adj_src_epilogue_kernel); }
void *adj_tgt_epilogue_kernel() { return reinterpret_cast<void *>(&po_adj_tgt_epilogue_kernel); }

}  // namespace po
