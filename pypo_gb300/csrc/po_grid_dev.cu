// po_grid_dev.cu -- FP64 reflector grid generation on the device.
//
// The same formulas as the host generator po_grid.cpp (reference
// src/common/InterfaceReflector.cpp: paraboloid xy / uv :84-135, :166-244,
// hyperboloid :271-322, :353-434, ellipsoid :460-509, :540-621, plane xy / uv /
// AoE :645-686, :712-768, :794-849, 4x4 transform :35-57), one thread per grid
// point, written straight into the 7-row device layout the propagation entry
// points take (x, y, z, nx, ny, nz, area; index i*ncy + j). The optional
// surface error (:852-866) keeps the reference's random sequence, drawn on
// the device (normal_deviates_dev): mt19937 seeded with rms_seed and a fresh
// normal distribution per point (src/include/Random.h:112-116), applied along
// the normals where the deviates are formed.
//
// The correlated surface error (po_correlated_error_dev) is a spectral
// synthesis over random modes drawn from the same generator, evaluated on
// the device at every grid point.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include "po_internal.h"

namespace po {

// Scalars of a reflparams, by value.
struct GridSpec {
    int type, gmode, ncx, ncy, nfac, spheric, transform;
    double a, b, c;
    double lxu0, lxu1, lyv0, lyv1, gcx, gcy, ecc, rot;
    double m[12];   // first three rows of the 4x4 transform
};

namespace {

constexpr double kPiD = 3.14159265358979323846;

__device__ void quadric_d(int type, double a, double b, double c, double x, double y, double &z, double n[3])
{
    switch (type) {
    case 0:
        z = x * x / (a * a) + y * y / (b * b);
        n[0] = -2 * x / (a * a); n[1] = -2 * y / (b * b); n[2] = 1;
        break;
    case 1:
        z = c * sqrt(x * x / (a * a) + y * y / (b * b) + 1);
        n[0] = -2 * x / (a * a); n[1] = -2 * y / (b * b); n[2] = 2 * z / (c * c);
        break;
    case 2:
        z = c * sqrt(1 - x * x / (a * a) - y * y / (b * b));
        n[0] = 2 * x / (a * a); n[1] = 2 * y / (b * b); n[2] = 2 * z / (c * c);
        break;
    default:
        z = 0;
        n[0] = 0; n[1] = 0; n[2] = 1;
        break;
    }
}

__device__ void slope_d(int type, double a, double b, double c, double x, double y, double z, double &zx, double &zy)
{
    switch (type) {
    case 0: zx = 2 * x / (a * a); zy = 2 * y / (b * b); break;
    case 1: zx = c * c / z * x / (a * a); zy = c * c / z * y / (b * b); break;
    case 2: zx = -c * c / z * x / (a * a); zy = -c * c / z * y / (b * b); break;
    default: zx = 0; zy = 0; break;
    }
}

}  // namespace

__global__ void po_grid_kernel(GridSpec g, double *__restrict__ out)
{
    const long n = (long)g.ncx * g.ncy;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    const int i = (int)(idx / g.ncy), j = (int)(idx - (long)i * g.ncy);
    double x = 0, y = 0, z = 0, nx = 0, ny = 0, nz = 1, area = 0;
    if (g.gmode == 0) {
        const double dx = (g.lxu1 - g.lxu0) / (g.ncx - 1), dy = (g.lyv1 - g.lyv0) / (g.ncy - 1);
        const bool centred = g.type == 0 || g.type == 1;   // quadrics offset by gcenter; ellipsoids, planes not
        x = i * dx + g.lxu0 + (centred ? g.gcx : 0.0);
        y = j * dy + g.lyv0 + (centred ? g.gcy : 0.0);
        double q[3];
        quadric_d(g.type, g.a, g.b, g.c, x, y, z, q);
        if (g.type == 3) {
            nx = 0; ny = 0; nz = g.nfac;
            area = dx * dy;
        } else {
            const double nrm = sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]);
            nx = g.nfac * q[0] / nrm; ny = g.nfac * q[1] / nrm; nz = g.nfac * q[2] / nrm;
            area = nrm * dx * dy;
        }
    } else if (g.gmode == 1) {
        const double du0 = (g.lxu1 - g.lxu0) / (g.ncx - 1), dv = (g.lyv1 - g.lyv0) / g.ncy;
        const double rot = g.rot * kPiD / 180, cr = cos(rot), sr = sin(rot);
        const double v = (j * dv + g.lyv0) * kPiD / 180, sv = sin(v), cv = cos(v);
        const double ef = sqrt(1 - g.ecc * g.ecc * sv * sv);
        const double duv = du0 / ef;
        const double u = i * duv + g.lxu0 / ef;
        const double dudv = u / (ef * ef) * g.ecc * g.ecc * cv * sv;
        x = u * cv * cr - u * sv * sr + g.gcx;
        y = u * cv * sr + u * sv * cr + g.gcy;
        double q[3];
        quadric_d(g.type, g.a, g.b, g.c, x, y, z, q);
        if (g.type == 3) {
            nx = 0; ny = 0; nz = g.nfac;
            area = u * duv * dv * kPiD / 180;
        } else {
            const double nrm = sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]);
            nx = g.nfac * q[0] / nrm; ny = g.nfac * q[1] / nrm; nz = g.nfac * q[2] / nrm;
            // |dQ/du x dQ/dv| with Q(u, v) = (x, y, z(x, y))
            const double xu = cv * cr - sv * sr;
            const double xv = cv * cr * dudv - u * sv * cr - sv * sr * dudv - u * cv * sr;
            const double yu = cv * sr + sv * cr;
            const double yv = cv * sr * dudv - u * sv * sr + sv * cr * dudv + u * cv * cr;
            double zx, zy;
            slope_d(g.type, g.a, g.b, g.c, x, y, z, zx, zy);
            const double zu = zx * xu + zy * yu, zv = zx * xv + zy * yv;
            const double cx = yu * zv - zu * yv, cy = zu * xv - xu * zv, cz = xu * yv - yu * xv;
            area = sqrt(cx * cx + cy * cy + cz * cz) * duv * dv * kPiD / 180;
        }
    } else {
        const double dA = (g.lxu1 - g.lxu0) / (g.ncx - 1), dE = (g.lyv1 - g.lyv0) / (g.ncy - 1);
        const double az = i * dA + g.lxu0, el = j * dE + g.lyv0;
        x = az; y = el; z = 0; nx = 0; ny = 0; nz = 1;
        if (g.spheric) {
            x = sqrt(az * az + el * el) * kPiD / 180;
            y = atan2(el, az);
            if (y != y) y = 0;
        }
        area = cos(el * kPiD / 180) * dA * dE * kPiD * kPiD / 180 / 180;
    }
    if (g.transform) {
        const double p[3] = {x, y, z}, q[3] = {nx, ny, nz};
        double po[3], qo[3];
        for (int r = 0; r < 3; ++r) {
            po[r] = g.m[r * 4] * p[0] + g.m[r * 4 + 1] * p[1] + g.m[r * 4 + 2] * p[2] + g.m[r * 4 + 3];
            qo[r] = g.m[r * 4] * q[0] + g.m[r * 4 + 1] * q[1] + g.m[r * 4 + 2] * q[2];
        }
        x = po[0]; y = po[1]; z = po[2];
        nx = qo[0]; ny = qo[1]; nz = qo[2];
    }
    out[idx] = x;
    out[n + idx] = y;
    out[2 * n + idx] = z;
    out[3 * n + idx] = nx;
    out[4 * n + idx] = ny;
    out[5 * n + idx] = nz;
    out[6 * n + idx] = area;
}

int generate_grid_dev(const reflparams &r, double *out7, bool transform, bool spheric, cudaStream_t s)
{
    if (!r.n_cells || r.n_cells[0] < 1 || r.n_cells[1] < 1) return fail(1, "bad n_cells");
    if (!out7) return fail(1, "null output buffer");
    if (r.gmode < 0 || r.gmode > 2) return fail(1, "gmode must be 0 (xy), 1 (uv) or 2 (AoE)");
    if (!r.coeffs || !r.lxu || !r.lyv || !r.gcenter || (transform && !r.transf)) return fail(1, "null reflparams array");
    GridSpec g{};
    g.type = r.type;
    g.gmode = r.gmode;
    g.ncx = r.n_cells[0];
    g.ncy = r.n_cells[1];
    g.nfac = r.flip ? -1 : 1;
    g.spheric = spheric ? 1 : 0;
    g.transform = transform ? 1 : 0;
    g.a = r.coeffs[0];
    g.b = r.coeffs[1];
    g.c = r.coeffs[2];
    g.lxu0 = r.lxu[0];
    g.lxu1 = r.lxu[1];
    g.lyv0 = r.lyv[0];
    g.lyv1 = r.lyv[1];
    g.gcx = r.gcenter[0];
    g.gcy = r.gcenter[1];
    g.ecc = r.ecc_uv;
    g.rot = r.rot_uv;
    if (transform)
        for (int q = 0; q < 12; ++q) g.m[q] = r.transf[q];
    const long n = (long)g.ncx * g.ncy;
    const unsigned nblk = (unsigned)((n + 255) / 256);
    po_grid_kernel<<<nblk, 256, 0, s>>>(g, out7);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(2, std::string("grid kernel launch: ") + cudaGetErrorString(e));
    note_launches(1);
    if (r.rms > 0) {
        int *err = error_word();
        if (!err) return fail(2, "could not allocate the device error word");
        return normal_deviates_dev((unsigned)r.rms_seed, n, r.rms, nullptr, out7, err, s);
    }
    return 0;
}

// ------------------------------------------------- mt19937 normal deviates
//
// MT19937 (Matsumoto and Nishimura, 1998) and the reference's draw of one
// normal deviate per fresh distribution: a double in [0, 1) from two
// outputs, low word first, (w0 + w1 2^32) 2^-64 (at most the double below 1);
// Marsaglia's polar method, x, y = 2U - 1 until 0 < r2 = x^2 + y^2 <= 1, then
// y sqrt(-2 ln r2 / r2) stdev, the other deviate of the pair dropped. So each
// attempt takes four outputs, and a block of 624 outputs is exactly 156
// attempts, of which pi / 4 are accepted.
//
// Only the twist is a serial chain: one CTA writes the generator's words, then
// all SMs count the accepted attempts and write their deviates in order. (One
// CTA for all of it waited 13 us per block, most of it for the FP64 logarithm,
// division and root: 2,070 deviates 174 us, now 22; 200,000 21.1 ms, now 0.39.)

namespace {

constexpr int kMtN = 624;
constexpr int kMtThreads = 256;          // the twist's CTA: 227 threads work
constexpr long kMtRound = 4096;          // blocks of words kept at a time (10 MB)
constexpr int kMtAttempts = 256;         // attempts per CTA
// CTAs from which a kernel of its own counts the accepted attempts: 121 deviates
// (2 CTAs) take 5 us less without it, 289 (4 CTAs, whose attempts one CTA would
// try one after the other) 4 us more.
constexpr unsigned kMtCountFrom = 3;

__device__ __forceinline__ uint32_t mt_twist(uint32_t cur, uint32_t next, uint32_t tap)
{
    const uint32_t y = (cur & 0x80000000u) | (next & 0x7fffffffu);
    return tap ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}

__device__ __forceinline__ double mt_canonical(uint32_t w0, uint32_t w1)
{
    const double u = __dmul_rn(__dadd_rn((double)w0, __dmul_rn((double)w1, 4294967296.0)), 0x1p-64);
    return u < 1.0 ? u : 1.0 - 0x1p-53;
}

__device__ __forceinline__ uint32_t mt_temper(uint32_t w)
{
    w ^= w >> 11;
    w ^= (w << 7) & 0x9d2c5680u;
    w ^= (w << 15) & 0xefc60000u;
    return w ^ (w >> 18);
}

// Attempt a of the round: accepted or not; y and r2 of the polar method.
__device__ __forceinline__ bool mt_attempt(const uint4 *words, long a, long n, double &y, double &r2)
{
    if (a >= n) return false;
    const uint4 w = words[a];
    const double x = __dsub_rn(__dmul_rn(2.0, mt_canonical(mt_temper(w.x), mt_temper(w.y))), 1.0);
    y = __dsub_rn(__dmul_rn(2.0, mt_canonical(mt_temper(w.z), mt_temper(w.w))), 1.0);
    r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
    return r2 <= 1.0 && r2 != 0.0;
}

}  // namespace

// nblk blocks of the generator's words, before tempering; state: the words of
// the last block, where a later round goes on (start: from the seed, and the
// deviates' count *start is cleared). Word i
// of a block needs the old words i and i + 1 and the word 227 before it (the
// old word i + 397 where there is none), so thread t has t, t + 227 and t + 454
// in one go, and two buffers need one barrier a block.
__global__ void __launch_bounds__(kMtThreads)
po_mt_words_kernel(unsigned seed, long long *__restrict__ start, long nblk, uint32_t *__restrict__ state,
                   uint32_t *__restrict__ words)
{
    __shared__ uint32_t mt[2][kMtN];
    const int t = threadIdx.x;
    if (!start) {
        for (int i = t; i < kMtN; i += kMtThreads) mt[0][i] = state[i];
    } else if (t == 0) {
        *start = 0;
        uint32_t v = seed;
        mt[0][0] = v;
        for (int i = 1; i < kMtN; ++i) {
            v = 1812433253u * (v ^ (v >> 30)) + (uint32_t)i;
            mt[0][i] = v;
        }
    }
    __syncthreads();
    for (long b = 0; b < nblk; ++b) {
        const uint32_t *cur = mt[b & 1];
        uint32_t *nxt = mt[1 - (b & 1)], *out = words + b * kMtN;
        if (t < 227) {
            const uint32_t v0 = mt_twist(cur[t], cur[t + 1], cur[t + 397]);
            const uint32_t v1 = mt_twist(cur[t + 227], cur[t + 228], v0);
            nxt[t] = v0;
            nxt[t + 227] = v1;
            out[t] = v0;
            out[t + 227] = v1;
            if (t < 170) {
                // the last word's successor is the new word 0
                const uint32_t next = t < 169 ? cur[t + 455] : mt_twist(cur[0], cur[1], cur[397]);
                const uint32_t v2 = mt_twist(cur[t + 454], next, v1);
                nxt[t + 454] = v2;
                out[t + 454] = v2;
            }
        }
        __syncthreads();
    }
    for (int i = t; i < kMtN; i += kMtThreads) state[i] = mt[nblk & 1][i];
}

// Accepted attempts of each CTA's kMtAttempts.
__global__ void __launch_bounds__(kMtAttempts)
po_mt_count_kernel(const uint4 *__restrict__ words, long na, int *__restrict__ count)
{
    double y, r2;
    const int c = __syncthreads_count(mt_attempt(words, (long)blockIdx.x * kMtAttempts + threadIdx.x, na, y, r2));
    if (threadIdx.x == 0) count[blockIdx.x] = c;
}

// The accepted attempts' deviates, in order, from where the rounds before
// ended (base[0]; the last CTA leaves the new end in base[1] and, at the last
// round, reports deviates that are missing). Without counts (a few CTAs) each
// CTA counts the attempts before its own itself. Deviate i goes into out[i] or,
// with g7 (7 rows of n), moves point i along its normal.
__global__ void __launch_bounds__(kMtAttempts)
po_mt_emit_kernel(const uint4 *__restrict__ words, long na, const int *__restrict__ count, long long *__restrict__ base,
                  int last, long n, double stdev, double *__restrict__ out, double *__restrict__ g7,
                  int *__restrict__ err)
{
    __shared__ unsigned long long before;
    __shared__ int warp_ok[kMtAttempts / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double y, r2;
    const bool ok = mt_attempt(words, (long)blockIdx.x * kMtAttempts + t, na, y, r2);
    const unsigned ball = __ballot_sync(0xffffffffu, ok);
    if (t == 0) before = (unsigned long long)base[0];
    if (lane == 0) warp_ok[warp] = __popc(ball);
    __syncthreads();
    unsigned long long mine = 0;
    if (count)
        for (int c = t; c < (int)blockIdx.x; c += kMtAttempts) mine += (unsigned)count[c];
    else
        for (int c = 0; c < (int)blockIdx.x; ++c) {
            double u, v;
            mine += mt_attempt(words, (long)c * kMtAttempts + t, na, u, v);
        }
    if (mine) atomicAdd(&before, mine);
    __syncthreads();
    long at = (long)before + __popc(ball & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) at += warp_ok[w];
    if (ok && at < n) {
        const double d = __dmul_rn(__dmul_rn(y, __dsqrt_rn(__ddiv_rn(__dmul_rn(-2.0, log(r2)), r2))), stdev);
        if (g7)
            for (int c = 0; c < 3; ++c) g7[c * n + at] += d * g7[(3 + c) * n + at];
        else
            out[at] = d;
    }
    if (blockIdx.x == gridDim.x - 1 && t == kMtAttempts - 1) {
        const long end = at + ok;
        base[1] = end;
        if (last && end < n) atomicExch(err, kErrRngBound);
    }
}

int normal_deviates_dev(unsigned seed, long n, double stdev, double *out, double *g7, int *err, cudaStream_t s)
{
    if (n <= 0) return 0;
    // attempts for n deviates at pi / 4 a piece, with 12 standard deviations to
    // spare: the bound is never met in practice
    const double need = n / 0.78539816339744831;
    const long blocks = (long)((need + 12.0 * sqrt(0.27 * need) + 200.0) / (kMtN / 4)) + 1;
    const long most = std::min(blocks, kMtRound), na = most * (kMtN / 4);
    uint32_t *words = nullptr, *state = nullptr;
    int *count = nullptr;
    long long *base = nullptr;
    const long ctas = (na + kMtAttempts - 1) / kMtAttempts, rounds = (blocks + kMtRound - 1) / kMtRound;
    int rc = 0;
    if (!(rc = scratch_alloc(reinterpret_cast<void **>(&words), sizeof(uint32_t) * kMtN * (most + 1) +
                             sizeof(long long) * (rounds + 1) + sizeof(int) * ctas, s))) {
        // words first (16-byte aligned), then the state, the bases, the counts
        state = words + kMtN * most;
        base = reinterpret_cast<long long *>(state + kMtN);
        count = reinterpret_cast<int *>(base + rounds + 1);
        cudaError_t e = cudaSuccess;
        for (long r = 0; r < rounds && e == cudaSuccess; ++r) {
            const long nb = std::min(kMtRound, blocks - r * kMtRound), a = nb * (kMtN / 4);
            const unsigned grid = (unsigned)((a + kMtAttempts - 1) / kMtAttempts);
            const uint4 *w4 = reinterpret_cast<const uint4 *>(words);
            const bool counts = grid >= kMtCountFrom;
            po_mt_words_kernel<<<1, kMtThreads, 0, s>>>(seed, r == 0 ? base : nullptr, nb, state, words);
            if (counts) po_mt_count_kernel<<<grid, kMtAttempts, 0, s>>>(w4, a, count);
            po_mt_emit_kernel<<<grid, kMtAttempts, 0, s>>>(w4, a, counts ? count : nullptr, base + r, r == rounds - 1, n, stdev,
                                                          out, g7, err);
            e = cudaGetLastError();
            if (e == cudaSuccess) note_launches(counts ? 3 : 2);
        }
        if (e != cudaSuccess) rc = fail(2, std::string("normal deviates: ") + cudaGetErrorString(e));
    }
    scratch_free(words, s);
    return rc;
}

// ------------------------------------------------- correlated surface error

// The cosines' phases and values are 64-bit integers: this device's FP64 unit
// takes 16 clocks of an SM per warp operation, the 32 of a cos() with its
// argument 512 clocks, where a hundred integer operations take some 25.
//
// Phase, in units of 2^-64 turns (mod 1 by wrapping): with x = X 2^(ex - 62)
// and k_x / 2 pi = K 2^(ek - 62), X and K rounded to integers, the exact
// 128-bit sum of the two products is shifted down by 60 - ek - ex. Against
// the FP64 argument (three roundings of 53 bits) its error is 2^(ex + ek - 61)
// turns. Cosine: table values C, S at the nearest of 1024 points, and the
// remainder A (|A| <= pi / 1024) by the addition theorem,
//   cos = C - S sin A - C (1 - cos A),
// with Taylor's sin A = A (1 - A^2/6 + A^4/120), 1 - cos A = A^2/2 - A^4/24
// (the next terms are below 2^-59). The terms are rounded once, to 2^-55, and
// summed exactly. Errors of the sum of 700 modes (against 113-bit arithmetic,
// 60 points each, correlation length 30): 8 10^-15 at 50 and at 300 from the
// origin (FP64 cos: 5 and 8 10^-14), 6 10^-14 at 10^5 (10^-11).

constexpr int kCosN = 1024;          // table points per turn
constexpr int kCorrModes = 256;      // modes per stage
constexpr int kCorrPoints = 32;      // points per CTA; 256 / kCorrPoints threads share a point's modes
constexpr long long kTwoOverPi63 = 0x517cc1b727220a95ll;   // 2 / pi, 2^-63
constexpr long long kTwoPi60 = 0x6487ed5110b4611all;       // 2 pi, 2^-60

// e with |x| < 2^e (at least -1022; above 1023 for infinities and NaN).
__device__ __forceinline__ int above_exponent(double x) { return ((__double2hiint(x) >> 20) & 0x7ff) - 1022; }

// v / 2 pi 2^(62 - e) for |v| < 2^(e + 2), to the nearest integer
__device__ __forceinline__ long long turns62(double v, int e)
{
    const __int128 p = (__int128)__double2ll_rn(scalbn(v, 60 - e)) * kTwoOverPi63;
    return (long long)((p + ((__int128)1 << 62)) >> 63);
}

// cos(2 pi ph 2^-64) 2^62 + 2^6, in about 2^-54: tab[i] = (cos 2^62 + 2^6, sin 2^62) of i / kCosN turns.
__device__ __forceinline__ long long cos_turns62(unsigned long long ph, const longlong2 *tab)
{
    const unsigned i = ((unsigned)(ph >> 32) + (1u << 21)) >> 22;
    const longlong2 cs = tab[i & (kCosN - 1)];
    const long long d = (long long)(ph - ((unsigned long long)i << 54));   // |d| <= 2^53
    const long long A = __mul64hi((long long)((unsigned long long)d << 10), kTwoPi60);   // A 2^70
    const long long q = __mul64hi(A << 1, A << 1);                                       // A^2 2^78
    const unsigned q2 = (unsigned)(q >> 30);                                             // A^2 2^48
    const unsigned q4 = __umulhi(q2, q2);                                                // A^4 2^64
    const unsigned w = __umulhi(q2, 2863311531u) - __umulhi(q4, 2185u);                  // (A^2/6 - A^4/120) 2^50
    const long long sn = A - (((long long)(int)(A >> 32) * (int)w) >> 18);               // sin A 2^70
    const long long v = q - (long long)(((unsigned long long)q4 * 87381u) >> 6);         // (1 - cos A) 2^79
    return cs.x - (__mul64hi(sn, cs.y) >> 6) - (__mul64hi(v, cs.x) >> 15);
}

// Modes of the synthesis from four standard normal deviates each:
// (kx, ky) = (g0, g1) / corr_len, phase atan2(g2, g3). And the cosine table.
__global__ void po_modes_kernel(int m, const double *__restrict__ g, double inv_len, double *__restrict__ modes,
                                longlong2 *__restrict__ tab)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kCosN) {
        double s, c;
        sincospi(2.0 * i / kCosN, &s, &c);
        tab[i] = make_longlong2(__double2ll_rn(c * 0x1p62) + 64, __double2ll_rn(s * 0x1p62));
    }
    if (i >= m) return;
    modes[i] = g[4 * i] * inv_len;
    modes[m + i] = g[4 * i + 1] * inv_len;
    modes[2 * m + i] = atan2(g[4 * i + 2], g[4 * i + 3]);
}

// delta_i = scale sum_m cos(kx_m x_i + ky_m y_i + ph_m), the modes staged
// through shared memory kCorrModes at a time; with `apply`, the point also
// moves by delta_i along its normal. A point's modes are shared by the
// threads l, l + kCorrPoints, ... of the CTA (warps of one kind: the modes are
// broadcast), whose FP64 sums are added in that order: few points still fill
// the chip, and many are spread evenly. A thread whose products are outside the
// integers' range (phases of 2^28 turns and more, infinities) takes cos().
// 90,601 points x 512 modes: 2.46 ms with FP64 cos and a thread a point, 0.30
// now; 10^6 points 21.2 and 3.2; 1,000 points 0.80 and 0.04. 32 points a CTA: 64
// 2 % faster at 10^6 and 2 % slower at 90,601, 256 23 % slower there.
__global__ void __launch_bounds__(256)
po_correlated_kernel(long n, double *__restrict__ g7, int m, const double *__restrict__ modes,
                     const longlong2 *__restrict__ tab, double scale, double *__restrict__ delta, int apply)
{
    constexpr int G = 256 / kCorrPoints, PER = kCorrModes / G;
    __shared__ longlong2 st[kCosN];
    __shared__ longlong2 sk[kCorrModes];            // k_x, k_y
    __shared__ unsigned long long sp[kCorrModes];   // phase
    __shared__ int se;
    __shared__ double part[G][kCorrPoints];
    const int l = threadIdx.x % kCorrPoints, grp = threadIdx.x / kCorrPoints;
    const long i = (long)blockIdx.x * kCorrPoints + l;
    for (int q = threadIdx.x; q < kCosN; q += 256) st[q] = tab[q];
    const double x = i < n ? g7[i] : 0.0, y = i < n ? g7[n + i] : 0.0;
    const int epoint = max(above_exponent(x), above_exponent(y));
    double sum = 0.0;
    for (int c = 0; c < m; c += kCorrModes) {
        const int cnt = min(kCorrModes, m - c), j = threadIdx.x;
        const bool have = j < cnt;
        const double kx = have ? modes[c + j] : 0.0, ky = have ? modes[m + c + j] : 0.0;
        const double kp = have ? modes[2 * m + c + j] : 0.0;
        __syncthreads();
        if (j == 0) se = -4000;
        __syncthreads();
        if (have) atomicMax(&se, max(above_exponent(kx), above_exponent(ky)) - 2);
        __syncthreads();
        const int ek = se;   // |k| / 2 pi < 2^ek
        if (have && ek < 1000) {
            sk[j] = make_longlong2(turns62(kx, ek), turns62(ky, ek));
            // |ph| < 4: ph 2^64 / 2 pi, mod 2^64
            sp[j] = (unsigned long long)(((__int128)__double2ll_rn(kp * 0x1p60) * kTwoOverPi63) >> 61);
        }
        __syncthreads();
        const int j0 = grp * PER, j1 = min(cnt, j0 + PER);
        const int ex = max(epoint, -3 - ek), sh = 60 - ek - ex - 32;   // the shift, less a word
        if (ek < 1000 && sh >= 0) {
            const long long X = __double2ll_rn(scalbn(x, 62 - ex)), Y = __double2ll_rn(scalbn(y, 62 - ex));
            long long acc = 0;   // 2^-55
            for (int q = j0; q < j1; ++q) {
                const longlong2 k = sk[q];
                const __int128 p = (__int128)X * k.x + (__int128)Y * k.y;
                const unsigned w1 = (unsigned)(p >> 32), w2 = (unsigned)(p >> 64), w3 = (unsigned)(p >> 96);
                const unsigned long long t =
                    ((unsigned long long)__funnelshift_r(w2, w3, sh) << 32) | __funnelshift_r(w1, w2, sh);
                acc += cos_turns62(t + sp[q], st) >> 7;
            }
            sum += (double)acc * 0x1p-55;
        } else {
            for (int q = c + j0; q < c + j1; ++q) sum += cos(modes[q] * x + modes[m + q] * y + modes[2 * m + q]);
        }
    }
    part[grp][l] = sum;
    __syncthreads();
    if (grp > 0 || i >= n) return;
    for (int q = 1; q < G; ++q) sum += part[q][l];
    const double d = scale * sum;
    if (delta) delta[i] = d;
    if (apply) {
        g7[i] += d * g7[3 * n + i];
        g7[n + i] += d * g7[4 * n + i];
        g7[2 * n + i] += d * g7[5 * n + i];
    }
}

int correlated_error_dev(long n, double *g7, double rms, double corr_len, unsigned seed, int n_modes, double *delta,
                         int apply, cudaStream_t s)
{
    if (n < 0 || n_modes < 1 || !(corr_len > 0.0) || !(rms >= 0.0)) return fail(1, "bad surface-error arguments");
    if (n > 0 && !g7) return fail(1, "null grid");
    if (n == 0) return 0;
    int *err = error_word();
    if (!err) return fail(2, "could not allocate the device error word");
    double *g = nullptr, *modes = nullptr;
    longlong2 *tab = nullptr;
    int rc = 0;
    if ((rc = scratch_alloc(reinterpret_cast<void **>(&g), sizeof(double) * 4 * n_modes, s)) ||
        (rc = scratch_alloc(reinterpret_cast<void **>(&modes), sizeof(double) * 3 * n_modes, s)) ||
        (rc = scratch_alloc(reinterpret_cast<void **>(&tab), sizeof(longlong2) * kCosN, s))) {
        scratch_free(g, s);
        scratch_free(modes, s);
        return rc;
    }
    rc = normal_deviates_dev(seed, 4L * n_modes, 1.0, g, nullptr, err, s);
    if (!rc) {
        po_modes_kernel<<<(std::max(n_modes, kCosN) + 127) / 128, 128, 0, s>>>(n_modes, g, 1.0 / corr_len, modes, tab);
        po_correlated_kernel<<<(unsigned)((n + kCorrPoints - 1) / kCorrPoints), 256, 0, s>>>(
            n, g7, n_modes, modes, tab, rms * sqrt(2.0 / n_modes), delta, apply);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = fail(2, std::string("surface error: ") + cudaGetErrorString(e));
        else note_launches(2);
    }
    scratch_free(g, s);
    scratch_free(modes, s);
    scratch_free(tab, s);
    return rc;
}

}  // namespace po
