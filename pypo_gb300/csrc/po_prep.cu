// po_prep.cu -- set-up kernels of the mixed-precision paths: the frame of the
// split representation, and the packed records of sources and targets.
//
// A small propagation is bound by its launches (2.1 us each on the device,
// and as much per stream-ordered allocation), so its set-up is two kernels:
// the frame in one thread-block cluster (no partial buffer, no second
// launch), and one pack kernel for the source records, their tile boxes and
// the targets. Many points take their box from all SMs, in one kernel more.
// Each later kernel of a call is launched with programmatic
// stream serialisation and begins with pdl_wait().
#include <cuda_runtime.h>
#include <math_constants.h>

#include <cstdint>

#include "po_device.cuh"
#include "po_kernels.cuh"

namespace po {

namespace {

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Store into the shared memory of cluster rank `rank` at this CTA's address p.
__device__ __forceinline__ void st_cluster(long long *p, uint32_t rank, long long v)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.s64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

// Smallest power of two q >= need, at least 2^-40 (need NaN: 2^-40; need
// infinite or past the largest power of two: infinity).
__device__ __forceinline__ double quantum(double need)
{
    const double least = 0x1p-40;
    if (!(need > least)) return least;
    const long long bits = __double_as_longlong(need);
    const long long e = bits >> 52;   // need > 2^-40: positive and normal
    return __longlong_as_double(((bits & 0xfffffffffffffll) ? e + 1 : e) << 52);
}

// The box of the points of a (na) and b (nb; rows x, y, z first) that the CTAs
// first, first + step, ... of THREADS threads take, THREADS points at a time: thread
// q < 6 returns lowest x, y, z, highest x, y, z as order keys (NaN coordinates
// are left out). wbox: shared.
template <int THREADS>
__device__ __forceinline__ long long cta_box(const double *__restrict__ a, long na, const double *__restrict__ b,
                                             long nb, long first, long step, long long (*wbox)[THREADS / 32])
{
    long long v[6] = {kKeyInf, kKeyInf, kKeyInf, ~kKeyInf, ~kKeyInf, ~kKeyInf};
    auto scan = [&](const double *__restrict__ p, long n) {
#pragma unroll 4
        for (long i = first * THREADS + threadIdx.x; i < n; i += step * THREADS)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long x = __double_as_longlong(p[c * n + i]), y = order_key(x);
                const bool nan = (x & 0x7fffffffffffffffll) > kKeyInf;
                v[c] = nan ? v[c] : min(v[c], y);
                v[3 + c] = nan ? v[3 + c] : max(v[3 + c], y);
            }
    };
    scan(a, na);
    scan(b, nb);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const long long u = __shfl_xor_sync(0xffffffffu, v[q], o);
            v[q] = q < 3 ? min(v[q], u) : max(v[q], u);
        }
        if ((threadIdx.x & 31) == 0) wbox[q][threadIdx.x >> 5] = v[q];
    }
    __syncthreads();
    long long r = 0;
    if (threadIdx.x < 6) {
        const int q = threadIdx.x;
        r = wbox[q][0];
        for (int w = 1; w < THREADS / 32; ++w) r = q < 3 ? min(r, wbox[q][w]) : max(r, wbox[q][w]);
    }
    return r;
}

// The frame of the box k (order keys: lowest x, y, z, highest x, y, z).
__device__ __forceinline__ void write_frame(const long long *k, double kappa, int centred, Frame *fr)
{
    double m = 0.0;
    for (int c = 0; c < 3; ++c) {
        const double lo = __longlong_as_double(order_key(k[c])), hi = __longlong_as_double(order_key(k[3 + c]));
        double o = 0.0;
        if (centred && lo <= hi) o = 0.5 * (lo + hi);
        fr->o[c] = o;
        if (lo <= hi) m = fmax(m, fmax(fabs(hi - o), fabs(lo - o)));
        fr->lo[c] = lo;
        fr->hi[c] = hi;
    }
    m *= kappa;
    // 2 m / q <= 2048, so |hi/q| <= 1024.5
    const double q = quantum(2.0 * m / 2048.0);
    fr->kappa = kappa;
    fr->q = q;
    fr->inv_q = 1.0 / q;
    fr->m = m;
}

}  // namespace

// Box of the points of a (na) and b (nb; rows x, y, z first), and from it the
// frame: origin, scale and quantum. One cluster of kFrameCtas CTAs: minima and
// maxima are exact in any order, so the split does not show in the result.
// centred: origin at the box centre (near field, scalar); otherwise origin 0
// (far field: the phase reference is the coordinate origin). zero: a word
// cleared for the call's later kernels (the band list's count), or null.
__global__ void __launch_bounds__(kFrameThreads) __cluster_dims__(kFrameCtas, 1, 1)
po_frame_kernel(const double *__restrict__ a, long na, const double *__restrict__ b, long nb, double kappa,
                int centred, Frame *__restrict__ fr, unsigned *__restrict__ zero)
{
    __shared__ long long box[6][kFrameCtas];   // rank 0's copy gathers the cluster's
    __shared__ long long wbox[6][kFrameThreads / 32];
    pdl_trigger();
    cluster_arrive();   // completed below: every CTA has started before one writes into rank 0's memory
    const uint32_t rank = cluster_rank();
    if (rank == 0 && threadIdx.x == 0 && zero) *zero = 0u;
    const long long r = cta_box<kFrameThreads>(a, na, b, nb, rank, kFrameCtas, wbox);
    cluster_wait();
    if (threadIdx.x < 6) st_cluster(&box[threadIdx.x][rank], 0, r);
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (rank != 0 || threadIdx.x != 0) return;
    long long k[6];
    for (int q = 0; q < 6; ++q) {
        k[q] = box[q][0];
        for (int c = 1; c < kFrameCtas; ++c) k[q] = q < 3 ? min(k[q], box[q][c]) : max(k[q], box[q][c]);
    }
    write_frame(k, kappa, centred, fr);
}

// The same in two kernels, for many points and for devices that cannot hold the
// cluster: the boxes of gridDim.x CTAs, then the frame of their box.
__global__ void __launch_bounds__(kFrameThreads)
po_box_kernel(const double *__restrict__ a, long na, const double *__restrict__ b, long nb,
              long long *__restrict__ boxes)
{
    __shared__ long long wbox[6][kFrameThreads / 32];
    const long long r = cta_box<kFrameThreads>(a, na, b, nb, blockIdx.x, gridDim.x, wbox);
    if (threadIdx.x < 6) boxes[6L * blockIdx.x + threadIdx.x] = r;
    pdl_trigger();
}

__global__ void __launch_bounds__(192)
po_box_frame_kernel(const long long *boxes, int n, double kappa, int centred, Frame *__restrict__ fr,
                    unsigned *__restrict__ zero)
{
    __shared__ long long k[6];
    pdl_wait();
    pdl_trigger();
    // warp q: word q of the boxes
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long long v = q < 3 ? kKeyInf : ~kKeyInf;
    for (int i = lane; i < n; i += 32) {
        const long long u = boxes[6L * i + q];
        v = q < 3 ? min(v, u) : max(v, u);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long u = __shfl_xor_sync(0xffffffffu, v, o);
        v = q < 3 ? min(v, u) : max(v, u);
    }
    if (lane == 0) k[q] = v;
    __syncthreads();
    if (threadIdx.x > 0) return;
    if (zero) *zero = 0u;
    write_frame(k, kappa, centred, fr);
}

// Packed target i. Near field / scalar: hi/lo split position in the frame.
// Far field: direction r_hat from (polar, azimuth), hi part on 2^-11.
__device__ __forceinline__ void pack_target(long i, long nt, const double *tgt7, const Frame &fr, int far, float4 *out)
{
    float h[3], l[3];
    if (far) {
        const double th = tgt7[i], ph = tgt7[nt + i];
        const double r[3] = {cos(ph) * sin(th), sin(ph) * sin(th), cos(th)};
        for (int c = 0; c < 3; ++c) {
            const double hd = rint(r[c] * 2048.0) / 2048.0;
            h[c] = (float)hd;
            l[c] = (float)(r[c] - hd);
        }
    } else {
        for (int c = 0; c < 3; ++c) split_hi_lo((tgt7[c * nt + i] - fr.o[c]) * fr.kappa, fr, h[c], l[c]);
    }
    out[2 * i] = make_float4(h[0], h[1], h[2], l[0]);
    out[2 * i + 1] = make_float4(l[1], l[2], 0.f, 0.f);
}

// Blocks 0 .. tiles-1: one tile of kTile sources each (layout in
// po_kernels.cu), assembled in shared memory and written out in coalesced
// float4. Near field, M = 0: the tile's box for the lit-tile proof goes ahead
// of the records: lowest normal xyz, highest normal xyz, largest n.s, largest
// |s|_1 (s = hi + lo, turns).
// The remaining blocks: kTile targets each. far: no source tiles here (the
// far field packs them in curve order), and the targets are directions.
template <bool SCALAR, bool HAS_M>
__global__ void __launch_bounds__(kTile)
po_pack_kernel(long ns, const double *__restrict__ src7, const double *__restrict__ cur, int gmode, int ncx, int ncy,
               const Frame *frp, double fac_re, double fac_im, long tiles,
               float4 *__restrict__ src, long nt, const double *__restrict__ tgt7, int far, float4 *__restrict__ tgt)
{
    constexpr int KIND = SCALAR ? kKindScalar : kKindNF;
    constexpr int HEAD = pk_head(KIND, HAS_M), R4 = pk_rec4(KIND, HAS_M), T4 = pk_tile4(KIND, HAS_M, kTile);
    __shared__ __align__(16) float4 buf[T4];
    __shared__ float wbox[kTile / 32][kBoxF];
    pdl_wait();
    const Frame fr = *frp;
    if ((long)blockIdx.x >= tiles) {
        const long i = ((long)blockIdx.x - tiles) * kTile + threadIdx.x;
        if (i < nt) pack_target(i, nt, tgt7, fr, far, tgt);
        pdl_trigger();
        return;
    }
    const long first = (long)blockIdx.x * kTile, i = first + threadIdx.x;
    const int n = (int)min((long)kTile, ns - first);   // sources of this tile
    const bool real = (int)threadIdx.x < n;
    float v[4 * R4 + 1];
    if (real) {
        for (int c = 0; c < 3; ++c) split_hi_lo((src7[c * ns + i] - fr.o[c]) * fr.kappa, fr, v[c], v[3 + c]);
        const double w = trap_weight(i, gmode, ncx, ncy) * src7[6 * ns + i];
        const double fr_ = fac_re * w, fi_ = fac_im * w;
        if (SCALAR) {
            const double re = cur[i], im = cur[ns + i];
            v[6] = (float)(fr_ * re - fi_ * im);
            v[7] = (float)(fr_ * im + fi_ * re);
        } else {
            for (int c = 0; c < 3; ++c) v[6 + c] = (float)src7[(3 + c) * ns + i];
#pragma unroll
            for (int q = 0; q < (HAS_M ? 6 : 3); ++q) {
                const int grp = q / 3, ax = q % 3;
                const double re = cur[(grp * 6 + ax) * ns + i];
                const double im = cur[(grp * 6 + 3 + ax) * ns + i];
                v[9 + 2 * q] = (float)(fr_ * re - fi_ * im);
                v[10 + 2 * q] = (float)(fr_ * im + fi_ * re);
            }
            if (!HAS_M) v[15] = 0.f;
        }
        // even sources first, then the odd ones
        const int pos = (threadIdx.x >> 1) + (threadIdx.x & 1) * ((n + 1) / 2);
#pragma unroll
        for (int q = 0; q < R4; ++q)
            buf[HEAD + pos * R4 + q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        if (!SCALAR && HAS_M) reinterpret_cast<float *>(buf + n * R4)[pos] = v[4 * R4];
    }
    if (!SCALAR && HAS_M && (int)threadIdx.x >= n && (int)threadIdx.x < (n + 3) / 4 * 4)
        reinterpret_cast<float *>(buf + n * R4)[threadIdx.x] = 0.f;
    if (HEAD > 0) {
        float x[kBoxF] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F,
                          -CUDART_INF_F, 0.0f};
        if (real) {
            float s[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                s[c] = v[c] + v[3 + c];
                x[c] = x[3 + c] = v[6 + c];
            }
            x[6] = fmaf(v[8], s[2], fmaf(v[7], s[1], v[6] * s[0]));
            x[7] = fabsf(s[0]) + fabsf(s[1]) + fabsf(s[2]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < kBoxF; ++q) {
                const float u = __shfl_xor_sync(0xffffffffu, x[q], o);
                x[q] = q < 3 ? fminf(x[q], u) : fmaxf(x[q], u);
            }
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int q = 0; q < kBoxF; ++q) wbox[threadIdx.x >> 5][q] = x[q];
        __syncthreads();
        if (threadIdx.x < kBoxF) {
            const int q = threadIdx.x;
            float r = wbox[0][q];
            for (int w = 1; w < kTile / 32; ++w) r = q < 3 ? fminf(r, wbox[w][q]) : fmaxf(r, wbox[w][q]);
            reinterpret_cast<float *>(buf)[q] = r;
        }
    }
    __syncthreads();
    float4 *dst = src + (size_t)blockIdx.x * T4;
    for (int q = threadIdx.x; q < pk_tile4(KIND, HAS_M, n); q += kTile) dst[q] = buf[q];
    pdl_trigger();
}

void *frame_kernel() { return reinterpret_cast<void *>(&po_frame_kernel); }
void *box_kernel() { return reinterpret_cast<void *>(&po_box_kernel); }
void *box_frame_kernel() { return reinterpret_cast<void *>(&po_box_frame_kernel); }

void *pack_kernel(bool scalar, bool has_m)
{
    if (scalar) return reinterpret_cast<void *>(&po_pack_kernel<true, false>);
    return has_m ? reinterpret_cast<void *>(&po_pack_kernel<false, true>)
                 : reinterpret_cast<void *>(&po_pack_kernel<false, false>);
}

}  // namespace po
