// po_kernels.cuh -- constants and kernel handles shared by the PO kernels and
// their host launcher.
#pragma once
#include <cstdint>

namespace po {

// Propagation modes (numbering of the reference's GpropagateBeam_0..5).
enum Mode { kJM = 0, kEH = 1, kJMEH = 2, kEHP = 3, kFF = 4, kScalar = 5 };

// Kernel families.
constexpr int kKindNF = 0;      // near field (JM, EH, JMEH, EHP)
constexpr int kKindFF = 1;      // far field
constexpr int kKindScalar = 2;  // scalar Green's function

// Mixed-precision N-body kernel geometry (the PO_* macros exist for tuning
// sweeps; the defaults are the shipped configuration).
#ifndef PO_THREADS
#define PO_THREADS 128
#endif
#ifndef PO_TILE
#define PO_TILE 128
#endif
#ifndef PO_MINB
#define PO_MINB 1
#endif
#ifndef PO_THREADS_A
#define PO_THREADS_A 128
#endif
constexpr int kThreads = PO_THREADS;   // threads per CTA
constexpr int kTile = PO_TILE;         // sources per shared-memory stage
constexpr int kMinBlocks = PO_MINB;    // resident CTAs per SM asked of ptxas
// The near-field and scalar forward: resident CTAs per SM asked of ptxas and
// records per iteration. Near field, M = 0, dish to focal plane 251,001 x
// 90,601, ms: 66.98 at 4 CTAs and 3 records (1 record 67.51, 2 67.43, 4 67.30;
// 3 CTAs 67.4-68.2, 5 CTAs 67.1-68.0, 6 68.9). With M, 40,602 x 10,100: 2.039
// at 5 and 4 (1 record 2.084, 3 2.056; 4 CTAs 2.047-2.089). Scalar, same size:
// 0.443 with 4 records (1 0.478, 2 0.452, 3 0.441; 10,403 x 14,399 0.173,
// 0.199, 0.177, 0.177).
// FEW: a grid that leaves an SM two CTAs or fewer has nothing to hide a warp's
// latencies but its own instructions, so the near field then takes eight
// records at a time and the registers that this needs (156): 1,023 x 899 with M
// 35.8 -> 34.0 us, M = 0 1 to 4 % (at four CTAs an SM up to 30 % slower).
__host__ __device__ constexpr int pk_min_blocks(int kind, bool has_m, bool few)
{
    return kind == kKindScalar || few ? 1 : (has_m ? 5 : 4);
}
__host__ __device__ constexpr int pk_unroll(int kind, bool has_m, bool few)
{
    return few ? 8 : (kind == kKindNF && !has_m ? 3 : 4);
}
#ifndef PO_STAGES
#define PO_STAGES 3
#endif
constexpr int kStages = PO_STAGES;     // TMA pipeline depth
constexpr int kRec = 6;         // float4 per packed source record (96 B)
constexpr int kAcc = 12;        // accumulators per target (E, H re/im x y z)
constexpr int kBoxF = 8;        // floats per source-tile box (lit-tile proof)
#ifndef PO_MUFU_SINCOS
#define PO_MUFU_SINCOS 1         // 0: the polynomial sin/cos (accuracy comparisons)
#endif
constexpr uint32_t kWaitLimit = 1u << 24;   // bounded mbarrier polls

// Adjoint kernels: one source (or target) per thread; 12 current
// accumulators + 1 displacement accumulator.
constexpr int kThreadsA = PO_THREADS_A;
#ifndef PO_UNROLL_A
#define PO_UNROLL_A 1            // target pairs per iteration of the adjoint pair loop
#endif
#ifndef PO_PAIRS_A
#define PO_PAIRS_A 32            // target pairs per stage of the pair-packed adjoint
#endif
#ifndef PO_MINB_A2
// Resident CTAs per SM asked of ptxas for the pair-packed adjoint: 3 holds the
// fused near-field kernel at 150-165 registers with no spills (182 at 2), and
// dish_eh's adjoint measured 208.6 -> 206.1 ms with it.
#define PO_MINB_A2 3
#endif
constexpr int kMinBlocksA2 = PO_MINB_A2;
#ifndef PO_MINB_A2M
// The same with magnetic source currents: 2 (feed -> dish JM adjoint
// 1.394 -> 1.348 ms against 3).
#define PO_MINB_A2M 2
#endif
constexpr int kMinBlocksA2M = PO_MINB_A2M;
// Without the currents' gradient (120 and 140 registers needed). 40,000
// sources x 20,000 targets, both displacement gradients, ms: 4.73 at 4 blocks
// without M (4.83 at 3, 4.80 at 5), 6.61 at 3 with M (6.71 at 2 and at 4).
constexpr int kMinBlocksA2N = 4, kMinBlocksA2MN = 3;
constexpr int kMinBlocksFA = 6, kMinBlocksFAM = 4;   // resident CTAs per SM asked of ptxas (M = 0, with M)
constexpr int kStagesFA = 2;
constexpr int kFFDirs = 64;   // directions per stage of the far-field adjoint
// The far-field forward without magnetic currents, two pair records an
// iteration at 5 CTAs/SM: 105.1 ms on 1,002,001 x 160,801 (one record 112.3;
// at 4 CTAs/SM 109.7 with one, 111.7 with two, 109.4 with four).
// FEW (at most two CTAs an SM), as in the near field: eight pair records an
// iteration, 2,652 x 1,722 61.2 -> 58.9 us.
__host__ __device__ constexpr int ff0_min_blocks(bool few) { return few ? 1 : 5; }
__host__ __device__ constexpr int ff0_unroll(bool few) { return few ? 8 : 2; }
constexpr int kUnrollA = PO_UNROLL_A;   // target pairs per iteration of the adjoint pair loop
constexpr int kAccAdj = 13;   // the pair formulas' accumulators: 12 of the currents, 1 of the displacement
// Of those, the ones that a call's kernels keep, as rows of the partials: the
// currents' (c; the scalar kind has two, E.x re and im) where that gradient is
// wanted, then the source displacement's (d). adj_row: accumulator a's row, or -1.
__host__ __device__ constexpr int adj_rows(int kind, bool c, bool d)
{
    return (c ? (kind == kKindScalar ? 2 : 12) : 0) + (d ? 1 : 0);
}
__host__ __device__ constexpr int adj_row(int kind, bool c, bool d, int a)
{
    if (a == 12) return d ? adj_rows(kind, c, false) : -1;
    if (!c) return -1;
    if (kind != kKindScalar) return a;
    return a == 0 ? 0 : (a == 3 ? 1 : -1);
}

// Plain FP64 kernels (po_fp64.cu).
constexpr int kThreadsD = 128;
constexpr int kTileD = 64;
// Granularity of a chunk of the streamed axis: 16 lets a few hundred points
// fill the GPU (13 x 13 -> 5 x 5 forward and adjoint 0.45 ms; 0.61 with 32,
// 0.78 with 64) and even the SMs' loads (101 x 99 -> 41 x 43: 12.6 ms).
constexpr int kChunkD = 16;
constexpr int kRecD = 18;       // x y z nx ny nz, J' 6, M' 6 (doubles)
// Doubles per source record (scalar: point, normal, S'; M = 0: no M') and
// per target record of the adjoint.
__host__ __device__ constexpr int fp64_rec(int kind, bool has_m) { return kind == kKindScalar ? 8 : (has_m ? kRecD : 12); }
__host__ __device__ constexpr int adj64_rec(int kind) { return kind == kKindScalar ? 8 : (kind == kKindFF ? 18 : 22); }
// The wave as the FP64 kernels take it: k, 1/k and the sign bit of t.
struct Wave64 {
    double k, inv_k;
    unsigned neg;
};
Wave64 wave64(double k, double t);

// The frame kernel: one thread-block cluster (16 is the most a cluster may
// have, past the portable 8). Past kFrameClusterMax points, and where a context's
// share of the device cannot hold the cluster, the box comes from a CTA an SM and
// the frame from a second kernel. A call of n sources and 25 targets, cluster /
// two kernels, in us: 4,000 28.6 / 29.5, 48,000 54.8 / 55.3, 64,000 67.8 / 67.8,
// 161,202 126.2 / 122.1, 1,002,001 600 / 554.
constexpr int kFrameThreads = 512;
constexpr int kFrameCtas = 16;
constexpr long kFrameClusterMax = 60000;

// Illumination test of the mixed-precision kernels: a pair with
// n . R_hat >= kTangentBand is lit, one below -kTangentBand is not (the FP32
// test's own error is below 4.2e-7). A pair inside the band is left out of
// the FP32 sums and listed; a fixup kernel then decides it with the
// reference's FP64 rounding, as the FP64 kernels decide every pair, and adds
// its FP64 term if it is lit. The lit-tile proofs keep a margin of 1e-5.
constexpr float kTangentBand = 1e-6f;

// The list of pairs inside the band: (source, target) entries, their count
// (zeroed before the main kernel) and the capacity; a count above the
// capacity is reported as kErrBandOverflow by the fixup.
struct BandList {
    int2 *pairs;
    unsigned *count;
    unsigned cap;
};
constexpr unsigned kBandCap = 1u << 22;        // entries, calls on the library's pool: every pair up
                                               // to this many, else at least this many
constexpr unsigned kBandCapMax = 1u << 24;     // ... and at most (one entry per 2^16 pairs between)
constexpr unsigned kBandCapStatic = 1u << 14;  // entries, the allocation-free entry

// Band-list entries of a call on the library's pool with ns x nt pairs: a
// call of up to 2^22 pairs can list all of them (targets in the sources'
// own plane put every pair in the band); larger calls one per 2^16 pairs.
inline unsigned band_cap_for(long ns, long nt)
{
    const double pairs = (double)ns * (double)nt;
    if (pairs <= (double)kBandCap) return pairs < 1.0 ? 1u : (unsigned)pairs;
    const double want = pairs / 65536.0;
    return want <= kBandCap ? kBandCap : (want >= kBandCapMax ? kBandCapMax : (unsigned)want);
}
constexpr unsigned kFixupBlocks = 152;         // grid of the fixup kernels (grid-stride over the list)

// Device error codes (written to the call's error word).
constexpr int kErrWaitTimeout = 101;
constexpr int kErrRngBound = 102;   // the device normal generator ran past its bound (never expected)
constexpr int kErrBandOverflow = 103;   // more near-tangent pairs than the band list holds

// Frame of the split representation: positions in turns (mm * kappa),
// relative to origin o, hi parts on multiples of q.
struct Frame {
    double o[3];
    double kappa;
    double q;
    double inv_q;
    double m;   // half-extent in wavelengths (turns), which sets q and the precision
    double lo[3], hi[3];   // the points' box (mm), from which the far field orders its sources
};

// Far-field forward (po_farfield.cu): sources in tiles of kTile along a
// Hilbert curve, each tile a 64-byte header and kTile / 2 pair records of
// ff_rec4 float4 (offset from the tile centre, J', normal, the offset's lo
// part in a wide tile, M').
constexpr int kFFHead = 4;
__host__ __device__ constexpr int ff_rec4(bool has_m) { return has_m ? 11 : 8; }
// Tiles up to this radius (turns) take the per-pair phase in plain FP32;
// wider ones (sparse sampling) split their offsets into hi + lo. At 64 turns
// the FP32 phase leaves about 2e-6 relative L2 error on a sum of random
// (incoherent) currents, the worst case (FP32 emulation on a 501 x 501 dish
// of 2000 wavelengths), and 1.2 % of that dish's tiles are wide; the full
// 1001 x 1001 configuration has 0.1 %.
constexpr float kFFNarrow = 64.0f;
__host__ __device__ constexpr int ff_tile4(bool has_m) { return kFFHead + (kTile / 2) * ff_rec4(has_m); }
int ff_smem_bytes(bool has_m);
// Up to this many sources the far field's order comes from ff_rank_kernel, past
// it from the radix sort: calls with 41 x 40 directions, sort / rank, in us:
// 2,652 sources 132 / 60, 8,190 152 / 86, 14,520 179 / 133, 19,740 194 / 187,
// 22,650 204 / 207, 32,580 229 / 313.
constexpr long kFFRankMax = 20000;
void *ff_key_kernel();
void *ff_rank_kernel();
void *ff_pack_kernel(bool has_m);
void *ff_kernel(int t_sign, bool has_m, bool few);

// Source tiles of the near-field and scalar forward (layout in po_kernels.cu):
// float4 ahead of the records, per record, and of a tile of n sources.
__host__ __device__ constexpr int pk_head(int kind, bool has_m) { return kind != kKindScalar && !has_m ? kBoxF / 4 : 0; }
__host__ __device__ constexpr int pk_rec4(int kind, bool has_m) { return kind == kKindScalar ? 2 : (has_m ? 5 : 4); }
__host__ __device__ constexpr int pk_tile4(int kind, bool has_m, int n)
{
    return pk_head(kind, has_m) + n * pk_rec4(kind, has_m) + (kind != kKindScalar && has_m ? (n + 3) / 4 : 0);
}

// Stages, the halves' exchange and the compensation words.
inline int pk_smem_bytes(int kind, bool has_m)
{
    const int na = kind == kKindScalar ? 1 : kAcc / 2;
    return kStages * pk_tile4(kind, has_m, kTile) * 16 + 2 * na * kThreads * 8;
}

void *pk_kernel(int kind, int t_sign, bool has_m, bool few);
void *pack_kernel(bool scalar, bool has_m);   // source tiles (near field, scalar) and targets
void *fp64_kernel(int kind, bool has_m);
void *frame_kernel();
void *box_kernel();
void *box_frame_kernel();   // 192 threads
void *pack_src_d_kernel();
constexpr int kEpiThreads = 256;
void *epilogue_kernel(int groups);   // 1, 8, 32 or 64 threads share a target's chunks
void *f2d_kernel();   // float -> double, grid-stride over n
void *d2f_kernel();   // double -> float
void *fp32_probe_kernel();
void *band_fixup_kernel(int kind, bool has_m);
void *adj_band_fixup_kernel(int kind, bool want_t);
void *wait_selftest_kernel();
void *adj_fp64_kernel(int kind, bool has_m, bool want_c, bool want_d, bool want_t);
void *adj_tsum_kernel();
void *adj_pack_tgt_d_kernel(int kind);
void *adj_cot_kernel();
void *adj_pack_kernel();                 // near field, scalar: sources, targets and cotangents
void *adj_epilogue_kernel(int groups, int rows);   // 1 or 8 threads share a source's chunks of `rows` rows
void *adj_ehp_cot_kernel();
// Far-field adjoint (po_ff_adjoint.cu): stages of kFFDirs packed directions.
void *ff_pack_cot_kernel();
void *ff_adj_kernel(int t_sign, bool has_m, bool want_c, bool want_d);
int ff_adj_smem_bytes(bool want_c, bool want_d);
int ff_adj_threads();
int ff_adj_stage4();   // float4 per stage
// Pair-packed adjoint, near field and scalar, fused: currents, source and
// target displacement.
void *adj_pk_kernel(int kind, int t_sign, bool has_m, bool want_c, bool want_d, bool want_t);
int adj_pk_smem_bytes(int kind, bool has_m, bool want_c, bool want_d, bool want_t);
int adj_pk_pairs_per_tile();
int adj_pk_rec4(bool has_m, bool want_t);   // float4 per pair-packed cotangent record

}  // namespace po
