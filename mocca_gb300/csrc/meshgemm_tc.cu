// meshgemm_tc.cu -- the mesh-sized contractions on the tcgen05 tensor cores
// (exact BF16 digit products, ozaki.cuh), in the mixed form with six digits and
// in the FP64 form with eight: the Gram-Schmidt overlap and apply, the
// canonical-basis transform and the contractions of the pairing field and gaps.
//
// Blocks of up to kMeshTcMax (80) spinors in the mixed form, kMeshTcMin64 to
// kMeshTcMax64 (24 to 64) in the FP64 form, whose results are rounded once to FP64
// (norm-wise errors of the Gram-Schmidt of blocks of 22 to 50, mean over the spinors:
// 1.27e-16 to 1.49e-16, with FP64 FMAs 1.31e-16 to 1.59e-16).
//
// Gram-Schmidt (gs.cu; GramSchmidt, src/SpwfStorage.f90:372-480, as
// Q = Psi R^{-1} with S = R^T R per (isospin, parity, signature) block in
// energy order):
//   k_gs_overlap_tc : S partial sums over chunks of 256 points (128).  Rows of
//                     the MMA are the block's spinors, K the chunk's points; A
//                     and B are the same digit planes.  Each (spinor, chunk) row
//                     gets its own power of two.  The partials go to the same
//                     kind of table as the FP64 kernel's, so k_gs_sum /
//                     k_gs_factor (gs.cu) finish the job.
// Block apply, out_l(p) = sum_k C[k][l] in_k(p) per block of spinors:
//   k_coef_digits   : digit planes of C (rows: output l, K: input k), one
//                     power of two per row;
//   k_apply_tc      : tiles of 128 points (MMA M), K = the block's spinors, FP64
//                     output.  Gram-Schmidt: C = R^{-1}, in place, plus the
//                     GradDesc history upd_l = out_l - upd_l.  Canonical basis
//                     (HFBOccupations, src/HFB.f90:3448-3487): C = CanTransfo,
//                     HF basis in, canonical basis out.
// A chunk keeps the digit weights of the overlap that have an accumulator of their own
// within 2^24 (at most 3 pairs x 256 points x 2^14, in the FP64 form 8 x 128), so their
// FP32 sums are exact.
#include <algorithm>
#include <vector>

#include "df.cuh"
#include "mg_internal.cuh"
#include "ozaki.cuh"
#include "tc.cuh"

namespace mg {

namespace {

using oz::kDigits;
constexpr int kRows = 128;            // MMA M
constexpr int kChunk = 256;           // overlap points per CTA
constexpr int kStage = 32;            // overlap points per MMA stage (K)
constexpr long kXdStride = (long)kMeshTcMax * kMeshTcMax;   // per block in the coefficient planes
constexpr long long kWaitCycles = 4000000000LL;

// Block sizes and list offsets: Gram-Schmidt blocks come from a start table,
// pairing blocks have hsz[b] members listed at b * hmax.
struct BlockIdx {
    const int* starts;
    const int* hsz;
    int hmax;
    __device__ int nb(int b) const { return starts ? starts[b + 1] - starts[b] : hsz[b]; }
    __device__ int off(int b) const { return starts ? starts[b] : b * hmax; }
};

__device__ __forceinline__ double pow2d(int x) {
    return x < -1022 ? 0.0 : __longlong_as_double((long long)(min(x, 1023) + 1023) << 52);
}

// Sum over a chunk of points of psi_k psi_l for the pairs k <= l of a block, or of
// psi_k z_l for all pairs (kTwo), to part.
//
// A unit is a chunk of one block, 256 points in the mixed form, 128 in the FP64 form
// (what keeps the sums of a weight exact).  One CTA per SM takes a run of units with
// the roles of k_apply_tc: the slicers cut stages of kStage points into a ring of
// plane buffers, one thread issues a stage's MMAs, the epilogue writes a unit's sums
// while the next unit's stages go on.  A's rows are the planes' own, one after the
// other, so that the planes are B's stacked columns too, behind the planes of zeros that
// the stack begins with; what A reads past a plane's NP rows gives rows of D that
// nothing reads.  Bound by the latency of the slicers' loads (160 spwfs of 24^3: a
// quarter of the issue slots used, the tensor pipe active 27% in the mixed form, 40% in
// the FP64 form).  300 spwfs of 36^3 (blocks of 75, 38 MMAs a stage of 32 points) 572
// us, 834 with a CTA per chunk; the FP64 form for 160 of 24^3 (40, 24 MMAs) 150, 512
// by FP64 FMAs.
constexpr int kRoleWarps = 8;                       // epilogue: warps 0-7, slicers: 8-15
constexpr int kRoleThreads = 2 * kRoleWarps * 32 + 32;   // and the MMA warp
constexpr int kSmemCap = 225 * 1024;
constexpr int kNone = 255;

__host__ __device__ constexpr int accs_for(int nd) { return nd == oz::kDigits64 ? oz::kAccs64 : (int)oz::kAccs; }
__host__ __device__ constexpr int chunk_for(int nd) { return nd == oz::kDigits64 ? 128 : kChunk; }
__host__ __device__ constexpr int tbufs_for(int nd, int np) { return 2 * accs_for(nd) * np <= 512 ? 2 : 1; }
// A stage's planes: of two operands A's, zeros, B's; of one zeros and the planes of both.
__host__ __device__ constexpr int overlap_a(int nd, int np, bool two) {
    return two ? 0 : oz::stack_zeros(nd, np);
}
__host__ __device__ constexpr int overlap_b(int nd, int np, bool two) {
    return (two ? nd : 0) + oz::stack_zeros(nd, np);
}
__host__ __device__ constexpr int overlap_stage(int nd, int np, bool two) {
    return (overlap_b(nd, np, two) + nd) * np * kStage * 2;
}
// A's reads past its last plane: of two operands they end in the planes behind it
__host__ __device__ constexpr int overlap_tail(bool two) { return two ? 0 : kRows * kStage * 2; }
__host__ __device__ constexpr int overlap_bufs(int nd, int np, bool two) {
    // (8 KB left for the kernels' static shared memory)
    const int n = (kSmemCap - 8192 - 128 - overlap_tail(two)) / overlap_stage(nd, np, two);
    return n >= 6 ? 6 : n;
}
// (more than half of an SM's, so that no second CTA comes beside one that holds all
// TMEM columns and waits for them)
constexpr size_t kOneCtaSmem = 116 * 1024;
__host__ __device__ constexpr size_t one_cta(size_t bytes) {
    return bytes > kOneCtaSmem ? bytes : kOneCtaSmem;
}
__host__ __device__ constexpr size_t overlap_smem(int nd, int np, bool two) {
    return one_cta((size_t)overlap_bufs(nd, np, two) * overlap_stage(nd, np, two) +
                   overlap_tail(two) + 128);
}

__device__ __forceinline__ bool wait_warp(uint64_t* mbar, uint32_t parity) {
    return __all_sync(0xffffffffu, tc::mbar_wait(mbar, parity, kWaitCycles)) != 0;
}
__device__ __forceinline__ void arrive_warp(uint64_t* mbar, int lane) {
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(mbar);
}

// psi_k = psi[list[off + k]], z_l = z[b nbmax + l]; part[chunk of b][k ldo + l].
template <int ND, int NP, bool kTwo>
__global__ void __launch_bounds__(kRoleThreads, 1)
k_gs_overlap_tc(const double* __restrict__ psi, const double* __restrict__ z, BlockIdx bi,
                const int* __restrict__ list, int nbmax, long V4, int nchunk, int nunits,
                double* __restrict__ part, int* __restrict__ status) {
    constexpr int NACC = accs_for(ND), NBUF = overlap_bufs(ND, NP, kTwo), NTB = tbufs_for(ND, NP);
    constexpr int CH = chunk_for(ND), kPlane = NP * kStage * 2, kBuf = overlap_stage(ND, NP, kTwo);
    constexpr int kArr = kTwo ? 2 : 1;
    constexpr int kA = overlap_a(ND, NP, kTwo) * kPlane, kB = overlap_b(ND, NP, kTwo) * kPlane;
    static_assert(!kTwo || kBuf >= (ND - 1) * kPlane + kRows * kStage * 2, "A's reads past its planes");
    constexpr int kPasses = (NP + 63) / 64;   // rows of a slicer: row0, row0 + 64
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t full[6], empty[6], fullT[2], emptyT[2], expReady[8];
    __shared__ uint32_t tmem_slot;
    __shared__ int sE[8][kArr * NP];   // of the last units
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t s0a = tc::smem_u32(smraw);
    uint8_t* base = smraw + ((128u - (s0a & 127u)) & 127u);
    for (int t = tid; t < (NBUF * kBuf + overlap_tail(kTwo)) / 16; t += kRoleThreads)
        reinterpret_cast<uint4*>(base)[t] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) tc::alloc(&tmem_slot, 512u);
    if (tid == 0) {
        for (int q = 0; q < NBUF; ++q) {
            tc::mbar_init(&full[q], kRoleWarps);
            tc::mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            tc::mbar_init(&fullT[q], 1);
            tc::mbar_init(&emptyT[q], kRoleWarps);
        }
        for (int q = 0; q < 8; ++q) tc::mbar_init(&expReady[q], kRoleWarps);
    }
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_slot;
    const int u0 = (int)((long)nunits * blockIdx.x / gridDim.x);
    const int u1 = (int)((long)nunits * (blockIdx.x + 1) / gridDim.x);
    bool ok = true;
    // units of empty blocks are passed over by every role
    const auto stages_of = [&](int unit, int& b, int& s0, int& nb, long& p0, int& npts) {
        b = unit / nchunk;
        s0 = bi.off(b);
        nb = bi.nb(b);
        p0 = (long)(unit - b * nchunk) * CH;
        npts = (int)min((long)CH, V4 - p0);
        return nb > 0 ? (npts + kStage - 1) / kStage : 0;
    };
    int b, s0, nb, npts;
    long p0;
    if (warp >= kRoleWarps && warp < 2 * kRoleWarps) {
        // ---------------- slicers ----------------
        // a row's 4 K groups sit on 4 neighbouring lanes
        const int st = tid - 32 * kRoleWarps, row0 = st >> 2, g = st & 3;
        int stage = 0;   // stages of this CTA so far
        for (int unit = u0, k = 0; unit < u1 && ok; ++unit) {
            const int nst = stages_of(unit, b, s0, nb, p0, npts);
            if (nst == 0) continue;
            const double* src[kArr][kPasses];
            int emax[kArr][kPasses];
#pragma unroll
            for (int y = 0; y < kArr; ++y)
#pragma unroll
                for (int r = 0; r < kPasses; ++r) {
                    const int row = row0 + 64 * r;
                    src[y][r] = row >= nb ? nullptr
                                : y == 0  ? psi + (long)list[s0 + row] * V4 + p0
                                          : z + ((long)b * nbmax + row) * V4 + p0;
                    int e = 0;
                    if (src[y][r])
                        for (int s = 0; s < nst; ++s) {
#pragma unroll
                            for (int h = 0; h < 8; ++h) {
                                const int q = s * kStage + 8 * g + h;
                                if (q < npts) e = max(e, oz::bexp(src[y][r][q]));
                            }
                        }
                    e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
                    emax[y][r] = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
                }
            // (the epilogue of unit k - 8 has read its slot: the ring's stages and the
            // accumulators let the slicers run at most five units ahead)
#pragma unroll
            for (int y = 0; y < kArr; ++y)
#pragma unroll
                for (int r = 0; r < kPasses; ++r)
                    if (src[y][r] && g == 0) sE[k & 7][y * NP + row0 + 64 * r] = emax[y][r];
            arrive_warp(&expReady[k & 7], lane);
            ++k;
            for (int s = 0; s < nst; ++s, ++stage) {
                const int buf = stage % NBUF;
                uint8_t* planes = base + buf * kBuf;
#pragma unroll
                for (int y = 0; y < kArr; ++y) {
                    double v[kPasses][8];
#pragma unroll
                    for (int r = 0; r < kPasses; ++r)
#pragma unroll
                        for (int h = 0; h < 8; ++h) {
                            const int q = s * kStage + 8 * g + h;
                            v[r][h] = src[y][r] && q < npts ? src[y][r][q] : 0.0;
                        }
                    if (y == 0 && stage >= NBUF) {
                        ok = wait_warp(&empty[buf], ((stage - NBUF) / NBUF) & 1);
                        if (!ok) break;
                    }
#pragma unroll
                    for (int r = 0; r < kPasses; ++r) {
                        const int row = row0 + 64 * r;
                        if (row >= NP) continue;
                        const oz::FixedRow<ND> fixed(emax[y][r]);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const double v4[4] = {v[r][4 * h], v[r][4 * h + 1], v[r][4 * h + 2],
                                                  v[r][4 * h + 3]};
                            uint2 w[ND];
                            oz::digits4<ND>(v4, fixed, w);
#pragma unroll
                            for (int a = 0; a < ND; ++a)
                                *reinterpret_cast<uint2*>(planes + (y == 0 ? kA : kB) + a * kPlane +
                                                          tc::kmajor_off(row, 8 * g + 4 * h)) = w[a];
                        }
                    }
                }
                if (!ok) break;
                tc::fence_proxy_async();
                arrive_warp(&full[buf], lane);
            }
        }
    } else if (warp == 2 * kRoleWarps) {
        // ---------------- MMA issue ----------------
        if (lane == 0) {
            int stage = 0, k = 0;
            for (int unit = u0; unit < u1 && ok; ++unit) {
                const int nst = stages_of(unit, b, s0, nb, p0, npts);
                if (nst == 0) continue;
                const int tb = k % NTB;
                if (k >= NTB) ok = tc::mbar_wait(&emptyT[tb], ((k - NTB) / NTB) & 1, kWaitCycles);
                for (int s = 0; s < nst && ok; ++s, ++stage) {
                    const int buf = stage % NBUF;
                    ok = tc::mbar_wait(&full[buf], (stage / NBUF) & 1, kWaitCycles);
                    if (!ok) break;
                    tc::fence_after();
                    const uint32_t pa = tc::smem_u32(base + buf * kBuf);
                    oz::issue_stacked<ND, NP, kStage / 16>(tmem + (uint32_t)(tb * NACC * NP), pa + kA,
                                                           kPlane, pa + kB, tc::kSbo, s > 0);
                    tc::commit(&empty[buf]);
                }
                if (!ok) break;
                tc::commit(&fullT[tb]);
                ++k;
            }
            // the last commit covers every MMA of this CTA (after a timeout: the
            // buffers' last ones)
            if (k > 0) ok &= tc::mbar_wait(&fullT[(k - 1) % NTB], ((k - 1) / NTB) & 1, kWaitCycles);
            if (!ok && stage > 0)
                tc::mbar_wait(&empty[(stage - 1) % NBUF], ((stage - 1) / NBUF) & 1, kWaitCycles);
        }
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        // D[k][l], k = TMEM lane (row), l = column; warps w and w + 4 share lane quarter w % 4
        const int quarter = warp & 3, colh = warp >> 2, kr = quarter * 32 + lane;
        for (int unit = u0, k = 0; unit < u1; ++unit) {
            const int nst = stages_of(unit, b, s0, nb, p0, npts);
            if (nst == 0) continue;
            const int tb = k % NTB;
            ok = wait_warp(&expReady[k & 7], (k >> 3) & 1);
            if (ok) ok = wait_warp(&fullT[tb], (k / NTB) & 1);
            if (!ok) break;
            tc::fence_after();
            const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) +
                                  (uint32_t)(tb * NACC * NP + 8 * colh);
            double* out = part + (long)unit * nbmax * nbmax;
            const int* se = sE[k & 7] + (kTwo ? NP : 0);   // of the columns
            const int ldo = kTwo ? nb : nbmax;
            const int ek = kr < nb ? sE[k & 7][kr] : 0;
            // rows past the block have nothing to write
            const int nch = quarter * 32 < nb ? (nb - 8 * colh + 15) / 16 : 0;
#pragma unroll 1
            for (int c = 0; c < nch; ++c) {
                const int l0 = 16 * c + 8 * colh;
                uint32_t r[NACC][8];
                __syncwarp();
#pragma unroll
                for (int q = 0; q < NACC; ++q) tc::ld8(trow + (uint32_t)(q * NP + 16 * c), r[q]);
#pragma unroll
                for (int q = 0; q < NACC; ++q) tc::wait_ld(r[q]);
                if (kr >= nb) continue;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int l = l0 + u;
                    if (l >= nb || (!kTwo && l < kr)) continue;
                    double val;
                    if constexpr (ND == oz::kDigits64) {
                        uint32_t acc[NACC];
#pragma unroll
                        for (int q = 0; q < NACC; ++q) acc[q] = r[q][u];
                        val = oz::combine64_any(acc, ek - 1023 + se[l] - 1023 - oz::kUnit64);
                        if (ek == 0 || se[l] == 0) val = 0.0;
                        if (ek == 2047 || se[l] == 2047)
                            val = __longlong_as_double(0x7FF8000000000000ll);
                    } else {
                        const dfl o = oz::combine4(__uint_as_float(r[0][u]), __uint_as_float(r[1][u]),
                                                   __uint_as_float(r[2][u]), __uint_as_float(r[3][u]));
                        val = (f2d_bits(o.h) + f2d_bits(o.l)) * pow2d(ek - 1023 + se[l] - 1023 - 12);
                    }
                    out[kr * ldo + l] = val;
                }
            }
            tc::fence_before();
            arrive_warp(&emptyT[tb], lane);
            ++k;
        }
    }
    ok = __syncthreads_and(ok) != 0;
    if (!ok && tid == 0) tc::report_timeout(status);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::dealloc(tmem_slot, 512u);
}

// Digit planes of C (per block: ND planes of NP rows x NP, row l = output l, K =
// input k; C[k][l] = coef[b * bstride + k * ld + l], ld = nb when 0) and the row
// exponents (biased).  Thread (l, y): entries k = y, y + kCoefRows, ...
constexpr int kCoefRows = 8;

template <int ND, int NP>
__global__ void __launch_bounds__(NP * kCoefRows)
k_coef_digits(const double* __restrict__ coef, long bstride, int ld, BlockIdx bi,
              uint16_t* __restrict__ xd, int* __restrict__ xe) {
    __shared__ int se[kCoefRows][NP];
    const int b = blockIdx.x;
    const int nb = bi.nb(b);
    const int l = threadIdx.x, y = threadIdx.y;
    if (nb == 0) return;
    const int ldc = ld > 0 ? ld : nb;
    const double* X = coef + (long)b * bstride;
    uint16_t* out = xd + (long)b * ND * kXdStride;
    double v[NP / kCoefRows];
    int emax = 0;
#pragma unroll
    for (int q = 0; q < NP / kCoefRows; ++q) {
        const int k = y + q * kCoefRows;
        v[q] = (l < nb && k < nb) ? X[k * ldc + l] : 0.0;
        emax = max(emax, oz::bexp(v[q]));
    }
    se[y][l] = emax;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kCoefRows; ++q) emax = max(emax, se[q][l]);
    if (y == 0) xe[b * kMeshTcMax + l] = emax;
    const oz::FixedRow<ND> fixed(emax);
#pragma unroll
    for (int q = 0; q < NP / kCoefRows; ++q) {
        uint32_t d[ND];
        oz::digits_of<ND>(fixed.biased(v[q]), d);
        const uint32_t o = tc::kmajor_off_g(l, y + q * kCoefRows, NP / 8) / 2;
#pragma unroll
        for (int a = 0; a < ND; ++a) out[(long)a * NP * NP + o] = (uint16_t)(d[a] >> 16);
    }
}

// out_l = sum_k C[k][l] in_k over 128 points (in_k = in[in_list[off + k]],
// out_l = out[out_list[off + l]] or out[out_base[b] + l]); when upd is given,
// upd_l = out_l - upd_l.  in and out may be the same array (in place).
//
// One CTA per SM takes a run of the (block, 128 points) tiles.  Three roles work on
// different tiles at a time: the slicers hold a tile's values (two threads a point)
// and cut them once the planes of the tile before are free, one thread issues the
// MMAs, the epilogue takes the accumulators to registers, gives them back and
// writes.  The integer and FP32 work of cutting and combining bounds it (about 160
// instructions per entry, 55 to 61% of the issue slots at 24^3), the MMAs come next (one of up to
// 192 columns holds the tensor pipe ~130 clocks: 54 of them for a tile of 48
// spinors, 95 for 80).  A CTA per tile went through the same steps one after the
// other: 1628 us for the 300 spwfs of 36^3 (blocks of 75), now 573; 110 for the 160
// of 24^3 (40), now 77.
// Epilogue warps.  Up to 48 spinors a slicer's values leave the registers for sixteen:
// 160 spwfs of 24^3 77 us, FP64 form 102, with eight 87 and 150.  Above them not: 300
// of 36^3 573 us with eight of each, 709 with sixteen slicer warps and eight.
__host__ __device__ constexpr int apply_epilogue(int np) { return np <= 48 ? 16 : 8; }
__host__ __device__ constexpr int apply_threads(int np) { return 32 * (apply_epilogue(np) + kRoleWarps + 1); }
__device__ __forceinline__ void tmem_load(uint32_t t, uint32_t (&r)[4]) { tc::ld4(t, r); }
__device__ __forceinline__ void tmem_load(uint32_t t, uint32_t (&r)[8]) { tc::ld8(t, r); }
__host__ __device__ constexpr int apply_plane(int np) { return kRows * np * 2; }
// the coefficients' planes behind the zeros that their stack begins with
__host__ __device__ constexpr int apply_zeros(int nd, int np) { return oz::stack_zeros(nd, np) * np * np * 2; }
__host__ __device__ constexpr int apply_coef(int nd, int np) { return oz::stack_planes(nd, np) * np * np * 2; }
// operand and accumulator buffers that fit
__host__ __device__ constexpr int apply_bufs(int nd, int np) {
    return 2 * nd * apply_plane(np) + apply_coef(nd, np) + 128 <= kSmemCap ? 2 : 1;
}
__host__ __device__ constexpr size_t apply_smem(int nd, int np) {
    return one_cta((size_t)apply_bufs(nd, np) * nd * apply_plane(np) + apply_coef(nd, np) + 128);
}

template <int ND, int NP, bool kInPlace>
__global__ void __launch_bounds__(apply_threads(NP), 1)
k_apply_tc(const double* in, double* out, double* __restrict__ upd, BlockIdx bi,
           const int* __restrict__ in_list, const int* __restrict__ out_list,
           const int* __restrict__ out_base, const uint16_t* __restrict__ xd,
           const int* __restrict__ xe, const double* __restrict__ coef, long bstride, int ld,
           long V4, int tpb, int ntiles, int* __restrict__ status) {
    constexpr int NACC = accs_for(ND), NBUF = apply_bufs(ND, NP), NTB = tbufs_for(ND, NP);
    constexpr int kg = NP / 8, kPlane = apply_plane(NP), kZeros = apply_zeros(ND, NP);
    constexpr int EW = apply_epilogue(NP);
    static_assert(apply_smem(ND, NP) <= kSmemCap, "operands");
    constexpr int W = 64 / EW;   // columns of an epilogue chunk, 16 / W warps side by side
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t fullA[2], emptyA[2], fullT[2], emptyT[2], emaxReady[4];
    __shared__ uint32_t tmem_slot;
    __shared__ int sEx[2][2 * kRows];          // the two slicers of a point
    __shared__ int sEmax[4][kRows];            // of the last tiles
    __shared__ int sXe[NP], sIdx[NP], sOut[NP];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t s0a = tc::smem_u32(smraw);
    uint8_t* sA = smraw + ((128u - (s0a & 127u)) & 127u);
    uint8_t* sB = sA + NBUF * ND * kPlane;
    if (warp == 0) tc::alloc(&tmem_slot, 512u);
    if (tid == 0) {
        for (int q = 0; q < 2; ++q) {
            tc::mbar_init(&fullA[q], kRoleWarps);
            tc::mbar_init(&emptyA[q], 1);
            tc::mbar_init(&fullT[q], 1);
            tc::mbar_init(&emptyT[q], EW);
        }
        for (int q = 0; q < 4; ++q) tc::mbar_init(&emaxReady[q], kRoleWarps);
    }
    const int t0 = (int)((long)ntiles * blockIdx.x / gridDim.x);
    const int t1 = (int)((long)ntiles * (blockIdx.x + 1) / gridDim.x);
    bool ok = true;
    int k0 = 0;   // tiles of this CTA before the block at hand
    uint32_t tmem = 0;
    for (int ta = t0; ta < t1;) {
        const int b = ta / tpb, te = min(t1, (b + 1) * tpb);
        const int off = bi.off(b), nb = bi.nb(b);
        const long first = (long)(ta - b * tpb) * kRows;
        const int count = nb > 0 ? te - ta : 0;
        ta = te;
        if (count == 0) continue;
        {
            const uint4* src = reinterpret_cast<const uint4*>(xd + (long)b * ND * kXdStride);
            uint4* dst = reinterpret_cast<uint4*>(sB);
            for (int t = tid; t < apply_coef(ND, NP) / 16; t += apply_threads(NP))
                dst[t] = t < kZeros / 16 ? make_uint4(0u, 0u, 0u, 0u) : src[t - kZeros / 16];
            // K groups past the block's spinors stay zero
            uint4* a = reinterpret_cast<uint4*>(sA);
            for (int t = tid; t < NBUF * ND * kPlane / 16; t += apply_threads(NP))
                a[t] = make_uint4(0u, 0u, 0u, 0u);
            if (tid < NP) {
                sXe[tid] = xe[b * kMeshTcMax + tid];
                sIdx[tid] = tid < nb ? in_list[off + tid] : 0;
                sOut[tid] = tid < nb ? (out_list ? out_list[off + tid] : out_base[b] + tid) : 0;
            }
        }
        tc::fence_proxy_async();
        tc::fence_before();
        const bool xbad = __syncthreads_or(tid < NP && xe[b * kMeshTcMax + tid] == 2047) != 0;
        tc::fence_after();
        tmem = tmem_slot;
        if (warp >= EW && warp < EW + kRoleWarps) {
            // ---------------- slicers ----------------
            // thread: point `row`, K groups half, half + 2, ...
            const int st = tid - 32 * EW, row = st & (kRows - 1), half = st >> 7;
            constexpr int own = (kg + 1) / 2;
            // (a warp whose wait has run out stays in the loop: the barrier below counts it)
            for (int q = 0, k = k0; q < count; ++q, ++k) {
                const int buf = k % NBUF;
                const long p = first + (long)q * kRows + row;
                double v[8 * own];
                int emax = 0;
#pragma unroll
                for (int u = 0; u < 8 * own; ++u) {
                    const int kk = 8 * (half + 2 * (u >> 3)) + (u & 7);
                    v[u] = (p < V4 && kk < nb) ? in[(long)sIdx[kk] * V4 + p] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 8 * own; ++u) emax = max(emax, oz::bexp(v[u]));
                int bad = kNone;   // FP64 form: the first spinor with an infinity or a NaN
                if (ND == oz::kDigits64 && emax == 2047) {
                    emax = 0;
#pragma unroll
                    for (int u = 0; u < 8 * own; ++u) {
                        if (oz::bexp(v[u]) == 2047) {
                            bad = min(bad, 8 * (half + 2 * (u >> 3)) + (u & 7));
                            v[u] = 0.0;
                        }
                        emax = max(emax, oz::bexp(v[u]));
                    }
                }
                sEx[k & 1][st] = emax * 256 + bad;
                asm volatile("bar.sync 1, %0;" ::"n"(32 * kRoleWarps) : "memory");
                {
                    const int e0 = sEx[k & 1][row], e1 = sEx[k & 1][row + kRows];
                    emax = max(e0 >> 8, e1 >> 8);
                    bad = min(e0 & 255, e1 & 255);
                }
                if (ok && k >= NBUF) ok = wait_warp(&emptyA[buf], ((k - NBUF) / NBUF) & 1);
                if (!ok) continue;
                if (half == 0) sEmax[k & 3][row] = emax * 256 + bad;
                arrive_warp(&emaxReady[k & 3], lane);
                const oz::FixedRow<ND> fixed(emax);
                uint8_t* planes = sA + buf * ND * kPlane;
#pragma unroll
                for (int gg = 0; gg < own; ++gg) {
                    const int g = half + 2 * gg;
                    if (8 * g >= nb) continue;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const double v4[4] = {v[8 * gg + 4 * h], v[8 * gg + 4 * h + 1],
                                              v[8 * gg + 4 * h + 2], v[8 * gg + 4 * h + 3]};
                        uint2 w[ND];
                        oz::digits4<ND>(v4, fixed, w);
#pragma unroll
                        for (int a = 0; a < ND; ++a)
                            *reinterpret_cast<uint2*>(planes + a * kPlane +
                                                      tc::kmajor_off_g(row, 8 * g + 4 * h, kg)) = w[a];
                    }
                }
                tc::fence_proxy_async();
                arrive_warp(&fullA[buf], lane);
            }
        } else if (warp == EW + kRoleWarps) {
            // ---------------- MMA issue ----------------
            if (lane == 0) {
                int k = k0;
                for (int q = 0; q < count; ++q, ++k) {
                    const int buf = k % NBUF, tb = k % NTB;
                    ok = tc::mbar_wait(&fullA[buf], (k / NBUF) & 1, kWaitCycles);
                    if (ok && k >= NTB)
                        ok = tc::mbar_wait(&emptyT[tb], ((k - NTB) / NTB) & 1, kWaitCycles);
                    if (!ok) break;
                    tc::fence_after();
                    oz::issue_stacked<ND, NP, NP / 16>(
                        tmem + (uint32_t)(tb * NACC * NP), tc::smem_u32(sA + buf * ND * kPlane),
                        kPlane, tc::smem_u32(sB + kZeros), (uint32_t)kg * 128u);
                    tc::commit(&emptyA[buf]);
                    tc::commit(&fullT[tb]);
                }
                // the last commit covers every MMA of this CTA
                if (k > k0) ok &= tc::mbar_wait(&fullT[(k - 1) % NTB], ((k - 1) / NTB) & 1, kWaitCycles);
            }
            __syncwarp();
        } else {
            // ---------------- epilogue ----------------
            // lane: point quarter * 32 + lane of the tile; columns 16 c + W colh + ...
            const int quarter = warp & 3, colh = warp >> 2, erow = quarter * 32 + lane;
            for (int q = 0, k = k0; q < count; ++q, ++k) {
                const int tb = k % NTB;
                const long pe = first + (long)q * kRows + erow;
                ok = wait_warp(&emaxReady[k & 3], (k >> 2) & 1);
                if (ok) ok = wait_warp(&fullT[tb], (k / NTB) & 1);
                if (!ok) break;
                tc::fence_after();
                const int emax = sEmax[k & 3][erow] >> 8, bad = sEmax[k & 3][erow] & 255;
                const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) +
                                      (uint32_t)(tb * NACC * NP + W * colh);
                const int nch = max(0, (nb - W * colh + 15) / 16);
                if (nch == 0) {
                    tc::fence_before();
                    arrive_warp(&emptyT[tb], lane);
                }
#pragma unroll 1
                for (int c = 0; c < nch; ++c) {
                    const int l0 = 16 * c + W * colh;
                    uint32_t r[NACC][W];
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < NACC; ++g) tmem_load(trow + (uint32_t)(g * NP + 16 * c), r[g]);
                    double was[W];
                    if (upd && pe < V4)
#pragma unroll
                        for (int u = 0; u < W; ++u)
                            if (l0 + u < nb) was[u] = upd[(long)sOut[l0 + u] * V4 + pe];
#pragma unroll
                    for (int g = 0; g < NACC; ++g) tc::wait_ld(r[g]);
                    if (c == nch - 1) {
                        // the last accumulators of this tile are in registers
                        tc::fence_before();
                        arrive_warp(&emptyT[tb], lane);
                    }
                    if (pe >= V4) continue;
#pragma unroll
                    for (int u = 0; u < W; ++u) {
                        if (l0 + u >= nb) break;
                        const int ex = sXe[l0 + u];
                        double x = 0.0;
                        if constexpr (ND == oz::kDigits64) {
                            uint32_t acc[NACC];
#pragma unroll
                            for (int g = 0; g < NACC; ++g) acc[g] = r[g][u];
                            const int e = emax - 1023 + ex - 1023 - oz::kUnit64;
                            // 6 pairs x 42 x 2^14 < 2^22: the magic numbers' range (weights
                            // 6 and 7 are taken far below theirs)
                            if (nb <= 42 && e >= -900 && e <= 900)
                                x = oz::combine64(acc, e);
                            else
                                x = oz::combine64_any(acc, e);
                            if (emax == 0 || ex == 0) x = 0.0;
                            // in place C is triangular, and NaN from a spinor with an
                            // infinity or a NaN on (else: below)
                            if (l0 + u >= bad || ex == 2047) x = __longlong_as_double(0x7FF8000000000000ll);
                        } else if (emax > 0) {
                            dfl o = oz::combine4(__uint_as_float(r[0][u]), __uint_as_float(r[1][u]),
                                                 __uint_as_float(r[2][u]), __uint_as_float(r[3][u]));
                            const float sc = oz::pow2f(emax - 1023 + ex - 1023 - 12);
                            o.h = __fmul_rn(o.h, sc);
                            o.l = __fmul_rn(o.l, sc);
                            x = f2d_bits(o.h) + f2d_bits(o.l);
                        }
                        const long o = (long)sOut[l0 + u] * V4 + pe;
                        out[o] = x;
                        if (upd) upd[o] = x - was[u];
                    }
                }
                if (ND == oz::kDigits64 && !kInPlace && pe < V4 && (bad != kNone || xbad))
                    // an infinity or a NaN at this point or in C: the plain sums
                    for (int l = W * colh; l < nb; l += (l & (W - 1)) == W - 1 ? 17 - W : 1) {
                        const double* C = coef + (long)b * bstride + l;
                        double x = 0.0;
#pragma unroll 1
                        for (int q2 = 0; q2 < nb; ++q2)
                            x = fma(C[q2 * (ld > 0 ? ld : nb)], in[(long)sIdx[q2] * V4 + pe], x);
                        out[(long)sOut[l] * V4 + pe] = x;
                    }
            }
        }
        k0 += count;
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;
    }
    if (!ok && tid == 0) tc::report_timeout(status);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::dealloc(tmem_slot, 512u);
}

// Pairing gaps, HFBGaps (src/HFB.f90:520-632), per block b (isospin b / 2):
//   G_ij = sum_p sum_c psi_ic(p) Z_jc(p)  over a 64-point chunk,
//   Z_j0 = -Fr psi_j0 + Fi psi_j1, Z_j1 = -Fi psi_j0 - Fr psi_j1 (same for 2, 3),
// the form of k_pair_gaps (pairing.cu).  K runs over (component, point):
// stage s covers 8 points, K group c = component c.  A rows are the spinors
// (one power of two per spinor and chunk), B rows their Z, formed in
// double-float and cut into digits through the fixed-point form with the
// exponent bound 2 max|F| max|psi_j| of the chunk.  Units, roles and rings as in
// k_gs_overlap_tc.  160 spwfs of 24^3 (blocks of 40): 225 us with a CTA per chunk and
// its stages one after the other, now 178 (298 with eight slicer warps).
constexpr int kGapPts = 64;
constexpr int kGapSlicers = 16;   // forming and cutting Z is most of the work
constexpr int kGapThreads = 32 * (kRoleWarps + kGapSlicers + 1);

template <int NP>
__global__ void __launch_bounds__(kGapThreads, 1)
k_gaps_tc(const double* __restrict__ psi, const int* __restrict__ members,
          const int* __restrict__ hsz, int hmax, const double* __restrict__ fre,
          const double* __restrict__ fim, long V, int nchunk, double* __restrict__ gpart,
          int* __restrict__ status) {
    constexpr int NACC = oz::kAccs, NBUF = overlap_bufs(kDigits, NP, true),
                  NTB = tbufs_for(kDigits, NP);
    constexpr int kPlane = NP * kStage * 2, kBuf = overlap_stage(kDigits, NP, true), nst = kGapPts / 8;
    constexpr int kB = overlap_b(kDigits, NP, true) * kPlane;
    static_assert(kBuf >= (kDigits - 1) * kPlane + kRows * kStage * 2, "A's reads past its planes");
    constexpr int kPasses = (NP + 63) / 64;   // rows of a slicer: row0, row0 + 64
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t full[6], empty[6], fullT[2], emptyT[2], expReady[8];
    __shared__ uint32_t tmem_slot;
    __shared__ int sE[8][2 * NP];      // of the last units: psi, then Z
    __shared__ int sFe[2][kGapPts];
    __shared__ float4 sF[2][kGapPts];  // (Fr hi, Fr lo, Fi hi, Fi lo)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t s0a = tc::smem_u32(smraw);
    uint8_t* base = smraw + ((128u - (s0a & 127u)) & 127u);
    for (int t = tid; t < NBUF * kBuf / 16; t += kGapThreads)
        reinterpret_cast<uint4*>(base)[t] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) tc::alloc(&tmem_slot, 512u);
    if (tid == 0) {
        for (int q = 0; q < NBUF; ++q) {
            tc::mbar_init(&full[q], kGapSlicers);
            tc::mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            tc::mbar_init(&fullT[q], 1);
            tc::mbar_init(&emptyT[q], kRoleWarps);
        }
        for (int q = 0; q < 8; ++q) tc::mbar_init(&expReady[q], kGapSlicers);
    }
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_slot;
    const int nunits = 4 * nchunk;
    const int u0 = (int)((long)nunits * blockIdx.x / gridDim.x);
    const int u1 = (int)((long)nunits * (blockIdx.x + 1) / gridDim.x);
    bool ok = true;
    if (warp >= kRoleWarps && warp < kRoleWarps + kGapSlicers) {
        // ------- slicers: rows row0 and row0 + 64, component c, half of the points -------
        const int st = tid - 32 * kRoleWarps, row0 = st >> 3, c = (st >> 1) & 3, half = st & 1;
        int stage = 0;
        // (a warp whose wait has run out stays in the loop: the barrier below counts it)
        for (int unit = u0, k = 0; unit < u1; ++unit) {
            const int b = unit / nchunk, it = b >> 1, h = hsz[b];
            if (h == 0) continue;
            const long p0 = (long)(unit - b * nchunk) * kGapPts;
            const int npts = (int)min((long)kGapPts, V - p0);
            // the pairing field of the chunk, double-float, and its largest exponent
            if (st < kGapPts) {
                double fr = 0.0, fi = 0.0;
                if (st < npts) {
                    fr = fre[(long)it * V + p0 + st];
                    fi = fim[(long)it * V + p0 + st];
                }
                const dfl a = df_split(fr), d = df_split(fi);
                sF[k & 1][st] = make_float4(a.h, a.l, d.h, d.l);
                sFe[k & 1][st] = max(oz::bexp(fr), oz::bexp(fi));
            }
            const double *src[kPasses], *srp[kPasses];   // psi_c and its partner component
            int emax[kPasses], ez[kPasses];
#pragma unroll
            for (int r = 0; r < kPasses; ++r) {
                const int row = row0 + 64 * r;
                const bool live = row < h;
                const double* p = psi + (long)members[b * hmax + (live ? row : 0)] * 4 * V + p0;
                src[r] = live ? p + c * V : nullptr;
                srp[r] = p + (c ^ 1) * V;
                int e = 0;
                if (live)
#pragma unroll 8
                    for (int q = half; q < npts; q += 2) e = max(e, oz::bexp(src[r][q]));
                e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
                e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
                emax[r] = max(e, __shfl_xor_sync(0xffffffffu, e, 4));
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kGapSlicers) : "memory");
            int efmax = 0;
            for (int q = 0; q < kGapPts; ++q) efmax = max(efmax, sFe[k & 1][q]);
#pragma unroll
            for (int r = 0; r < kPasses; ++r) {
                // |Z| <= |F| (|psi_c| + |psi_c'|) < 2^(E_F + E_psi + 3)
                ez[r] = (emax[r] == 0 || efmax == 0) ? 0 : emax[r] + efmax - 1023 + 2;
                if (src[r] && c == 0 && half == 0) {
                    sE[k & 7][row0 + 64 * r] = emax[r];
                    sE[k & 7][NP + row0 + 64 * r] = ez[r];
                }
            }
            arrive_warp(&expReady[k & 7], lane);
            const float4* F = sF[k & 1];
            ++k;
            for (int s = 0; s < nst && ok; ++s, ++stage) {
                const int buf = stage % NBUF;
                uint8_t* planes = base + buf * kBuf;
                double a[kPasses][4], ap[kPasses][4];
#pragma unroll
                for (int r = 0; r < kPasses; ++r)
#pragma unroll
                    for (int hh = 0; hh < 4; ++hh) {
                        const int q = 8 * s + 4 * half + hh;
                        const bool in = src[r] && q < npts;
                        a[r][hh] = in ? src[r][q] : 0.0;
                        ap[r][hh] = in ? srp[r][q] : 0.0;
                    }
                if (stage >= NBUF) {
                    ok = wait_warp(&empty[buf], ((stage - NBUF) / NBUF) & 1);
                    if (!ok) break;
                }
#pragma unroll
                for (int r = 0; r < kPasses; ++r) {
                    const int row = row0 + 64 * r;
                    if (row >= NP) continue;
                    long long zx[4];
#pragma unroll
                    for (int hh = 0; hh < 4; ++hh) {
                        const float4 f = F[8 * s + 4 * half + hh];
                        const dfl fr = {f.x, f.y}, fi = {f.z, f.w};
                        const dfl ac = df_split(a[r][hh]), ao = df_split(ap[r][hh]);
                        // c even: Z = -Fr a_c + Fi a_c' ; c odd: Z = -Fi a_c' - Fr a_c
                        const dfl t1 = df_mul(fr, ac), t2 = df_mul(fi, ao);
                        const dfl z = (c & 1) ? df_neg(df_add(t1, t2)) : df_sub(t2, t1);
                        zx[hh] = ez[r] ? oz::fixed_f(z.h, ez[r]) + oz::fixed_f(z.l, ez[r]) : 0ll;
                    }
                    uint2 w[kDigits];
                    const uint32_t o = tc::kmajor_off(row, 8 * c + 4 * half);
                    oz::digits4<kDigits>(a[r], oz::FixedRow<kDigits>(emax[r]), w);
#pragma unroll
                    for (int d = 0; d < kDigits; ++d)
                        *reinterpret_cast<uint2*>(planes + d * kPlane + o) = w[d];
                    oz::digits4_fixed(zx, w);
#pragma unroll
                    for (int d = 0; d < kDigits; ++d)
                        *reinterpret_cast<uint2*>(planes + kB + d * kPlane + o) = w[d];
                }
                tc::fence_proxy_async();
                arrive_warp(&full[buf], lane);
            }
        }
    } else if (warp == kRoleWarps + kGapSlicers) {
        // ---------------- MMA issue ----------------
        if (lane == 0) {
            int stage = 0, k = 0;
            for (int unit = u0; unit < u1 && ok; ++unit) {
                if (hsz[unit / nchunk] == 0) continue;
                const int tb = k % NTB;
                if (k >= NTB) ok = tc::mbar_wait(&emptyT[tb], ((k - NTB) / NTB) & 1, kWaitCycles);
                for (int s = 0; s < nst && ok; ++s, ++stage) {
                    const int buf = stage % NBUF;
                    ok = tc::mbar_wait(&full[buf], (stage / NBUF) & 1, kWaitCycles);
                    if (!ok) break;
                    tc::fence_after();
                    const uint32_t pa = tc::smem_u32(base + buf * kBuf);
                    oz::issue_stacked<kDigits, NP, kStage / 16>(
                        tmem + (uint32_t)(tb * NACC * NP), pa, kPlane, pa + kB, tc::kSbo, s > 0);
                    tc::commit(&empty[buf]);
                }
                if (!ok) break;
                tc::commit(&fullT[tb]);
                ++k;
            }
            // the last commit covers every MMA of this CTA (after a timeout: the
            // buffers' last ones)
            if (k > 0) ok &= tc::mbar_wait(&fullT[(k - 1) % NTB], ((k - 1) / NTB) & 1, kWaitCycles);
            if (!ok && stage > 0)
                tc::mbar_wait(&empty[(stage - 1) % NBUF], ((stage - 1) / NBUF) & 1, kWaitCycles);
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: G[i][j], i = TMEM lane, j = column ----------------
        const int quarter = warp & 3, colh = warp >> 2, i = quarter * 32 + lane;
        for (int unit = u0, k = 0; unit < u1; ++unit) {
            const int h = hsz[unit / nchunk];
            if (h == 0) continue;
            const int tb = k % NTB;
            ok = wait_warp(&expReady[k & 7], (k >> 3) & 1);
            if (ok) ok = wait_warp(&fullT[tb], (k / NTB) & 1);
            if (!ok) break;
            tc::fence_after();
            const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) +
                                  (uint32_t)(tb * NACC * NP + 8 * colh);
            double* out = gpart + (long)unit * hmax * hmax;
            const int ei = i < h ? sE[k & 7][i] : 0;
            const int* sz = sE[k & 7] + NP;
            const int nch = quarter * 32 < h ? (h - 8 * colh + 15) / 16 : 0;
#pragma unroll 1
            for (int c = 0; c < nch; ++c) {
                const int l0 = 16 * c + 8 * colh;
                uint32_t r[NACC][8];
                __syncwarp();
#pragma unroll
                for (int q = 0; q < NACC; ++q) tc::ld8(trow + (uint32_t)(q * NP + 16 * c), r[q]);
#pragma unroll
                for (int q = 0; q < NACC; ++q) tc::wait_ld(r[q]);
                if (i >= h) continue;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int j = l0 + u;
                    if (j >= h) break;
                    double val = 0.0;
                    if (ei != 0 && sz[j] != 0) {
                        const dfl o = oz::combine4(__uint_as_float(r[0][u]), __uint_as_float(r[1][u]),
                                                   __uint_as_float(r[2][u]), __uint_as_float(r[3][u]));
                        val = (f2d_bits(o.h) + f2d_bits(o.l)) * pow2d(ei - 1023 + sz[j] - 1023 - 12);
                    }
                    out[i * h + j] = val;
                }
            }
            tc::fence_before();
            arrive_warp(&emptyT[tb], lane);
            ++k;
        }
    }
    ok = __syncthreads_and(ok) != 0;
    if (!ok && tid == 0) tc::report_timeout(status);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::dealloc(tmem_slot, 512u);
}

// Chunk partials of the gaps summed per entry, one warp each (fixed order):
// gsum[b][i * h + j].
__global__ void k_gaps_sum(const double* __restrict__ gpart, const int* __restrict__ hsz,
                           int hmax, int nchunk, double* __restrict__ gsum) {
    const int b = blockIdx.y;
    const int h = hsz[b];
    const int t = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (t >= h * h) return;
    const double* pb = gpart + (long)b * nchunk * hmax * hmax;
    double s = 0.0;
    for (int q = lane; q < nchunk; q += 32) s += pb[(long)q * hmax * hmax + t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncwarp();
    if (lane == 0) gsum[(long)b * hmax * hmax + t] = s;
}

// Pairing field (HFBPairingField, src/HFB.f90:350-518) after the block apply
// Y_i = sum_j Ktilde[j][i] psi_j (tensor cores): per point and block,
//   Fr = sum_i sum_c Y_ic psi_ic,  Fi = sum_i (-Y_i0 psi_i1 + Y_i1 psi_i0
//                                               - Y_i2 psi_i3 + Y_i3 psi_i2)
// in double-float, as k_pair_field (pairing.cu) forms it; part[b][0|1][V].
// Four lanes per point (spinors i = sub, sub + 4, ...), combined by a fixed
// shuffle order.
template <bool kF64>
__global__ void __launch_bounds__(256)
k_field_contract(const double* __restrict__ Y, const double* __restrict__ psi,
                 const int* __restrict__ members, const int* __restrict__ hsz, int hmax, long V,
                 double* __restrict__ part) {
    const int b = blockIdx.y, h = hsz[b];
    const long v = (long)blockIdx.x * (blockDim.x / 4) + threadIdx.x / 4;
    const int sub = threadIdx.x & 3;
    if constexpr (kF64) {
        double fr = 0.0, fi = 0.0;
        for (int i = sub; i < h && v < V; i += 4) {
            const double* y = Y + (long)(b * hmax + i) * 4 * V + v;
            const double* p = psi + (long)members[b * hmax + i] * 4 * V + v;
            const double y0 = y[0], y1 = y[V], y2 = y[2 * V], y3 = y[3 * V];
            const double a0 = p[0], a1 = p[V], a2 = p[2 * V], a3 = p[3 * V];
            fr = fma(y0, a0, fr);
            fr = fma(y1, a1, fr);
            fr = fma(y2, a2, fr);
            fr = fma(y3, a3, fr);
            fi = fi - (y0 * a1 - y1 * a0 + y2 * a3 - y3 * a2);
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            fr += __shfl_xor_sync(0xffffffffu, fr, o);
            fi += __shfl_xor_sync(0xffffffffu, fi, o);
        }
        if (sub == 0 && v < V) {
            part[((long)b * 2 + 0) * V + v] = fr;
            part[((long)b * 2 + 1) * V + v] = fi;
        }
        return;
    }
    float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f;
    for (int i = sub; i < h && v < V; i += 4) {
        const double* y = Y + (long)(b * hmax + i) * 4 * V + v;
        const double* p = psi + (long)members[b * hmax + i] * 4 * V + v;
        dfl yy[4], pp[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            yy[c] = df_split(y[c * V]);
            pp[c] = df_split(p[c * V]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) df_acc(rh, rl, yy[c], pp[c]);
        df_acc(ih, il, yy[0], df_neg(pp[1]));
        df_acc(ih, il, yy[1], pp[0]);
        df_acc(ih, il, yy[2], df_neg(pp[3]));
        df_acc(ih, il, yy[3], pp[2]);
    }
    dfl re = df_norm(dfl{rh, rl}), im = df_norm(dfl{ih, il});
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        re = df_add(re, dfl{__shfl_xor_sync(0xffffffffu, re.h, o),
                            __shfl_xor_sync(0xffffffffu, re.l, o)});
        im = df_add(im, dfl{__shfl_xor_sync(0xffffffffu, im.h, o),
                            __shfl_xor_sync(0xffffffffu, im.l, o)});
    }
    if (sub == 0 && v < V) {
        part[((long)b * 2 + 0) * V + v] = df_to_fast(re);
        part[((long)b * 2 + 1) * V + v] = df_to_fast(im);
    }
}

// The gaps' right factors in FP64, as k_pair_gaps (pairing.cu) forms them:
// Z_j0 = -Fr psi_j0 + Fi psi_j1, Z_j1 = -Fi psi_j0 - Fr psi_j1 (same for 2, 3), to
// z[b hmax + j].
__global__ void __launch_bounds__(128)
k_gaps_factor(const double* __restrict__ psi, const int* __restrict__ members,
              const int* __restrict__ hsz, int hmax, const double* __restrict__ fre,
              const double* __restrict__ fim, long V, double* __restrict__ z) {
    const int b = blockIdx.z, j = blockIdx.y, it = b / 2;
    const long v = (long)blockIdx.x * 128 + threadIdx.x;
    if (j >= hsz[b] || v >= V) return;
    const double* a = psi + (long)members[b * hmax + j] * 4 * V + v;
    double* o = z + ((long)b * hmax + j) * 4 * V + v;
    const double r = fre[it * V + v], m = fim[it * V + v];
    const double a0 = a[0], a1 = a[V], a2 = a[2 * V], a3 = a[3 * V];
    o[0] = fma(m, a1, -r * a0);
    o[V] = fma(-m, a0, -r * a1);
    o[2 * V] = fma(m, a3, -r * a2);
    o[3 * V] = fma(-m, a2, -r * a3);
}

}  // namespace

// Largest and smallest blocks of the FP64 form.  Above 64 its eight accumulators do
// not fit the 512 TMEM columns.  Below 24 the FP64 kernels of gs.cu are as fast or
// faster, but on large meshes; the whole Gram-Schmidt of four blocks at 10^3 / 16^3 /
// 24^3 in us, there and here: blocks of 16: 44 / 73 / 158 and 52 / 77 / 143, of 20: 53 /
// 96 / 220 and 59 / 88 / 163, of 24: 66 / 131 / 320 and 64 / 92 / 171, of 40: 118 / 280 /
// 750 and 92 / 146 / 297, of 64: 243 / 636 / 1776 and 144 / 230 / 480.
constexpr int kMeshTcMax64 = 64, kMeshTcMin64 = 24;

// Whether blocks of up to nbmax spinors go to the kernels of this file.
bool mesh_tc_serves(const mg_ctx* c, int nbmax, bool f64) {
    return c->tc_mesh_ok &&
           (f64 ? nbmax >= kMeshTcMin64 && nbmax <= kMeshTcMax64 : nbmax <= kMeshTcMax);
}

static void gs_tc_free(mg_ctx* c) {
    cudaFree(c->gs_Stc);
    cudaFree(c->gs_xd);
    cudaFree(c->gs_xe);
    c->gs_Stc = nullptr;
    c->gs_xd = nullptr;
    c->gs_xe = nullptr;
}

// Buffers of the tensor-core Gram-Schmidt, for both forms; new quantum numbers can
// change the number and the size of the blocks they are for.  Returns false where the
// FP64 kernels of gs.cu are the ones to run, also when the device has no room for them.
bool gs_tc_prepare(mg_ctx* c, bool f64) {
    if (!mesh_tc_serves(c, c->gs_nbmax, f64)) return false;
    if (c->gs_tc_nblk != c->gs_nblk || c->gs_tc_nbmax != c->gs_nbmax) gs_tc_free(c);
    if (c->gs_xd == nullptr) {
        const int nblk = c->gs_nblk;
        const bool both = c->gs_nbmax <= kMeshTcMax64;   // the FP64 form's chunks are smaller
        const long chunks = div_up(4 * c->V, chunk_for(both ? oz::kDigits64 : kDigits));
        if (cudaMalloc(&c->gs_Stc, (size_t)nblk * chunks * c->gs_nbmax * c->gs_nbmax *
                                       sizeof(double)) != cudaSuccess ||
            cudaMalloc(&c->gs_xd, (size_t)nblk * oz::kDigits64 * kXdStride * sizeof(uint16_t)) !=
                cudaSuccess ||
            cudaMalloc(&c->gs_xe, (size_t)nblk * kMeshTcMax * sizeof(int)) != cudaSuccess) {
            cudaGetLastError();
            gs_tc_free(c);
            return false;
        }
        c->gs_tc_nblk = nblk;
        c->gs_tc_nbmax = c->gs_nbmax;
    }
    return true;
}

template <int ND, int NP, bool kTwo>
static int overlap_launch(mg_ctx* c, const double* psi, const double* z, BlockIdx bi,
                          const int* list, int nblk, int nbmax, int nchunk, double* part) {
    const auto kernel = k_gs_overlap_tc<ND, NP, kTwo>;
    constexpr size_t sm = overlap_smem(ND, NP, kTwo);
    MG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    const int nunits = nchunk * nblk;
    kernel<<<std::min(c->num_sms, nunits), kRoleThreads, sm, c->stream>>>(
        psi, z, bi, list, nbmax, 4 * c->V, nchunk, nunits, part, c->tc_status);
    MG_LAUNCHED(c);
    return MG_OK;
}

// Chunk partials of the blocks' overlaps in gs_Stc, *nchunk of them.
int gs_overlap_tc(mg_ctx* c, const double* psi, const int* d_lists, const int* d_ordered, bool f64,
                  int* nchunk) {
    *nchunk = div_up(4 * c->V, chunk_for(f64 ? oz::kDigits64 : kDigits));
    const auto run = [&](auto launch) {
        return launch(c, psi, nullptr, BlockIdx{d_lists, nullptr, 0}, d_ordered, c->gs_nblk,
                      c->gs_nbmax, *nchunk, c->gs_Stc);
    };
    const int steps = std::max(1, div_up(c->gs_nbmax, 16));
    if (f64) return steps <= 2   ? run(overlap_launch<oz::kDigits64, 32, false>)
                    : steps == 3 ? run(overlap_launch<oz::kDigits64, 48, false>)
                                 : run(overlap_launch<oz::kDigits64, 64, false>);
    switch (steps) {
        case 1: return run(overlap_launch<kDigits, 16, false>);
        case 2: return run(overlap_launch<kDigits, 32, false>);
        case 3: return run(overlap_launch<kDigits, 48, false>);
        case 4: return run(overlap_launch<kDigits, 64, false>);
        default: return run(overlap_launch<kDigits, 80, false>);
    }
}

template <int ND, int NP>
static int apply_launch(mg_ctx* c, int nblk, const double* coef, long bstride, int ld, BlockIdx bi,
                        const double* in, double* out, double* upd, const int* in_list,
                        const int* out_list, const int* out_base, uint16_t* xd, int* xe) {
    k_coef_digits<ND, NP><<<nblk, dim3(NP, kCoefRows), 0, c->stream>>>(coef, bstride, ld, bi, xd, xe);
    MG_LAUNCHED(c);
    // (in place matters to the FP64 form's treatment of infinities alone)
    auto kernel = k_apply_tc<ND, NP, true>;
    if constexpr (ND == oz::kDigits64)
        if (in != out) kernel = k_apply_tc<ND, NP, false>;
    MG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)apply_smem(ND, NP)));
    const long V4 = 4 * c->V;
    const int tpb = div_up(V4, kRows), ntiles = tpb * nblk;
    const int sms = c->tc_grid_cap > 0 ? std::min(c->tc_grid_cap, c->num_sms) : c->num_sms;
    kernel<<<std::min(sms, ntiles), apply_threads(NP), apply_smem(ND, NP), c->stream>>>(
        in, out, upd, bi, in_list, out_list, out_base, xd, xe, coef, bstride, ld, V4, tpb, ntiles,
        c->tc_status);
    MG_LAUNCHED(c);
    return MG_OK;
}

template <class... A>
static int apply_tc(mg_ctx* c, int nblk, int nbmax, bool f64, A... args) {
    const int steps = std::max(1, div_up(nbmax, 16));
    if (f64) return steps <= 2   ? apply_launch<oz::kDigits64, 32>(c, nblk, args...)
                    : steps == 3 ? apply_launch<oz::kDigits64, 48>(c, nblk, args...)
                                 : apply_launch<oz::kDigits64, 64>(c, nblk, args...);
    switch (steps) {
        case 1: return apply_launch<kDigits, 16>(c, nblk, args...);
        case 2: return apply_launch<kDigits, 32>(c, nblk, args...);
        case 3: return apply_launch<kDigits, 48>(c, nblk, args...);
        case 4: return apply_launch<kDigits, 64>(c, nblk, args...);
        default: return apply_launch<kDigits, 80>(c, nblk, args...);
    }
}

int gs_apply_tc(mg_ctx* c, double* psi, double* upd, const int* d_lists, const int* d_ordered,
                bool f64) {
    const BlockIdx bi{d_lists, nullptr, 0};
    return apply_tc(c, c->gs_nblk, c->gs_nbmax, f64, c->gs_R, (long)c->gs_nbmax * c->gs_nbmax,
                    c->gs_nbmax, bi, psi, psi, upd, d_ordered, d_ordered, nullptr, c->gs_xd,
                    c->gs_xe);
}

// Buffers of the tensor-core canonical transform.  False where the kernels of
// pairing.cu are the ones to run, also when the device has no room for them.
bool can_tc_prepare(mg_ctx* c, bool f64) {
    if (!mesh_tc_serves(c, c->hfb.hmax, f64)) return false;
    if (c->can_xe == nullptr) {   // allocated last
        if ((c->can_xd == nullptr &&
             cudaMalloc(&c->can_xd, (size_t)4 * oz::kDigits64 * kXdStride * sizeof(uint16_t)) !=
                 cudaSuccess) ||
            cudaMalloc(&c->can_xe, (size_t)4 * kMeshTcMax * sizeof(int)) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
    }
    return true;
}

// Canonical basis of the four pairing blocks (hsz[b] <= kMeshTcMax), behind
// can_tc_prepare: CanTransfo is stored densely per block (ld = h) at b * hmax^2.
int can_transform_tc(mg_ctx* c, bool f64) {
    Hfb& H = c->hfb;
    const BlockIdx bi{nullptr, H.hsz, H.hmax};
    return apply_tc(c, 4, H.hmax, f64, H.cantr, (long)H.hmax * H.hmax, 0, bi,
                    c->bas[MG_HF_BASIS].psi, c->bas[MG_CAN_BASIS].psi, nullptr, H.members,
                    nullptr, H.cstart, c->can_xd, c->can_xe);
}

template <int NP>
static int gaps_launch(mg_ctx* c, int nchunk) {
    Hfb& H = c->hfb;
    constexpr size_t sm = overlap_smem(kDigits, NP, true);
    MG_CUDA(cudaFuncSetAttribute(k_gaps_tc<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_gaps_tc<NP><<<std::min(c->num_sms, 4 * nchunk), kGapThreads, sm, c->stream>>>(
        c->bas[MG_HF_BASIS].psi, H.members, H.hsz, H.hmax, H.fre, H.fim, c->V, nchunk, c->gap_part,
        c->tc_status);
    MG_LAUNCHED(c);
    return MG_OK;
}

// Gaps partial sums of the four pairing blocks on the tensor cores into
// gsum[b][i * h + j] (to be finished by k_gaps_finish with one chunk).
int gaps_tc(mg_ctx* c, double* gsum) {
    Hfb& H = c->hfb;
    if (!mesh_tc_serves(c, H.hmax, false)) return MG_ERR_STATE;
    const int nchunk = div_up(c->V, kGapPts);
    if (c->gap_part == nullptr)
        MG_CUDA(cudaMalloc(&c->gap_part, (size_t)4 * nchunk * H.hmax * H.hmax * sizeof(double)));
    switch (std::max(1, div_up(H.hmax, 16))) {
        case 1: MG_TRY(gaps_launch<16>(c, nchunk)); break;
        case 2: MG_TRY(gaps_launch<32>(c, nchunk)); break;
        case 3: MG_TRY(gaps_launch<48>(c, nchunk)); break;
        case 4: MG_TRY(gaps_launch<64>(c, nchunk)); break;
        default: MG_TRY(gaps_launch<80>(c, nchunk)); break;
    }
    k_gaps_sum<<<dim3(div_up((long)H.hmax * H.hmax, 8), 4), 256, 0, c->stream>>>(
        c->gap_part, H.hsz, H.hmax, nchunk, gsum);
    MG_LAUNCHED(c);
    return MG_OK;
}

// Scratch of the pairing contractions.  False where the kernels of pairing.cu are the
// ones to run, in the FP64 form also when the device has no room for the scratch.
bool pair_tc_prepare(mg_ctx* c, bool f64) {
    Hfb& H = c->hfb;
    if (!mesh_tc_serves(c, H.hmax, f64)) return false;
    if (c->field_ybase == nullptr) {
        const int yb[4] = {0, H.hmax, 2 * H.hmax, 3 * H.hmax};
        const auto room = [](auto** p, size_t bytes) {
            return *p != nullptr || cudaMalloc(p, bytes) == cudaSuccess;
        };
        if (!room(&c->field_y, (size_t)4 * H.hmax * 4 * c->V * sizeof(double)) ||
            !room(&c->field_xd, (size_t)4 * oz::kDigits64 * kXdStride * sizeof(uint16_t)) ||
            !room(&c->field_xe, (size_t)4 * kMeshTcMax * sizeof(int)) ||
            !room(&c->field_ybase, sizeof(yb)) ||
            cudaMemcpy(c->field_ybase, yb, sizeof(yb), cudaMemcpyHostToDevice) != cudaSuccess) {
            cudaGetLastError();
            if (c->field_ybase) cudaFree(c->field_ybase);
            c->field_ybase = nullptr;   // not complete
            return !f64;                // mixed: the launch reports the missing scratch
        }
    }
    if (f64 && c->gap_part64 == nullptr &&
        cudaMalloc(&c->gap_part64, (size_t)4 * div_up(4 * c->V, chunk_for(oz::kDigits64)) * H.hmax *
                                       H.hmax * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        c->gap_part64 = nullptr;
        return false;
    }
    return true;
}

// Pairing-field partials of the four blocks: Y = block apply of Ktilde
// (tensor cores) into the scratch basis, then the pointwise contraction.
int pair_field_tc(mg_ctx* c, bool f64) {
    Hfb& H = c->hfb;
    if (c->field_ybase == nullptr) return MG_ERR_CUDA;   // pair_tc_prepare
    const long V = c->V;
    const BlockIdx bi{nullptr, H.hsz, H.hmax};
    MG_TRY(apply_tc(c, 4, H.hmax, f64, H.ktil, (long)H.hmax * H.hmax, 0, bi,
                    c->bas[MG_HF_BASIS].psi, c->field_y, nullptr, H.members, nullptr,
                    c->field_ybase, c->field_xd, c->field_xe));
    const auto contract = f64 ? k_field_contract<true> : k_field_contract<false>;
    contract<<<dim3(div_up(V, 64), 4), 256, 0, c->stream>>>(
        c->field_y, c->bas[MG_HF_BASIS].psi, H.members, H.hsz, H.hmax, V, H.fpart);
    MG_LAUNCHED(c);
    return MG_OK;
}

// The same in the FP64 form, behind pair_field_tc, whose scratch basis takes the
// factors Z.  Pairing field and gaps of 108 spwfs at 18^3 (blocks of 26 and 28): 136
// and 152 us by FP64 FMAs, here 56 and 100.
int gaps_tc64(mg_ctx* c, double* gsum) {
    Hfb& H = c->hfb;
    if (c->field_y == nullptr || c->gap_part64 == nullptr) return MG_ERR_STATE;
    const long V = c->V;
    const int nchunk = div_up(4 * V, chunk_for(oz::kDigits64));
    const double* psi = c->bas[MG_HF_BASIS].psi;
    k_gaps_factor<<<dim3(div_up(V, 128), H.hmax, 4), 128, 0, c->stream>>>(
        psi, H.members, H.hsz, H.hmax, H.fre, H.fim, V, c->field_y);
    MG_LAUNCHED(c);
    const auto run = [&](auto launch) {
        return launch(c, psi, c->field_y, BlockIdx{nullptr, H.hsz, H.hmax}, H.members, 4, H.hmax,
                      nchunk, c->gap_part64);
    };
    const int steps = div_up(H.hmax, 16);
    MG_TRY(steps <= 2   ? run(overlap_launch<oz::kDigits64, 32, true>)
           : steps == 3 ? run(overlap_launch<oz::kDigits64, 48, true>)
                        : run(overlap_launch<oz::kDigits64, 64, true>));
    k_gaps_sum<<<dim3(div_up((long)H.hmax * H.hmax, 8), 4), 256, 0, c->stream>>>(
        c->gap_part64, H.hsz, H.hmax, nchunk, gsum);
    MG_LAUNCHED(c);
    return MG_OK;
}

}  // namespace mg
