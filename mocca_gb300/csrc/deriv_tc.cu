// deriv_tc.cu -- DeriveAll on the tcgen05 tensor cores: the mixed form, and
// the FP64 form on lines of up to 32 points.
//
// Same operation as the kernels of deriv.cu (Opt_LAG{X,Y,Z}_EV8 and
// Lapla_LAG_EV8, src/OptimizedDerivatives.f90:115-148, :306-338, :432-464,
// :551-615): per line of a real grid, out(i) = sum_q M(i,q) in(q) for the
// first- and second-derivative matrices of the axis, as exact BF16 digit
// products (ozaki.cuh).  A line is one MMA row; the Lagrange block of the
// axis is two column blocks (first, then second derivative); rows and K are n
// padded to 16, 32 or 48.
//   mixed form  six digits (47-bit operands), four accumulators, stored as
//               {hi, lo} float pairs, the format the double-float consumers
//               read;
//   FP64 form   eight digits (62-bit operands), eight accumulators, rounded once
//               to FP64.  Its error is below that of the FP64 FMA chain it
//               replaces (ozaki.cuh), which is bound by the FP64 pipe: 2104 us
//               against 327 us here at 24^3 with 160 spwfs.
//
// One persistent CTA per SM walks 128-line tiles of one matrix slot (the
// basis' jobs are sorted by slot, the CTAs divided between the two slots by
// their tile counts, so that a CTA holds one slot's matrices) with
// warp-specialised roles:
//   warps 0-7   slicers: two lanes per line (lanes l and l + 16 of a warp),
//               each with every other chunk of four points; they prefetch the
//               next tile's points with cp.async into slots of their own, before
//               they turn the current ones into digit planes or, where shared
//               memory has one slot only, behind their last reads of it;
//   warp 8      MMA issue (one thread): the digit pairs of both derivatives'
//               columns together (mixed form), or of the first's, then of the
//               second's, with a commit each (FP64 form, whose accumulators
//               leave TMEM room for one set only);
//   warps 9-24  epilogue: eight warps per column block (two per TMEM lane
//               quarter, alternating chunks of four columns), combine the
//               accumulators, scale, store.  The Laplacian values a chunk adds
//               to are loaded while the chunk before it is worked on.
// The kernel is bound by instruction issue (58 to 66% of the slots at 24^3; HBM
// below 34%, the tensor pipe below 36%).  Two things brought it there.  The digit planes
// of a column block's matrix are stacked, so that an MMA of up to 192 columns
// serves several pairs of a line digit (stacked_pairs in ozaki.cuh): with one MMA
// of 32 columns per pair, about 125 clocks each, the MMAs bound the kernel
// (FP64 form 660 us, now 327).  And separate column blocks give the two
// epilogue groups straight code and let one block's MMAs run under the other's
// epilogue, while every plane, slot and address that one thread alone uses
// needs no barrier.  DeriveAll of one basis, mixed form, against one epilogue
// group, both slots' matrices per CTA, a pair per MMA and eight-byte stores
// on every axis: 240 us (336 before) at 24^3 with 160 spwfs, 25 us (37) at
// 10^3 with 40, 1.50 ms (3.03) at 36^3 with 300.
//
// Hand-offs are mbarriers: fullA (one arrival per slicer warp), emptyA and
// fullT (tcgen05.commit), emptyT (one arrival per epilogue warp of the block);
// every wait is bounded and a timeout sets the context's status word.  The
// line exponents the epilogue reads sit in a four-tile ring.
// Three launches, one per axis: x writes d/dx and Lxx, y writes d/dy and
// adds Lyy, z writes d/dz and adds Lzz, so the Laplacian is summed
// (X + Y) + Z as in Lapla_LAG_EV8.
// A line that holds an infinity or a NaN has no digits: its outputs come
// from the plain FP64 sum.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "df.cuh"
#include "mg_internal.cuh"
#include "ozaki.cuh"
#include "tc.cuh"

namespace mg {

namespace {

constexpr int kTile = 128;                      // lines per tile (MMA M)
constexpr int kSliceWarps = 8;
constexpr int kSlicers = 32 * kSliceWarps;      // warps 0-7
constexpr int kMmaWarp = kSliceWarps;
constexpr int kBlockWarps = 8;                  // epilogue warps of one column block
constexpr int kThreads = kSlicers + 32 + 2 * 32 * kBlockWarps;   // 800
constexpr long long kWaitCycles = 4000000000LL; // ~2 s at the top SM clock
constexpr int kMaxLine = 48;                    // mixed form
constexpr int kMaxLine64 = 32;                  // FP64 form (eight accumulators of 2 x 32 columns)

// Buffers by K: up to 32 points two plane buffers, at 48 one (the planes of 128 x 48
// digits take 74 KB); a second staging slot where there is room for it beside them and
// the matrices with their planes of zeros.
constexpr int nbuf_of(int kp) { return kp <= 32 ? 2 : 1; }
constexpr int nslot_of(int kp, bool f64) { return kp == 48 || (f64 && kp == 32) ? 1 : 2; }
constexpr int blocks_of(bool f64) { return f64 ? 2 : 1; }   // MMA blocks, see k_deriv_tc
constexpr int digits_of_form(bool f64) { return f64 ? oz::kDigits64 : oz::kDigits; }
// bytes of a matrix plane of a block, planes of both derivatives with their zeros
constexpr int plane_bytes(int kp, bool f64) { return 2 * kp / blocks_of(f64) * kp * 2; }
constexpr int matrix_planes(int kp, bool f64) {
    return blocks_of(f64) * oz::stack_planes(digits_of_form(f64), 2 * kp / blocks_of(f64));
}
constexpr int accs_of(bool f64) { return f64 ? oz::kAccs64 : (int)oz::kAccs; }
// TMEM accumulator sets: two where 512 columns hold them
constexpr int tbuf_of(int kp, int nacc) { return 4 * nacc * kp <= 512 ? 2 : 1; }
constexpr uint32_t tmem_cols(int kp, int nacc) {
    const int need = 2 * tbuf_of(kp, nacc) * nacc * kp;
    return need <= 128 ? 128u : (need <= 256 ? 256u : 512u);
}

struct TcPass {
    const GridJob* jobs;
    const int* perm;           // jobs sorted by the axis' slot
    int njobs[2];              // jobs of each slot
    int ctas0;                 // CTAs on slot 0, the rest on slot 1
    const uint16_t* bmat[2];   // per slot: 2 x ND planes of KP rows x KP, K-major core matrices
    const int* erow[2];        // per slot: 2 x kMaxLine row exponents
    const double* mat[2][2];   // [kind][slot] FP64 matrices, transposed (lines with infinities)
    int axis, n, nlines, tpj, nx, ny;
    uint32_t tpj_inv, nx_inv;  // ceil(2^32 / d), quotients by a multiply
    int* status;
};

// a / d by the rounded-up reciprocal: exact while a (d inv - 2^32) < 2^32,
// which holds for a < 2^32 / d
__device__ __forceinline__ int quotient(int a, uint32_t inv) {
    return inv == 0 ? a : (int)__umulhi((uint32_t)a, inv);   // inv 0: d = 1
}

template <int NBUF, int NTB, int NBLK>
struct TcShared {
    uint64_t fullA[NBUF], emptyA[NBUF];
    uint64_t fullT[NBLK][NTB], emptyT[NBLK][NTB];   // [MMA block][buffer]
    uint64_t emaxReady[4];   // tile k's line exponents written
    uint32_t tmem;
    // line exponents of the last four tiles: the slicers write tile k's after
    // the MMAs of tile k - NBUF, which waited for the epilogue of tile
    // k - NBUF - NTB, so a ring of four is never overwritten early
    uint16_t emax[4][kTile];
    alignas(16) int erow[2][kMaxLine];
    alignas(16) float srow[2][kMaxLine];
};

// global offset of element 0 of line l of a grid (axis order: x, y, z)
__device__ __forceinline__ long line_offset(const TcPass& P, int l) {
    if (P.axis == 0) return (long)l * P.n;
    if (P.axis == 1) {
        const int z = quotient(l, P.nx_inv);
        return (long)z * P.nx * P.ny + (l - z * P.nx);
    }
    return l;
}

__device__ __forceinline__ double* out_of(const GridJob& J, int axis) {
    return axis == 0 ? J.dx : (axis == 1 ? J.dy : J.dz);
}

__device__ __forceinline__ bool wait_warp(uint64_t* mbar, uint32_t parity) {
    return __all_sync(0xffffffffu, tc::mbar_wait(mbar, parity, kWaitCycles)) != 0;
}

__device__ __forceinline__ void arrive_warp(uint64_t* mbar, int lane) {
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(mbar);
}

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(sdst)), "l"(gsrc)
                 : "memory");
}

// 8-byte words of four consecutive outputs of an x line
__device__ __forceinline__ void store4(double* p, const double (&o)[4], int left, int n) {
    if (left >= 4 && (n & 3) == 0) {
        // a whole 32-byte sector
        asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(o[0]), "d"(o[1]),
                     "d"(o[2]), "d"(o[3])
                     : "memory");
    } else if ((n & 1) == 0) {
        *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
        if (left > 2) *reinterpret_cast<double2*>(p + 2) = make_double2(o[2], o[3]);
    } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (u < left) p[u] = o[u];
    }
}

// KP: padded K; F64: the FP64 form; XP: the x pass (lines contiguous in memory)
template <int KP, bool F64, bool XP>
__global__ void __launch_bounds__(kThreads, 1)
k_deriv_tc(TcPass P) {
    constexpr int ND = digits_of_form(F64);
    constexpr int NACC = accs_of(F64);
    static_assert(!F64 || KP <= kMaxLine64, "combine64 holds sums of at most 32 terms");
    constexpr int NBUF = nbuf_of(KP), NSLOT = nslot_of(KP, F64), NTB = tbuf_of(KP, NACC);
    // FP64 form: the two derivatives' columns are two MMA blocks with commits of
    // their own; mixed form: one block of 2 KP columns
    constexpr int NBLK = blocks_of(F64), COLS = 2 * KP / NBLK;
    constexpr int kPlane = kTile * KP * 2;     // bytes of one digit plane of a tile
    constexpr int kKg = KP / 8;                // K groups of 8
    constexpr uint32_t kSboK = 128u * kKg;     // stride byte offset of the planes
    constexpr int kPlaneB = plane_bytes(KP, F64);
    constexpr int kZerosB = oz::stack_zeros(ND, COLS) * kPlaneB, kBlockB = ND * kPlaneB;
    extern __shared__ uint8_t smraw[];
    __shared__ TcShared<NBUF, NTB, NBLK> S;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = P.n;
    const int slot = (int)blockIdx.x < P.ctas0 ? 0 : 1;
    const int cta = slot == 0 ? blockIdx.x : blockIdx.x - P.ctas0;
    const int nctas = slot == 0 ? P.ctas0 : gridDim.x - P.ctas0;
    const int* perm = P.perm + (slot == 0 ? 0 : P.njobs[0]);
    const int ntiles = P.njobs[slot] * P.tpj;

    const uint32_t s0 = tc::smem_u32(smraw);
    uint8_t* sA = smraw + ((128u - (s0 & 127u)) & 127u);        // NBUF x ND planes
    uint8_t* sB = sA + NBUF * ND * kPlane;                      // per block zeros, ND planes
    uint8_t* sIn = sB + NBLK * (kZerosB + kBlockB);             // NSLOT x nch8 x 2 x kSlicers x 16

    if (warp == 0) tc::alloc(&S.tmem, tmem_cols(KP, NACC));
    if (tid == 0) {
        for (int b = 0; b < NBUF; ++b) {
            tc::mbar_init(&S.fullA[b], kSliceWarps);
            tc::mbar_init(&S.emptyA[b], 1);
        }
        for (int h = 0; h < NBLK; ++h)
            for (int b = 0; b < NTB; ++b) {
                tc::mbar_init(&S.fullT[h][b], 1);
                tc::mbar_init(&S.emptyT[h][b], 2 * kBlockWarps / NBLK);
            }
        for (int b = 0; b < 4; ++b) tc::mbar_init(&S.emaxReady[b], kSliceWarps);
    }
    {
        for (int h = 0; h < NBLK; ++h) {
            const uint4* src = reinterpret_cast<const uint4*>(P.bmat[slot]) + h * (kBlockB / 16);
            uint4* dst = reinterpret_cast<uint4*>(sB + h * (kZerosB + kBlockB));
            for (int t = tid; t < (kZerosB + kBlockB) / 16; t += kThreads)
                dst[t] = t < kZerosB / 16 ? make_uint4(0u, 0u, 0u, 0u) : src[t - kZerosB / 16];
        }
        // K columns past the line stay zero
        uint4* a = reinterpret_cast<uint4*>(sA);
        for (int t = tid; t < NBUF * ND * kPlane / 16; t += kThreads)
            a[t] = make_uint4(0u, 0u, 0u, 0u);
        if (tid < 2 * kMaxLine) {
            const int e = P.erow[slot][tid];
            S.erow[tid / kMaxLine][tid % kMaxLine] = e;
            S.srow[tid / kMaxLine][tid % kMaxLine] = oz::pow2f(e);
        }
    }
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    // the set-up above may run while the pass before this one ends; the
    // Laplacian that pass wrote is read after this
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tmem = S.tmem;
    const long lstride = XP ? 1 : (P.axis == 1 ? (long)P.nx : (long)P.nx * P.ny);
    bool ok = true;

    if (warp < kSliceWarps) {
        // ---------------- slicers ----------------
        const int row = warp * 16 + (lane & 15), h = lane >> 4;
        const int nch8 = (n + 7) >> 3;   // chunks of four points per lane
        // slot of chunk i, pair u of this thread: consecutive threads 16 bytes apart
        auto slot_at = [&](int sbuf, int i, int pair) {
            return reinterpret_cast<double*>(
                sIn + ((size_t)((sbuf * nch8 + i) * 2 + pair) * kSlicers + tid) * 16);
        };
        // this lane's first point of the tile, null where its line does not exist
        auto first_point = [&](int T) -> const double* {
            if (T >= ntiles) return nullptr;
            const int job = quotient(T, P.tpj_inv), l = (T - job * P.tpj) * kTile + row;
            if (l >= P.nlines) return nullptr;
            return P.jobs[perm[job]].in + line_offset(P, l) + 4 * h * lstride;
        };
        // copies chunk i (points k0 = 4 h + 8 i, ...) at `in`, which moves on to the next
        auto prefetch = [&](const double*& in, int sbuf, int i) {
            const int k0 = 4 * h + 8 * i;
            if (XP && (n & 1) == 0) {
                // even lines: 16-byte copies (line starts and k0 are even)
                cp_async16(slot_at(sbuf, i, 0), in);
                if (k0 + 2 < n) cp_async16(slot_at(sbuf, i, 1), in + 2);
                in += 8;
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (k0 + u < n) tc::cp_async8(slot_at(sbuf, i, u >> 1) + (u & 1), in);
                    in += lstride;
                }
                in += 4 * lstride;
            }
        };
        auto prefetch_all = [&](const double* in, int sbuf) {
            if (in)
#pragma unroll 1
                for (int i = 0; 4 * h + 8 * i < n; ++i) prefetch(in, sbuf, i);
        };
        int T = cta;
        const double* next = first_point(T);
        prefetch_all(next, 0);
        tc::cp_async_commit();
        for (int k = 0; T < ntiles; T += nctas, ++k) {
            const int buf = k % NBUF, sbuf = k % NSLOT;
            const bool live = next != nullptr;
            tc::cp_async_wait_all();
            // the points of chunk i, zero past the line's end
            auto chunk = [&](int i, double (&v)[4]) {
#pragma unroll
                for (int pair = 0; pair < 2; ++pair) {
                    const double2 x = *reinterpret_cast<const double2*>(slot_at(sbuf, i, pair));
                    const int q = 4 * (2 * i + h) + 2 * pair;
                    v[2 * pair] = live && q < n ? x.x : 0.0;
                    v[2 * pair + 1] = live && q + 1 < n ? x.y : 0.0;
                }
            };
            uint32_t top = 0;
            for (int i = 0; 4 * (2 * i + h) < n; ++i) {
                double v[4];
                chunk(i, v);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    top = max(top, (uint32_t)__double2hiint(v[u]) & 0x7FFFFFFFu);
            }
            top = max(top, __shfl_xor_sync(0xffffffffu, top, 16));
            const int emax = (int)(top >> 20);
            next = first_point(T + nctas);
            const double* ahead = next;
            if (NSLOT == 2) {
                // the other staging slot was read in the iteration before
                prefetch_all(next, sbuf ^ 1);
                tc::cp_async_commit();
            }
            if (k >= NBUF) {
                ok = wait_warp(&S.emptyA[buf], ((k - NBUF) / NBUF) & 1);
                if (!ok) break;
            }
            if (h == 0) S.emax[k & 3][row] = (uint16_t)emax;
            arrive_warp(&S.emaxReady[k & 3], lane);
            const oz::FixedRow<ND> fixed(emax);
            uint8_t* planes = sA + buf * ND * kPlane + (row >> 3) * (kKg * 128) + (row & 7) * 16 + 8 * h;
            // chunk 2 i + h of a row is half h of its K group i
#pragma unroll 1
            for (int i = 0; 4 * (2 * i + h) < n; ++i) {
                double v[4];
                chunk(i, v);
                if (NSLOT == 1 && NBUF == 2 && ahead) prefetch(ahead, 0, i);
                uint2 w[ND];
                oz::digits4<ND>(v, fixed, w);
#pragma unroll
                for (int a = 0; a < ND; ++a)
                    *reinterpret_cast<uint2*>(planes + a * kPlane + i * 128) = w[a];
            }
            tc::fence_proxy_async();
            arrive_warp(&S.fullA[buf], lane);
            if (NSLOT == 1) {
                // with one plane buffer the MMAs leave time for all of the next tile's
                // points (36^3: 1016 us this way, 1072 chunk by chunk; FP64 at 24^3 with
                // two buffers 335 and 328)
                if (NBUF == 1) prefetch_all(next, 0);
                tc::cp_async_commit();
            }
        }
        tc::cp_async_wait_all();
    } else if (warp == kMmaWarp) {
        // ---------------- MMA issue ----------------
        if (lane == 0) {
            int k = 0;
            for (int T = cta; T < ntiles; T += nctas, ++k) {
                const int buf = k % NBUF, tb = k % NTB;
                ok = tc::mbar_wait(&S.fullA[buf], (k / NBUF) & 1, kWaitCycles);
                for (int h = 0; h < NBLK && ok; ++h) {
                    if (k >= NTB)
                        ok = tc::mbar_wait(&S.emptyT[h][tb], ((k - NTB) / NTB) & 1, kWaitCycles);
                    if (!ok) break;
                    tc::fence_after();
                    oz::issue_stacked<ND, COLS, KP / 16>(
                        tmem + (uint32_t)((tb * NBLK + h) * NACC * COLS),
                        tc::smem_u32(sA + buf * ND * kPlane), kPlane,
                        tc::smem_u32(sB + h * (kZerosB + kBlockB) + kZerosB), kSboK);
                    if (h == NBLK - 1) tc::commit(&S.emptyA[buf]);
                    tc::commit(&S.fullT[h][tb]);
                }
                if (!ok) break;
            }
            // the last commit of each block covers every MMA of this CTA
            for (int h = 0; h < NBLK && k > 0; ++h)
                ok &= tc::mbar_wait(&S.fullT[h][(k - 1) % NTB], ((k - 1) / NTB) & 1, kWaitCycles);
        }
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        const int e = warp - (kMmaWarp + 1);
        const int h = e / kBlockWarps;            // column block: first or second derivative
        const int c0 = (e % kBlockWarps) >> 2;    // chunks c0, c0 + 2, ...
        const int blk = NBLK == 2 ? h : 0;        // its MMA block
        const int quarter = warp & 3;             // TMEM lanes of this warp
        const int erow = quarter * 32 + lane;     // tile row
        const int nch = (n + 3) >> 2;
        for (int k = 0, T = cta; T < ntiles; T += nctas, ++k) {
            const int tb = k % NTB;
            const int job = quotient(T, P.tpj_inv), l = (T - job * P.tpj) * kTile + erow;
            const GridJob& J = P.jobs[perm[job]];
            double* dst = h == 0 ? out_of(J, P.axis) : J.lap;
            bool live = l < P.nlines && dst != nullptr;
            if (live) dst += line_offset(P, l) + 4 * c0 * lstride;
            // Laplacian values of the next chunk (y and z passes)
            const bool add = !XP && h == 1;
            double prev[4];
            auto load_prev = [&](const double* p, int left) {
#pragma unroll
                for (int u = 0; u < 4; ++u, p += lstride)
                    if (u < left) prev[u] = *p;
            };
            if (add && live) load_prev(dst, n - 4 * c0);
            ok = wait_warp(&S.emaxReady[k & 3], (k >> 2) & 1);
            if (ok) ok = wait_warp(&S.fullT[blk][tb], (k / NTB) & 1);
            if (!ok) break;
            tc::fence_after();
            const int emax = S.emax[k & 3][erow];
            const uint32_t tq = tmem + ((uint32_t)(quarter * 32) << 16) +
                                (uint32_t)((tb * NBLK + blk) * NACC * COLS + (NBLK == 2 ? 0 : h * KP));
            const float sline = emax == 0 ? 0.0f : oz::pow2f(emax - 1023 - 12);
            if (c0 >= nch) {
                tc::fence_before();
                arrive_warp(&S.emptyT[blk][tb], lane);
            }
            if (live && emax != 0 && (F64 ? emax < 128 || emax > 1900 : emax == 2047)) {
                // an infinity or a NaN in the line (FP64 form: also a line near
                // the ends of the exponent range): this lane's outputs by the plain sum
                const double* src = J.in + line_offset(P, l);
                const double* mt = P.mat[h][slot];
                double* d = dst;
#pragma unroll 1
                for (int j = 4 * c0; j < n;) {
                    double s = 0.0;
#pragma unroll 1
                    for (int q = 0; q < n; ++q) s = fma(mt[q * n + j], src[q * lstride], s);
                    if (F64) {
                        *d = add ? *d + s : s;
                    } else {
                        float2* f = reinterpret_cast<float2*>(d);
                        *f = make_float2((float)(add ? (double)f->x + s : s), 0.0f);
                    }
                    const int step = (j & 3) == 3 ? 5 : 1;
                    j += step;
                    d += step * lstride;
                }
                live = false;
            }
            for (int ch = c0; ch < nch; ch += 2) {
                uint32_t r[NACC][4];
                __syncwarp();
#pragma unroll
                for (int g = 0; g < NACC; ++g) tc::ld4(tq + (uint32_t)(g * COLS + 4 * ch), r[g]);
                double was[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) was[u] = prev[u];
                const int left = n - 4 * ch;   // outputs of this chunk, at least 1
                if (add && live) load_prev(dst + 8 * lstride, left - 8);
#pragma unroll
                for (int g = 0; g < NACC; ++g) tc::wait_ld(r[g]);
                if (ch + 2 >= nch) {
                    // the last accumulators of this tile are in registers
                    tc::fence_before();
                    arrive_warp(&S.emptyT[blk][tb], lane);
                }
                if (live) {
                    double o[4];
                    if constexpr (F64) {
                        const int4 ec = *reinterpret_cast<const int4*>(&S.erow[h][4 * ch]);
                        const int x = emax - 1023 - oz::kUnit64;
                        const int xs[4] = {x + ec.x, x + ec.y, x + ec.z, x + ec.w};
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            uint32_t a[NACC];
#pragma unroll
                            for (int g = 0; g < NACC; ++g) a[g] = r[g][u];
                            o[u] = oz::combine64(a, xs[u]);
                            if (add) o[u] = was[u] + o[u];
                        }
                    } else {
                        const float4 sc = *reinterpret_cast<const float4*>(&S.srow[h][4 * ch]);
                        const float scs[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            dfl x = oz::combine4(__uint_as_float(r[0][u]), __uint_as_float(r[1][u]),
                                                 __uint_as_float(r[2][u]), __uint_as_float(r[3][u]));
                            const float f = __fmul_rn(sline, scs[u]);
                            x.h = __fmul_rn(x.h, f);
                            x.l = __fmul_rn(x.l, f);
                            if (add)
                                x = df_add(dfl{__int_as_float(__double2loint(was[u])),
                                               __int_as_float(__double2hiint(was[u]))}, x);
                            o[u] = __hiloint2double(__float_as_int(x.l), __float_as_int(x.h));
                        }
                    }
                    if (XP) {
                        store4(dst, o, left, n);
                    } else {
                        double* p = dst;
#pragma unroll
                        for (int u = 0; u < 4; ++u, p += lstride)
                            if (u < left) *p = o[u];
                    }
                }
                dst += 8 * lstride;
            }
        }
    }
    if (!ok) tc::report_timeout(P.status);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::dealloc(tmem, tmem_cols(KP, NACC));
}

int kp_of(int n) { return n <= 16 ? 16 : (n <= 32 ? 32 : 48); }

size_t smem_bytes(int n, bool f64) {
    const int kp = kp_of(n);
    return 128 + (size_t)nbuf_of(kp) * digits_of_form(f64) * kTile * kp * 2 +
           (size_t)matrix_planes(kp, f64) * plane_bytes(kp, f64) +
           (size_t)nslot_of(kp, f64) * ((n + 7) / 8) * 2 * kSlicers * 16;
}

template <bool F64>
const void* kernel_of(int kp, bool xp) {
    if (kp == 16) return xp ? (const void*)k_deriv_tc<16, F64, true> : (const void*)k_deriv_tc<16, F64, false>;
    if constexpr (!F64)
        if (kp == 48) return xp ? (const void*)k_deriv_tc<48, false, true> : (const void*)k_deriv_tc<48, false, false>;
    return xp ? (const void*)k_deriv_tc<32, F64, true> : (const void*)k_deriv_tc<32, F64, false>;
}

const void* kernel_for(bool f64, int kp, bool xp) {
    return f64 ? kernel_of<true>(kp, xp) : kernel_of<false>(kp, xp);
}

constexpr size_t kSmemCap = 225 * 1024;   // plus under 2 KB of static TcShared

}  // namespace

// Digit planes of the Lagrange blocks, built once per context and form: per
// (axis, slot) stacked planes of 2 x n rows rounded up to 16, 32 or 48: the
// FP64 form's all planes of the first derivative before those of the second,
// the mixed form's the two derivatives of a plane together.  Row exponents
// sit at a stride of 2 kMaxLine per (axis, slot).  The mixed form serves
// lines of up to 48 points, the FP64 form up to 32.
int tc_setup(mg_ctx* c) {
    const int ns[3] = {c->nx, c->ny, c->nz};
    c->tc_ok = c->tc_ok64 = false;
    // the mesh-sized GEMMs of meshgemm_tc.cu need no Lagrange planes: they
    // run on any mesh
    if (!c->h_tc_status) {
        MG_CUDA(cudaHostAlloc(&c->h_tc_status, sizeof(int), cudaHostAllocMapped));
        *c->h_tc_status = 0;
    }
    MG_CUDA(cudaHostGetDevicePointer(&c->tc_status, c->h_tc_status, 0));
    c->tc_mesh_ok = true;
    const int nmax = std::max(ns[0], std::max(ns[1], ns[2]));
    if (nmax > kMaxLine) return MG_OK;
    const bool f64 = nmax <= kMaxLine64;
    long total = 0;
    for (int form = 0; form < (f64 ? 2 : 1); ++form)
        for (int a = 0; a < 3; ++a)
            for (int s = 0; s < 2; ++s) {
                c->tc_off[form][a][s] = total;
                total += (long)(form ? oz::kDigits64 : oz::kDigits) * 2 * kp_of(ns[a]) * kp_of(ns[a]);
            }
    std::vector<uint16_t> h(total, 0);
    std::vector<int> he(3 * 2 * 2 * kMaxLine, 0);
    for (int a = 0; a < 3; ++a) {
        const int n = ns[a], kp = kp_of(n);
        const long nn = (long)n * n;
        std::vector<double> d1(2 * nn), d2(2 * nn);
        MG_TRY(mg_lagrange_matrices(n, c->p.dx, c->folded ? 1 : 0, d1.data(), d2.data()));
        for (int s = 0; s < 2; ++s)
            for (int kind = 0; kind < 2; ++kind)
                for (int j = 0; j < n; ++j) {
                    const double* row = (kind ? d2.data() : d1.data()) + s * nn + (long)j * n;
                    double mx = 0.0;
                    for (int k = 0; k < n; ++k) mx = std::max(mx, std::fabs(row[k]));
                    const int E = oz::host_row_exponent(mx);
                    he[((a * 2 + s) * 2 + kind) * kMaxLine + j] = E;
                    for (int form = 0; form < (f64 ? 2 : 1); ++form) {
                        const int nd = form ? oz::kDigits64 : oz::kDigits;
                        const double scale = std::ldexp(1.0, form ? oz::fixed_power<oz::kDigits64>(E)
                                                                  : oz::fixed_power<oz::kDigits>(E));
                        for (int k = 0; k < n; ++k) {
                            uint16_t dg[oz::kDigits64];
                            oz::host_digits(row[k], scale, dg, nd);
                            for (int b = 0; b < nd; ++b)
                                h[c->tc_off[form][a][s] +
                                  tc::kmajor_off_g((form ? kind * nd + b : 2 * b + kind) * kp + j, k,
                                                   kp / 8) / 2] = dg[b];
                        }
                    }
                }
    }
    MG_CUDA(cudaMalloc(&c->tcmats, total * sizeof(uint16_t)));
    MG_CUDA(cudaMemcpy(c->tcmats, h.data(), total * sizeof(uint16_t), cudaMemcpyHostToDevice));
    MG_CUDA(cudaMalloc(&c->tc_erow, he.size() * sizeof(int)));
    MG_CUDA(cudaMemcpy(c->tc_erow, he.data(), he.size() * sizeof(int), cudaMemcpyHostToDevice));
    // the kernels of this mesh (each is loaded when it is first touched)
    for (int form = 0; form < (f64 ? 2 : 1); ++form)
        for (int a = 0; a < 3; ++a)
            MG_CUDA(cudaFuncSetAttribute(kernel_for(form == 1, kp_of(ns[a]), a == 0),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap));
    c->tc_ok = true;
    c->tc_ok64 = f64;
    return MG_OK;
}

// DeriveAll of a basis on the tensor cores: the mixed form with double-float
// output, or the FP64 form.
int derive_basis_tc(mg_ctx* c, int b, bool f64) {
    const Basis& B = c->bas[b];
    const int njobs = 4 * c->p.nwt;
    const int ns[3] = {c->nx, c->ny, c->nz};
    for (int axis = 0; axis < 3; ++axis) {
        const int n = ns[axis];
        TcPass P{};
        P.jobs = B.jobs;
        P.perm = B.job_perm + (long)axis * njobs;
        P.njobs[0] = B.job_slot0[axis];
        P.njobs[1] = njobs - P.njobs[0];
        for (int s = 0; s < 2; ++s) {
            P.bmat[s] = c->tcmats + c->tc_off[f64 ? 1 : 0][axis][s];
            P.erow[s] = c->tc_erow + (axis * 2 + s) * 2 * kMaxLine;
            for (int kind = 0; kind < 2; ++kind) P.mat[kind][s] = c->mats + c->mat_off[axis][kind][s];
        }
        P.axis = axis;
        P.n = n;
        P.nlines = (int)(c->V / n);
        P.tpj = div_up(P.nlines, kTile);
        P.nx = c->nx;
        P.ny = c->ny;
        const auto inverse = [](int d) { return d <= 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); };
        P.tpj_inv = inverse(P.tpj);
        P.nx_inv = inverse(P.nx);
        P.status = c->tc_status;
        const int sms = c->tc_grid_cap > 0 ? std::min(c->tc_grid_cap, c->num_sms) : c->num_sms;
        const int t0 = P.njobs[0] * P.tpj, t1 = P.njobs[1] * P.tpj;
        // one CTA per SM, divided between the slots by their tiles
        int grid = std::min(sms, t0 + t1);
        if (t0 > 0 && t1 > 0) grid = std::max(grid, 2);
        P.ctas0 = (int)(((long)grid * t0 + (t0 + t1) / 2) / (t0 + t1));
        if (t0 > 0) P.ctas0 = std::max(P.ctas0, 1);
        if (t1 > 0) P.ctas0 = std::min(P.ctas0, grid - 1);
        // the y and z passes' set-up (matrix planes, zeroed buffers, TMEM) overlaps
        // the end of the pass before (36 -> 29 us at 10^3 with 40 spwfs); not
        // beside other work, whose SMs the early CTAs would hold
        cudaLaunchAttribute early{};
        early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        early.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem_bytes(n, f64);
        cfg.stream = c->stream;
        cfg.attrs = &early;
        cfg.numAttrs = axis == 0 || c->tc_grid_cap > 0 ? 0 : 1;
        void* args[] = {&P};
        MG_CUDA(cudaLaunchKernelExC(&cfg, kernel_for(f64, kp_of(n), axis == 0), args));
        MG_LAUNCHED(c);
    }
    return MG_OK;
}

int tc_result(mg_ctx* c) {
    volatile int* word = c->h_tc_status;
    if (*word == 0) return MG_OK;
    *word = 0;
    return MG_ERR_TIMEOUT;
}

int sync_results(mg_ctx* c) {
    MG_CUDA(cudaStreamSynchronize(c->stream));
    return tc_result(c);
}

}  // namespace mg
