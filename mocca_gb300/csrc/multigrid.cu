// multigrid.cu -- Coulomb Poisson solve by FP32 multigrid V-cycles inside an
// FP64 iteration (CoulombSolver = 2).
//
// The reference's MGSolve / VCycle / Restrict / Prolong
// (src/MultiGrid.f90:14-348, with Gauss_Seidel_Update
// src/CoulombDerivatives.f90:20-141) are a multigrid for the same problem as
// ConjugGrad: the 4th-order difference Laplacian on the stored box, mirror
// planes at the low end of each axis, the multipole Dirichlet values on the
// two planes beyond the high end (src/Coulomb.f90:255-346, :583-674).  Here
// the multigrid is the preconditioner of a conjugate-gradient iteration
// carried in FP64:
//   - FP64: the residual with the 4th-order operator and the Dirichlet
//     planes, the search directions, the two dot products of an iteration
//     (deterministic block partials summed in a fixed order), the updates of
//     the solution and the residual, the stopping test |r| <= tol |b|;
//   - FP32: one V-cycle per iteration on the 7-point Laplacian of each level
//     (spacing dx 2^l), with red-black Gauss-Seidel smoothing (one sweep red
//     then black before the coarse correction, one black then red after, so
//     the cycle is a symmetric operator), cell-centred restriction
//     R = P^T / 8 (weights 1/8, 3/8, 3/8, 1/8 per axis) and trilinear
//     prolongation P (3/4, 1/4 per axis), the mirror planes and the
//     homogeneous Dirichlet planes of the correction on every level, and a
//     single-block Gauss-Seidel solve of the coarsest level in shared memory.
// Coarsening halves every axis while all of them are even and the halves
// stay >= 3 (64 -> 32 -> 16 -> 8 -> 4, 24 -> 12 -> 6 -> 3); the coarsest
// level must fit the shared-memory solve (4096 points), so an odd line
// length above 16 is refused (MG_ERR_ARG).  The 7-point operator is
// spectrally equivalent to the 4th-order one (ratio between 1 and 4/3), so
// the preconditioned iteration needs few steps whatever the mesh.
//
// The work of an iteration is small (48^3: a few MB through L2); one kernel per
// half sweep, transfer and vector operation, ~40 launches, took 132 us of launch
// and memory latency.  Now a level's way down (both half sweeps from zero, the
// residual, the restriction) is one kernel that keeps a tile with its halo in
// shared memory and computes the halo again instead of exchanging it, its way up
// (prolongation, both half sweeps) another, and the levels of at most kCoarseMax
// points are one block's work in shared memory from end to end.  Directions and
// matrix-vector product share a kernel, updates and stopping test another: 7
// kernels for 48^3, started early (chain.cuh), 52 us an iteration.  Every
// kernel of an iteration first reads the convergence flag and returns once it is
// set; the host reads the flag every kChunk iterations, which replay as one CUDA
// graph, while the next ones run.
#include <algorithm>
#include <cmath>
#include <vector>

#include "chain.cuh"
#include "mg_internal.cuh"

namespace mg {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxLevels = 8;
constexpr int kChunk = 4;           // iterations between host checks of the flag (even)
static_assert(kChunk % 2 == 0);
constexpr int kCoarseMax = 4096;    // points of a level solved in one block's shared memory
constexpr int kCoarseThreads = 1024;
constexpr int kMatrixMax = 1024;    // points of a coarsest level whose sweeps are one matrix
constexpr int kTile = 8;            // edge of a block's cells on the levels above
constexpr int kTileThreads = 288;   // two of the 12 x 12 columns of a tile with a halo of 2
constexpr int kDirDepth = 4;        // ... of k_pcg_direction along z
constexpr int kDirThreads = kTile * kTile * kDirDepth;
constexpr int kPartBlocks = 256;    // blocks of the FP64 dot products
static_assert(kPartBlocks == kThreads);

struct Level {
    int n[3];
    long V;
    float inv_h2;
    float *u, *f, *r;
};

struct PcgScalars {
    int conv;       // 1 once |r| <= tol |b|; 2 when the cap is reached first
    int iters;      // iterations run
    double bb;      // |b|^2
    double rz_old;  // r.z of the previous iteration
    double rr;      // |r|^2 of the last iteration
    unsigned ticket;   // blocks of the update that are done
};

// The levels one block solves, the finest first.
struct CoarseLevels {
    int count;
    int sweeps;                 // of the last one
    int n[kMaxLevels][3];
    uint32_t inv[kMaxLevels][2];   // ceil(2^32 / nx), ceil(2^32 / (nx ny))
    int parts[kMaxLevels];      // threads per column (0: columns per thread)
    float inv_h2[kMaxLevels];
    int at[kMaxLevels];         // the level's arrays in shared memory
};

// One Gauss-Seidel value of A u = f at cell (i, j, k): g = f / inv_h2, nb the sum of the
// neighbours.  Low end: mirror (the neighbour is the cell itself); high end: zero.
__device__ __forceinline__ float gs_value(float g, float nb, int i, int j, int k) {
    return (g - nb) / (float)((i == 0) + (j == 0) + (k == 0) - 6);
}

// Sum of the neighbours of u[at] (strides 1, sy, sz); cells outside the box hold zero.
__device__ __forceinline__ float neighbours(const float* u, int at, int sy, int sz) {
    return u[at - 1] + u[at + 1] + u[at - sy] + u[at + sy] + u[at - sz] + u[at + sz];
}

// f - A u at u[at], which is cell (i, j, k)
__device__ __forceinline__ float residual(const float* u, float f, float inv_h2, int at, int sy,
                                          int sz, int i, int j, int k) {
    const float c = u[at];
    float a = -6.0f * c;
    a += i > 0 ? u[at - 1] : c;
    a += u[at + 1];
    a += j > 0 ? u[at - sy] : c;
    a += u[at + sy];
    a += k > 0 ? u[at - sz] : c;
    a += u[at + sz];
    return f - inv_h2 * a;
}

// per-axis restriction weights of coarse c: fine 2c-1 .. 2c+2 (P^T / 2)
__device__ __forceinline__ void rweights(int c, int nf, float* w) {
    w[0] = c > 0 ? 0.125f : 0.0f;
    w[1] = c > 0 ? 0.375f : 0.5f;
    w[2] = 0.375f;
    w[3] = 2 * c + 2 < nf ? 0.125f : 0.0f;
}

// Restriction: fine cell a of coarse (I, J, K)'s 4 x 4 x 4 is r[at + ax[a0] + ay[a1] + az[a2]].
__device__ __forceinline__ float restricted(const float* r, const int* ax, const int* ay,
                                            const int* az, const float* wx, const float* wy,
                                            const float* wz) {
    float s = 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            float sr = 0.0f;
#pragma unroll
            for (int a = 0; a < 4; ++a) sr = fmaf(wx[a], r[ax[a] + ay[b] + az[c]], sr);
            s = fmaf(wy[b] * wz[c], sr, s);
        }
    return s;
}

// per-axis prolongation of fine f: coarse f/2 (3/4) and its neighbour on the
// side of f (1/4); the low-end neighbour is the mirror image, the high-end
// one the zero Dirichlet value
__device__ __forceinline__ void pweights(int f, int nc, int* ci, float* w) {
    const int c = f >> 1;
    ci[0] = c;
    w[0] = 0.75f;
    if (f & 1) {
        ci[1] = c + 1 < nc ? c + 1 : c;
        w[1] = c + 1 < nc ? 0.25f : 0.0f;
    } else {
        ci[1] = c > 0 ? c - 1 : 0;
        w[1] = 0.25f;
    }
}

// Prolongation at fine cell (i, j, k) from coarse values uc (strides 1, sy, sz; cell
// (x, y, z) at uc[x - x0 + ...]).
__device__ __forceinline__ float prolonged(const float* uc, int sy, int sz, int x0, int y0, int z0,
                                           int i, int j, int k, const int* nc) {
    int ix[2], iy[2], iz[2];
    float wx[2], wy[2], wz[2];
    pweights(i, nc[0], ix, wx);
    pweights(j, nc[1], iy, wy);
    pweights(k, nc[2], iz, wz);
    float s = 0.0f;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int a = 0; a < 2; ++a)
                s = fmaf(wx[a] * wy[b] * wz[c],
                         uc[ix[a] - x0 + sy * (iy[b] - y0) + sz * (iz[c] - z0)], s);
    return s;
}

struct Box {
    int n[3];
};

__device__ __forceinline__ bool inside(int i, int j, int k, const int* n) {
    return (unsigned)i < (unsigned)n[0] && (unsigned)j < (unsigned)n[1] && (unsigned)k < (unsigned)n[2];
}

// The passes of a tile kernel: fn(a, b, first, step) on the columns of the square [o,
// o + R) in x and y, for the planes (or pairs of planes) first, first + step, ...
// A thread keeps its column: the box, the mirrors and the colour along x and y are
// worked out once, and a half sweep takes the cell of its colour out of each pair of
// planes, so that no lane waits for the other colour.
template <int R, class F>
__device__ __forceinline__ void columns(int o, F fn) {
    constexpr int parts = kTileThreads / (R * R);
    const int col = threadIdx.x % (R * R), part = threadIdx.x / (R * R);
    if (part < parts) fn(o + col % R, o + col / R, part, parts);
}

// A level's way down: u = one red, one black half sweep from zero, fc = the
// restricted residual.  A block's cells are 8^3 of the level and the 4^3 coarse
// ones below them; f comes with a halo of 3, for red there, black at 2, the residual
// at 1 (5 times the block's own work, all of it small beside a launch).
__global__ void __launch_bounds__(kTileThreads)
k_mg_down(const float* __restrict__ f, float* __restrict__ u, float* __restrict__ fc, Box N, Box C,
          float inv_h2, const int* __restrict__ conv) {
    constexpr int E = kTile + 6, S2 = E * E, B = kTile + 4, R = kTile + 2;
    __shared__ float sf[E * S2], su[E * S2], sr[R * R * R];
    chain_wait();
    if (*conv) return;
    const int x0 = blockIdx.x * kTile - 3, y0 = blockIdx.y * kTile - 3, z0 = blockIdx.z * kTile - 3;
    const int* n = N.n;
    const long sy = n[0], sz = (long)n[0] * n[1];
    columns<E>(0, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        const bool in = inside(i, j, 0, n);
        const float* col = f + i + sy * j;
        float x[E];
#pragma unroll
        for (int c = 0; c < E; ++c)
            x[c] = in && (unsigned)(z0 + c) < (unsigned)n[2] ? col[sz * (z0 + c)] : 0.0f;
        const int odd = (i + j + z0) & 1;   // the red cell of a pair
#pragma unroll
        for (int c = 0; c < E; c += 2) {
            const int k = z0 + c + odd, at = a + E * b + S2 * c;
            const float v = gs_value((odd ? x[c + 1] : x[c]) / inv_h2, 0.0f, i, j, k);
            sf[at] = x[c];
            sf[at + S2] = x[c + 1];
            su[at] = odd ? 0.0f : v;   // zero outside, where f is
            su[at + S2] = odd ? v : 0.0f;
        }
    });
    __syncthreads();
    columns<B>(1, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        if (!inside(i, j, 0, n)) return;
        const int odd = (i + j + z0) & 1;   // planes 1 + 2m, 2 + 2m: the black one
        for (int c = 1 + odd + 2 * first; c < B + 1; c += 2 * step) {
            const int k = z0 + c, at = a + E * b + S2 * c;
            if ((unsigned)k < (unsigned)n[2])
                su[at] = gs_value(sf[at] / inv_h2, neighbours(su, at, E, S2), i, j, k);
        }
    });
    __syncthreads();
    columns<R>(2, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        const bool in = inside(i, j, 0, n);
        for (int c = 2 + first; c < R + 2; c += step) {
            const int k = z0 + c, at = a + E * b + S2 * c;
            sr[a - 2 + R * (b - 2 + R * (c - 2))] =
                in && (unsigned)k < (unsigned)n[2]
                    ? residual(su, sf[at], inv_h2, at, E, S2, i, j, k) : 0.0f;
        }
    });
    columns<kTile>(3, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        if (!inside(i, j, 0, n)) return;
        for (int c = 3 + first; c < kTile + 3; c += step)
            if (z0 + c < n[2]) u[i + sy * j + sz * (z0 + c)] = su[a + E * b + S2 * c];
    });
    __syncthreads();
    constexpr int H = kTile / 2;
    if (threadIdx.x < H * H * H) {
        const int a = threadIdx.x % H, b = threadIdx.x / H % H, c = threadIdx.x / (H * H);
        const int I = blockIdx.x * H + a, J = blockIdx.y * H + b, K = blockIdx.z * H + c;
        if (inside(I, J, K, C.n)) {
            float wx[4], wy[4], wz[4];
            rweights(I, n[0], wx);
            rweights(J, n[1], wy);
            rweights(K, n[2], wz);
            int ax[4], ay[4], az[4];
            // sr starts at fine -1 of the block, so fine 2c - 1 of coarse a is 2a
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ax[q] = 2 * a + q;
                ay[q] = R * (2 * b + q);
                az[q] = R * R * (2 * c + q);
            }
            fc[I + (long)C.n[0] * (J + (long)C.n[1] * K)] = restricted(sr, ax, ay, az, wx, wy, wz);
        }
    }
}

// Sum of the count values at x (shared or global memory) by one warp, the same in
// all its lanes: a lane adds every 32nd one.  FP64 adds are scarce (a warp's takes 16
// clocks of the SM), so a block's sum is not made by shuffles in every warp.
__device__ __forceinline__ double warp_total(const double* x, int count) {
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q = threadIdx.x & 31; q < count; q += 128)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (q + 32 * u < count) a[u] += x[q + 32 * u];
    double s = (a[0] + a[1]) + (a[2] + a[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Sum over the block (sh: one word a thread), on the threads of warp 0.
__device__ __forceinline__ double block_reduce(double x, double* sh) {
    sh[threadIdx.x] = x;
    __syncthreads();
    return threadIdx.x < 32 ? warp_total(sh, blockDim.x) : 0.0;
}

// A level's way up: u + P uc, one black and one red half sweep; to out, or on the
// finest level (kFinest) to z in FP64 with the block's partial of r.z.  Halos: u and
// the coarse correction 2, black 1.
template <bool kFinest>
__global__ void __launch_bounds__(kTileThreads)
k_mg_up(const float* __restrict__ u, const float* __restrict__ f, const float* __restrict__ uc,
        Box N, Box C, float inv_h2, float* __restrict__ out, double* __restrict__ z,
        const double* __restrict__ r, double* __restrict__ part, const int* __restrict__ conv) {
    constexpr int E = kTile + 4, S2 = E * E, G = kTile + 2, P = kTile / 2 + 4;
    constexpr int parts = kTileThreads / S2, depth = E / parts;
    static_assert(parts * depth == E);
    __shared__ float su[E * S2], sg[G * G * G], sc[P * P * P];
    __shared__ double sh[kTileThreads];
    chain_wait();
    if (*conv) return;
    const int x0 = blockIdx.x * kTile - 2, y0 = blockIdx.y * kTile - 2, z0 = blockIdx.z * kTile - 2;
    const int X0 = x0 / 2 - 1, Y0 = y0 / 2 - 1, Z0 = z0 / 2 - 1;   // x0, y0, z0 are even
    const int* n = N.n;
    const long sy = n[0], sz = (long)n[0] * n[1];
    for (int t = threadIdx.x; t < P * P * P; t += kTileThreads) {
        const int I = X0 + t % P, J = Y0 + t / P % P, K = Z0 + t / (P * P);
        sc[t] = inside(I, J, K, C.n) ? uc[I + (long)C.n[0] * (J + (long)C.n[1] * K)] : 0.0f;
    }
    columns<G>(1, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        const bool in = inside(i, j, 0, n);
        const float* col = f + i + sy * j;
#pragma unroll
        for (int c = 1 + first; c < G + 1; c += kTileThreads / (G * G))
            sg[a - 1 + G * (b - 1 + G * (c - 1))] =
                in && (unsigned)(z0 + c) < (unsigned)n[2] ? col[sz * (z0 + c)] : 0.0f;
    });
    float mine[depth];
    columns<E>(0, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        const bool in = inside(i, j, 0, n);
        const float* col = u + i + sy * j;
#pragma unroll
        for (int m = 0; m < depth; ++m) {
            const int k = z0 + first + m * parts;
            mine[m] = in && (unsigned)k < (unsigned)n[2] ? col[sz * k] : 0.0f;
        }
    });
    // r at the two cells of this thread's column (below)
    double rv[2] = {0.0, 0.0};
    if (kFinest)
        columns<kTile>(2, [&](int a, int b, int first, int step) {
            const int i = x0 + a, j = y0 + b;
            if (!inside(i, j, 0, n)) return;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int k = z0 + 2 + 2 * first + m;
                if (k < n[2]) rv[m] = r[i + sy * j + sz * k];
            }
        });
    __syncthreads();
    columns<E>(0, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        const bool in = inside(i, j, 0, n);
        int ix[2], iy[2];
        float wx[2], wy[2];
        pweights(i, C.n[0], ix, wx);
        pweights(j, C.n[1], iy, wy);
        const float w[2][2] = {{wx[0] * wy[0], wx[1] * wy[0]}, {wx[0] * wy[1], wx[1] * wy[1]}};
        // the place of column (ix, iy) in sc, held inside it for a cell outside the box
        const int px[2] = {min(max(ix[0] - X0, 0), P - 1), min(max(ix[1] - X0, 0), P - 1)};
        const int py[2] = {P * min(max(iy[0] - Y0, 0), P - 1), P * min(max(iy[1] - Y0, 0), P - 1)};
#pragma unroll
        for (int m = 0; m < depth; ++m) {
            const int c = first + m * parts, k = z0 + c;
            float x = 0.0f;
            if (in && (unsigned)k < (unsigned)n[2]) {
                int iz[2];
                float wz[2];
                pweights(k, C.n[2], iz, wz);
#pragma unroll
                for (int cc = 0; cc < 2; ++cc)
#pragma unroll
                    for (int bb = 0; bb < 2; ++bb)
#pragma unroll
                        for (int aa = 0; aa < 2; ++aa)
                            x = fmaf(w[bb][aa] * wz[cc], sc[px[aa] + py[bb] + P * P * (iz[cc] - Z0)],
                                     x);
                x += mine[m];
            }
            su[a + E * b + S2 * c] = x;
        }
    });
    __syncthreads();
    columns<G>(1, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        if (!inside(i, j, 0, n)) return;
        const int odd = (i + j + z0) & 1;   // planes 1 + 2m, 2 + 2m: the black one
        for (int c = 1 + odd + 2 * first; c < G + 1; c += 2 * step) {
            const int k = z0 + c, at = a + E * b + S2 * c;
            if ((unsigned)k < (unsigned)n[2])
                su[at] = gs_value(sg[a - 1 + G * (b - 1 + G * (c - 1))] / inv_h2,
                                  neighbours(su, at, E, S2), i, j, k);
        }
    });
    __syncthreads();
    double loc = 0.0;
    columns<kTile>(2, [&](int a, int b, int first, int step) {
        const int i = x0 + a, j = y0 + b;
        if (!inside(i, j, 0, n)) return;
        const int odd = (i + j + z0) & 1;   // planes 2 + 2m, 3 + 2m: the red one
        static_assert(kTileThreads / (kTile * kTile) == kTile / 2);   // one pair a thread
        const int c0 = 2 + 2 * first, cr = c0 + odd;
        const int at = a + E * b + S2 * cr;
        float v[2] = {su[a + E * b + S2 * c0], su[a + E * b + S2 * (c0 + 1)]};
        const float red = gs_value(sg[a - 1 + G * (b - 1 + G * (cr - 1))] / inv_h2,
                                   neighbours(su, at, E, S2), i, j, z0 + cr);
        v[0] = odd ? v[0] : red;
        v[1] = odd ? red : v[1];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int k = z0 + c0 + m;
            if (k >= n[2]) continue;
            const long o = i + sy * j + sz * k;
            if (kFinest) {
                z[o] = (double)v[m];
                loc = fma(rv[m], (double)v[m], loc);
            } else {
                out[o] = v[m];
            }
        }
    });
    if (kFinest) {
        const double s = block_reduce(loc, sh);
        if (threadIdx.x == 0)
            part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = s;
    }
}

// The coarsest level's sweeps from u = 0 are linear in f: column blockIdx.x of their
// matrix (row-major), by the sweeps of one block on a unit vector.
__global__ void __launch_bounds__(kThreads)
k_mg_sweep_matrix(Box N, float inv_h2, int sweeps, float* __restrict__ mat) {
    extern __shared__ float su[];
    const int nx = N.n[0], ny = N.n[1], nz = N.n[2], V = nx * ny * nz;
    const int sy = nx + 2, sz = sy * (ny + 2);
    for (int t = threadIdx.x; t < sz * (nz + 2); t += kThreads) su[t] = 0.0f;
    __syncthreads();
    for (int s = 0; s < 2 * sweeps; ++s) {
        for (int v = threadIdx.x; v < V; v += kThreads) {
            const int i = v % nx, j = v / nx % ny, k = v / (nx * ny);
            if (((i + j + k) & 1) != (s & 1)) continue;
            const int at = i + 1 + sy * (j + 1) + sz * (k + 1);
            const float g = (v == (int)blockIdx.x ? 1.0f : 0.0f) / inv_h2;
            su[at] = gs_value(g, neighbours(su, at, sy, sz), i, j, k);
        }
        __syncthreads();
    }
    for (int v = threadIdx.x; v < V; v += kThreads)
        mat[(long)v * V + blockIdx.x] = su[v % nx + 1 + sy * (v / nx % ny + 1) + sz * (v / (nx * ny) + 1)];
}

// Way down, coarsest solve and way up of the levels of at most kCoarseMax points,
// in shared memory: per level f, the residual, and u in a frame of zeros.  The
// coarsest level's sweeps are 36 dependent half sweeps even for 3^3: up to kMatrixMax
// points they are one product with their matrix (k_mg_sweep_matrix), a warp per row
// (at the limit 4 MB through L2, ~20 us, against ~60 of sweeps).
__global__ void __launch_bounds__(kCoarseThreads)
k_mg_coarse(const float* __restrict__ f, float* __restrict__ out, CoarseLevels L, int floats,
            const float* __restrict__ mat, const int* __restrict__ conv) {
    extern __shared__ float sm[];
    chain_wait();
    if (*conv) return;
    const int tid = threadIdx.x;
    const auto volume = [&](int l) { return L.n[l][0] * L.n[l][1] * L.n[l][2]; };
    // fn(v, place in u, i, j, k) over the cells of level l of colour c (-1: all): a
    // thread takes a column's planes (pairs of planes) first, first + step, ...
    const auto cells = [&](int l, int c, auto fn) {
        const int nx = L.n[l][0], ny = L.n[l][1], nz = L.n[l][2], ncol = nx * ny;
        const int part = ncol > 1 ? (int)__umulhi((uint32_t)tid, L.inv[l][1]) : tid;
        const int parts = max(1, L.parts[l]);
        if (L.parts[l] > 0 && part >= parts) return;
        for (int col = L.parts[l] > 0 ? tid - part * ncol : tid; col < ncol; col += kCoarseThreads) {
            const int j = nx > 1 ? (int)__umulhi((uint32_t)col, L.inv[l][0]) : col, i = col - j * nx;
            const int step = c < 0 ? parts : 2 * parts;
            int k = L.parts[l] > 0 ? part : 0;
            if (c >= 0) k = 2 * k + ((i + j + c) & 1);
            for (; k < nz; k += step)
                fn(col + ncol * k, i + 1 + (nx + 2) * (j + 1 + (ny + 2) * (k + 1)), i, j, k);
        }
    };
    const int V0 = volume(0);
    for (int t = tid; t < floats; t += kCoarseThreads) sm[t] = t < V0 ? f[t] : 0.0f;
    __syncthreads();
    for (int l = 0; l + 1 < L.count; ++l) {
        const int* n = L.n[l];
        const int V = volume(l), sy = n[0] + 2, sz = sy * (n[1] + 2);
        const float inv_h2 = L.inv_h2[l];
        float *sf = sm + L.at[l], *r = sf + V, *u = r + V;
        cells(l, 0, [&](int v, int at, int i, int j, int k) {
            u[at] = gs_value(sf[v] / inv_h2, 0.0f, i, j, k);
        });
        __syncthreads();
        cells(l, 1, [&](int v, int at, int i, int j, int k) {
            u[at] = gs_value(sf[v] / inv_h2, neighbours(u, at, sy, sz), i, j, k);
        });
        __syncthreads();
        cells(l, -1, [&](int v, int at, int i, int j, int k) {
            r[v] = residual(u, sf[v], inv_h2, at, sy, sz, i, j, k);
        });
        __syncthreads();
        float* fc = sm + L.at[l + 1];
        cells(l + 1, -1, [&](int v, int, int I, int J, int K) {
            float wx[4], wy[4], wz[4];
            rweights(I, n[0], wx);
            rweights(J, n[1], wy);
            rweights(K, n[2], wz);
            int ax[4], ay[4], az[4];
            // a cell outside the box has weight zero
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ax[q] = min(max(2 * I - 1 + q, 0), n[0] - 1);
                ay[q] = n[0] * min(max(2 * J - 1 + q, 0), n[1] - 1);
                az[q] = n[0] * n[1] * min(max(2 * K - 1 + q, 0), n[2] - 1);
            }
            fc[v] = restricted(r, ax, ay, az, wx, wy, wz);
        });
        __syncthreads();
    }
    {
        const int l = L.count - 1, V = volume(l), nx = L.n[l][0], ny = L.n[l][1];
        const int sy = nx + 2, sz = sy * (ny + 2);
        const float inv_h2 = L.inv_h2[l];
        float *sf = sm + L.at[l], *u = sf + 2 * V;
        if (mat) {
            const int lane = tid & 31;
            for (int v = tid >> 5; v < V; v += kCoarseThreads / 32) {
                const float* row = mat + (long)v * V;
                float x = 0.0f;
#pragma unroll 4
                for (int q = lane; q < V; q += 32) x = fmaf(row[q], sf[q], x);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                const int k = v / (nx * ny), j = v / nx % ny, i = v % nx;
                if (lane == 0) u[i + 1 + sy * (j + 1) + sz * (k + 1)] = x;
            }
        } else {
            for (int s = 0; s < 2 * L.sweeps; ++s) {
                cells(l, s & 1, [&](int v, int at, int i, int j, int k) {
                    u[at] = gs_value(sf[v] / inv_h2, neighbours(u, at, sy, sz), i, j, k);
                });
                __syncthreads();
            }
        }
        __syncthreads();
    }
    for (int l = L.count - 2; l >= 0; --l) {
        const int *n = L.n[l], *nc = L.n[l + 1];
        const int V = volume(l), sy = n[0] + 2, sz = sy * (n[1] + 2);
        const int cy = nc[0] + 2, cz = cy * (nc[1] + 2);
        const float inv_h2 = L.inv_h2[l];
        float *sf = sm + L.at[l], *u = sf + 2 * V;
        const float* uc = sm + L.at[l + 1] + 2 * volume(l + 1);
        cells(l, -1, [&](int, int at, int i, int j, int k) {
            u[at] += prolonged(uc, cy, cz, -1, -1, -1, i, j, k, nc);
        });
        __syncthreads();
        for (int color = 1; color >= 0; --color) {
            cells(l, color, [&](int v, int at, int i, int j, int k) {
                u[at] = gs_value(sf[v] / inv_h2, neighbours(u, at, sy, sz), i, j, k);
            });
            __syncthreads();
        }
    }
    const float* u = sm + L.at[0] + 2 * V0;
    cells(0, -1, [&](int v, int at, int, int, int) { out[v] = u[at]; });
}

// z in FP64 and the partials of r.z where the finest level is one block's
__global__ void __launch_bounds__(kThreads)
k_mg_out(const float* __restrict__ u, const double* __restrict__ r, double* __restrict__ z, long V,
         double* __restrict__ part, const int* __restrict__ conv) {
    __shared__ double sh[kThreads];
    chain_wait();
    if (*conv) return;
    double loc = 0.0;
    for (long v = (long)blockIdx.x * kThreads + threadIdx.x; v < V; v += (long)gridDim.x * kThreads) {
        z[v] = (double)u[v];
        loc = fma(r[v], z[v], loc);
    }
    const double s = block_reduce(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// ---- FP64 preconditioned conjugate gradients --------------------------------

// |b|^2 over the stored box (b: the source), and the state reset
__global__ void __launch_bounds__(kThreads)
k_pcg_start(const double* __restrict__ src, int nx, int ny, int nz, int mx, int my,
            double* __restrict__ e, double* __restrict__ p, double* __restrict__ part) {
    __shared__ double sh[kThreads];
    const long V = (long)nx * ny * nz;
    double loc = 0.0;
    for (long v = (long)blockIdx.x * kThreads + threadIdx.x; v < V;
         v += (long)kPartBlocks * kThreads) {
        const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
        const double s = src[i + mx * (j + (long)my * k)];
        loc = fma(s, s, loc);
        e[v] = 0.0;
        p[v] = 0.0;
    }
    const double s = block_reduce(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void __launch_bounds__(32)
k_pcg_init_scalars(const double* __restrict__ part, PcgScalars* __restrict__ S) {
    const double bb = warp_total(part, kPartBlocks);
    if (threadIdx.x == 0) {
        S->conv = bb == 0.0 ? 1 : 0;
        S->iters = 0;
        S->bb = bb;
        S->rz_old = 1.0;
        S->rr = 0.0;
        S->ticket = 0;
    }
}

// p = z + beta p_old, beta = rz / rz_old (0 on the first iteration), q = L p (the
// 4th-order Laplacian, zero on the Dirichlet planes, mirrors at the low ends) and the
// partials of p.q.  A block makes p on its 8 x 8 x 4 cells and their two neighbours on
// each side of an axis, so the new p goes to another buffer than p_old.  Bound by the
// FP64 pipe, hence the scalars in one warp.
__global__ void __launch_bounds__(kDirThreads)
k_pcg_direction(const double* __restrict__ z, const double* __restrict__ p_old,
                double* __restrict__ p, double* __restrict__ q, Box N, double inv_dx2,
                const double* __restrict__ part_rz, int n_rz, double* __restrict__ part_pq,
                const PcgScalars* __restrict__ S) {
    constexpr int E = kTile + 4, S2 = E * E, D = kDirDepth + 4;
    __shared__ double sp[D * S2];
    __shared__ double sh[kDirThreads];
    __shared__ double sbeta;
    chain_wait();
    if (S->conv) return;
    const int* n = N.n;
    const int x0 = blockIdx.x * kTile - 2, y0 = blockIdx.y * kTile - 2,
              z0 = blockIdx.z * kDirDepth - 2;
    // the words come in while warp 0 makes beta
    constexpr int kWords = (D * S2 + kDirThreads - 1) / kDirThreads;
    double zw[kWords], pw[kWords];
#pragma unroll
    for (int m = 0; m < kWords; ++m) {
        const int t = threadIdx.x + m * kDirThreads;
        const int a = t % E, b = t / E % E, c = t / S2;
        const int out = (a < 2 || a >= kTile + 2) + (b < 2 || b >= kTile + 2) +
                        (c < 2 || c >= kDirDepth + 2);
        int i = x0 + a, j = y0 + b, k = z0 + c;
        i = i < 0 ? -i - 1 : i;
        j = j < 0 ? -j - 1 : j;
        k = k < 0 ? -k - 1 : k;
        zw[m] = 0.0;
        pw[m] = 0.0;
        if (out <= 1 && i < n[0] && j < n[1] && k < n[2]) {
            const long v = i + (long)n[0] * (j + (long)n[1] * k);
            zw[m] = z[v];
            pw[m] = p_old[v];
        }
    }
    if (threadIdx.x < 32) {
        const double rz = warp_total(part_rz, n_rz);
        if (threadIdx.x == 0) sbeta = S->iters == 0 ? 0.0 : rz / S->rz_old;
    }
    __syncthreads();
    const double beta = sbeta;
#pragma unroll
    for (int m = 0; m < kWords; ++m) {
        const int t = threadIdx.x + m * kDirThreads;
        if (t < D * S2) sp[t] = fma(beta, pw[m], zw[m]);
    }
    __syncthreads();
    const int a = threadIdx.x % kTile + 2, b = threadIdx.x / kTile % kTile + 2,
              c = threadIdx.x / (kTile * kTile) + 2;
    const int i = x0 + a, j = y0 + b, k = z0 + c;
    double loc = 0.0;
    if (inside(i, j, k, n)) {
        const int at = a + E * b + S2 * c;
        const double cf[5] = {-1.0 / 12.0, 4.0 / 3.0, -5.0 / 2.0, 4.0 / 3.0, -1.0 / 12.0};
        double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll
        for (int w = -2; w <= 2; ++w) {
            ax = fma(cf[w + 2], sp[at + w], ax);
            ay = fma(cf[w + 2], sp[at + w * E], ay);
            az = fma(cf[w + 2], sp[at + w * S2], az);
        }
        const double x = ax * inv_dx2 + ay * inv_dx2 + az * inv_dx2;
        const long v = i + (long)n[0] * (j + (long)n[1] * k);
        p[v] = sp[at];
        q[v] = x;
        loc = sp[at] * x;
    }
    const double s = block_reduce(loc, sh);
    if (threadIdx.x == 0)
        part_pq[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = s;
}

// alpha = rz / pq; e += alpha p; r -= alpha q, also to f in FP32 for the next cycle;
// partials of r.r, and by the last block to come the stopping test.
__global__ void __launch_bounds__(kThreads)
k_pcg_update(double* __restrict__ e, double* __restrict__ r, const double* __restrict__ p,
             const double* __restrict__ q, float* __restrict__ f, long V,
             const double* __restrict__ part_rz, int n_rz, const double* __restrict__ part_pq,
             int n_pq, double* part_rr, double tol2, int maxit, PcgScalars* S) {
    __shared__ double sh[kThreads];
    __shared__ double total[2], salpha;
    __shared__ bool last;
    chain_wait();
    if (S->conv) return;
    // the first words come in while two warps make alpha
    long v = (long)blockIdx.x * kThreads + threadIdx.x;
    bool have = v < V;
    double pv = 0.0, qv = 0.0, ev = 0.0, xv = 0.0;
    if (have) {
        pv = p[v];
        qv = q[v];
        ev = e[v];
        xv = r[v];
    }
    if (threadIdx.x < 64) {   // warp 0 the r.z, warp 1 the p.q
        const bool first = threadIdx.x < 32;
        const double t = warp_total(first ? part_rz : part_pq, first ? n_rz : n_pq);
        if (threadIdx.x % 32 == 0) total[threadIdx.x / 32] = t;
    }
    __syncthreads();
    const double rz = total[0];
    if (threadIdx.x == 0) salpha = rz / total[1];
    __syncthreads();
    const double alpha = salpha;
    double loc = 0.0;
    for (; v < V; v += (long)kPartBlocks * kThreads) {
        if (!have) {
            pv = p[v];
            qv = q[v];
            ev = e[v];
            xv = r[v];
        }
        have = false;
        e[v] = fma(alpha, pv, ev);
        const double x = fma(-alpha, qv, xv);
        r[v] = x;
        f[v] = (float)x;
        loc = fma(x, x, loc);
    }
    const double s = block_reduce(loc, sh);
    if (threadIdx.x == 0) {
        part_rr[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(&S->ticket, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    __syncthreads();
    sh[threadIdx.x] = __ldcg(part_rr + threadIdx.x);   // kPartBlocks = kThreads of them
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const double rr = warp_total(sh, kPartBlocks);
    if (threadIdx.x == 0) {
        S->ticket = 0;
        S->rz_old = rz;
        S->rr = rr;
        S->iters += 1;
        if (rr <= tol2 * S->bb) S->conv = 1;
        else if (S->iters >= maxit) S->conv = 2;
    }
}

__global__ void k_pcg_finish(double* __restrict__ sol, const double* __restrict__ e, int nx,
                             int ny, int nz, int mx, int my) {
    const long V = (long)nx * ny * nz;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
    sol[i + mx * (j + (long)my * k)] += e[v];
}

// r = src - L sol on the stored box, with sol's Dirichlet planes
__global__ void k_pcg_residual(const double* __restrict__ sol, const double* __restrict__ src,
                               double* __restrict__ r, float* __restrict__ f, int nx, int ny,
                               int nz, int mx, int my, double inv_dx2) {
    const long V = (long)nx * ny * nz;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
    const double cf[5] = {-1.0 / 12.0, 4.0 / 3.0, -5.0 / 2.0, 4.0 / 3.0, -1.0 / 12.0};
    double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll
    for (int q = -2; q <= 2; ++q) {
        const int ii = i + q < 0 ? -(i + q) - 1 : i + q;
        const int jj = j + q < 0 ? -(j + q) - 1 : j + q;
        const int kk = k + q < 0 ? -(k + q) - 1 : k + q;
        ax = fma(cf[q + 2], sol[ii + mx * (j + (long)my * k)], ax);
        ay = fma(cf[q + 2], sol[i + mx * (jj + (long)my * k)], ay);
        az = fma(cf[q + 2], sol[i + mx * (j + (long)my * kk)], az);
    }
    const double x = src[i + mx * (j + (long)my * k)] - (ax * inv_dx2 + ay * inv_dx2 + az * inv_dx2);
    r[v] = x;
    f[v] = (float)x;   // of the first cycle
}

}  // namespace

// Multigrid hierarchy and FP64 work vectors of one context.
struct Multigrid {
    int nlev = 0;
    Level lev[kMaxLevels];
    int first_coarse = 0;               // this level and the ones below: k_mg_coarse
    CoarseLevels coarse{};
    size_t coarse_smem = 0;
    float* mat = nullptr;               // the coarsest level's sweeps, or nullptr
    float* f32 = nullptr;               // every level's u, f, r
    double *r = nullptr, *z = nullptr, *q = nullptr, *e = nullptr;
    double* p[2] = {nullptr, nullptr};  // directions, old and new in turn
    double* part = nullptr;             // 3 x n_part partials (r.z, p.q, r.r)
    int n_part = 0, n_rz = 0, n_pq = 0;
    PcgScalars* S = nullptr;
    PcgScalars* h_S = nullptr;          // pinned, of two chunks in turn
    cudaEvent_t read[2] = {nullptr, nullptr};   // ... has come
    cudaGraphExec_t chunk = nullptr;    // kChunk iterations, captured on first use
    double tol2 = 0.0;                  // ... for this tolerance and cap
    int maxit = 0;
    long long chunk_launches = 0;
    bool no_graph = false;
};

void multigrid_free(Multigrid* M) {
    if (!M) return;
    for (void* p : {(void*)M->f32, (void*)M->mat, (void*)M->r, (void*)M->z, (void*)M->p[0], (void*)M->p[1],
                    (void*)M->q, (void*)M->e, (void*)M->part, (void*)M->S})
        if (p) cudaFree(p);
    if (M->h_S) cudaFreeHost(M->h_S);
    for (cudaEvent_t e : M->read)
        if (e) cudaEventDestroy(e);
    if (M->chunk) cudaGraphExecDestroy(M->chunk);
    delete M;
}

static int multigrid_build(mg_ctx* c, Multigrid* M) {
    int n[3] = {c->nx, c->ny, c->nz};
    double h = c->p.dx;
    long total = 0;
    while (M->nlev < kMaxLevels) {
        Level& L = M->lev[M->nlev++];
        for (int a = 0; a < 3; ++a) L.n[a] = n[a];
        L.V = (long)n[0] * n[1] * n[2];
        L.inv_h2 = (float)(1.0 / (h * h));
        total += 3 * L.V;
        const bool even = n[0] % 2 == 0 && n[1] % 2 == 0 && n[2] % 2 == 0;
        const bool room = n[0] / 2 >= 3 && n[1] / 2 >= 3 && n[2] / 2 >= 3;
        if (!(even && room)) break;
        for (int a = 0; a < 3; ++a) n[a] /= 2;
        h *= 2.0;
    }
    // the last level is solved in shared memory
    if (M->lev[M->nlev - 1].V > kCoarseMax) return MG_ERR_ARG;
    const Level& C = M->lev[M->nlev - 1];
    const int nm = std::max(C.n[0], std::max(C.n[1], C.n[2]));
    CoarseLevels& K = M->coarse;
    K.sweeps = std::min(200, 2 * nm * nm);
    while (M->lev[M->first_coarse].V > kCoarseMax) ++M->first_coarse;
    K.count = M->nlev - M->first_coarse;
    int floats = 0;
    for (int l = 0; l < K.count; ++l) {
        const Level& L = M->lev[M->first_coarse + l];
        for (int a = 0; a < 3; ++a) K.n[l][a] = L.n[a];
        // exact quotients of cell numbers below 2^16
        K.inv[l][0] = 0xFFFFFFFFu / (uint32_t)L.n[0] + 1u;
        K.inv[l][1] = 0xFFFFFFFFu / (uint32_t)(L.n[0] * L.n[1]) + 1u;
        K.parts[l] = kCoarseThreads / (L.n[0] * L.n[1]);
        K.inv_h2[l] = L.inv_h2;
        K.at[l] = floats;
        floats += 2 * (int)L.V + (L.n[0] + 2) * (L.n[1] + 2) * (L.n[2] + 2);
    }
    M->coarse_smem = floats * sizeof(float);
    MG_CUDA(cudaFuncSetAttribute(k_mg_coarse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)M->coarse_smem));
    M->n_pq = div_up(c->nx, kTile) * div_up(c->ny, kTile) * div_up(c->nz, kDirDepth);
    M->n_rz = M->first_coarse > 0
                  ? div_up(c->nx, kTile) * div_up(c->ny, kTile) * div_up(c->nz, kTile)
                  : kPartBlocks;
    M->n_part = std::max(M->n_pq, kPartBlocks);
    MG_CUDA(cudaMalloc(&M->f32, total * sizeof(float)));
    float* q = M->f32;
    for (int l = 0; l < M->nlev; ++l) {
        Level& L = M->lev[l];
        L.u = q; q += L.V;
        L.f = q; q += L.V;
        L.r = q; q += L.V;
    }
    const long V = c->V;
    for (double** b : {&M->r, &M->z, &M->p[0], &M->p[1], &M->q, &M->e})
        MG_CUDA(cudaMalloc(b, V * sizeof(double)));
    MG_CUDA(cudaMalloc(&M->part, 3 * (size_t)M->n_part * sizeof(double)));
    MG_CUDA(cudaMalloc(&M->S, sizeof(PcgScalars)));
    if (C.V <= kMatrixMax) {
        MG_CUDA(cudaMalloc(&M->mat, (size_t)C.V * C.V * sizeof(float)));
        const size_t frame = (size_t)(C.n[0] + 2) * (C.n[1] + 2) * (C.n[2] + 2) * sizeof(float);
        MG_CUDA(cudaFuncSetAttribute(k_mg_sweep_matrix, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)frame));
        k_mg_sweep_matrix<<<(unsigned)C.V, kThreads, frame, c->stream>>>(
            Box{{C.n[0], C.n[1], C.n[2]}}, C.inv_h2, K.sweeps, M->mat);
        MG_LAUNCHED(c);
    }
    MG_CUDA(cudaMallocHost(&M->h_S, 2 * sizeof(PcgScalars)));
    for (cudaEvent_t& e : M->read) MG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return MG_OK;
}

// The context's hierarchy; none when it cannot be had (MG_ERR_ARG: a mesh without one).
static int multigrid_setup(mg_ctx* c) {
    Multigrid* M = new Multigrid();
    const int st = multigrid_build(c, M);
    if (st != MG_OK) {
        multigrid_free(M);
        return st;
    }
    c->mgrid = M;
    return MG_OK;
}

static dim3 tiles_of(const int* n) {
    return dim3(div_up(n[0], kTile), div_up(n[1], kTile), div_up(n[2], kTile));
}

static Box box_of(const Level& L) { return Box{{L.n[0], L.n[1], L.n[2]}}; }

// One V-cycle from the finest level's f: z = M^{-1} r (FP32 inside) and the partials
// of r.z.  A level's result is in its r.
static int vcycle(mg_ctx* c, Multigrid* M, double* p_rz) {
    const int* conv = &M->S->conv;
    const int fc = M->first_coarse;
    for (int l = 0; l < fc; ++l) {
        const Level &L = M->lev[l], &C = M->lev[l + 1];
        MG_TRY(launch_early(c, k_mg_down, tiles_of(L.n), kTileThreads, 0, L.f, L.u, C.f, box_of(L),
                            box_of(C), L.inv_h2, conv));
    }
    MG_TRY(launch_early(c, k_mg_coarse, dim3(1), kCoarseThreads, M->coarse_smem, M->lev[fc].f,
                        M->lev[fc].r, M->coarse, (int)(M->coarse_smem / sizeof(float)), M->mat, conv));
    for (int l = fc - 1; l >= 0; --l) {
        const Level &L = M->lev[l], &C = M->lev[l + 1];
        MG_TRY(launch_early(c, l == 0 ? k_mg_up<true> : k_mg_up<false>, tiles_of(L.n), kTileThreads,
                            0, L.u, L.f, C.r, box_of(L), box_of(C), L.inv_h2, L.r, M->z, M->r,
                            p_rz, conv));
    }
    if (fc == 0)
        MG_TRY(launch_early(c, k_mg_out, dim3(M->n_rz), kThreads, 0, M->lev[0].r, M->r, M->z,
                            M->lev[0].V, p_rz, conv));
    return MG_OK;
}

// Solve L phi = src on the stored box (cpot holds the start and the
// Dirichlet planes) to |r| <= tol |src|; *iters: PCG iterations.
// Returns MG_NOT_CONVERGED when maxit iterations did not reach tol.
int coulomb_multigrid(mg_ctx* c, double tol, int maxit, int* iters) {
    if (!c->mgrid) MG_TRY(multigrid_setup(c));
    Multigrid* M = c->mgrid;
    const int nx = c->nx, ny = c->ny, nz = c->nz;
    const long V = c->V;
    const double inv_dx2 = 1.0 / (c->p.dx * c->p.dx);
    double *p_rz = M->part, *p_pq = M->part + M->n_part, *p_rr = M->part + 2 * M->n_part;
    k_pcg_start<<<kPartBlocks, kThreads, 0, c->stream>>>(c->csource, nx, ny, nz, c->mx, c->my,
                                                          M->e, M->p[0], M->part);
    MG_LAUNCHED(c);
    k_pcg_init_scalars<<<1, 32, 0, c->stream>>>(M->part, M->S);
    MG_LAUNCHED(c);
    k_pcg_residual<<<div_up(V, kThreads), kThreads, 0, c->stream>>>(
        c->cpot, c->csource, M->r, M->lev[0].f, nx, ny, nz, c->mx, c->my, inv_dx2);
    MG_LAUNCHED(c);
    const double tol2 = tol * tol;
    const Level& L0 = M->lev[0];
    // kChunk is even: every chunk starts with the old direction in p[0]
    auto iterations = [&](int count) -> int {
        for (int s = 0; s < count; ++s) {
            const double* p_old = M->p[s & 1];
            double* p_new = M->p[1 - (s & 1)];
            MG_TRY(vcycle(c, M, p_rz));
            MG_TRY(launch_early(c, k_pcg_direction,
                                dim3(div_up(nx, kTile), div_up(ny, kTile), div_up(nz, kDirDepth)),
                                kDirThreads, 0, M->z, p_old, p_new, M->q, box_of(L0), inv_dx2,
                                p_rz, M->n_rz, p_pq, M->S));
            MG_TRY(launch_early(c, k_pcg_update, dim3(kPartBlocks), kThreads, 0, M->e, M->r, p_new,
                                M->q, L0.f, V, p_rz, M->n_rz, p_pq, M->n_pq, p_rr, tol2, maxit,
                                M->S));
        }
        return MG_OK;
    };
    // the launches of kChunk iterations replay as one CUDA graph; tol and maxit are baked
    // into it, so it is rebuilt when they change
    if (M->chunk && (M->tol2 != tol2 || M->maxit != maxit)) {
        cudaGraphExecDestroy(M->chunk);
        M->chunk = nullptr;
    }
    if (!M->chunk && !M->no_graph) {
        if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();   // e.g. the legacy default stream: launch directly
            M->no_graph = true;
        } else {
            const long long l0 = c->launches;
            const int st = iterations(kChunk);
            cudaGraph_t graph = nullptr;
            const cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
            if (st != MG_OK || ce != cudaSuccess) {
                if (graph) cudaGraphDestroy(graph);
                return st != MG_OK ? st : MG_ERR_CUDA;
            }
            const cudaError_t ie = cudaGraphInstantiate(&M->chunk, graph, 0);
            cudaGraphDestroy(graph);
            if (ie != cudaSuccess) {
                M->chunk = nullptr;
                return MG_ERR_CUDA;
            }
            M->chunk_launches = c->launches - l0;
            c->launches = l0;
            M->tol2 = tol2;
            M->maxit = maxit;
        }
    }
    // a chunk is launched before the flag of the one before it is read (20 us of
    // waiting for the host a chunk; after convergence its kernels return at once)
    const PcgScalars* last = nullptr;
    for (int done = 0, turn = 0; done < maxit; turn ^= 1) {
        const int chunk = std::min(kChunk, maxit - done);
        if (M->chunk && chunk == kChunk) {
            MG_CUDA(cudaGraphLaunch(M->chunk, c->stream));
            c->launches += M->chunk_launches;
        } else {
            MG_TRY(iterations(chunk));
        }
        MG_CUDA(cudaMemcpyAsync(&M->h_S[turn], M->S, sizeof(PcgScalars), cudaMemcpyDeviceToHost,
                                c->stream));
        MG_CUDA(cudaEventRecord(M->read[turn], c->stream));
        if (done > 0) {
            MG_CUDA(cudaEventSynchronize(M->read[turn ^ 1]));
            last = &M->h_S[turn ^ 1];
            if (last->conv) break;
        }
        done += chunk;
        if (done >= maxit) {
            MG_CUDA(cudaEventSynchronize(M->read[turn]));
            last = &M->h_S[turn];
            break;
        }
    }
    k_pcg_finish<<<div_up(V, kThreads), kThreads, 0, c->stream>>>(c->cpot, M->e, nx, ny, nz, c->mx,
                                                                  c->my);
    MG_LAUNCHED(c);
    if (iters) *iters = last->iters;
    return last->conv == 1 ? MG_OK : MG_NOT_CONVERGED;
}

int multigrid_levels(const mg_ctx* c) { return c->mgrid ? c->mgrid->nlev : 0; }

}  // namespace mg
