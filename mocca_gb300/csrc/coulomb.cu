// coulomb.cu -- Coulomb Poisson solve on the symmetry-reduced box, FP64.
//
// Replaces SolveCoulomb with CoulombSolver = 1 (src/Coulomb.f90:255-346):
//   CoulombBound (:583-674): source -4 pi e2 rho_p on the stored box and
//     Dirichlet values sum_lm e2 4pi/(2l+1) Q_lm r^l Y_lm / r^(2l+1) on the
//     BCNumber = 2 extra planes of the extended box;
//   ConjugGrad (:755-900) with CoulombLaplacian (5-point FD, even mirror at
//     the low end of each axis, src/CoulombDerivatives.f90:144-281);
//   Slater exchange -(3/pi)^(1/3) e2 rho_p^(1/3) (:338-344).
// The CG runs as ONE cooperative kernel: every thread owns up to eight points
// of the stored box and keeps their solution, residual, direction and its
// Laplacian in registers; only the residual, which the stencil reads at the
// neighbours, goes to memory.  The recurrences are those of Chronopoulos and
// Gear (J. Comput. Appl. Math. 25 (1989) 153): w = Lap(r) and the sums r.r and
// r.w give both coefficients, so an iteration has one meeting of all blocks,
// where a block posts its partial sums and adds up everybody's in the same
// order (so every block takes the same branch).  The blocks come in clusters
// of eight, which add up their partials through distributed shared memory; one
// block of a cluster sends the sum to a mailbox of every block.  Everything
// that travels through memory (sums and residuals) is a pair of 64-bit words
// that carry a running number beside the halves of the value, so a reader sees
// by itself whether the value is there: no counters, flags or fences.  The
// waits are bounded: one that runs out of its cap sets the timeout status and
// the kernel returns instead of hanging.  A block leaves with its cluster, after
// a meeting that all eight attend (no rank writes to the shared memory of one
// that is gone), and decides nothing from sums that did not come.
// The kernel is a chain of latencies: an FP64 add or FMA takes 64 clocks, a
// divide 549, a cluster barrier 400, a word written by one block and polled by
// another about a thousand (but ten thousand where many blocks poll the lines
// that are to be written: the reason for clusters and mailboxes).  With three
// meetings through a counter and fences, serial sums of the partials and FP64
// divides an iteration took 19.8 us on a 24^3 box, 14.1 on 10^3 and 48 on 64^3
// (solve times over iterations); now 4.8, 3.9 and 20.
#include <algorithm>
#include <cmath>

#include "cgsum.cuh"
#include "mg_internal.cuh"

namespace mg {

namespace {

constexpr int kThreads = 256;
constexpr long long kWaitCycles = 4000000000LL;   // ~2 s at the top SM clock
constexpr int kMaxClusters = 32;  // sums of a meeting, one per lane

struct CgArgs {
    double* sol;            // extended box
    const double* src;      // extended box
    ulonglong2* res;        // stored box, tagged
    ulonglong2* mail;       // [2][blocks][kMaxClusters][2] sums of the clusters, tagged
    unsigned tag;           // every tag of this launch is above it, every earlier one at most it
    int* status;            // [0] state, [1] iterations
    int nx, ny, nz, mx, my;
    double inv_dx2;
    double prec;
    double rel;             // > 0: stop at |r| <= rel |src| instead of |r|^2 <= prec
    int maxit;
    long long sum_wait;     // limit in clocks of the waits for the clusters' sums,
    int sum_wait_from;      // from this iteration on (tests make single waits run out)
};

__device__ __forceinline__ double lap_at(const double* g, int i, int j, int k, int mx, int my,
                                         double inv_dx2) {
    const double cf[5] = {-1.0 / 12.0, 4.0 / 3.0, -5.0 / 2.0, 4.0 / 3.0, -1.0 / 12.0};
    double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll
    for (int q = -2; q <= 2; ++q) {
        const int ii = i + q < 0 ? -(i + q) - 1 : i + q;
        const int jj = j + q < 0 ? -(j + q) - 1 : j + q;
        const int kk = k + q < 0 ? -(k + q) - 1 : k + q;
        ax = fma(cf[q + 2], g[ii + mx * (j + (long)my * k)], ax);
        ay = fma(cf[q + 2], g[i + mx * (jj + (long)my * k)], ay);
        az = fma(cf[q + 2], g[i + mx * (j + (long)my * kk)], az);
    }
    return ax * inv_dx2 + ay * inv_dx2 + az * inv_dx2;
}

// A double as two words, each half of the value's bits below a 32-bit tag.
__device__ __forceinline__ void put_tagged(ulonglong2* p, double x, unsigned tag) {
    const unsigned long long e = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p),
                 "l"(e | (unsigned)__double2hiint(x)), "l"(e | (unsigned)__double2loint(x))
                 : "memory");
}
__device__ __forceinline__ ulonglong2 get_words(const ulonglong2* p) {
    ulonglong2 w;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
    return w;
}
// zero when both words carry the tag
__device__ __forceinline__ unsigned differs(const ulonglong2& w, unsigned tag) {
    return ((unsigned)(w.x >> 32) ^ tag) | ((unsigned)(w.y >> 32) ^ tag);
}
__device__ __forceinline__ double value_of(const ulonglong2& w) {
    return __hiloint2double((int)(unsigned)w.x, (int)(unsigned)w.y);
}

// Sums x and y over the grid; warp 0 of every block applies `then` to the
// totals (the same bits everywhere) and gives its two results to its threads.
// `meanwhile` is work of warp 0 for the time that the cluster's barrier takes.
// The tag's parity picks the turn: what is left for a turn has been read when
// that turn comes again, because the call in between needed every block.
// Waits for `limit` clocks.  False when this block gives up, which the other ranks
// of its cluster learn at their next meeting, the one of the next tag.
template <class Meanwhile, class Then>
__device__ bool grid_sum(ClusterSum& S, ulonglong2* mail, int* status, unsigned tag, long long limit,
                         double x, double y, double& a, double& b, Meanwhile meanwhile, Then then) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int turn = (int)(tag & 1u);
    const int rank = (int)(blockIdx.x % kCluster), cluster = (int)(blockIdx.x / kCluster);
    const int nclusters = (int)(gridDim.x / kCluster);
    if (!cluster_sum(S, turn, rank, x, y, meanwhile)) {
        // all ranks of the cluster leave here together
        if (threadIdx.x == 0) atomicExch(status, 2);
        return false;
    }
    if (warp == 0) {
        bool all = true;
        if (nclusters > 1) {
            ulonglong2* box = mail + (size_t)turn * gridDim.x * kMaxClusters * 2;
            if (rank == 0) {
                for (int q = lane; q < (int)gridDim.x; q += 32) {
                    ulonglong2* to = box + ((size_t)q * kMaxClusters + cluster) * 2;
                    put_tagged(to, x, tag);
                    put_tagged(to + 1, y, tag);
                }
            }
            const ulonglong2* mine = box + ((size_t)blockIdx.x * kMaxClusters + lane) * 2;
            x = y = 0.0;
            bool ok = true;
            if (lane < nclusters) {
                const long long t0 = clock64();
                while (true) {
                    const ulonglong2 w = get_words(mine), z = get_words(mine + 1);
                    if ((differs(w, tag) | differs(z, tag)) == 0) {
                        x = value_of(w);
                        y = value_of(z);
                        break;
                    }
                    if (clock64() - t0 > limit) {
                        ok = false;
                        break;
                    }
                }
            }
            all = __all_sync(0xffffffffu, ok) != 0;
            const double v = warp_sum2(x, y);
            x = __shfl_sync(0xffffffffu, v, 0);
            y = __shfl_sync(0xffffffffu, v, 16);
        }
        if (all) {
            double ra, rb;
            then(x, y, ra, rb);
            if (lane == 0) {
                S.result[0] = ra;
                S.result[1] = rb;
            }
        }
        if (lane == 0) {
            S.late = all ? 0 : 1;
            if (!all) S.fail = 1;
        }
    }
    __syncthreads();
    if (S.late) {
        x = y = 0.0;
        cluster_sum(S, turn ^ 1, rank, x, y, []() {});
        if (threadIdx.x == 0) atomicExch(status, 2);
        return false;
    }
    a = S.result[0];
    b = S.result[1];
    return true;
}

// A stored point's twelve neighbours: offsets per axis to -1, +1, -2, +2, the
// low ones mirrored (-1 to 0, -2 to 1); `have` leaves out the Dirichlet planes,
// where the residual is zero.
struct Neighbours {
    int off[12];
    unsigned have;
    __device__ __forceinline__ Neighbours(int i, int j, int k, int nx, int ny, int nz) {
        const int at[3] = {i, j, k}, n[3] = {nx, ny, nz}, st[3] = {1, nx, nx * ny};
        have = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int q = at[d], s = st[d];
            const bool in[4] = {true, q + 1 < n[d], q > 0 || n[d] > 1, q + 2 < n[d]};
            const int o[4] = {q >= 1 ? -s : 0, s, q >= 2 ? -2 * s : (q == 1 ? -s : s), 2 * s};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                off[4 * d + u] = in[u] ? o[u] : 0;
                have |= (in[u] ? 1u : 0u) << (4 * d + u);
            }
        }
    }
};

// Laplacian of the residual at the point c, whose neighbours carry `tag`.
__device__ __forceinline__ double lap_res(const ulonglong2* c, double centre, const Neighbours& nb,
                                          double k0, double k1, double k2, unsigned tag, int* fail) {
    double v[12];
    const long long t0 = clock64();
    while (true) {
        ulonglong2 w[12];
#pragma unroll
        for (int u = 0; u < 12; ++u) w[u] = get_words(c + nb.off[u]);
        unsigned bad = 0;
#pragma unroll
        for (int u = 0; u < 12; ++u) {
            bad |= differs(w[u], tag);
            v[u] = nb.have >> u & 1u ? value_of(w[u]) : 0.0;
        }
        if (bad == 0) break;
        if (clock64() - t0 > kWaitCycles) {
            *fail = 1;
            break;
        }
    }
    const double one = ((v[0] + v[1]) + (v[4] + v[5])) + (v[8] + v[9]);
    const double two = ((v[2] + v[3]) + (v[6] + v[7])) + (v[10] + v[11]);
    return fma(k2, two, fma(k1, one, k0 * centre));
}

// R points per thread: point q of thread t is t + q * (threads of the grid).
template <int R>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(512, 1) k_cg(CgArgs a) {
    __shared__ ClusterSum S;
    if (!in_cluster()) {
        if (blockIdx.x == 0 && threadIdx.x == 0) a.status[0] = 3;
        return;
    }
    if (threadIdx.x == 0) S.fail = 0;
    cluster_barrier();   // no rank writes to another's shared memory before that one has started
    unsigned tag = a.tag;   // of the last sums and of the residual before them
    const int V = a.nx * a.ny * a.nz;
    const int stride = (int)(gridDim.x * blockDim.x);
    const int t0 = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    const double k0 = -7.5 * a.inv_dx2, k1 = 4.0 / 3.0 * a.inv_dx2, k2 = -1.0 / 12.0 * a.inv_dx2;
    double sol[R], res[R], p[R], s[R];   // s = Lap(p)
    int ci[R], cj[R], ck[R];

    long long limit = a.sum_wait_from > 0 ? kWaitCycles : a.sum_wait;

    // r0 = src - Lap(sol)
    double bb = 0.0, unused;
    if (a.rel > 0.0) ++tag;
    ++tag;
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int v = t0 + q * stride;
        sol[q] = res[q] = p[q] = s[q] = 0.0;
        ci[q] = v % a.nx;
        cj[q] = (v / a.nx) % a.ny;
        ck[q] = v / (a.nx * a.ny);
        if (v >= V) continue;
        const long o = ci[q] + a.mx * (cj[q] + (long)a.my * ck[q]);
        sol[q] = a.sol[o];
        res[q] = a.src[o] - lap_at(a.sol, ci[q], cj[q], ck[q], a.mx, a.my, a.inv_dx2);
        put_tagged(a.res + v, res[q], tag);
        bb = fma(a.src[o], a.src[o], bb);
    }
    double prec = a.prec;
    if (a.rel > 0.0) {
        // |src|^2 over the stored box for the relative test
        if (!grid_sum(S, a.mail, a.status, tag - 1, limit, bb, 0.0, bb, unused, []() {},
                      [](double x, double, double& u, double& w) { u = x; w = 0.0; }))
            return;
        prec = a.rel * a.rel * bb;
    }
    const Neighbours nb0(ci[0], cj[0], ck[0], a.nx, a.ny, a.nz);
    // of warp 0: |r|^2 and |r|^2 / alpha of the iteration before, the inverses
    // of |r|^2 and alpha
    double rr_old = 0.0, d_old = 0.0, inv_rr = 0.0, inv_alpha = 0.0;
    int it = 0;
    bool done = false;
    for (;; ++it) {
        if (it == a.sum_wait_from) limit = a.sum_wait;
        double rr = 0.0, rw = 0.0, lap[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            lap[q] = 0.0;
            const int v = t0 + q * stride;
            if (v >= V) continue;
            lap[q] = lap_res(a.res + v, res[q],
                             q == 0 ? nb0 : Neighbours(ci[q], cj[q], ck[q], a.nx, a.ny, a.nz), k0, k1, k2,
                             tag, &S.fail);
            rr = fma(res[q], res[q], rr);
            rw = fma(res[q], lap[q], rw);
        }
        double alpha, beta;
        // beta = rr / rr_old, alpha = rr / (rw - beta rr / alpha_old); a negative
        // beta says that the test is met (rr <= prec)
        if (!grid_sum(
                S, a.mail, a.status, tag, limit, rr, rw, alpha, beta,
                [&]() {
                    if (it == 0) return;
                    inv_rr = inverse(rr_old);
                    inv_alpha = d_old * inv_rr;
                },
                [&](double x, double y, double& u, double& w) {
                    const double b = x * inv_rr;
                    d_old = fma(-b, x * inv_alpha, y);
                    rr_old = x;
                    u = x * inverse(d_old);
                    w = it > 0 && x <= prec ? -1.0 : b;
                }))
            return;
        done = beta < 0.0;
        if (done || it == a.maxit) break;
        ++tag;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            s[q] = fma(beta, s[q], lap[q]);
            const double r = fma(-alpha, s[q], res[q]);
            if (t0 + q * stride < V) put_tagged(a.res + t0 + q * stride, r, tag);
            p[q] = fma(beta, p[q], res[q]);
            sol[q] = fma(alpha, p[q], sol[q]);
            res[q] = r;
        }
    }
    // the last meeting: a rank whose last sums did not come is at it too
    double none[2] = {0.0, 0.0};
    if (!cluster_sum(S, (int)((tag + 1) & 1u), (int)(blockIdx.x % kCluster), none[0], none[1], []() {})) {
        if (threadIdx.x == 0) atomicExch(a.status, 2);
        return;
    }
#pragma unroll
    for (int q = 0; q < R; ++q)
        if (t0 + q * stride < V) a.sol[ci[q] + a.mx * (cj[q] + (long)a.my * ck[q])] = sol[q];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.status[1] = it;
        if (!done) atomicCAS(a.status, 0, 1);
    }
}

// Launch shape of the CG: clusters of eight blocks with up to 128 points each
// until the card is full, then more threads, then two, four or eight points
// per thread.  More blocks cost mail, more points per block FP64 issue: per
// iteration at 10^3 3.9 us with 64 points a block, 3.25 with 128, 4.2 with 256;
// at 16^3 4.27, 4.29 and 4.8; at 20^3 4.37 with 128 and 5.2 with 256.
struct CgShape {
    const void* fn;
    int blocks, threads;
};
constexpr int kCgThreads = 512;
CgShape cg_shape(const mg_ctx* c) {
    constexpr long kPer = 128L * kCluster;
    const int clusters = (int)std::max<long>(1, std::min<long>(c->cg_clusters, (c->V + kPer - 1) / kPer));
    const int blocks = clusters * kCluster;
    const long per = (c->V + blocks - 1) / blocks;
    int r = 1;
    while (r < 8 && (per + r - 1) / r > 256) r *= 2;
    const int threads = (int)(((per + r - 1) / r + 31) / 32 * 32);
    const void* fn = r == 1   ? (const void*)k_cg<1>
                     : r == 2 ? (const void*)k_cg<2>
                     : r == 4 ? (const void*)k_cg<4>
                              : (const void*)k_cg<8>;
    return CgShape{fn, blocks, threads};
}
// the residuals, then the mailboxes
size_t cg_tagged_bytes(const mg_ctx* c) {
    return ((size_t)c->V + 4 * (size_t)cg_shape(c).blocks * kMaxClusters) * sizeof(ulonglong2);
}

// Source and multipole Dirichlet values on the extended box.
//
// A Dirichlet value is a sum of nmom terms with an FP64 divide each (~550 clocks
// one after the other).  A block takes kBoundPoints of the points beyond the box, its
// warps share the terms, and one warp adds them in their order.  The blocks after
// those take the box.  24^3: 25 us with a thread per point of the extended box, now
// 7.4; 48^3: 67 and 14.
constexpr int kBoundPoints = 32;
constexpr int kBoundThreads = 256;
constexpr int kBoundTerms = 64;   // at a time

__global__ void __launch_bounds__(kBoundThreads)
k_coulomb_bound(const double* __restrict__ rho_p, const double* __restrict__ sh,
                const double* __restrict__ rpow, const double* __restrict__ mval,
                const double* __restrict__ mfac, int nmom, int nx, int ny, int nz, int mx, int my,
                int mz, double e2, double* __restrict__ src, double* __restrict__ sol) {
    __shared__ double term[kBoundTerms][kBoundPoints];
    const long M = (long)mx * my * mz, V = (long)nx * ny * nz;
    const long nb = (M - V + kBoundPoints - 1) / kBoundPoints;
    if (blockIdx.x >= nb) {
        const long t = (blockIdx.x - nb) * kBoundThreads + threadIdx.x;
        if (t >= V) return;
        const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / ((long)nx * ny));
        const double pi = 4.0 * atan2(1.0, 1.0);
        src[i + mx * (j + (long)my * k)] = -4 * pi * e2 * rho_p[t];
        return;
    }
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    long t = (long)blockIdx.x * kBoundPoints + lane;
    const bool in = t < M - V;
    // the points beyond the box, by their z, y or x
    const long nzs = (long)mx * my * (mz - nz), nys = (long)mx * (my - ny) * nz;
    long o = 0;
    if (t < nzs) {
        o = (long)mx * my * nz + t;
    } else if (t < nzs + nys) {
        t -= nzs;
        const long row = t / mx;
        o = t % mx + mx * (ny + row % (my - ny) + my * (row / (my - ny)));
    } else if (in) {
        t -= nzs + nys;
        const long row = t / (mx - nx);
        o = nx + t % (mx - nx) + mx * (row % ny + my * (row / ny));
    }
    double bc = 0.0;
    for (int m0 = 0; m0 < nmom; m0 += kBoundTerms) {
        const int m1 = min(nmom, m0 + kBoundTerms);
        for (int m = m0 + warp; m < m1; m += kBoundThreads / 32)
            if (in) {
                const double value = mval[2 * m + 1] * mfac[m];
                term[m - m0][lane] = value * sh[(long)m * M + o] * e2 / rpow[(long)m * M + o];
            }
        __syncthreads();
        if (in && warp == 0)
            for (int m = 0; m < m1 - m0; ++m) bc = bc + term[m][lane];
        __syncthreads();
    }
    if (!in || warp > 0) return;
    src[o] = 0.0;
    if (bc != 0.0) sol[o] = bc;
}

static dim3 bound_blocks(const mg_ctx* c) {
    return dim3(div_up(c->M - c->V, kBoundPoints) + div_up(c->V, kBoundThreads));
}

// (blocks of two warps: the power is FP64 work, spread over all SMs)
constexpr int kOutThreads = 64;

__global__ void k_coulomb_out(const double* __restrict__ sol, const double* __restrict__ rho_p,
                              int nx, int ny, int nz, int mx, int my, double fac,
                              double* __restrict__ coul, double* __restrict__ coulex) {
    const long V = (long)nx * ny * nz;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
    coul[v] = sol[i + mx * (j + (long)my * k)];
    coulex[v] = fac * pow(rho_p[v], 1 / 3.0);
}

// ---- direct separable solve (mixed form) ---------------------------------------
//
// The CG operator is the 4th-order difference Laplacian on the stored box
// with a mirror at each symmetry plane and the two Dirichlet planes of the
// extended box moved to the right-hand side: a Kronecker sum
// L = (L_x + L_y + L_z) / dx^2 of three 1-D symmetric operators.  With the
// 1-D eigendecompositions L_a = C_a diag(mu_a) C_a^T (computed once on the
// host), L^{-1} r = (C_x C_y C_z) diag(dx^2 / (mu_x + mu_y + mu_z))
// (C_x C_y C_z)^T r: six small contractions along the axes and one scaling
// instead of ~140 CG iterations with four grid barriers each.  Two rounds of
// FP64 iterative refinement (residual with the full stencil, correction
// from the direct solve) leave a residual at FP64 rounding.

__global__ void k_cfast_residual(const double* __restrict__ sol, const double* __restrict__ src,
                                 double* __restrict__ r, int nx, int ny, int nz, int mx, int my,
                                 double inv_dx2) {
    const long V = (long)nx * ny * nz;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
    const long o = i + mx * (j + (long)my * k);
    r[v] = src[o] - lap_at(sol, i, j, k, mx, my, inv_dx2);
}

// out = M^T in (fwd) or M in (back) along one axis of an nx x ny x nz grid;
// C is the axis' n x n eigenvector matrix, C[i * n + kk] = component i of
// eigenvector kk.
__global__ void k_cfast_axis(const double* __restrict__ in, double* __restrict__ out,
                             const double* __restrict__ C, int axis, int nx, int ny, int nz,
                             int fwd) {
    const long V = (long)nx * ny * nz;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int c3[3] = {(int)(v % nx), (int)((v / nx) % ny), (int)(v / ((long)nx * ny))};
    const int n = axis == 0 ? nx : axis == 1 ? ny : nz;
    const long step = axis == 0 ? 1 : axis == 1 ? nx : (long)nx * ny;
    const int a = c3[axis];
    const long base = v - a * step;
    double s = 0.0;
    for (int q = 0; q < n; ++q) {
        const double m = fwd ? C[q * n + a] : C[a * n + q];
        s = fma(m, in[base + q * step], s);
    }
    out[v] = s;
}

__global__ void k_cfast_scale(double* __restrict__ x, const double* __restrict__ mux,
                              const double* __restrict__ muy, const double* __restrict__ muz,
                              int nx, int ny, int nz, double dx2) {
    const long V = (long)nx * ny * nz;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
    x[v] *= dx2 / (mux[i] + muy[j] + muz[k]);
}

__global__ void k_cfast_update(double* __restrict__ sol, const double* __restrict__ e, int nx,
                               int ny, int nz, int mx, int my) {
    const long V = (long)nx * ny * nz;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
    sol[i + mx * (j + (long)my * k)] += e[v];
}

// 1-D operator of one axis (mirror at -1/2, Dirichlet planes beyond n-1
// dropped) and its eigendecomposition by cyclic Jacobi in FP64.
void axis_eigen(int n, std::vector<double>& C, std::vector<double>& mu) {
    const double cf[5] = {-1.0 / 12.0, 4.0 / 3.0, -5.0 / 2.0, 4.0 / 3.0, -1.0 / 12.0};
    std::vector<double> A((size_t)n * n, 0.0);
    for (int i = 0; i < n; ++i)
        for (int q = -2; q <= 2; ++q) {
            int m = i + q;
            if (m < 0) m = -m - 1;
            if (m >= n) continue;
            A[(size_t)i * n + m] += cf[q + 2];
        }
    C.assign((size_t)n * n, 0.0);
    for (int i = 0; i < n; ++i) C[(size_t)i * n + i] = 1.0;
    for (int sweep = 0; sweep < 60; ++sweep) {
        double off = 0.0, nrm = 0.0;
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < n; ++j) {
                nrm += A[(size_t)i * n + j] * A[(size_t)i * n + j];
                if (i != j) off += A[(size_t)i * n + j] * A[(size_t)i * n + j];
            }
        if (off <= 1e-30 * nrm) break;
        for (int p = 0; p < n - 1; ++p)
            for (int q = p + 1; q < n; ++q) {
                const double apq = A[(size_t)p * n + q];
                if (std::fabs(apq) < 1e-300) continue;
                const double th = (A[(size_t)q * n + q] - A[(size_t)p * n + p]) / (2.0 * apq);
                const double t = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1.0));
                const double cs = 1.0 / std::sqrt(t * t + 1.0), sn = t * cs;
                for (int k = 0; k < n; ++k) {
                    const double akp = A[(size_t)k * n + p], akq = A[(size_t)k * n + q];
                    A[(size_t)k * n + p] = cs * akp - sn * akq;
                    A[(size_t)k * n + q] = sn * akp + cs * akq;
                }
                for (int k = 0; k < n; ++k) {
                    const double apk = A[(size_t)p * n + k], aqk = A[(size_t)q * n + k];
                    A[(size_t)p * n + k] = cs * apk - sn * aqk;
                    A[(size_t)q * n + k] = sn * apk + cs * aqk;
                }
                for (int k = 0; k < n; ++k) {
                    const double vkp = C[(size_t)k * n + p], vkq = C[(size_t)k * n + q];
                    C[(size_t)k * n + p] = cs * vkp - sn * vkq;
                    C[(size_t)k * n + q] = sn * vkp + cs * vkq;
                }
            }
    }
    mu.resize(n);
    for (int i = 0; i < n; ++i) mu[i] = A[(size_t)i * n + i];
}

}  // namespace

// ---- host-side restatement of the spherical harmonics of the moments -----
// legendre_pnm src/Mesh.f90:96-262; SphericalHarmonics src/Moments.f90:584-691
static void legendre(int n, int m, double x, double* cx) {
    for (int i = 0; i < m; ++i) cx[i] = 0.0;
    cx[m] = 1.0;
    const double somx2 = std::sqrt(1.0 - x * x);
    double fact = 1.0;
    for (int i = 1; i <= m; ++i) { cx[m] = -cx[m] * fact * somx2; fact += 2.0; }
    if (m == n) return;
    cx[m + 1] = x * double(2 * m + 1) * cx[m];
    for (int i = m + 2; i <= n; ++i)
        cx[i] = (double(2 * i - 1) * x * cx[i - 1] - double(i + m - 1) * cx[i - 2]) / double(i - m);
}

static double ipow(double x, int n) {
    double r = 1.0;
    for (int i = 0; i < n; ++i) r *= x;
    return r;
}

double rlylm(int l, int m, int im, double X, double Y, double Z) {
    const double pi = 4.0 * std::atan2(1.0, 1.0);
    const int maxl = 10;
    const double r = std::sqrt(X * X + Y * Y + Z * Z);
    double leg[16];
    legendre(maxl, m, Z / r, leg);
    double fq = 1.0;
    for (int q = 1; q <= 2 * m; ++q) fq = fq / double(l + m - q + 1);
    double fac = ((m % 2) ? -1.0 : 1.0) * std::sqrt(fq) * ipow(r, l);
    fac = fac * std::sqrt(double(2 * l + 1) / (4 * pi));
    const double phi = std::atan2(Y, X);
    return fac * leg[l] * (im ? std::sin(m * phi) : std::cos(m * phi));
}

// Moment table (IniMoments, src/Moments.f90:372-582; EV8 selection of
// NewMoment_Electric), spherical harmonics on the stored and extended
// meshes, the extended-box geometry and the initial guess (SetupCoulomb
// :348-540, InitialGuess :542-581).
int coulomb_setup(mg_ctx* c) {
    const double pi = 4.0 * std::atan2(1.0, 1.0);
    const int maxl = c->p.max_l_coul > 0 ? std::min(c->p.max_l_coul, 10) : 10;
    std::vector<int> L, Mm, Im;
    L.push_back(0); Mm.push_back(0); Im.push_back(0);
    for (int l = 1; l <= 10; ++l)
        for (int m = 0; m <= l; ++m)
            for (int im = 0; im <= 1; ++im) {
                if (c->p.pc && (l % 2)) continue;
                if (c->p.tsc && im == 1) continue;
                if (c->p.sc && (m % 2)) continue;
                if (m == 0 && im == 1) continue;
                L.push_back(l); Mm.push_back(m); Im.push_back(im);
            }
    const int nmom_all = (int)L.size();
    int nmom_bc = 0;
    while (nmom_bc < nmom_all && L[nmom_bc] <= maxl) ++nmom_bc;
    c->n_moments = nmom_all;
    for (int q = 0; q < nmom_all && q < kNumMoments; ++q) c->h_moment_l[q] = L[q];
    const int nx = c->nx, ny = c->ny, nz = c->nz;
    const long V = c->V;
    std::vector<double> sh(nmom_all * V);
    for (int q = 0; q < nmom_all; ++q)
        for (int k = 0; k < nz; ++k)
            for (int j = 0; j < ny; ++j)
                for (int i = 0; i < nx; ++i) {
                    const double X = c->p.dx / 2.0 + c->p.dx * i, Y = c->p.dx / 2.0 + c->p.dx * j,
                                 Z = c->p.dx / 2.0 + c->p.dx * k;
                    sh[q * V + i + nx * (j + (long)ny * k)] =
                        q == 0 ? 1.0 / std::sqrt(4.0 * pi) : rlylm(L[q], Mm[q], Im[q], X, Y, Z);
                }
    MG_CUDA(cudaMalloc(&c->sh_mesh, sh.size() * sizeof(double)));
    MG_CUDA(cudaMemcpy(c->sh_mesh, sh.data(), sh.size() * sizeof(double), cudaMemcpyHostToDevice));
    MG_CUDA(cudaMalloc(&c->moment_values, 2 * nmom_all * sizeof(double)));
    MG_CUDA(cudaMemset(c->moment_values, 0, 2 * nmom_all * sizeof(double)));

    // extended box: BCNumber = 2 planes beyond the stored box on each axis
    c->mx = nx + 2; c->my = ny + 2; c->mz = nz + 2;
    const long M = (long)c->mx * c->my * c->mz;
    c->M = M;
    std::vector<double> shx(nmom_bc * M), rp(nmom_bc * M), guess(M, 0.0), mfac(nmom_bc);
    for (int q = 0; q < nmom_bc; ++q) mfac[q] = 4 * pi / (2 * L[q] + 1);
    const double R = 1.25 * std::pow(c->p.neutrons + c->p.protons, 1.0 / 3.0);
    const double charge = c->p.protons * c->f.e2, fac = charge / (2 * R);
    for (int k = 0; k < c->mz; ++k)
        for (int j = 0; j < c->my; ++j)
            for (int i = 0; i < c->mx; ++i) {
                const long o = i + c->mx * (j + (long)c->my * k);
                const double X = (0.5 + i) * c->p.dx, Y = (0.5 + j) * c->p.dx, Z = (0.5 + k) * c->p.dx;
                const double r = std::sqrt(X * X + Y * Y + Z * Z);
                for (int q = 0; q < nmom_bc; ++q) {
                    shx[q * M + o] = rlylm(L[q], Mm[q], Im[q], X, Y, Z);
                    rp[q * M + o] = ipow(r, 2 * L[q] + 1);
                }
                if (i < nx && j < ny && k < nz) guess[o] = r <= R ? fac * (3 - r * r / (R * R)) : charge / r;
            }
    c->n_bc_moments = nmom_bc;
    MG_CUDA(cudaMalloc(&c->sh_ext, shx.size() * sizeof(double) + 8));
    MG_CUDA(cudaMalloc(&c->rpow_ext, rp.size() * sizeof(double) + 8));
    MG_CUDA(cudaMalloc(&c->mfac, mfac.size() * sizeof(double) + 8));
    MG_CUDA(cudaMemcpy(c->sh_ext, shx.data(), shx.size() * sizeof(double), cudaMemcpyHostToDevice));
    MG_CUDA(cudaMemcpy(c->rpow_ext, rp.data(), rp.size() * sizeof(double), cudaMemcpyHostToDevice));
    MG_CUDA(cudaMemcpy(c->mfac, mfac.data(), mfac.size() * sizeof(double), cudaMemcpyHostToDevice));
    for (double** b : {&c->cpot, &c->csource, &c->cres, &c->cp, &c->ct})
        MG_CUDA(cudaMalloc(b, M * sizeof(double)));
    MG_CUDA(cudaMemcpy(c->cpot, guess.data(), M * sizeof(double), cudaMemcpyHostToDevice));
    MG_CUDA(cudaMalloc(&c->cguess, M * sizeof(double)));
    MG_CUDA(cudaMemcpy(c->cguess, guess.data(), M * sizeof(double), cudaMemcpyHostToDevice));
    MG_CUDA(cudaMalloc(&c->cg_status, 4 * sizeof(int)));
    // clusters that the card holds at once, whatever the shape
    c->cg_clusters = kMaxClusters;
    for (const void* fn : {(const void*)k_cg<1>, (const void*)k_cg<2>, (const void*)k_cg<4>,
                           (const void*)k_cg<8>}) {
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kCluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kCluster);
        cfg.blockDim = dim3(kCgThreads);
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        MG_CUDA(cudaOccupancyMaxActiveClusters(&n, fn, &cfg));
        c->cg_clusters = std::min(c->cg_clusters, n);
    }
    if (c->cg_clusters < 1 || cg_shape(c).threads > kCgThreads) return MG_ERR_CUDA;
    MG_CUDA(cudaMalloc(&c->cg_tagged, cg_tagged_bytes(c)));
    MG_CUDA(cudaMemset(c->cg_tagged, 0, cg_tagged_bytes(c)));
    // eigendecompositions of the three 1-D operators for the direct solve
    {
        const int ns[3] = {nx, ny, nz};
        std::vector<double> all;
        for (int a = 0; a < 3; ++a) {
            std::vector<double> Ca, mua;
            axis_eigen(ns[a], Ca, mua);
            c->cfast_off[a][0] = (long)all.size();
            all.insert(all.end(), Ca.begin(), Ca.end());
            c->cfast_off[a][1] = (long)all.size();
            all.insert(all.end(), mua.begin(), mua.end());
        }
        MG_CUDA(cudaMalloc(&c->cfast, all.size() * sizeof(double)));
        MG_CUDA(cudaMemcpy(c->cfast, all.data(), all.size() * sizeof(double),
                           cudaMemcpyHostToDevice));
    }
    c->coulomb_init = true;
    return MG_OK;
}

// Sums of r^2 and of the source's square over the stored box (a diagnostic:
// atomics, so the last bits vary between runs).
__global__ void k_residual_norms(const double* __restrict__ r, const double* __restrict__ src,
                                 int nx, int ny, int nz, int mx, int my,
                                 double* __restrict__ out) {
    const long V = (long)nx * ny * nz;
    double a = 0.0, b = 0.0;
    for (long v = (long)blockIdx.x * blockDim.x + threadIdx.x; v < V;
         v += (long)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long)nx * ny));
        const double s = src[i + mx * (j + (long)my * k)];
        a = fma(r[v], r[v], a);
        b = fma(s, s, b);
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (threadIdx.x % 32 == 0) {
        atomicAdd(out, a);
        atomicAdd(out + 1, b);
    }
}

// Mixed form: two rounds of (FP64 residual, direct separable correction).
static int coulomb_direct_launches(mg_ctx* c) {
    const int nx = c->nx, ny = c->ny, nz = c->nz;
    const long V = c->V;
    const int g = div_up(V, kThreads);
    const double dx2 = c->p.dx * c->p.dx;
    double *r = c->cres, *t1 = c->cp, *t2 = c->ct;   // CG buffers, unused here
    const double* C[3] = {c->cfast + c->cfast_off[0][0], c->cfast + c->cfast_off[1][0],
                          c->cfast + c->cfast_off[2][0]};
    const double* mu[3] = {c->cfast + c->cfast_off[0][1], c->cfast + c->cfast_off[1][1],
                           c->cfast + c->cfast_off[2][1]};
    for (int round = 0; round < 2; ++round) {
        k_cfast_residual<<<g, kThreads, 0, c->stream>>>(c->cpot, c->csource, r, nx, ny, nz, c->mx,
                                                        c->my, 1.0 / dx2);
        MG_LAUNCHED(c);
        k_cfast_axis<<<g, kThreads, 0, c->stream>>>(r, t1, C[0], 0, nx, ny, nz, 1);
        MG_LAUNCHED(c);
        k_cfast_axis<<<g, kThreads, 0, c->stream>>>(t1, t2, C[1], 1, nx, ny, nz, 1);
        MG_LAUNCHED(c);
        k_cfast_axis<<<g, kThreads, 0, c->stream>>>(t2, t1, C[2], 2, nx, ny, nz, 1);
        MG_LAUNCHED(c);
        k_cfast_scale<<<g, kThreads, 0, c->stream>>>(t1, mu[0], mu[1], mu[2], nx, ny, nz, dx2);
        MG_LAUNCHED(c);
        k_cfast_axis<<<g, kThreads, 0, c->stream>>>(t1, t2, C[2], 2, nx, ny, nz, 0);
        MG_LAUNCHED(c);
        k_cfast_axis<<<g, kThreads, 0, c->stream>>>(t2, t1, C[1], 1, nx, ny, nz, 0);
        MG_LAUNCHED(c);
        k_cfast_axis<<<g, kThreads, 0, c->stream>>>(t1, t2, C[0], 0, nx, ny, nz, 0);
        MG_LAUNCHED(c);
        k_cfast_update<<<g, kThreads, 0, c->stream>>>(c->cpot, t2, nx, ny, nz, c->mx, c->my);
        MG_LAUNCHED(c);
    }
    return MG_OK;
}

// The eighteen launches of the two rounds replay as one CUDA graph (fixed
// buffers per context): a few microseconds each, they would otherwise run at
// the host's enqueue rate.
static int coulomb_direct(mg_ctx* c) {
    if (c->cfast_no_graph) return coulomb_direct_launches(c);
    if (!c->cfast_graph) {
        if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            c->cfast_no_graph = true;
            return coulomb_direct_launches(c);
        }
        const long long l0 = c->launches;
        const int st = coulomb_direct_launches(c);
        cudaGraph_t graph = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
        if (st != MG_OK || ce != cudaSuccess) {
            if (graph) cudaGraphDestroy(graph);
            return st != MG_OK ? st : MG_ERR_CUDA;
        }
        const cudaError_t ie = cudaGraphInstantiate(&c->cfast_graph, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) {
            c->cfast_graph = nullptr;
            return MG_ERR_CUDA;
        }
        c->cfast_graph_launches = c->launches - l0;
        c->launches = l0;
    }
    MG_CUDA(cudaGraphLaunch(c->cfast_graph, c->stream));
    c->launches += c->cfast_graph_launches;
    return MG_OK;
}

// |b - L phi| / |b| of the current Coulomb potential on the stored box, with
// the solver's own Laplacian (CoulombLaplacian with the boundary planes).
int coulomb_residual(mg_ctx* c, double* rel) {
    if (!c->coulomb_init) return MG_ERR_STATE;
    const long V = c->V;
    const double dx2 = c->p.dx * c->p.dx;
    k_cfast_residual<<<div_up(V, kThreads), kThreads, 0, c->stream>>>(
        c->cpot, c->csource, c->cres, c->nx, c->ny, c->nz, c->mx, c->my, 1.0 / dx2);
    MG_LAUNCHED(c);
    MG_CUDA(cudaMemsetAsync(c->red, 0, 2 * sizeof(double), c->stream));
    k_residual_norms<<<std::min(div_up(V, kThreads), 4 * c->num_sms), kThreads, 0, c->stream>>>(
        c->cres, c->csource, c->nx, c->ny, c->nz, c->mx, c->my, c->red);
    MG_LAUNCHED(c);
    double h[2];
    MG_CUDA(cudaMemcpyAsync(h, c->red, 2 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    MG_CUDA(cudaStreamSynchronize(c->stream));
    *rel = h[1] > 0.0 ? std::sqrt(h[0] / h[1]) : std::sqrt(h[0]);
    return MG_OK;
}

// The potential back to InitialGuess (the start of a cold solve).
int coulomb_reset(mg_ctx* c) {
    if (!c->coulomb_init) MG_TRY(coulomb_setup(c));
    MG_CUDA(cudaMemcpyAsync(c->cpot, c->cguess, c->M * sizeof(double), cudaMemcpyDeviceToDevice,
                            c->stream));
    return MG_OK;
}

int coulomb_solve(mg_ctx* c, int* iters) {
    if (!c->coulomb_init) MG_TRY(coulomb_setup(c));
    k_coulomb_bound<<<bound_blocks(c), kBoundThreads, 0, c->stream>>>(
        c->rho + c->V, c->sh_ext, c->rpow_ext, c->moment_values, c->mfac, c->n_bc_moments, c->nx,
        c->ny, c->nz, c->mx, c->my, c->mz, c->f.e2, c->csource, c->cpot);
    MG_LAUNCHED(c);
    if (c->p.coulomb_solver == 2) {
        const double pi_ = 4.0 * std::atan2(1.0, 1.0);
        const int maxit = c->p.coulomb_max > 0 ? c->p.coulomb_max : 500;
        const int st = coulomb_multigrid(c, c->p.coulomb_prec > 0 ? c->p.coulomb_prec : 1e-10,
                                         maxit, iters);
        if (st < 0) return st;
        k_coulomb_out<<<div_up(c->V, kOutThreads), kOutThreads, 0, c->stream>>>(
            c->cpot, c->rho + c->V, c->nx, c->ny, c->nz, c->mx, c->my,
            -std::pow(3 / pi_, 1 / 3.0) * c->f.e2, c->coulomb, c->coulex);
        MG_LAUNCHED(c);
        return st;
    }
    if (c->cur_precision == MG_MIXED) {
        MG_TRY(coulomb_direct(c));
        const double pi = 4.0 * std::atan2(1.0, 1.0);
        const double fac = -std::pow(3 / pi, 1 / 3.0) * c->f.e2;
        k_coulomb_out<<<div_up(c->V, kOutThreads), kOutThreads, 0, c->stream>>>(
            c->cpot, c->rho + c->V, c->nx, c->ny, c->nz, c->mx, c->my, fac, c->coulomb,
            c->coulex);
        MG_LAUNCHED(c);
        if (iters) *iters = 2;
        return MG_OK;
    }
    MG_CUDA(cudaMemsetAsync(c->cg_status, 0, 4 * sizeof(int), c->stream));
    const int maxit = c->p.coulomb_max > 0 ? c->p.coulomb_max : 500;
    // tags run on from solve to solve, so nothing is cleared between them
    // until they come near the end of 32 bits
    const unsigned span = (unsigned)maxit + 8u;
    if (c->cg_tag > 0xFFFFFFFFu - span) {
        MG_CUDA(cudaMemsetAsync(c->cg_tagged, 0, cg_tagged_bytes(c), c->stream));
        c->cg_tag = 0;
    }
    CgArgs a;
    a.sol = c->cpot; a.src = c->csource;
    a.res = c->cg_tagged; a.mail = c->cg_tagged + c->V;
    a.tag = c->cg_tag;
    c->cg_tag += span;
    a.status = c->cg_status;
    a.nx = c->nx; a.ny = c->ny; a.nz = c->nz; a.mx = c->mx; a.my = c->my;
    a.inv_dx2 = 1.0 / (c->p.dx * c->p.dx);
    a.prec = 1.0e-9 / (c->p.dx * c->p.dx * c->p.dx * c->nx * c->ny * c->nz);
    a.rel = c->p.coulomb_prec > 0 ? c->p.coulomb_prec : 0.0;
    a.maxit = maxit;
    a.sum_wait = c->cg_sum_wait > 0 ? c->cg_sum_wait : kWaitCycles;
    a.sum_wait_from = c->cg_sum_wait_from;
    void* args[] = {&a};
    const CgShape shape = cg_shape(c);
    // cooperative: its blocks wait for one another
    MG_CUDA(cudaLaunchCooperativeKernel(shape.fn, dim3(shape.blocks), dim3(shape.threads), args, 0,
                                        c->stream));
    ++c->launches;
    const double pi = 4.0 * std::atan2(1.0, 1.0);
    const double fac = -std::pow(3 / pi, 1 / 3.0) * c->f.e2;
    k_coulomb_out<<<div_up(c->V, kOutThreads), kOutThreads, 0, c->stream>>>(
        c->cpot, c->rho + c->V, c->nx, c->ny, c->nz, c->mx, c->my, fac, c->coulomb, c->coulex);
    MG_LAUNCHED(c);
    MG_CUDA(cudaMemcpyAsync(c->h_cg_status, c->cg_status, 4 * sizeof(int), cudaMemcpyDeviceToHost,
                            c->stream));
    if (iters) {
        MG_CUDA(cudaStreamSynchronize(c->stream));
        *iters = c->h_cg_status[1];
        if (c->h_cg_status[0] == 1) return MG_NOT_CONVERGED;
        return coulomb_status(c);
    }
    return MG_OK;
}

// Whether a wait of the last CG solve ran out, read after a synchronisation behind it;
// reported once.
int coulomb_status(mg_ctx* c) {
    const int st = c->h_cg_status[0];
    if (st != 2 && st != 3) return MG_OK;
    c->h_cg_status[0] = 0;
    return st == 2 ? MG_ERR_TIMEOUT : MG_ERR_CUDA;
}

}  // namespace mg
