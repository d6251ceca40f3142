// mixing.cu -- the reference's mixing between iterations, FP64.
//
//   scheme 0 (default): MixDensities, src/DensityMixing.f90:38-47: every
//     density is mixed with the previous iteration's,
//     Density = (1 - DampingParam) Density + DampingParam DensityHistory(1);
//     UpdateDensities(0) (src/Densities.f90:406-429) keeps the replaced
//     densities as that history.
//   scheme 2: the U update is preconditioned instead,
//     Upot = UpotOld + PreconditionPotential(Upot - UpotOld)
//     and, without time reversal, each component of the S update with the
//     symmetries of s, and with PreConW > 0 each W component's
//     (src/PotentialMixing.f90:143-210,
//     src/Damping.f90:158-228): per isospin
//     a CG on (beta + alpha Lap) x = dU with alpha = -preconu, beta = 1 and
//     the Lagrange Laplacian, at most 300 steps, stopping when
//     sum(residual^2) dv < 1e-8.  Meshes that a cluster's shared memory holds
//     run it as one kernel, a cluster of eight blocks per isospin; on larger
//     ones the host drives the steps: both isospins step together with their
//     own scalars, an isospin that has converged stops changing, and the sums
//     are block partials added on the host in block order (deterministic).
#include <cmath>
#include <vector>

#include "cgsum.cuh"
#include "mg_internal.cuh"

namespace mg {

namespace {

constexpr int kThreads = 256;

__global__ void k_mix(double* __restrict__ x, const double* __restrict__ h, long n, double d) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) x[t] = (1.0 - d) * x[t] + d * h[t];
}

// rho, tau, nablaj, derrho and laprho as one list of 14V values, and their
// history in that order: one launch each to keep and to mix it (with five
// copies UpdateDensities of two spwfs at 8^3 took 39 us, now 20)
struct Densities {
    double* p[5];
};

__device__ __forceinline__ double* density_at(const Densities& d, long t, long V) {
    // rho, tau, nablaj and laprho have 2V values, derrho 6V
    if (t < 6 * V) return t < 2 * V ? d.p[0] + t : (t < 4 * V ? d.p[1] + t - 2 * V : d.p[2] + t - 4 * V);
    return t < 12 * V ? d.p[3] + t - 6 * V : d.p[4] + t - 12 * V;
}

__global__ void k_keep_densities(Densities d, double* __restrict__ h, long V) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 14 * V) h[t] = *density_at(d, t, V);
}

__global__ void k_mix_densities(Densities den, const double* __restrict__ h, long V, double d) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 14 * V) return;
    double* x = density_at(den, t, V);
    *x = (1.0 - d) * *x + d * h[t];
}

__device__ double block_sum(double s, double* red) {
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = s;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < kThreads / 32; ++q) t += red[q];
    return t;
}

// upd = beta dir + alpha lap (isospin blockIdx.y) and block partials of dir.upd
__global__ void __launch_bounds__(kThreads)
k_pc_update(const double* __restrict__ dir, const double* __restrict__ lap,
            double* __restrict__ upd, long V, double alpha, double beta,
            double* __restrict__ part) {
    __shared__ double red[kThreads / 32];
    const int it = blockIdx.y;
    const long v = (long)blockIdx.x * kThreads + threadIdx.x;
    double s = 0.0;
    if (v < V) {
        const long o = it * V + v;
        const double u = beta * dir[o] + alpha * lap[o];
        upd[o] = u;
        s = dir[o] * u;
    }
    const double t = block_sum(s, red);
    if (threadIdx.x == 0) part[(long)it * gridDim.x + blockIdx.x] = t;
}

// inv += a dir, res -= a upd (per isospin), block partials of res.res
__global__ void __launch_bounds__(kThreads)
k_pc_step(double* __restrict__ inv, double* __restrict__ res, const double* __restrict__ dir,
          const double* __restrict__ upd, long V, double a0, double a1,
          double* __restrict__ part) {
    __shared__ double red[kThreads / 32];
    const int it = blockIdx.y;
    const double a = it == 0 ? a0 : a1;
    const long v = (long)blockIdx.x * kThreads + threadIdx.x;
    double s = 0.0;
    if (v < V) {
        const long o = it * V + v;
        inv[o] = inv[o] + a * dir[o];
        const double r = res[o] - a * upd[o];
        res[o] = r;
        s = r * r;
    }
    const double t = block_sum(s, red);
    if (threadIdx.x == 0) part[(long)it * gridDim.x + blockIdx.x] = t;
}

// dir = res + b dir (isospins with b < 0 are left alone: converged)
__global__ void k_pc_direction(double* __restrict__ dir, const double* __restrict__ res, long V,
                               double b0, double b1) {
    const int it = blockIdx.y;
    const double b = it == 0 ? b0 : b1;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V || b < 0.0) return;
    dir[it * V + v] = res[it * V + v] + b * dir[it * V + v];
}

// dir = res = dU, inv = 0, block partials of dU.dU (the potential's
// isospins stride apart)
__global__ void __launch_bounds__(kThreads)
k_pc_start(const double* __restrict__ U, const double* __restrict__ Uold, long stride,
           double* __restrict__ res, double* __restrict__ dir, double* __restrict__ inv, long V,
           double* __restrict__ part) {
    __shared__ double red[kThreads / 32];
    const int it = blockIdx.y;
    const long v = (long)blockIdx.x * kThreads + threadIdx.x;
    double s = 0.0;
    if (v < V) {
        const long o = it * V + v;
        const double d = U[it * stride + v] - Uold[it * stride + v];
        res[o] = d;
        dir[o] = d;
        inv[o] = 0.0;
        s = d * d;
    }
    const double t = block_sum(s, red);
    if (threadIdx.x == 0) part[(long)it * gridDim.x + blockIdx.x] = t;
}

__global__ void k_pc_finish(double* __restrict__ U, const double* __restrict__ Uold, long stride,
                            const double* __restrict__ inv, long V) {
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int it = blockIdx.y;
    if (v < V) U[it * stride + v] = Uold[it * stride + v] + inv[it * V + v];
}

// The whole CG of one potential, a cluster of eight blocks per isospin: every
// rank keeps the residual of the whole mesh in shared memory (its line sums
// read it along all axes) and a slice of the other vectors in registers, R
// points per thread; a step has the two meetings of the cluster that the
// Chronopoulos-Gear recurrences need (J. Comput. Appl. Math. 25 (1989) 153):
// one for the sums r.r and r.Ar, one for the new residual.
struct PcArgs {
    double* F;              // isospins stride apart
    const double* Fold;
    long stride;
    const double* m[3];     // second-derivative matrices of the symmetry class, transposed
    int nx, ny, nz;
    double alpha, beta, dv;
};
constexpr int kPcThreads = 512;
constexpr int kPcMaxIter = 300;

template <int R>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kPcThreads, 1)
k_precondition(PcArgs a) {
    extern __shared__ double sm[];
    __shared__ ClusterSum S;
    if (!in_cluster()) return;
    const int V = a.nx * a.ny * a.nz;
    const int rank = (int)(blockIdx.x % kCluster), it = (int)(blockIdx.x / kCluster);
    double* sx = sm;
    double* sy = sx + a.nx * a.nx;
    double* sz = sy + a.ny * a.ny;
    double* sr = sz + a.nz * a.nz;
    for (int t = threadIdx.x; t < a.nx * a.nx; t += blockDim.x) sx[t] = a.m[0][t];
    for (int t = threadIdx.x; t < a.ny * a.ny; t += blockDim.x) sy[t] = a.m[1][t];
    for (int t = threadIdx.x; t < a.nz * a.nz; t += blockDim.x) sz[t] = a.m[2][t];
    if (threadIdx.x == 0) S.fail = 0;
    cluster_barrier();   // no rank writes to another's shared memory before that one has started
    const int per = (V + kCluster - 1) / kCluster;
    const int v0 = rank * per + threadIdx.x, v1 = min(V, (rank + 1) * per), step = blockDim.x;
    double* F = a.F + it * a.stride;
    const double* Fold = a.Fold + it * a.stride;
    double x[R], r[R], p[R], s[R];   // s = A p
    const auto publish = [&](int v, double value) {
#pragma unroll
        for (int q = 0; q < kCluster; ++q) put_remote(remote(sr + v, q), value);
    };
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int v = v0 + q * step;
        x[q] = p[q] = s[q] = r[q] = 0.0;
        if (v >= v1) continue;
        r[q] = F[v] - Fold[v];
        publish(v, r[q]);
    }
    cluster_barrier();
    double rr_old = 0.0, d_old = 0.0, inv_rr = 0.0, inv_alpha = 0.0;   // of warp 0
    for (int k = 0;; ++k) {
        double rr = 0.0, rw = 0.0, w[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int v = v0 + q * step;
            w[q] = 0.0;
            if (v >= v1) continue;
            const int i = v % a.nx, j = (v / a.nx) % a.ny, l = v / (a.nx * a.ny);
            double lx = 0.0, ly = 0.0, lz = 0.0;
            const double* row = sr + v - i;
#pragma unroll 2
            for (int u = 0; u < a.nx; ++u) lx = fma(sx[u * a.nx + i], row[u], lx);
            const double* col = sr + v - j * a.nx;
#pragma unroll 2
            for (int u = 0; u < a.ny; ++u) ly = fma(sy[u * a.ny + j], col[u * a.nx], ly);
            const double* pil = sr + v - l * a.nx * a.ny;
#pragma unroll 2
            for (int u = 0; u < a.nz; ++u) lz = fma(sz[u * a.nz + l], pil[u * a.nx * a.ny], lz);
            w[q] = fma(a.alpha, lx + ly + lz, a.beta * r[q]);
            rr = fma(r[q], r[q], rr);
            rw = fma(r[q], w[q], rw);
        }
        cluster_sum(S, k & 1, rank, rr, rw, [&]() {
            if (k == 0) return;
            inv_rr = inverse(rr_old);
            inv_alpha = d_old * inv_rr;
        });
        if (threadIdx.x < 32) {
            // beta = rr / rr_old, alpha = rr / (rw - beta rr / alpha_old); a negative
            // beta ends the steps (an identically zero update stays as it is)
            const double b = rr * inv_rr;
            d_old = fma(-b, rr * inv_alpha, rw);
            rr_old = rr;
            const bool done = rr == 0.0 || (k > 0 && rr * a.dv < 1e-8) || k == kPcMaxIter;
            if (threadIdx.x == 0) {
                S.result[0] = rr * inverse(d_old);
                S.result[1] = done ? -1.0 : b;
            }
        }
        __syncthreads();
        const double alpha = S.result[0], beta = S.result[1];
        if (beta < 0.0) break;   // the same on every rank
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int v = v0 + q * step;
            if (v >= v1) continue;
            s[q] = fma(beta, s[q], w[q]);
            const double rn = fma(-alpha, s[q], r[q]);
            publish(v, rn);
            p[q] = fma(beta, p[q], r[q]);
            x[q] = fma(alpha, p[q], x[q]);
            r[q] = rn;
        }
        cluster_barrier();
    }
#pragma unroll
    for (int q = 0; q < R; ++q)
        if (v0 + q * step < v1) F[v0 + q * step] = Fold[v0 + q * step] + x[q];
}

// Where the one-kernel form is taken: the mesh and the matrices fit a block's
// shared memory, and the eight SMs of a cluster are quicker at a step's line
// sums (V (nx + ny + nz) FMAs, two per clock and SM) than the host's loop with
// its five launches and two synchronisations per step.  One potential: 145 us
// against 1605 at 10^3, 0.31 ms against 2.21 at 14^3, 1.80 against 3.27 at
// 24^3, 3.06 against 3.98 at 28^3 (1.84e6 in the units below); the host's loop
// takes 4.4 ms at 29^3, where the cluster would take about as long.
constexpr size_t kPcSmem = 220 * 1024;
constexpr double kPcMaxWork = 2.0e6;

size_t pc_smem(const mg_ctx* c) {
    return ((size_t)c->V + c->nx * c->nx + c->ny * c->ny + c->nz * c->nz) * sizeof(double);
}
bool pc_one_kernel(const mg_ctx* c) {
    return pc_smem(c) <= kPcSmem && (double)c->V * (c->nx + c->ny + c->nz) <= kPcMaxWork;
}

int pc_launch(mg_ctx* c, double* F, const double* Fold, long stride, const int8_t* slot) {
    PcArgs a;
    a.F = F;
    a.Fold = Fold;
    a.stride = stride;
    for (int d = 0; d < 3; ++d) a.m[d] = c->mats + c->mat_off[d][1][slot[d]];
    a.nx = c->nx;
    a.ny = c->ny;
    a.nz = c->nz;
    a.alpha = -c->p.precon_u;
    a.beta = 1.0;
    a.dv = c->dv;
    const int per = (int)((c->V + kCluster - 1) / kCluster);
    int r = 1;
    while (r < 8 && (per + r - 1) / r > 256) r *= 2;
    const void* fn = r == 1   ? (const void*)k_precondition<1>
                     : r == 2 ? (const void*)k_precondition<2>
                     : r == 4 ? (const void*)k_precondition<4>
                              : (const void*)k_precondition<8>;
    const int threads = ((per + r - 1) / r + 31) / 32 * 32;
    if (threads > kPcThreads) return MG_ERR_ARG;
    void* args[] = {&a};
    MG_CUDA(cudaLaunchKernel(fn, dim3(2 * kCluster), dim3(threads), args, pc_smem(c), c->stream));
    MG_LAUNCHED(c);
    return MG_OK;
}

}  // namespace

// Device buffers and the two Laplacian jobs of the preconditioner.
int mixing_setup(mg_ctx* c) {
    const long V = c->V;
    auto A = [&](double** p, long n) {
        return cudaMalloc(p, n * sizeof(double)) == cudaSuccess &&
               cudaMemset(*p, 0, n * sizeof(double)) == cudaSuccess;
    };
    if (!(A(&c->dhist, 14 * V) && A(&c->Uold, 2 * V) && A(&c->pc_buf, 10 * V)))
        return MG_ERR_CUDA;
    if (!c->p.trc && !A(&c->Sold, 6 * V)) return MG_ERR_CUDA;
    if (c->p.precon_w > 0.0 && !A(&c->Wold, 18 * V)) return MG_ERR_CUDA;
    // the Laplacian of the direction: U (P, S, TS, 1); the S components
    // (P, -S, TS, 1), (P, -S, TS, 2), (P, S, TS, 1); the W classes
    // (-P, S, TS, 2) of W_11, W_22, W_33, (-P, S, TS, 1) of W_12, W_21,
    // (-P, -S, TS, 2) of W_13, W_31, (-P, -S, TS, 1) of W_23, W_32
    std::vector<GridJob> jobs(16);
    const int P = c->p.pc, S = c->p.sc, TS = c->p.tsc;
    const int sym[8][3] = {{P, S, 1},   {P, -S, 1},  {P, -S, 2},  {P, S, 1},
                           {-P, S, 2},  {-P, S, 1},  {-P, -S, 2}, {-P, -S, 1}};
    for (int k = 0; k < 8; ++k)
        for (int it = 0; it < 2; ++it) {
            GridJob J{};
            J.in = c->pc_buf + (2 + it) * V;        // direction
            J.lap = c->pc_buf + (6 + it) * V;       // Laplacian of the direction
            for (int d = 0; d < 3; ++d)
                J.slot[d] = c->pc_slots[k][d] =
                    (int8_t)lag_slot(d, sym[k][0], sym[k][1], TS, sym[k][2]);
            jobs[2 * k + it] = J;
        }
    for (const void* fn : {(const void*)k_precondition<1>, (const void*)k_precondition<2>,
                           (const void*)k_precondition<4>, (const void*)k_precondition<8>})
        MG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPcSmem));
    MG_CUDA(cudaMalloc(&c->pc_jobs, jobs.size() * sizeof(GridJob)));
    MG_CUDA(cudaMemcpy(c->pc_jobs, jobs.data(), jobs.size() * sizeof(GridJob),
                       cudaMemcpyHostToDevice));
    return MG_OK;
}

static Densities all_densities(const mg_ctx* c) {
    return Densities{{c->rho, c->tau, c->nablaj, c->derrho, c->laprho}};
}

// UpdateDensities(0): the current densities become the history.
int save_density_history(mg_ctx* c) {
    const long V = c->V;
    k_keep_densities<<<div_up(14 * V, kThreads), kThreads, 0, c->stream>>>(all_densities(c), c->dhist,
                                                                           V);
    MG_LAUNCHED(c);
    if (c->odd)
        MG_CUDA(cudaMemcpyAsync(c->odd_hist, c->odd, c->odd_len * V * sizeof(double),
                                cudaMemcpyDeviceToDevice, c->stream));
    if (c->tensor)
        MG_CUDA(cudaMemcpyAsync(c->jmunu_hist, c->jmunu, 18 * V * sizeof(double),
                                cudaMemcpyDeviceToDevice, c->stream));
    c->have_dhist = true;
    return MG_OK;
}

int mix_densities(mg_ctx* c) {
    if (c->p.mixing_scheme != 0 || !c->have_dhist) return MG_OK;
    const long V = c->V;
    k_mix_densities<<<div_up(14 * V, kThreads), kThreads, 0, c->stream>>>(all_densities(c), c->dhist, V,
                                                                          c->p.damping);
    MG_LAUNCHED(c);
    if (c->odd) {   // the time-odd densities mix with the rest
        k_mix<<<div_up(c->odd_len * V, kThreads), kThreads, 0, c->stream>>>(c->odd, c->odd_hist, c->odd_len * V,
                                                                    c->p.damping);
        MG_LAUNCHED(c);
    }
    if (c->tensor) {   // and J_{mu nu}
        k_mix<<<div_up(18 * V, kThreads), kThreads, 0, c->stream>>>(c->jmunu, c->jmunu_hist,
                                                                    18 * V, c->p.damping);
        MG_LAUNCHED(c);
    }
    return MG_OK;
}

static int read_pair(mg_ctx* c, int nblk, std::vector<double>& h, double out[2]) {
    MG_CUDA(cudaMemcpyAsync(h.data(), c->red, 2 * nblk * sizeof(double), cudaMemcpyDeviceToHost,
                            c->stream));
    MG_CUDA(cudaStreamSynchronize(c->stream));
    for (int it = 0; it < 2; ++it) {
        double s = 0.0;
        for (int q = 0; q < nblk; ++q) s += h[(size_t)it * nblk + q];
        out[it] = s * c->dv;
    }
    return MG_OK;
}

// F = Fold + PreconditionPotential(F - Fold) for a potential whose two
// isospins lie stride apart, with the Laplacian of its symmetry class
static int precondition_pot(mg_ctx* c, double* F, const double* Fold, long stride, int cls) {
    if (pc_one_kernel(c)) return pc_launch(c, F, Fold, stride, c->pc_slots[cls]);
    const GridJob* jobs = c->pc_jobs + 2 * cls;
    const long V = c->V;
    const int nblk = div_up(V, kThreads);
    const dim3 g2(nblk, 2);
    double* res = c->pc_buf;
    double* dir = c->pc_buf + 2 * V;
    double* upd = c->pc_buf + 4 * V;
    double* lap = c->pc_buf + 6 * V;
    double* inv = c->pc_buf + 8 * V;
    const double alpha = -c->p.precon_u, beta = 1.0;
    std::vector<double> h((size_t)2 * nblk);
    double nn[2], dd[2], nn_new[2];
    k_pc_start<<<g2, kThreads, 0, c->stream>>>(F, Fold, stride, res, dir, inv, V, c->red);
    MG_LAUNCHED(c);
    MG_TRY(read_pair(c, nblk, h, nn));
    // an isospin whose update is identically zero keeps it (its first CG
    // step would divide 0 by 0), e.g. W_11 of a functional without J^2 terms
    bool conv[2] = {nn[0] == 0.0, nn[1] == 0.0};
    for (int iter = 1; iter <= 300 && !(conv[0] && conv[1]); ++iter) {
        MG_TRY(run_jobs(c, jobs, 2));
        k_pc_update<<<g2, kThreads, 0, c->stream>>>(dir, lap, upd, V, alpha, beta, c->red);
        MG_LAUNCHED(c);
        MG_TRY(read_pair(c, nblk, h, dd));
        double a[2];
        for (int it = 0; it < 2; ++it) a[it] = conv[it] ? 0.0 : nn[it] / dd[it];
        k_pc_step<<<g2, kThreads, 0, c->stream>>>(inv, res, dir, upd, V, a[0], a[1], c->red);
        MG_LAUNCHED(c);
        MG_TRY(read_pair(c, nblk, h, nn_new));
        double b[2] = {-1.0, -1.0};
        for (int it = 0; it < 2; ++it) {
            if (conv[it]) continue;
            b[it] = nn_new[it] / nn[it];
            nn[it] = nn_new[it];
        }
        k_pc_direction<<<g2, kThreads, 0, c->stream>>>(dir, res, V, b[0], b[1]);
        MG_LAUNCHED(c);
        for (int it = 0; it < 2; ++it)
            if (!conv[it] && nn[it] < 1e-8) conv[it] = true;
    }
    k_pc_finish<<<g2, kThreads, 0, c->stream>>>(F, Fold, stride, inv, V);
    MG_LAUNCHED(c);
    return MG_OK;
}

// Upot = UpotOld + PreconditionPotential(Upot - UpotOld); without time
// reversal each S component the same way
int precondition_u(mg_ctx* c) {
    const long V = c->V;
    MG_TRY(precondition_pot(c, c->U, c->Uold, V, 0));
    if (!c->p.trc)
        for (int m = 0; m < 3; ++m)
            MG_TRY(precondition_pot(c, c->Spot + m * V, c->Sold + m * V, 3 * V, m + 1));
    if (c->Wold) {
        // W (mu, nu) at [it][nu][mu]; its symmetry class by (mu, nu)
        const int cls[3][3] = {{4, 5, 6}, {5, 4, 7}, {6, 7, 4}};
        for (int mu = 0; mu < 3; ++mu)
            for (int nu = 0; nu < 3; ++nu) {
                const long off = (nu * 3 + mu) * V;
                MG_TRY(precondition_pot(c, c->W + off, c->Wold + off, 9 * V, cls[mu][nu]));
            }
    }
    return MG_OK;
}

}  // namespace mg
