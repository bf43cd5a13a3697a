// See krylov_team.cuh.
#include "krylov_team.cuh"

#include <algorithm>
#include <cstdlib>

#include <cooperative_groups.h>

#include "mc_reduce.cuh"

namespace mcb {

namespace {

namespace cg = cooperative_groups;

// Rows of a block up to which a thread holds one; above, two: their gathers
// overlap and half as many warps are left to reduce (16,000 rows in 16 blocks:
// 4.0 us per PCG iteration with one row per thread, 3.5 with two; four were no
// faster).
constexpr int TEAM_R1 = 256;
// Threads of a block: at most 1024 rows in a cluster's blocks, 2048 in the grid's.
template <bool CLUSTER, int RPT>
constexpr int team_threads = RPT == 1 ? TEAM_R1 : CLUSTER ? 512 : 1024;
constexpr int TEAM_CLUSTER = 16;      // blocks of the largest cluster
constexpr unsigned TEAM_POLLS = 1u << 20;  // bound of a grid barrier's wait (about a second)

// Bound of the waits; MC_TEAM_WAIT_POLLS lowers it (to make them run out).
unsigned team_polls()
{
    const char *v = std::getenv("MC_TEAM_WAIT_POLLS");
    if (v && *v) {
        const long n = std::strtol(v, nullptr, 10);
        if (n >= 0 && n < (long)TEAM_POLLS) return (unsigned)n;
    }
    return TEAM_POLLS;
}

// Device memory of the grid form's barrier, as a kernel gets it.
struct TeamMem {
    unsigned int *words;  // arrivals; a block's wait ran out (both zero at the launch)
    double *partials;
    unsigned int polls;
};

// The blocks of the team and their sum-and-barrier.  Every thread of every
// block calls sums() the same number of times; the totals are the same bits in
// every thread, so all blocks take the same branches.
template <bool CLUSTER>
struct Team {
    int rank, size;
    unsigned epoch = 0;
    TeamMem m;
    double (*sw)[32];                 // [3][32] shared
    double (*sp)[3][TEAM_CLUSTER];    // cluster: [2][3][16] shared, filled by the other blocks
    double *tot;                      // [4] shared: totals, tot[3] != 0: a wait ran out

    // Totals of v over the team, and a barrier: what any thread stored before
    // is visible to loads after.  False when this block's wait ran out, which
    // m.words[1] then tells the host: the other blocks need not notice (the
    // last one to arrive waits for none).
    template <int K>
    __device__ __forceinline__ bool sums(double (&v)[K])
    {
        const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
        const int buf = epoch & 1;
        epoch++;
        warp_sums<K>(v, lane);
#pragma unroll
        for (int k = 0; k < K; k++)
            if (lane == ((k & 1) && k < (K & ~1) ? 16 : 0)) sw[k][warp] = v[k];
        __syncthreads();
        if (CLUSTER) {
            cg::cluster_group cl = cg::this_cluster();
            if (warp == 0) {
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const double b = warp_sum_all(lane < nw ? sw[k][lane] : 0.0);
                    if (lane < size) *cl.map_shared_rank(&sp[buf][k][rank], lane) = b;
                }
            }
            cl.sync();
            if (warp == 0) {
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const double s = warp_sum_all(lane < size ? sp[buf][k][lane] : 0.0);
                    if (lane == 0) tot[k] = s;
                }
            }
        } else if (warp == 0) {
            double *part = m.partials + (size_t)buf * 3 * size;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const double b = warp_sum_all(lane < nw ? sw[k][lane] : 0.0);
                if (lane == 0) part[(size_t)k * size + rank] = b;
            }
            if (lane == 0) {
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(m.words) : "memory");
                unsigned seen, polls = 0;
                do {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(m.words) : "memory");
                } while (seen < epoch * (unsigned)size && ++polls < m.polls);
                tot[3] = seen < epoch * (unsigned)size ? 1.0 : 0.0;
                if (seen < epoch * (unsigned)size) *(volatile unsigned int *)(m.words + 1) = 1u;
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < K; k++) {
                double s = 0.0;
                for (int r = lane; r < size; r += 32) s += __ldcg(part + (size_t)k * size + r);
                s = warp_sum_all(s);
                if (lane == 0) tot[k] = s;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = tot[k];
        return CLUSTER || tot[3] == 0.0;
    }
};

// Shared memory of a team kernel's dynamic part: per row of the block six
// couplings, six columns and `extra` further doubles.
size_t team_smem(int rows, int extra) { return (size_t)rows * (6 * 8 + 6 * 4 + 8 * extra); }

#define TEAM_SETUP                                                                                       \
    extern __shared__ double team_smem_base[];                                                           \
    __shared__ double sw[3][32], sp[2][3][TEAM_CLUSTER], stot[4];                                        \
    Team<CLUSTER> team;                                                                                  \
    team.m = m;                                                                                          \
    team.sw = sw;                                                                                        \
    team.sp = sp;                                                                                        \
    team.tot = stot;                                                                                     \
    team.rank = blockIdx.x;                                                                              \
    team.size = gridDim.x;                                                                               \
    const int N = A.N, t = threadIdx.x, nt = blockDim.x, base = blockIdx.x * rows;                                  \
    double *so = team_smem_base;           /* [6][rows] couplings */                                     \
    int *sc = reinterpret_cast<int *>(so + (size_t)6 * rows); /* [6][rows] columns */                    \
    double *se = reinterpret_cast<double *>(sc + (size_t)6 * rows); /* [extra][rows] */                  \
    if (CLUSTER) cg::this_cluster().sync() /* every block has started before its memory is written */

// Rows of a block: thread t holds rows t, t + blockDim, ... of it (`RPT` of them).
template <bool CLUSTER, int RPT>
__global__ void __launch_bounds__((team_threads<CLUSTER, RPT>), 1)
    k_pcg_team(Ell A, PcgVectors v, double rtol, double abs_floor, int max_iters, int use_x0, int rows, TeamMem m)
{
    TEAM_SETUP;
    (void)se;
    double2 *__restrict__ zp = v.zp[0];
    const double mean = v.st->mean;
    double x[RPT], r[RPT], z[RPT], p[RPT], d[RPT], di[RPT], q[RPT];
    bool on[RPT];
    double a3[3] = {0.0, 0.0, 0.0};  // b.b, r.z, r.r
#pragma unroll
    for (int e = 0; e < RPT; e++) {
        const int l = t + e * nt, i = base + l;
        on[e] = l < rows && i < N;
        x[e] = r[e] = z[e] = p[e] = q[e] = 0.0;
        d[e] = di[e] = 1.0;
        if (!on[e]) continue;
        int c[6];
        row_cols(A, i, c);
        d[e] = A.diag[i];
        double ax = 0.0;
        if (use_x0) {
            x[e] = v.x[i];
            ax = d[e] * x[e];
        }
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const double o = ell_val(A.dc, A.off, N, i, k, c[k]);
            so[(size_t)k * rows + l] = o;
            sc[(size_t)k * rows + l] = c[k];
            if (use_x0) ax += o * v.x[c[k]];
        }
        const double bi = v.b[i] - mean;
        r[e] = use_x0 ? bi - ax : bi;
        if (d[e] != 0.0) di[e] = 1.0 / d[e];  // a zero row (isolated cell) is left unpreconditioned
        z[e] = r[e] * di[e];
        zp[i] = make_double2(z[e], 0.0);
        a3[0] += bi * bi;
        a3[1] += r[e] * z[e];
        a3[2] += r[e] * r[e];
    }
    if (!team.sums(a3)) return;
    const double tol = fmax(rtol * sqrt(a3[0]), abs_floor), tol2 = tol * tol;
    double rz = a3[1], rz_old = 1.0, rr = a3[2];
    int iter = 0, status = KRYLOV_OK;
    bool done = a3[0] == 0.0 || rr <= tol2;
    if (!isfinite(a3[0]) || !isfinite(rz)) {
        done = true;
        status = KRYLOV_NONFINITE;
    }
    while (!done) {
        const double beta = iter == 0 ? 0.0 : rz / rz_old;
        double a1[1] = {0.0};
#pragma unroll
        for (int e = 0; e < RPT; e++) {
            if (!on[e]) continue;
            const int l = t + e * nt;
            p[e] = z[e] + beta * p[e];
            double s = d[e] * p[e];
            double2 g[6];
#pragma unroll
            for (int k = 0; k < 6; k++) g[k] = zp[sc[(size_t)k * rows + l]];
#pragma unroll
            for (int k = 0; k < 6; k++) s += so[(size_t)k * rows + l] * (g[k].x + beta * g[k].y);
            q[e] = s;
            a1[0] += p[e] * s;
        }
        if (!team.sums(a1)) {
            status = KRYLOV_TIMEOUT;
            break;
        }
        const double alpha = rz / a1[0];
        if (!isfinite(alpha)) {
            status = KRYLOV_NONFINITE;
            break;
        }
        double a2[2] = {0.0, 0.0};
#pragma unroll
        for (int e = 0; e < RPT; e++) {
            if (!on[e]) continue;
            x[e] += alpha * p[e];
            r[e] -= alpha * q[e];
            z[e] = r[e] * di[e];
            zp[base + t + e * nt] = make_double2(z[e], p[e]);
            a2[0] += r[e] * z[e];
            a2[1] += r[e] * r[e];
        }
        if (!team.sums(a2)) {
            status = KRYLOV_TIMEOUT;
            break;
        }
        rz_old = rz;
        rz = a2[0];
        rr = a2[1];
        iter++;
        if (!isfinite(rz) || !isfinite(rr)) {
            status = KRYLOV_NONFINITE;
            done = true;
        } else if (rr <= tol2) {
            done = true;
        } else if (iter >= max_iters) {
            status = KRYLOV_NOT_CONVERGED;
            done = true;
        }
    }
    double xm = 0.0;
    if (status != KRYLOV_TIMEOUT && (iter > 0 || use_x0)) {
        double a1[1] = {0.0};
#pragma unroll
        for (int e = 0; e < RPT; e++) a1[0] += x[e];
        if (!team.sums(a1)) status = KRYLOV_TIMEOUT;
        xm = a1[0] / (double)N;
    }
#pragma unroll
    for (int e = 0; e < RPT; e++)
        if (on[e]) v.x[base + t + e * nt] = x[e] - xm;
    if (blockIdx.x == 0 && t == 0) {
        PcgState *st = v.st;
        st->bb = a3[0];
        st->rz = rz;
        st->rz_old = rz_old;
        st->rr = rr;
        st->tol2 = tol2;
        st->xmean = xm;
        st->iter = iter;
        st->max_iters = max_iters;
        st->done = 1;
        st->status = status;
    }
}

template <bool CLUSTER, int RPT>
__global__ void __launch_bounds__((team_threads<CLUSTER, RPT>), 1)
    k_bicg_team(Ell A, const double *__restrict__ b, double *__restrict__ xout, double2 *rp, double *vv0, double *vv1,
                BicgState<1> *st, double rtol, int max_iters, int rows, TeamMem m)
{
    TEAM_SETUP;
    double *sx = se, *sr0 = se + rows;  // own rows only
    double r[RPT], p[RPT], vn[RPT], d[RPT], s[RPT], tt[RPT];
    bool on[RPT];
    double a1[1] = {0.0};
#pragma unroll
    for (int e = 0; e < RPT; e++) {
        const int l = t + e * nt, i = base + l;
        on[e] = l < rows && i < N;
        r[e] = p[e] = vn[e] = d[e] = s[e] = tt[e] = 0.0;
        if (!on[e]) continue;
        int c[6];
        row_cols(A, i, c);
        d[e] = A.diag[i];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            so[(size_t)k * rows + l] = ell_val(A.dc, A.off, N, i, k, c[k]);
            sc[(size_t)k * rows + l] = c[k];
        }
        r[e] = b[i];
        sr0[l] = r[e];
        sx[l] = 0.0;
        rp[i] = make_double2(r[e], 0.0);
        vv0[i] = 0.0;
        a1[0] += r[e] * r[e];
    }
    bool fine = team.sums(a1);
    const double bb = a1[0], tol2 = rtol * rtol * bb;
    double rho = 1.0, rho_new = bb, alpha = 1.0, omega = 1.0, rr = bb;
    int iter = 0, status = isfinite(bb) ? KRYLOV_OK : KRYLOV_NONFINITE;
    bool done = !fine || bb == 0.0 || !isfinite(bb);
    while (!done) {
        // p = r + beta (p - omega v) on the own row and, evaluated there, the
        // neighbours'; v = A p
        const double beta = (rho_new / rho) * (alpha / omega);
        double *const vo = (iter & 1) ? vv1 : vv0, *const vw = (iter & 1) ? vv0 : vv1;
        a1[0] = 0.0;
#pragma unroll
        for (int e = 0; e < RPT; e++) {
            if (!on[e]) continue;
            const int l = t + e * nt;
            p[e] = r[e] + beta * (p[e] - omega * vn[e]);
            double2 g[6];
            double h[6];
#pragma unroll
            for (int k = 0; k < 6; k++) {
                const int c = sc[(size_t)k * rows + l];
                g[k] = rp[c];
                h[k] = vo[c];
            }
            double q = d[e] * p[e];
#pragma unroll
            for (int k = 0; k < 6; k++) q += so[(size_t)k * rows + l] * (g[k].x + beta * (g[k].y - omega * h[k]));
            vn[e] = q;
            vw[base + l] = q;
            a1[0] += sr0[l] * q;
        }
        if (!(fine = team.sums(a1))) break;
        alpha = rho_new / a1[0];
        if (!isfinite(alpha)) {
            status = KRYLOV_NONFINITE;
            break;
        }
        // s = r - alpha v; t = A s
        double a2[2] = {0.0, 0.0};
#pragma unroll
        for (int e = 0; e < RPT; e++) {
            if (!on[e]) continue;
            const int l = t + e * nt;
            s[e] = r[e] - alpha * vn[e];
            double g[6], h[6];
#pragma unroll
            for (int k = 0; k < 6; k++) {
                const int c = sc[(size_t)k * rows + l];
                g[k] = rp[c].x;
                h[k] = vw[c];
            }
            double q = d[e] * s[e];
#pragma unroll
            for (int k = 0; k < 6; k++) q += so[(size_t)k * rows + l] * (g[k] - alpha * h[k]);
            tt[e] = q;
            a2[0] += q * s[e];
            a2[1] += q * q;
        }
        if (!(fine = team.sums(a2))) break;
        omega = a2[1] != 0.0 ? a2[0] / a2[1] : 0.0;
        // x += alpha p + omega s; r = s - omega t
        a2[0] = a2[1] = 0.0;
#pragma unroll
        for (int e = 0; e < RPT; e++) {
            if (!on[e]) continue;
            const int l = t + e * nt;
            sx[l] += alpha * p[e] + omega * s[e];
            r[e] = s[e] - omega * tt[e];
            rp[base + l] = make_double2(r[e], p[e]);
            a2[0] += sr0[l] * r[e];
            a2[1] += r[e] * r[e];
        }
        if (!(fine = team.sums(a2))) break;
        rho = rho_new;
        rho_new = a2[0];
        rr = a2[1];
        iter++;
        if (!isfinite(rho_new) || !isfinite(rr)) {
            status = KRYLOV_NONFINITE;
            done = true;
        } else if (rr <= tol2) {
            done = true;
        } else if (omega == 0.0 || rho_new == 0.0 || iter >= max_iters) {
            status = KRYLOV_NOT_CONVERGED;
            done = true;
        }
    }
#pragma unroll
    for (int e = 0; e < RPT; e++) {
        const int l = t + e * nt;
        if (on[e]) xout[base + l] = sx[l];
    }
    if (blockIdx.x == 0 && t == 0) {
        st->bb[0] = bb;
        st->rr[0] = rr;
        st->tol2[0] = tol2;
        st->rho[0] = rho;
        st->rho_new[0] = rho_new;
        st->alpha[0] = alpha;
        st->omega[0] = omega;
        st->iter[0] = iter;
        st->done[0] = 1;
        st->status[0] = status;
        st->all_done = 1;
        st->max_iters = max_iters;
    }
}

#undef TEAM_SETUP

// The team for N rows: a cluster up to 16 x 1024 rows (its sum costs 1.1 us,
// the grid's 2.5 us), then one block per SM with one or two rows per thread.
// Blocks get 128 rows or more: fewer gain nothing from another SM.  Larger
// systems stream from memory, and the per-kernel solvers' full occupancy makes
// the better use of that.
struct TeamShape {
    bool cluster = false;
    int blocks = 0, threads = 0, rows = 0, rpt = 0;
    int smem_max = 0;  // dynamic shared memory a block may have
};
constexpr int TEAM_STATIC_SMEM = 2048;  // at least the static part of a team kernel

TeamShape team_shape(int N)
{
    TeamShape s;
    int dev = 0, sms = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return s;
    s.smem_max = optin - TEAM_STATIC_SMEM;
    if (N <= TEAM_CLUSTER * 1024) {
        s.cluster = true;
        s.blocks = std::max(1, N / 128);
        if (s.blocks > 8) s.blocks = s.blocks >= TEAM_CLUSTER ? TEAM_CLUSTER : 8;
    } else if (N <= sms * 2048) {
        s.blocks = sms;
    } else {
        return s;
    }
    s.rows = (N + s.blocks - 1) / s.blocks;
    s.rpt = s.rows <= TEAM_R1 ? 1 : 2;
    s.threads = ((s.rows + s.rpt - 1) / s.rpt + 31) / 32 * 32;
    return s;
}

// Launch k on the team, or false (no error left behind) when the device does
// not take the launch.
template <typename... KArgs, typename... Args>
bool team_launch(void (*k)(KArgs...), const TeamShape &sh, size_t smem, cudaStream_t s, unsigned int *words,
                 Args &&...args)
{
    // (a kernel's limit is shared by the process: always the same value, so that
    // a thread with a smaller system does not lower another's between its two calls)
    bool ok = smem <= (size_t)sh.smem_max &&
              cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sh.smem_max) == cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(sh.blocks);
    cfg.blockDim = dim3(sh.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (sh.cluster) {
        if (sh.blocks > 8)
            ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = sh.blocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        int fit = 0;
        ok = ok && cudaOccupancyMaxActiveClusters(&fit, k, &cfg) == cudaSuccess && fit > 0;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        int fit = 0;
        ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k, sh.threads, smem) == cudaSuccess && fit > 0;
        // (a cluster waits in hardware: its words stay zero, as the state's memory was made)
        ok = ok && cudaMemsetAsync(words, 0, 2 * sizeof(unsigned int), s) == cudaSuccess;
    }
    ok = ok && cudaLaunchKernelEx(&cfg, k, static_cast<Args &&>(args)...) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
}

} // namespace

bool pcg_team(cudaStream_t s, const Ell &A, const PcgVectors &v, double rtol, double abs_floor, int max_iters,
              int use_x0)
{
    const TeamShape sh = team_shape(A.N);
    if (!sh.blocks) return false;
    const size_t smem = team_smem(sh.rows, 0);
    auto k = sh.rpt == 1 ? (sh.cluster ? k_pcg_team<true, 1> : k_pcg_team<false, 1>)
                         : (sh.cluster ? k_pcg_team<true, 2> : k_pcg_team<false, 2>);
    return team_launch(k, sh, smem, s, v.st->team, A, v, rtol, abs_floor, max_iters, use_x0, sh.rows,
                       TeamMem{v.st->team, v.partials, team_polls()});
}

bool bicg_team(cudaStream_t s, const Ell &A, const double *b, double *x, double2 *rp, double *vv0, double *vv1,
               double *partials, BicgState<1> *st, double rtol, int max_iters)
{
    const TeamShape sh = team_shape(A.N);
    if (!sh.blocks) return false;
    const size_t smem = team_smem(sh.rows, 2);
    auto k = sh.rpt == 1 ? (sh.cluster ? k_bicg_team<true, 1> : k_bicg_team<false, 1>)
                         : (sh.cluster ? k_bicg_team<true, 2> : k_bicg_team<false, 2>);
    return team_launch(k, sh, smem, s, st->team, A, b, x, rp, vv0, vv1, st, rtol, max_iters, sh.rows,
                       TeamMem{st->team, partials, team_polls()});
}

} // namespace mcb
