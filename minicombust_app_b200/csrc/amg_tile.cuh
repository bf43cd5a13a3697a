// The smoothing halves of a V-cycle level in one kernel each, on levels that
// are boxes in x-fastest order (included by amg.cu).
//
// Three damped-Jacobi sweeps and the restriction of the residual (or, coming
// back up, the prolongation and three sweeps) are seven kernels that each
// stream the level's matrix and vectors: 189 of level 0's 378 bytes per row in
// FP64 each way.  Here a block walks a column of TX x TY cells along z with all
// of a half's steps in flight one plane apart -- at step k it takes plane k in,
// computes the first iterate there, the second on plane k - 1, the third on
// k - 2 and the residual (or last sweep) on k - 3 -- so every array is read from
// HBM once: about 50 bytes per row.  A step needs the one before it on
// neighbouring cells, so three cells of overlap on each side of the tile and
// plane range are computed twice (26 x 10 of 32 x 16 cells are the block's own);
// these re-reads come from L2.  Values of the own column stay in registers, a
// plane of each iterate in shared memory for the x and y neighbours; planes are
// copied to shared memory five steps ahead (cp.async).  A step is bound by the
// chain through shared memory and FP64 arithmetic, 0.65 us a plane at 16 warps: a
// plain pass at 2 x 128^3, with six V-cycles that find work, takes 6.90 ms, 7.21
// by sweeps.  (V-cycle time of an event-timed pass, ten launches: 2.64 ms; with
// what only the own column reads loaded into registers two steps ahead 3.05,
// with the reciprocals a plane ahead and split sums 2.72, by sweeps 3.23.)
#pragma once

#include <type_traits>

namespace mcb {

namespace {

constexpr int TILE_X = 32, TILE_Y = 16, TILE_T = TILE_X * TILE_Y, TILE_H = 3;
constexpr int TILE_UX = TILE_X - 2 * TILE_H, TILE_UY = TILE_Y - 2 * TILE_H;
constexpr int TILE_SLOTS = 8, TILE_AHEAD = 5;  // planes in shared memory; copies run this many steps ahead

// A level as the tile kernels see it: sizes and the couplings of each cell to
// its +x, +y and +z neighbour (the other three are the neighbours').
template <typename T>
struct TileLevel {
    int nx = 0, ny = 0, nz = 0;
    const T *diag = nullptr, *cx = nullptr, *cy = nullptr, *cz = nullptr;
};

template <typename T>
struct TileArgs {
    TileLevel<T> L;
    int zc;            // planes of a block (even)
    T w[3];            // damping of the three sweeps, in order
    const T *r;        // right-hand side
    T *e;              // down: the iterate after three sweeps (out); up: the same (in)
    T *rc;             // down: the coarse right-hand side
    const T *ec;       // up: the coarse correction
    T alpha;           // up: its scaling
    T *eout;           // up: the result, or with zp ...
    typename Pair<T>::type *zp;  // ... z into zp[i].x and r . z into the state
    PcgState *st;
    double *partials;
    unsigned int *counter;
    int is_init;
};

__device__ __forceinline__ void tile_copy(double *dst, const double *src, bool in)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(in ? 8 : 0) : "memory");
}
__device__ __forceinline__ void tile_copy(float *dst, const float *src, bool in)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// Shared memory: five (up: six) arrays of TILE_SLOTS planes, three iterates of
// two planes, the residual's x sums.
template <typename T, bool UP>
constexpr size_t tile_smem()
{
    return sizeof(T) * TILE_T * ((UP ? 6 : 5) * TILE_SLOTS + 6 + 2);
}

template <typename T, bool UP>
__global__ void __launch_bounds__(TILE_T, sizeof(T) == 4 ? 2 : 1) k_amg_tile(const __grid_constant__ TileArgs<T> a)
{
    pdl_wait();
    extern __shared__ __align__(16) unsigned char tile_raw[];
    __shared__ double sh[1][32];
    if (a.st->done) return;
    const int nx = a.L.nx, ny = a.L.ny, nz = a.L.nz, t = threadIdx.x, tx = t & (TILE_X - 1), ty = t / TILE_X;
    const int x = (int)blockIdx.x * TILE_UX - TILE_H + tx, y = (int)blockIdx.y * TILE_UY - TILE_H + ty;
    const int z0 = (int)blockIdx.z * a.zc, z1 = min(z0 + a.zc, nz);
    const bool in = x >= 0 && x < nx && y >= 0 && y < ny;
    const bool own = in && tx >= TILE_H && tx < TILE_X - TILE_H && ty >= TILE_H && ty < TILE_Y - TILE_H;
    const size_t plane = (size_t)nx * ny, col = in ? (size_t)y * nx + x : 0;
    const int cnx = (nx + 1) / 2, cny = (ny + 1) / 2;
    // neighbours in the tile (clamped at its rim, whose values no own cell sees)
    const int txm = max(t - 1, 0), txp = min(t + 1, TILE_T - 1);
    const int tym = max(t - TILE_X, 0), typ = min(t + TILE_X, TILE_T - 1);
    T *const base = reinterpret_cast<T *>(tile_raw);
    auto slot = [&](int array, int k) { return base + ((size_t)array * TILE_SLOTS + (k & (TILE_SLOTS - 1))) * TILE_T; };
    T *const it = base + (size_t)(UP ? 6 : 5) * TILE_SLOTS * TILE_T;  // [3][2][TILE_T]
    T *const sr = it + 6 * TILE_T;
    auto copy_plane = [&](int k) {
        const bool ok = in && k >= 0 && k < nz;
        const size_t i = ok ? (size_t)k * plane + col : 0;
        tile_copy(slot(0, k) + t, a.r + i, ok);
        tile_copy(slot(1, k) + t, a.L.diag + i, ok);
        tile_copy(slot(2, k) + t, a.L.cx + i, ok);
        tile_copy(slot(3, k) + t, a.L.cy + i, ok);
        tile_copy(slot(4, k) + t, a.L.cz + i, ok);
        if (UP) tile_copy(slot(5, k) + t, a.e + i, ok);
    };
    // rings over the planes, index k mod 4
    T r[4], di[4], dg[4], cx[4], cxm[4], cy[4], cym[4], cz[4], a0[4], a1[4], a2[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        r[q] = di[q] = dg[q] = cx[q] = cxm[q] = cy[q] = cym[q] = cz[q] = a0[q] = a1[q] = a2[q] = (T)0;
    }
    for (int q = 0; q < 6; q++) it[(size_t)q * TILE_T + t] = (T)0;
    const int ks = z0 - TILE_H, ke = z1 - 1 + TILE_H;
    for (int q = 0; q < (UP ? 6 : 5); q++) slot(q, ks - 1)[t] = (T)0;
#pragma unroll
    for (int q = 0; q < TILE_AHEAD; q++) {
        copy_plane(ks + q);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    T rsum = (T)0;       // residual of the two planes of a coarse plane
    double dot = 0.0;    // r . z
    // One step: S = step number mod 4 (the rings' index of plane k).
    auto step = [&](auto sc, int k) {
        constexpr int S = decltype(sc)::value;
        constexpr int P1 = (S + 3) & 3, P2 = (S + 2) & 3, P3 = (S + 1) & 3;  // planes k - 1, k - 2, k - 3; k - 4 is S
        const int wr = k & 1, rd = wr ^ 1;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(TILE_AHEAD - 1) : "memory");
        __syncthreads();  // plane k has landed for every thread; the last step's iterates are written
        copy_plane(k + TILE_AHEAD);  // into the slot of plane k - 3, last read a step ago
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        {
            const T *px = slot(2, k - 1), *py = slot(3, k - 1);
            cx[P1] = px[t];
            cxm[P1] = px[txm];
            cy[P1] = py[t];
            cym[P1] = py[tym];
            cz[P1] = slot(4, k - 1)[t];
        }
        r[S] = slot(0, k)[t];
        const T d = slot(1, k)[t];
        const T dinv = d != (T)0 ? (T)1 / d : (T)0;
        if (UP) {
            T v = slot(5, k)[t];
            if (in && k >= 0 && k < nz) v += a.alpha * a.ec[((size_t)(k >> 1) * cny + (y >> 1)) * cnx + (x >> 1)];
            a0[S] = v;
        } else {
            a0[S] = a.w[0] * r[S] * dinv;
        }
        auto nb = [&](const T *p, int P, T c4, const T (&v)[4], int up, int dn) {
            return cx[P] * p[txp] + cxm[P] * p[txm] + cy[P] * p[typ] + cym[P] * p[tym] + cz[P] * v[up] + c4 * v[dn];
        };
        const T s1 = nb(it + (size_t)(0 * 2 + rd) * TILE_T, P1, cz[P2], a0, S, P2);
        a1[P1] = a0[P1] + a.w[UP ? 0 : 1] * ((r[P1] - s1) * di[P1] - a0[P1]);
        const T s2 = nb(it + (size_t)(1 * 2 + rd) * TILE_T, P2, cz[P3], a1, P1, P3);
        a2[P2] = a1[P2] + a.w[UP ? 1 : 2] * ((r[P2] - s2) * di[P2] - a1[P2]);
        // (a2's ring: the plane k - 4 of the last term has index S)
        const T s3 = nb(it + (size_t)(2 * 2 + rd) * TILE_T, P3, cz[S], a2, P2, S);
        const int q = k - TILE_H;  // plane of the last stage
        if (UP) {
            const T z = a2[P3] + a.w[2] * ((r[P3] - s3) * di[P3] - a2[P3]);
            if (own && q >= z0 && q < z1) {
                const size_t i = (size_t)q * plane + col;
                if (a.zp) {
                    a.zp[i].x = z;
                    dot += (double)r[P3] * (double)z;
                } else {
                    a.eout[i] = z;
                }
            }
        } else {
            if (own && k - 2 >= z0 && k - 2 < z1) a.e[(size_t)(k - 2) * plane + col] = a2[P2];
            // restriction: z pair in the thread, x pair by a shuffle, y pair through shared memory a step later
            if (q >= z0 && q < z1) {
                const T res = own ? (r[P3] - s3) - dg[P3] * a2[P3] : (T)0;
                if ((q & 1) == 0) rsum = (T)0;
                rsum += res;
                if ((q & 1) || q == z1 - 1) sr[((q >> 1) & 1) * TILE_T + t] = rsum + __shfl_down_sync(0xffffffffu, rsum, 1);
            }
            const int qp = q - 1;  // the plane whose sums were written in the last step
            if (qp >= z0 && qp < z1 && ((qp & 1) || qp == z1 - 1) && own && !(x & 1) && !(y & 1))
                a.rc[((size_t)(qp >> 1) * cny + (y >> 1)) * cnx + (x >> 1)] =
                    sr[((qp >> 1) & 1) * TILE_T + t] + sr[((qp >> 1) & 1) * TILE_T + t + TILE_X];
        }
        it[(size_t)(0 * 2 + wr) * TILE_T + t] = a0[S];
        it[(size_t)(1 * 2 + wr) * TILE_T + t] = a1[P1];
        it[(size_t)(2 * 2 + wr) * TILE_T + t] = a2[P2];
        di[S] = dinv;
        dg[S] = d;
    };
    // down: one more step writes the last coarse plane
    const int last = UP ? ke : ke + 1;
    for (int k = ks; k <= last; k += 4) {
        step(std::integral_constant<int, 0>{}, k);
        if (k + 1 <= last) step(std::integral_constant<int, 1>{}, k + 1);
        if (k + 2 <= last) step(std::integral_constant<int, 2>{}, k + 2);
        if (k + 3 <= last) step(std::integral_constant<int, 3>{}, k + 3);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (UP && a.zp) {
        const unsigned nb = gridDim.x * gridDim.y * gridDim.z;
        double v[1] = {dot};
        if (publish_sums<1>(v, a.partials, a.counter, sh, (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x,
                            nb)) {
            double tot[1];
            reduce_sums<1>(tot, a.partials, a.counter, sh, nb);
            if (t == 0) {
                PcgState *st = a.st;
                st->rz_old = a.is_init ? 1.0 : st->rz;
                st->rz = tot[0];
                if (!isfinite(tot[0])) {
                    st->done = 1;
                    st->status = KRYLOV_NONFINITE;
                }
            }
        }
    }
}

} // namespace

} // namespace mcb
