// kernels_bottom.cu -- coarsest-level solve: the exact product with the inverse
// of the level's operator where that is small enough, else BiCGStab in one CTA.
//
// BiCGStab restates AMReX MLMG's bottom step as Alamo configures it
// (Solver/Nonlocal/Linear.H:258 selects BiCGStab):
//   cor = 0; BiCGStab on the diagonally scaled system (MLCGSolver::solve_bicgstab
//   with Operator<Node>::normalize = divide by the diagonal, Operator.cpp:156-165);
//   a failed solve (anything but a clean convergence) zeroes the correction;
//   then `bottom_smooth` (after success) or `final_smooth` (after failure)
//   Fsmooth calls of 2 damped-Jacobi sweeps each.
// On a fully periodic box (singular: rigid translations) the Krylov residual
// and every operator application are projected to zero mean per component
// before the diagonal scaling, so that BiCGStab works on a consistent system;
// the smoothing uses the right-hand side as given.
// Every loop is bounded by maxiter / the smoothing counts; there is no
// spin-wait.  The return code lands in ret_slot: 0 converged, 1-4 breakdown,
// 8 not converged in maxiter.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>


#include "agb_internal.h"
#include "stencil.cuh"
#include "bottom.cuh"

namespace agb {

constexpr int BOT_THREADS = 512;

__device__ __forceinline__ double blk_sum(double v, double* red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0;
    if (threadIdx.x < 32) {
        t = threadIdx.x < (BOT_THREADS / 32) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

__device__ __forceinline__ double blk_max(double v, double* red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        double w = __shfl_xor_sync(0xffffffffu, v, o);
        v = (w > v || w != w) ? w : v;
    }
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = threadIdx.x < (BOT_THREADS / 32) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            double w = __shfl_xor_sync(0xffffffffu, t, o);
            t = (w > t || w != w) ? w : t;
        }
        if (threadIdx.x == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

struct BotAcc {
    const double* x;
    const double* c;
    long long S;
    long long base;
    long long o[3][3];
    __device__ __forceinline__ long long off(int di, int dj, int dk) const
    {
        return base + o[0][di + 1] + o[1][dj + 1] + o[2][dk + 1];
    }
    __device__ __forceinline__ double u(int p, int di, int dj, int dk) const { return x[p * S + off(di, dj, dk)]; }
    __device__ __forceinline__ double C(int m, int di, int dj, int dk) const { return c[m * S + off(di, dj, dk)]; }
};

// y = A x over all nodes of the level (threads stride over nodes)
template <int SYM>
__device__ void cta_apply(const LevelDesc& L, const BCTable& bc, const Geo<double>& g, int uniform,
                          const double* ddw, const double* x, double* y)
{
    const long long cnt = L.count();
    const long long st[3] = {1, (long long)L.P, (long long)L.P * L.nn[1]};
    for (long long e = threadIdx.x; e < cnt; e += blockDim.x) {
        const int i = (int)(e % L.nn[0]);
        const int j = (int)((e / L.nn[0]) % L.nn[1]);
        const int k = (int)(e / ((long long)L.nn[0] * L.nn[1]));
        const int pos[3] = {i, j, k};
        BotAcc acc;
        acc.x = x;
        acc.c = ddw;
        acc.S = L.S;
        acc.base = L.idx(i, j, k);
        int mn[3], mx[3];
        bool bnd = false;
        for (int d = 0; d < 3; d++) {
            mn[d] = !L.per[d] && pos[d] == 0;
            mx[d] = !L.per[d] && pos[d] == L.n[d];
            bnd = bnd || mn[d] || mx[d];
            acc.o[d][0] = -st[d];
            acc.o[d][1] = 0;
            acc.o[d][2] = st[d];
            if (L.per[d]) {
                if (pos[d] == 0) acc.o[d][0] = st[d] * (L.n[d] - 1);
                if (pos[d] == L.n[d] - 1) acc.o[d][2] = -st[d] * (L.n[d] - 1);
            }
        }
        double f[3];
        if (bnd) boundary_row<double, SYM>(acc, g, bc, mn, mx, f);
        else interior_row<double, SYM>(acc, g, uniform != 0, f);
        for (int c = 0; c < 3; c++) y[c * L.S + acc.base] = f[c];
    }
}

// per-component means over the level's nodes (every stored node is unique on
// a fully periodic level)
__device__ void cta_mean3(const LevelDesc& L, const double* v, double* red, double m[3])
{
    const long long cnt = L.count();
    double s0 = 0, s1 = 0, s2 = 0;
    for (long long e = threadIdx.x; e < cnt; e += blockDim.x) {
        const long long q = L.idx((int)(e % L.nn[0]), (int)((e / L.nn[0]) % L.nn[1]),
                                  (int)(e / ((long long)L.nn[0] * L.nn[1])));
        s0 += v[q];
        s1 += v[L.S + q];
        s2 += v[2 * L.S + q];
    }
    m[0] = blk_sum(s0, red) / (double)cnt;
    m[1] = blk_sum(s1, red) / (double)cnt;
    m[2] = blk_sum(s2, red) / (double)cnt;
}

#define FOR_NODES(q)                                                                                     \
    for (long long e_ = threadIdx.x; e_ < cnt; e_ += blockDim.x)                                         \
        for (int c_ = 0, i_ = (int)(e_ % L.nn[0]), j_ = (int)((e_ / L.nn[0]) % L.nn[1]),                  \
                 k_ = (int)(e_ / ((long long)L.nn[0] * L.nn[1]));                                        \
             c_ < 3; c_++)                                                                               \
            for (long long q = c_ * L.S + L.idx(i_, j_, k_), once_ = 0; once_ < 1; once_++)

// cor = A^-1 res with the inverse row-major, in the inverse's arithmetic I: one
// row a warp, the right-hand side in shared memory.  Every CTA of the grid takes
// its rows.
template <typename T, typename I>
__device__ __forceinline__ void exact_product(const LevelDesc& L, const I* __restrict__ inv, T* __restrict__ cor,
                                              const T* __restrict__ res, I* __restrict__ xs, int* ret_slot)
{
    const int cnt = (int)L.count(), nu = 3 * cnt;
    for (int q = threadIdx.x; q < nu; q += blockDim.x) xs[q] = (I)__ldcg(res + dense_to_padded(L, q, cnt));
    __syncthreads();
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int row = blockIdx.x * nw + (threadIdx.x >> 5); row < nu; row += gridDim.x * nw) {
        const I* a = inv + (long long)row * nu;
        I y0 = 0, y1 = 0;
        int j = lane;
        for (; j + 32 < nu; j += 64) {
            y0 += a[j] * xs[j];
            y1 += a[j + 32] * xs[j + 32];
        }
        if (j < nu) y0 += a[j] * xs[j];
        y0 += y1;
        for (int o = 16; o > 0; o >>= 1) y0 += __shfl_xor_sync(0xffffffffu, y0, o);
        if (lane == 0) cor[dense_to_padded(L, row, cnt)] = (T)y0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && ret_slot) *ret_slot = 0;
}

template <typename T, int SYM>
__global__ void __launch_bounds__(BOT_THREADS) k_bottom(LevelDesc L, BCTable bc, Geo<double> g, int uniform,
                                                        const double* __restrict__ ddw,
                                                        const double* __restrict__ diag, T* __restrict__ cor,
                                                        const T* __restrict__ res, double* __restrict__ work,
                                                        int maxiter, double eps_rel, double eps_abs, int nub,
                                                        int nuf, double omega, int* ret_slot,
                                                        const double* __restrict__ inv, const int* __restrict__ inv_ok)
{
    __shared__ double red[33];
    if (inv && *inv_ok) {
        extern __shared__ __align__(16) unsigned char bsm_raw[];
        exact_product(L, inv, cor, res, reinterpret_cast<double*>(bsm_raw), ret_slot);
        return;
    }
    if (blockIdx.x) return;   // the BiCGStab solve is one CTA's
    const long long n3 = 3 * L.S, cnt = L.count();
    double *r = work, *rh = work + n3, *p = work + 2 * n3, *v = work + 3 * n3, *s = work + 4 * n3,
           *t = work + 5 * n3, *sol = work + 6 * n3, *b = work + 7 * n3;
    FOR_NODES(q)
    {
        b[q] = (double)res[q];
        sol[q] = 0.0;
    }
    __syncthreads();
    const bool sing = L.singular();
    double mb[3] = {0, 0, 0};
    if (sing) cta_mean3(L, b, red, mb);
    // r = P(b - A*0)/D, P the zero-mean projection on a singular level (identity otherwise)
    double lm = 0;
    FOR_NODES(q)
    {
        r[q] = (b[q] - mb[c_]) / diag[q];
        rh[q] = r[q];
        const double a = fabs(r[q]);
        lm = (a > lm || a != a) ? a : lm;
    }
    double rnorm = blk_max(lm, red);
    const double rnorm0 = rnorm;
    int ret = 0;
    double rho_1 = 0, alpha = 0, om = 0;
    if (!(rnorm0 == 0 || rnorm0 < eps_abs)) {
        for (int iter = 1; iter <= maxiter; iter++) {
            double acc = 0;
            FOR_NODES(q) acc += rh[q] * r[q];
            const double rho = blk_sum(acc, red);
            if (rho == 0) { ret = 1; break; }
            if (iter == 1) {
                FOR_NODES(q) p[q] = r[q];
            } else {
                const double beta = (rho / rho_1) * (alpha / om);
                FOR_NODES(q) p[q] = r[q] + beta * (p[q] - om * v[q]);
            }
            __syncthreads();
            cta_apply<SYM>(L, bc, g, uniform, ddw, p, v);
            __syncthreads();
            double mv[3] = {0, 0, 0};
            if (sing) cta_mean3(L, v, red, mv);
            acc = 0;
            FOR_NODES(q)
            {
                v[q] = (v[q] - mv[c_]) / diag[q];
                acc += rh[q] * v[q];
            }
            const double rhTv = blk_sum(acc, red);
            if (rhTv != 0) alpha = rho / rhTv;
            else { ret = 2; break; }
            lm = 0;
            FOR_NODES(q)
            {
                sol[q] += alpha * p[q];
                s[q] = r[q] - alpha * v[q];
                const double a = fabs(s[q]);
                lm = (a > lm || a != a) ? a : lm;
            }
            rnorm = blk_max(lm, red);
            if (rnorm < eps_rel * rnorm0 || rnorm < eps_abs) break;
            cta_apply<SYM>(L, bc, g, uniform, ddw, s, t);
            __syncthreads();
            double mt[3] = {0, 0, 0};
            if (sing) cta_mean3(L, t, red, mt);
            double tt = 0, ts = 0;
            FOR_NODES(q)
            {
                t[q] = (t[q] - mt[c_]) / diag[q];
                tt += t[q] * t[q];
                ts += t[q] * s[q];
            }
            tt = blk_sum(tt, red);
            ts = blk_sum(ts, red);
            if (tt != 0) om = ts / tt;
            else { ret = 3; break; }
            lm = 0;
            FOR_NODES(q)
            {
                sol[q] += om * s[q];
                r[q] = s[q] - om * t[q];
                const double a = fabs(r[q]);
                lm = (a > lm || a != a) ? a : lm;
            }
            rnorm = blk_max(lm, red);
            if (rnorm < eps_rel * rnorm0 || rnorm < eps_abs) break;
            if (om == 0) { ret = 4; break; }
            rho_1 = rho;
        }
        if (ret == 0 && rnorm > eps_rel * rnorm0 && rnorm > eps_abs) ret = 8;
        if (!((ret == 0 || ret == 8) && rnorm < rnorm0)) {
            FOR_NODES(q) sol[q] = 0.0;
        }
        // MLMG::actualBottomSolve: anything but a clean solve discards the correction
        if (ret != 0) {
            FOR_NODES(q) sol[q] = 0.0;
        }
    }
    __syncthreads();
    // post-smoothing: Fsmooth = 2 Jacobi sweeps each
    const int nsm = 2 * ((ret == 0) ? nub : nuf);
    for (int sw = 0; sw < nsm; sw++) {
        cta_apply<SYM>(L, bc, g, uniform, ddw, sol, t);
        __syncthreads();
        FOR_NODES(q)
        {
            const double Rx = t[q] - sol[q] * diag[q];
            s[q] = (1. - omega) * sol[q] + omega * (b[q] - Rx) / diag[q];
        }
        __syncthreads();
        FOR_NODES(q) sol[q] = s[q];
        __syncthreads();
    }
    FOR_NODES(q) cor[q] = (T)sol[q];
    if (threadIdx.x == 0 && ret_slot) *ret_slot = ret;
}

// Neighbour offsets of node (i,j,k) in the padded layout, periodic wrap included.
struct UnitAcc {
    const double* c;
    long long S, base, unit;   // unit: padded node index of the unit vector's node
    int comp;                  // and its component
    long long o[3][3];
    __device__ __forceinline__ long long off(int di, int dj, int dk) const
    {
        return base + o[0][di + 1] + o[1][dj + 1] + o[2][dk + 1];
    }
    __device__ __forceinline__ double u(int p, int di, int dj, int dk) const
    {
        return (p == comp && off(di, dj, dk) == unit) ? 1.0 : 0.0;
    }
    __device__ __forceinline__ double C(int m, int di, int dj, int dk) const { return c[m * S + off(di, dj, dk)]; }
};

// A (column-major, entry (row r, column j) at j * nu + r) of the level:
// one thread per (row node, column unknown), rows of its three components.
template <int SYM>
__global__ void k_bottom_assemble(LevelDesc L, BCTable bc, Geo<double> g, int uniform,
                                  const double* __restrict__ ddw, double* __restrict__ A)
{
    const int cnt = (int)L.count(), nu = 3 * cnt;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= cnt * nu) return;
    const int e = t % cnt, col = t / cnt;
    const int i = e % L.nn[0], j = (e / L.nn[0]) % L.nn[1], k = e / (L.nn[0] * L.nn[1]);
    const int ce = col % cnt;
    UnitAcc acc;
    acc.c = ddw;
    acc.S = L.S;
    acc.base = L.idx(i, j, k);
    acc.comp = col / cnt;
    const int cpos[3] = {ce % L.nn[0], (ce / L.nn[0]) % L.nn[1], ce / (L.nn[0] * L.nn[1])};
    acc.unit = L.idx(cpos[0], cpos[1], cpos[2]);
    const long long st[3] = {1, (long long)L.P, (long long)L.P * L.nn[1]};
    const int pos[3] = {i, j, k};
    int mn[3], mx[3];
    bool bnd = false;
    for (int d = 0; d < 3; d++) {
        mn[d] = !L.per[d] && pos[d] == 0;
        mx[d] = !L.per[d] && pos[d] == L.n[d];
        bnd = bnd || mn[d] || mx[d];
        acc.o[d][0] = -st[d];
        acc.o[d][1] = 0;
        acc.o[d][2] = st[d];
        if (L.per[d]) {
            if (pos[d] == 0) acc.o[d][0] = st[d] * (L.n[d] - 1);
            if (pos[d] == L.n[d] - 1) acc.o[d][2] = -st[d] * (L.n[d] - 1);
        }
    }
    bool near = true;   // a row reaches the 26 neighbours (periodic images included) only
    for (int d = 0; d < 3; d++) {
        const int a = abs(cpos[d] - pos[d]);
        near = near && (a <= 1 || (L.per[d] && a == L.n[d] - 1));
    }
    double f[3] = {0, 0, 0};
    if (near) {
        if (bnd) boundary_row<double, SYM>(acc, g, bc, mn, mx, f);
        else interior_row<double, SYM>(acc, g, uniform != 0, f);
    }
    for (int c = 0; c < 3; c++) A[(long long)col * nu + c * cnt + e] = f[c];
}

// The CTA copies the operator (FP64, column-major) into shared memory in R.
template <typename R> __device__ __forceinline__ void dense_load(R* A, const double* __restrict__ Ag, int nu)
{
    for (int q = threadIdx.x; q < nu * nu; q += blockDim.x) A[q] = (R)Ag[q];
}

// With `inv` set and *inv_ok (an exact inverse exists, launch_bottom_invert),
// the bottom is the product cor = A^-1 res instead of the BiCGStab solve.
template <typename T, typename R>
__global__ void __launch_bounds__(DENSE_MAX) k_bottom_dense(LevelDesc L, const double* __restrict__ Ag,
                                                            const double* __restrict__ diag, T* __restrict__ cor,
                                                            const T* __restrict__ res, int maxiter, double eps_rel_d,
                                                            double eps_abs_d, int nub, int nuf, double omega_d,
                                                            int* ret_slot, const T* __restrict__ inv,
                                                            const int* __restrict__ inv_ok)
{
    pdl_entry();
    extern __shared__ __align__(16) unsigned char dsm_raw[];
    __shared__ R red[2 * 3 * 32];
    const int nu = 3 * (int)L.count();
    if (inv && *inv_ok) {
        exact_product(L, inv, cor, res, reinterpret_cast<T*>(dsm_raw), ret_slot);
        return;
    }
    if (blockIdx.x) return;   // the BiCGStab solve is one CTA's
    R* A = reinterpret_cast<R*>(dsm_raw);
    dense_load<R>(A, Ag, nu);
    __syncthreads();
    R* xs = A + nu * nu;
    dense_bottom_block<T, R>(L, DenseRow<R>{A, xs, nu, (int)threadIdx.x}, xs, red, diag, cor, res, maxiter, eps_rel_d,
                             eps_abs_d, nub, nuf, omega_d, ret_slot);
}

bool bottom_dense_fits(const LevelDesc& L) { return 3 * L.count() <= DENSE_MAX; }

// ---------------------------------------------------------------------------
// Exact coarsest solve.  Once per solve the dense operator (FP64,
// column-major) is inverted by Gauss-Jordan elimination with partial pivoting
// in FP64 and stored row-major in FP64, or in FP32 for the FP32 cycles of a level
// of up to DENSE_MAX unknowns, whose BiCGStab is in FP32 as well.  (Above, the
// BiCGStab of both is FP64, and so is the product: an inverse in 24 bits is off
// by the level's condition times 6e-8, which grows with the level.)  A
// displacement row is 1 and an interior row C/dx^2, so each row is first scaled
// to a largest |entry| in [1, 2) by a power of two, which the columns of the
// inverse take back: (S A)^-1 S = A^-1, exact, and the same pivots in any units.  A
// fully periodic level (singular), or a pivot at or below 1e-13 of the scaled
// rows, clears *ok and the cycles keep the BiCGStab bottom.  (Compared with the
// largest entry of the whole matrix instead, a level of 2^3 cells has a smallest
// pivot of 2e-2 with C = 1 on a unit box and 1e-17 with C = 2e11 on one of 1 cm.)
//
// BiCGStab runs in one CTA, whose SM has two FP64 lanes per clock and whose
// reductions are barriers: 37 us (isotropic) to 248 us a call on 81 unknowns,
// 2.7 ms on the 588 of a 6 x 6 x 3-cell level, six calls and more a cycle.
// The product takes 4 to 6 us and the inversion is paid once per solve (0.3 ms
// for 81 unknowns; 4.8 ms for 588, of which 74 panels are 53 us each): the FP64 solve of a 65^3 polycrystal (81
// unknowns) went from 176 to 113 ms, the mixed solve of a 96 x 96 x 48-cell
// one (588) from 391 to 34 ms.  Above EXACT_MAX the inversion (cubic in the
// unknowns) and its two copies of the matrix cost more than they save.
//
// Up to DENSE_MAX unknowns the matrix fits the shared memory of one CTA
// (k_bottom_invert).  Up to EXACT_MAX it is eliminated eight columns at a
// time: k_inv_panel (one CTA, a row or two of the panel in each thread's
// registers) runs the eight steps with their row interchanges and leaves the
// panel's transformation T; k_inv_update applies it to every other column,
// new(r, c) = (r in panel ? 0 : old(perm r, c)) + sum_q T(r, q) old(perm(k + q), c),
// from one copy of the matrix into another, so that its tiles are independent.
// ---------------------------------------------------------------------------
constexpr double PIVOT_MIN = 1e-13;

// Power of two that brings a row whose largest |entry| is amax to [1, 2) (NaN
// for an infinite entry, which no pivot passes).
__device__ __forceinline__ double row_factor(double amax)
{
    if (amax == 0.0) return 1.0;
    return isinf(amax) ? amax - amax : scalbn(1.0, min(-ilogb(amax), 1000));
}

__global__ void __launch_bounds__(1024) k_bottom_invert(LevelDesc L, const double* __restrict__ Ag,
                                                       double* __restrict__ inv64, float* __restrict__ inv32,
                                                       int* __restrict__ ok)
{
    extern __shared__ __align__(16) unsigned char inv_raw[];
    double* M = reinterpret_cast<double*>(inv_raw);   // nu x nu, row-major
    __shared__ double fcol[DENSE_MAX], scale[DENSE_MAX];
    __shared__ int piv[DENSE_MAX];
    __shared__ double pinv_s;
    __shared__ int bad_s;
    const int nu = 3 * (int)L.count();
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    if (L.singular() || nu > DENSE_MAX) {
        if (tid == 0) *ok = 0;
        return;
    }
    for (int t = tid; t < nu * nu; t += nt) M[(t % nu) * nu + t / nu] = Ag[t];
    if (tid == 0) bad_s = 0;
    __syncthreads();
    for (int r = tid; r < nu; r += nt) {
        double a = 0.0;
        for (int c = 0; c < nu; c++) a = fmax(a, fabs(M[r * nu + c]));
        scale[r] = row_factor(a);
    }
    __syncthreads();
    for (int t = tid; t < nu * nu; t += nt) M[t] *= scale[t / nu];
    __syncthreads();
    for (int k = 0; k < nu; k++) {
        if (tid < 32) {
            // pivot: the largest |M(r, k)| for r >= k (ties to the lower row)
            double best = -1.0;
            int br = k;
            for (int r = k + lane; r < nu; r += 32) {
                const double v = fabs(M[r * nu + k]);
                if (v > best) {
                    best = v;
                    br = r;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int orow = __shfl_xor_sync(0xffffffffu, br, o);
                if (ob > best || (ob == best && orow < br)) {
                    best = ob;
                    br = orow;
                }
            }
            if (lane == 0) {
                piv[k] = br;
                if (!(best > PIVOT_MIN)) bad_s = 1;
            }
        }
        __syncthreads();
        if (bad_s) break;   // uniform: every thread reads it after the barrier
        const int pr = piv[k];
        if (pr != k)
            for (int c = tid; c < nu; c += nt) {
                const double t = M[k * nu + c];
                M[k * nu + c] = M[pr * nu + c];
                M[pr * nu + c] = t;
            }
        __syncthreads();
        if (tid == 0) pinv_s = 1.0 / M[k * nu + k];
        __syncthreads();
        const double pinv = pinv_s;
        for (int c = tid; c < nu; c += nt) M[k * nu + c] = (c == k ? 1.0 : M[k * nu + c]) * pinv;
        for (int r = tid; r < nu; r += nt) fcol[r] = r == k ? 0.0 : M[r * nu + k];
        __syncthreads();
        for (int t = tid; t < nu * nu; t += nt) {
            const int r = t / nu, c = t - r * nu;
            if (r == k) continue;
            M[t] = (c == k ? 0.0 : M[t]) - fcol[r] * M[k * nu + c];
        }
        __syncthreads();
    }
    if (bad_s) {
        if (tid == 0) *ok = 0;
        return;
    }
    // undo the row interchanges: swap columns k <-> piv[k], last interchange first
    for (int k = nu - 1; k >= 0; k--) {
        const int pc = piv[k];
        if (pc != k)
            for (int r = tid; r < nu; r += nt) {
                const double t = M[r * nu + k];
                M[r * nu + k] = M[r * nu + pc];
                M[r * nu + pc] = t;
            }
        __syncthreads();
    }
    for (int t = tid; t < nu * nu; t += nt) {
        const double v = M[t] * scale[t % nu];
        if (inv64) inv64[t] = v;
        if (inv32) inv32[t] = (float)v;
    }
    if (tid == 0) *ok = 1;
}

constexpr int INV_NB = 8;           // panel width
constexpr int EXACT_MAX = 1536;     // unknowns

// The factor of every row of A (column-major); a block takes 32 rows.
__global__ void __launch_bounds__(256) k_inv_scale(int nu, const double* __restrict__ A, double* __restrict__ scale)
{
    __shared__ double m[8][32];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5, r = blockIdx.x * 32 + x;
    double a = 0.0;
    if (r < nu) {
#pragma unroll 8
        for (int c = y; c < nu; c += 8) a = fmax(a, fabs(A[(long long)c * nu + r]));
    }
    m[y][x] = a;
    __syncthreads();
    if (y || r >= nu) return;
    for (int q = 1; q < 8; q++) a = fmax(a, m[q][x]);
    scale[r] = row_factor(a);
}

// M = A with scaled rows, row-major
__global__ void __launch_bounds__(256) k_inv_begin(int nu, const double* __restrict__ A,
                                                   const double* __restrict__ scale, double* __restrict__ M)
{
    __shared__ double t[32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const double f = r0 + x < nu ? scale[r0 + x] : 0.0;
    for (int q = y; q < 32; q += 8)   // column c0 + q, rows r0 + x
        if (c0 + q < nu && r0 + x < nu) t[q][x] = A[(long long)(c0 + q) * nu + r0 + x] * f;
    __syncthreads();
    for (int q = y; q < 32; q += 8)
        if (r0 + q < nu && c0 + x < nu) M[(long long)(r0 + q) * nu + c0 + x] = t[x][q];
}

// Gauss-Jordan on columns k .. k + w of M (w <= INV_NB): T (nu x INV_NB), the
// source row of every row after the interchanges (perm), the pivots (piv).
template <int INV_ROWS>   // rows a thread holds: blocks of 1024 (one row) or 768 (two) threads at most
__global__ void __launch_bounds__(INV_ROWS == 1 ? 1024 : 768) k_inv_panel(int nu, int k, const double* __restrict__ M,
                                                    double* __restrict__ T, int* __restrict__ perm,
                                                    int* __restrict__ piv, int* ok)
{
    __shared__ double best_s[32], prow[INV_NB + 1], srow[INV_NB];
    __shared__ int row_s[32], src_s[2];
    if (!*ok) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int w = min(INV_NB, nu - k);
    double a[INV_ROWS][INV_NB];
    int src[INV_ROWS];
#pragma unroll
    for (int q = 0; q < INV_ROWS; q++) {
        const int r = tid + q * blockDim.x;
        src[q] = r;
#pragma unroll
        for (int c = 0; c < INV_NB; c++) a[q][c] = r < nu && c < w ? M[(long long)r * nu + k + c] : 0.0;
    }
#pragma unroll
    for (int s = 0; s < INV_NB; s++) {
        if (s >= w) break;
        // pivot: the largest |a| of column s in rows >= k + s (ties to the lower row)
        double best = -1.0;
        int br = k + s;
#pragma unroll
        for (int q = 0; q < INV_ROWS; q++) {
            const int r = tid + q * blockDim.x;
            const double v = fabs(a[q][s]);
            if (r >= k + s && r < nu && v > best) {
                best = v;
                br = r;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int orow = __shfl_xor_sync(0xffffffffu, br, o);
            if (ob > best || (ob == best && orow < br)) {
                best = ob;
                br = orow;
            }
        }
        if (lane == 0) {
            best_s[warp] = best;
            row_s[warp] = br;
        }
        __syncthreads();
        best = lane < nw ? best_s[lane] : -1.0;
        br = lane < nw ? row_s[lane] : nu;
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int orow = __shfl_xor_sync(0xffffffffu, br, o);
            if (ob > best || (ob == best && orow < br)) {
                best = ob;
                br = orow;
            }
        }
        if (!(best > PIVOT_MIN)) {   // uniform over the CTA
            if (tid == 0) *ok = 0;
            return;
        }
        const int pr = br;
        // the owners publish the pivot row, scaled, and the row it changes places with
#pragma unroll
        for (int q = 0; q < INV_ROWS; q++) {
            const int r = tid + q * blockDim.x;
            if (r == pr) {
                const double pinv = 1.0 / a[q][s];
#pragma unroll
                for (int c = 0; c < INV_NB; c++) prow[c] = (c == s ? 1.0 : a[q][c]) * pinv;
                src_s[0] = src[q];
                piv[k + s] = pr;
            }
            if (r == k + s) {
#pragma unroll
                for (int c = 0; c < INV_NB; c++) srow[c] = a[q][c];
                src_s[1] = src[q];
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < INV_ROWS; q++) {
            const int r = tid + q * blockDim.x;
            if (r == k + s) {
#pragma unroll
                for (int c = 0; c < INV_NB; c++) a[q][c] = prow[c];
                src[q] = src_s[0];
            } else {
                if (r == pr) {
#pragma unroll
                    for (int c = 0; c < INV_NB; c++) a[q][c] = srow[c];
                    src[q] = src_s[1];
                }
                const double f = a[q][s];
#pragma unroll
                for (int c = 0; c < INV_NB; c++) a[q][c] = (c == s ? 0.0 : a[q][c]) - f * prow[c];
            }
        }
    }
#pragma unroll
    for (int q = 0; q < INV_ROWS; q++) {
        const int r = tid + q * blockDim.x;
        if (r < nu) {
            perm[r] = src[q];
#pragma unroll
            for (int c = 0; c < INV_NB; c++) T[(long long)r * INV_NB + c] = a[q][c];
        }
    }
}

__global__ void __launch_bounds__(256) k_inv_update(int nu, int k, const double* __restrict__ Mo,
                                                    double* __restrict__ Mn, const double* __restrict__ T,
                                                    const int* __restrict__ perm, const int* ok)
{
    __shared__ double t[32][INV_NB + 1], p[INV_NB][32];
    if (!*ok) return;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int r0 = blockIdx.y * 32, c = blockIdx.x * 32 + x;
    const int w = min(INV_NB, nu - k);
    if (r0 + (int)(threadIdx.x >> 3) < nu)
        t[threadIdx.x >> 3][threadIdx.x & 7] = T[(long long)(r0 + (threadIdx.x >> 3)) * INV_NB + (threadIdx.x & 7)];
    p[y][x] = y < w && c < nu ? Mo[(long long)perm[k + y] * nu + c] : 0.0;
    __syncthreads();
    if (c >= nu) return;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int rl = y + 8 * q, r = r0 + rl;
        if (r >= nu) continue;
        double v;
        if (c >= k && c < k + w) {
            v = t[rl][c - k];
        } else {
            v = r >= k && r < k + w ? 0.0 : Mo[(long long)perm[r] * nu + c];
#pragma unroll
            for (int s = 0; s < INV_NB; s++) v += (s < w ? t[rl][s] : 0.0) * p[s][x];
        }
        Mn[(long long)r * nu + c] = v;
    }
}

// Undo the row interchanges (swap columns k <-> piv[k], last first) on the way
// into the row-major inverses, and the rows' factors into their columns.
__global__ void __launch_bounds__(256) k_inv_end(int nu, const double* __restrict__ M, const int* __restrict__ piv,
                                                 const double* __restrict__ scale, double* __restrict__ inv64,
                                                 float* __restrict__ inv32, const int* ok)
{
    __shared__ int col[EXACT_MAX];
    __shared__ int pv[EXACT_MAX];
    if (!*ok) return;
    for (int j = threadIdx.x; j < nu; j += blockDim.x) {
        col[j] = j;
        pv[j] = piv[j];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int j = nu - 1; j >= 0; j--) {
            const int t = col[j];
            col[j] = col[pv[j]];
            col[pv[j]] = t;
        }
    __syncthreads();
    for (int r = blockIdx.x; r < nu; r += gridDim.x)
        for (int j = threadIdx.x; j < nu; j += blockDim.x) {
            const double v = M[(long long)r * nu + col[j]] * scale[j];
            if (inv64) inv64[(long long)r * nu + j] = v;
            if (inv32) inv32[(long long)r * nu + j] = (float)v;
        }
}

// Exact coarsest solve unless AGB_BOTTOM_EXACT=0 (read when an operator is created).
bool use_exact_bottom()
{
    const char* s = getenv("AGB_BOTTOM_EXACT");
    return !(s && s[0] == '0');
}

bool bottom_exact_fits(const LevelDesc& L) { return !L.singular() && 3 * L.count() <= EXACT_MAX; }

// Work of the panel elimination: two copies of the matrix, T, scale, perm, piv.
size_t bottom_invert_work_bytes(const LevelDesc& L)
{
    const size_t nu = 3 * (size_t)L.count();
    return bottom_dense_fits(L) ? 0 : (2 * nu * nu + nu * INV_NB + nu) * sizeof(double) + 2 * nu * sizeof(int);
}

// *ok = 1 and the inverses of A, or *ok = 0 (a kernel of the chain that finds
// *ok cleared leaves at once).
void launch_bottom_invert(cudaStream_t st, const LevelDesc& L, const double* A, double* inv64, float* inv32,
                          double* work, int* ok)
{
    const int nu = 3 * (int)L.count();
    if (bottom_dense_fits(L)) {
        k_bottom_invert<<<1, 1024, (size_t)nu * nu * sizeof(double), st>>>(L, A, inv64, inv32, ok);
        count_launch();
        return;
    }
    const size_t n2 = (size_t)nu * nu;
    double *M0 = work, *M1 = work + n2, *T = work + 2 * n2;
    double* scale = T + (size_t)nu * INV_NB;
    int *perm = (int*)(scale + nu), *piv = perm + nu;
    const dim3 tiles((nu + 31) / 32, (nu + 31) / 32);
    const int rows = nu <= 1024 ? 1 : 2, threads = ((nu + rows - 1) / rows + 31) / 32 * 32;
    cudaMemsetAsync(ok, 1, sizeof(int), st);   // any value but 0
    k_inv_scale<<<(nu + 31) / 32, 256, 0, st>>>(nu, A, scale);
    k_inv_begin<<<tiles, 256, 0, st>>>(nu, A, scale, M0);
    count_launch();
    count_launch();
    for (int k = 0; k < nu; k += INV_NB) {
        if (rows == 1) k_inv_panel<1><<<1, threads, 0, st>>>(nu, k, M0, T, perm, piv, ok);
        else k_inv_panel<2><<<1, threads, 0, st>>>(nu, k, M0, T, perm, piv, ok);
        k_inv_update<<<tiles, 256, 0, st>>>(nu, k, M0, M1, T, perm, ok);
        count_launch();
        count_launch();
        double* t = M0;
        M0 = M1;
        M1 = t;
    }
    k_inv_end<<<64, 256, 0, st>>>(nu, M0, piv, scale, inv64, inv32, ok);
    count_launch();
}

// Small bottom levels use the dense path unless AGB_BOTTOM_DENSE=0.
bool use_dense_bottom()
{
    static bool v = [] {
        const char* s = getenv("AGB_BOTTOM_DENSE");
        return !(s && s[0] == '0');
    }();
    return v;
}

size_t bottom_dense_bytes(const LevelDesc& L)
{
    const size_t nu = 3 * (size_t)L.count();
    return nu * nu * sizeof(double);
}

void launch_bottom_assemble(cudaStream_t st, int sym, const LevelDesc& L, const BCTable& bc, bool uniform,
                            const double* ddw64, double* A)
{
    const Geo<double> g = make_geo<double>(L);
    const int cnt = (int)L.count(), work = cnt * 3 * cnt;
    const int blocks = (work + 255) / 256;
    if (sym == SYM_ISO) k_bottom_assemble<SYM_ISO><<<blocks, 256, 0, st>>>(L, bc, g, uniform ? 1 : 0, ddw64, A);
    else k_bottom_assemble<SYM_MM><<<blocks, 256, 0, st>>>(L, bc, g, uniform ? 1 : 0, ddw64, A);
    count_launch();
}

template <typename T>
void launch_bottom_dense(cudaStream_t st, const LevelDesc& L, const double* A, const double* diag64, T* cor,
                         const T* res, int maxiter, double tol_rel, double tol_abs, int* ret_slot, int nub, int nuf,
                         double omega, const T* inv, const int* inv_ok)
{
    const size_t nu = 3 * (size_t)L.count();
    const size_t smem = (nu * nu + nu) * sizeof(T);
    // the exact product takes a row a warp; the BiCGStab solve the first CTA
    const unsigned grid = inv ? (unsigned)((nu + DENSE_MAX / 32 - 1) / (DENSE_MAX / 32)) : 1u;
    pdl_launch(k_bottom_dense<T, T>, dim3(grid), dim3(DENSE_MAX), smem, st, L, A, diag64, cor, res, maxiter, tol_rel,
               tol_abs, nub, nuf, omega, ret_slot, inv, inv_ok);
    count_launch();
}

void init_bottom_attributes()
{
    const int smem = (DENSE_MAX * DENSE_MAX + DENSE_MAX) * (int)sizeof(double);
    cudaFuncSetAttribute(k_bottom_dense<double, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_bottom_dense<float, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_bottom_invert, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         DENSE_MAX * DENSE_MAX * (int)sizeof(double));
}

template void launch_bottom_dense<double>(cudaStream_t, const LevelDesc&, const double*, const double*, double*,
                                          const double*, int, double, double, int*, int, int, double, const double*,
                                          const int*);
template void launch_bottom_dense<float>(cudaStream_t, const LevelDesc&, const double*, const double*, float*,
                                         const float*, int, double, double, int*, int, int, double, const float*,
                                         const int*);

template <typename T>
void launch_bottom(cudaStream_t st, int sym, const LevelDesc& L, const BCTable& bc, bool uniform, const double* ddw64,
                   const double* diag64, T* cor, const T* res, double* work, int maxiter, double tol_rel,
                   double tol_abs, int* ret_slot, int nub, int nuf, double omega, const double* inv,
                   const int* inv_ok)
{
    const Geo<double> g = make_geo<double>(L);
    const size_t nu = 3 * (size_t)L.count();
    const unsigned grid = inv ? (unsigned)((nu + BOT_THREADS / 32 - 1) / (BOT_THREADS / 32)) : 1u;
    const size_t smem = inv ? nu * sizeof(double) : 0;
    if (sym == SYM_ISO)
        k_bottom<T, SYM_ISO><<<grid, BOT_THREADS, smem, st>>>(L, bc, g, uniform ? 1 : 0, ddw64, diag64, cor, res, work,
                                                              maxiter, tol_rel, tol_abs, nub, nuf, omega, ret_slot,
                                                              inv, inv_ok);
    else
        k_bottom<T, SYM_MM><<<grid, BOT_THREADS, smem, st>>>(L, bc, g, uniform ? 1 : 0, ddw64, diag64, cor, res, work,
                                                             maxiter, tol_rel, tol_abs, nub, nuf, omega, ret_slot,
                                                             inv, inv_ok);
    count_launch();
}

template void launch_bottom<double>(cudaStream_t, int, const LevelDesc&, const BCTable&, bool, const double*,
                                    const double*, double*, const double*, double*, int, double, double, int*, int,
                                    int, double, const double*, const int*);
template void launch_bottom<float>(cudaStream_t, int, const LevelDesc&, const BCTable&, bool, const double*,
                                   const double*, float*, const float*, double*, int, double, double, int*, int, int,
                                   double, const double*, const int*);

}  // namespace agb

// ---------------------------------------------------------------------------
// Allocation-free coarsest-level solve (agb_bottom_solve_noalloc in agb.h)
//
// Some callers may not allocate device memory at the moment they need a
// bottom solve: a host framework that owns every device byte through its own
// arena and forbids cudaMalloc inside its solver hooks, or a time-stepping
// code that must not stall on cudaMalloc's implicit synchronisation in the
// middle of a step.  For them the BiCGStab
// work vectors live in a file-scope device array instead of a buffer of an
// operator handle.  The array is sized for boxes of at most
// AGB_NOALLOC_MAX_NODES nodes (a 16^3-cell box); every GPU that loads this
// library holds it (943 KB) until the process exits.
// ---------------------------------------------------------------------------
#include <mutex>

#include "agb.h"

namespace {

constexpr long long kScratchDoubles = 8LL * 3LL * AGB_NOALLOC_MAX_NODES;
static __device__ __align__(256) double g_bottom_scratch[kScratchDoubles];

constexpr int kMaxDevices = 256;
std::mutex g_scratch_mutex;
double* g_scratch_addr[kMaxDevices] = {nullptr};

// Device address of g_bottom_scratch on the current device.  The name
// g_bottom_scratch is only a host-side stand-in: a kernel must be given the
// address that cudaGetSymbolAddress returns for the device it runs on.  The
// address is cached per device for the life of the process, which assumes
// one CUDA context per device: after cudaDeviceReset the cached address is
// stale, so a caller that resets a device must not call this entry point
// again in that process.
agb_status scratch_for_current_device(double** out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        agb::set_error("no usable CUDA device for the allocation-free bottom solve");
        return AGB_CUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) {
        agb::set_error("device index out of range");
        return AGB_CUDA;
    }
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_bottom_scratch);
        if (e != cudaSuccess || !p) {
            agb::set_error("cudaGetSymbolAddress of the bottom-solve scratch failed");
            return AGB_CUDA;
        }
        g_scratch_addr[dev] = (double*)p;
    }
    *out = g_scratch_addr[dev];
    return AGB_OK;
}

}  // namespace

extern "C" agb_status agb_bottom_solve_noalloc(const int n_cells[3], const double dx[3], int sym, int uniform,
                                               const agb_bc* bc, const double* ddw, const double* diag,
                                               const double* res, double* cor, int* ret, int max_iter,
                                               double tol_rel, double tol_abs, int bottom_smooth, int final_smooth,
                                               double omega, void* stream)
{
    using namespace agb;
    if (!n_cells || !dx || !bc || !ddw || !diag || !res || !cor || !ret) {
        set_error("null argument");
        return AGB_BADARG;
    }
    if (sym != AGB_ISO && sym != AGB_MAJORMINOR) {
        set_error("sym must be AGB_ISO or AGB_MAJORMINOR");
        return AGB_BADARG;
    }
    long long nodes = 1;
    for (int d = 0; d < 3; d++) {
        if (n_cells[d] < 1 || !(dx[d] > 0)) {
            set_error("n_cells must be >= 1 and dx > 0");
            return AGB_BADARG;
        }
        nodes *= (long long)(n_cells[d] + 1);
    }
    if (nodes > AGB_NOALLOC_MAX_NODES) {
        set_error("box too large for the allocation-free bottom solve: more than AGB_NOALLOC_MAX_NODES nodes");
        return AGB_BADARG;
    }
    if (cor == res) {
        set_error("res and cor must be distinct, non-overlapping arrays");
        return AGB_BADARG;
    }
    if (max_iter < 0 || bottom_smooth < 0 || final_smooth < 0 || !(omega > 0 && omega < 2)) {
        set_error("bad iteration count, smoothing count or omega");
        return AGB_BADARG;
    }
    BCTable t;
    for (int f = 0; f < F_NFACES; f++)
        for (int c = 0; c < 3; c++) {
            if (bc->type[f][c] < AGB_BC_DISP || bc->type[f][c] > AGB_BC_NONE) {
                set_error("bad BC type");
                return AGB_BADARG;
            }
            // The box has no periodic direction: a periodic row would be an
            // empty row (zero diagonal) of the scaled system.
            if (bc->type[f][c] == AGB_BC_PERIODIC) {
                set_error("the allocation-free bottom solve takes no periodic BC type");
                return AGB_BADARG;
            }
            t.type[f][c] = (int8_t)bc->type[f][c];
            t.val[f][c] = bc->val[f][c];
        }
    // The caller's arrays are the unpadded reference layout: row pitch n0+1,
    // component stride = node count.
    LevelDesc L;
    for (int d = 0; d < 3; d++) {
        L.n[d] = n_cells[d];
        L.nn[d] = n_cells[d] + 1;
        L.per[d] = 0;
        L.dx[d] = dx[d];
    }
    L.P = L.nn[0];
    L.S = nodes;
    double* work = nullptr;
    const agb_status s = scratch_for_current_device(&work);
    if (s != AGB_OK) return s;
    // An error pending from earlier, unrelated work is not this call's: clear
    // it, so that the check after the launch sees only the launch's own
    // error (a broken context makes the launch itself fail).
    if (cudaPeekAtLastError() != cudaSuccess) cudaGetLastError();
    // Every scratch element the kernel reads is written earlier in the same
    // launch, so the contents left by a previous call need no clearing.
    launch_bottom<double>((cudaStream_t)stream, sym, L, t, uniform != 0, ddw, diag, cor, res, work, max_iter, tol_rel,
                          tol_abs, ret, bottom_smooth, final_smooth, omega);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(cudaGetErrorString(e));
        return AGB_CUDA;
    }
    return AGB_OK;
}
