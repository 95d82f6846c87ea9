// kernels_stencil.cu -- Fapply / residual / damped-Jacobi / diagonal kernels.
//
//   MODE_APPLY   out = A x                          (Elastic::Fapply, Elastic.cpp:141-292)
//   MODE_RESID   out = b - A x, max|out| -> slot    (solutionResidual, Operator.cpp:636-657)
//   MODE_JACOBI  out = x + omega * (b - A x) / D    (one sweep of Operator<Node>::Fsmooth,
//                                                    Operator.cpp:107-147, with the reference's
//                                                    (1-w)x + w(b-(Ax-Dx))/D regrouped;
//                                                    `diag` carries 1/D)
//
// Kernels, all on the per-node arithmetic of stencil.cuh:
//   k_rows, k_column   rows from the node's own moduli (and their divergence):
//                      FP64 on every level, FP32 on those the TMA kernel
//                      (kernels_tma.cu) does not take
//   k_stencil_pipe     FP32 interiors of large levels by cp.async (behind a switch)
//   k_stencil_shell    the boundary rows beside the TMA and cp.async kernels
//   k_stencil_node     one thread per node from the moduli of the neighbours:
//                      levels whose divergence field found no memory
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>

#include "agb_internal.h"
#include "stencil.cuh"

namespace agb {

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

template <typename T> struct MaxBits;
template <> struct MaxBits<double> {
    typedef unsigned long long U;
    static __device__ __forceinline__ U bits(double v) { return (U)__double_as_longlong(v); }
    static __device__ __forceinline__ void atomic(void* slot, double v)
    {
        atomicMax((unsigned long long*)slot, bits(v));
    }
};
template <> struct MaxBits<float> {
    typedef unsigned int U;
    static __device__ __forceinline__ U bits(float v) { return (U)__float_as_uint(v); }
    static __device__ __forceinline__ void atomic(void* slot, float v) { atomicMax((unsigned int*)slot, bits(v)); }
};

// max of |v| over the block (v >= 0 or NaN); one atomic per block.  NaN has the
// largest bit pattern of the non-negative encodings, so it propagates.
template <typename T>
__device__ __forceinline__ void block_max_to_slot(T v, void* slot)
{
    __shared__ T red[32];
    const int lane = (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)) & 31;
    const int warp = (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)) >> 5;
    const int nwarp = (blockDim.x * blockDim.y * blockDim.z + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T w = __shfl_xor_sync(0xffffffffu, v, o);
        v = (w > v || w != w) ? w : v;
    }
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = lane < nwarp ? red[lane] : (T)0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            T w = __shfl_xor_sync(0xffffffffu, v, o);
            v = (w > v || w != w) ? w : v;
        }
        if (lane == 0) MaxBits<T>::atomic(slot, v);
    }
}

template <typename T> struct GlobalAcc {
    const T* __restrict__ x;
    const T* __restrict__ c;
    long long S;
    Nbr nb;
    __device__ __forceinline__ long long off(int di, int dj, int dk) const
    {
        return nb.base + nb.o[0][di + 1] + nb.o[1][dj + 1] + nb.o[2][dk + 1];
    }
    __device__ __forceinline__ T u(int p, int di, int dj, int dk) const { return __ldg(x + p * S + off(di, dj, dk)); }
    __device__ __forceinline__ T C(int m, int di, int dj, int dk) const { return __ldg(c + m * S + off(di, dj, dk)); }
};

template <typename T, int MODE>
__device__ __forceinline__ void epilogue(const T f[3], const T* __restrict__ x, const T* __restrict__ b,
                                         const T* __restrict__ dinv, T* __restrict__ out, long long S, long long p,
                                         T omega, T& nrm)
{
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const long long q = c * S + p;
        if (MODE == MODE_APPLY) {
            out[q] = f[c];
        } else if (MODE == MODE_RESID) {
            const T r = b[q] - f[c];
            out[q] = r;
            const T a = fabs(r);
            nrm = (a > nrm || a != a) ? a : nrm;
        } else {
            out[q] = x[q] + omega * ((b[q] - f[c]) * dinv[q]);
        }
    }
}

// ---------------------------------------------------------------------------
// one thread per node: general moduli without their divergence
// ---------------------------------------------------------------------------
template <typename T, int MODE>
__global__ void __launch_bounds__(256) k_stencil_node(LevelDesc L, BCTable bc, Geo<T> g, const T* __restrict__ ddw,
                                                      const T* __restrict__ x, const T* __restrict__ b,
                                                      const T* __restrict__ dinv, T* __restrict__ out, T omega,
                                                      void* norm_slot)
{
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    T nrm = 0;
    if (i < L.nn[0] && j < L.nn[1] && k < L.nn[2]) {
        const int pos[3] = {i, j, k};
        int mn[3], mx[3];
        bool bnd = false;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            mn[d] = !L.per[d] && pos[d] == 0;
            mx[d] = !L.per[d] && pos[d] == L.n[d];
            bnd = bnd || mn[d] || mx[d];
        }
        GlobalAcc<T> acc{x, ddw, L.S, make_nbr(L, i, j, k)};
        T f[3];
        if (bnd) boundary_row<T, SYM_MM>(acc, g, bc, mn, mx, f);
        else interior_row<T, SYM_MM>(acc, g, false, f);
        epilogue<T, MODE>(f, x, b, dinv, out, L.S, acc.nb.base, omega, nrm);
    }
    if (MODE == MODE_RESID && norm_slot) block_max_to_slot<T>(nrm, norm_slot);
}

// ---------------------------------------------------------------------------
// boundary shell of a box with no periodic direction: one thread per boundary
// node, enumerated plane k=0, plane k=n2, then the rings of the planes between
// ---------------------------------------------------------------------------
// (with xf = 0 the x-face nodes between the y rows are left out: the TMA
// interior kernel computes them)
__host__ __device__ inline long long shell_count(const LevelDesc& L, int xf)
{
    const long long a = (long long)L.nn[0] * L.nn[1];
    return 2 * a + (long long)(L.nn[2] - 2) * (2LL * L.nn[0] + (xf ? 2LL * (L.nn[1] - 2) : 0LL));
}

__device__ __forceinline__ void shell_node(const LevelDesc& L, long long e, int xf, int& i, int& j, int& k)
{
    const long long a = (long long)L.nn[0] * L.nn[1];
    if (e < 2 * a) {
        k = e < a ? 0 : L.nn[2] - 1;
        const long long r = e < a ? e : e - a;
        j = (int)(r / L.nn[0]);
        i = (int)(r % L.nn[0]);
        return;
    }
    const long long e2 = e - 2 * a, pm = 2LL * L.nn[0] + (xf ? 2LL * (L.nn[1] - 2) : 0LL);
    k = 1 + (int)(e2 / pm);
    const int r = (int)(e2 % pm);
    if (r < 2 * L.nn[0]) {
        j = r < L.nn[0] ? 0 : L.nn[1] - 1;
        i = r < L.nn[0] ? r : r - L.nn[0];
    } else {
        const int r2 = r - 2 * L.nn[0];
        j = 1 + r2 / 2;
        i = (r2 & 1) ? L.nn[0] - 1 : 0;
    }
}

template <typename T, int SYM, int MODE>
__global__ void __launch_bounds__(256) k_stencil_shell(LevelDesc L, BCTable bc, Geo<T> g, const T* __restrict__ ddw,
                                                       const T* __restrict__ x, const T* __restrict__ b,
                                                       const T* __restrict__ dinv, T* __restrict__ out, T omega,
                                                       void* norm_slot, int xf)
{
    pdl_entry();
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    T nrm = 0;
    if (e < shell_count(L, xf)) {
        int i, j, k;
        shell_node(L, e, xf, i, j, k);
        const int pos[3] = {i, j, k};
        int mn[3], mx[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            mn[d] = pos[d] == 0;
            mx[d] = pos[d] == L.n[d];
        }
        GlobalAcc<T> acc{x, ddw, L.S, make_nbr(L, i, j, k)};
        T f[3];
        boundary_row<T, SYM>(acc, g, bc, mn, mx, f);
        epilogue<T, MODE>(f, x, b, dinv, out, L.S, acc.nb.base, omega, nrm);
    }
    if (MODE == MODE_RESID && norm_slot) block_max_to_slot<T>(nrm, norm_slot);
}

// ---------------------------------------------------------------------------
// Rows from the node's own moduli.
//
// General moduli enter an interior row through the node's 21 coefficients and
// the 18 of their divergence (mm_row_div), a field made once per
// prepareForSolve by k_div_moduli; isotropic moduli through the node and its
// six neighbours.  So there is no halo of moduli to stage, every coefficient
// is read once, coalesced, by the thread that uses it, and the displacement's
// neighbours come through L1.
//
// What bounds it: in FP64 the FP64 pipe (two lanes per clock and SM on GB300; a
// Jacobi sweep is 146 operations a node in k_rows and 144 in k_column, counted by
// ncu, against 262 with the moduli of the neighbours, and the extra 144 bytes a node of the divergence cost a tenth of that time);
// in FP32, on the levels that fit in L2, latency.  A Jacobi sweep with general
// moduli went from 10.10 to 4.37 ms at 257^3 nodes in FP64 (0.89 of what the
// pipe issues at 144 operations a node), 338 to 88 us at 65^3, 34.8 to 14.4 us at
// 33^3, 27.7 to 10.3 us at 9^3; isotropic 671 to 433 us at 129^3; FP32 general
// moduli 18.4 to 10.3 us at 49^3.
//
//   k_rows    one thread per node, any level.  On a box with no periodic
//             direction the threads are numbered interior nodes first, then
//             the boundary shell, so that no warp runs both kinds of row; 64
//             threads a block, so that the 9^3- to 33^3-node levels spread over all SMs.
//   k_column  FP64 on large levels: a thread marches up a column, carrying the
//             x and y differences of three planes in registers, from which the
//             mixed xz and yz differences cost one subtraction each and a node
//             27 instead of 57 displacement loads; the boundary shell is done by
//             the last blocks of the same launch.
// ---------------------------------------------------------------------------
constexpr int ROW_THREADS = 64;

template <typename T, int SYM, bool CUBE, class A>
__device__ __forceinline__ void row_from_diffs(const A& acc, const Geo<T>& g, bool uniform, const RowD<T>& r,
                                               const T* __restrict__ div, T f[3])
{
    if constexpr (SYM == SYM_ISO) {
        iso_row<T, CUBE>(acc, g, uniform, r, f);
    } else {
        mm_row_div<T, CUBE>([&](int m) { return acc.C(m, 0, 0, 0); },
                            [&](int m) { return __ldg(div + m * acc.S + acc.nb.base); }, uniform, r, f);
    }
    if (CUBE) {
        const T h = row_scale<T, CUBE>(g);
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] *= h;
    }
}

// nint: interior nodes of a box with no periodic direction, rounded up to a
// warp (the shell's numbers start there); 0: nodes numbered by their place.
template <typename T, int SYM, int MODE, bool CUBE>
__global__ void __launch_bounds__(ROW_THREADS) k_rows(LevelDesc L, BCTable bc, Geo<T> g, int uniform, int nint,
                                                      const T* __restrict__ ddw, const T* __restrict__ div,
                                                      const T* __restrict__ x, const T* __restrict__ b,
                                                      const T* __restrict__ dinv, T* __restrict__ out, T omega,
                                                      void* norm_slot)
{
    pdl_entry();
    const int e = blockIdx.x * ROW_THREADS + threadIdx.x;
    int i = 0, j = 0, k = 0;
    bool ok;
    if (nint > 0) {
        const int I = L.n[0] - 1, J = L.n[1] - 1;
        if (e < nint) {
            i = 1 + e % I;
            j = 1 + (e / I) % J;
            k = 1 + e / (I * J);
            ok = k < L.n[2];
        } else {
            ok = e - nint < shell_count(L, 1);
            if (ok) shell_node(L, e - nint, 1, i, j, k);
        }
    } else {
        i = e % L.nn[0];
        j = (e / L.nn[0]) % L.nn[1];
        k = e / (L.nn[0] * L.nn[1]);
        ok = k < L.nn[2];
    }
    T nrm = 0;
    if (ok) {
        const int pos[3] = {i, j, k};
        int mn[3], mx[3];
        bool bnd = false;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            mn[d] = !L.per[d] && pos[d] == 0;
            mx[d] = !L.per[d] && pos[d] == L.n[d];
            bnd = bnd || mn[d] || mx[d];
        }
        GlobalAcc<T> acc{x, ddw, L.S, make_nbr(L, i, j, k)};
        T f[3];
        if (bnd) {
            boundary_row<T, SYM>(acc, g, bc, mn, mx, f);
        } else {
            RowD<T> r;
            row_diffs<T, CUBE>(acc, g, r);
            row_from_diffs<T, SYM, CUBE>(acc, g, uniform != 0, r, div, f);
        }
        epilogue<T, MODE>(f, x, b, dinv, out, L.S, acc.nb.base, omega, nrm);
    }
    if (MODE == MODE_RESID && norm_slot) block_max_to_slot<T>(nrm, norm_slot);
}

constexpr int COL_X = 32, COL_Y = 2;   // threads of a block (64)
constexpr int COL_RESIDENT = 8;         // blocks an SM holds (128 registers a thread)

template <typename T, int SYM, int MODE, bool CUBE>
__global__ void __launch_bounds__(COL_X* COL_Y, COL_RESIDENT) k_column(LevelDesc L, BCTable bc, Geo<T> g, int uniform, int kz,
                                                         int chunks, const T* __restrict__ ddw,
                                                         const T* __restrict__ div, const T* __restrict__ x,
                                                         const T* __restrict__ b, const T* __restrict__ dinv,
                                                         T* __restrict__ out, T omega, void* norm_slot)
{
    pdl_entry();
    const int tx = threadIdx.x, ty = threadIdx.y;
    T nrm = 0;
    if ((int)blockIdx.z >= chunks) {
        // boundary shell
        const long long e = (((long long)(blockIdx.z - chunks) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) *
                                (COL_X * COL_Y) + ty * COL_X + tx;
        if (e < shell_count(L, 1)) {
            int i, j, k;
            shell_node(L, e, 1, i, j, k);
            const int mn[3] = {i == 0, j == 0, k == 0}, mx[3] = {i == L.n[0], j == L.n[1], k == L.n[2]};
            GlobalAcc<T> acc{x, ddw, L.S, make_nbr(L, i, j, k)};
            T f[3];
            boundary_row<T, SYM>(acc, g, bc, mn, mx, f);
            epilogue<T, MODE>(f, x, b, dinv, out, L.S, acc.nb.base, omega, nrm);
        }
    } else {
        const int i = 1 + blockIdx.x * COL_X + tx, j = 1 + blockIdx.y * COL_Y + ty;
        const int k0 = 1 + blockIdx.z * kz, k1 = min(k0 + kz, L.n[2]);
        if (i < L.n[0] && j < L.n[1]) {
            const long long S = L.S, P = L.P, plane = P * L.nn[1];
            GlobalAcc<T> acc{x, ddw, S, make_nbr(L, i, j, k0)};
            // differences of a plane at the column, unscaled: x and y first
            // and second ones, and the displacement itself
            T gx[3][3], gy[3][3], uc[3][3], dx2[3], dy2[3];   // [plane k-1, k, k+1][component]
            auto take = [&](int s, long long q, T* d2x, T* d2y) {
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const T* a = x + p * S + q;
                    const T c = __ldg(a), xp = __ldg(a + 1), xm = __ldg(a - 1), yp = __ldg(a + P), ym = __ldg(a - P);
                    uc[s][p] = c;
                    gx[s][p] = xp - xm;
                    gy[s][p] = yp - ym;
                    if (d2x) {
                        d2x[p] = (xp - (T)2 * c) + xm;
                        d2y[p] = (yp - (T)2 * c) + ym;
                    }
                }
            };
            long long q = acc.nb.base;
            take(0, q - plane, nullptr, nullptr);
            take(1, q, dx2, dy2);
#pragma unroll 1
            for (int k = k0; k < k1; k++, q += plane) {
                T nx2[3], ny2[3];
                take(2, q + plane, nx2, ny2);
                acc.nb.base = q;
                RowD<T> r;
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const T* a = x + p * S + q;
                    r.d2[0][p] = dx2[p];
                    r.d2[1][p] = dy2[p];
                    r.d2[2][p] = (uc[2][p] - (T)2 * uc[1][p]) + uc[0][p];
                    r.mx[0][p] = (__ldg(a + 1 + P) - __ldg(a - 1 + P)) - (__ldg(a + 1 - P) - __ldg(a - 1 - P));
                    r.mx[1][p] = gx[2][p] - gx[0][p];
                    r.mx[2][p] = gy[2][p] - gy[0][p];
                    r.G[0][p] = gx[1][p];
                    r.G[1][p] = gy[1][p];
                    r.G[2][p] = uc[2][p] - uc[0][p];
                    scale_diffs<T, CUBE>(g, r, p);
                }
                T f[3];
                row_from_diffs<T, SYM, CUBE>(acc, g, uniform != 0, r, div, f);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const long long o = c * S + q;
                    if (MODE == MODE_APPLY) {
                        out[o] = f[c];
                    } else if (MODE == MODE_RESID) {
                        const T rr = __ldg(b + o) - f[c];
                        out[o] = rr;
                        const T a = fabs(rr);
                        nrm = (a > nrm || a != a) ? a : nrm;
                    } else {
                        out[o] = uc[1][c] + omega * ((__ldg(b + o) - f[c]) * __ldg(dinv + o));
                    }
                }
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    gx[0][p] = gx[1][p];
                    gx[1][p] = gx[2][p];
                    gy[0][p] = gy[1][p];
                    gy[1][p] = gy[2][p];
                    uc[0][p] = uc[1][p];
                    uc[1][p] = uc[2][p];
                    dx2[p] = nx2[p];
                    dy2[p] = ny2[p];
                }
            }
        }
    }
    if (MODE == MODE_RESID && norm_slot) block_max_to_slot<T>(nrm, norm_slot);
}

// The divergence of general moduli at the interior nodes, D(i, m) = sum_j w_j
// (C(+e_j) - C(-e_j))_{ij,m}, w_j = 1 on cubic cells (the row is scaled as a
// whole) and 0.5/dx_j otherwise; 18 planes, zero on the boundary.
template <typename T, bool CUBE>
__global__ void __launch_bounds__(128) k_div_moduli(LevelDesc L, Geo<T> g, const T* __restrict__ ddw,
                                                    T* __restrict__ div)
{
    const int e = blockIdx.x * 128 + threadIdx.x;
    const int i = e % L.nn[0], j = (e / L.nn[0]) % L.nn[1], k = e / (L.nn[0] * L.nn[1]);
    if (k >= L.nn[2]) return;
    const int pos[3] = {i, j, k};
#pragma unroll
    for (int d = 0; d < 3; d++)
        if (!L.per[d] && (pos[d] == 0 || pos[d] == L.n[d])) return;
    const Nbr nb = make_nbr(L, i, j, k);
    constexpr int slot[6][6] = {{0, 1, 2, 3, 4, 5},     {1, 6, 7, 8, 9, 10},    {2, 7, 11, 12, 13, 14},
                                {3, 8, 12, 15, 16, 17}, {4, 9, 13, 16, 18, 19}, {5, 10, 14, 17, 19, 20}};
    constexpr int pair[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    T D[3][6];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        T dc[21];   // the 15 of them that row d uses
#pragma unroll
        for (int m = 0; m < 21; m++) {
            const T* c = ddw + m * L.S + nb.base;
            dc[m] = __ldg(c + nb.o[d][2]) - __ldg(c + nb.o[d][0]);
            if (!CUBE) dc[m] *= g.h1[d];
        }
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int m = 0; m < 6; m++) D[r][m] = d ? D[r][m] + dc[slot[pair[r][d]][m]] : dc[slot[pair[r][d]][m]];
    }
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int m = 0; m < 6; m++) div[(r * 6 + m) * L.S + nb.base] = D[r][m];
}

// ---------------------------------------------------------------------------
// cp.async-pipelined marching kernel (FP32 cycles on the finest levels)
//
// A 32 x 8 column tile marches in k; the planes of the tile (+1 halo) are
// copied global -> shared with 16-byte cp.async (L1 bypassed) two planes ahead
// of the compute: u in a ring of 4 planes, moduli in a ring of 3, so the loads
// of plane k+3 overlap the arithmetic of plane k.  Every halo row is 36
// elements wide and starts at i = 32t, 16-byte aligned (the level's row pitch
// leaves room for it).  Own-column values at k-1 (moduli) are kept in
// registers.
// ---------------------------------------------------------------------------
constexpr int MT_X = 32, MT_Y = 8;  // tile
constexpr int MH_Y = MT_Y + 2;      // with halo
constexpr int PT_Z = 32;            // k-chunk of one CTA
constexpr int PW = 36;              // halo row width loaded (9 x 16 bytes)
constexpr int PU = 4, PC = 3;       // ring depths (u, moduli)

template <typename T, int SYM> struct PipeSmem {
    static constexpr int NC = NCoef<SYM>::value;
    T u[PU][3][MH_Y][PW];
    T c[PC][NC][MH_Y][PW];
};

template <typename T, int SYM> struct PipeAcc {
    const PipeSmem<T, SYM>* s;
    int tx, ty;            // halo-tile position of the node (1-based)
    int um, u0, up;        // u ring slots of planes k-1, k, k+1
    int c0, cp;            // moduli ring slots of planes k, k+1
    T cm[NCoef<SYM>::value];
    __device__ __forceinline__ T u(int p, int di, int dj, int dk) const
    {
        const int r = dk < 0 ? um : (dk > 0 ? up : u0);
        return s->u[r][p][ty + dj][tx + di];
    }
    __device__ __forceinline__ T C(int m, int di, int dj, int dk) const
    {
        if (dk < 0) return cm[m];
        if (dk > 0) return s->c[cp][m][ty][tx];
        return s->c[c0][m][ty + dj][tx + di];
    }
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    unsigned long long ga;
    asm volatile("cvta.to.global.u64 %0, %1;" : "=l"(ga) : "l"(gmem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(ga) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Queue the copy of plane kk of `ncomp` planes of src into dst[ncomp][MH_Y][PW].
template <typename T>
__device__ __forceinline__ void issue_plane(T* dst, const T* __restrict__ src, int ncomp, const LevelDesc& L, int i0,
                                            int j0, int kk, int tid)
{
    constexpr int VEC = 16 / sizeof(T);        // elements per 16-byte chunk
    constexpr int QPR = PW / VEC;              // chunks per halo row
    const int per_comp = MH_Y * QPR;
    const long long plane = (long long)L.P * L.nn[1] * kk;
    for (int e = tid; e < ncomp * per_comp; e += MT_X * MT_Y) {
        const int c = e / per_comp, rem = e - c * per_comp;
        const int row = rem / QPR, q = rem - row * QPR;
        const int gj = j0 - 1 + row;
        if (gj > L.n[1]) continue;   // rows past the hi boundary are never read
        const T* g = src + c * L.S + plane + (long long)L.P * gj + (i0 - 1) + q * VEC;
        cp_async16(dst + ((c * MH_Y + row) * PW + q * VEC), g);
    }
}

template <typename T, int SYM, int MODE>
__global__ void __launch_bounds__(MT_X* MT_Y) k_stencil_pipe(LevelDesc L, Geo<T> g, int uniform,
                                                                const T* __restrict__ ddw, const T* __restrict__ x,
                                                                const T* __restrict__ b, const T* __restrict__ dinv,
                                                                T* __restrict__ out, T omega, void* norm_slot)
{
    pdl_entry();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PipeSmem<T, SYM>& s = *reinterpret_cast<PipeSmem<T, SYM>*>(smem_raw);
    constexpr int NC = NCoef<SYM>::value;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + MT_X * ty;
    const int i0 = 1 + blockIdx.x * MT_X, j0 = 1 + blockIdx.y * MT_Y;
    const int k0 = 1 + blockIdx.z * PT_Z;
    const int k1 = min(k0 + PT_Z, L.n[2]);   // exclusive
    const int i = i0 + tx, j = j0 + ty;
    const bool mine = (i < L.n[0]) && (j < L.n[1]);
    const long long S = L.S;

    PipeAcc<T, SYM> acc;
    acc.s = &s;
    acc.tx = tx + 1;
    acc.ty = ty + 1;
    {
        const long long p = L.idx(min(i, L.n[0]), min(j, L.n[1]), k0 - 1);
#pragma unroll
        for (int m = 0; m < NC; m++) acc.cm[m] = __ldg(ddw + m * S + p);
    }
    // prologue: planes k0-1, k0, k0+1 of u and k0, k0+1 of the moduli, then k0+2
    issue_plane<T>(&s.u[0][0][0][0], x, 3, L, i0, j0, k0 - 1, tid);
    issue_plane<T>(&s.u[1][0][0][0], x, 3, L, i0, j0, k0, tid);
    issue_plane<T>(&s.u[2][0][0][0], x, 3, L, i0, j0, k0 + 1, tid);
    issue_plane<T>(&s.c[0][0][0][0], ddw, NC, L, i0, j0, k0, tid);
    issue_plane<T>(&s.c[1][0][0][0], ddw, NC, L, i0, j0, k0 + 1, tid);
    cp_async_commit();
    if (k0 + 2 <= k1) {
        issue_plane<T>(&s.u[3][0][0][0], x, 3, L, i0, j0, k0 + 2, tid);
        issue_plane<T>(&s.c[2][0][0][0], ddw, NC, L, i0, j0, k0 + 2, tid);
    }
    cp_async_commit();

    T nrm = 0;
    for (int k = k0; k < k1; k++) {
        const int it = k - k0;
        long long q = 0;
        T bq[3] = {0, 0, 0}, dq[3] = {0, 0, 0};
        if (mine) {
            q = L.idx(i, j, k);
            if (MODE != MODE_APPLY)
#pragma unroll
                for (int c = 0; c < 3; c++) bq[c] = __ldg(b + c * S + q);
            if (MODE == MODE_JACOBI)
#pragma unroll
                for (int c = 0; c < 3; c++) dq[c] = __ldg(dinv + c * S + q);
        }
        cp_async_wait1();
        __syncthreads();
        acc.um = it % PU;
        acc.u0 = (it + 1) % PU;
        acc.up = (it + 2) % PU;
        acc.c0 = it % PC;
        acc.cp = (it + 1) % PC;
        if (mine) {
            T f[3];
            interior_row<T, SYM>(acc, g, uniform != 0, f);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const long long o = c * S + q;
                if (MODE == MODE_APPLY) {
                    out[o] = f[c];
                } else if (MODE == MODE_RESID) {
                    const T r = bq[c] - f[c];
                    out[o] = r;
                    const T a = fabs(r);
                    nrm = (a > nrm || a != a) ? a : nrm;
                } else {
                    const T xc = s.u[acc.u0][c][ty + 1][tx + 1];
                    out[o] = xc + omega * ((bq[c] - f[c]) * dq[c]);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < NC; m++) acc.cm[m] = s.c[acc.c0][m][ty + 1][tx + 1];
        __syncthreads();
        // refill the slots of u(k-1) and C(k) with plane k+3
        const int kk = k + 3;
        if (kk <= k1) {
            issue_plane<T>(&s.u[it % PU][0][0][0], x, 3, L, i0, j0, kk, tid);
            issue_plane<T>(&s.c[it % PC][0][0][0], ddw, NC, L, i0, j0, kk, tid);
        }
        cp_async_commit();
    }
    cp_async_wait0();
    if (MODE == MODE_RESID && norm_slot) block_max_to_slot<T>(nrm, norm_slot);
}

// ---------------------------------------------------------------------------
// diagonal
// ---------------------------------------------------------------------------
// diag (may be null) = D and dinv = 1/D (0 where D is 0), the latter in T or FP32.
template <typename T, int SYM, typename TI>
__global__ void __launch_bounds__(256) k_diagonal(LevelDesc L, DiagGeo<T> dg, BCTable bc, const T* __restrict__ ddw,
                                                  T* __restrict__ diag, TI* __restrict__ dinv)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i >= L.nn[0] || j >= L.nn[1] || k >= L.nn[2]) return;
    const int pos[3] = {i, j, k};
    int mn[3], mx[3];
    bool bnd = false;
    for (int d = 0; d < 3; d++) {
        mn[d] = !L.per[d] && pos[d] == 0;
        mx[d] = !L.per[d] && pos[d] == L.n[d];
        bnd = bnd || mn[d] || mx[d];
    }
    const long long p = L.idx(i, j, k);
    auto cf = [&](int m) { return __ldg(ddw + m * L.S + p); };
    T d[3];
    if (bnd) diag_boundary<T, SYM>(cf, dg, bc, mn, mx, d);
    else diag_interior<T, SYM>(cf, dg, d);
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (diag) diag[q * L.S + p] = d[q];
        dinv[q * L.S + p] = d[q] != (T)0 ? (TI)((T)1 / d[q]) : (TI)0;
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline dim3 node_grid(const LevelDesc& L, dim3 blk)
{
    return dim3((L.nn[0] + blk.x - 1) / blk.x, (L.nn[1] + blk.y - 1) / blk.y, (L.nn[2] + blk.z - 1) / blk.z);
}

// Smallest x cell count for which the interior goes to the marching kernels
// (AGB_MARCH_MIN_CELLS overrides; used for tile studies).
int march_min_cells()
{
    static int v = [] {
        const char* s = getenv("AGB_MARCH_MIN_CELLS");
        return s ? atoi(s) : 64;
    }();
    return v;
}

// Without the TMA kernel FP32 interiors use the cp.async one unless AGB_PIPE=0.
bool use_pipe_kernel()
{
    static bool v = [] {
        const char* s = getenv("AGB_PIPE");
        return !(s && s[0] == '0');
    }();
    return v;
}

// Whether the interior of a level may go to the marching kernels: a box with
// no periodic direction, large enough to fill every SM several times.
static bool big_level(const LevelDesc& L)
{
    return !L.per[0] && !L.per[1] && !L.per[2] && L.n[0] >= march_min_cells() && L.n[1] >= 16 && L.n[2] >= 16;
}
// FP32: the tiled kernels read each value from HBM once (132 bytes a node and
// Jacobi sweep with general moduli, 56 isotropic); k_rows reads 204 (56) with the
// divergence but has neither a shared-memory ring to fill nor a second launch
// for the shell, so it wins while a level's sweep stays in half of the L2.
// Jacobi, tiled / k_rows: general 65^3 nodes 20.5 / 13.2 us, 81^3 32.8 / 33.7,
// 113^3 70.7 / 82.6, 129^3 84.3 / 108.6; isotropic 65^3 15.4 / 10.3, 97^3 27.6 /
// 20.5, 129^3 56.1 / 63.7.
static bool tiled_f32(int sym, const LevelDesc& L)
{
    const long long bytes = 4LL * L.count() * (sym == SYM_MM ? 21 + 18 + 12 : 2 + 12);
    return big_level(L) && bytes > (64LL << 20) && (use_tma_kernel() || use_pipe_kernel());
}

bool stencil_uses_div(int sym, bool fp32, const LevelDesc& L)
{
    return sym == SYM_MM && !(fp32 && tiled_f32(sym, L));
}

template <typename T, int SYM, int MODE, bool CUBE>
static void rows_dispatch(cudaStream_t st, const LevelDesc& L, const BCTable& bc, const Geo<T>& g, bool uniform,
                          const T* ddw, const T* div, const T* x, const T* b, const T* diag, T* out, T omega,
                          void* norm_slot)
{
    if constexpr (sizeof(T) == 8) {
        if (big_level(L)) {
            // chunk: the longest march (fewest planes loaded twice) up to 16
            // that leaves at least two waves of blocks, and no shorter than 2
            // (general moduli, 65^3 / 129^3 nodes: one wave 97 / 677 us, two
            // 88 / 580 us, six 88 / 585 us)
            const int gx = (L.n[0] - 1 + COL_X - 1) / COL_X, gy = (L.n[1] - 1 + COL_Y - 1) / COL_Y;
            int kz = 16;
            while (kz > 2 && (long long)gx * gy * ((L.n[2] - 1 + kz - 1) / kz) < 2LL * COL_RESIDENT * sm_count()) kz /= 2;
            const int chunks = (L.n[2] - 1 + kz - 1) / kz;
            const long long per_z = (long long)gx * gy * COL_X * COL_Y;
            const int shell_z = (int)((shell_count(L, 1) + per_z - 1) / per_z);
            if (gy <= 65535 && chunks + shell_z <= 65535) {   // the most blocks a grid has in y and z
                pdl_launch(k_column<T, SYM, MODE, CUBE>, dim3(gx, gy, chunks + shell_z), dim3(COL_X, COL_Y), 0, st, L,
                           bc, g, uniform ? 1 : 0, kz, chunks, ddw, div, x, b, diag, out, omega, norm_slot);
                count_launch();
                return;
            }
        }
    }
    long long threads = L.count();
    int nint = 0;
    if (!L.per[0] && !L.per[1] && !L.per[2]) {
        nint = (((L.n[0] - 1) * (L.n[1] - 1) * (L.n[2] - 1) + 31) / 32) * 32;
        threads = nint + shell_count(L, 1);
    }
    pdl_launch(k_rows<T, SYM, MODE, CUBE>, dim3((unsigned)((threads + ROW_THREADS - 1) / ROW_THREADS)),
               dim3(ROW_THREADS), 0, st, L, bc, g, uniform ? 1 : 0, nint, ddw, div, x, b, diag, out, omega, norm_slot);
    count_launch();
}

template <typename T, int SYM, int MODE>
static void stencil_dispatch(cudaStream_t st, const LevelDesc& L, const BCTable& bc, bool uniform, const T* ddw,
                             const T* div, const T* x, const T* b, const T* diag, T* out, T omega, void* norm_slot)
{
    const Geo<T> g = make_geo<T>(L);
    if constexpr (sizeof(T) == 4) {
        if (tiled_f32(SYM, L)) {
            // interior by the tiled kernel, boundary shell by the per-node
            // kernel (the TMA kernel also takes the x-face nodes)
            bool tma = false;
            if (use_tma_kernel() && tma_supported(L) &&
                launch_stencil_tma(st, SYM, MODE, L, bc, uniform, ddw, x, b, diag, out, omega, norm_slot)) {
                tma = true;   // launched by launch_stencil_tma
            } else {
                const size_t smem = sizeof(PipeSmem<T, SYM>);
                dim3 grd((L.n[0] - 1 + MT_X - 1) / MT_X, (L.n[1] - 1 + MT_Y - 1) / MT_Y,
                         (L.n[2] - 1 + PT_Z - 1) / PT_Z);
                pdl_launch(k_stencil_pipe<T, SYM, MODE>, grd, dim3(MT_X, MT_Y, 1), smem, st, L, g, uniform ? 1 : 0,
                           ddw, x, b, diag, out, omega, norm_slot);
            }
            count_launch();
            const int xf = tma ? 0 : 1;
            const long long ns = shell_count(L, xf);
            pdl_launch(k_stencil_shell<T, SYM, MODE>, dim3((unsigned)((ns + 255) / 256)), dim3(256), 0, st, L, bc, g,
                       ddw, x, b, diag, out, omega, norm_slot, xf);
            count_launch();
            return;
        }
    }
    if constexpr (SYM == SYM_MM) {
        if (!div && !uniform) {
            dim3 b2(32, 4, 2);
            if (L.nn[0] <= 40) b2 = dim3(8, 8, 4);   // fewer idle lanes on short rows
            pdl_launch(k_stencil_node<T, MODE>, node_grid(L, b2), b2, 0, st, L, bc, g, ddw, x, b, diag, out, omega,
                       norm_slot);
            count_launch();
            return;
        }
    }
    if (g.cube)
        rows_dispatch<T, SYM, MODE, true>(st, L, bc, g, uniform, ddw, div, x, b, diag, out, omega, norm_slot);
    else
        rows_dispatch<T, SYM, MODE, false>(st, L, bc, g, uniform, ddw, div, x, b, diag, out, omega, norm_slot);
}

template <typename T>
void launch_div_moduli(cudaStream_t st, const LevelDesc& L, const T* ddw, T* div)
{
    const Geo<T> g = make_geo<T>(L);
    const unsigned blocks = (unsigned)((L.count() + 127) / 128);
    if (g.cube) k_div_moduli<T, true><<<blocks, 128, 0, st>>>(L, g, ddw, div);
    else k_div_moduli<T, false><<<blocks, 128, 0, st>>>(L, g, ddw, div);
    count_launch();
}

template <typename T>
void launch_stencil(cudaStream_t st, int sym, int mode, const LevelDesc& L, const BCTable& bc, bool uniform,
                    const T* ddw, const T* div, const T* x, const T* b, const T* diag, T* out, T omega,
                    void* norm_slot)
{
#define DISP(S, M) stencil_dispatch<T, S, M>(st, L, bc, uniform, ddw, div, x, b, diag, out, omega, norm_slot)
    if (sym == SYM_ISO) {
        if (mode == MODE_APPLY) DISP(SYM_ISO, MODE_APPLY);
        else if (mode == MODE_RESID) DISP(SYM_ISO, MODE_RESID);
        else DISP(SYM_ISO, MODE_JACOBI);
    } else {
        if (mode == MODE_APPLY) DISP(SYM_MM, MODE_APPLY);
        else if (mode == MODE_RESID) DISP(SYM_MM, MODE_RESID);
        else DISP(SYM_MM, MODE_JACOBI);
    }
#undef DISP
}

template <int SYM>
static void set_attr()
{
    const int ps = (int)sizeof(PipeSmem<float, SYM>);
    cudaFuncSetAttribute(k_stencil_pipe<float, SYM, MODE_APPLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, ps);
    cudaFuncSetAttribute(k_stencil_pipe<float, SYM, MODE_RESID>, cudaFuncAttributeMaxDynamicSharedMemorySize, ps);
    cudaFuncSetAttribute(k_stencil_pipe<float, SYM, MODE_JACOBI>, cudaFuncAttributeMaxDynamicSharedMemorySize, ps);
}

// Opt the cp.async kernel into its shared-memory size; called once per
// process before any launch (and so before any graph capture).
void init_kernel_attributes()
{
    set_attr<SYM_ISO>();
    set_attr<SYM_MM>();
}

template <typename T, typename TI>
void launch_diagonal(cudaStream_t st, int sym, const LevelDesc& L, const BCTable& bc, const T* ddw, T* diag, TI* dinv)
{
    dim3 blk(32, 4, 2);
    const DiagGeo<T> dg = make_diag_geo<T>(L);
    if (sym == SYM_ISO) k_diagonal<T, SYM_ISO, TI><<<node_grid(L, blk), blk, 0, st>>>(L, dg, bc, ddw, diag, dinv);
    else k_diagonal<T, SYM_MM, TI><<<node_grid(L, blk), blk, 0, st>>>(L, dg, bc, ddw, diag, dinv);
    count_launch();
}

template void launch_stencil<double>(cudaStream_t, int, int, const LevelDesc&, const BCTable&, bool, const double*,
                                     const double*, const double*, const double*, const double*, double*, double,
                                     void*);
template void launch_stencil<float>(cudaStream_t, int, int, const LevelDesc&, const BCTable&, bool, const float*,
                                    const float*, const float*, const float*, const float*, float*, float, void*);
template void launch_div_moduli<double>(cudaStream_t, const LevelDesc&, const double*, double*);
template void launch_div_moduli<float>(cudaStream_t, const LevelDesc&, const float*, float*);
template void launch_diagonal<double, double>(cudaStream_t, int, const LevelDesc&, const BCTable&, const double*,
                                              double*, double*);
template void launch_diagonal<float, float>(cudaStream_t, int, const LevelDesc&, const BCTable&, const float*, float*,
                                            float*);

}  // namespace agb
