// kernels_newton.cu -- the steps either side of the linear solve.
//
//   dw, post      DW = C : (grad u - F0) per node with one-sided gradients on the
//                 boundary: Newton::prepareForSolve, Solver/Nonlocal/Newton.H:157-185;
//                 Model/Solid/Affine/Isotropic.H:42-45; stress output of
//                 Integrator/Base/Mechanics.H:210-236
//   newton_rhs    rhs = b - div DW (interior) | b - BC(u, grad u, DW) (boundary),
//                 Newton.H:199-231
//   bc_init       BC values into the RHS, BC/Operator/Elastic/Constant.H:100-194
//   traction_xhi  trac_hi[0] face integral, Integrator/Base/Mechanics.H:391-431
//   strain        eps = (grad u + grad u^T) / 2, Operator/Elastic.cpp:447-490
//   energy        W = sig : eps / 2 with sig = C : grad u, Operator/Elastic.cpp:552-597
#include <cuda_runtime.h>

#include "agb_internal.h"
#include "stencil.cuh"

namespace agb {

struct NAcc {
    const double* x;
    long long S;
    long long base;
    long long o[3][3];
    __device__ __forceinline__ double u(int p, int di, int dj, int dk) const
    {
        return x[p * S + base + o[0][di + 1] + o[1][dj + 1] + o[2][dk + 1]];
    }
};

__device__ __forceinline__ void node_setup(const LevelDesc& L, int i, int j, int k, NAcc& a, int mn[3], int mx[3])
{
    const long long st[3] = {1, (long long)L.P, (long long)L.P * L.nn[1]};
    const int pos[3] = {i, j, k};
    a.base = L.idx(i, j, k);
    a.S = L.S;
    for (int d = 0; d < 3; d++) {
        mn[d] = !L.per[d] && pos[d] == 0;
        mx[d] = !L.per[d] && pos[d] == L.n[d];
        a.o[d][0] = mn[d] ? 0 : -st[d];
        a.o[d][1] = 0;
        a.o[d][2] = mx[d] ? 0 : st[d];
        if (L.per[d]) {
            if (pos[d] == 0) a.o[d][0] = st[d] * (L.n[d] - 1);
            if (pos[d] == L.n[d] - 1) a.o[d][2] = -st[d] * (L.n[d] - 1);
        }
    }
}

// grad u with the grid factors as reciprocals (FP64 division costs a dozen
// operations of the pipe that bounds these kernels).  On a face the offset of
// the missing neighbour is 0 (node_setup, post_node), so that the one-sided
// difference is the same expression with the factor 1/dx.
__device__ __forceinline__ void gradient(const NAcc& a, const Geo<double>& g, const int mn[3], const int mx[3],
                                         double G[3][3])
{
    for (int d = 0; d < 3; d++) {
        const double f = (mn[d] || mx[d]) ? g.i1[d] : g.h1[d];
        const int ox = d == 0, oy = d == 1, oz = d == 2;
        for (int p = 0; p < 3; p++) G[p][d] = (a.u(p, ox, oy, oz) - a.u(p, -ox, -oy, -oz)) * f;
    }
}

template <int SYM>
__global__ void k_dw(LevelDesc L, Geo<double> g, const double* __restrict__ ddw, const double* __restrict__ F0,
                     const double* __restrict__ u, double* __restrict__ dw)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i >= L.nn[0] || j >= L.nn[1] || k >= L.nn[2]) return;
    NAcc a;
    a.x = u;
    int mn[3], mx[3];
    node_setup(L, i, j, k, a, mn, mx);
    double G[3][3], E[3][3], D[3][3], c[NCoef<SYM>::value];
    gradient(a, g, mn, mx, G);
    for (int r = 0; r < 3; r++)
        for (int s = 0; s < 3; s++) E[r][s] = G[r][s] - (F0 ? F0[(r * 3 + s) * L.S + a.base] : 0.0);
    for (int m = 0; m < NCoef<SYM>::value; m++) c[m] = ddw[m * L.S + a.base];
    c_mul_mat<double, SYM>(c, E, D);
    for (int r = 0; r < 3; r++)
        for (int s = 0; s < 3; s++) dw[(r * 3 + s) * L.S + a.base] = D[r][s];
}

// The fields of a displacement as a caller holds them: stress DW = C : (grad u
// - F0), Elastic::Strain (non-Voigt) and Elastic::Energy, with the gradient
// stencils of Numeric::GetStencil (one-sided on the boundary).  Any output may
// be null.  A block takes 128 consecutive nodes of the full (n+1)^3 box
// (periodic images included) and passes its 9 values a node through shared
// memory, so the interleaved output is written in whole lines; the moduli are
// read once, coalesced, and u in place in the caller's layout when it is device
// memory (U: the strides of u; the host imports u where an output overlaps it).
// Bound by the FP64 pipe, 57 operations a node for the stress and 70 for strain
// and energy: 520 us together at 129^3 nodes
// with general moduli (430 us of FP64 work; with padded intermediate fields, their
// export, FP64 divisions and three forms of every difference evaluated, 1690 us
// besides two allocations a call).
struct UField {
    const double* p;
    long long P, plane, S;   // row, plane and component strides
};
constexpr int POST_NODES = 128;

__device__ __forceinline__ void post_node(const LevelDesc& L, const UField& U, int i, int j, int k, NAcc& a, int mn[3],
                                          int mx[3])
{
    const int pos[3] = {i, j, k};
    const long long st[3] = {1, U.P, U.plane};
    a.x = U.p;
    a.S = U.S;
    a.base = i + U.P * j + U.plane * k;
    for (int d = 0; d < 3; d++) {
        mn[d] = !L.per[d] && pos[d] == 0;
        mx[d] = !L.per[d] && pos[d] == L.n[d];
        a.o[d][0] = mn[d] ? 0 : -st[d];
        a.o[d][1] = 0;
        a.o[d][2] = mx[d] ? 0 : st[d];
        if (L.per[d]) {
            if (pos[d] == 0) a.o[d][0] = st[d] * (L.n[d] - 1);
            if (pos[d] == L.n[d] - 1) a.o[d][2] = -st[d] * (L.n[d] - 1);
        }
    }
}

template <int SYM>
__global__ void __launch_bounds__(POST_NODES) k_post(LevelDesc L, Geo<double> g, const double* __restrict__ ddw,
                                                     const double* __restrict__ F0, UField U,
                                                     double* __restrict__ sigma, double* __restrict__ eps,
                                                     double* __restrict__ energy)
{
    __shared__ double sh[POST_NODES * 9];
    const int N0 = L.n[0] + 1, N1 = L.n[1] + 1;
    const long long total = (long long)N0 * N1 * (L.n[2] + 1), e0 = blockIdx.x * (long long)POST_NODES;
    const long long e = e0 + threadIdx.x;
    const int cnt = (int)min((long long)POST_NODES, total - e0);
    auto write = [&](const double v[3][3], double* out) {
        for (int r = 0; r < 3; r++)
            for (int s = 0; s < 3; s++) sh[threadIdx.x * 9 + 3 * r + s] = v[r][s];
        __syncthreads();
        for (int t = threadIdx.x; t < cnt * 9; t += POST_NODES) out[e0 * 9 + t] = sh[t];
        __syncthreads();
    };
    double G[3][3], S[3][3], E[3][3];
    if (e < total) {
        int i = (int)(e % N0), j = (int)((e / N0) % N1), k = (int)(e / ((long long)N0 * N1));
        if (L.per[0] && i == L.n[0]) i = 0;
        if (L.per[1] && j == L.n[1]) j = 0;
        if (L.per[2] && k == L.n[2]) k = 0;
        NAcc a;
        int mn[3], mx[3];
        post_node(L, U, i, j, k, a, mn, mx);
        gradient(a, g, mn, mx, G);
        const long long q = L.idx(i, j, k);
        if (eps || energy) {
            for (int r = 0; r < 3; r++) {
                E[r][r] = G[r][r];
                for (int s = 0; s < r; s++) E[r][s] = E[s][r] = 0.5 * (G[r][s] + G[s][r]);
            }
        }
        if (sigma || energy) {
            double c[NCoef<SYM>::value];
            for (int m = 0; m < NCoef<SYM>::value; m++) c[m] = __ldg(ddw + m * L.S + q);
            if (F0)
                for (int r = 0; r < 3; r++)
                    for (int s = 0; s < 3; s++) G[r][s] -= F0[(r * 3 + s) * L.S + q];
            c_mul_mat<double, SYM>(c, G, S);
        }
        // sig : eps / 2, both symmetric
        if (energy)
            energy[e] = 0.5 * (S[0][0] * E[0][0] + S[1][1] * E[1][1] + S[2][2] * E[2][2]) + S[0][1] * E[0][1] +
                        S[0][2] * E[0][2] + S[1][2] * E[1][2];
    }
    if (sigma) write(S, sigma);
    if (eps) write(E, eps);
}

// Sum over the x = hi face of the traction sigma_r0 dA: the mean of a quad's
// four corners times its area, summed over the quads, is each face node's
// stress times the share of the quads around it (1/4 of an area for each).
// Blocks leave their sums in part; k_traction_sum adds them in order.
template <int SYM>
__global__ void __launch_bounds__(128) k_traction_face(LevelDesc L, Geo<double> g, const double* __restrict__ ddw,
                                                       const double* __restrict__ F0, UField U,
                                                       double* __restrict__ part)
{
    __shared__ double red[3][4];
    const int i = (L.per[0]) ? 0 : L.n[0];
    const int nj = L.nn[1], nk = L.nn[2];
    const double da = 0.25 * L.dx[1] * L.dx[2];
    double acc[3] = {0, 0, 0};
    for (int e = blockIdx.x * 128 + threadIdx.x; e < nj * nk; e += gridDim.x * 128) {
        const int j = e % nj, k = e / nj;
        const double wj = (!L.per[1] && (j == 0 || j == L.n[1])) ? 1.0 : 2.0;
        const double wk = (!L.per[2] && (k == 0 || k == L.n[2])) ? 1.0 : 2.0;
        NAcc a;
        int mn[3], mx[3];
        double G[3][3], S[3][3], c[NCoef<SYM>::value];
        post_node(L, U, i, j, k, a, mn, mx);
        gradient(a, g, mn, mx, G);
        const long long q = L.idx(i, j, k);
        if (F0)
            for (int r = 0; r < 3; r++)
                for (int s = 0; s < 3; s++) G[r][s] -= F0[(r * 3 + s) * L.S + q];
        for (int m = 0; m < NCoef<SYM>::value; m++) c[m] = __ldg(ddw + m * L.S + q);
        c_mul_mat<double, SYM>(c, G, S);
        for (int r = 0; r < 3; r++) acc[r] += wj * wk * da * S[r][0];
    }
    for (int r = 0; r < 3; r++) {
        for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
        if ((threadIdx.x & 31) == 0) red[r][threadIdx.x >> 5] = acc[r];
    }
    __syncthreads();
    if (threadIdx.x < 3)
        part[blockIdx.x * 3 + threadIdx.x] =
            (red[threadIdx.x][0] + red[threadIdx.x][1]) + (red[threadIdx.x][2] + red[threadIdx.x][3]);
}

__global__ void k_traction_sum(int blocks, const double* __restrict__ part, double* __restrict__ out)
{
    const int r = threadIdx.y, lane = threadIdx.x;
    double s = 0;
    for (int b = lane; b < blocks; b += 32) s += part[3 * b + r];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[r] = s;
}

__global__ void k_newton_rhs(LevelDesc L, Geo<double> g, BCTable bc, const double* __restrict__ u, const double* __restrict__ b,
                             const double* __restrict__ dw, double* __restrict__ rhs)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i >= L.nn[0] || j >= L.nn[1] || k >= L.nn[2]) return;
    NAcc a;
    a.x = u;
    int mn[3], mx[3];
    node_setup(L, i, j, k, a, mn, mx);
    const bool bnd = mn[0] | mx[0] | mn[1] | mx[1] | mn[2] | mx[2];
    double ret[3];
    if (bnd) {
        double G[3][3], S[3][3], uc[3], nrm[3];
        gradient(a, g, mn, mx, G);
        for (int r = 0; r < 3; r++) {
            uc[r] = u[r * L.S + a.base];
            for (int s = 0; s < 3; s++) S[r][s] = dw[(r * 3 + s) * L.S + a.base];
        }
        const int face = face_of(mn, mx, nrm);
        bc_set<double>(bc.type[face], uc, G, S, nrm, ret);
    } else {
        // Numeric::Divergence, Numeric/Stencil.H:588-657 (central)
        for (int r = 0; r < 3; r++) ret[r] = 0.0;
        for (int d = 0; d < 3; d++) {
            const long long pp = a.base + a.o[d][2], pm = a.base + a.o[d][0];
            for (int r = 0; r < 3; r++)
                ret[r] += (dw[(r * 3 + d) * L.S + pp] - dw[(r * 3 + d) * L.S + pm]) * g.h1[d];
        }
    }
    for (int r = 0; r < 3; r++) rhs[r * L.S + a.base] = b[r * L.S + a.base] - ret[r];
}

__global__ void k_bc_init(LevelDesc L, BCTable bc, double* __restrict__ rhs, int homogeneous)
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
    if (!bnd) return;
    double nrm[3];
    const int face = face_of(mn, mx, nrm);
    const long long q = L.idx(i, j, k);
    for (int d = 0; d < 3; d++)
        rhs[d * L.S + q] = (homogeneous && bc.type[face][d] == BCT_DISP) ? 0.0 : bc.val[face][d];
}

static inline dim3 grid_of(const LevelDesc& L, dim3 blk)
{
    return dim3((L.nn[0] + blk.x - 1) / blk.x, (L.nn[1] + blk.y - 1) / blk.y, (L.nn[2] + blk.z - 1) / blk.z);
}

static UField ufield(const LevelDesc& L, const double* u, bool full)
{
    if (!full) return UField{u, L.P, (long long)L.P * L.nn[1], L.S};
    const long long P = L.n[0] + 1, plane = P * (L.n[1] + 1);
    return UField{u, P, plane, plane * (L.n[2] + 1)};
}

void launch_post(cudaStream_t st, int sym, const LevelDesc& L, const double* ddw, const double* F0, const double* u,
                 bool full, double* sigma, double* eps, double* energy)
{
    const Geo<double> g = make_geo<double>(L);
    const long long total = (long long)(L.n[0] + 1) * (L.n[1] + 1) * (L.n[2] + 1);
    const unsigned blocks = (unsigned)((total + POST_NODES - 1) / POST_NODES);
    const UField U = ufield(L, u, full);
    if (sym == SYM_ISO) k_post<SYM_ISO><<<blocks, POST_NODES, 0, st>>>(L, g, ddw, F0, U, sigma, eps, energy);
    else k_post<SYM_MM><<<blocks, POST_NODES, 0, st>>>(L, g, ddw, F0, U, sigma, eps, energy);
    count_launch();
}

void launch_traction_xhi(cudaStream_t st, int sym, const LevelDesc& L, const double* ddw, const double* F0,
                         const double* u, bool full, double* part, double* out3)
{
    const Geo<double> g = make_geo<double>(L);
    const int nodes = L.nn[1] * L.nn[2], blocks = (nodes + 127) / 128 < 256 ? (nodes + 127) / 128 : 256;
    const UField U = ufield(L, u, full);
    if (sym == SYM_ISO) k_traction_face<SYM_ISO><<<blocks, 128, 0, st>>>(L, g, ddw, F0, U, part);
    else k_traction_face<SYM_MM><<<blocks, 128, 0, st>>>(L, g, ddw, F0, U, part);
    k_traction_sum<<<1, dim3(32, 3), 0, st>>>(blocks, part, out3);
    count_launch();
    count_launch();
}

void launch_newton_rhs(cudaStream_t st, int sym, const LevelDesc& L, const BCTable& bc, const double* ddw,
                       const double* F0, const double* u, const double* b, double* rhs, double* dw_work)
{
    const Geo<double> g = make_geo<double>(L);
    dim3 blk(32, 4, 2);
    if (sym == SYM_ISO) k_dw<SYM_ISO><<<grid_of(L, blk), blk, 0, st>>>(L, g, ddw, F0, u, dw_work);
    else k_dw<SYM_MM><<<grid_of(L, blk), blk, 0, st>>>(L, g, ddw, F0, u, dw_work);
    count_launch();
    k_newton_rhs<<<grid_of(L, blk), blk, 0, st>>>(L, g, bc, u, b, dw_work, rhs);
    count_launch();
}

void launch_bc_init(cudaStream_t st, const LevelDesc& L, const BCTable& bc, double* rhs, int homogeneous)
{
    dim3 blk(32, 4, 2);
    k_bc_init<<<grid_of(L, blk), blk, 0, st>>>(L, bc, rhs, homogeneous); count_launch();
}

}  // namespace agb
