// kernels_transfer.cu -- inter-level transfers and vector kernels.
//
//   restriction       Operator<Node>::restriction, Operator/Operator.cpp:262-363
//   interpolation     Operator<Node>::interpolation (additive), Operator.cpp:365-434;
//                     `assign` variant = MLMG interpAssign used by the F-cycle
//   average_ddw       Elastic::averageDownCoeffsSameAmrLevel, Operator/Elastic.cpp:748-910
//   import / export   reference nodal-box images (n+1 nodes per direction, SoA
//                     MultiFab components or AoS BaseFab<Matrix4>) <-> padded storage
#include <cuda_runtime.h>

#include <algorithm>

#include "agb_internal.h"
#include "transfer.cuh"

namespace agb {

static inline dim3 grid_for(const LevelDesc& L, dim3 blk)
{
    return dim3((L.nn[0] + blk.x - 1) / blk.x, (L.nn[1] + blk.y - 1) / blk.y, (L.nn[2] + blk.z - 1) / blk.z);
}

// One coarse node and component a thread (blockIdx.x counts blocks of a
// row and components: the other two have only 65535): on the coarse levels the three components side by side are
// three times the threads, and the FP64 sums a third as long.  257^3 -> 129^3
// nodes, FP32: 103 us (27 reads and a loop over the components: 135); 9^3 -> 5^3,
// FP64: 5.3 us (10.5).
template <typename T>
__global__ void __launch_bounds__(256) k_restrict(LevelDesc Lf, LevelDesc Lc, const T* __restrict__ fine,
                                                  T* __restrict__ crse, int ncomp)
{
    pdl_entry();
    const int c = blockIdx.x % ncomp, I = (blockIdx.x / ncomp) * blockDim.x + threadIdx.x;
    const int J = blockIdx.y * blockDim.y + threadIdx.y;
    const int K = blockIdx.z * blockDim.z + threadIdx.z;
    if (I >= Lc.nn[0] || J >= Lc.nn[1] || K >= Lc.nn[2]) return;
    const RestrictNode<T> r(Lf, Lc, I, J, K);
    crse[c * Lc.S + Lc.idx(I, J, K)] = r(fine + c * Lf.S);
}

// One coarse cell and component a thread.  129^3 -> 257^3 nodes, FP32, additive:
// 72 us (a fine pair a thread, looping over the components: 175).
template <typename T>
__global__ void __launch_bounds__(256) k_interp(LevelDesc Lf, LevelDesc Lc, T* __restrict__ fine,
                                                const T* __restrict__ crse, int assign)
{
    pdl_entry();
    const int c = blockIdx.x % 3, I = (blockIdx.x / 3) * blockDim.x + threadIdx.x;
    const int J = blockIdx.y * blockDim.y + threadIdx.y;
    const int K = blockIdx.z * blockDim.z + threadIdx.z;
    if (I >= Lc.nn[0] || J >= Lc.nn[1] || K >= Lc.nn[2]) return;
    const InterpCell<T> cell(Lf, Lc, I, J, K);
    cell(crse + c * Lc.S, fine + c * Lf.S, assign != 0);
}

template <typename T>
__global__ void k_avg_ddw(LevelDesc Lf, LevelDesc Lc, const T* __restrict__ fine, T* __restrict__ crse, int ncoef)
{
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    const int J = blockIdx.y * blockDim.y + threadIdx.y;
    const int K = blockIdx.z * blockDim.z + threadIdx.z;
    if (I >= Lc.nn[0] || J >= Lc.nn[1] || K >= Lc.nn[2]) return;
    const long long q = Lc.idx(I, J, K);
    const RestrictNode<T> r(Lf, Lc, I, J, K);
    for (int m = 0; m < ncoef; m++) crse[m * Lc.S + q] = r(fine + m * Lf.S);
}

template <typename TD, typename TS>
__global__ void k_convert(long long n, const TS* __restrict__ src, TD* __restrict__ dst, double scale)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        dst[e] = (TD)((double)src[e] * scale);
}

template <typename T>
__global__ void k_axpy(long long n, T* __restrict__ y, const T* __restrict__ x, T a)
{
    pdl_entry();
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        y[e] += a * x[e];
}

template <typename T> struct MaxSlot;
template <> struct MaxSlot<double> {
    static __device__ void put(void* s, double v) { atomicMax((unsigned long long*)s, (unsigned long long)__double_as_longlong(v)); }
};
template <> struct MaxSlot<float> {
    static __device__ void put(void* s, float v) { atomicMax((unsigned int*)s, __float_as_uint(v)); }
};

template <typename T>
__global__ void k_norm_inf(long long n, const T* __restrict__ x, void* slot)
{
    pdl_entry();
    T m = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const T a = fabs(x[e]);
        m = (a > m || a != a) ? a : m;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const T w = __shfl_xor_sync(0xffffffffu, m, o);
        m = (w > m || w != w) ? w : m;
    }
    if ((threadIdx.x & 31) == 0) MaxSlot<T>::put(slot, m);
}

// Reference nodal box (n+1 nodes per direction) -> padded storage, for the
// k-planes [k0, k0+nk).  With `chunk`, src holds only those planes (a staging
// slab); otherwise src is the whole box.  Component planes (SoA): a warp copies one row of
// one component, COPY_UNROLL elements a lane in flight at once; bound by HBM.  A
// thread for each node has three loads in flight and leaves the last warp of a row
// of 2^k + 1 nodes nearly empty: 192 x 160 x 144 cells in FP32 (109 MB moved) 33 us
// against 16 in and 21 out; two sweeps through the public call 431 against 389 us.
constexpr int COPY_UNROLL = 8;
template <typename TD, typename TS>
__global__ void __launch_bounds__(256) k_import_rows(LevelDesc L, long long rows, const TS* __restrict__ src,
                                                     TD* __restrict__ dst, int k0, int nk, long long Nsrc, int chunk)
{
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= rows) return;
    const int j = (int)(r % L.nn[1]);
    const long long t = r / L.nn[1];
    const int k = k0 + (int)(t % nk), c = (int)(t / nk);
    const TS* s = src + c * Nsrc + (long long)(L.n[0] + 1) * (j + (long long)(L.n[1] + 1) * (chunk ? k - k0 : k));
    TD* d = dst + c * L.S + L.idx(0, j, k);
    for (int i0 = lane; i0 < L.nn[0]; i0 += 32 * COPY_UNROLL) {
        TS v[COPY_UNROLL];
#pragma unroll
        for (int u = 0; u < COPY_UNROLL; u++)
            if (i0 + 32 * u < L.nn[0]) v[u] = __ldg(s + i0 + 32 * u);
#pragma unroll
        for (int u = 0; u < COPY_UNROLL; u++)
            if (i0 + 32 * u < L.nn[0]) d[i0 + 32 * u] = (TD)v[u];
    }
}

// and back, periodic images filled
template <typename TD, typename TS>
__global__ void __launch_bounds__(256) k_export_rows(LevelDesc L, long long rows, const TS* __restrict__ src,
                                                     TD* __restrict__ dst, int k0, int nk, long long Ndst, int chunk)
{
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= rows) return;
    const int n0 = L.n[0] + 1, n1 = L.n[1] + 1;
    const int j = (int)(r % n1);
    const long long t = r / n1;
    const int k = k0 + (int)(t % nk), c = (int)(t / nk);
    const TS* s = src + c * L.S + L.idx(0, L.per[1] && j == L.n[1] ? 0 : j, L.per[2] && k == L.n[2] ? 0 : k);
    TD* d = dst + c * Ndst + (long long)n0 * (j + (long long)n1 * (chunk ? k - k0 : k));
    const int wrap = L.per[0] ? L.n[0] : -1;   // this column is column 0
    for (int i0 = lane; i0 < n0; i0 += 32 * COPY_UNROLL) {
        TS v[COPY_UNROLL];
#pragma unroll
        for (int u = 0; u < COPY_UNROLL; u++) {
            const int i = i0 + 32 * u;
            if (i < n0) v[u] = __ldg(s + (i == wrap ? 0 : i));
        }
#pragma unroll
        for (int u = 0; u < COPY_UNROLL; u++)
            if (i0 + 32 * u < n0) d[i0 + 32 * u] = (TD)v[u];
    }
}

// The same for interleaved (AoS) sources, through shared memory: a warp
// copies the contiguous 32 x ncomp source values of 32 consecutive nodes of a
// row into shared memory (coalesced), then writes each component's 32 values
// (coalesced).  Block (32, 8): one row segment per warp.
template <typename TD, typename TS>
__global__ void __launch_bounds__(256) k_import_aos(LevelDesc L, int ncomp, const TS* __restrict__ src,
                                                   TD* __restrict__ dst, int k0, int kc, int chunk)
{
    extern __shared__ __align__(16) unsigned char imp_raw[];
    TS* buf = reinterpret_cast<TS*>(imp_raw) + threadIdx.y * 32 * ncomp;
    const int lane = threadIdx.x;
    const long long r = (long long)blockIdx.y * blockDim.y + threadIdx.y;   // (j, k) row of the chunk
    const int j = (int)(r % L.nn[1]);
    const int k = k0 + (int)(r / L.nn[1]);
    const int i0 = blockIdx.x * 32;
    if (k >= k0 + kc || k >= L.nn[2]) return;   // uniform over the warp
    const int cnt = min(32, L.nn[0] - i0);
    const long long planeN = (long long)(L.n[0] + 1) * (L.n[1] + 1);
    const long long sb = ((long long)i0 + (long long)(L.n[0] + 1) * j + planeN * (chunk ? k - k0 : k)) * ncomp;
    for (int t = lane; t < cnt * ncomp; t += 32) buf[t] = src[sb + t];
    __syncwarp();
    if (lane < cnt) {
        const long long q = L.idx(i0 + lane, j, k);
        for (int c = 0; c < ncomp; c++) dst[c * L.S + q] = (TD)buf[lane * ncomp + c];
    }
}

// and back to interleaved fields, periodic images filled
template <typename TD, typename TS>
__global__ void k_export_aos(LevelDesc L, int ncomp, const TS* __restrict__ src, TD* __restrict__ dst, int k0, int kc,
                             int chunk)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = k0 + blockIdx.z * blockDim.z + threadIdx.z;
    if (i > L.n[0] || j > L.n[1] || k > L.n[2] || k >= k0 + kc) return;
    const long long planeN = (long long)(L.n[0] + 1) * (L.n[1] + 1);
    const long long s = (long long)i + (long long)(L.n[0] + 1) * j + planeN * (chunk ? k - k0 : k);
    const int ii = (L.per[0] && i == L.n[0]) ? 0 : i;
    const int jj = (L.per[1] && j == L.n[1]) ? 0 : j;
    const int kk = (L.per[2] && k == L.n[2]) ? 0 : k;
    const long long q = L.idx(ii, jj, kk);
    for (int c = 0; c < ncomp; c++) dst[s * ncomp + c] = (TD)src[c * L.S + q];
}

// The first damped-Jacobi sweep from x = 0: A 0 = 0 in every row (interior,
// displacement, traction and Neumann rows alike), so x + omega (b - A x) / D
// is omega (b / D) node by node -- the sweep kernels' expression with x = 0,
// equal to theirs up to the sign of a zero.
template <typename T>
__global__ void k_jacobi_zero(long long n, T* __restrict__ out, const T* __restrict__ b, const T* __restrict__ dinv,
                              T omega)
{
    pdl_entry();
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        out[e] = omega * (b[e] * dinv[e]);
}

// y += a * x with x in FP32, y in FP64 (refinement accumulation)
__global__ void k_axpy_mixed(long long n, double* __restrict__ y, const float* __restrict__ x, double a)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        y[e] += a * (double)x[e];
}

template <typename TD>
__global__ void k_recip(long long n, const double* __restrict__ d, TD* __restrict__ r)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        r[e] = d[e] != 0.0 ? (TD)(1.0 / d[e]) : (TD)0;
}

// per-component sums over the stored nodes (sums[0..2], accumulated) or, with
// `subtract`, x -= sums / count: the zero-mean normalization of a fully
// periodic box's displacement
template <typename T>
__global__ void k_mean3(LevelDesc L, T* __restrict__ x, double* __restrict__ sums, int subtract, void* norm_slot)
{
    pdl_entry();
    const long long cnt = L.count();
    double s[3] = {0, 0, 0};
    T m = 0;
    T mean[3] = {0, 0, 0};
    if (subtract)
        for (int c = 0; c < 3; c++) mean[c] = (T)(sums[c] / (double)cnt);
    const bool small = cnt <= 0x7fffffffLL;   // 32-bit index arithmetic
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt; e += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        if (small) {
            const int ei = (int)e;
            i = ei % L.nn[0];
            j = (ei / L.nn[0]) % L.nn[1];
            k = ei / (L.nn[0] * L.nn[1]);
        } else {
            i = (int)(e % L.nn[0]);
            j = (int)((e / L.nn[0]) % L.nn[1]);
            k = (int)(e / ((long long)L.nn[0] * L.nn[1]));
        }
        const long long q = L.idx(i, j, k);
        for (int c = 0; c < 3; c++) {
            if (subtract) {
                const T v = x[c * L.S + q] - mean[c];
                x[c * L.S + q] = v;
                const T a = fabs(v);
                m = (a > m || a != a) ? a : m;
            } else s[c] += (double)x[c * L.S + q];
        }
    }
    if (subtract) {
        if (!norm_slot) return;
        for (int o = 16; o > 0; o >>= 1) {
            const T w = __shfl_xor_sync(0xffffffffu, m, o);
            m = (w > m || w != w) ? w : m;
        }
        if ((threadIdx.x & 31) == 0) MaxSlot<T>::put(norm_slot, m);
        return;
    }
    for (int c = 0; c < 3; c++) {
        double v = s[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(&sums[c], v);
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline int blocks_1d(long long n)
{
    long long b = (n + 255) / 256;
    const long long cap = 16LL * sm_count();
    return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

// Blocks over the coarse nodes: 32-wide rows, 8 x 8 x 4 (and 8 x 4 x 2, which
// spread over more SMs, on the smallest levels) where rows are short.
static inline dim3 transfer_block(const LevelDesc& Lc)
{
    if (Lc.nn[0] > 20) return dim3(32, 4, 2);
    return Lc.count() <= 1000 ? dim3(8, 4, 2) : dim3(8, 8, 4);
}

template <typename T>
void launch_restriction(cudaStream_t st, const LevelDesc& Lf, const LevelDesc& Lc, const T* fine, T* crse, int ncomp)
{
    const dim3 blk = transfer_block(Lc);
    dim3 grd = grid_for(Lc, blk);
    grd.x *= ncomp;
    pdl_launch(k_restrict<T>, grd, blk, 0, st, Lf, Lc, fine, crse, ncomp); count_launch();
}

template <typename T>
void launch_interpolation(cudaStream_t st, const LevelDesc& Lf, const LevelDesc& Lc, T* fine, const T* crse,
                          bool assign)
{
    const dim3 blk = transfer_block(Lc);
    dim3 grd = grid_for(Lc, blk);
    grd.x *= 3;
    pdl_launch(k_interp<T>, grd, blk, 0, st, Lf, Lc, fine, crse, assign ? 1 : 0); count_launch();
}

template <typename T>
void launch_average_ddw(cudaStream_t st, const LevelDesc& Lf, const LevelDesc& Lc, const T* fine, T* crse, int ncoef)
{
    dim3 blk(32, 4, 2);
    k_avg_ddw<T><<<grid_for(Lc, blk), blk, 0, st>>>(Lf, Lc, fine, crse, ncoef); count_launch();
}

template <typename TD, typename TS>
void launch_convert(cudaStream_t st, const LevelDesc& L, int ncomp, const TS* src, TD* dst, double scale)
{
    const long long n = (long long)ncomp * L.S;
    k_convert<TD, TS><<<blocks_1d(n), 256, 0, st>>>(n, src, dst, scale); count_launch();
}

template <typename T>
void launch_axpy(cudaStream_t st, const LevelDesc& L, int ncomp, T* y, const T* x, T a)
{
    const long long n = (long long)ncomp * L.S;
    pdl_launch(k_axpy<T>, dim3(blocks_1d(n)), dim3(256), 0, st, n, y, x, a); count_launch();
}

template <typename T>
void launch_jacobi_zero(cudaStream_t st, const LevelDesc& L, int ncomp, T* out, const T* b, const T* dinv, T omega)
{
    const long long n = (long long)ncomp * L.S;
    pdl_launch(k_jacobi_zero<T>, dim3(blocks_1d(n)), dim3(256), 0, st, n, out, b, dinv, omega); count_launch();
}

template <typename T>
void launch_zero(cudaStream_t st, const LevelDesc& L, int ncomp, T* y)
{
    cudaMemsetAsync(y, 0, sizeof(T) * (size_t)ncomp * (size_t)L.S, st);
}

template <typename T>
void launch_norm_inf(cudaStream_t st, const LevelDesc& L, int ncomp, const T* x, void* slot)
{
    const long long n = (long long)ncomp * L.S;
    pdl_launch(k_norm_inf<T>, dim3(blocks_1d(n)), dim3(256), 0, st, n, x, slot); count_launch();
}

template <typename TD, typename TS>
void launch_import(cudaStream_t st, const LevelDesc& L, int ncomp, const TS* src, TD* dst, bool aos, int k0, int kc,
                   bool chunk)
{
    const int nk = std::min(kc, L.nn[2] - k0);
    if (nk <= 0 || ncomp <= 0) return;
    const long long rows = (long long)nk * L.nn[1];
    if (aos && ncomp > 1) {   // 21 components at most: 43 KB of shared memory
        const dim3 grd((L.nn[0] + 31) / 32, (unsigned)((rows + 7) / 8));
        const size_t smem = 8 * 32 * (size_t)ncomp * sizeof(TS);
        k_import_aos<TD, TS><<<grd, dim3(32, 8), smem, st>>>(L, ncomp, src, dst, k0, kc, chunk ? 1 : 0);
    } else {
        const long long Nsrc = (long long)(L.n[0] + 1) * (L.n[1] + 1) * (chunk ? kc : L.n[2] + 1);
        k_import_rows<TD, TS><<<(unsigned)((rows * ncomp + 7) / 8), 256, 0, st>>>(L, rows * ncomp, src, dst, k0, nk, Nsrc,
                                                                                  chunk ? 1 : 0);
    }
    count_launch();
}

template <typename TD, typename TS>
void launch_export(cudaStream_t st, const LevelDesc& L, int ncomp, const TS* src, TD* dst, bool aos, int k0, int kc,
                   bool chunk)
{
    if (!aos || ncomp == 1) {
        const int nk = std::min(kc, L.n[2] + 1 - k0);
        if (nk <= 0 || ncomp <= 0) return;
        const long long rows = (long long)ncomp * nk * (L.n[1] + 1);
        const long long Ndst = (long long)(L.n[0] + 1) * (L.n[1] + 1) * (chunk ? kc : L.n[2] + 1);
        k_export_rows<TD, TS><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(L, rows, src, dst, k0, nk, Ndst, chunk ? 1 : 0);
        count_launch();
        return;
    }
    dim3 blk(32, 4, 2);
    dim3 grd((L.n[0] + 1 + blk.x - 1) / blk.x, (L.n[1] + 1 + blk.y - 1) / blk.y, (kc + blk.z - 1) / blk.z);
    k_export_aos<TD, TS><<<grd, blk, 0, st>>>(L, ncomp, src, dst, k0, kc, chunk ? 1 : 0); count_launch();
}

template <typename T>
void launch_remove_mean(cudaStream_t st, const LevelDesc& L, T* x, double* sums3, void* norm_slot)
{
    cudaMemsetAsync(sums3, 0, 3 * sizeof(double), st);
    const int g = blocks_1d(L.count());
    pdl_launch(k_mean3<T>, dim3(g), dim3(256), 0, st, L, x, sums3, 0, (void*)nullptr);
    count_launch();
    pdl_launch(k_mean3<T>, dim3(g), dim3(256), 0, st, L, x, sums3, 1, norm_slot);
    count_launch();
}

// sum x y (w == nullptr) or sum x y w^2
__global__ void k_dot(long long n, const double* __restrict__ x, const double* __restrict__ y,
                      const double* __restrict__ w, double* __restrict__ out)
{
    double s = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        s += w ? x[e] * y[e] * (w[e] * w[e]) : x[e] * y[e];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

void launch_dot(cudaStream_t st, long long n, const double* x, const double* y, double* out, const double* w)
{
    k_dot<<<blocks_1d(n), 256, 0, st>>>(n, x, y, w, out);
    count_launch();
}

// ---------------------------------------------------------------------------
// Vector kernels of the inner FP32 GCR (flexible, weighted inner product
// <a, b> = sum a b d^2 with d = 1/diag: the rows of the operator scaled to a
// unit diagonal, so that displacement, traction and interior rows weigh
// alike).  All scalars stay on the device; sums accumulate in FP64.
// ---------------------------------------------------------------------------

// out[i] += sum_e x[e] v_i[e] d[e]^2, i < k (out zeroed by the caller).  Each
// thread sums its elements in FP32 (a few dozen terms; FP64 arithmetic per
// element would bind on GB300's FP64 rate); threads, warps and blocks are
// combined in FP64.
template <int K>
__global__ void __launch_bounds__(256) k_multidot_w(long long n, const float* __restrict__ x, GcrVecs V,
                                                    const float* __restrict__ d, double* __restrict__ out)
{
    pdl_entry();
    float acc[K];
#pragma unroll
    for (int i = 0; i < K; i++) acc[i] = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float dd = d[e];
        const float xw = x[e] * dd * dd;
#pragma unroll
        for (int i = 0; i < K; i++) acc[i] += xw * V.v[i][e];
    }
    __shared__ double red[8][K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = K;
#pragma unroll
    for (int i = 0; i < K; i++) {
        double a = (double)acc[i];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) red[warp][i] = a;
    }
    __syncthreads();
    if (threadIdx.x < k) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w][threadIdx.x];
        atomicAdd(out + threadIdx.x, t);
    }
}

// w -= sum_i beta_i W_i and z -= sum_i beta_i Z_i, i < K (classical Gram-Schmidt step)
template <int K>
__global__ void k_gcr_orth(long long n, const double* __restrict__ beta, GcrVecs W, GcrVecs Z,
                           float* __restrict__ w, float* __restrict__ z)
{
    pdl_entry();
    float b[K];
#pragma unroll
    for (int i = 0; i < K; i++) b[i] = (float)beta[i];
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        float tw = w[e], tz = z[e];
#pragma unroll
        for (int i = 0; i < K; i++) {
            tw -= b[i] * W.v[i][e];
            tz -= b[i] * Z.v[i][e];
        }
        w[e] = tw;
        z[e] = tz;
    }
}

// With ww = <w, w> and rw = <r, w> (dots[0], dots[1]): w, z scaled to unit
// norm, c += (rw / ww) z, r -= (rw / ww) w, and max |r| after it -> slot.
__global__ void k_gcr_step(long long n, const double* __restrict__ dots, float* __restrict__ w,
                           float* __restrict__ z, float* __restrict__ c, float* __restrict__ r, void* slot)
{
    pdl_entry();
    const double ww = dots[0], rw = dots[1];
    const float inv = ww > 0 ? (float)(1.0 / sqrt(ww)) : 0.0f;
    const float a = ww > 0 ? (float)(rw / sqrt(ww)) : 0.0f;   // coefficient of the unit direction
    float m = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float wu = w[e] * inv, zu = z[e] * inv;
        w[e] = wu;
        z[e] = zu;
        c[e] += a * zu;
        const float rn = r[e] - a * wu;
        r[e] = rn;
        const float t = fabsf(rn);
        m = (t > m || t != t) ? t : m;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const float q = __shfl_xor_sync(0xffffffffu, m, o);
        m = (q > m || q != q) ? q : m;
    }
    if ((threadIdx.x & 31) == 0) MaxSlot<float>::put(slot, m);
}

void launch_multidot_w(cudaStream_t st, long long n, int k, const float* x, const GcrVecs& V, const float* d,
                       double* out)
{
    const int nb = blocks_1d(n);
    switch (k) {
#define K_(K) case K: pdl_launch(k_multidot_w<K>, dim3(nb), dim3(256), 0, st, n, x, V, d, out); break;
        K_(1) K_(2) K_(3) K_(4) K_(5) K_(6) K_(7) K_(8) K_(9) K_(10) K_(11) K_(12) K_(13) K_(14) K_(15) K_(16)
#undef K_
    default: return;
    }
    count_launch();
}

void launch_gcr_orth(cudaStream_t st, long long n, int k, const double* beta, const GcrVecs& W, const GcrVecs& Z,
                     float* w, float* z)
{
    const int nb = blocks_1d(n);
    switch (k) {
#define K_(K) case K: pdl_launch(k_gcr_orth<K>, dim3(nb), dim3(256), 0, st, n, beta, W, Z, w, z); break;
        K_(1) K_(2) K_(3) K_(4) K_(5) K_(6) K_(7) K_(8) K_(9) K_(10) K_(11) K_(12) K_(13) K_(14) K_(15) K_(16)
#undef K_
    default: return;
    }
    count_launch();
}

void launch_gcr_step(cudaStream_t st, long long n, const double* dots, float* w, float* z, float* c, float* r,
                     void* slot)
{
    pdl_launch(k_gcr_step, dim3(blocks_1d(n)), dim3(256), 0, st, n, dots, w, z, c, r, slot);
    count_launch();
}

void launch_axpy_mixed(cudaStream_t st, const LevelDesc& L, int ncomp, double* y, const float* x, double a)
{
    const long long n = (long long)ncomp * L.S;
    k_axpy_mixed<<<blocks_1d(n), 256, 0, st>>>(n, y, x, a); count_launch();
}

template <typename TD>
void launch_recip(cudaStream_t st, const LevelDesc& L, int ncomp, const double* d, TD* r)
{
    const long long n = (long long)ncomp * L.S;
    k_recip<TD><<<blocks_1d(n), 256, 0, st>>>(n, d, r); count_launch();
}

#define INST(T)                                                                                              \
    template void launch_restriction<T>(cudaStream_t, const LevelDesc&, const LevelDesc&, const T*, T*, int); \
    template void launch_interpolation<T>(cudaStream_t, const LevelDesc&, const LevelDesc&, T*, const T*, bool); \
    template void launch_average_ddw<T>(cudaStream_t, const LevelDesc&, const LevelDesc&, const T*, T*, int); \
    template void launch_axpy<T>(cudaStream_t, const LevelDesc&, int, T*, const T*, T);                      \
    template void launch_zero<T>(cudaStream_t, const LevelDesc&, int, T*);                                   \
    template void launch_jacobi_zero<T>(cudaStream_t, const LevelDesc&, int, T*, const T*, const T*, T);     \
    template void launch_norm_inf<T>(cudaStream_t, const LevelDesc&, int, const T*, void*);                  \
    template void launch_remove_mean<T>(cudaStream_t, const LevelDesc&, T*, double*, void*);                 \
    template void launch_import<T, double>(cudaStream_t, const LevelDesc&, int, const double*, T*, bool, int, int, bool); \
    template void launch_import<T, float>(cudaStream_t, const LevelDesc&, int, const float*, T*, bool, int, int, bool);   \
    template void launch_export<T, double>(cudaStream_t, const LevelDesc&, int, const double*, T*, bool, int, int, bool); \
    template void launch_export<T, float>(cudaStream_t, const LevelDesc&, int, const float*, T*, bool, int, int, bool);
INST(double)
INST(float)
#undef INST
template void launch_recip<float>(cudaStream_t, const LevelDesc&, int, const double*, float*);
template void launch_convert<float, double>(cudaStream_t, const LevelDesc&, int, const double*, float*, double);
template void launch_convert<double, float>(cudaStream_t, const LevelDesc&, int, const float*, double*, double);
template void launch_convert<double, double>(cudaStream_t, const LevelDesc&, int, const double*, double*, double);

}  // namespace agb
