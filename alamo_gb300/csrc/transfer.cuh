// transfer.cuh -- per-node arithmetic of the inter-level transfers, shared
// by the single-box and batched kernels.
//
//   restriction     Operator<Node>::restriction, Operator/Operator.cpp:262-363
//   prolongation    Operator<Node>::interpolation, Operator.cpp:365-434
#pragma once
#include "agb_internal.h"

namespace agb {

// index i of a direction of n cells, folded into [0, n) when periodic
__device__ __forceinline__ int wrapn(int i, int n, int per)
{
    if (per) {
        if (i < 0) return i + n;
        if (i >= n) return i - n;
    }
    return i;
}

template <typename T> struct Pair;
template <> struct Pair<float> { typedef float2 type; };
template <> struct Pair<double> { typedef double2 type; };

// Full weighting of one coarse node as the product of one-dimensional weights,
// (1/4, 1/2, 1/4) in a direction or (0, 1, 0) on the coarse domain boundary
// (Operator.cpp:294-352 written out by cases): the fine values 2I and 2I+1 of
// a row are one vector (rows start on 32-byte boundaries and 2I is even; past
// the last node lies zero padding), so nine rows are 18 loads.  On the
// boundary the offsets of the missing rows are those of the node itself, so
// that a zero weight never meets a value the node does not depend on.
template <typename T> struct RestrictNode {
    int x0, xm;              // 2I and 2I - 1
    long long oy[3], oz[3];  // row and plane offsets of 2J + b - 1, 2K + d - 1
    T wc[3], wm[3];          // centre and side weights by direction
    __device__ __forceinline__ RestrictNode(const LevelDesc& Lf, const LevelDesc& Lc, int I, int J, int K)
    {
        const int pos[3] = {I, J, K};
        int at[3][3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const bool b = !Lc.per[d] && (pos[d] == 0 || pos[d] == Lc.n[d]);
            wc[d] = b ? (T)1 : (T)0.5;
            wm[d] = b ? (T)0 : (T)0.25;
#pragma unroll
            for (int q = 0; q < 3; q++) at[d][q] = b ? 2 * pos[d] : wrapn(2 * pos[d] + q - 1, Lf.n[d], Lf.per[d]);
        }
        x0 = at[0][1];
        xm = at[0][0];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            oy[q] = (long long)Lf.P * at[1][q];
            oz[q] = (long long)Lf.P * Lf.nn[1] * at[2][q];
        }
    }
    __device__ __forceinline__ T operator()(const T* __restrict__ src) const
    {
        typedef typename Pair<T>::type V;
        T c[3][3], s[3][3];   // centre value and the sum of its x neighbours, by plane and row
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const T* row = src + oy[b] + oz[d];
                const V v = __ldg(reinterpret_cast<const V*>(row + x0));
                c[d][b] = v.x;
                s[d][b] = wm[0] != (T)0 ? __ldg(row + xm) + v.y : (T)0;
            }
        T C[3], S[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            C[d] = wc[1] * c[d][1] + wm[1] * (c[d][0] + c[d][2]);
            S[d] = wc[1] * s[d][1] + wm[1] * (s[d][0] + s[d][2]);
        }
        return wc[0] * (wc[2] * C[1] + wm[2] * (C[0] + C[2])) + wm[0] * (wc[2] * S[1] + wm[2] * (S[0] + S[2]));
    }
};

// Trilinear prolongation (Operator.cpp:365-434) from one coarse cell: the fine
// nodes (2I, 2I+1) x (2J, 2J+1) x (2K, 2K+1) that exist, from the eight coarse
// values at its corners, read once.  Each fine value is the mean of the
// corners it lies between, summed in the reference's order.
template <typename T> struct InterpCell {
    long long f[4];          // fine offsets of the rows (j, k) = (0,0), (1,0), (0,1), (1,1), at 2I; -1 absent
    bool two;                // 2I + 1 exists
    int I0, I1;
    long long r00, r10, r01, r11;   // coarse rows
    __device__ __forceinline__ InterpCell(const LevelDesc& Lf, const LevelDesc& Lc, int I, int J, int K)
    {
        I0 = I;
        I1 = min(wrapn(I + 1, Lc.n[0], Lc.per[0]), Lc.nn[0] - 1);
        const int J1 = min(wrapn(J + 1, Lc.n[1], Lc.per[1]), Lc.nn[1] - 1);
        const int K1 = min(wrapn(K + 1, Lc.n[2], Lc.per[2]), Lc.nn[2] - 1);
        r00 = Lc.idx(0, J, K);
        r10 = Lc.idx(0, J1, K);
        r01 = Lc.idx(0, J, K1);
        r11 = Lc.idx(0, J1, K1);
        two = 2 * I + 1 < Lf.nn[0];
        const bool j1 = 2 * J + 1 < Lf.nn[1], k1 = 2 * K + 1 < Lf.nn[2];
        f[0] = Lf.idx(2 * I, 2 * J, 2 * K);
        f[1] = j1 ? Lf.idx(2 * I, 2 * J + 1, 2 * K) : -1;
        f[2] = k1 ? Lf.idx(2 * I, 2 * J, 2 * K + 1) : -1;
        f[3] = j1 && k1 ? Lf.idx(2 * I, 2 * J + 1, 2 * K + 1) : -1;
    }
    __device__ __forceinline__ void operator()(const T* __restrict__ crse, T* __restrict__ fine, bool assign) const
    {
        typedef typename Pair<T>::type V;
        const T c000 = __ldg(crse + r00 + I0), c100 = __ldg(crse + r00 + I1);
        const T c010 = __ldg(crse + r10 + I0), c110 = __ldg(crse + r10 + I1);
        const T c001 = __ldg(crse + r01 + I0), c101 = __ldg(crse + r01 + I1);
        const T c011 = __ldg(crse + r11 + I0), c111 = __ldg(crse + r11 + I1);
        V old[4];
        if (!assign) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (f[q] >= 0) {
                    if (two) old[q] = *reinterpret_cast<const V*>(fine + f[q]);
                    else old[q].x = fine[f[q]];
                }
        }
        V v[4];
        v[0].x = c000;
        v[0].y = (T)0.5 * (c000 + c100);
        v[1].x = (T)0.5 * (c000 + c010);
        v[1].y = (T)0.25 * (c000 + c100 + c010 + c110);
        v[2].x = (T)0.5 * (c000 + c001);
        v[2].y = (T)0.25 * (c000 + c001 + c100 + c101);
        v[3].x = (T)0.25 * (c000 + c010 + c001 + c011);
        v[3].y = (T)0.125 * (c000 + c100 + c010 + c001 + c011 + c101 + c110 + c111);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (f[q] < 0) continue;
            if (!assign) {
                v[q].x = old[q].x + v[q].x;
                v[q].y = old[q].y + v[q].y;
            }
            if (two) *reinterpret_cast<V*>(fine + f[q]) = v[q];
            else fine[f[q]] = v[q].x;
        }
    }
};

}  // namespace agb
