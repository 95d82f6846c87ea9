// kernels_batch.cu -- batched solves of many independent boxes (periodic RVEs
// of different sizes) with persistent tile kernels.
//
// A level arena holds every problem's fields of that level back to back
// (BProb gives the offsets).  A tile list names (problem, block) pairs; each
// kernel is launched with a grid sized to the GPU (a few CTAs per SM) and its
// CTAs stride over the tile list, so one launch covers all problems of the
// level whatever their sizes.  Problems already converged are skipped through
// the `active` flags, so the same captured graph serves every iteration.
//
// Per-node arithmetic is the single-box arithmetic of stencil.cuh
// (Operator/Elastic.cpp:141-292; transfers Operator.cpp:262-434).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "agb_internal.h"
#include "bottom.cuh"
#include "stencil.cuh"
#include "transfer.cuh"

namespace agb {

// The persistent launches ask for `grid` CTAs (a few per SM).  A CTA that is
// not resident from the start runs its share of the tiles after a resident
// one has finished all of its own, which adds a second wave; so each launch is
// trimmed to the CTAs of that kernel (256 threads) that fit on the device at
// once.  Queried once per kernel (the occupancy query is no stream operation,
// so it may also run while a graph is being captured).
static int fit_grid(const void* kernel, int grid, cudaStream_t)
{
    static std::mutex mu;
    static std::unordered_map<const void*, int> cache;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(kernel);
    if (it != cache.end()) return std::min(grid, it->second);
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 256, 0) != cudaSuccess || per < 1 || sms < 1)
        return grid;
    cache[kernel] = sms * per;
    return std::min(grid, sms * per);
}

// Shapes 0-4: one node per thread (k_batch_stencil).  Shapes 5 and 6: 32 x 8 and
// 16 x 16 columns marching through 16 planes (k_batch_march), for fully periodic
// isotropic batches only.  32 x 8 leaves a half or a quarter of a warp's row
// empty on edges that 32 does not divide.  The tuner times 16 x 16 where it has
// at least half as many tiles as there are SMs: with fewer most of the chip is
// idle for the 18 steps of a tile.
static const int kShapes[7][3] = {{32, 4, 2}, {32, 8, 1}, {16, 8, 2}, {8, 8, 4}, {64, 4, 1}, {32, 8, 16}, {16, 16, 16}};
constexpr int kMarchShape = 5, kMarchShape16 = 6;
int batch_shape_count() { return 7; }
bool batch_shape_worth(int shape, int tiles, int sms) { return shape != kMarchShape16 || 2 * tiles >= sms; }
void batch_shape_dims(int shape, int dims[3])
{
    for (int d = 0; d < 3; d++) dims[d] = kShapes[shape][d];
}
bool batch_shape_ok(int shape, int sym, const int per[3])
{
    if (shape < 0 || shape >= batch_shape_count()) return false;
    if (shape == kMarchShape || shape == kMarchShape16) return sym == SYM_ISO && per[0] && per[1] && per[2];
    return true;
}

template <typename T> __device__ __forceinline__ Geo<T> geo_of(const BProb& p)
{
    Geo<T> g;
    for (int d = 0; d < 3; d++) {
        if constexpr (sizeof(T) == 4) {
            g.h1[d] = p.h1f[d];
            g.i1[d] = p.i1f[d];
            g.h2[d] = p.h2f[d];
            g.hm[d] = p.hmf[d];
        } else {
            g.h1[d] = p.h1[d];
            g.i1[d] = p.i1[d];
            g.h2[d] = p.h2[d];
            g.hm[d] = p.hm[d];
        }
    }
    g.cube = p.cube;
    return g;
}

template <typename T> struct BAcc {
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

template <typename T> struct SlotMax;
template <> struct SlotMax<double> {
    static __device__ void put(void* s, int p, double v)
    {
        atomicMax((unsigned long long*)s + p, (unsigned long long)__double_as_longlong(v));
    }
};
template <> struct SlotMax<float> {
    static __device__ void put(void* s, int p, float v) { atomicMax((unsigned int*)s + 2 * p, __float_as_uint(v)); }
};

// block max of v over threads sharing the tile (all of the CTA) -> slot[prob]
template <typename T> __device__ __forceinline__ void tile_max(T v, void* slots, int prob)
{
    __shared__ T red[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        const T w = __shfl_xor_sync(0xffffffffu, v, o);
        v = (w > v || w != w) ? w : v;
    }
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = lane < (int)(blockDim.x >> 5) ? red[lane] : (T)0;
        for (int o = 16; o > 0; o >>= 1) {
            const T w = __shfl_xor_sync(0xffffffffu, v, o);
            v = (w > v || w != w) ? w : v;
        }
        if (lane == 0) SlotMax<T>::put(slots, prob, v);
    }
}

// The CTA's next tile, read while the current one is computed; past the list an
// end marker.  With the grid factors kept in FP32 beside the FP64 ones (twelve
// conversions a thread and tile ran at the FP64 rate) the node-per-thread
// sweeps of 17.3 M nodes went from 626-816 to 521-669 us, of a quarter of a
// million nodes from 33 to 26 us.
__device__ __forceinline__ BTile next_tile(const BTile* __restrict__ tiles, int t, int ntiles)
{
    BTile e;
    e.prob = -1;
    return t < ntiles ? tiles[t] : e;
}

// |v| by its bits: order-preserving, NaN above all, and no FP64 compare
__device__ __forceinline__ unsigned int abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned long long abs_bits(double v)
{
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ float as_value(unsigned int b) { return __uint_as_float(b); }
__device__ __forceinline__ double as_value(unsigned long long b) { return __longlong_as_double((long long)b); }

// node of the tile handled by this thread (1D CTA of 256 threads)
template <int BX, int BY, int BZ>
__device__ __forceinline__ bool tile_node(const BTile& t, const LevelDesc& L, int& i, int& j, int& k)
{
    const int tid = threadIdx.x;
    i = t.bx * BX + tid % BX;
    j = t.by * BY + (tid / BX) % BY;
    k = t.bz * BZ + tid / (BX * BY);
    return i < L.nn[0] && j < L.nn[1] && k < L.nn[2];
}

template <typename T, int SYM, int MODE, int BX, int BY, int BZ>
__global__ void __launch_bounds__(256) k_batch_stencil(const BProb* __restrict__ probs, const BTile* __restrict__ tiles,
                                                       int ntiles, const int* __restrict__ active, BCTable bc,
                                                       int uniform, const T* __restrict__ ddw,
                                                       const T* __restrict__ x, const T* __restrict__ b,
                                                       const T* __restrict__ dinv, T* __restrict__ out, T omega,
                                                       void* norm_slots)
{
    // residual norms: each thread keeps its max while the CTA's tiles stay in
    // one problem (tiles are ordered by problem) and the CTA flushes it to the
    // problem's slot when the problem changes
    T nrm = 0;
    int cur = -1;
    BTile ahead = next_tile(tiles, blockIdx.x, ntiles);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BTile tl = ahead;
        if (tl.prob < 0) break;   // compacted list: only end markers follow (uniform over the CTA)
        ahead = next_tile(tiles, t + gridDim.x, ntiles);
        if (active && !active[tl.prob]) continue;   // uniform over the CTA
        if (MODE == MODE_RESID && norm_slots && tl.prob != cur) {
            if (cur >= 0) tile_max<T>(nrm, norm_slots, cur);
            nrm = 0;
            cur = tl.prob;
        }
        const BProb& P = probs[tl.prob];
        const LevelDesc& L = P.L;
        int i, j, k;
        const bool ok = tile_node<BX, BY, BZ>(tl, L, i, j, k);
        if (ok) {
            const Geo<T> g = geo_of<T>(P);
            const T* xp = x + P.vo;
            BAcc<T> acc{xp, ddw + P.co, L.S, make_nbr(L, i, j, k)};
            const int pos[3] = {i, j, k};
            int mn[3], mx[3];
            bool bnd = false;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                mn[d] = !L.per[d] && pos[d] == 0;
                mx[d] = !L.per[d] && pos[d] == L.n[d];
                bnd = bnd || mn[d] || mx[d];
            }
            T f[3];
            if (bnd) boundary_row<T, SYM>(acc, g, bc, mn, mx, f);
            else interior_row<T, SYM>(acc, g, uniform != 0, f);
            const long long q = P.vo + acc.nb.base;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const long long o = q + c * L.S;
                if (MODE == MODE_APPLY) out[o] = f[c];
                else if (MODE == MODE_RESID) {
                    const T r = b[o] - f[c];
                    out[o] = r;
                    const T a = fabs(r);
                    nrm = (a > nrm || a != a) ? a : nrm;
                } else {
                    out[o] = x[o] + omega * ((b[o] - f[c]) * dinv[o]);
                }
            }
        }
    }
    if (MODE == MODE_RESID && norm_slots && cur >= 0) tile_max<T>(nrm, norm_slots, cur);
}

// ---------------------------------------------------------------------------
// Marching tile kernel for fully periodic batches with isotropic moduli.
//
// A tile is a 32 x 8 block of columns of one problem and a chunk of up to 16
// planes.  The halo wraps periodically (node -1 is node n-1, node n is node 0),
// so every stored node is an interior node of the stencil.  The CTA walks the
// chunk plane by plane; every thread copies its halo values of a plane global
// -> shared with cp.async (the wrapped rows are not contiguous), D - 2 planes
// ahead of their use, into a ring of D planes: one is in use, one just landed.
//
// What a column needs of a plane it forms once, when the plane lands: the value,
// the central differences and the second differences in x and y (five reads a
// component).  They go from "above" to "own" to "below" in registers, so the
// mixed differences xz and yz are differences of registers and only the four
// corners of xy are read again: 27 + 10 shared reads a node where the row read
// from the ring takes 57 + 12.  Sweeps of 17.3 M nodes in 48 RVEs (edges 32 to
// 96): FP32 296 us with every difference read from the ring, 256 as it is on
// tiles of 32 x 8, 230 on tiles of 16 x 16 (32 columns leave a quarter of the lanes of an
// edge of 48 empty); 112 us is HBM's time.  The FP64 residual went from 4.0 to
// 3.3 ms, the next coarser FP32 level from 60 to 44 us.  Issue bound.
// The row is iso_row's, of the same differences as interior_row's.
// ---------------------------------------------------------------------------
constexpr int BM_Z = 16;
template <typename T, int BX> struct BMarch {
    static constexpr int BY = 256 / BX;
    static constexpr int HX = BX + 2, HALO = HX * (BY + 2);   // halo nodes of a plane: 340 or 324, two a thread at most
    static constexpr int D = sizeof(T) == 4 ? 4 : 3;          // planes in the ring (static shared memory: 48 KB)
};

__device__ __forceinline__ int pwrap(int i, int n)
{
    i %= n;
    return i < 0 ? i + n : i;
}

template <int B> __device__ __forceinline__ void cp_async(void* smem, const void* gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(sa), "l"(gmem), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// the moduli of a node and its neighbours for iso_row: own column in registers
template <typename T, int BX> struct BMarchModuli {
    const T (*s)[BMarch<T, BX>::HALO];   // the plane's two moduli
    int h;
    const T *cm, *c0, *cp;    // own column below, at and above the node
    __device__ __forceinline__ T C(int m, int di, int dj, int dk) const
    {
        if (dk < 0) return cm[m];
        if (dk > 0) return cp[m];
        return di || dj ? s[m][h + di + BMarch<T, BX>::HX * dj] : c0[m];
    }
};

template <typename T, int MODE, int BX>
__global__ void __launch_bounds__(256, sizeof(T) == 4 && MODE != MODE_RESID ? 3 : 2)
    k_batch_march(const BProb* __restrict__ probs, const BTile* __restrict__ tiles, int ntiles,
                  const int* __restrict__ active, int uniform, const T* __restrict__ ddw, const T* __restrict__ x,
                  const T* __restrict__ b, const T* __restrict__ dinv, T* __restrict__ out, T omega, void* norm_slots)
{
    constexpr int D = BMarch<T, BX>::D, BY = BMarch<T, BX>::BY, HX = BMarch<T, BX>::HX, HALO = BMarch<T, BX>::HALO;
    __shared__ __align__(16) T su[D][3][HALO];
    __shared__ __align__(16) T sc[D][2][HALO];
    // a warp's rows: one of 32, or rows w and w + 8 of 16 (8 rows of 18 words
    // apart: the other 16 banks)
    const int tid = threadIdx.x, tx = tid % BX, ty = BX == 32 ? tid / 32 : tid / 32 + 8 * (tid / 16 % 2);
    const int h = (tx + 1) + HX * (ty + 1);
    typedef decltype(abs_bits(T())) Bits;
    Bits nrm = 0;
    int cur = -1;
    BTile ahead = next_tile(tiles, blockIdx.x, ntiles);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BTile tl = ahead;
        if (tl.prob < 0) break;   // compacted list: only end markers follow (uniform over the CTA)
        ahead = next_tile(tiles, t + gridDim.x, ntiles);
        if (active && !active[tl.prob]) continue;
        if (MODE == MODE_RESID && norm_slots && tl.prob != cur) {
            if (cur >= 0) tile_max<T>(as_value(nrm), norm_slots, cur);
            nrm = 0;
            cur = tl.prob;
        }
        const BProb& P = probs[tl.prob];
        const LevelDesc& L = P.L;
        const Geo<T> g = geo_of<T>(P);
        // offsets inside a problem fit 32 bits: three components of 2^31 / 1.5 nodes
        // would not fit the device beside their moduli and vectors
        const unsigned S = (unsigned)L.S, plane = (unsigned)L.P * L.nn[1];
        const int n2 = L.n[2];
        const int i0 = tl.bx * BX, j0 = tl.by * BY, k0 = tl.bz * BM_Z;
        const int k1 = min(k0 + BM_Z, n2);
        const int i = i0 + tx, j = j0 + ty;
        const bool mine = i < L.n[0] && j < L.n[1];
        const T *xq = x + P.vo, *cq = ddw + P.co, *bv = b + P.vo, *dv = dinv + P.vo;
        T* ov = out + P.vo;
        unsigned own = i + (unsigned)L.P * j + plane * k0;   // the own node of plane kk (from plane k0 on)
        unsigned hoff[2];   // in-plane offsets of this thread's halo nodes, wrapped
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int e = min(tid + 256 * q, HALO - 1);
            hoff[q] = pwrap(i0 - 1 + e % HX, L.n[0]) + (unsigned)L.P * pwrap(j0 - 1 + e / HX, L.n[1]);
        }
        // copies of plane kk into ring slot w; one commit group (empty past the chunk)
        auto issue = [&](int kk, int w) {
            if (kk <= k1) {
                const unsigned pk = plane * (kk < 0 ? n2 - 1 : (kk >= n2 ? kk - n2 : kk));
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int e = tid + 256 * q;
                    if (e < HALO) {
                        const unsigned o = hoff[q] + pk;
#pragma unroll
                        for (int c = 0; c < 3; c++) cp_async<sizeof(T)>(&su[w][c][e], xq + (o + c * S));
#pragma unroll
                        for (int m = 0; m < 2; m++) cp_async<sizeof(T)>(&sc[w][m][e], cq + (o + m * S));
                    }
                }
            }
            cp_commit();
        };
#pragma unroll
        for (int d = 0; d < D - 2; d++) issue(k0 - 1 + d, d);
        // of the planes below (m), at (0) and above: value, x and y differences
        T um[3] = {}, u0[3] = {}, dxm[3] = {}, dx0[3] = {}, dym[3] = {}, dy0[3] = {}, xx0[3] = {}, yy0[3] = {};
        T cm[2] = {}, c0[2] = {};
        T bq[3] = {}, dq[3] = {};   // b and 1/D of the own node, read when the plane below it is done
        int w0 = D - 1, wu = 0, wi = D - 2;   // slots of planes kk - 1, kk and of the plane to copy
#pragma unroll 3   // the state moves by renaming, not by copies
        for (int kk = k0 - 1; kk <= k1; kk++) {
            cp_wait<D - 3>();   // plane kk has landed
            __syncthreads();    // for every thread; and plane kk - 2, whose slot is filled next, was read by all
            issue(kk + D - 2, wi);
            T uu[3], dxu[3], dyu[3], xxu[3], yyu[3], cu[2];
#pragma unroll
            for (int p = 0; p < 3; p++) {
                const T* q = &su[wu][p][h];
                uu[p] = q[0];
                const T c2 = (T)2 * uu[p], xp = q[1], xm = q[-1], yp = q[HX], ym = q[-HX];
                dxu[p] = xp - xm;
                dyu[p] = yp - ym;
                xxu[p] = (xp - c2) + xm;
                yyu[p] = (yp - c2) + ym;
            }
#pragma unroll
            for (int m = 0; m < 2; m++) cu[m] = sc[wu][m][h];
            if (mine && kk > k0) {
                RowD<T> r;
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const T* q = &su[w0][p][h];
                    r.d2[0][p] = xx0[p];
                    r.d2[1][p] = yy0[p];
                    r.d2[2][p] = (uu[p] - (T)2 * u0[p]) + um[p];
                    r.mx[0][p] = (q[1 + HX] - q[HX - 1]) - (q[1 - HX] - q[-1 - HX]);
                    r.mx[1][p] = dxu[p] - dxm[p];
                    r.mx[2][p] = dyu[p] - dym[p];
                    r.G[0][p] = dx0[p];
                    r.G[1][p] = dy0[p];
                    r.G[2][p] = uu[p] - um[p];
                }
                const BMarchModuli<T, BX> mod{sc[w0], h, cm, c0, cu};
                T f[3];
                if (g.cube) {
                    iso_row<T, true>(mod, g, uniform != 0, r, f);
#pragma unroll
                    for (int c = 0; c < 3; c++) f[c] *= row_scale<T, true>(g);
                } else {
#pragma unroll
                    for (int p = 0; p < 3; p++) scale_diffs<T, false>(g, r, p);
                    iso_row<T, false>(mod, g, uniform != 0, r, f);
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const unsigned o = own - plane + c * S;
                    if (MODE == MODE_APPLY) ov[o] = f[c];
                    else if (MODE == MODE_RESID) {
                        const T v = bq[c] - f[c];
                        ov[o] = v;
                        const Bits a = abs_bits(v);
                        nrm = a > nrm ? a : nrm;
                    } else {
                        ov[o] = u0[c] + omega * ((bq[c] - f[c]) * dq[c]);
                    }
                }
            }
#pragma unroll
            for (int p = 0; p < 3; p++) {
                um[p] = u0[p];
                u0[p] = uu[p];
                dxm[p] = dx0[p];
                dx0[p] = dxu[p];
                dym[p] = dy0[p];
                dy0[p] = dyu[p];
                xx0[p] = xxu[p];
                yy0[p] = yyu[p];
            }
            if (mine && kk >= k0 && kk < k1) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    if (MODE != MODE_APPLY) bq[c] = __ldg(bv + (own + c * S));
                    if (MODE == MODE_JACOBI) dq[c] = __ldg(dv + (own + c * S));
                }
            }
            if (kk >= k0) own += plane;
#pragma unroll
            for (int m = 0; m < 2; m++) {
                cm[m] = c0[m];
                c0[m] = cu[m];
            }
            w0 = wu;
            wu = wu + 1 == D ? 0 : wu + 1;
            wi = wi + 1 == D ? 0 : wi + 1;
        }
        __syncthreads();   // every copy has landed and been read: the next tile's may start
    }
    if (MODE == MODE_RESID && norm_slots && cur >= 0) tile_max<T>(as_value(nrm), norm_slots, cur);
}

// Full weighting (restriction) or trilinear prolongation between the levels of
// every listed problem.  Tiles cover the coarse level (32 x 4 x 2 shape): a
// thread takes one coarse node or cell (RestrictNode, InterpCell).
template <typename T>
__global__ void __launch_bounds__(256) k_batch_transfer(int restrict_not_interp, int assign,
                                                        const BProb* __restrict__ pf, const BProb* __restrict__ pc,
                                                        const BTile* __restrict__ tiles, int ntiles,
                                                        const int* __restrict__ active, const T* __restrict__ src,
                                                        T* __restrict__ dst)
{
    BTile ahead = next_tile(tiles, blockIdx.x, ntiles);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BTile tl = ahead;
        if (tl.prob < 0) break;   // compacted list: only end markers follow (uniform over the CTA)
        ahead = next_tile(tiles, t + gridDim.x, ntiles);
        if (active && !active[tl.prob]) continue;
        const LevelDesc& Lf = pf[tl.prob].L;
        const LevelDesc& Lc = pc[tl.prob].L;
        int i, j, k;
        if (!tile_node<32, 4, 2>(tl, Lc, i, j, k)) continue;
        const long long vf = pf[tl.prob].vo, vc = pc[tl.prob].vo;
        if (restrict_not_interp) {
            const RestrictNode<T> r(Lf, Lc, i, j, k);
            const long long q = vc + Lc.idx(i, j, k);
#pragma unroll
            for (int c = 0; c < 3; c++) dst[q + c * Lc.S] = r(src + vf + c * Lf.S);
        } else {
            const InterpCell<T> cell(Lf, Lc, i, j, k);
#pragma unroll
            for (int c = 0; c < 3; c++) cell(src + vc + c * Lc.S, dst + vf + c * Lf.S, assign != 0);
        }
    }
}

__global__ void __launch_bounds__(256) k_batch_avg_ddw(const BProb* __restrict__ pf, const BProb* __restrict__ pc,
                                                       const BTile* __restrict__ tiles, int ntiles,
                                                       const double* __restrict__ fine, double* __restrict__ crse,
                                                       int ncoef)
{
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BTile tl = tiles[t];
        const LevelDesc& Lf = pf[tl.prob].L;
        const LevelDesc& Lc = pc[tl.prob].L;
        int I, J, K;
        if (!tile_node<32, 4, 2>(tl, Lc, I, J, K)) continue;
        const long long q = pc[tl.prob].co + Lc.idx(I, J, K);
        const RestrictNode<double> r(Lf, Lc, I, J, K);
        for (int m = 0; m < ncoef; m++) crse[q + m * Lc.S] = r(fine + pf[tl.prob].co + m * Lf.S);
    }
}

template <int SYM>
__global__ void __launch_bounds__(256) k_batch_diag(const BProb* __restrict__ probs, const BTile* __restrict__ tiles,
                                                    int ntiles, BCTable bc, const double* __restrict__ ddw,
                                                    double* __restrict__ diag, double* __restrict__ dinv64,
                                                    float* __restrict__ dinv32)
{
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BTile tl = tiles[t];
        const BProb& P = probs[tl.prob];
        const LevelDesc& L = P.L;
        int i, j, k;
        if (!tile_node<32, 4, 2>(tl, L, i, j, k)) continue;
        const int pos[3] = {i, j, k};
        int mn[3], mx[3];
        for (int d = 0; d < 3; d++) {
            mn[d] = !L.per[d] && pos[d] == 0;
            mx[d] = !L.per[d] && pos[d] == L.n[d];
        }
        const long long p = L.idx(i, j, k);
        DiagGeo<double> dg;
        for (int d = 0; d < 3; d++) {
            dg.h2m[d] = -2.0 * P.h2[d];
            dg.i1[d] = P.i1[d];
        }
        auto cf = [&](int m) { return __ldg(ddw + P.co + m * L.S + p); };
        double dd[3];
        if (mn[0] | mx[0] | mn[1] | mx[1] | mn[2] | mx[2]) diag_boundary<double, SYM>(cf, dg, bc, mn, mx, dd);
        else diag_interior<double, SYM>(cf, dg, dd);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const double d = dd[q], inv = d != 0.0 ? 1.0 / d : 0.0;
            const long long o = P.vo + q * L.S + p;
            diag[o] = d;
            dinv64[o] = inv;
            if (dinv32) dinv32[o] = (float)inv;
        }
    }
}

// ---------------------------------------------------------------------------
// Elementwise and reducing kernels over segments: runs of up to BSEG
// consecutive elements of one component of one problem (padded rows included:
// padding is zero in every vector and stays zero).  A CTA takes a contiguous
// part of the list, so its segments mostly belong to one problem and its sums
// go out once; a thread has four 16-byte vectors of every array in flight.
// The node tiles these kernels used before cost a chain of dependent loads (tile,
// problem, node) for 256 nodes, and their per-problem scalars were FP64 roots
// and divisions in every thread; here one thread makes them once a problem.
// Bound by HBM.  48 RVEs (17.3 M nodes), finest level, us before and now: GCR
// step 872 and 175, the sums and the subtraction of the FP32 zero-mean
// projection 305 and 37, 305 and 75; the solve 160 to 124 ms with the copies
// around the cycle gone.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void seg_range(const BSegList& list, int& s0, int& s1)
{
    const long long n = *list.n;
    s0 = (int)(n * blockIdx.x / gridDim.x);
    s1 = (int)(n * (blockIdx.x + 1) / gridDim.x);
}

// f(element offset, q): every vector of VE elements of a segment, q = 0 .. per thread
template <int VE, class F> __device__ __forceinline__ void seg_each(const BSeg& s, const F& f)
{
#pragma unroll
    for (int q = 0; q < BSEG / (256 * VE); q++) {
        const int e = (threadIdx.x + 256 * q) * VE;
        if (e < s.count) f(s.base + e);
    }
}

//   BV_ZERO        y = 0
//   BV_COPY        y = x
//   BV_AXPY        y += a x
//   BV_SCALE_TO32  y(float) = x(double) / scale[prob]
//   BV_ACC_FROM32  y(double) += x(float) * scale[prob]
//   BV_JACOBI0     y = a (x * x2): the first damped-Jacobi sweep from a zero
//                  guess (x the right-hand side, x2 = 1/D, a = omega), the
//                  sweep kernels' expression with A 0 = 0
template <int OP, typename T>
__global__ void __launch_bounds__(256) k_seg_vec(BSegList list, const int* __restrict__ active, void* yv,
                                                 const void* xv, double a, const double* __restrict__ scale,
                                                 const void* x2v)
{
    int s0, s1;
    seg_range(list, s0, s1);
    int prob = -1;
    double sc = 1.0;   // 1 / scale or scale of the current problem (an FP64 division a problem, not an element)
    for (int t = s0; t < s1; t++) {
        const BSeg s = list.d[t];
        if (active && !active[s.prob]) continue;   // uniform over the CTA
        if constexpr (OP == BV_SCALE_TO32 || OP == BV_ACC_FROM32) {
            if (s.prob != prob) {
                prob = s.prob;
                sc = OP == BV_SCALE_TO32 ? 1.0 / scale[prob] : scale[prob];
            }
            seg_each<2>(s, [&](long long e) {
                if (OP == BV_SCALE_TO32) {
                    const double2 x = *reinterpret_cast<const double2*>((const double*)xv + e);
                    *reinterpret_cast<float2*>((float*)yv + e) = make_float2((float)(x.x * sc), (float)(x.y * sc));
                } else {
                    const float2 x = *reinterpret_cast<const float2*>((const float*)xv + e);
                    double2* y = reinterpret_cast<double2*>((double*)yv + e);
                    double2 v = *y;
                    v.x += (double)x.x * sc;
                    v.y += (double)x.y * sc;
                    *y = v;
                }
            });
        } else if constexpr (sizeof(T) == 4) {
            const float f = (float)a;
            seg_each<4>(s, [&](long long e) {
                float4* y = reinterpret_cast<float4*>((float*)yv + e);
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (OP != BV_ZERO) {
                    const float4 x = *reinterpret_cast<const float4*>((const float*)xv + e);
                    if (OP == BV_COPY) v = x;
                    else if (OP == BV_JACOBI0) {
                        const float4 d = *reinterpret_cast<const float4*>((const float*)x2v + e);
                        v = make_float4(f * (x.x * d.x), f * (x.y * d.y), f * (x.z * d.z), f * (x.w * d.w));
                    } else {
                        v = *y;
                        v = make_float4(v.x + f * x.x, v.y + f * x.y, v.z + f * x.z, v.w + f * x.w);
                    }
                }
                *y = v;
            });
        } else {
            seg_each<2>(s, [&](long long e) {
                double2* y = reinterpret_cast<double2*>((double*)yv + e);
                double2 v = make_double2(0.0, 0.0);
                if (OP != BV_ZERO) {
                    const double2 x = *reinterpret_cast<const double2*>((const double*)xv + e);
                    if (OP == BV_COPY) v = x;
                    else if (OP == BV_JACOBI0) {
                        const double2 d = *reinterpret_cast<const double2*>((const double*)x2v + e);
                        v = make_double2(a * (x.x * d.x), a * (x.y * d.y));
                    } else {
                        v = *y;
                        v = make_double2(v.x + a * x.x, v.y + a * x.y);
                    }
                }
                *y = v;
            });
        }
    }
}

// Sum over the CTA of K values a thread (every thread calls it); the totals,
// added in FP64, are left in out[0 .. K) of shared memory.
template <int K> __device__ __forceinline__ void seg_reduce(const double (&v)[K], double (&red)[K][8], double* out)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < K; i++) {
        double t = v[i];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[i][warp] = t;
    }
    __syncthreads();
    if (threadIdx.x < K) {
        double t = 0;
        for (int w = 0; w < 8; w++) t += red[threadIdx.x][w];
        out[threadIdx.x] = t;
    }
    __syncthreads();
}

// A thread's running sum over segments: of FP32 partial sums the sum and what
// its rounding lost (Knuth's two-sum), added in FP64 when the problem changes.  So
// the error does not grow with the run, and the FP64 pipe stays out of the loop:
// 48 RVEs (edges 32 to 96) 92.7 ms, 92.4 with FP32 sums alone, 92.9 with an FP64
// addition a segment (against 91.6 in its run).
template <typename T> struct RunSum {
    double s = 0;
    __device__ __forceinline__ void add(T x) { s += x; }
    __device__ __forceinline__ double value() const { return s; }
};
template <> struct RunSum<float> {
    float hi = 0, lo = 0;
    __device__ __forceinline__ void add(float x)
    {
        const float t = hi + x, z = t - hi;
        lo += (hi - (t - z)) + (x - z);
        hi = t;
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Per-problem component sums (sums[3 prob + c]), or with subtract y -= sums /
// count over the nodes (not the padding), and the per-problem max |y| after it.
// A thread's sum over its elements of one segment is in T, the rest as RunSum.
template <typename T, int SUB>
__global__ void __launch_bounds__(256) k_seg_mean3(const BProb* __restrict__ probs, BSegList list,
                                                   const int* __restrict__ active, T* __restrict__ y,
                                                   double* __restrict__ sums, void* norm_slots)
{
    constexpr int VE = 16 / sizeof(T);
    typedef typename std::conditional<sizeof(T) == 4, float4, double2>::type V;
    typedef decltype(abs_bits(T())) Bits;
    __shared__ double red[1][8], tot[1];
    __shared__ T mean_s;
    int s0, s1;
    seg_range(list, s0, s1);
    RunSum<T> acc;
    T mean = 0;
    Bits m = 0;   // max |y| by its bits: order-preserving for |y|, NaN above all, and no FP64 compare
    int prob = -1, comp = -1;
    auto flush = [&]() {   // every thread of the CTA together
        if (prob < 0) return;
        if (SUB) {
            if (norm_slots) tile_max<T>(as_value(m), norm_slots, prob);
        } else {
            const double v[1] = {acc.value()};
            seg_reduce<1>(v, red, tot);
            if (threadIdx.x == 0) atomicAdd(&sums[prob * 3 + comp], tot[0]);
        }
        acc = RunSum<T>();
        m = 0;
    };
    for (int t = s0; t < s1; t++) {
        const BSeg s = list.d[t];
        if (active && !active[s.prob]) continue;
        if (s.prob != prob || s.comp != comp) {
            flush();
            prob = s.prob;
            comp = s.comp;
            if (SUB) {
                __syncthreads();
                if (threadIdx.x == 0) mean_s = (T)(sums[prob * 3 + comp] / (double)probs[prob].L.count());
                __syncthreads();
                mean = mean_s;
            }
        }
        const int P = s.pitch, nn0 = s.row;
        T part = 0;
        seg_each<VE>(s, [&](long long e) {
            V* p = reinterpret_cast<V*>(y + e);
            V v = *p;
            T* w = reinterpret_cast<T*>(&v);
            if (!SUB) {
#pragma unroll
                for (int i = 0; i < VE; i++) part += w[i];
                return;
            }
            const int i0 = P == nn0 ? 0 : (int)((s.first + (e - s.base)) % P);   // VE divides the pitch
#pragma unroll
            for (int i = 0; i < VE; i++)
                if (i0 + i < nn0) {
                    w[i] -= mean;
                    const Bits a = abs_bits(w[i]);
                    m = a > m ? a : m;
                }
            *p = v;
        });
        if (!SUB) acc.add(part);
    }
    flush();
}

// ---------------------------------------------------------------------------
// bottom solves: one CTA per problem (BiCGStab on the diagonally scaled
// system + smoothing, as the single-box k_bottom).  On a fully periodic box
// the Krylov residual and every operator application are projected to zero
// mean per component (the box is singular: rigid translations).
// ---------------------------------------------------------------------------
constexpr int BB_THREADS = 256;

template <typename R> __device__ __forceinline__ R bsum(R v, R* red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        R t = threadIdx.x < (BB_THREADS / 32) ? red[threadIdx.x] : (R)0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

template <typename R> __device__ __forceinline__ R bmax(R v, R* red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        const R w = __shfl_xor_sync(0xffffffffu, v, o);
        v = (w > v || w != w) ? w : v;
    }
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        R t = threadIdx.x < (BB_THREADS / 32) ? red[threadIdx.x] : (R)0;
        for (int o = 16; o > 0; o >>= 1) {
            const R w = __shfl_xor_sync(0xffffffffu, t, o);
            t = (w > t || w != w) ? w : t;
        }
        if (threadIdx.x == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

template <typename R, int SYM>
__device__ void bapply(const BProb& P, const BCTable& bc, int uniform, const R* ddw, const R* x, R* y)
{
    const LevelDesc& L = P.L;
    const Geo<R> g = geo_of<R>(P);
    const long long cnt = L.count();
    for (long long e = threadIdx.x; e < cnt; e += blockDim.x) {
        const int i = (int)(e % L.nn[0]), j = (int)((e / L.nn[0]) % L.nn[1]),
                  k = (int)(e / ((long long)L.nn[0] * L.nn[1]));
        BAcc<R> acc{x, ddw, L.S, make_nbr(L, i, j, k)};
        const int pos[3] = {i, j, k};
        int mn[3], mx[3];
        bool bnd = false;
        for (int d = 0; d < 3; d++) {
            mn[d] = !L.per[d] && pos[d] == 0;
            mx[d] = !L.per[d] && pos[d] == L.n[d];
            bnd = bnd || mn[d] || mx[d];
        }
        R f[3];
        if (bnd) boundary_row<R, SYM>(acc, g, bc, mn, mx, f);
        else interior_row<R, SYM>(acc, g, uniform != 0, f);
        for (int c = 0; c < 3; c++) y[c * L.S + acc.nb.base] = f[c];
    }
}

template <typename R> __device__ void bmean3(const LevelDesc& L, const R* v, R* red, R m[3])
{
    const long long cnt = L.count();
    R s0 = 0, s1 = 0, s2 = 0;
    for (long long e = threadIdx.x; e < cnt; e += blockDim.x) {
        const long long q = L.idx((int)(e % L.nn[0]), (int)((e / L.nn[0]) % L.nn[1]),
                                  (int)(e / ((long long)L.nn[0] * L.nn[1])));
        s0 += v[q];
        s1 += v[L.S + q];
        s2 += v[2 * L.S + q];
    }
    m[0] = bsum(s0, red) / (R)cnt;
    m[1] = bsum(s1, red) / (R)cnt;
    m[2] = bsum(s2, red) / (R)cnt;
}

#define BFOR(q)                                                                                        \
    for (long long e_ = threadIdx.x; e_ < cnt; e_ += blockDim.x)                                       \
        for (int c_ = 0, i_ = (int)(e_ % L.nn[0]), j_ = (int)((e_ / L.nn[0]) % L.nn[1]),                \
                 k_ = (int)(e_ / ((long long)L.nn[0] * L.nn[1]));                                      \
             c_ < 3; c_++)                                                                             \
            for (long long q = c_ * L.S + L.idx(i_, j_, k_), once_ = 0; once_ < 1; once_++)

template <typename T, int SYM>
__global__ void __launch_bounds__(BB_THREADS) k_batch_bottom(const BProb* __restrict__ probs, const int* __restrict__ plist,
                                                            const int* __restrict__ active, BCTable bc, int uniform,
                                                            const T* __restrict__ ddw_all,
                                                            const double* __restrict__ diag_all, T* __restrict__ cor_all,
                                                            const T* __restrict__ res_all, double* __restrict__ work_all,
                                                            int maxiter, double eps_rel_d, double eps_abs_d, int nub,
                                                            int nuf, double omega_d)
{
    typedef T R;   // arithmetic in the cycle's precision
    const R eps_rel = (R)eps_rel_d, eps_abs = (R)eps_abs_d, omega = (R)omega_d;
    __shared__ R red[33];
    const int pid = plist[blockIdx.x];
    if (active && !active[pid]) return;
    const BProb& P = probs[pid];
    const LevelDesc& L = P.L;
    const long long n3 = 3 * L.S, cnt = L.count();
    const R* ddw = ddw_all + P.co;
    const double* diag = diag_all + P.vo;
    T* cor = cor_all + P.vo;
    const T* res = res_all + P.vo;
    R* w = reinterpret_cast<R*>(work_all + P.wo);
    R *r = w, *rh = w + n3, *p = w + 2 * n3, *v = w + 3 * n3, *s = w + 4 * n3, *t = w + 5 * n3, *sol = w + 6 * n3,
           *b = w + 7 * n3;
    BFOR(q)
    {
        b[q] = (R)res[q];
        sol[q] = 0.0;
    }
    __syncthreads();
    const bool sing = L.singular();
    R mb[3] = {0, 0, 0};
    if (sing) bmean3(L, b, red, mb);
    R lm = 0;
    BFOR(q)
    {
        r[q] = (b[q] - mb[c_]) / (R)diag[q];
        rh[q] = r[q];
        const R a = fabs(r[q]);
        lm = (a > lm || a != a) ? a : lm;
    }
    R rnorm = bmax(lm, red);
    const R rnorm0 = rnorm;
    int ret = 0;
    R rho_1 = 0, alpha = 0, om = 0;
    if (!(rnorm0 == 0 || rnorm0 < eps_abs)) {
        for (int iter = 1; iter <= maxiter; iter++) {
            R acc = 0;
            BFOR(q) acc += rh[q] * r[q];
            const R rho = bsum(acc, red);
            if (rho == 0) { ret = 1; break; }
            if (iter == 1) {
                BFOR(q) p[q] = r[q];
            } else {
                const R beta = (rho / rho_1) * (alpha / om);
                BFOR(q) p[q] = r[q] + beta * (p[q] - om * v[q]);
            }
            __syncthreads();
            bapply<R, SYM>(P, bc, uniform, ddw, p, v);
            __syncthreads();
            R mv[3] = {0, 0, 0};
            if (sing) bmean3(L, v, red, mv);
            acc = 0;
            BFOR(q)
            {
                v[q] = (v[q] - mv[c_]) / (R)diag[q];
                acc += rh[q] * v[q];
            }
            const R rhTv = bsum(acc, red);
            if (rhTv != 0) alpha = rho / rhTv;
            else { ret = 2; break; }
            lm = 0;
            BFOR(q)
            {
                sol[q] += alpha * p[q];
                s[q] = r[q] - alpha * v[q];
                const R a = fabs(s[q]);
                lm = (a > lm || a != a) ? a : lm;
            }
            rnorm = bmax(lm, red);
            if (rnorm < eps_rel * rnorm0 || rnorm < eps_abs) break;
            bapply<R, SYM>(P, bc, uniform, ddw, s, t);
            __syncthreads();
            R mt[3] = {0, 0, 0};
            if (sing) bmean3(L, t, red, mt);
            R tt = 0, ts = 0;
            BFOR(q)
            {
                t[q] = (t[q] - mt[c_]) / (R)diag[q];
                tt += t[q] * t[q];
                ts += t[q] * s[q];
            }
            tt = bsum(tt, red);
            ts = bsum(ts, red);
            if (tt != 0) om = ts / tt;
            else { ret = 3; break; }
            lm = 0;
            BFOR(q)
            {
                sol[q] += om * s[q];
                r[q] = s[q] - om * t[q];
                const R a = fabs(r[q]);
                lm = (a > lm || a != a) ? a : lm;
            }
            rnorm = bmax(lm, red);
            if (rnorm < eps_rel * rnorm0 || rnorm < eps_abs) break;
            if (om == 0) { ret = 4; break; }
            rho_1 = rho;
        }
        if (ret == 0 && rnorm > eps_rel * rnorm0 && rnorm > eps_abs) ret = 8;
        if (ret != 0) {
            BFOR(q) sol[q] = 0.0;
        }
    }
    __syncthreads();
    const int nsm = 2 * ((ret == 0) ? nub : nuf);
    for (int sw = 0; sw < nsm; sw++) {
        bapply<R, SYM>(P, bc, uniform, ddw, sol, t);
        __syncthreads();
        BFOR(q)
        {
            const R Rx = t[q] - sol[q] * (R)diag[q];
            s[q] = ((R)1 - omega) * sol[q] + omega * (b[q] - Rx) / (R)diag[q];
        }
        __syncthreads();
        BFOR(q) sol[q] = s[q];
        __syncthreads();
    }
    BFOR(q) cor[q] = (T)sol[q];
}

// ---------------------------------------------------------------------------
// FP32 bottom solves on stored rows.  A coarsest level of up to ROWS_MAX
// unknowns keeps its operator's rows, 19 neighbours (no row reaches a corner)
// x 3 components an unknown, made once a model from the FP64 moduli
// (k_batch_rows); the solve runs one thread an unknown with its row and its
// Krylov entries in registers, the vector that is multiplied in shared memory
// and one barrier a reduction (dense_bottom_block).  k_batch_bottom evaluates
// the row from the moduli in every product, with all vectors in global memory
// and three barriers a sum: its time is a chain of latencies.  48 RVEs (8 to
// 125 coarsest nodes): 92 and 182 us a call before, 43 now; the solve 119 to
// 108 ms.
// Above ROWS_MAX unknowns the registers of a CTA do not hold a row for each; FP64 cycles keep
// k_batch_bottom: 57 FP64 multiply-adds an unknown cost more than the row.
// ---------------------------------------------------------------------------
constexpr int ROW_OFFS = 19;

__host__ __device__ constexpr int row_off(int o, int d)   // offset o of the 19 in direction d
{
    int n = 0;
    for (int k = -1; k <= 1; k++)
        for (int j = -1; j <= 1; j++)
            for (int i = -1; i <= 1; i++) {
                if (i && j && k) continue;
                if (n++ == o) return d == 0 ? i : (d == 1 ? j : k);
            }
    return 0;
}

// u = the unit vector of component p at offset (i, j, k) of the node, whatever
// node that is (on two cells a periodic node is its own two neighbours')
struct RowAcc {
    const double* __restrict__ c;
    long long S;
    Nbr nb;
    int p, i, j, k;
    __device__ __forceinline__ double u(int q, int di, int dj, int dk) const
    {
        return q == p && di == i && dj == j && dk == k ? 1.0 : 0.0;
    }
    __device__ __forceinline__ double C(int m, int di, int dj, int dk) const
    {
        return __ldg(c + m * S + nb.base + nb.o[0][di + 1] + nb.o[1][dj + 1] + nb.o[2][dk + 1]);
    }
};

// rows[P.ro + (3 o + p) nu + q]: the coefficient of component p at offset o in row q
template <int SYM>
__global__ void __launch_bounds__(256) k_batch_rows(const BProb* __restrict__ probs, const int* __restrict__ plist,
                                                    BCTable bc, const double* __restrict__ ddw,
                                                    float* __restrict__ rows)
{
    const BProb& P = probs[plist[blockIdx.x]];
    const LevelDesc& L = P.L;
    const int cnt = (int)L.count(), nu = 3 * cnt;
    const Geo<double> g = geo_of<double>(P);
    for (int t = threadIdx.x; t < cnt * ROW_OFFS * 3; t += blockDim.x) {
        const int e = t % cnt, col = t / cnt, o = col / 3;
        const int i = e % L.nn[0], j = (e / L.nn[0]) % L.nn[1], k = e / (L.nn[0] * L.nn[1]);
        const RowAcc acc{ddw + P.co, L.S, make_nbr(L, i, j, k), col % 3, row_off(o, 0), row_off(o, 1), row_off(o, 2)};
        const int pos[3] = {i, j, k};
        int mn[3], mx[3];
        bool bnd = false;
        for (int d = 0; d < 3; d++) {
            mn[d] = !L.per[d] && pos[d] == 0;
            mx[d] = !L.per[d] && pos[d] == L.n[d];
            bnd = bnd || mn[d] || mx[d];
        }
        double f[3];
        if (bnd) boundary_row<double, SYM>(acc, g, bc, mn, mx, f);
        else interior_row<double, SYM>(acc, g, false, f);
        for (int c = 0; c < 3; c++) rows[P.ro + (long long)col * nu + c * cnt + e] = (float)f[c];
    }
}

// One thread's row, its coefficients in registers.
struct StoredRow {
    const float* __restrict__ xs;
    int cnt;
    int ex[3], ey[3], ez[3];   // places of the neighbours in a component, by direction
    float w[3 * ROW_OFFS];
    __device__ __forceinline__ float operator()() const
    {
        float y[3] = {0, 0, 0};
#pragma unroll
        for (int o = 0; o < ROW_OFFS; o++) {
            const int at = ex[row_off(o, 0) + 1] + ey[row_off(o, 1) + 1] + ez[row_off(o, 2) + 1];
#pragma unroll
            for (int p = 0; p < 3; p++) y[p] += w[3 * o + p] * xs[p * cnt + at];
        }
        return (y[0] + y[1]) + y[2];
    }
};

__global__ void __launch_bounds__(ROWS_MAX) k_batch_bottom_rows(const BProb* __restrict__ probs,
                                                                const int* __restrict__ plist,
                                                                const int* __restrict__ active,
                                                                const float* __restrict__ rows,
                                                                const double* __restrict__ diag_all,
                                                                float* __restrict__ cor_all,
                                                                const float* __restrict__ res_all, int maxiter,
                                                                double eps_rel, double eps_abs, int nub, int nuf,
                                                                double omega)
{
    __shared__ float xs[ROWS_MAX], red[2 * 3 * 32];
    const int pid = plist[blockIdx.x];
    if (active && !active[pid]) return;
    const BProb& P = probs[pid];
    const LevelDesc& L = P.L;
    StoredRow row;
    row.cnt = (int)L.count();
    row.xs = xs;
    const int nu = 3 * row.cnt;
    const int q = min((int)threadIdx.x, nu - 1), e = q % row.cnt;   // a thread past the unknowns multiplies nothing
#pragma unroll
    for (int m = 0; m < 3 * ROW_OFFS; m++) row.w[m] = __ldg(rows + P.ro + (long long)m * nu + q);
    const int pos[3] = {e % L.nn[0], (e / L.nn[0]) % L.nn[1], e / (L.nn[0] * L.nn[1])};
    for (int s = 0; s < 3; s++) {
        int at[3];
        for (int d = 0; d < 3; d++) {
            at[d] = pos[d] + s - 1;
            if (L.per[d]) at[d] = at[d] < 0 ? L.n[d] - 1 : (at[d] >= L.n[d] ? 0 : at[d]);
            else at[d] = min(max(at[d], 0), L.n[d]);   // past a face the coefficient is zero
        }
        row.ex[s] = at[0];
        row.ey[s] = L.nn[0] * at[1];
        row.ez[s] = L.nn[0] * L.nn[1] * at[2];
    }
    dense_bottom_block<float, float>(L, row, xs, red, diag_all + P.vo, cor_all + P.vo, res_all + P.vo, maxiter, eps_rel,
                                     eps_abs, nub, nuf, omega, nullptr);
}

// Faces a node lies on: the directions that are not periodic.
__device__ __forceinline__ bool node_faces(const LevelDesc& L, int i, int j, int k, int mn[3], int mx[3])
{
    const int pos[3] = {i, j, k};
    bool bnd = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        mn[d] = !L.per[d] && pos[d] == 0;
        mx[d] = !L.per[d] && pos[d] == L.n[d];
        bnd = bnd || mn[d] || mx[d];
    }
    return bnd;
}

// rhs = b - div(C : (0 - F0)) with a uniform eigenstrain F0 per problem: the
// Newton right-hand side at u = 0 of an affine model (Newton.H:144-231,
// Model/Solid/Affine/Isotropic.H:42-45).  On the faces of a box that is not
// periodic in every direction the boundary condition's value less its row of the
// same stress (a node there has no neighbour on one side); b is 0 elsewhere.
template <int SYM>
__global__ void __launch_bounds__(256) k_batch_rhs(const BProb* __restrict__ probs, const BTile* __restrict__ tiles,
                                                   int ntiles, BCTable bc, const double* __restrict__ ddw,
                                                   const double* __restrict__ F0, double* __restrict__ rhs)
{
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const BTile tl = tiles[t];
        const BProb& P = probs[tl.prob];
        const LevelDesc& L = P.L;
        int i, j, k;
        if (!tile_node<32, 4, 2>(tl, L, i, j, k)) continue;
        const Nbr nb = make_nbr(L, i, j, k);
        double E[3][3], b[3] = {0, 0, 0}, ret[3] = {0, 0, 0};
        for (int a = 0; a < 3; a++)
            for (int c = 0; c < 3; c++) E[a][c] = 0.0 - F0[tl.prob * 9 + a * 3 + c];
        int mn[3], mx[3];
        if (node_faces(L, i, j, k, mn, mx)) {
            double c[NCoef<SYM>::value], S[3][3], nrm[3];
            const double zero[3] = {0, 0, 0}, G[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            for (int m = 0; m < NCoef<SYM>::value; m++) c[m] = ddw[P.co + m * L.S + nb.base];
            c_mul_mat<double, SYM>(c, E, S);
            const int face = face_of(mn, mx, nrm);
            bc_set<double>(bc.type[face], zero, G, S, nrm, ret);
            for (int r = 0; r < 3; r++) b[r] = bc.val[face][r];
        } else {
            for (int d = 0; d < 3; d++) {
                // (C+ - C-) : E, the difference of the moduli first
                double dc[NCoef<SYM>::value], D[3][3];
                for (int m = 0; m < NCoef<SYM>::value; m++)
                    dc[m] = ddw[P.co + m * L.S + nb.base + nb.o[d][2]] - ddw[P.co + m * L.S + nb.base + nb.o[d][0]];
                c_mul_mat<double, SYM>(dc, E, D);
                for (int r = 0; r < 3; r++) ret[r] += D[r][d] * P.h1[d];
            }
        }
        for (int r = 0; r < 3; r++) rhs[P.vo + r * L.S + nb.base] = b[r] - ret[r];
    }
}

// Per-problem sums of sigma = C : (grad u - F0) over the stored nodes
// (central differences, one-sided on faces), for the homogenized stress.  A
// CTA takes a contiguous part of the list and a thread keeps its six sums while
// the problem stays the same: reducing nine a tile by shuffles was most of its
// FP64 work (17.3 M nodes 2.8 ms before, 1.2 now).
template <int SYM>
__global__ void __launch_bounds__(256) k_batch_mean_stress(const BProb* __restrict__ probs,
                                                           const BTile* __restrict__ tiles, int ntiles,
                                                           const double* __restrict__ ddw,
                                                           const double* __restrict__ F0,
                                                           const double* __restrict__ u, double* __restrict__ sums)
{
    __shared__ double red[6][8], tot[6];
    double acc[6] = {0, 0, 0, 0, 0, 0};   // xx, xy, xz, yy, yz, zz
    int prob = -1;
    auto flush = [&]() {   // every thread of the CTA together
        if (prob < 0) return;
        seg_reduce<6>(acc, red, tot);
        if (threadIdx.x < 9) {
            const int r = threadIdx.x / 3, c = threadIdx.x % 3, lo = min(r, c), hi = max(r, c);
            atomicAdd(&sums[prob * 9 + threadIdx.x], tot[lo == 0 ? hi : (lo == 1 ? 2 + hi : 5)]);
        }
        for (int q = 0; q < 6; q++) acc[q] = 0;
    };
    const int t0 = (int)((long long)ntiles * blockIdx.x / gridDim.x);
    const int t1 = (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);
    for (int t = t0; t < t1; t++) {
        const BTile tl = tiles[t];
        if (tl.prob != prob) {
            flush();
            prob = tl.prob;
        }
        const BProb& P = probs[tl.prob];
        const LevelDesc& L = P.L;
        int i, j, k;
        if (!tile_node<32, 4, 2>(tl, L, i, j, k)) continue;
        const Nbr nb = make_nbr(L, i, j, k);
        double G[3][3], S[3][3], c[NCoef<SYM>::value];
        int mn[3], mx[3];
        node_faces(L, i, j, k, mn, mx);
        for (int d = 0; d < 3; d++) {
            const long long hi = mx[d] ? 0 : nb.o[d][2], lo = mn[d] ? 0 : nb.o[d][0];
            const double h = mn[d] || mx[d] ? P.i1[d] : P.h1[d];
            for (int p = 0; p < 3; p++)
                G[p][d] = (u[P.vo + p * L.S + nb.base + hi] - u[P.vo + p * L.S + nb.base + lo]) * h -
                          F0[tl.prob * 9 + p * 3 + d];
        }
        for (int m = 0; m < NCoef<SYM>::value; m++) c[m] = ddw[P.co + m * L.S + nb.base];
        c_mul_mat<double, SYM>(c, G, S);
        acc[0] += S[0][0];
        acc[1] += S[0][1];
        acc[2] += S[0][2];
        acc[3] += S[1][1];
        acc[4] += S[1][2];
        acc[5] += S[2][2];
    }
    flush();
}

template <typename T>
void launch_batch_mean3(cudaStream_t st, int grid, const BProb* probs, BSegList segs, const int* active, T* y,
                        double* sums, int subtract, void* norm_slots)
{
    grid = std::min(grid, segs.max);
    if (grid < 1) return;
    if (subtract) k_seg_mean3<T, 1><<<grid, 256, 0, st>>>(probs, segs, active, y, sums, norm_slots);
    else k_seg_mean3<T, 0><<<grid, 256, 0, st>>>(probs, segs, active, y, sums, norm_slots);
    count_launch();
}
template void launch_batch_mean3<double>(cudaStream_t, int, const BProb*, BSegList, const int*, double*, double*, int,
                                         void*);
template void launch_batch_mean3<float>(cudaStream_t, int, const BProb*, BSegList, const int*, float*, double*, int,
                                        void*);

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename T, int SYM, int MODE>
static void bst_shape(cudaStream_t st, int shape, int grid, const BProb* probs, const BTile* tiles, int ntiles,
                      const int* active, const BCTable& bc, bool uniform, const T* ddw, const T* x, const T* b,
                      const T* dinv, T* out, T omega, void* norm)
{
#define L_(BX, BY, BZ)                                                                                      \
    grid = fit_grid((const void*)k_batch_stencil<T, SYM, MODE, BX, BY, BZ>, grid, st);                           \
    k_batch_stencil<T, SYM, MODE, BX, BY, BZ><<<grid, 256, 0, st>>>(probs, tiles, ntiles, active, bc, uniform ? 1 : 0, \
                                                                     ddw, x, b, dinv, out, omega, norm)
    // the marching shape is only chosen for isotropic fully periodic batches
    // (batch_shape_ok)
    if constexpr (SYM == SYM_ISO) {
#define M_(BX)                                                                                                       \
    do {                                                                                                             \
        grid = fit_grid((const void*)k_batch_march<T, MODE, BX>, grid, st);                                          \
        k_batch_march<T, MODE, BX><<<grid, 256, 0, st>>>(probs, tiles, ntiles, active, uniform ? 1 : 0, ddw, x, b,   \
                                                         dinv, out, omega, norm);                                    \
        count_launch();                                                                                              \
        return;                                                                                                      \
    } while (0)
        if (shape == kMarchShape) M_(32);
        if (shape == kMarchShape16) M_(16);
#undef M_
    }
    switch (shape) {
    case 0: L_(32, 4, 2); break;
    case 1: L_(32, 8, 1); break;
    case 2: L_(16, 8, 2); break;
    case 3: L_(8, 8, 4); break;
    default: L_(64, 4, 1); break;
    }
#undef L_
    count_launch();
}

template <typename T>
void launch_batch_stencil(cudaStream_t st, int sym, int mode, int shape, int grid, const BProb* probs,
                          const BTile* tiles, int ntiles, const int* active, const BCTable& bc, bool uniform,
                          const T* ddw, const T* x, const T* b, const T* dinv, T* out, T omega, void* norm_slots)
{
#define D_(S, M) bst_shape<T, S, M>(st, shape, grid, probs, tiles, ntiles, active, bc, uniform, ddw, x, b, dinv, out, omega, norm_slots)
    if (sym == SYM_ISO) {
        if (mode == MODE_APPLY) D_(SYM_ISO, MODE_APPLY);
        else if (mode == MODE_RESID) D_(SYM_ISO, MODE_RESID);
        else D_(SYM_ISO, MODE_JACOBI);
    } else {
        if (mode == MODE_APPLY) D_(SYM_MM, MODE_APPLY);
        else if (mode == MODE_RESID) D_(SYM_MM, MODE_RESID);
        else D_(SYM_MM, MODE_JACOBI);
    }
#undef D_
}

template <typename T>
void launch_batch_transfer(cudaStream_t st, int restrict_not_interp, bool assign, int grid, const BProb* pf,
                           const BProb* pc, const BTile* tiles, int ntiles, const int* active, const T* src, T* dst)
{
    grid = fit_grid((const void*)k_batch_transfer<T>, grid, st);
    k_batch_transfer<T><<<grid, 256, 0, st>>>(restrict_not_interp, assign ? 1 : 0, pf, pc, tiles, ntiles, active, src,
                                              dst);
    count_launch();
}

void launch_batch_avg_ddw(cudaStream_t st, int grid, const BProb* pf, const BProb* pc, const BTile* tiles, int ntiles,
                          const double* fine, double* crse, int ncoef)
{
    k_batch_avg_ddw<<<grid, 256, 0, st>>>(pf, pc, tiles, ntiles, fine, crse, ncoef);
    count_launch();
}

void launch_batch_diag(cudaStream_t st, int sym, int grid, const BProb* probs, const BTile* tiles, int ntiles,
                       const BCTable& bc, const double* ddw, double* diag, double* dinv64, float* dinv32)
{
    if (sym == SYM_ISO) k_batch_diag<SYM_ISO><<<grid, 256, 0, st>>>(probs, tiles, ntiles, bc, ddw, diag, dinv64, dinv32);
    else k_batch_diag<SYM_MM><<<grid, 256, 0, st>>>(probs, tiles, ntiles, bc, ddw, diag, dinv64, dinv32);
    count_launch();
}

void launch_batch_vec(cudaStream_t st, int op, int grid, BSegList segs, const int* active, void* y, const void* x,
                      double a, const double* scale, int fp32, const void* x2)
{
    grid = std::min(grid, segs.max);
    if (grid < 1) return;
#define V_(OP)                                                                                          \
    case OP:                                                                                            \
        if (fp32) k_seg_vec<OP, float><<<grid, 256, 0, st>>>(segs, active, y, x, a, scale, x2);         \
        else k_seg_vec<OP, double><<<grid, 256, 0, st>>>(segs, active, y, x, a, scale, x2);             \
        break;
    switch (op) {
        V_(BV_ZERO) V_(BV_COPY) V_(BV_AXPY) V_(BV_SCALE_TO32) V_(BV_ACC_FROM32) V_(BV_JACOBI0)
    }
#undef V_
    count_launch();
}

// ---------------------------------------------------------------------------
// Per-problem GCR over the batched FP32 cycle (the single-box inner_gcr32 on
// every problem at once), over segments.  Inner products are weighted by d^2
// (d = 1/diag); a thread sums its 16 elements of a segment in FP32, segments by
// RunSum, threads in FP64.
// Directions are kept as they come, with ww_i = <w_i, w_i> beside them
// (dots[i][2 prob]), so the step writes only the solution and the residual.
// ---------------------------------------------------------------------------

// out[prob * stride + i] += sum of x v_i d^2, i < K
template <int K>
__global__ void __launch_bounds__(256) k_seg_multidot(BSegList list, const int* __restrict__ active,
                                                      const float* __restrict__ x, GcrVecs V,
                                                      const float* __restrict__ d, double* __restrict__ out,
                                                      int stride)
{
    __shared__ double red[K][8], tot[K];
    int s0, s1;
    seg_range(list, s0, s1);
    RunSum<float> sum[K];
    int prob = -1;
    auto flush = [&]() {
        if (prob < 0) return;
        double v[K];
#pragma unroll
        for (int i = 0; i < K; i++) {
            v[i] = sum[i].value();
            sum[i] = RunSum<float>();
        }
        seg_reduce<K>(v, red, tot);
        if (threadIdx.x < K) atomicAdd(out + (long long)prob * stride + threadIdx.x, tot[threadIdx.x]);
    };
    for (int t = s0; t < s1; t++) {
        const BSeg s = list.d[t];
        if (active && !active[s.prob]) continue;
        if (s.prob != prob) {
            flush();
            prob = s.prob;
        }
        float acc[K];
#pragma unroll
        for (int i = 0; i < K; i++) acc[i] = 0;
        seg_each<4>(s, [&](long long e) {
            const float4 dd = __ldg(reinterpret_cast<const float4*>(d + e));
            const float4 xx = __ldg(reinterpret_cast<const float4*>(x + e));
            const float4 w = make_float4(xx.x * dd.x * dd.x, xx.y * dd.y * dd.y, xx.z * dd.z * dd.z,
                                         xx.w * dd.w * dd.w);
#pragma unroll
            for (int i = 0; i < K; i++) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(V.v[i] + e));
                acc[i] += (w.x * v.x + w.y * v.y) + (w.z * v.z + w.w * v.w);
            }
        });
#pragma unroll
        for (int i = 0; i < K; i++) sum[i].add(acc[i]);
    }
    flush();
}

// w -= sum_i (beta_i / ww_i) W_i and z likewise (i < K), and the new direction's
// <w, w> and <w, r> into dots[2 prob], dots[2 prob + 1].  beta_i at beta[prob *
// stride + i], ww_i at all[(i * np + prob) * 2].
template <int K>
__global__ void __launch_bounds__(256) k_seg_gcr_orth(BSegList list, const int* __restrict__ active,
                                                      const double* __restrict__ beta, int stride,
                                                      const double* __restrict__ all, int np, GcrVecs W, GcrVecs Z,
                                                      float* __restrict__ w, float* __restrict__ z,
                                                      const float* __restrict__ r, const float* __restrict__ d,
                                                      double* __restrict__ dots)
{
    __shared__ double red[2][8], tot[2];
    __shared__ float coef[K > 0 ? K : 1];
    int s0, s1;
    seg_range(list, s0, s1);
    RunSum<float> sww, swr;
    float b[K > 0 ? K : 1];
    int prob = -1;
    auto flush = [&]() {
        if (prob < 0) return;
        const double v[2] = {sww.value(), swr.value()};
        seg_reduce<2>(v, red, tot);
        if (threadIdx.x < 2) atomicAdd(dots + 2 * (long long)prob + threadIdx.x, tot[threadIdx.x]);
        sww = swr = RunSum<float>();
    };
    for (int t = s0; t < s1; t++) {
        const BSeg s = list.d[t];
        if (active && !active[s.prob]) continue;
        if (s.prob != prob) {
            flush();
            prob = s.prob;
            if (K > 0) {
                __syncthreads();
                if (threadIdx.x < K) {
                    const double n = all[((long long)threadIdx.x * np + prob) * 2];
                    coef[threadIdx.x] = n > 0 ? (float)(beta[(long long)prob * stride + threadIdx.x] / n) : 0.0f;
                }
                __syncthreads();
#pragma unroll
                for (int i = 0; i < K; i++) b[i] = coef[i];
            }
        }
        float ww = 0, wr = 0;
        seg_each<4>(s, [&](long long e) {
            float4 tw = *reinterpret_cast<const float4*>(w + e);
            if (K > 0) {
                float4 tz = *reinterpret_cast<const float4*>(z + e);
#pragma unroll
                for (int i = 0; i < K; i++) {
                    const float4 wi = __ldg(reinterpret_cast<const float4*>(W.v[i] + e));
                    const float4 zi = __ldg(reinterpret_cast<const float4*>(Z.v[i] + e));
                    tw = make_float4(tw.x - b[i] * wi.x, tw.y - b[i] * wi.y, tw.z - b[i] * wi.z, tw.w - b[i] * wi.w);
                    tz = make_float4(tz.x - b[i] * zi.x, tz.y - b[i] * zi.y, tz.z - b[i] * zi.z, tz.w - b[i] * zi.w);
                }
                *reinterpret_cast<float4*>(w + e) = tw;
                *reinterpret_cast<float4*>(z + e) = tz;
            }
            const float4 dd = __ldg(reinterpret_cast<const float4*>(d + e));
            const float4 rr = __ldg(reinterpret_cast<const float4*>(r + e));
            const float4 u = make_float4(tw.x * dd.x * dd.x, tw.y * dd.y * dd.y, tw.z * dd.z * dd.z,
                                         tw.w * dd.w * dd.w);
            ww += (u.x * tw.x + u.y * tw.y) + (u.z * tw.z + u.w * tw.w);
            wr += (u.x * rr.x + u.y * rr.y) + (u.z * rr.z + u.w * rr.w);
        });
        sww.add(ww);
        swr.add(wr);
    }
    flush();
}

// with ww = dots[2p], wr = dots[2p+1]: c += (wr / ww) z, r -= (wr / ww) w, max |r|
// per problem -> norm_slots
__global__ void __launch_bounds__(256) k_seg_gcr_step(BSegList list, const int* __restrict__ active,
                                                      const double* __restrict__ dots, const float* __restrict__ w,
                                                      const float* __restrict__ z, float* __restrict__ c,
                                                      float* __restrict__ r, void* norm_slots)
{
    __shared__ float a_s;
    int s0, s1;
    seg_range(list, s0, s1);
    float nrm = 0, a = 0;
    int prob = -1;
    for (int t = s0; t < s1; t++) {
        const BSeg s = list.d[t];
        if (active && !active[s.prob]) continue;
        if (s.prob != prob) {
            if (prob >= 0) tile_max<float>(nrm, norm_slots, prob);
            nrm = 0;
            prob = s.prob;
            __syncthreads();
            if (threadIdx.x == 0) {
                const double ww = dots[2 * prob];
                a_s = ww > 0 ? (float)(dots[2 * prob + 1] / ww) : 0.0f;
            }
            __syncthreads();
            a = a_s;
        }
        seg_each<4>(s, [&](long long e) {
            const float4 ww = __ldg(reinterpret_cast<const float4*>(w + e));
            const float4 zz = __ldg(reinterpret_cast<const float4*>(z + e));
            float4 cc = *reinterpret_cast<const float4*>(c + e), rr = *reinterpret_cast<const float4*>(r + e);
            cc = make_float4(cc.x + a * zz.x, cc.y + a * zz.y, cc.z + a * zz.z, cc.w + a * zz.w);
            rr = make_float4(rr.x - a * ww.x, rr.y - a * ww.y, rr.z - a * ww.z, rr.w - a * ww.w);
            *reinterpret_cast<float4*>(c + e) = cc;
            *reinterpret_cast<float4*>(r + e) = rr;
            const float v[4] = {fabsf(rr.x), fabsf(rr.y), fabsf(rr.z), fabsf(rr.w)};
#pragma unroll
            for (int i = 0; i < 4; i++) nrm = (v[i] > nrm || v[i] != v[i]) ? v[i] : nrm;
        });
    }
    if (prob >= 0) tile_max<float>(nrm, norm_slots, prob);
}

void launch_batch_multidot(cudaStream_t st, int grid, BSegList segs, const int* active, int k, const float* x,
                           const GcrVecs& V, const float* d, double* out, int stride)
{
    grid = std::min(grid, segs.max);
    if (grid < 1) return;
    switch (k) {
#define K_(K) case K: k_seg_multidot<K><<<grid, 256, 0, st>>>(segs, active, x, V, d, out, stride); break;
        K_(1) K_(2) K_(3) K_(4) K_(5) K_(6) K_(7) K_(8) K_(9) K_(10) K_(11) K_(12) K_(13) K_(14) K_(15)
#undef K_
    default: return;
    }
    count_launch();
}

void launch_batch_gcr_orth(cudaStream_t st, int grid, BSegList segs, const int* active, int k, const double* beta,
                           int stride, const double* all, int np, const GcrVecs& W, const GcrVecs& Z, float* w,
                           float* z, const float* r, const float* d, double* dots)
{
    grid = std::min(grid, segs.max);
    if (grid < 1) return;
    switch (k) {
#define K_(K)                                                                                                         \
    case K:                                                                                                           \
        k_seg_gcr_orth<K><<<grid, 256, 0, st>>>(segs, active, beta, stride, all, np, W, Z, w, z, r, d, dots);          \
        break;
        K_(0) K_(1) K_(2) K_(3) K_(4) K_(5) K_(6) K_(7) K_(8) K_(9) K_(10) K_(11) K_(12) K_(13) K_(14) K_(15)
#undef K_
    default: return;
    }
    count_launch();
}

void launch_batch_gcr_step(cudaStream_t st, int grid, BSegList segs, const int* active, const double* dots,
                           const float* w, const float* z, float* c, float* r, void* norm_slots)
{
    grid = std::min(grid, segs.max);
    if (grid < 1) return;
    k_seg_gcr_step<<<grid, 256, 0, st>>>(segs, active, dots, w, z, c, r, norm_slots);
    count_launch();
}

void launch_batch_bottom(cudaStream_t st, int sym, int fp32, const BProb* probs, const int* plist, int np,
                         const int* active, const BCTable& bc, bool uniform, const void* ddw, const double* diag,
                         void* cor, const void* res, double* work, int maxiter, double tol_rel, double tol_abs, int nub,
                         int nuf, double omega)
{
    if (np <= 0) return;
#define B_(T, S)                                                                                                     \
    k_batch_bottom<T, S><<<np, BB_THREADS, 0, st>>>(probs, plist, active, bc, uniform ? 1 : 0, (const T*)ddw, diag,  \
                                                    (T*)cor,                                                           \
                                                    (const T*)res, work, maxiter, tol_rel, tol_abs, nub, nuf, omega)
    if (fp32) {
        if (sym == SYM_ISO) B_(float, SYM_ISO);
        else B_(float, SYM_MM);
    } else {
        if (sym == SYM_ISO) B_(double, SYM_ISO);
        else B_(double, SYM_MM);
    }
#undef B_
    count_launch();
}

void launch_batch_rows(cudaStream_t st, int sym, const BProb* probs, const int* plist, int np, const BCTable& bc,
                       const double* ddw64, float* rows)
{
    if (np <= 0) return;
    if (sym == SYM_ISO) k_batch_rows<SYM_ISO><<<np, 256, 0, st>>>(probs, plist, bc, ddw64, rows);
    else k_batch_rows<SYM_MM><<<np, 256, 0, st>>>(probs, plist, bc, ddw64, rows);
    count_launch();
}

void launch_batch_bottom_rows(cudaStream_t st, const BProb* probs, const int* plist, int np, int max_unknowns,
                              const int* active, const float* rows, const double* diag, float* cor, const float* res,
                              int maxiter, double tol_rel, double tol_abs, int nub, int nuf, double omega)
{
    if (np <= 0) return;
    k_batch_bottom_rows<<<np, (max_unknowns + 31) / 32 * 32, 0, st>>>(probs, plist, active, rows, diag, cor, res,
                                                                     maxiter, tol_rel, tol_abs, nub, nuf, omega);
    count_launch();
}

void launch_batch_rhs(cudaStream_t st, int sym, int grid, const BProb* probs, const BTile* tiles, int ntiles,
                      const BCTable& bc, const double* ddw, const double* F0, double* rhs)
{
    if (sym == SYM_ISO) k_batch_rhs<SYM_ISO><<<grid, 256, 0, st>>>(probs, tiles, ntiles, bc, ddw, F0, rhs);
    else k_batch_rhs<SYM_MM><<<grid, 256, 0, st>>>(probs, tiles, ntiles, bc, ddw, F0, rhs);
    count_launch();
}

void launch_batch_mean_stress(cudaStream_t st, int sym, int grid, const BProb* probs, const BTile* tiles, int ntiles,
                              const double* ddw, const double* F0, const double* u, double* sums)
{
    if (sym == SYM_ISO) k_batch_mean_stress<SYM_ISO><<<grid, 256, 0, st>>>(probs, tiles, ntiles, ddw, F0, u, sums);
    else k_batch_mean_stress<SYM_MM><<<grid, 256, 0, st>>>(probs, tiles, ntiles, ddw, F0, u, sums);
    count_launch();
}

template void launch_batch_stencil<double>(cudaStream_t, int, int, int, int, const BProb*, const BTile*, int,
                                           const int*, const BCTable&, bool, const double*, const double*,
                                           const double*, const double*, double*, double, void*);
template void launch_batch_stencil<float>(cudaStream_t, int, int, int, int, const BProb*, const BTile*, int,
                                          const int*, const BCTable&, bool, const float*, const float*, const float*,
                                          const float*, float*, float, void*);
template void launch_batch_transfer<double>(cudaStream_t, int, bool, int, const BProb*, const BProb*, const BTile*,
                                            int, const int*, const double*, double*);
template void launch_batch_transfer<float>(cudaStream_t, int, bool, int, const BProb*, const BProb*, const BTile*, int,
                                           const int*, const float*, float*);

}  // namespace agb
