// kernels_wgrad_tc.cu -- weight and bias gradients of the learned
// correction's 3x3x3 convolutions; the weight gradient on the
// fifth-generation tensor cores.
//
//   dw[tap][co][ci] += sum_v dy[v][co] x[v + off(tap)][ci]   (FP32, zero padding)
//
// Voxels are the contraction.  Fields are channels-last, so both operands are
// MN-major: 8 channels of a voxel are 16 bytes, and eight voxels of them are
// one core matrix.  A batch is T lines (y .. y+T-1 at one z) of dy and the T+2
// lines around them of x at z + dz; lines and 8-channel groups lie one after
// the other in shared memory at one pitch, so the M side of one MMA takes, from
// line y-1 of x on, the lines y-1, y and y+1 (all three dy taps) of a block of
// CB input channels, the N side the line y of CO output channels, and the
// three dx taps are three MMAs whose M operand starts one voxel (16 bytes)
// further.  A line that ends inside its last 16 voxels is filled up with zeros:
// behind it for the taps 0 and +1, before it for the tap -1 (both operands start
// `pad` voxels earlier), so that dy's zeros meet zeros of x and a NaN or infinity
// in x reaches the taps that use it only.  Rows of the 128 beyond 3 CB are whatever follows in shared memory;
// they are never read back.  CTAs are (dz, channel blocks, run of batches); the
// accumulators are read out, added in FP32 registers and started again after
// every batch: tensor cores do not round their FP32 sums to nearest, and a
// batch is at most T KX / 16 steps long (20 on a 65-voxel line), which keeps
// the error against 64 bits below the scalar kernel's (1.8e-7 relative against
// 3.0e-7 at 65^3 voxels, 32 x 32 channels).
//
// Roles: warps 0-3 read the accumulators, warp 4 issues the MMAs, the others
// copy (16-byte cp.async, zeros outside the grid; a TMA box of 8 channels moves
// 16 bytes a request); two to four stages of shared memory, two sets of
// accumulators.  Every wait is bounded (about 1 s); one that runs out sets the
// error flag, and the CTA stops, waits (bounded) for what it issued, frees its
// tensor memory and adds nothing.
//
// What bounds it: issuing the copies (33 a thread and batch of four 80-voxel
// lines, 2500 clocks) beside the MMAs (60 a batch, 2900 clocks).  65^3 voxels, 32
// x 32 channels: 63.5 us (60.7 with the zeros of all taps behind the line: the
// shifted dy operand of the tap -1 starts inside a core matrix); 64^3, which has
// none, 51; with TMA boxes and MMAs issued from one thread's branch 82 us at 65^3;
// the scalar kernel below 3080 us.  The bias gradient reads 8 channels a thread:
// 7 against 21 us.
//
// The scalar kernel stays for slices and pointers that are not 16-byte aligned.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "agb.h"
#include "agb_internal.h"
#include "tma.cuh"
#include "umma.cuh"

namespace agb {
namespace {

// threads that copy: as many as the registers of the accumulators leave room for
template <int CO> struct WtThreads {
    static constexpr int copy = CO == 16 ? 224 : 96;
    static constexpr int all = 160 + copy;
};
constexpr int WT_M = 128;

struct WtArgs {
    int nx, ny, nz;
    int kx, ntx;               // voxels of a line tile (multiple of 16, 128 at most), tiles of a line
    const __nv_bfloat16 *x, *dy;   // first channel of each slice
    int x_cs, dy_cs;
    int cin, cout;
    int T, chunks, stages;     // lines of a batch, CTAs along the batches, stages of shared memory (2 to 4)
    int lead;                  // voxels of zeros before each line: 16 where lines end inside their last 16
    float* dw;
    int* err;
};

// Bytes from one 8-channel group of a line to the next.  The copying threads
// write the groups of a voxel side by side; the odd multiples of 32 (16 for 8
// groups) bytes put them in different banks.
__host__ __device__ inline int x_pitch(int kx, int lead) { return (lead + kx + 2) * 16; }
__host__ __device__ inline int dy_pitch(int kx, int lead, int co) { return (lead + kx) * 16 + (co == 64 ? 16 : 32); }
__host__ __device__ inline int stage_bytes(int kx, int lead, int cb, int co, int T)
{
    return (T + 2) * (cb / 8) * x_pitch(kx, lead) + T * (co / 8) * dy_pitch(kx, lead, co);
}
// the 16 M groups of the last line reach past the x lines: room behind the stages
__host__ __device__ inline int smem_bytes(int kx, int lead, int cb, int co, int T, int stages)
{
    return 128 + stages * stage_bytes(kx, lead, cb, co, T) + 16 * x_pitch(kx, lead) + 128;
}

// `lines` lines from (x0, y0, z) of GROUPS x 8 channels into dst, `len` voxels each
template <int GROUPS, int COPY>
__device__ __forceinline__ void copy_lines(uint32_t dst, int pitch, int lines, int len, const __nv_bfloat16* base,
                                           int cs, int x0, int y0, int z, const WtArgs& a, int t)
{
    constexpr int VS = COPY / GROUPS;   // a thread keeps its group and takes every VS-th voxel
    const int g = t % GROUPS, v0 = t / GROUPS;
    for (int l = 0; l < lines; l++) {
        const int y = y0 + l;
        const bool row = y >= 0 && y < a.ny;
        const __nv_bfloat16* p = base + (((long long)z * a.ny + y) * a.nx + x0 + v0) * cs + 8 * g;
        uint32_t d = dst + (l * GROUPS + g) * pitch + v0 * 16;
        int x = x0 + v0;
#pragma unroll 4
        for (int v = v0; v < len; v += VS) {
            const bool in = row && (unsigned)x < (unsigned)a.nx;
            copy16(d, in ? p : base, in);
            p += VS * cs;
            d += VS * 16;
            x += VS;
        }
    }
}

template <int CB, int CO>
__global__ void __launch_bounds__(WtThreads<CO>::all, 1) k_wgrad_tc(WtArgs a)
{
    constexpr int COPY = WtThreads<CO>::copy;
    constexpr int COLS = 3 * CO;   // columns of one set of accumulators
    constexpr int TMEM = 2 * COLS <= 128 ? 128 : (2 * COLS <= 256 ? 256 : 512);
    constexpr uint32_t idesc = umma_idesc_bf16(WT_M, CO, true);
    extern __shared__ __align__(128) unsigned char wt_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(wt_raw) + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t bars[10];   // full[4], done[4] (by stage), accfree[2]
    __shared__ uint32_t tmem_slot;
    __shared__ int bad;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full = smem_u32(&bars[0]), done = smem_u32(&bars[4]), accfree = smem_u32(&bars[8]);
    const int NS = a.stages;
    const int xp = x_pitch(a.kx, a.lead), dp = dy_pitch(a.kx, a.lead, CO);
    const int xbytes = (a.T + 2) * (CB / 8) * xp, stage = stage_bytes(a.kx, a.lead, CB, CO, a.T);
    const int dz = blockIdx.y;
    const int nci = a.cin / CB;
    const int ci0 = (blockIdx.z % nci) * CB, co0 = (blockIdx.z / nci) * CO;
    const int ybatches = (a.ny + a.T - 1) / a.T;
    const long long total = (long long)a.nz * ybatches * a.ntx;
    const long long b0 = total * blockIdx.x / a.chunks, b1 = total * (blockIdx.x + 1) / a.chunks;
    // batch -> tile; batches whose x plane lies outside the grid add nothing
    auto tile = [&](long long b, int& x0, int& y0, int& z) {
        x0 = (int)(b % a.ntx) * a.kx;
        y0 = (int)((b / a.ntx) % ybatches) * a.T;
        z = (int)(b / ((long long)a.ntx * ybatches));
        return z + dz - 1 >= 0 && z + dz - 1 < a.nz;
    };

    if (warp == 4) tmem_alloc(smem_u32(&tmem_slot), TMEM);
    if (tid == 0) {
        for (int s = 0; s < 4; s++) {
            mbar_init(full + 8 * s, COPY);
            mbar_init(done + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) mbar_init(accfree + 8 * s, 128);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bad = 0;
    }
    // the zeros before the lines: written once, the copies leave them alone
    const int xlines = (a.T + 2) * (CB / 8), lines_all = xlines + a.T * (CO / 8);
    if (a.lead)
        for (int s = 0; s < NS; s++)
            for (int l = tid >> 4; l < lines_all; l += WtThreads<CO>::all / 16) {
                unsigned char* line = sm + s * stage + (l < xlines ? l * xp : xbytes + (l - xlines) * dp);
                *reinterpret_cast<uint4*>(line + 16 * (tid & 15)) = make_uint4(0, 0, 0, 0);
            }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    umma_fence_before();
    __syncthreads();
    umma_fence_after();
    const uint32_t tmem = tmem_slot;

    constexpr int W = CO == 32 ? 32 : 16;   // columns read at once
    float acc[COLS];
#pragma unroll
    for (int i = 0; i < COLS; i++) acc[i] = 0.f;
    bool ok = true;
    if (warp >= 5) {
        const int t = tid - 160;
        int n = 0;   // batches issued
        for (long long b = b0; b < b1; b++) {
            int x0, y0, z;
            if (!tile(b, x0, y0, z)) continue;
            const int s = n % NS;
            if (n >= NS && !mbar_wait(done + 8 * s, (uint32_t)((n / NS - 1) & 1))) {
                ok = false;
                break;
            }
            const uint32_t dst = smem_u32(sm + s * stage) + 16 * a.lead;
            copy_lines<CB / 8, COPY>(dst, xp, a.T + 2, a.kx + 2, a.x + ci0, a.x_cs, x0 - 1, y0 - 1, z + dz - 1, a, t);
            copy_lines<CO / 8, COPY>(dst + xbytes, dp, a.T, a.kx, a.dy + co0, a.dy_cs, x0, y0, z, a, t);
            // the thread's arrival, once its copies so far have landed
            copy_arrive(full + 8 * s);
            n++;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");   // the shared memory outlives the copies
    } else if (warp == 4) {
        int n = 0;
        const int la = (CB / 8) * xp / 16, lb = (CO / 8) * dp / 16;   // a line further, in 16-byte units
        for (long long b = b0; b < b1; b++) {
            int x0, y0, z;
            if (!tile(b, x0, y0, z)) continue;
            const int s = n % NS;
            ok = mbar_wait(full + 8 * s, (uint32_t)((n / NS) & 1)) &&
                 (n < 2 || mbar_wait(accfree + 8 * (n & 1), (uint32_t)((n / 2 - 1) & 1)));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            // the copies were generic writes; the MMAs read through the async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            umma_fence_after();
            const uint32_t xs = smem_u32(sm) + s * stage + 16 * a.lead, d = tmem + (uint32_t)((n & 1) * COLS);
            const uint64_t ax = umma_desc(xs, 128, xp), bd = umma_desc(xs + xbytes, 128, dp);
            const int lines = min(a.T, a.ny - y0), steps = min(a.kx, (a.nx - x0 + 15) / 16 * 16) / 16;
            const int pad = max(16 * steps - (a.nx - x0), 0);
            const uint64_t ap = umma_advance(ax, -pad), bp = umma_advance(bd, -pad);
            uint32_t more = 0;   // the first step of a batch starts the accumulators
            for (int l = 0; l < lines; l++)
#pragma unroll 2
                for (int k = 0; k < steps; k++) {
                    const uint64_t ak = umma_advance(ax, l * la + 16 * k), bk = umma_advance(bd, l * lb + 16 * k);
                    umma_bf16(d, umma_advance(ap, l * la + 16 * k), umma_advance(bp, l * lb + 16 * k), idesc, more);
#pragma unroll
                    for (int dx = 1; dx < 3; dx++)
                        umma_bf16(d + (uint32_t)(dx * CO), umma_advance(ak, dx), bk, idesc, more);
                    more = 1;
                }
            umma_commit(done + 8 * s);
            n++;
        }
        // nothing may be in flight when the tensor memory is freed
        for (int q = n > NS ? n - NS : 0; q < n; q++) mbar_wait(done + 8 * (q % NS), (uint32_t)((q / NS) & 1));
    } else {
        int n = 0;
        for (long long b = b0; b < b1 && ok; b++) {
            int x0, y0, z;
            if (!tile(b, x0, y0, z)) continue;
            const int s = n & 1;
            ok = mbar_wait(done + 8 * (n % NS), (uint32_t)((n / NS) & 1));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            umma_fence_after();
            if (32 * warp < 3 * CB) {
#pragma unroll
                for (int c = 0; c < COLS / W; c++) {
                    float v[W];
                    const uint32_t at = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(s * COLS + W * c);
                    if constexpr (W == 32) tmem_ld32(at, v);
                    else tmem_ld16(at, v);
#pragma unroll
                    for (int i = 0; i < W; i++) acc[W * c + i] += v[i];
                }
            }
            umma_fence_before();
            mbar_arrive(accfree + 8 * s);
            n++;
        }
    }
    if (!ok) {
        atomicExch(a.err, 1);
        bad = 1;
    }
    umma_fence_before();
    __syncthreads();
    umma_fence_after();
    if (warp == 4) tmem_free(tmem, TMEM);
    if (bad) return;
    const int row = 32 * warp + lane;   // M row: (line offset, input channel)
    if (warp < 4 && row < 3 * CB) {
        const int oy = row / CB, ci = ci0 + row % CB;
        float* w = a.dw + ((long long)(3 * oy + 9 * dz) * a.cout + co0) * a.cin + ci;
#pragma unroll
        for (int dx = 0; dx < 3; dx++, w += (long long)(a.cout - CO) * a.cin)
#pragma unroll
            for (int n = 0; n < CO; n++, w += a.cin) atomicAdd(w, acc[dx * CO + n]);
    }
}

// ---------------------------------------------------------------------------
// scalar weight gradient: one CTA per (tap, 16-output block, 16-input block, voxel
// chunk); thread (co, ci) of a 16 x 16 block accumulates in FP32 over the
// chunk, staged 64 voxels at a time in shared memory; one atomic per output.
// ---------------------------------------------------------------------------
struct Grid {
    int g[3];
};
constexpr int WG_V = 64;          // voxels per staging step
constexpr int WG_CHUNK = 4096;    // voxels per CTA

__global__ void __launch_bounds__(256) k_wgrad0(Grid G, int cin, int cout, const __nv_bfloat16* __restrict__ x, int x_cs,
                                                int x_c0, const __nv_bfloat16* __restrict__ dy, int dy_cs, int dy_c0,
                                                float* __restrict__ dw)
{
    __shared__ float ds[WG_V][17], xs[WG_V][17];
    const int tap = blockIdx.y;
    const int nb_ci = cin / 16;
    const int co0 = (blockIdx.z / nb_ci) * 16, ci0 = (blockIdx.z % nb_ci) * 16;
    const int dx = tap % 3 - 1, dyy = (tap / 3) % 3 - 1, dz = tap / 9 - 1;
    const int tid = threadIdx.x, tco = tid >> 4, tci = tid & 15;
    const long long V = (long long)G.g[0] * G.g[1] * G.g[2];
    const long long v0 = (long long)blockIdx.x * WG_CHUNK;
    const long long v1 = min(V, v0 + WG_CHUNK);
    float acc = 0.f;
    for (long long vb = v0; vb < v1; vb += WG_V) {
        // stage dy[v][co0..+15] and x[v + off][ci0..+15] for 64 voxels (4 values per thread each)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int e = tid + 256 * q;   // 0 .. 1023
            const int vl = e >> 4, c = e & 15;
            const long long v = vb + vl;
            float d = 0.f, xv = 0.f;
            if (v < v1) {
                d = __bfloat162float(dy[v * dy_cs + dy_c0 + co0 + c]);
                const int ix = (int)(v % G.g[0]), iy = (int)((v / G.g[0]) % G.g[1]), iz = (int)(v / ((long long)G.g[0] * G.g[1]));
                const int jx = ix + dx, jy = iy + dyy, jz = iz + dz;
                if (jx >= 0 && jx < G.g[0] && jy >= 0 && jy < G.g[1] && jz >= 0 && jz < G.g[2]) {
                    const long long w = jx + (long long)G.g[0] * (jy + (long long)G.g[1] * jz);
                    xv = __bfloat162float(x[w * x_cs + x_c0 + ci0 + c]);
                }
            }
            ds[vl][c] = d;
            xs[vl][c] = xv;
        }
        __syncthreads();
#pragma unroll 8
        for (int v = 0; v < WG_V; v++) acc = fmaf(ds[v][tco], xs[v][tci], acc);
        __syncthreads();
    }
    atomicAdd(dw + ((long long)tap * cout + co0 + tco) * cin + ci0 + tci, acc);
}

// db[co] += sum_v dy[v][c0 + co]: threads read 8 channels (16 bytes) of a voxel
__global__ void __launch_bounds__(256) k_bgrad8(long long V, int groups, const uint4* __restrict__ dy, int cs8,
                                                int g0, float* __restrict__ db)
{
    __shared__ float red[8][8];
    const int g = blockIdx.y;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (long long v = blockIdx.x * 256LL + threadIdx.x; v < V; v += (long long)gridDim.x * 256) {
        const uint4 q = __ldg(dy + v * cs8 + g0 + g);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            s[2 * i] += __uint_as_float(w[i] << 16);
            s[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        for (int o = 16; o > 0; o >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][i] = s[i];
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        float t = 0;
        for (int w = 0; w < 8; w++) t += red[w][threadIdx.x];
        atomicAdd(db + 8 * g + threadIdx.x, t);
    }
}

// the same for slices that are not 16-byte aligned
__global__ void k_bgrad0(long long V, int cout, const __nv_bfloat16* __restrict__ dy, int dy_cs, int dy_c0,
                         float* __restrict__ db)
{
    __shared__ float red[32];
    const int co = blockIdx.y;
    float s = 0.f;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x)
        s += __bfloat162float(dy[v * dy_cs + dy_c0 + co]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (int)(blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) atomicAdd(db + co, s);
    }
}

constexpr int WT_SMEM = 220 * 1024;

template <int CB, int CO>
bool launch_wt(cudaStream_t st, WtArgs a)
{
    static DeviceOnce once;
    if (!allow_smem(once, k_wgrad_tc<CB, CO>, WT_SMEM)) return false;
    a.T = 4;
    a.lead = a.nx % 16 ? 16 : 0;
    while (a.T > 1 && smem_bytes(a.kx, a.lead, CB, CO, a.T, 2) > WT_SMEM) a.T--;
    a.stages = 4;
    while (a.stages > 2 && smem_bytes(a.kx, a.lead, CB, CO, a.T, a.stages) > WT_SMEM) a.stages--;
    const int blocks = 3 * (a.cin / CB) * (a.cout / CO);
    const long long total = (long long)a.nz * ((a.ny + a.T - 1) / a.T) * a.ntx;
    // one CTA a SM over all channel blocks and dz
    a.chunks = (int)std::min<long long>(std::max(1, sm_count() / blocks), total);
    k_wgrad_tc<CB, CO><<<dim3(a.chunks, 3, (a.cin / CB) * (a.cout / CO)), WtThreads<CO>::all,
                         smem_bytes(a.kx, a.lead, CB, CO, a.T, a.stages), st>>>(a);
    return true;
}

template <int CB> bool launch_wt_cb(cudaStream_t st, const WtArgs& a)
{
    if (a.cout % 64 == 0) return launch_wt<CB, 64>(st, a);
    if (a.cout % 32 == 0) return launch_wt<CB, 32>(st, a);
    return launch_wt<CB, 16>(st, a);
}

bool aligned8(const void* p, int cs, int c0)
{
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && cs % 8 == 0 && c0 % 8 == 0;
}

agb_status check_launch()
{
    count_launch();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(cudaGetErrorString(e));
        return AGB_CUDA;
    }
    return AGB_OK;
}

}  // namespace
}  // namespace agb

using namespace agb;

extern "C" agb_status agb_conv3_wgrad0(const int g[3], int cin, int cout, const void* x, int x_cs, int x_c0,
                                       const void* dy, int dy_cs, int dy_c0, float* dw, float* db, void* stream)
{
    auto slice_ok = [](int cs, int c0, int C) { return cs > 0 && c0 >= 0 && C > 0 && c0 + C <= cs; };
    if (!g || g[0] < 1 || g[1] < 1 || g[2] < 1 || !x || !dy || !dw || cin < 16 || cin % 16 || cout < 16 ||
        cout % 16 || !slice_ok(x_cs, x_c0, cin) || !slice_ok(dy_cs, dy_c0, cout)) {
        set_error("agb_conv3_wgrad0: bad argument (channels multiples of 16, slices inside their strides)");
        return AGB_BADARG;
    }
    const long long V = (long long)g[0] * g[1] * g[2];
    cudaStream_t st = (cudaStream_t)stream;
    bool tc = false;
    if (aligned8(x, x_cs, x_c0) && aligned8(dy, dy_cs, dy_c0)) {
        WtArgs a;
        a.nx = g[0];
        a.ny = g[1];
        a.nz = g[2];
        a.ntx = (g[0] + 127) / 128;
        a.kx = ((g[0] + a.ntx - 1) / a.ntx + 15) / 16 * 16;
        a.x = (const __nv_bfloat16*)x + x_c0;
        a.dy = (const __nv_bfloat16*)dy + dy_c0;
        a.x_cs = x_cs;
        a.dy_cs = dy_cs;
        a.cin = cin;
        a.cout = cout;
        a.dw = dw;
        a.err = conv_tc_error_address();
        if (a.err) tc = cin % 32 == 0 ? launch_wt_cb<32>(st, a) : launch_wt_cb<16>(st, a);
    }
    if (!tc) {
        Grid G{{g[0], g[1], g[2]}};
        const long long chunks = (V + WG_CHUNK - 1) / WG_CHUNK;
        dim3 grid((unsigned)chunks, 27, (unsigned)((cout / 16) * (cin / 16)));
        k_wgrad0<<<grid, 256, 0, st>>>(G, cin, cout, (const __nv_bfloat16*)x, x_cs, x_c0, (const __nv_bfloat16*)dy,
                                       dy_cs, dy_c0, dw);
    }
    agb_status s = check_launch();
    if (s != AGB_OK || !db) return s;
    if (aligned8(dy, dy_cs, dy_c0)) {
        const unsigned blocks = (unsigned)std::min<long long>((V + 1023) / 1024, 1LL * sm_count());
        k_bgrad8<<<dim3(blocks, cout / 8), 256, 0, st>>>(V, cout / 8, (const uint4*)dy, dy_cs / 8, dy_c0 / 8, db);
    } else {
        k_bgrad0<<<dim3(sm_count(), cout), 256, 0, st>>>(V, cout, (const __nv_bfloat16*)dy, dy_cs, dy_c0, db);
    }
    return check_launch();
}
