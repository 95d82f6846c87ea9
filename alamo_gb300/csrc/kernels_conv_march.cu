// kernels_conv_march.cu -- 3x3x3 convolutions of the learned correction that
// march in z: the layers whose weights fit beside the input in shared memory.
//
//   out[v][co] = act(bias[co] + sum_tap sum_ci in[v + off(tap)][ci] W[tap][co][ci])
//
// An MMA with M = 128 voxels and K = 16 channels reads 4 KB of shared memory for
// its voxels, 32 clocks, whatever N is: with N = cout = 16 and one MMA a tap the
// tensor cores wait for shared memory three quarters of the time.  So an input
// plane is multiplied once for the three output planes it reaches: N = 3 CO, 9
// MMAs (the taps in the plane) instead of 27.  The accumulators of an output
// plane are one of three slots of CO columns (plane mod 3); the weights of the
// three dz sit in the order 1 0 2 1 0, so that for every plane the three blocks
// that match the slots 0, 1, 2 follow one another.  A finished slot is read,
// stored and zeroed before the plane after the next adds to it.
//
// A plane is laid out flat with rows of nx + 2 voxels (the zero padding left
// and right): tile m is the flat positions 128 m .. 128 m + 127 of the output,
// and its operand for tap (dy, dx) starts dy (nx + 2) + dx voxels of 16 bytes
// further, so lines of any length fill the tiles but for two voxels.  A CTA
// takes mt tiles of a run of planes and CO output channels; 16 channels of a
// plane (with the two halo rows) are one unit of a ring that its copying
// threads fill with 16-byte cp.async, zeros outside the grid.
//
// Roles: two groups of four warps read the accumulators and store, one warp
// issues the MMAs, seven copy.  Every wait is bounded (about 1 s); one that runs out sets the
// error flag, and the CTA stops, waits (bounded) for what it issued, frees its
// tensor memory and returns.
//
// Measured (line kernel of kernels_conv_tc.cu -> this one), 129^3 voxels: 48 ->
// 16 channels 858 -> 142 us, 32 -> 32 712 -> 168, 64 -> 64 2020 -> 470 (1010
// TFLOP/s), 96 -> 32 1858 -> 476; 65^3: 32 -> 32 99 -> 33, 64 -> 64 262 -> 93.  What
// bounds it: the MMAs (56 clocks each at CO = 16, of which the voxels' operand is
// 32), and on short runs of planes the two halo planes and the start.
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

constexpr int MC_EPI = 256;                  // threads that read the accumulators, in two groups
constexpr int MC_COPY = 224;                 // copying threads
constexpr int MC_THREADS = MC_EPI + 32 + MC_COPY;
constexpr int MC_PIECES = 14;                // 16-byte pieces of a unit a copying thread brings at most
constexpr int MC_TILES = 8;                  // tiles of a CTA at most
constexpr int MC_RING = 4;
constexpr int MC_SMEM = 224 * 1024;

struct McArgs {
    int nx, ny, nz, px;        // px = nx + 2
    int cin, cout, cs;         // cs: channel stride of the input
    int mt, ring, zc;          // tiles, units of the ring, output planes of a CTA
    int np;                    // positions of a unit: 128 mt + 2 px + 2
    int half;                  // positions between its two 8-channel halves: np, up to 4 mod 8
    const __nv_bfloat16* in;   // first channel of the slice
    const __nv_bfloat16* wp;   // packed weights [stage][tap][2][cout][8]
    const float* bias;
    void* out;
    int out_cs, out_c0, out_f32, relu;
    int* err;
};

__host__ __device__ inline int weight_bytes(int cin, int co) { return cin / 16 * 9 * 2 * 5 * co * 16; }

template <int CO>
__global__ void __launch_bounds__(MC_THREADS, 1) k_conv3_march(McArgs a)
{
    extern __shared__ __align__(128) unsigned char mc_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(mc_raw) + 127) & ~(uintptr_t)127);
    // full[MC_RING], empty[MC_RING], accdone[MC_TILES], accfree[MC_TILES], weights
    __shared__ __align__(8) uint64_t bars[2 * MC_RING + 2 * MC_TILES + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ float bias[CO];
    __shared__ int bad;
    const uint32_t full = smem_u32(&bars[0]), empty = full + 8 * MC_RING, accdone = empty + 8 * MC_RING,
                   accfree = accdone + 8 * MC_TILES, wbar = accfree + 8 * MC_TILES;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int stages = a.cin / 16, unit = a.half * 32;
    const uint32_t sw = smem_u32(sm), sx = sw + weight_bytes(a.cin, CO);
    const int f0 = blockIdx.x * a.mt * 128;
    const int z0 = blockIdx.y * a.zc, z1 = min(z0 + a.zc, a.nz), planes = z1 - z0 + 2;   // input planes z0-1 .. z1
    const int co0 = blockIdx.z * CO;
    const int cols = a.mt * 3 * CO;
    const uint32_t tcols = cols <= 64 ? 64 : (cols <= 128 ? 128 : (cols <= 256 ? 256 : 512));

    if (warp == 8) tmem_alloc(smem_u32(&tmem_slot), tcols);
    if (tid == 0) {
        for (int s = 0; s < MC_RING; s++) {
            mbar_init(full + 8 * s, MC_COPY);
            mbar_init(empty + 8 * s, 1);
        }
        for (int m = 0; m < MC_TILES; m++) {
            mbar_init(accdone + 8 * m, 1);
            mbar_init(accfree + 8 * m, 128);
        }
        mbar_init(wbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bad = 0;
    }
    if (tid < CO) bias[tid] = a.bias ? __ldg(a.bias + co0 + tid) : 0.f;
    umma_fence_before();
    __syncthreads();
    umma_fence_after();
    const uint32_t tmem = tmem_slot;
    if (warp < 4) {   // lanes 32 warp .. of every column
        for (int c = 0; c < cols; c += 16) tmem_zero16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c);
        tmem_wait_st();
    } else if (warp == 8) {
        if (lane == 0) mbar_expect(wbar, (uint32_t)weight_bytes(a.cin, CO));
        __syncwarp();
        // block b of a (stage, tap in the plane, half): dz = 1, 0, 2, 1, 0
        for (int q = lane; q < stages * 9 * 2 * 5; q += 32) {
            const int b = q % 5, h = q / 5 % 2, t9 = q / 10 % 9, s = q / 90;
            const int tz = b == 2 ? 2 : (b % 3 == 0 ? 1 : 0);
            bulk_load(sw + (uint32_t)(q * CO * 16), a.wp + (((size_t)(s * 27 + tz * 9 + t9) * 2 + h) * a.cout + co0) * 8,
                      CO * 16, wbar);
        }
    }
    umma_fence_before();
    __syncthreads();
    umma_fence_after();

    bool ok = true;
    if (warp > 8) {
        // a thread keeps its half of 8 channels: two lanes bring the 32 bytes
        // of a voxel, so a warp touches as few lines as the channel stride allows
        const int t = tid - MC_EPI - 32, h = t & 1, p0 = t >> 1;
        // offsets of this thread's pieces in an input plane, -1 outside it
        int off[MC_PIECES];
#pragma unroll
        for (int j = 0; j < MC_PIECES; j++) {
            const int p = p0 + MC_COPY / 2 * j, f = f0 + p, y = f / a.px - 1, x = f % a.px - 1;
            off[j] = p < a.np && y >= 0 && y < a.ny && x >= 0 && x < a.nx ? (y * a.nx + x) * a.cs + 8 * h : -1;
        }
        const long long plane = (long long)a.nx * a.ny * a.cs;
        int u = 0;
        for (int n = 0; n < planes && ok; n++) {
            const int z = z0 - 1 + n;
            const bool zin = z >= 0 && z < a.nz;
            const __nv_bfloat16* src = a.in + (zin ? z : 0) * plane;
            for (int s = 0; s < stages; s++, u++) {
                const int slot = u % a.ring;
                if (u >= a.ring && !mbar_wait(empty + 8 * slot, (uint32_t)((u / a.ring - 1) & 1))) {
                    ok = false;
                    break;
                }
                const uint32_t dst = sx + slot * unit + (h * a.half + p0) * 16;
#pragma unroll
                for (int j = 0; j < MC_PIECES; j++) {
                    if (p0 + MC_COPY / 2 * j < a.np) {
                        const bool in = zin && off[j] >= 0;
                        copy16(dst + j * (MC_COPY / 2 * 16), src + (in ? off[j] + 16 * s : 0), in);
                    }
                }
                copy_arrive(full + 8 * slot);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");   // the shared memory outlives the copies
    } else if (warp == 8) {
        constexpr uint32_t idesc = umma_idesc_bf16(128, 3 * CO, false);
        const uint64_t wd = umma_desc(sw, 5 * CO * 16, 128);
        ok = __all_sync(0xffffffffu, mbar_wait(wbar, 0));
        if (!ok) mbar_wait(wbar, 0);   // bounded: the weights' copies must not outlive the shared memory
        int u = 0;
        for (int n = 0; n < planes && ok; n++) {
            const int r = (z0 - 1 + n + 3) % 3;
            const uint64_t wr = umma_advance(wd, (r == 0 ? 0 : 3 - r) * CO);   // first of the three blocks
            for (int s = 0; s < stages && ok; s++, u++) {
                const int slot = u % a.ring;
                ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * slot, (uint32_t)((u / a.ring) & 1)));
                if (!ok) break;
                // the copies were generic writes; the MMAs read through the async proxy
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                const uint64_t ad = umma_desc(sx + slot * unit, a.half * 16, 128), ws = umma_advance(wr, s * 90 * CO);
                for (int m = 0; m < a.mt; m++) {
                    if (s == 0 && n > 0) {
                        // the slot this plane starts was read and zeroed with the plane before
                        ok = __all_sync(0xffffffffu, mbar_wait(accfree + 8 * m, (uint32_t)((n - 1) & 1)));
                        if (!ok) break;
                    }
                    umma_fence_after();
                    const uint64_t am = umma_advance(ad, m * 128);
                    const uint32_t d = tmem + (uint32_t)(m * 3 * CO);
#pragma unroll
                    for (int dy = 0; dy < 3; dy++)
#pragma unroll
                        for (int dx = 0; dx < 3; dx++)
                            umma_bf16(d, umma_advance(am, dy * a.px + dx), umma_advance(ws, (dy * 3 + dx) * 10 * CO),
                                      idesc, 1u);
                    if (s == stages - 1) umma_commit(accdone + 8 * m);
                }
                umma_commit(empty + 8 * slot);
            }
        }
        // nothing may be in flight when the tensor memory is freed
        for (int q = u > a.ring ? u - a.ring : 0; q < u; q++)
            mbar_wait(empty + 8 * (q % a.ring), (uint32_t)((q / a.ring) & 1));
    } else {
        // two groups of four warps take the tiles in turn
        const int group = warp >> 2, row = 32 * (warp & 3) + lane;
        const uint32_t lanes = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        int vox[MC_TILES / 2];   // this thread's voxel of each of its tiles in a plane, -1 outside it
#pragma unroll
        for (int q = 0; q < MC_TILES / 2; q++) {
            const int f = f0 + (2 * q + group) * 128 + row, y = f / a.px, x = f % a.px;
            vox[q] = x < a.nx && y < a.ny ? y * a.nx + x : -1;
        }
        for (int n = 0; n < planes && ok; n++) {
            const int zo = z0 - 2 + n;   // complete once input plane zo + 1 has been added
            const int slot = (zo + 3) % 3;
            const bool keep = zo >= z0 && zo < z1;
#pragma unroll
            for (int q = 0; q < MC_TILES / 2; q++) {
                const int m = 2 * q + group;
                if (m >= a.mt || !ok) continue;
                ok = __all_sync(0xffffffffu, mbar_wait(accdone + 8 * m, (uint32_t)(n & 1)));
                if (!ok) continue;
                umma_fence_after();
                const uint32_t at = lanes + (uint32_t)((m * 3 + slot) * CO);
                float v[CO];
                if (keep) {
#pragma unroll
                    for (int cb = 0; cb < CO / 16; cb++) tmem_ld16(at + (uint32_t)(cb * 16), v + cb * 16);
                }
#pragma unroll
                for (int cb = 0; cb < CO / 16; cb++) tmem_zero16(at + (uint32_t)(cb * 16));
                tmem_wait_st();
                umma_fence_before();
                mbar_arrive(accfree + 8 * m);
                if (!keep || vox[q] < 0) continue;
                const long long o = ((long long)vox[q] + (long long)a.nx * a.ny * zo) * a.out_cs + a.out_c0 + co0;
#pragma unroll
                for (int i = 0; i < CO; i++) {
                    const float w = v[i] + bias[i];
                    v[i] = (a.relu && w < 0.f) ? 0.f : w;
                }
                if (a.out_f32) {
                    float4* d = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + o);
#pragma unroll
                    for (int i = 0; i < CO / 4; i++)
                        d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                } else {
                    uint4* d = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + o);
#pragma unroll
                    for (int i = 0; i < CO / 8; i++) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const __nv_bfloat162 hb = __floats2bfloat162_rn(v[8 * i + 2 * e], v[8 * i + 2 * e + 1]);
                            w[e] = *reinterpret_cast<const uint32_t*>(&hb);
                        }
                        d[i] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        }
    }
    if (!ok) {
        atomicExch(a.err, 1);
        bad = 1;
    }
    umma_fence_before();
    __syncthreads();
    umma_fence_after();
    if (warp == 8) tmem_free(tmem, tcols);
}

template <int CO> bool launch_march(cudaStream_t st, const McArgs& a, int smem)
{
    static DeviceOnce once;
    if (!allow_smem(once, k_conv3_march<CO>, MC_SMEM)) return false;
    const int tiles = (a.ny * a.px + a.mt * 128 - 1) / (a.mt * 128);
    k_conv3_march<CO><<<dim3(tiles, (a.nz + a.zc - 1) / a.zc, a.cout / CO), MC_THREADS, smem, st>>>(a);
    return true;
}

}  // namespace

// Plan: the block of output channels, the tiles and the planes of a CTA with
// the smallest estimate of waves x clocks of a CTA.  A unit costs the MMAs'
// clocks (32 for the voxels' operand and a quarter of N, half of N at least) or
// its copy at 45 bytes a clock; a CTA its weights and start.  False: no plan
// fits (weights too large, rows too long), the line kernel serves.
bool launch_conv3_march(cudaStream_t st, const int n[3], int cin, int cout, const void* in, int in_cs, int in_c0,
                        const void* wp, const float* bias, void* out, int out_cs, int out_c0, int out_f32, int relu,
                        int* err)
{
    McArgs a;
    a.nx = n[0];
    a.ny = n[1];
    a.nz = n[2];
    a.px = n[0] + 2;
    if ((long long)a.nx * a.ny * in_cs > 0x3fffffffLL || (long long)a.px * (a.ny + 2) > 0x3fffffffLL || n[2] > 65535)
        return false;
    a.cin = cin;
    a.cout = cout;
    a.cs = in_cs;
    a.in = (const __nv_bfloat16*)in + in_c0;
    a.wp = (const __nv_bfloat16*)wp;
    a.bias = bias;
    a.out = out;
    a.out_cs = out_cs;
    a.out_c0 = out_c0;
    a.out_f32 = out_f32;
    a.relu = relu;
    a.err = err;
    const int sms = std::max(1, sm_count()), stages = cin / 16;
    if ((long long)((a.nx + 127) / 128) * a.ny * a.nz <= 2LL * sms) return false;
    const int blocks[4] = {64, 48, 32, 16};
    const double lines = std::max(21.0, in_cs * 2 * 16 / 128.0);   // clocks of a warp's copy of 16 voxels
    double best = 0;
    int best_co = 0, best_smem = 0;
    McArgs plan = a;
    for (int co : blocks) {
        if (cout % co) continue;
        for (int mt = 1; mt <= MC_TILES && mt * 3 * co <= 512; mt++) {
            a.mt = mt;
            a.np = 128 * mt + 2 * a.px + 2;
            a.half = (a.np + 3) / 8 * 8 + 4;
            if (a.half < a.np) a.half += 8;
            if (2 * a.np > MC_PIECES * MC_COPY) break;
            a.ring = MC_RING;
            auto bytes = [&] { return 128 + weight_bytes(cin, co) + a.ring * a.half * 32 + 128; };
            while (a.ring > 2 && bytes() > MC_SMEM) a.ring--;
            if (bytes() > MC_SMEM) break;
            const long long ctas = (long long)((a.ny * a.px + mt * 128 - 1) / (mt * 128)) * (cout / co);
            const double mma = std::max(44 + 0.75 * co, 1.5 * co) * 9 * mt, copy = a.np * 2 / 32.0 * lines;
            const double u = std::max(std::max(mma, copy) * stages, mt * (300.0 + 5 * co)), start = 4000 + weight_bytes(cin, co) / 40.0;
            for (int zch = 1; zch <= std::min(a.nz, 64); zch++) {
                a.zc = (a.nz + zch - 1) / zch;
                const long long waves = (ctas * ((a.nz + a.zc - 1) / a.zc) + sms - 1) / sms;
                const double cost = waves * ((a.zc + 2) * u + start);
                if (!best_co || cost < best) {
                    best = cost;
                    best_co = co;
                    best_smem = bytes();
                    plan = a;
                }
            }
        }
    }
    switch (best_co) {
    case 64: return launch_march<64>(st, plan, best_smem);
    case 48: return launch_march<48>(st, plan, best_smem);
    case 32: return launch_march<32>(st, plan, best_smem);
    case 16: return launch_march<16>(st, plan, best_smem);
    }
    return false;
}

}  // namespace agb
