// wp_conv.cu -- 3x3x3 "same" convolutions of channels-last BF16 volumes on the tcgen05 tensor cores
// (FP32 accumulation in TMEM), the building block of the warm-start network.  No reference
// counterpart: the reference has no learned component.
//
// Layouts.  Activations: [z][x][y][c] BF16 (c fastest), c in {16, 32, 64}.  Weights of one input
// part: [tap][cout][cin] BF16 with tap = (dz * 3 + dx) * 3 + dy, offsets d - 1 (zero padding).
//
// Forward / input-gradient kernels (implicit GEMM, K-major operands).  Layers whose weights and a ring of input
// planes fit shared memory take conv3_walk_kernel (described there), the others conv3_fwd_kernel: a CTA owns a tile of
// M = 128 voxels of one z plane (yt consecutive y times xt consecutive x, yt * xt = 128) and all
// cout outputs.  K runs over (input part, tap, cin): per tap a TMA load brings the shifted
// [128 voxels][cin] block of the input (out-of-range voxels arrive as zeros = the padding) and the
// [cout][cin] weight block, each row one swizzle span (cin * 2 bytes = 32/64/128 B), which is the
// canonical K-major UMMA layout; cin / 16 tcgen05.mma (M=128, N=cout, K=16) accumulate into TMEM.
// Warp roles: warp 0 issues TMA, warp 1 owns TMEM and issues the MMAs, warps 2-5 drain TMEM
// (tcgen05.ld, one voxel per thread) and apply bias / skip-add / ReLU mask / ReLU, storing BF16.
// The input gradient of a convolution is the same kernel on the output gradient with the weights
// transposed and flipped ([26 - tap][cin][cout]).
//
// Weight-gradient kernel (MN-major operands).  dW[tap][co][ci] = sum_v dY[v][co] X[v + off(tap)][ci]
// is a GEMM with M = (tap, ci) rows, N = cout, K = voxels: a CTA owns 128 / cin taps (one M tile
// of 128 rows) and a range of voxel tiles; per voxel tile it TMA-loads the shifted input block of
// each of its taps (each an MN-major swizzle atom of width cin, stacked along M) and the output
// gradient block (MN-major, width cout), issues 8 MMAs of K = 16 voxels, and finally adds its
// partial [128][cout] tile into the FP32 weight gradient with atomics.
#include "wp_common.cuh"
#include "wp_tc.cuh"

#include <algorithm>
#include <cstring>
#include <mutex>

using namespace wptc;

namespace {

constexpr int kThreads = 192;
constexpr int kStagesF = 4;
constexpr int kSlotA = 16384;  // 128 rows x 64 channels x 2 B
constexpr int kSlotB = 8192;   // 64 x 64 x 2 B
constexpr int kWalkThreads = 320; // weights, MMA, 4 epilogue and 4 producer warps
constexpr int kStagesWalk = 6;  // input planes of the walk kernel's ring at most
constexpr int kStagesW = 3;
constexpr int kSlotWA = 32768;  // 128 x 128 x 2 B
constexpr int kSlotWB = 16384;  // 128 x 64 x 2 B

__device__ __forceinline__ void store_bf16_row(__nv_bfloat16* dst, const float* v, int n) {
    for (int c = 0; c < n; c += 8) {
        __nv_bfloat162 h[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(v[c + 2 * k], v[c + 2 * k + 1]);
        *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<uint4*>(h);
    }
}

__device__ __forceinline__ void load_bf16_row(const __nv_bfloat16* src, float* v, int n) {
    for (int c = 0; c < n; c += 8) {
        uint4 u = *reinterpret_cast<const uint4*>(src + c);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = __bfloat1622float2(h[k]);
            v[c + 2 * k] = f.x;
            v[c + 2 * k + 1] = f.y;
        }
    }
}

struct TileGeo {
    int yt, xt, nty, ntx;
};

// one voxel's outputs: bias, skip addend, mask, ReLU, BF16 store
template <int COUT>
__device__ __forceinline__ void store_voxel(float* acc, long v, __nv_bfloat16* __restrict__ out,
                                            const float* __restrict__ bias, const __nv_bfloat16* __restrict__ addend,
                                            const __nv_bfloat16* __restrict__ mask, int relu) {
    if (bias)
#pragma unroll
        for (int c = 0; c < COUT; ++c) acc[c] += bias[c];
    if (addend) {
        float a2[COUT];
        load_bf16_row(addend + v * COUT, a2, COUT);
#pragma unroll
        for (int c = 0; c < COUT; ++c) acc[c] += a2[c];
    }
    if (mask) {
        float mk[COUT];
        load_bf16_row(mask + v * COUT, mk, COUT);
#pragma unroll
        for (int c = 0; c < COUT; ++c) acc[c] = mk[c] > 0.f ? acc[c] : 0.f;
    }
    if (relu)
#pragma unroll
        for (int c = 0; c < COUT; ++c) acc[c] = fmaxf(acc[c], 0.f);
    store_bf16_row(out + v * COUT, acc, COUT);
}

// After a pipeline wait gave up: waits (bounded) for the tile loads issued but never consumed, steps
// [consumed, issued) of the ring of full barriers, so that no copy into this CTA's shared memory is
// in flight when it exits.  The withheld step was never issued.
__device__ __forceinline__ void drain_copies(uint32_t bar_full, int stages, int consumed, int issued, int withheld,
                                             int* err) {
    for (int k = consumed; k < issued; ++k)
        if (k != withheld && !mbar_wait(bar_full + 8 * (k % stages), (k / stages) & 1, err)) return;
}

template <int COUT>
__global__ void __launch_bounds__(kThreads, 1)
    conv3_fwd_kernel(const __grid_constant__ CUtensorMap xm0, const __grid_constant__ CUtensorMap wm0,
                     const __grid_constant__ CUtensorMap xm1, const __grid_constant__ CUtensorMap wm1, int cin0,
                     int cin1, int nparts, __nv_bfloat16* __restrict__ out, const float* __restrict__ bias,
                     const __nv_bfloat16* __restrict__ addend, const __nv_bfloat16* __restrict__ mask, int relu, int nx,
                     int ny, int nz, TileGeo tg, int* err, int withhold, unsigned long long lim) {
    constexpr int NCOL = COUT < 32 ? 32 : COUT;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* basep = smem_raw + (base - raw);
    const uint32_t bar_full = base + kStagesF * (kSlotA + kSlotB);
    const uint32_t bar_empty = bar_full + 8 * kStagesF;
    const uint32_t bar_acc = bar_empty + 8 * kStagesF;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(basep + kStagesF * (kSlotA + kSlotB) + 16 * kStagesF + 8);
    volatile int* s_consumed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* s_fail = reinterpret_cast<volatile int*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x != 0) withhold = -1;
    long t = blockIdx.x;
    const int ty = (int)(t % tg.nty);
    t /= tg.nty;
    const int tx = (int)(t % tg.ntx);
    const int z = (int)(t / tg.ntx);
    const int y0 = ty * tg.yt, x0 = tx * tg.xt;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStagesF; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init_fence();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), NCOL);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int nk = 27 * nparts;

    int issued = 0;
    if (warp == 0 && lane == 0) {
        for (int k = 0; k < nk; ++k) {
            const int s = k % kStagesF;
            if (!mbar_wait(bar_empty + 8 * s, ((k / kStagesF) & 1) ^ 1, err, lim)) break;
            issued = k + 1;
            if (k == withhold) continue;
            const int part = k / 27, tap = k % 27;
            const int cin = part ? cin1 : cin0;
            const int dz = tap / 9, dx = (tap / 3) % 3, dy = tap % 3;
            const uint32_t a = base + s * (kSlotA + kSlotB), b = a + kSlotA;
            mbar_expect_tx(bar_full + 8 * s, (uint32_t)(128 * cin * 2 + COUT * cin * 2));
            tma_load_4d(a, part ? &xm1 : &xm0, bar_full + 8 * s, 0, y0 + dy - 1, x0 + dx - 1, z + dz - 1);
            tma_load_2d(b, part ? &wm1 : &wm0, bar_full + 8 * s, 0, tap * COUT);
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t idesc = idesc_bf16_f32(128, COUT, 0, 0);
        int k = 0;
        for (; k < nk; ++k) {
            const int s = k % kStagesF;
            if (!mbar_wait(bar_full + 8 * s, (k / kStagesF) & 1, err, lim)) break;
            tc_fence_after();
            const int cin = (k / 27) ? cin1 : cin0;
            const uint32_t rowb = (uint32_t)cin * 2, lay = sw_code(cin * 2);
            const uint32_t a = base + s * (kSlotA + kSlotB), b = a + kSlotA;
            for (int j = 0; j < cin / 16; ++j) {
                const uint64_t ad = smem_desc(a + 32 * j, 16, 8 * rowb, lay);
                const uint64_t bd = smem_desc(b + 32 * j, 16, 8 * rowb, lay);
                umma_f16(tmem, ad, bd, idesc, (k | j) != 0);
            }
            umma_commit(bar_empty + 8 * s);
        }
        *s_consumed = k;
        *s_fail = k < nk;
        umma_commit(bar_acc);  // also on failure: bar_acc then tracks the MMAs already issued
    }
    bool ready = false;
    if (warp >= 2) ready = mbar_wait(bar_acc, 0, err);
    __syncthreads();
    if (warp == 0 && lane == 0) drain_copies(bar_full, kStagesF, *s_consumed, issued, withhold, err);
    if (warp >= 2) {
        const int q = warp & 3;
        const int m = q * 32 + lane;
        ready = ready && !*s_fail;
        __syncwarp();  // tcgen05.ld is warp-collective
        tc_fence_after();
        float acc[COUT];
#pragma unroll
        for (int c = 0; c < COUT; c += 16) tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + c, acc + c);
        tmem_wait_ld();
        const int xi = m / tg.yt, yi = m - xi * tg.yt;
        const int x = x0 + xi, y = y0 + yi;
        if (ready && x < nx && y < ny) {
            const long v = ((long)z * nx + x) * ny + y;
            store_voxel<COUT>(acc, v, out, bias, addend, mask, relu);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, NCOL);
    }
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Forward / input-gradient kernel that walks the planes of a column of tiles.  conv3_fwd_kernel fetches the
// shifted input once per tap, 27 times in all (250 MB through L2 for 16 channels at 64^3, 70 us); here a CTA
// keeps the layer's weights and a ring of input planes resident, each plane's halo block fetched once and
// used for three output planes, and the x and y offsets are taken by moving the operand's start address.
// That needs rows at a fixed pitch in one run, so a block is stored without swizzle, one part per 8 channels
// of 16-byte rows [x][y = -1 .. ny], and the 128 rows of a tile are 128 consecutive positions of the padded
// plane index x (ny + 2) + y: a tap (dx, dy) is the run that starts dx (ny + 2) + dy rows later.  Positions
// with y >= ny compute padding that is not stored (2 / (ny + 2) of the work).  The blocks arrive by
// 16-byte cp.async from four producer warps (zero-filled outside the volume).  Two accumulators in TMEM: the
// epilogue of a plane overlaps the next plane's products.
// What bounds it is the rate of the products, some 140 cycles each of 128 x N x 16 whatever N is.  Measured at
// 64^3 (B200): 16 -> 16 channels 70 -> 32 us, 32 -> 32 78 -> 62, 16 + 32 -> 16 123 -> 80; at 32^3 and 16^3 within
// 2 us of conv3_fwd_kernel, mostly below it.
struct WalkGeo {
    int pitch;     // ny + 2
    int rows;      // x rows of a block
    int tiles;     // per plane
    unsigned mpitch; // position / pitch = umulhi(position, mpitch)
    int lbo;       // bytes between the 8-channel parts of a block (a multiple of 128)
    int slot;      // bytes of a ring step (one input plane, all its channels)
    int w1, wbytes; // offset of the second part's weights, bytes of all
    int stages;    // 0: does not fit
    int zc;        // output planes per CTA
};

// 16 bytes, of which `bytes` (0 or 16) are read and the rest zero
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// The products of one input plane and part: 9 taps of CIN channels.  One thread issues them, so that building a
// descriptor (some forty dependent instructions, 220 cycles) cost more than its product: two are built and the
// others are sums (the address is their low field, in 16 bytes).
template <int COUT, int CIN>
__device__ __forceinline__ void walk_taps(uint32_t acc, uint32_t a, uint32_t b, const WalkGeo& g, uint32_t idesc, bool first) {
    const uint64_t da = smem_desc(a, g.lbo, 128, 0), db = smem_desc(b, 16, 16 * CIN, sw_code(2 * CIN));
    const uint32_t step = (uint32_t)g.lbo >> 3;  // two 8-channel parts
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int j = 0; j < CIN / 16; ++j)
            umma_f16(acc, da + (uint32_t)((t / 3) * g.pitch + t % 3 + j * step), db + (uint32_t)(t * COUT * CIN / 8 + 2 * j), idesc,
                     !first || (t | j) != 0);
}

template <int COUT>
__global__ void __launch_bounds__(kWalkThreads, 1)
    conv3_walk_kernel(const __nv_bfloat16* __restrict__ xin0, const __grid_constant__ CUtensorMap wm0,
                      const __nv_bfloat16* __restrict__ xin1, const __grid_constant__ CUtensorMap wm1, int cin0,
                      int cin1, int nparts, __nv_bfloat16* __restrict__ out, const float* __restrict__ bias,
                      const __nv_bfloat16* __restrict__ addend, const __nv_bfloat16* __restrict__ mask, int relu, int nx,
                      int ny, int nz, WalkGeo g, int* err, int withhold, unsigned long long lim) {
    constexpr int NCOL = COUT < 32 ? 32 : COUT;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // weights | ring | barriers
    unsigned char* basep = smem_raw + (base - raw);
    const uint32_t ring = base + g.wbytes;
    const uint32_t bar_full = ring + g.stages * g.slot;
    const uint32_t bar_empty = bar_full + 8 * kStagesWalk;
    const uint32_t bar_w = bar_empty + 8 * kStagesWalk;
    const uint32_t bar_accf = bar_w + 8, bar_acce = bar_accf + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(basep + (bar_acce + 16 - base));
    volatile int* s_fail = reinterpret_cast<volatile int*>(tmem_slot + 1);  // the first output plane without a sum

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chunk = blockIdx.x / g.tiles, p0 = (blockIdx.x - chunk * g.tiles) * 128;
    const int z0 = chunk * g.zc, nout = min(g.zc, nz - z0), nk = nout + 2;
    const int x0 = p0 / g.pitch, off0 = p0 - x0 * g.pitch;
    // a withheld step is numbered by taps, as in conv3_fwd_kernel
    withhold = blockIdx.x != 0 || withhold < 0 ? -1 : min(withhold / 9, nk - 1);

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; ++s) {
            mbar_init(bar_full + 8 * s, 128);  // the producer threads
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_w, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_accf + 8 * b, 1);
            mbar_init(bar_acce + 8 * b, 4);
        }
        mbar_init_fence();
        *s_fail = 1 << 30;
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 2 * NCOL);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        mbar_expect_tx(bar_w, (uint32_t)(27 * COUT * (cin0 + (nparts > 1 ? cin1 : 0)) * 2));
        for (int part = 0; part < nparts; ++part)
            for (int j = 0; j < 9; ++j) {
                const uint32_t at = part ? base + g.w1 + j * 3 * COUT * cin1 * 2 : base + j * 3 * COUT * cin0 * 2;
                tma_load_2d(at, part ? &wm1 : &wm0, bar_w, 0, 3 * j * COUT);
            }
    } else if (warp >= 6) {
        // input planes: step k is issued when its slot is free and handed over lag steps later, so that the
        // copies of up to lag + 1 steps are in flight (a product of plane o waits for three steps: lag + 3
        // <= stages)
        const int tid = threadIdx.x - 192, lag = min(2, g.stages - 3);
        auto hand_over = [&](int k) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (k != withhold) mbar_arrive(bar_full + 8 * (k % g.stages));
        };
        int k = 0;
        for (; k < nk; ++k) {
            const int s = k % g.stages;
            if (k >= g.stages && !mbar_wait(bar_empty + 8 * s, ((k / g.stages) & 1) ^ 1, err, lim)) break;
            const int zz = z0 + k - 1;
            const bool zin = zz >= 0 && zz < nz;
            uint32_t a = ring + s * g.slot;
            for (int part = 0; part < nparts; ++part) {
                const int cin = part ? cin1 : cin0, lg = cin == 16 ? 1 : cin == 32 ? 2 : 3;  // log2 of its 8-channel parts
                const __nv_bfloat16* src = (part ? xin1 : xin0) + (long)zz * nx * ny * cin;
                for (int e = tid; e < (g.rows * g.pitch) << lg; e += 128) {
                    const int pos = e >> lg, c = e & ((1 << lg) - 1);
                    const int r = (int)__umulhi((unsigned)pos, g.mpitch), yy = pos - r * g.pitch - 1, xx = x0 - 1 + r;
                    const bool in = zin && xx >= 0 && xx < nx && yy >= 0 && yy < ny;
                    cp_async16_zfill(a + c * g.lbo + 16 * pos, in ? src + ((long)xx * ny + yy) * cin + 8 * c : xin0, in ? 16 : 0);
                }
                a += cin / 8 * g.lbo;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (lag == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            if (k >= lag) hand_over(k - lag);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");  // none in flight when the CTA exits
        for (int j = max(k - lag, 0); j < k; ++j) hand_over(j);
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t idesc = idesc_bf16_f32(128, COUT, 0, 0);
        int have = 0, o = 0;
        bool ok = mbar_wait(bar_w, 0, err, lim);
        for (; ok && o < nout; ++o) {
            const uint32_t acc = tmem + (o & 1) * NCOL;
            if (o >= 2) ok = mbar_wait(bar_acce + 8 * (o & 1), ((o >> 1) & 1) ^ 1, err, lim);
            for (int dz = 0; ok && dz < 3; ++dz) {
                const int k = o + dz, s = k % g.stages;
                if (k >= have) {
                    ok = mbar_wait(bar_full + 8 * s, (k / g.stages) & 1, err, lim);
                    if (!ok) break;
                    have = k + 1;
                }
                tc_fence_after();
                uint32_t a = ring + s * g.slot + 16 * off0;
                for (int part = 0; part < nparts; ++part) {
                    const int cin = part ? cin1 : cin0;
                    const uint32_t b = base + (part ? g.w1 : 0) + dz * 9 * COUT * cin * 2;
                    if (cin == 16) walk_taps<COUT, 16>(acc, a, b, g, idesc, (dz | part) == 0);
                    else if (cin == 32) walk_taps<COUT, 32>(acc, a, b, g, idesc, (dz | part) == 0);
                    else walk_taps<COUT, 64>(acc, a, b, g, idesc, (dz | part) == 0);
                    a += cin / 8 * g.lbo;
                }
            }
            if (!ok) break;
            umma_commit(bar_empty + 8 * (o % g.stages));  // input plane o has had its last use
            umma_commit(bar_accf + 8 * (o & 1));
        }
        if (o < nout) {
            *s_fail = o;
            __threadfence_block();
            umma_commit(bar_accf + 8 * (o & 1));  // tracks the MMAs already issued
        }
    } else if (warp >= 2 && warp < 6) {
        const int q = warp & 3;
        const int p = p0 + q * 32 + lane;
        const int x = p / g.pitch, y = p - x * g.pitch;
        for (int o = 0; o < nout; ++o) {
            const bool ready = mbar_wait(bar_accf + 8 * (o & 1), (o >> 1) & 1, err);
            if (!__all_sync(0xffffffffu, ready && *s_fail > o)) break;
            tc_fence_after();
            float acc[COUT];
#pragma unroll
            for (int c = 0; c < COUT; c += 16) tmem_ld16(tmem + (o & 1) * NCOL + ((uint32_t)(q * 32) << 16) + c, acc + c);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_acce + 8 * (o & 1));
            if (x < nx && y < ny)
                store_voxel<COUT>(acc, ((long)(z0 + o) * nx + x) * ny + y, out, bias, addend, mask, relu);
        }
    }
    if (warp == 0 && lane == 0) mbar_wait(bar_w, 0, err);  // no copy in flight when the CTA exits
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 2 * NCOL);
    }
}

template <int COUT>
__global__ void __launch_bounds__(kThreads, 1)
    conv3_wgrad_kernel(const __grid_constant__ CUtensorMap xm, const __grid_constant__ CUtensorMap gm, int cin,
                       float* __restrict__ dw, int nx, int ny, int nz, TileGeo tg, long ntiles, int tiles_per_cta,
                       int* err, int withhold, unsigned long long lim) {
    constexpr int NCOL = COUT < 32 ? 32 : COUT;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* basep = smem_raw + (base - raw);
    const uint32_t bar_full = base + kStagesW * (kSlotWA + kSlotWB);
    const uint32_t bar_empty = bar_full + 8 * kStagesW;
    const uint32_t bar_acc = bar_empty + 8 * kStagesW;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(basep + kStagesW * (kSlotWA + kSlotWB) + 16 * kStagesW + 8);
    volatile int* s_consumed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* s_fail = reinterpret_cast<volatile int*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x != 0 || blockIdx.y != 0) withhold = -1;
    const int tpg = 128 / cin;             // taps per CTA (one M tile of 128 rows)
    const int tap0 = blockIdx.x * tpg;
    const int ntap = min(tpg, 27 - tap0);
    const long k0 = (long)blockIdx.y * tiles_per_cta;
    const int nk = (int)min((long)tiles_per_cta, ntiles - k0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStagesW; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init_fence();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), NCOL);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    int issued = 0;
    if (warp == 0 && lane == 0) {
        for (int k = 0; k < nk; ++k) {
            const int s = k % kStagesW;
            if (!mbar_wait(bar_empty + 8 * s, ((k / kStagesW) & 1) ^ 1, err, lim)) break;
            issued = k + 1;
            if (k == withhold) continue;
            long t = k0 + k;
            const int ty = (int)(t % tg.nty);
            t /= tg.nty;
            const int tx = (int)(t % tg.ntx);
            const int z = (int)(t / tg.ntx);
            const int y0 = ty * tg.yt, x0 = tx * tg.xt;
            const uint32_t a = base + s * (kSlotWA + kSlotWB), b = a + kSlotWA;
            mbar_expect_tx(bar_full + 8 * s, (uint32_t)(ntap * 128 * cin * 2 + 128 * COUT * 2));
            for (int j = 0; j < ntap; ++j) {
                const int tap = tap0 + j;
                const int dz = tap / 9, dx = (tap / 3) % 3, dy = tap % 3;
                tma_load_4d(a + j * 128 * cin * 2, &xm, bar_full + 8 * s, 0, y0 + dy - 1, x0 + dx - 1, z + dz - 1);
            }
            tma_load_4d(b, &gm, bar_full + 8 * s, 0, y0, x0, z);
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t idesc = idesc_bf16_f32(128, COUT, 1, 1);
        const uint32_t rowa = (uint32_t)cin * 2, laya = sw_code(cin * 2);
        constexpr uint32_t rowb = COUT * 2, layb = sw_code(COUT * 2);
        int k = 0;
        for (; k < nk; ++k) {
            const int s = k % kStagesW;
            if (!mbar_wait(bar_full + 8 * s, (k / kStagesW) & 1, err, lim)) break;
            tc_fence_after();
            const uint32_t a = base + s * (kSlotWA + kSlotWB), b = a + kSlotWA;
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                const uint64_t ad = smem_desc(a + kk * 16 * rowa, 128 * rowa, 8 * rowa, laya);
                const uint64_t bd = smem_desc(b + kk * 16 * rowb, 128 * rowb, 8 * rowb, layb);
                umma_f16(tmem, ad, bd, idesc, (k | kk) != 0);
            }
            umma_commit(bar_empty + 8 * s);
        }
        *s_consumed = k;
        *s_fail = k < nk || nk <= 0;
        umma_commit(bar_acc);  // also on failure: bar_acc then tracks the MMAs already issued
    }
    bool ready = false;
    if (warp >= 2) ready = mbar_wait(bar_acc, 0, err);
    __syncthreads();
    if (warp == 0 && lane == 0) drain_copies(bar_full, kStagesW, *s_consumed, issued, withhold, err);
    if (warp >= 2) {
        const int q = warp & 3;
        const int m = q * 32 + lane;
        ready = ready && !*s_fail;
        __syncwarp();  // tcgen05.ld is warp-collective
        tc_fence_after();
        float acc[COUT];
#pragma unroll
        for (int c = 0; c < COUT; c += 16) tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + c, acc + c);
        tmem_wait_ld();
        const int j = m / cin, ci = m - j * cin;
        if (ready && j < ntap) {
            float* d = dw + (long)(tap0 + j) * COUT * cin + ci;
#pragma unroll
            for (int co = 0; co < COUT; ++co) atomicAdd(d + (long)co * cin, acc[co]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, NCOL);
    }
}

// ------------------------------------------------------------------------------ host side
using wptc::EncodeTiledFn;
EncodeTiledFn encode_fn() { return wptc::encode_tiled(); }

CUtensorMapSwizzle swz(int bytes) {
    return bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

// [z][x][y][c] volume, box (c, yt, xt, 1)
bool map_volume(CUtensorMap* m, const void* p, int c, int nx, int ny, int nz, int yt, int xt) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)ny, (cuuint64_t)nx, (cuuint64_t)nz};
    const cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)c * 2 * ny, (cuuint64_t)c * 2 * ny * nx};
    const cuuint32_t box[4] = {(cuuint32_t)c, (cuuint32_t)yt, (cuuint32_t)xt, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swz(c * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// [27 * cout][cin] weights, box (cin, taps * cout)
bool map_weights(CUtensorMap* m, const void* p, int cin, int cout, int taps = 1) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cin, (cuuint64_t)27 * cout};
    const cuuint64_t strides[1] = {(cuuint64_t)cin * 2};
    const cuuint32_t box[2] = {(cuuint32_t)cin, (cuuint32_t)(taps * cout)};
    const cuuint32_t es[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swz(cin * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool chan_ok(int c) { return c == 16 || c == 32 || c == 64; }
bool pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }

TileGeo tile_geo(int nx, int ny) {
    TileGeo g;
    g.yt = ny < 128 ? ny : 128;
    g.xt = 128 / g.yt;
    g.nty = (ny + g.yt - 1) / g.yt;
    g.ntx = (nx + g.xt - 1) / g.xt;
    return g;
}

// The walk kernel's geometry for a layer, or stages = 0 where conv3_fwd_kernel takes it: where the weights and four
// input planes do not fit shared memory (64 channels on both sides, 96 into 32), and where few planes make
// a CTA's start dearer than the input it saves.  Both times in us as fitted to measured ones (B200; within 20%):
// conv3_fwd_kernel runs waves of two CTAs per SM, 8.6 a part and 0.05 a channel each; the walk kernel pays for the
// arrival of its first planes (some of it hidden in the waves after the first), then for every plane, 16 channels
// and CTA on the SM 1.5 of products or, for wide blocks, what they take to arrive.  conv3_fwd_kernel is taken where
// it is ahead by 2 us.  On planes of 256 x 256, 16 channels: 2 planes 41 against 51 us, 4 planes 69 against 74, 6
// planes 100 against 92; on 128 x 128, 32 channels: 2 planes 17.6 against 19.3, 3 planes 26.7 against 22.5; one plane
// of 128 x 128, 16 channels: 15.6 against 13.1.
WalkGeo walk_geo(int nx, int ny, int nz, int cin0, int cin1, int cout) {
    WalkGeo g{};
    g.pitch = ny + 2;
    if (g.pitch > 4096) return g;
    g.mpitch = (unsigned)((0x100000000ull + g.pitch - 1) / g.pitch);
    g.tiles = (nx * g.pitch + 127) / 128;
    // a tile starts up to ny + 1 positions into its first row and reads two rows and two positions further
    g.rows = 2 + (128 + ny + 1 + g.pitch - 1) / g.pitch;
    g.lbo = (g.rows * g.pitch * 16 + 127) / 128 * 128;
    // (the last rows of a tile's last taps may lie past the block: 64 bytes of slack)
    g.slot = ((cin0 + cin1) / 8 * g.lbo + 64 + 1023) / 1024 * 1024;
    // (a part's weights start on a 1024-byte boundary, the period of the widest swizzle)
    g.w1 = (27 * cout * cin0 * 2 + 1023) / 1024 * 1024;
    g.wbytes = g.w1 + (27 * cout * cin1 * 2 + 1023) / 1024 * 1024;
    // CTAs per SM: what the registers hold (56, 88 and 152 a thread for 16, 32 and 64 outputs), where the weights and a
    // ring of four planes fit their share of the shared memory
    int ctas = cout == 16 ? 3 : cout == 32 ? 2 : 1;
    for (; ctas >= 1; --ctas) {
        const int room = (226 * 1024 / ctas - 2560 - g.wbytes) / g.slot;
        if (226 * 1024 / ctas - 2560 > g.wbytes && room >= 4) {
            g.stages = std::min(room, kStagesWalk);
            break;
        }
    }
    if (!g.stages) return g;
    // as many chunks of planes as one wave of CTAs holds, one where it holds no tile of every column
    const long sms = wp_sm_count(), slots = ctas * sms, chunks = std::max(1L, std::min<long>(nz, slots / g.tiles));
    g.zc = (int)((nz + chunks - 1) / chunks);
    const long n = (long)g.tiles * ((nz + g.zc - 1) / g.zc), waves = (n + slots - 1) / slots;
    const double cin = cin0 + cin1, positions = (double)g.rows * g.pitch;
    const double start = 5.5 + positions * (0.0032 + 0.00016 * cin), plane = std::max(1.5, 0.0024 * positions) * cin / 16;
    const double walk = 3.0 + start * (0.4 + 0.6 * waves) + waves * g.zc * plane * std::min<long>(ctas, (n + sms - 1) / sms);
    const TileGeo t = tile_geo(nx, ny);
    const long nf = (long)t.nty * t.ntx * nz;
    const double fwd = 5.0 + (nf + 2 * sms - 1) / (2 * sms) * (8.6 * (cin1 ? 2 : 1) + 0.05 * cin);
    if (walk > fwd + 2.0) g.stages = 0;
    return g;
}

int* err_flag() {
    static int* d[64] = {nullptr};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(mu);
    if (!d[dev] && cudaMalloc((void**)&d[dev], sizeof(int)) == cudaSuccess) cudaMemset(d[dev], 0, sizeof(int));
    return d[dev];
}

template <int COUT>
cudaError_t launch_fwd(const CUtensorMap& x0, const CUtensorMap& w0, const CUtensorMap& x1, const CUtensorMap& w1,
                       int cin0, int cin1, int nparts, __nv_bfloat16* out, const float* bias,
                       const __nv_bfloat16* addend, const __nv_bfloat16* mask, int relu, int nx, int ny, int nz,
                       TileGeo tg, int* err, cudaStream_t s) {
    const size_t smem = 1024 + kStagesF * (kSlotA + kSlotB) + 16 * kStagesF + 32;
    int wh = -1;
    unsigned long long lim = wptc::kWaitLimitNs;
    if (!wp_take_withhold(WP_WAIT_SITE_CONV_PIPELINE, s, &wh, &lim)) wh = -1;
    auto k = conv3_fwd_kernel<COUT>;
    cudaError_t e = wp_set_smem(k, smem);
    if (e != cudaSuccess) return e;
    const long tiles = (long)tg.nty * tg.ntx * nz;
    k<<<(unsigned)tiles, kThreads, smem, s>>>(x0, w0, x1, w1, cin0, cin1, nparts, out, bias, addend, mask, relu, nx, ny,
                                              nz, tg, err, wh, lim);
    return cudaGetLastError();
}

template <int COUT>
cudaError_t launch_walk(const __nv_bfloat16* x0, const CUtensorMap& w0, const __nv_bfloat16* x1, const CUtensorMap& w1,
                        int cin0, int cin1, int nparts, __nv_bfloat16* out, const float* bias,
                        const __nv_bfloat16* addend, const __nv_bfloat16* mask, int relu, int nx, int ny, int nz,
                        WalkGeo g, int* err, cudaStream_t s) {
    const size_t smem = 1024 + (size_t)g.wbytes + (size_t)g.stages * g.slot + 16 * kStagesWalk + 8 + 32 + 32;
    int wh = -1;
    unsigned long long lim = wptc::kWaitLimitNs;
    if (!wp_take_withhold(WP_WAIT_SITE_CONV_PIPELINE, s, &wh, &lim)) wh = -1;
    auto k = conv3_walk_kernel<COUT>;
    cudaError_t e = wp_set_smem(k, smem);
    if (e != cudaSuccess) return e;
    const unsigned ctas = (unsigned)(g.tiles * ((nz + g.zc - 1) / g.zc));
    k<<<ctas, kWalkThreads, smem, s>>>(x0, w0, x1, w1, cin0, cin1, nparts, out, bias, addend, mask, relu, nx, ny, nz, g,
                                       err, wh, lim);
    return cudaGetLastError();
}

template <int COUT>
cudaError_t launch_wgrad(const CUtensorMap& xm, const CUtensorMap& gm, int cin, float* dw, int nx, int ny, int nz,
                         TileGeo tg, int* err, cudaStream_t s) {
    const size_t smem = 1024 + kStagesW * (kSlotWA + kSlotWB) + 16 * kStagesW + 32;
    int wh = -1;
    unsigned long long lim = wptc::kWaitLimitNs;
    if (!wp_take_withhold(WP_WAIT_SITE_CONV_PIPELINE, s, &wh, &lim)) wh = -1;
    auto k = conv3_wgrad_kernel<COUT>;
    cudaError_t e = wp_set_smem(k, smem);
    if (e != cudaSuccess) return e;
    const long ntiles = (long)tg.nty * tg.ntx * nz;
    const int groups = (27 + 128 / cin - 1) / (128 / cin);
    // about two CTAs per SM in total
    long chunks = (2L * wp_sm_count() + groups - 1) / groups;
    if (chunks > ntiles) chunks = ntiles;
    const int per = (int)((ntiles + chunks - 1) / chunks);
    chunks = (ntiles + per - 1) / per;
    k<<<dim3(groups, (unsigned)chunks), kThreads, smem, s>>>(xm, gm, cin, dw, nx, ny, nz, tg, ntiles, per, err, wh, lim);
    return cudaGetLastError();
}

}  // namespace

// Error flag of the tensor-core kernels on the current device (a bounded wait that gave up).
wp_status wp_conv_check_error(cudaStream_t s) {
    int* e = err_flag();
    if (!e) return WP_OK;
    int h = 0;
    WP_CUDA_TRY(cudaMemcpyAsync(&h, e, sizeof(int), cudaMemcpyDeviceToHost, s));
    WP_CUDA_TRY(cudaStreamSynchronize(s));
    if (h) {
        cudaMemsetAsync(e, 0, sizeof(int), s);
        wp_set_error_msg("tensor-core convolution: a pipeline wait gave up; the outputs of the call are invalid");
        return WP_ERR_DEVICE_WAIT;
    }
    return WP_OK;
}

// out = act(sum over parts conv(x_p, w_p) + bias + addend) [masked]; see the file comment.
wp_status wp_conv3_forward_impl(void* out, const void* x0, int cin0, const void* w0, const void* x1, int cin1,
                                const void* w1, const float* bias, int cout, int nx, int ny, int nz, int relu,
                                const void* addend, const void* mask, cudaStream_t s) {
    const int nparts = x1 ? 2 : 1;
    if (!out || !x0 || !w0 || !chan_ok(cin0) || (x1 && (!w1 || !chan_ok(cin1))) || !chan_ok(cout) || !pow2(nx) ||
        !pow2(ny) || nz < 1 || nz > 65535) {
        wp_set_error_msg("wp_conv3_forward: channels must be 16/32/64, nx and ny powers of two");
        return WP_ERR_INVALID_ARG;
    }
    const TileGeo tg = tile_geo(nx, ny);
    const WalkGeo wg = walk_geo(nx, ny, nz, cin0, x1 ? cin1 : 0, cout);
    // (its copies need 16-byte aligned inputs, as the tensor maps do)
    const bool walk = wg.stages > 0 && (((uintptr_t)x0 | (uintptr_t)x1) & 15u) == 0;
    auto maps = [&](CUtensorMap* mx, CUtensorMap* mw, const void* x, const void* w, int cin) {
        return walk ? map_weights(mw, w, cin, cout, 3)
                    : map_volume(mx, x, cin, nx, ny, nz, tg.yt, tg.xt) && map_weights(mw, w, cin, cout);
    };
    CUtensorMap mx0, mw0, mx1, mw1;
    if (!maps(&mx0, &mw0, x0, w0, cin0)) {
        wp_set_error_msg("wp_conv3_forward: tensor map encoding failed");
        return WP_ERR_CUDA;
    }
    if (x1) {
        if (!maps(&mx1, &mw1, x1, w1, cin1)) {
            wp_set_error_msg("wp_conv3_forward: tensor map encoding failed");
            return WP_ERR_CUDA;
        }
    } else {
        mx1 = mx0;
        mw1 = mw0;
        cin1 = cin0;
    }
    int* err = err_flag();
    if (!err) { wp_set_error_msg("wp_conv3_forward: error flag allocation failed"); return WP_ERR_CUDA; }
    auto o = static_cast<__nv_bfloat16*>(out);
    auto ad = static_cast<const __nv_bfloat16*>(addend);
    auto mk = static_cast<const __nv_bfloat16*>(mask);
    cudaError_t e;
    const int tok = wp_prof_start(s);
    auto go = [&](auto fwd, auto walkk) {
        return walk ? walkk(static_cast<const __nv_bfloat16*>(x0), mw0, static_cast<const __nv_bfloat16*>(x1), mw1, cin0, cin1,
                            nparts, o, bias, ad, mk, relu, nx, ny, nz, wg, err, s)
                    : fwd(mx0, mw0, mx1, mw1, cin0, cin1, nparts, o, bias, ad, mk, relu, nx, ny, nz, tg, err, s);
    };
    switch (cout) {
        case 16: e = go(launch_fwd<16>, launch_walk<16>); break;
        case 32: e = go(launch_fwd<32>, launch_walk<32>); break;
        default: e = go(launch_fwd<64>, launch_walk<64>); break;
    }
    const double flops = 2.0 * 27.0 * (cin0 + (x1 ? cin1 : 0)) * cout * (double)nx * ny * nz;
    wp_prof_stop(tok, "conv3_tc", flops, s);
    if (e != cudaSuccess) { wp_set_cuda_error(e, "conv3 forward", __FILE__, __LINE__); return WP_ERR_CUDA; }
    return WP_OK;
}

// dw[tap][cout][cin] += sum_v gy[v][co] x[v + off(tap)][ci] (FP32, caller zeroes dw)
wp_status wp_conv3_wgrad_impl(float* dw, const void* x, int cin, const void* gy, int cout, int nx, int ny, int nz,
                              cudaStream_t s) {
    if (!dw || !x || !gy || !chan_ok(cin) || !chan_ok(cout) || !pow2(nx) || !pow2(ny) || nz < 1 || nz > 65535) {
        wp_set_error_msg("wp_conv3_wgrad: channels must be 16/32/64, nx and ny powers of two");
        return WP_ERR_INVALID_ARG;
    }
    const TileGeo tg = tile_geo(nx, ny);
    CUtensorMap mx, mg;
    if (!map_volume(&mx, x, cin, nx, ny, nz, tg.yt, tg.xt) || !map_volume(&mg, gy, cout, nx, ny, nz, tg.yt, tg.xt)) {
        wp_set_error_msg("wp_conv3_wgrad: tensor map encoding failed");
        return WP_ERR_CUDA;
    }
    int* err = err_flag();
    if (!err) { wp_set_error_msg("wp_conv3_wgrad: error flag allocation failed"); return WP_ERR_CUDA; }
    cudaError_t e;
    const int tok = wp_prof_start(s);
    switch (cout) {
        case 16: e = launch_wgrad<16>(mx, mg, cin, dw, nx, ny, nz, tg, err, s); break;
        case 32: e = launch_wgrad<32>(mx, mg, cin, dw, nx, ny, nz, tg, err, s); break;
        default: e = launch_wgrad<64>(mx, mg, cin, dw, nx, ny, nz, tg, err, s); break;
    }
    wp_prof_stop(tok, "conv3_wgrad_tc", 2.0 * 27.0 * cin * cout * (double)nx * ny * nz, s);
    if (e != cudaSuccess) { wp_set_cuda_error(e, "conv3 wgrad", __FILE__, __LINE__); return WP_ERR_CUDA; }
    return WP_OK;
}

extern "C" CUWHHD_API wp_status wp_conv3_forward(void* out, const void* x0, int cin0, const void* w0, const void* x1,
                                                 int cin1, const void* w1, const float* bias, int cout, int nx, int ny,
                                                 int nz, int relu, const void* addend, const void* mask, void* stream) {
    wp_status st = wp_conv3_forward_impl(out, x0, cin0, w0, x1, cin1, w1, bias, cout, nx, ny, nz, relu, addend, mask,
                                         (cudaStream_t)stream);
    if (st != WP_OK) return st;
    return wp_conv_check_error((cudaStream_t)stream);
}

extern "C" CUWHHD_API wp_status wp_conv3_wgrad(float* dw, const void* x, int cin, const void* gy, int cout, int nx,
                                               int ny, int nz, void* stream) {
    wp_status st = wp_conv3_wgrad_impl(dw, x, cin, gy, cout, nx, ny, nz, (cudaStream_t)stream);
    if (st != WP_OK) return st;
    return wp_conv_check_error((cudaStream_t)stream);
}
