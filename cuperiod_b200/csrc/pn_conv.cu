// The proposal network's convolutions and matrix products as implicit GEMMs on the
// tensor cores (sm_100a), forward and backward, and the composite passes.
//
// The width-7, stride-2, padding-3 convolution of 64 channels needs no patch matrix:
// split by the parity of the position, output row o of tap k reads position 2o + k - 3,
// which is row o + (k >> 1) - 2 (k even) or o + (k >> 1) - 1 (k odd) of one parity plane.
// TMA views an activation [B][L][64] as {64, parity 2, L / 2, B}: one box is a run of
// rows of one plane, zero outside the curve, and every tap of that plane is the same
// rows shifted by whole 128-byte rows of the swizzled tile.  The backward passes use the
// same views, and read operands M- or N-major where the forward pass reads them K-major,
// so nothing is transposed in memory.
//
//  * conv_kernel<false>: Y = relu(conv(X) + b); 128 output rows a tile, M = 128, N = 64,
//    K = 7 x 64; the weights stay in shared memory.
//  * conv_kernel<true>: the input gradient of a tile of 128 row pairs, both parities, with
//    the ReLU mask of the input; each tap has its own accumulator, since its product is
//    rounded to bf16 before the taps are added.
//  * conv_wgrad_kernel: weight and bias gradients, M = 7 taps x 64 channels (+ a block of
//    ones, whose product is the bias gradient), N = 64, K = the rows.
//  * conv0_*: the first layer (two input channels, K = 14).
//  * fc_kernel: the MLP's products, K split over a cluster and summed through distributed
//    shared memory in rank order.
//
// With the patch matrices, transposes and column sums in memory a pass over 1,024 curves
// took 2,630 us and a training step of 256 curves 3,370 us; as built 240 and 374 us.
//
// Every wait on an mbarrier is bounded; one that runs out sets the error flag, after which
// the CTA's roles finish their loops without further waits or stores.
#include <math.h>

#include "../../include/bls_proposal.h"
#include "bls_launch.h"
#include "pn_net.h"
#include "pn_ptx.cuh"

namespace blsb200 {
namespace pn {
namespace {

constexpr int kCh = 64;
constexpr int kTaps = 7;
constexpr int kRows = 128;                          // rows of one output tile
constexpr uint32_t kTile = kRows * 128;             // a tile of 128 rows x 64 bf16
constexpr uint32_t kWTap = 64 * 128;                // one tap's weights
constexpr uint32_t kWeights = kTaps * kWTap;
constexpr int kWinRows = 136;                       // 128 rows and the taps' shifts, to 8
constexpr uint32_t kWin = kWinRows * 128;
constexpr int kMaxStages = 4;
constexpr int kConvThreads = 320;                   // producer, MMA, eight epilogue warps
constexpr uint32_t kSmemMax = 226 * 1024;

__device__ __forceinline__ uint32_t saddr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* tm, int x, int y, int z,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* tm, int x, int y, int z,
                                            int w, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tm, int x, int y, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(tm)),
                 "r"(x), "r"(y), "r"(src)
                 : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* tm, int x, int y, int z, int w,
                                             uint32_t src) {
    asm volatile(
        "cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(
            reinterpret_cast<uint64_t>(tm)),
        "r"(x), "r"(y), "r"(z), "r"(w), "r"(src)
        : "memory");
}
__device__ __forceinline__ void bulk_commit() {
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() {
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ uint32_t tmem_alloc(uint32_t slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    return 0;
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols)
                 : "memory");
}
// 32 consecutive fp32 columns of the accumulator for this warp's 32 rows.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10,"
        " %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27,"
        " %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w)
                 : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// (a, b) where the two bf16 of `act` are positive, else 0
__device__ __forceinline__ uint32_t pack2_masked(float a, float b, uint32_t act) {
    const float m0 = __uint_as_float(act << 16), m1 = __uint_as_float(act & 0xffff0000u);
    return pack2(m0 > 0.0f ? a : 0.0f, m1 > 0.0f ? b : 0.0f);
}
// 16-byte chunk j of row r of a 128-byte-swizzled tile
__device__ __forceinline__ uint32_t chunk(uint32_t tile, int r, int j) {
    return tile + (uint32_t)r * 128u + (uint32_t)((j ^ (r & 7)) << 4);
}

// ---- the convolution and its input gradient ---------------------------------------

// Backward: the masks' stages (2 tiles each) are their own, since they are read last: held
// with the input's they kept the next loads from starting until the epilogue was over.
template <bool BWD, bool WINDOW>
__host__ __device__ constexpr int conv_mask_stages() { return !BWD ? 0 : WINDOW ? 2 : 1; }

struct ConvArgs {
    int n_tiles;            // tiles of 128 rows (row pairs)
    int L;                  // rows (pairs) of one curve: 64 or a multiple of 128
    int stages;             // of the input
    const float* bias;      // forward
    int* error_flag;
};

template <bool BWD, bool WINDOW>
__host__ __device__ constexpr uint32_t conv_stage_bytes() {
    return BWD ? (WINDOW ? kWin : 4 * kTile) : (WINDOW ? 2 * kWin : kTaps * kTile);
}

// BWD: tmIn is dY as {64, L, B}, tmOut dX and tmMask the convolution's input, both as
// {64, 2, L, B}; forward: tmIn is X as {64, 2, L, B}, tmOut Y as {64, B L}.  WINDOW: a tile
// lies in one curve and its taps share windows; else (L = 64) it is two curves, a tap a
// tile.  Persistent, one CTA an SM, two accumulators: the epilogue of a tile overlaps the
// next tile's products.  Bound by HBM: at 1,024 curves layer 2 (2048 -> 1024 positions)
// reads 268 MB and writes 134 MB; a tile's loads are 34 KB with the shared windows, where
// a tile per tap is 112 KB, above what L2 hands an SM in the time HBM takes.
template <bool BWD, bool WINDOW>
__global__ void __launch_bounds__(kConvThreads, 1)
    conv_kernel(const __grid_constant__ CUtensorMap tmIn, const __grid_constant__ CUtensorMap tmW,
                const __grid_constant__ CUtensorMap tmOut,
                const __grid_constant__ CUtensorMap tmMask, const ConvArgs a) {
    constexpr uint32_t kStage = conv_stage_bytes<BWD, WINDOW>();
    constexpr int kMasks = BWD ? conv_mask_stages<BWD, WINDOW>() : 1;
    // accumulator columns: forward 64 a tile, two tiles; backward 64 a tap, three taps of
    // the even positions and four of the odd ones (N = 32 and halves of the channels
    // instead took 52 cycles a product, N = 64 about 60: both read all of A)
    constexpr int kAcc = BWD ? 3 * 64 : 64;
    constexpr int kCols = BWD ? 512 : 128;
    constexpr int kOut = BWD ? 2 : 1;                          // output tiles of a tile
    extern __shared__ uint8_t dsm_raw[];
    __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages];
    __shared__ __align__(8) uint64_t tfull_bar[2], tempty_bar[2], w_bar;
    __shared__ __align__(8) uint64_t mfull_bar[2], mempty_bar[2];
    __shared__ float s_bias[kCh];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sW = (saddr(dsm_raw) + 1023u) & ~1023u;
    const uint32_t sOut = sW + kWeights;                       // 2 x kOut tiles
    const uint32_t sIn = sOut + 2 * kOut * kTile;
    const uint32_t fb = saddr(full_bar), eb = saddr(empty_bar), tf = saddr(tfull_bar),
                   te = saddr(tempty_bar), wb = saddr(&w_bar), mf = saddr(mfull_bar),
                   me = saddr(mempty_bar);
    const uint32_t sMask = sIn + a.stages * kStage;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(fb + 8 * s, 1);
            mbar_init(eb + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(tf + 8 * s, 1);
            mbar_init(te + 8 * s, BWD ? 4 : 8);         // the warps that read it
            mbar_init(mf + 8 * s, 1);
            mbar_init(me + 8 * s, 1);
        }
        mbar_init(wb, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(saddr(&tmem_slot), kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) dependents_may_launch();
    wait_for_prior();
    if (!BWD) {
        if (threadIdx.x < kCh) s_bias[threadIdx.x] = a.bias[threadIdx.x];
        __syncthreads();
    }
    const uint32_t tmem = tmem_slot;
    const int S = a.stages;
    volatile int* dead = &abort_s;
    auto give_up = [&] {
        abort_s = 1;
        atomicExch(a.error_flag, 1);
    };

    if (threadIdx.x == 0) {
        mbar_expect_tx(wb, kWeights);
        for (int k = 0; k < kTaps; ++k) tma_load_2d(sW + k * kWTap, &tmW, k * 64, 0, wb);
        int n = 0;
        for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++n) {
            const int st = n % S;
            if (n >= S && !mbar_wait(eb + 8 * st, (uint32_t)(n / S - 1) & 1u)) {
                give_up();
                break;
            }
            if (*dead) break;
            const uint32_t in = sIn + st * kStage, bar = fb + 8 * st;
            const int row = t * kRows;
            const int b = row / a.L, o0 = row - b * a.L;
            mbar_expect_tx(bar, kStage);
            if (!BWD) {
                if (WINDOW) {
                    tma_load_4d(in, &tmIn, 0, 1, o0 - 2, b, bar);
                    tma_load_4d(in + kWin, &tmIn, 0, 0, o0 - 1, b, bar);
                } else {
                    for (int k = 0; k < kTaps; ++k)
                        tma_load_4d(in + k * kTile, &tmIn, 0, (k & 1) ^ 1,
                                    o0 + (k >> 1) - ((k & 1) ? 1 : 2), b, bar);
                }
            } else {
                if (WINDOW) tma_load_3d(in, &tmIn, 0, o0 - 1, b, bar);
                else
                    for (int k = 0; k < 4; ++k)
                        tma_load_3d(in + k * kTile, &tmIn, 0, o0 - 1 + k, b, bar);
                const int ms = n % kMasks;
                if (n >= kMasks && !mbar_wait(me + 8 * ms, (uint32_t)(n / kMasks - 1) & 1u)) {
                    give_up();
                    break;
                }
                const uint32_t mask = sMask + ms * 2 * kTile;
                mbar_expect_tx(mf + 8 * ms, 2 * kTile);
                tma_load_4d(mask, &tmMask, 0, 0, o0, b, mf + 8 * ms);
                tma_load_4d(mask + kTile, &tmMask, 0, 1, o0, b, mf + 8 * ms);
            }
        }
    } else if (threadIdx.x == 32) {
        constexpr uint32_t idesc = bf16_idesc(128, 64) | (BWD ? kIdescBMn : 0u);
        const uint64_t dW = BWD ? sw128_mn_desc(sW, 1024) : sw128_desc(sW);
        bool ok = mbar_wait(wb, 0u);
        if (!ok) give_up();
        int n = 0;
        for (int t = blockIdx.x; ok && t < a.n_tiles; t += gridDim.x, ++n) {
            const int st = n % S;
            const uint32_t in = sIn + st * kStage;
            if (!mbar_wait(fb + 8 * st, (uint32_t)(n / S) & 1u)) ok = false;
            const uint64_t dA = sw128_desc(in);
#pragma unroll
            for (int e = 0; e < (BWD ? 2 : 1); ++e) {
                if (!ok) break;
                // accumulator and how often it was used before
                const int acc = BWD ? e : n & 1, use = BWD ? n : n / 2;
                if (use >= 1 && !mbar_wait(te + 8 * acc, (uint32_t)(use - 1) & 1u)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t D = tmem + acc * kAcc;
#pragma unroll
                for (int k = BWD ? e ^ 1 : 0; k < kTaps; k += BWD ? 2 : 1) {
                    // forward: rows of the tap's parity plane.  Backward: parity 0 takes
                    // taps 1, 3, 5 at rows +1, 0, -1, parity 1 taps 0, 2, 4, 6 at rows
                    // +2 .. -1; the window starts at row -1, and a tap has its own
                    // accumulator
                    const int sh = (k & 1) ? 2 - (k >> 1) : 3 - (k >> 1);
                    const uint32_t A = BWD ? sh * (WINDOW ? 128 : kTile)
                                       : WINDOW ? (k & 1) * kWin + (k >> 1) * 128
                                                : k * kTile;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_bf16(BWD ? D + (k >> 1) * 64 : D, desc_at(dA, A + kk * 32),
                                  desc_at(dW, k * kWTap + kk * (BWD ? 2048 : 32)),
                                  idesc, kk == 0 && (BWD || k == 0) ? 0u : 1u);
                }
                umma_commit(tf + 8 * acc);
            }
            if (!ok) {
                give_up();
                break;
            }
            umma_commit(eb + 8 * st);
        }
    } else if (warp >= 2) {
        // warps 2-5 take channels 0-31 (backward: the even positions), 6-9 the others
        const int quarter = warp & 3, part = (warp - 2) >> 2, r = quarter * 32 + lane;
        bool ok = true;
        int n = 0;
        for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++n) {
            const int ms = n % kMasks;
            const uint32_t out = sOut + (n & 1) * kOut * kTile;
            const int acc = BWD ? part : n & 1, use = BWD ? n : n / 2;
            if (ok) ok = mbar_wait(tf + 8 * acc, (uint32_t)use & 1u) && !*dead;
            if (BWD && ok) ok = mbar_wait(mf + 8 * ms, (uint32_t)(n / kMasks) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok && lane == 0) give_up();
            auto release = [&] {                    // the accumulator is read
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(te + 8 * acc);
            };
            if (ok) {
                tc_fence_after();
                const uint32_t D = tmem + ((uint32_t)(quarter * 32) << 16) + acc * kAcc;
                if (BWD) {
                    const uint32_t mask = sMask + (ms * 2 + part) * kTile;
#pragma unroll 1
                    for (int c = 0; c < 2; ++c) {
                        // the taps' products are rounded to bf16 one by one and added
                        // in tap order
                        float sum[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) sum[i] = 0.0f;
#pragma unroll 1
                        for (int k = 0; k < 3 + part; ++k) {
                            float v[32];
                            tmem_ld32(D + k * 64 + c * 32, v);
#pragma unroll
                            for (int i = 0; i < 32; i += 2) {
                                const uint32_t p = pack2(v[i], v[i + 1]);
                                sum[i] += __uint_as_float(p << 16);
                                sum[i + 1] += __uint_as_float(p & 0xffff0000u);
                            }
                        }
                        if (c == 1) release();
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint4 m = lds128(chunk(mask, r, c * 4 + j));
                            sts128(chunk(out + part * kTile, r, c * 4 + j),
                                   make_uint4(pack2_masked(sum[8 * j], sum[8 * j + 1], m.x),
                                              pack2_masked(sum[8 * j + 2], sum[8 * j + 3], m.y),
                                              pack2_masked(sum[8 * j + 4], sum[8 * j + 5], m.z),
                                              pack2_masked(sum[8 * j + 6], sum[8 * j + 7], m.w)));
                        }
                    }
                } else {
                    float v[32];
                    tmem_ld32(D + part * 32, v);
                    release();
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            v[8 * j + i] =
                                fmaxf(v[8 * j + i] + s_bias[part * 32 + 8 * j + i], 0.0f);
                        sts128(chunk(out, r, part * 4 + j),
                               make_uint4(pack2(v[8 * j], v[8 * j + 1]),
                                          pack2(v[8 * j + 2], v[8 * j + 3]),
                                          pack2(v[8 * j + 4], v[8 * j + 5]),
                                          pack2(v[8 * j + 6], v[8 * j + 7])));
                    }
                }
            }
            // (the stores that may still read the other buffer are those of tile n - 1, so
            // past this barrier it is free for tile n + 1)
            if (threadIdx.x == 64) bulk_wait_read<0>();
            fence_async_smem();
            epi_sync();
            if (threadIdx.x == 64) {
                if (BWD) mbar_arrive(me + 8 * ms);          // the masks are read
                if (ok && !*dead) {
                    const int row = t * kRows;
                    if (BWD) {
                        const int b = row / a.L, o0 = row - b * a.L;
                        tma_store_4d(&tmOut, 0, 0, o0, b, out);
                        tma_store_4d(&tmOut, 0, 1, o0, b, out + kTile);
                    } else {
                        tma_store_2d(&tmOut, 0, row, out);
                    }
                }
                bulk_commit();
            }
        }
        if (threadIdx.x == 64) bulk_wait_all();
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_free(tmem, kCols);
}

// ---- weight gradients -----------------------------------------------------------------

constexpr int kWgRows = 64;                         // rows of one block
constexpr int kWgWinRows = 72;
constexpr uint32_t kWgWin = kWgWinRows * 128;
constexpr uint32_t kWgStage = 64 * 128 + 2 * kWgWin;        // dY, odd-plane and even-plane rows
constexpr int kWgStages = 6;
constexpr int kWgThreads = 192;                     // producer, MMA, four reading warps

struct WgradArgs {
    int n_blocks;           // blocks of 64 rows
    int L;                  // rows of one curve
    float* part;            // per CTA [8][64 n][64]: 7 taps of channels, then the bias row
    int* error_flag;
};
constexpr int kWgPart = 8 * 64 * 64;

// dW[n][k*64 + c] += sum over rows (b, o) of dY[b, o][n] X[b, 2o + k - 3][c], and db.  Each
// CTA sums its share of the 64-row blocks in tensor memory -- four products of M = 128
// (two taps, one row apart in their window, or tap 5 and the block of ones), N = 64 --
// and writes its sums to the workspace, which wgrad_sum_kernel adds up (adding them to the
// gradient with atomics took three times the products' time).
__global__ void __launch_bounds__(kWgThreads, 1)
    conv_wgrad_kernel(const __grid_constant__ CUtensorMap tmDy,
                      const __grid_constant__ CUtensorMap tmX, const WgradArgs a) {
    extern __shared__ uint8_t dsm_raw[];
    __shared__ __align__(8) uint64_t full_bar[kWgStages], empty_bar[kWgStages];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sIn = (saddr(dsm_raw) + 1023u) & ~1023u;
    const uint32_t sOnes = sIn + kWgStages * kWgStage;
    const uint32_t fb = saddr(full_bar), eb = saddr(empty_bar), db = saddr(&done_bar);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kWgStages; ++s) {
            mbar_init(fb + 8 * s, 1);
            mbar_init(eb + 8 * s, 1);
        }
        mbar_init(db, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (uint32_t i = threadIdx.x; i < 64 * 128 / 16; i += kWgThreads)
        sts128(sOnes + 16 * i, make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u));
    fence_async_smem();
    if (warp == 1) tmem_alloc(saddr(&tmem_slot), 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) dependents_may_launch();
    wait_for_prior();
    const uint32_t tmem = tmem_slot;
    volatile int* dead = &abort_s;
    auto give_up = [&] {
        abort_s = 1;
        atomicExch(a.error_flag, 1);
    };
    if (threadIdx.x == 0) {
        int n = 0;
        for (int t = blockIdx.x; t < a.n_blocks; t += gridDim.x, ++n) {
            const int st = n % kWgStages;
            if (n >= kWgStages && !mbar_wait(eb + 8 * st, (uint32_t)(n / kWgStages - 1) & 1u)) {
                give_up();
                break;
            }
            if (*dead) break;
            const uint32_t in = sIn + st * kWgStage, bar = fb + 8 * st;
            const int row = t * kWgRows;
            const int b = row / a.L, o0 = row - b * a.L;
            mbar_expect_tx(bar, kWgStage);
            tma_load_3d(in, &tmDy, 0, o0, b, bar);
            tma_load_4d(in + 8192, &tmX, 0, 1, o0 - 2, b, bar);
            tma_load_4d(in + 8192 + kWgWin, &tmX, 0, 0, o0 - 1, b, bar);
        }
    } else if (threadIdx.x == 32) {
        constexpr uint32_t idesc = bf16_idesc(128, 64) | kIdescAMn | kIdescBMn;
        int n = 0;
        for (int t = blockIdx.x; t < a.n_blocks; t += gridDim.x, ++n) {
            const int st = n % kWgStages;
            if (!mbar_wait(fb + 8 * st, (uint32_t)(n / kWgStages) & 1u)) {
                give_up();
                break;
            }
            tc_fence_after();
            const uint32_t dy = sIn + st * kWgStage, p1 = dy + 8192, p0 = p1 + kWgWin;
            const uint64_t dB = sw128_mn_desc(dy, 1024);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                // taps 0, 2 | 4, 6 of the odd plane, 1, 3 | 5 of the even one
                const uint32_t A = (m < 2 ? p1 : p0) + (m & 1) * 256;
                const uint64_t dA = sw128_mn_desc(A, m < 3 ? 128u : sOnes - A);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    umma_bf16(tmem + m * 64, desc_at(dA, kk * 2048), desc_at(dB, kk * 2048), idesc,
                              n > 0 || kk > 0 ? 1u : 0u);
            }
            umma_commit(eb + 8 * st);
        }
        umma_commit(db);            // arrives once every product above has completed
    }
    __syncwarp();
    if (warp >= 2) {
        bool ok = mbar_wait(db, 0u);
        ok = __all_sync(0xffffffffu, ok) && !*dead;
        if (!ok && lane == 0) give_up();
        tc_fence_after();
        if (ok && blockIdx.x < a.n_blocks) {
            const int quarter = warp & 3;
            const int half = quarter >> 1, c = (quarter & 1) * 32 + lane;
            const int taps[4][2] = {{0, 2}, {4, 6}, {1, 3}, {5, 7}};
            float* part = a.part + (int64_t)blockIdx.x * kWgPart;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                float* p = part + taps[m][half] * 64 * 64 + c;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float v[32];
                    tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + m * 64 + h * 32, v);
#pragma unroll
                    for (int j = 0; j < 32; ++j) p[(h * 32 + j) * 64] = v[j];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_free(tmem, 256);
}

// gw, gb += the sums of n_parts partial gradients, in order: a block takes one tap and four
// rows n, its 4 x 64 channels by 4 groups of threads that each sum a quarter of the parts.
__global__ void __launch_bounds__(1024)
    wgrad_sum_kernel(const float* part, int n_parts, float* gw, float* gb) {
    __shared__ float sum[4][256];
    const int tap = blockIdx.x >> 4, i = threadIdx.x & 255, group = threadIdx.x >> 8;
    const int n = (blockIdx.x & 15) * 4 + (i >> 6), c = i & 63;
    const float* p = part + tap * 64 * 64 + n * 64 + c;
    const int per = (n_parts + 3) / 4, end = min(n_parts, (group + 1) * per);
    float s = 0.0f;
    dependents_may_launch();
    wait_for_prior();
#pragma unroll 8
    for (int z = group * per; z < end; ++z) s += p[(int64_t)z * kWgPart];
    sum[group][i] = s;
    __syncthreads();
    if (group == 0) {
        s = (sum[0][i] + sum[1][i]) + (sum[2][i] + sum[3][i]);
        if (tap < 7) gw[n * (kTaps * kCh) + tap * kCh + c] += s;
        else if (c == 0) gb[n] += s;
    }
}

// ---- the first layer: two input channels ------------------------------------------------

// Elements of x are read two by two (one position) when the array is 4-byte aligned.
template <bool PAIRS>
__device__ __forceinline__ uint32_t position(const __nv_bfloat16* x, int i) {
    if (PAIRS) return __ldg(reinterpret_cast<const uint32_t*>(x) + i);
    const unsigned short* p = reinterpret_cast<const unsigned short*>(x) + 2 * (int64_t)i;
    return (uint32_t)__ldg(p) | ((uint32_t)__ldg(p + 1) << 16);
}

struct Conv0Args {
    const __nv_bfloat16* x;         // [B][2 L][2]
    const __nv_bfloat16* w;         // [64][16], columns 14 and 15 zero
    const float* bias;
    int n_tiles, L;
    int* error_flag;
};

constexpr int kConv0Ctas = 7;       // a CTA holds 64 of the 512 tensor-memory columns

// Y = relu(conv(x) + b), 128 rows a tile: a thread builds its row's 14 inputs in the
// unswizzled core-matrix layout, one product of K = 16, and stores through TMA.  Bound by
// the write of Y (268 MB at 1,024 curves); several CTAs an SM overlap one another's steps.
template <bool PAIRS>
__global__ void __launch_bounds__(128)
    conv0_kernel(const __grid_constant__ CUtensorMap tmOut, const Conv0Args a) {
    extern __shared__ uint8_t dsm_raw[];
    __shared__ __align__(128) uint8_t sa[128 * 32];
    __shared__ __align__(128) uint8_t sw[64 * 32];
    __shared__ float s_bias[kCh];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t out = (saddr(dsm_raw) + 1023u) & ~1023u;
    const uint32_t A = saddr(sa), W = saddr(sw), db = saddr(&done_bar);
    if (tid == 0) {
        mbar_init(db, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(saddr(&tmem_slot), 64);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) dependents_may_launch();
    wait_for_prior();
    if (tid < kCh) s_bias[tid] = a.bias[tid];
    {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.w) + tid);   // row tid / 2, half tid & 1
        const int r = tid >> 1;
        sts128(W + (uint32_t)((r >> 3) * 256 + (tid & 1) * 128 + (r & 7) * 16), v);
    }
    const uint32_t tmem = tmem_slot;
    const int L_in = 2 * a.L;
    auto load_row = [&](int t, uint32_t (&v)[7]) {
        const int row = t * kRows + tid;
        const int b = row / a.L, o = row - b * a.L;
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const int i = 2 * o + k - 3;
            v[k] = i >= 0 && i < L_in ? position<PAIRS>(a.x + (int64_t)b * L_in * 2, i) : 0u;
        }
    };
    uint32_t v[7];
    if (blockIdx.x < a.n_tiles) load_row(blockIdx.x, v);
    bool ok = true;
    uint32_t ph = 0u;
    for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ph ^= 1u) {
        const uint32_t at = A + (uint32_t)((tid >> 3) * 256 + (tid & 7) * 16);
        sts128(at, make_uint4(v[0], v[1], v[2], v[3]));
        sts128(at + 128, make_uint4(v[4], v[5], v[6], 0u));
        fence_async_smem();
        if (tid == 0) bulk_wait_read<0>();          // the previous tile's store
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            umma_bf16(tmem, plain_desc(A, 128, 256), plain_desc(W, 128, 256), bf16_idesc(128, 64),
                      0u);
            umma_commit(db);
        }
        if (t + (int)gridDim.x < a.n_tiles) load_row(t + gridDim.x, v);
        if (ok) ok = mbar_wait(db, ph);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float f[32];
                tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + c * 32, f);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        f[8 * j + i] = fmaxf(f[8 * j + i] + s_bias[c * 32 + 8 * j + i], 0.0f);
                    sts128(chunk(out, tid, c * 4 + j),
                           make_uint4(pack2(f[8 * j], f[8 * j + 1]),
                                      pack2(f[8 * j + 2], f[8 * j + 3]),
                                      pack2(f[8 * j + 4], f[8 * j + 5]),
                                      pack2(f[8 * j + 6], f[8 * j + 7])));
                }
            }
            tc_fence_before();
        } else if ((tid & 31) == 0) {
            atomicExch(a.error_flag, 1);
        }
        fence_async_smem();
        ok = __syncthreads_and(ok);
        if (tid == 0 && ok) {
            tma_store_2d(&tmOut, 0, t * kRows, out);
            bulk_commit();
        }
        if (!ok) break;             // the same for every thread
    }
    if (tid == 0) bulk_wait_all();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 64);
}

struct Wgrad0Args {
    const __nv_bfloat16* x;
    int n_blocks, L;
    float* part;            // per CTA [16][64 n]: 14 inputs, the bias, nothing
    int* error_flag;
};
constexpr int kWg0Stages = 4;
constexpr int kWg0Ctas = 3;         // an SM: laying out a block's rows is what takes the time
constexpr uint32_t kWg0Stage = 2 * 64 * 128;
constexpr int kWg0Part = 16 * 64;

// dW0[n][k*2 + c] += sum over rows of dY[b, o][n] x[b, 2o + k - 3][c], and db0, the same way:
// two warps lay out a block's 64 rows of 14 inputs and a 1 (the bias) as the M-major
// operand, M = 128 of which 15 are used, N = 64, K = 64 rows a block.
template <bool PAIRS>
__global__ void __launch_bounds__(128, kWg0Ctas)
    conv0_wgrad_kernel(const __grid_constant__ CUtensorMap tmDy, const Wgrad0Args a) {
    extern __shared__ uint8_t dsm_raw[];
    __shared__ __align__(8) uint64_t full_bar[kWg0Stages], empty_bar[kWg0Stages];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sIn = (saddr(dsm_raw) + 1023u) & ~1023u;
    const uint32_t fb = saddr(full_bar), eb = saddr(empty_bar), db = saddr(&done_bar);
    if (tid == 0) {
        for (int s = 0; s < kWg0Stages; ++s) {
            mbar_init(fb + 8 * s, 3);           // the load, and the two laying-out warps
            mbar_init(eb + 8 * s, 1);
        }
        mbar_init(db, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // M columns past the 16 of a row's inputs stay zero; the second half of M = 128 reads
    // the first again
    for (uint32_t i = tid; i < kWg0Stages * kWg0Stage / 16; i += 128)
        sts128(sIn + 16 * i, make_uint4(0u, 0u, 0u, 0u));
    fence_async_smem();
    if (warp == 0) tmem_alloc(saddr(&tmem_slot), 64);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) dependents_may_launch();
    wait_for_prior();
    const uint32_t tmem = tmem_slot;
    volatile int* dead = &abort_s;
    auto give_up = [&] {
        abort_s = 1;
        atomicExch(a.error_flag, 1);
    };
    if (tid == 0) {
        int n = 0;
        for (int t = blockIdx.x; t < a.n_blocks; t += gridDim.x, ++n) {
            const int st = n % kWg0Stages;
            if (n >= kWg0Stages && !mbar_wait(eb + 8 * st, (uint32_t)(n / kWg0Stages - 1) & 1u)) {
                give_up();
                break;
            }
            if (*dead) break;
            mbar_expect_tx(fb + 8 * st, 64 * 128);
            tma_load_2d(sIn + st * kWg0Stage, &tmDy, 0, t * 64, fb + 8 * st);
        }
    } else if (tid == 32) {
        constexpr uint32_t idesc = bf16_idesc(128, 64) | kIdescAMn | kIdescBMn;
        int n = 0;
        for (int t = blockIdx.x; t < a.n_blocks; t += gridDim.x, ++n) {
            const int st = n % kWg0Stages;
            if (!mbar_wait(fb + 8 * st, (uint32_t)(n / kWg0Stages) & 1u)) {
                give_up();
                break;
            }
            tc_fence_after();
            const uint32_t dy = sIn + st * kWg0Stage;
            const uint64_t dA = sw128_mn_desc(dy + 64 * 128, 0), dB = sw128_mn_desc(dy, 1024);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                umma_bf16(tmem, desc_at(dA, kk * 2048), desc_at(dB, kk * 2048), idesc, n > 0 || kk > 0 ? 1u : 0u);
            umma_commit(eb + 8 * st);
        }
        umma_commit(db);
    } else if (warp >= 2) {
        const int r = tid - 64, L_in = 2 * a.L;
        auto load_row = [&](int t, uint32_t (&v)[7]) {
            const int row = t * 64 + r;
            const int b = row / a.L, o = row - b * a.L;
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const int i = 2 * o + k - 3;
                v[k] = i >= 0 && i < L_in ? position<PAIRS>(a.x + (int64_t)b * L_in * 2, i) : 0u;
            }
        };
        uint32_t v[7];
        load_row(blockIdx.x, v);
        bool ok = true;
        int n = 0;
        for (int t = blockIdx.x; t < a.n_blocks; t += gridDim.x, ++n) {
            const int st = n % kWg0Stages;
            if (n >= kWg0Stages) ok = mbar_wait(eb + 8 * st, (uint32_t)(n / kWg0Stages - 1) & 1u);
            ok = __all_sync(0xffffffffu, ok) && !*dead;
            if (!ok) {
                if (lane == 0) give_up();
                break;
            }
            const uint32_t p = sIn + st * kWg0Stage + 64 * 128;
            sts128(chunk(p, r, 0), make_uint4(v[0], v[1], v[2], v[3]));
            sts128(chunk(p, r, 1), make_uint4(v[4], v[5], v[6], 0x3f80u));
            if (t + (int)gridDim.x < a.n_blocks) load_row(t + gridDim.x, v);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(fb + 8 * st);
        }
    }
    __syncwarp();
    bool ok = mbar_wait(db, 0u);
    ok = __all_sync(0xffffffffu, ok) && !*dead;
    if (!ok && lane == 0) give_up();
    tc_fence_after();
    if (ok && warp == 0) {
        float* part = a.part + (int64_t)blockIdx.x * kWg0Part + lane * 64;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v[32];
            tmem_ld32(tmem + h * 32, v);
            if (lane < 16)
#pragma unroll
                for (int j = 0; j < 32; ++j) part[h * 32 + j] = v[j];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 64);
}

// gw, gb += those partial sums: 16 runs of them, then the runs in order.
__global__ void __launch_bounds__(1024)
    wgrad0_sum_kernel(const float* part, int n_parts, float* gw, float* gb) {
    __shared__ float sum[16][64];
    const int k = blockIdx.x, n = threadIdx.x & 63, run = threadIdx.x >> 6;
    const int per = (n_parts + 15) / 16, end = min(n_parts, (run + 1) * per);
    float s = 0.0f;
    dependents_may_launch();
    wait_for_prior();
#pragma unroll 4
    for (int z = run * per; z < end; ++z) s += part[(int64_t)z * kWg0Part + k * 64 + n];
    sum[run][n] = s;
    __syncthreads();
    if (run != 0) return;
    for (int g = 1; g < 16; ++g) s += sum[g][n];
    if (k < 14) gw[n * 16 + k] += s;
    else gb[n] += s;
}

// db[n] += sum over rows of g[m][n] (bf16): a block takes 64 columns, its warps rows in turn.
__global__ void __launch_bounds__(256) bias_grad_kernel(const __nv_bfloat16* g, int M, int N,
                                                        float* db) {
    __shared__ float sum[8][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = blockIdx.x * 64;
    float s0 = 0.0f, s1 = 0.0f;
    dependents_may_launch();
    wait_for_prior();
#pragma unroll 8
    for (int m = warp; m < M; m += 8) {
        // (not __ldg: the kernel that writes g may still run when this one is launched)
        const uint32_t v = reinterpret_cast<const uint32_t*>(g + (int64_t)m * N + n)[lane];
        s0 += __uint_as_float(v << 16);
        s1 += __uint_as_float(v & 0xffff0000u);
    }
    sum[warp][2 * lane] = s0;
    sum[warp][2 * lane + 1] = s1;
    __syncthreads();
    if (threadIdx.x < 64) {
        float s = 0.0f;
        for (int w = 0; w < 8; ++w) s += sum[w][threadIdx.x];
        db[n + threadIdx.x] += s;
    }
}

// ---- the MLP's products --------------------------------------------------------------------

constexpr uint32_t kFcA = 128 * 128;
template <int BN>
__host__ __device__ constexpr uint32_t fc_stage() { return kFcA + BN * 128; }
// K blocks of one stage (one wait: the issuing thread spends about 300 cycles on a wait, as
// long as on five products), and as many stages as fit
constexpr int kFcBlocks = 3;
template <int BN>
__host__ __device__ constexpr int fc_stages() {
    return (int)((kSmemMax - 1024) / (kFcBlocks * fc_stage<BN>()));
}
template <int BN>
__host__ __device__ constexpr int fc_pitch() { return BN + 4; }     // floats of a partial row

struct FcArgs {
    int M, N, K;
    int kb_per;             // 64-wide K blocks of one CTA of the cluster
    void* out;
    long long ldo;
    int f32;                // fp32 output, else bf16
    int add;                // fp32: add to the output
    int relu;
    const float* bias;
    const __nv_bfloat16* mask;      // times (mask[m, n] > 0), stride ldo
    int* error_flag;
};

// D[M, N] = A B^T, 128 x BN tiles, K split over the cluster's CTAs (gradients only: a
// split changes the order of the sums, and with it what an activation rounds to).  A_MN /
// B_MN: the operand is stored K rows of M (N) elements, else M (N) rows of K.  Each CTA
// accumulates its K blocks in tensor memory, leaves the fp32 tile in its shared memory, and
// after the cluster barrier sums its share of the rows over the CTAs in rank order (the
// same bits every run).  The hidden layer (K = 4096) takes BN = 32: more CTAs, each bound by
// the 20 KB a K block brings from L2.
template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(128, 1)
    fc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
              const FcArgs g) {
    constexpr uint32_t kFcStage = fc_stage<BN>();
    constexpr int kFcPitch = fc_pitch<BN>(), kFcStages = fc_stages<BN>();
    extern __shared__ uint8_t dsm_raw[];
    __shared__ __align__(8) uint64_t full_bar[kFcStages], empty_bar[kFcStages];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sIn = (saddr(dsm_raw) + 1023u) & ~1023u;
    const uint32_t fb = saddr(full_bar), eb = saddr(empty_bar), db = saddr(&done_bar);
    const int splits = gridDim.z;
    const int nk_all = (g.K + 63) / 64, kb0 = blockIdx.z * g.kb_per;
    const int nk = max(0, min(g.kb_per, nk_all - kb0));
    const int m0 = blockIdx.x * 128, n0 = blockIdx.y * BN;
    if (tid == 0) {
        for (int s = 0; s < kFcStages; ++s) {
            mbar_init(fb + 8 * s, 1);
            mbar_init(eb + 8 * s, 1);
        }
        mbar_init(db, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(saddr(&tmem_slot), 64);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) dependents_may_launch();
    wait_for_prior();
    const uint32_t tmem = tmem_slot;
    volatile int* dead = &abort_s;
    auto give_up = [&] {
        abort_s = 1;
        atomicExch(g.error_flag, 1);
    };
    if (tid == 0) {
        for (int i = 0, n = 0; i < nk; i += kFcBlocks, ++n) {
            const int st = n % kFcStages, blocks = min(kFcBlocks, nk - i);
            if (n >= kFcStages && !mbar_wait(eb + 8 * st, (uint32_t)(n / kFcStages - 1) & 1u)) {
                give_up();
                break;
            }
            if (*dead) break;
            const uint32_t bar = fb + 8 * st;
            mbar_expect_tx(bar, blocks * kFcStage);
            for (int q = 0; q < blocks; ++q) {
                const uint32_t in = sIn + (st * kFcBlocks + q) * kFcStage;
                const int k0 = (kb0 + i + q) * 64;
                if (A_MN) {
                    tma_load_2d(in, &tmA, m0, k0, bar);
                    tma_load_2d(in + kFcA / 2, &tmA, m0 + 64, k0, bar);
                } else {
                    tma_load_2d(in, &tmA, k0, m0, bar);
                }
                if (B_MN) tma_load_2d(in + kFcA, &tmB, n0, k0, bar);
                else tma_load_2d(in + kFcA, &tmB, k0, n0, bar);
            }
        }
    } else if (tid == 32) {
        constexpr uint32_t idesc =
            bf16_idesc(128, BN) | (A_MN ? kIdescAMn : 0u) | (B_MN ? kIdescBMn : 0u);
        for (int i = 0, n = 0; i < nk; i += kFcBlocks, ++n) {
            const int st = n % kFcStages, blocks = min(kFcBlocks, nk - i);
            if (!mbar_wait(fb + 8 * st, (uint32_t)(n / kFcStages) & 1u)) {
                give_up();
                break;
            }
            tc_fence_after();
            const uint32_t A = sIn + st * kFcBlocks * kFcStage, B = A + kFcA;
            const uint64_t dA = A_MN ? sw128_mn_desc(A, kFcA / 2) : sw128_desc(A);
            const uint64_t dB = B_MN ? sw128_mn_desc(B, 1024) : sw128_desc(B);
#pragma unroll
            for (int q = 0; q < kFcBlocks; ++q) {
                if (q >= blocks) break;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    umma_bf16(tmem, desc_at(dA, q * kFcStage + kk * (A_MN ? 2048 : 32)),
                              desc_at(dB, q * kFcStage + kk * (B_MN ? 2048 : 32)), idesc,
                              i > 0 || q > 0 || kk > 0 ? 1u : 0u);
            }
            umma_commit(eb + 8 * st);
        }
        umma_commit(db);
    }
    __syncwarp();
    bool ok = mbar_wait(db, 0u);
    ok = __all_sync(0xffffffffu, ok) && !*dead;
    if (!ok && lane == 0) give_up();
    tc_fence_after();
    // every load has landed and been read: the stages hold the partial tile now
    const uint32_t row = sIn + (uint32_t)(warp * 32 + lane) * (kFcPitch * 4);
#pragma unroll
    for (int c = 0; c < BN / 32; ++c) {
        float v[32];
        if (ok && nk > 0) tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + c * 32, v);
        else
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            sts128(row + c * 128 + j * 16,
                   make_uint4(__float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]),
                              __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3])));
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    {
        // the cluster is (1, 1, splits): rank = blockIdx.z
        constexpr int kVec = BN / 4;
        const int per = 128 / splits, c4 = tid % kVec;
        const bool vec = (reinterpret_cast<uintptr_t>(g.out) & 15u) == 0u && (g.ldo & 7) == 0 &&
                         n0 + BN <= g.N;
        for (int i = tid / kVec; i < per; i += 128 / kVec) {
            const int r = blockIdx.z * per + i, m = m0 + r, n = n0 + 4 * c4;
            if (m >= g.M) break;
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int z = 0; z < splits; ++z) {
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                             : "=r"(remote)
                             : "r"(sIn + (uint32_t)r * (kFcPitch * 4) + 16u * c4), "r"(z));
                float p[4];
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(p[0]), "=f"(p[1]), "=f"(p[2]), "=f"(p[3])
                             : "r"(remote)
                             : "memory");
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += p[j];
            }
            const long long o = (long long)m * g.ldo + n;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n + j >= g.N) continue;
                if (g.bias != nullptr) v[j] += g.bias[n + j];
                if (g.relu) v[j] = fmaxf(v[j], 0.0f);
                if (g.mask != nullptr && !(__bfloat162float(g.mask[o + j]) > 0.0f)) v[j] = 0.0f;
            }
            if (!ok) continue;
            if (g.f32) {
                float* out = reinterpret_cast<float*>(g.out) + o;
                if (vec) {
                    float4 w = make_float4(v[0], v[1], v[2], v[3]);
                    if (g.add) {
                        const float4 old = *reinterpret_cast<const float4*>(out);
                        w = make_float4(w.x + old.x, w.y + old.y, w.z + old.z, w.w + old.w);
                    }
                    *reinterpret_cast<float4*>(out) = w;
                } else {
                    for (int j = 0; j < 4; ++j)
                        if (n + j < g.N) out[j] = g.add ? out[j] + v[j] : v[j];
                }
            } else {
                __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(g.out) + o;
                if (vec) *reinterpret_cast<uint2*>(out) = make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
                else
                    for (int j = 0; j < 4; ++j)
                        if (n + j < g.N) out[j] = __float2bfloat16(v[j]);
            }
        }
    }
    // no CTA leaves while another may still read its tile
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 64);
}

// ---- host side ------------------------------------------------------------------------------

// A bf16 tensor map of `rank` dimensions (innermost first), 128-byte swizzle.
int tmap(CUtensorMap* tm, const void* ptr, int rank, const cuuint64_t* dims,
         const cuuint64_t* strides, const cuuint32_t* box) {
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    if (!ptr || (reinterpret_cast<uintptr_t>(ptr) & 15u) != 0) return PN_E_INVALID;
    const CUresult r = g_encode(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank,
                                const_cast<void*>(ptr), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? PN_OK : PN_E_INVALID;
}
// rows x cols, row stride ld (elements), boxes of box_rows x 64
int tmap2(CUtensorMap* tm, const void* ptr, long long rows, long long cols, long long ld,
          int box_rows) {
    if ((ld * 2) % 16 != 0) return PN_E_INVALID;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    return tmap(tm, ptr, 2, dims, strides, box);
}
// an activation [B][L][64] as {64, L, B}, boxes of n rows of nb curves
int tmap3(CUtensorMap* tm, const void* ptr, int B, int L, int n, int nb) {
    const cuuint64_t dims[3] = {64, (cuuint64_t)L, (cuuint64_t)B};
    const cuuint64_t strides[2] = {128, (cuuint64_t)L * 128};
    const cuuint32_t box[3] = {64, (cuuint32_t)n, (cuuint32_t)nb};
    return tmap(tm, ptr, 3, dims, strides, box);
}
// an activation [B][2 L][64] as {64, parity 2, L, B}, boxes of n rows of one parity plane
int tmap4(CUtensorMap* tm, const void* ptr, int B, int L, int n, int nb) {
    const cuuint64_t dims[4] = {64, 2, (cuuint64_t)L, (cuuint64_t)B};
    const cuuint64_t strides[3] = {128, 256, (cuuint64_t)L * 256};
    const cuuint32_t box[4] = {64, 1, (cuuint32_t)n, (cuuint32_t)nb};
    return tmap(tm, ptr, 4, dims, strides, box);
}

int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return n;
}

// A launch that may begin before the kernel ahead of it on the stream has ended (each of these
// kernels waits for it): a pass is 8 to 34 launches, 1 to 2 us apart without this.
template <typename... Params, typename... Args>
int launch(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t st,
           const Args&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess ? PN_OK : PN_E_CUDA;
}

template <bool BWD, bool WINDOW>
int launch_conv(const CUtensorMap& in, const CUtensorMap& w, const CUtensorMap& out,
                const CUtensorMap& mask, ConvArgs a, int n_sm, cudaStream_t st) {
    constexpr uint32_t stage = conv_stage_bytes<BWD, WINDOW>();
    constexpr uint32_t fixed = 1024 + kWeights + 2 * (BWD ? 2 : 1) * kTile +
                               conv_mask_stages<BWD, WINDOW>() * 2 * kTile;
    constexpr int fit = (int)((kSmemMax - fixed) / stage);
    constexpr int stages = fit < kMaxStages ? fit : kMaxStages;
    static_assert(stages >= 1, "a stage must fit");
    constexpr size_t smem = fixed + stages * stage;
    if (raise_smem_limit((const void*)conv_kernel<BWD, WINDOW>, smem) != cudaSuccess)
        return PN_E_CUDA;
    a.stages = stages;
    return launch(conv_kernel<BWD, WINDOW>, a.n_tiles < n_sm ? a.n_tiles : n_sm, kConvThreads, smem,
                  st, in, w, out, mask, a);
}

// Y = relu(conv(X) + bias): X [B][2 L][64], Y [B][L][64], W [64][448] (tap-major columns).
int conv_forward(const void* X, const void* W, const float* bias, void* Y, int B, int L, int n_sm,
                 int* err, cudaStream_t st) {
    const bool window = L % kRows == 0;
    CUtensorMap in, w, out;
    int rc = tmap4(&in, X, B, L, window ? kWinRows : 64, window ? 1 : 2);
    if (!rc) rc = tmap2(&w, W, 64, kTaps * kCh, kTaps * kCh, 64);
    if (!rc) rc = tmap2(&out, Y, (long long)B * L, 64, 64, kRows);
    if (rc) return rc;
    ConvArgs a{(int)(((long long)B * L + kRows - 1) / kRows), L, 0, bias, err};
    return window ? launch_conv<false, true>(in, w, out, out, a, n_sm, st)
                  : launch_conv<false, false>(in, w, out, out, a, n_sm, st);
}

// dX = the input gradient of that convolution times (X > 0).
int conv_input_grad(const void* dY, const void* W, const void* X, void* dX, int B, int L, int n_sm,
                    int* err, cudaStream_t st) {
    const bool window = L % kRows == 0;
    CUtensorMap in, w, out, mask;
    int rc = tmap3(&in, dY, B, L, window ? kWinRows : 64, window ? 1 : 2);
    if (!rc) rc = tmap2(&w, W, 64, kTaps * kCh, kTaps * kCh, 64);
    if (!rc) rc = tmap4(&out, dX, B, L, window ? kRows : 64, window ? 1 : 2);
    if (!rc) rc = tmap4(&mask, X, B, L, window ? kRows : 64, window ? 1 : 2);
    if (rc) return rc;
    ConvArgs a{(int)(((long long)B * L + kRows - 1) / kRows), L, 0, nullptr, err};
    return window ? launch_conv<true, true>(in, w, out, mask, a, n_sm, st)
                  : launch_conv<true, false>(in, w, out, mask, a, n_sm, st);
}

// gw, gb += the weight and bias gradients of that convolution; part: kWgPart floats a CTA.
int conv_weight_grad(const void* dY, const void* X, float* gw, float* gb, float* part, int B, int L,
                     int n_sm, int* err, cudaStream_t st) {
    CUtensorMap dy, x;
    int rc = tmap3(&dy, dY, B, L, kWgRows, 1);
    if (!rc) rc = tmap4(&x, X, B, L, kWgWinRows, 1);
    if (rc) return rc;
    constexpr size_t smem = 1024 + kWgStages * kWgStage + 64 * 128;
    if (raise_smem_limit((const void*)conv_wgrad_kernel, smem) != cudaSuccess) return PN_E_CUDA;
    WgradArgs a{(int)((long long)B * L / kWgRows), L, part, err};
    // at least four blocks a CTA, so that adding the sums stays small beside forming them
    const int ctas = a.n_blocks / 4 < n_sm ? (a.n_blocks + 3) / 4 : n_sm;
    rc = launch(conv_wgrad_kernel, ctas, kWgThreads, smem, st, dy, x, a);
    return rc ? rc : launch(wgrad_sum_kernel, 8 * 16, 1024, 0, st, (const float*)part, ctas, gw, gb);
}

int conv0_forward(const void* x, const void* W, const float* bias, void* Y, int B, int L, int n_sm,
                  int* err, cudaStream_t st) {
    CUtensorMap out;
    const int rc = tmap2(&out, Y, (long long)B * L, 64, 64, kRows);
    if (rc || (reinterpret_cast<uintptr_t>(W) & 15u) != 0) return PN_E_INVALID;
    Conv0Args a{reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(W),
                bias, (int)((long long)B * L / kRows), L, err};
    const int ctas = a.n_tiles < n_sm * kConv0Ctas ? a.n_tiles : n_sm * kConv0Ctas;
    constexpr size_t smem = 1024 + kTile;
    return launch((reinterpret_cast<uintptr_t>(x) & 3u) == 0 ? conv0_kernel<true>
                                                             : conv0_kernel<false>,
                  ctas, 128, smem, st, out, a);
}

int conv0_weight_grad(const void* dY, const void* x, float* gw, float* gb, float* part, int B, int L,
                      int n_sm, int* err, cudaStream_t st) {
    CUtensorMap dy;
    const int rc = tmap2(&dy, dY, (long long)B * L, 64, 64, 64);
    if (rc) return rc;
    constexpr size_t smem = 1024 + kWg0Stages * kWg0Stage;
    Wgrad0Args a{reinterpret_cast<const __nv_bfloat16*>(x), (int)((long long)B * L / 64), L, part, err};
    const int ctas = a.n_blocks < n_sm * kWg0Ctas ? a.n_blocks : n_sm * kWg0Ctas;
    static_assert(kWg0Ctas * kWg0Part <= kWgPart, "the workspace holds kWgPart floats an SM");
    const bool pairs = (reinterpret_cast<uintptr_t>(x) & 3u) == 0;
    const auto k = pairs ? conv0_wgrad_kernel<true> : conv0_wgrad_kernel<false>;
    if (raise_smem_limit((const void*)k, smem) != cudaSuccess) return PN_E_CUDA;
    const int rc2 = launch(k, ctas, 128, smem, st, dy, a);
    return rc2 ? rc2 : launch(wgrad0_sum_kernel, 15, 1024, 0, st, (const float*)part, ctas, gw, gb);
}

// One product of the MLP; a_mn / b_mn as fc_kernel.
template <int BN>
int fc(const void* A, bool a_mn, const void* B, bool b_mn, FcArgs g, int n_sm, cudaStream_t st) {
    const long long lda = a_mn ? g.M : g.K, ldb = b_mn ? g.N : g.K;
    CUtensorMap ta, tb;
    int rc = a_mn ? tmap2(&ta, A, g.K, g.M, lda, 64) : tmap2(&ta, A, g.M, g.K, lda, 128);
    if (!rc) rc = b_mn ? tmap2(&tb, B, g.K, g.N, ldb, 64) : tmap2(&tb, B, g.N, g.K, ldb, BN);
    if (rc) return rc;
    const int nk = (g.K + 63) / 64;
    const int tiles = ((g.M + 127) / 128) * ((g.N + BN - 1) / BN);
    int splits = 1;             // enough CTAs for the SMs, at least two K blocks each
    while (g.add && splits < 8 && tiles * splits * 2 <= n_sm && nk >= splits * 4) splits *= 2;
    g.kb_per = (nk + splits - 1) / splits;
    constexpr size_t smem = 1024 + fc_stages<BN>() * kFcBlocks * fc_stage<BN>();
    using Kernel = void (*)(CUtensorMap, CUtensorMap, FcArgs);
    Kernel k;
    if constexpr (BN == 64)
        k = a_mn ? (b_mn ? fc_kernel<BN, true, true> : fc_kernel<BN, true, false>)
                 : (b_mn ? fc_kernel<BN, false, true> : fc_kernel<BN, false, false>);
    else k = fc_kernel<BN, false, false>;
    if (raise_smem_limit((const void*)k, smem) != cudaSuccess) return PN_E_CUDA;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((g.M + 127) / 128, (g.N + BN - 1) / BN, splits);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = splits;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k, ta, tb, g) == cudaSuccess ? PN_OK : PN_E_CUDA;
}

int bias_grad(const void* g, int M, int N, float* db, cudaStream_t st) {
    return launch(bias_grad_kernel, N / 64, 256, 0, st, reinterpret_cast<const __nv_bfloat16*>(g), M,
                  N, db);
}

constexpr int kNetBins = 4096, kNetConv = 6, kNetHidden = 256, kNetClasses = 1024;
constexpr int kNetFlat = kCh * (kNetBins >> kNetConv);

// Activation l of the workspace: [B][4096 >> (l + 1)][64]; the hidden layer after the last.
char* act_at(void* ws, int B, int l) {
    long long pos = 0;
    for (int i = 0; i < l; ++i) pos += kNetBins >> (i + 1);
    return static_cast<char*>(ws) + pos * B * 128;
}

}  // namespace
}  // namespace pn
}  // namespace blsb200

using namespace blsb200::pn;

extern "C" {

long long pn_workspace(int B) {
    return (long long)B * ((kNetBins - (kNetBins >> kNetConv)) * 128 + kNetHidden * 2);
}

long long pn_scratch(int B) {
    return pn_workspace(B) + (long long)sm_count() * kWgPart * (long long)sizeof(float);
}

int pn_forward(const PnNet* net, const void* x, int B, void* ws, float* logits, int* error_flag,
               void* stream) {
    if (!net || !x || !ws || !logits || !error_flag || B < 1 || B > (1 << 20)) return PN_E_INVALID;
    if (load_encode() != cudaSuccess || !g_encode) return PN_E_CUDA;
    const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int n_sm = sm_count();
    int L = kNetBins / 2;
    int rc = conv0_forward(x, net->conv_w[0], net->conv_b[0], act_at(ws, B, 0), B, L, n_sm,
                           error_flag, st);
    for (int l = 1; !rc && l < kNetConv; ++l) {
        L /= 2;
        rc = conv_forward(act_at(ws, B, l - 1), net->conv_w[l], net->conv_b[l], act_at(ws, B, l), B,
                          L, n_sm, error_flag, st);
    }
    if (rc) return rc;
    void* h = act_at(ws, B, kNetConv);
    rc = fc<32>(act_at(ws, B, kNetConv - 1), false, net->w1, false,
            FcArgs{B, kNetHidden, kNetFlat, 0, h, kNetHidden, 0, 0, 1, net->b1, nullptr, error_flag},
            n_sm, st);
    if (rc) return rc;
    return fc<64>(h, false, net->w2, false,
              FcArgs{B, kNetClasses, kNetHidden, 0, logits, kNetClasses, 1, 0, 0, net->b2, nullptr,
                     error_flag},
              n_sm, st);
}

int pn_backward(const PnNet* net, const PnGrads* g, const void* x, int B, const void* ws,
                const void* dlogits, void* dws, int* error_flag, void* stream) {
    if (!net || !g || !x || !ws || !dlogits || !dws || !error_flag || B < 8 || B % 8 != 0 ||
        B > (1 << 20))
        return PN_E_INVALID;
    if (load_encode() != cudaSuccess || !g_encode) return PN_E_CUDA;
    const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int n_sm = sm_count();
    void* acts = const_cast<void*>(ws);
    if ((reinterpret_cast<uintptr_t>(dws) & 15u) != 0) return PN_E_INVALID;
    const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(act_at(acts, B, kNetConv));
    const __nv_bfloat16* flat =
        reinterpret_cast<const __nv_bfloat16*>(act_at(acts, B, kNetConv - 1));
    void* dh = act_at(dws, B, kNetConv);
    // the CTAs' partial weight gradients, after the activations' gradients
    float* part = reinterpret_cast<float*>(static_cast<char*>(dws) + pn_workspace(B));
    void* dflat = act_at(dws, B, kNetConv - 1);
    // logits = h W2^T + b2
    int rc = fc<64>(dlogits, true, h, true,
                FcArgs{kNetClasses, kNetHidden, B, 0, g->w2, kNetHidden, 1, 1, 0, nullptr, nullptr,
                       error_flag},
                n_sm, st);
    if (!rc) rc = bias_grad(dlogits, B, kNetClasses, g->b2, st);
    if (!rc)
        rc = fc<64>(dlogits, false, net->w2, true,
                FcArgs{B, kNetHidden, kNetClasses, 0, dh, kNetHidden, 0, 0, 0, nullptr, h,
                       error_flag},
                n_sm, st);
    // h = relu(flat W1^T + b1)
    if (!rc)
        rc = fc<64>(dh, true, flat, true,
                FcArgs{kNetHidden, kNetFlat, B, 0, g->w1, kNetFlat, 1, 1, 0, nullptr, nullptr,
                       error_flag},
                n_sm, st);
    if (!rc) rc = bias_grad(dh, B, kNetHidden, g->b1, st);
    if (!rc)
        rc = fc<64>(dh, false, net->w1, true,
                FcArgs{B, kNetFlat, kNetHidden, 0, dflat, kNetFlat, 0, 0, 0, nullptr, flat,
                       error_flag},
                n_sm, st);
    // the convolutions, last to first
    for (int l = kNetConv - 1; !rc && l > 0; --l) {
        const int L = kNetBins >> (l + 1);
        rc = conv_weight_grad(act_at(dws, B, l), act_at(acts, B, l - 1), g->conv_w[l], g->conv_b[l],
                              part, B, L, n_sm, error_flag, st);
        if (!rc)
            rc = conv_input_grad(act_at(dws, B, l), net->conv_w[l], act_at(acts, B, l - 1),
                                 act_at(dws, B, l - 1), B, L, n_sm, error_flag, st);
    }
    if (rc) return rc;
    return conv0_weight_grad(act_at(dws, B, 0), x, g->conv_w[0], g->conv_b[0], part, B,
                             kNetBins / 2, n_sm, error_flag, st);
}

}  // extern "C"
