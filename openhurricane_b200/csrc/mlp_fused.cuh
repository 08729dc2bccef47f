// The surrogate network's inference in one kernel, sm_100a (tcgen05 + TMA): a
// tile of 128 rows goes through every layer with its activations in shared
// memory and its accumulators in tensor memory.
//
// What bounds it: the activation, 128 x width GELUs per layer and tile on the
// ordinary pipes (about 25 instructions each), not the tensor cores (1024 cycles
// a 256 x 256 layer) and no longer memory: the layer-by-layer form wrote and read
// every activation (512 bytes a row and layer) and padded the input to 128
// columns and the output to 128. So two tiles per SM, each with its own four
// epilogue warps, one's GELUs under the other's MMAs:
//
//   warp 0      streams the weights' K blocks (64 wide) by TMA through a ring
//   warp 1      issues tcgen05.mma (M = 128, N = layer width, K = 16), one tile's
//               layer after the other's
//   warps 2-5   tile slot 0: input rows to BF16, then per layer bias + GELU from
//   warps 6-9   tile slot 1: tensor memory back into the slot's operand buffer
//
// Shapes: up to kFusedLayers layers, inputs and widths up to 256, outputs up to
// 256; anything else takes the layer-by-layer form.
//
// Measured (B200, an ensemble's forward passes, three networks 12-256-256-256-10, fused /
// layer by layer with an earlier form of GELU): 4,096 rows 123 / 205 us, 65,536 rows
// 233 / 548 us, 300,000 rows 866 / 2497 us.
#pragma once

#include "mlp_gemm.cuh"

namespace hc {

constexpr int kFusedLayers = 6;
constexpr int kFusedRing = 3;
constexpr int kFusedThreads = 320;

struct FusedMlp {
    CUtensorMap w[kFusedLayers];       // [outp][inp] bf16, box {64, bn}
    const float *bias[kFusedLayers];
    int nk[kFusedLayers];              // K blocks of 64
    int bn[kFusedLayers];              // columns of the accumulator (multiple of 32, <= 256)
    int nl, n_in, n_out;
};

struct FusedSmem {
    static constexpr int kA = 4 * kGemmBM * kGemmBK * 2;       // a slot's operand: four K blocks, 64 KiB
    static constexpr int kB = 256 * kGemmBK * 2;               // a weight block, 32 KiB
    static constexpr size_t bytes() { return 1024 + 2 * (size_t)kA + (size_t)kFusedRing * kB + 256; }
};

__global__ void __launch_bounds__(kFusedThreads, 1)
mlp_fused_kernel(const __grid_constant__ FusedMlp net, const float *__restrict__ X, int64_t rows,
                 float *__restrict__ Y, int *err) {
    using S = FusedSmem;
    extern __shared__ uint8_t fused_smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(fused_smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = smem + 2 * S::kA;
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + kFusedRing * S::kB);
    uint64_t *empty = full + kFusedRing, *ready = empty + kFusedRing, *done = ready + 2;
    uint64_t *drain = done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *stop = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t tiles = (rows + kGemmBM - 1) / kGemmBM;
    // this block's tiles: pair p holds tiles 2 p (slot 0) and 2 p + 1 (slot 1)
    const int64_t pairs = (tiles + 1) / 2;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kFusedRing; ++s) {
            sm100::mbar_init(&full[s], 1);
            sm100::mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            sm100::mbar_init(&ready[s], 128);
            sm100::mbar_init(&done[s], 1);
        }
        sm100::mbar_init(drain, 1);
        *stop = 0;
        sm100::fence_mbar_init();
    }
    if (warp == 2) {
        sm100::tmem_alloc(tmem_slot, 512);
        sm100::tmem_relinquish();
    }
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
    const uint32_t taddr = *tmem_slot;
    // a bounded wait that also gives up when another role has
    auto wait = [&](uint64_t *bar, uint32_t parity, int code) {
        for (uint32_t i = 0; i < kWaitLimit; ++i) {
            if (sm100::mbar_try_wait(bar, parity)) return true;
            if (*stop) return false;
        }
        *stop = 1;
        atomicExch(err, code);
        return false;
    };

    if (warp == 0 && lane == 0) {
        uint32_t q = 0;
        bool ok = true;
        for (int64_t p = blockIdx.x; ok && p < pairs; p += gridDim.x)
            for (int l = 0; ok && l < net.nl; ++l)
                for (int s = 0; ok && s < 2; ++s) {
                    if (2 * p + s >= tiles) continue;
                    for (int k = 0; ok && k < net.nk[l]; ++k, ++q) {
                        const uint32_t st = q % kFusedRing, it = q / kFusedRing;
                        if (it > 0 && !wait(&empty[st], (it - 1) & 1, 1)) {
                            ok = false;
                            break;
                        }
                        sm100::mbar_arrive_expect_tx(&full[st], (uint32_t)net.bn[l] * kGemmBK * 2);
                        sm100::tma_load_2d(ring + st * S::kB, &net.w[l], &full[st], k * kGemmBK, 0);
                    }
                }
        // where a role gave up, loads may still be on their way into this block's memory
        for (uint32_t i = q < kFusedRing ? 0 : q - kFusedRing; i < q; ++i)
            sm100::mbar_wait(&full[i % kFusedRing], (i / kFusedRing) & 1, kWaitLimit);
    } else if (warp == 1 && lane == 0) {
        uint32_t q = 0, phase[2] = {0, 0};
        bool ok = true;
        for (int64_t p = blockIdx.x; ok && p < pairs; p += gridDim.x)
            for (int l = 0; ok && l < net.nl; ++l)
                for (int s = 0; ok && s < 2; ++s) {
                    if (2 * p + s >= tiles) continue;
                    if (!wait(&ready[s], phase[s], 2)) {
                        ok = false;
                        break;
                    }
                    phase[s] ^= 1;
                    sm100::tc_fence_after();
                    const uint32_t idesc = sm100::idesc_bf16_f32(kGemmBM, net.bn[l]);
                    for (int k = 0; k < net.nk[l]; ++k, ++q) {
                        const uint32_t st = q % kFusedRing, it = q / kFusedRing;
                        if (!wait(&full[st], it & 1, 3)) {
                            ok = false;
                            break;
                        }
                        sm100::tc_fence_after();
                        const uint32_t a = sm100::smem_u32(smem + s * S::kA + k * kGemmBM * kGemmBK * 2);
                        const uint32_t b = sm100::smem_u32(ring + st * S::kB);
#pragma unroll
                        for (int j = 0; j < kGemmBK / 16; ++j)
                            sm100::mma_bf16(taddr + 256 * s, sm100::desc_kmajor_sw128(a + 32 * j),
                                            sm100::desc_kmajor_sw128(b + 32 * j), idesc, (k | j) != 0 ? 1u : 0u);
                        sm100::mma_commit(&empty[st]);
                    }
                    if (ok) sm100::mma_commit(&done[s]);
                }
        // and MMAs into the tensor memory that is freed below
        sm100::mma_commit(drain);
        sm100::mbar_wait(drain, 0, kWaitLimit);
    } else if (warp >= 2) {
        const int s = (warp - 2) >> 2, quarter = warp & 3;    // the lanes of tensor memory a warp can read
        const int r = quarter * 32 + lane;                    // the thread's row of the tile
        uint8_t *A = smem + s * S::kA + r * 128;
        const uint32_t lane_base = taddr + 256 * s + ((uint32_t)(quarter * 32) << 16);
        uint32_t phase = 0;
        bool ok = true;
        // chunk of 8 columns to its place in the 128-byte swizzled K block
        auto put = [&](int c, const uint4 &v) {
            *reinterpret_cast<uint4 *>(A + (c >> 3) * (kGemmBM * kGemmBK * 2) + (((c & 7) ^ (r & 7)) << 4)) = v;
        };
        auto pack = [](float x, float y) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
            return *reinterpret_cast<const uint32_t *>(&h);
        };
        auto publish = [&]() {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes before the MMAs' reads
            sm100::tc_fence_before();
            sm100::mbar_arrive(&ready[s]);
        };
        for (int64_t p = blockIdx.x; p < pairs; p += gridDim.x) {
            const int64_t tile = 2 * p + s;
            if (tile >= tiles) break;
            const int64_t row = tile * kGemmBM + r;
            const float *x = X + row * net.n_in;
            for (int c = 0; c < 8 * net.nk[0]; ++c) {
                float v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = (row < rows && 8 * c + j < net.n_in) ? __ldg(&x[8 * c + j]) : 0.0f;
                put(c, make_uint4(pack(v[0], v[1]), pack(v[2], v[3]), pack(v[4], v[5]), pack(v[6], v[7])));
            }
            publish();
            for (int l = 0; l < net.nl; ++l) {
                // warp-uniform: the tensor-memory loads below are .sync.aligned
                ok = __all_sync(0xffffffffu, wait(&done[s], phase, 4));
                if (!ok) break;
                phase ^= 1;
                sm100::tc_fence_after();
                const float *b = net.bias[l];
                const bool last = l + 1 == net.nl;
#pragma unroll 1
                for (int c0 = 0; c0 < net.bn[l]; c0 += 32) {
                    uint32_t t[32];
                    sm100::tmem_ld_32x32b_x32(lane_base + (uint32_t)c0, t);
                    sm100::tmem_ld_wait();
                    if (last) {
                        if (row < rows) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (c0 + j < net.n_out)
                                    Y[row * net.n_out + c0 + j] = __uint_as_float(t[j]) + __ldg(&b[c0 + j]);
                        }
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        const float4 b0 = __ldg(reinterpret_cast<const float4 *>(b + c0 + j));
                        const float4 b1 = __ldg(reinterpret_cast<const float4 *>(b + c0 + j + 4));
                        float v[8] = {__uint_as_float(t[j]) + b0.x, __uint_as_float(t[j + 1]) + b0.y,
                                      __uint_as_float(t[j + 2]) + b0.z, __uint_as_float(t[j + 3]) + b0.w,
                                      __uint_as_float(t[j + 4]) + b1.x, __uint_as_float(t[j + 5]) + b1.y,
                                      __uint_as_float(t[j + 6]) + b1.z, __uint_as_float(t[j + 7]) + b1.w};
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] = gelu_f(v[k]);
                        put((c0 + j) >> 3, make_uint4(pack(v[0], v[1]), pack(v[2], v[3]), pack(v[4], v[5]), pack(v[6], v[7])));
                    }
                }
                if (!last) publish();
                else sm100::tc_fence_before();
            }
            if (!ok) break;
        }
    }
    __syncwarp();
    sm100::tc_fence_before();
    __syncthreads();
    if (warp == 2) sm100::tmem_dealloc(taddr, 512);
}

}  // namespace hc
