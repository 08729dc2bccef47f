// Pipeline depth of the tensor-core GEMM by its grid (host; tests compile it alone).
#pragma once

namespace hc {

// Two stages leave room for two blocks on an SM, one's epilogue under the other's loads
// and MMAs; that pays only where the grid has more blocks than the GPU has SMs. A smaller
// grid has its SMs to itself and takes four, which load a layer's whole K (four 64-wide
// blocks) at once instead of waiting for the MMAs. Measured (B200, us, two / four stages):
// training step of 12-256-256-256-10 on 64 rows 248 / 240, 512 rows 258 / 248, 8192 rows
// 447 / 438 (no grid above 128 blocks); forward pass of a 320-wide network on 200 rows
// 49.9 / 47.8, on 65,536 rows 223 / 336. A long K keeps four: 32,768 x 1024, K = 1024,
// 134 / 129.
constexpr int kLongRing = 4, kShortRing = 2, kShortK = 512;

constexpr int gemm_stages(int tiles_m, int tiles_n, int K, int sms) {
    return K <= kShortK && (long long)tiles_m * tiles_n > sms ? kShortRing : kLongRing;
}

}  // namespace hc
