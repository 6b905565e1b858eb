// Launch description of an fp32 product on the FMA pipe (gemm32.cu), made by the plan compiler.
#pragma once

namespace b200 {
struct Gemm32Launch {
  int M = 0, N = 0, K = 0, G = 1;
  int a_kc = 1, b_kc = 0;                   // k contiguous in the operand (else m, n)
  long long a_ld = 0, b_ld = 0;             // stride of the other index
  long long a_gs = 0, b_gs = 0;             // group strides
  int a_vec = 0, b_vec = 0;                 // rows start on 16 bytes and are multiples of 16 bytes long
  int tile = 0;                             // CTA tile: 0 32 x 64 (eight warps share k), 1 64 x 64 (four), 2 64 x 128 (two), 3 64 x 128 (four warps)
  int split = 0;                            // CTAs of a cluster that share K (1, 2, 4 or 8); 0: this kernel is not used
};

// CTAs of clusters of `split` that are resident at one per SM (cudaOccupancyMaxActiveClusters on a B200: a cluster stays
// inside a GPC, and GPCs have between 16 and 20 SMs).
inline int gemm32_resident(int split) { return split == 8 ? 120 : split == 4 ? 132 : 148; }
}  // namespace b200
