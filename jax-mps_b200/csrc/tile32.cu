// fp32 contractions whose operands arrive in whole tiles: the 3xTF32 product of kernels.cu (hi*hi + hi*lo + lo*hi, fp32
// accumulation in tensor memory) for everything whose A is a dense matrix or the image of a stride-1 convolution.
//
// The table-driven kernels gather both operands with hundreds of threads and split B again in every CTA; a k-tile of
// 128 x 64 x 32 took an SM about 1000 cycles of which the tensor core needs 390. What is left to do per k-tile here:
//   * A: one tiled copy (or four) by one thread; two groups of four converter warps move it to tensor memory as high and
//     low words, as before.
//   * B: split once per product by a kernel of its own (split_b_kernel) into an image of finished tiles, high then low
//     part, swizzled as the tensor core reads them, so that a k-tile of B is one untiled copy of 16 or 32 KB. Weights are
//     small against what they are multiplied with, and the split runs beside whatever is in front of the product.
//   * The CTA is persistent over its tiles with two accumulators: four warps of their own read one back while the tensor
//     core fills the other.
// Per k-tile that leaves (16 + 16 for A, 16 + 24 for B) = 72 KB through shared memory for a 64-wide tile, 112 KB for a
// 128-wide one: bound by shared memory at about 560 and 880 cycles; measured 830 and 960. 3x3 convolutions, forward and input
// gradient, kernel alone, table-driven -> here: 131072 x 64 x 576 88 -> 63 us (153 TFLOP/s), 32768 x 128 x 1152 74 -> 48 us,
// 8192 x 256 x 2304 67 -> 45 us (213 TFLOP/s). Weight gradients were tried and stay table-driven: their B is the large operand,
// and writing and reading its image costs what the product gains.
// The first version took 1180 and 1370 cycles a k-tile, bound by latencies of single warps: divisions in the copying warp
// (now one lane each for A and B, and divisions once a tile), and two waits, a flag and a vote in the MMA warp's loop.
// Roles (16 warps): 0 copies of A, 1 MMA, 2 copies of B, 4-11 converters, 12-15 read-back. Every wait is bounded; a role that
// times out raises the flag, the others give up at it, everybody meets at the end, tensor memory is released.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstring>
#include <algorithm>

#include "kernels.h"
#include "launch.h"
#include "tc_util.cuh"

namespace b200 {
namespace {

bool g_programmatic = true;

constexpr int VM = 128, VK = 32, GROUPS = 2;                 // GROUPS warpgroups turn A into its two parts
constexpr int READ_WARP = 4 + 4 * GROUPS, VTHREADS = 32 * (READ_WARP + 4);

template <int BN_>
struct TileCfg {
  static constexpr int BN = BN_;
  static constexpr int STAGES = BN == 64 ? 6 : 4;
  static constexpr int A_BYTES = VM * VK * 4, B_BYTES = 2 * BN * VK * 4;      // B: high and low part
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 512;
  static constexpr int A_COL0 = 2 * BN;                                       // after the two accumulators, 64 columns a stage
  static_assert(A_COL0 + 64 * STAGES <= 512, "tensor memory");
};

struct TileParams {
  int M, N, K, G, mode, split, tiles_m, tiles_n, ktiles, kt_per_split;
  int ow, oh, kw, pad_h, pad_w, dil_h, dil_w, cin, c_vec;
};

__device__ __forceinline__ float low_part(float x) {
  // x less its TF32 bits (exact), half a TF32 unit added so that the tensor core's truncation rounds; inf - inf would be NaN
  const float l = x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
  return fabsf(x) == INFINITY ? 0.f : __uint_as_float(__float_as_uint(l) + 0x1000u);
}

// B(k, n) = B[b_grp[g] + b_row[k] + b_col[n]] as tiles [group][n-tile][k-tile][part][n][32 k]: rows of 128 bytes in the
// 128-byte swizzle. A thread makes four consecutive k of one n. LANES_N: neighbouring threads take neighbouring n.
template <bool LANES_N>
__global__ void __launch_bounds__(256) split_b_kernel(const float* __restrict__ B, float* __restrict__ image, const long long* __restrict__ b_row,
                                                     const long long* __restrict__ b_col, const long long* __restrict__ b_grp, int N, int K, int bn,
                                                     int tiles_n, int ktiles, long long total) {
  pdl_prologue();
  const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
  if (t >= total) return;
  const int np = tiles_n * bn, kc = ktiles * 8;
  int n, c;
  long long rest;
  if (LANES_N) { n = (int)(t % np); rest = t / np; c = (int)(rest % kc); rest /= kc; }
  else { c = (int)(t % kc); rest = t / kc; n = (int)(rest % np); rest /= np; }
  const int g = (int)rest;
  float v[4];
  const float* src = B + b_grp[g] + (n < N ? b_col[n] : 0);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int k = 4 * c + e;
    v[e] = (n < N && k < K) ? src[b_row[k]] : 0.f;
  }
  const int row = n % bn, chunk = c & 7;
  float* tile = image + (((long long)g * tiles_n + n / bn) * ktiles + (c >> 3)) * (2ll * bn * 32);
  const int at = (row >> 3) * 256 + (row & 7) * 32 + ((chunk ^ (row & 7)) << 2);
  *reinterpret_cast<float4*>(tile + at) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(tile + bn * 32 + at) = make_float4(low_part(v[0]), low_part(v[1]), low_part(v[2]), low_part(v[3]));
}

template <int BN, bool A_MC>
__global__ void __launch_bounds__(VTHREADS, 1) tile32_kernel(const __grid_constant__ CUtensorMap tm_a, const float* __restrict__ image, float* __restrict__ C,
                                                            float* __restrict__ partial, const long long* __restrict__ c_row,
                                                            const long long* __restrict__ c_col, const long long* __restrict__ c_grp,
                                                            int* __restrict__ error_flag, TileParams p) {
  using Cfg = TileCfg<BN>;
  constexpr int S = Cfg::STAGES;
  extern __shared__ uint8_t v_smem[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)v_smem + 1023) & ~(uintptr_t)1023);
  uint64_t* landed = (uint64_t*)(smem + S * Cfg::STAGE_BYTES);
  uint64_t* a_ready = landed + S;
  uint64_t* empty = a_ready + S;
  uint64_t* acc_full = empty + S;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* drained = acc_empty + 2;
  uint32_t* tmem_slot = (uint32_t*)(drained + 1);
  volatile int* failed = (volatile int*)(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(&landed[s]), 2);                    // the copies of A and those of B
      mbar_init(smem_u32(&a_ready[s]), 4);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), 4);
    }
    mbar_init(smem_u32(drained), 1);
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_prologue();

  // work items (each with at least one k-tile) in the order [group][split][n-tile][m-tile]; every role walks the same ones and counts their k-tiles in `it`
  const int items = p.G * p.split * p.tiles_n * p.tiles_m;
  struct Item { int g, sp, nt, mt, k0, k1; };
  auto item_of = [&](int w) -> Item {
    Item i;
    i.mt = w % p.tiles_m; w /= p.tiles_m;
    i.nt = w % p.tiles_n; w /= p.tiles_n;
    i.sp = w % p.split; i.g = w / p.split;
    i.k0 = min(p.ktiles, i.sp * p.kt_per_split);
    i.k1 = min(p.ktiles, i.k0 + p.kt_per_split);
    return i;
  };

  if (warp == 0 || warp == 2) {
    // ------------------------------ copies: warp 0 those of A, warp 2 those of B (one lane each) --------------------
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const Item i = item_of(w);
        const int m0 = i.mt * VM;
        const char* b_tiles = (const char*)image + ((long long)i.g * p.tiles_n + i.nt) * p.ktiles * (long long)Cfg::B_BYTES;
        // Where the tile starts: divisions once per tile, additions per k-tile.
        int c0 = 0, kw = 0, kh = 0, px_n = 0, px_h = 0;
        if (p.mode == 1) {
          const int c_tiles = p.cin / VK, tap = i.k0 / c_tiles;
          c0 = (i.k0 - tap * c_tiles) * VK, kh = tap / p.kw, kw = tap - kh * p.kw;
          px_n = m0 / (p.oh * p.ow), px_h = (m0 - px_n * p.oh * p.ow) / p.ow;
        }
        for (int kt = i.k0; kt < i.k1; ++kt, ++it) {
          const int s = it % S;
          if (it >= S && !(ok = role_wait(smem_u32(&empty[s]), (uint32_t)((it / S - 1) & 1), failed))) break;
          const uint32_t bar = smem_u32(&landed[s]), at = smem_u32(smem + s * Cfg::STAGE_BYTES);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)(warp == 0 ? Cfg::A_BYTES : Cfg::B_BYTES)) : "memory");
          auto box = [&](uint32_t dst, int x, int y, int z, int u) {
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                ::"r"(dst), "l"(&tm_a), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(u) : "memory");
          };
          if (warp == 2) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(at + (uint32_t)Cfg::A_BYTES), "l"(b_tiles + (long long)kt * Cfg::B_BYTES), "r"((uint32_t)Cfg::B_BYTES), "r"(bar) : "memory");
          } else if (A_MC) {
#pragma unroll
            for (int q = 0; q < 4; ++q) box(at + 4096u * q, m0 + 32 * q, kt * VK, i.g, 0);      // 32 rows at 32 k each
          } else if (p.mode == 1) {                  // 32 channels at one filter tap, 128 output pixels
            box(at, c0, kw * p.dil_w - p.pad_w, px_h + kh * p.dil_h - p.pad_h, px_n);
            if ((c0 += VK) >= p.cin) { c0 = 0; if (++kw == p.kw) kw = 0, ++kh; }
          } else box(at, kt * VK, m0, i.g, 0);       // 32 k of 128 rows
        }
      }
      if (!ok)                                       // nothing may be in flight when the block leaves
        for (int j = it > S ? it - S : 0; j < it; ++j) mbar_wait(smem_u32(&landed[j % S]), (uint32_t)((j / S) & 1));
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA (whole warp, one elected lane issues) -------------------------------------
    // The tensor core keeps only a few instructions in its queue, so what this loop does between two k-tiles has to be
    // short: one wait (A's parts in tensor memory also mean that B has landed), asked for before the MMAs in front of it.
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(VM >> 4) << 24);
    const uint64_t d_b = umma_desc(smem_u32(smem) + Cfg::A_BYTES);
    constexpr uint64_t LOW = (uint64_t)((Cfg::B_BYTES / 2) >> 4);
    int done = 0, s = 0;
    uint32_t ph = 0;
    bool ready = false;
    for (int w = blockIdx.x; w < items; w += gridDim.x, ++done) {
      const Item i = item_of(w);
      const uint32_t acc = tmem + (uint32_t)((done & 1) * BN);
      if (done >= 2) role_wait(smem_u32(&acc_empty[done & 1]), (uint32_t)((done / 2 - 1) & 1), failed);
      __syncwarp();
      for (int kt = i.k0; kt < i.k1; ++kt) {
        if (!ready) role_wait(smem_u32(&a_ready[s]), ph, failed);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int s1 = s + 1 < S ? s + 1 : 0;
        const uint32_t ph1 = s + 1 < S ? ph : ph ^ 1u;
        ready = phase_done(smem_u32(&a_ready[s1]), ph1);
        const uint64_t st = (uint64_t)((s * Cfg::STAGE_BYTES) >> 4);
        const uint32_t a_hi = tmem + (uint32_t)(Cfg::A_COL0 + s * 64);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < VK / 8; ++kk) {
            const uint64_t db = d_b + st + (uint64_t)(kk * 2);       // 8 floats = 32 bytes along K inside the swizzle atom
            umma_tf32_ta(acc, a_hi + kk * 8, db, idesc, (kt > i.k0 || kk > 0) ? 1u : 0u);
            umma_tf32_ta(acc, a_hi + kk * 8, db + LOW, idesc, 1);
            umma_tf32_ta(acc, a_hi + 32 + kk * 8, db, idesc, 1);
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&empty[s])) : "memory");
          if (kt + 1 == i.k1)
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&acc_full[done & 1])) : "memory");
        }
        __syncwarp();
        s = s1, ph = ph1;
      }
    }
    if (*failed) {                                   // tensor memory goes back only when no MMA is left
      if (elect_one()) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(drained)) : "memory");
      __syncwarp();
      mbar_wait(smem_u32(drained), 0);
    }
  } else if (warp >= 4 && warp < READ_WARP) {
    // ------------------------------ A: shared memory -> registers -> tensor memory ---------------------------------
    const int group = (warp - 4) >> 2, quad = warp & 3, row = 32 * quad + lane;
    int it = 0, turn = 0;
    for (int w = blockIdx.x; w < items; w += gridDim.x) {
      const Item i = item_of(w);
      for (int kt = i.k0; kt < i.k1; ++kt, ++it) {
        const bool mine = turn == group;
        if (++turn == GROUPS) turn = 0;
        if (!mine) continue;
        const int s = it % S;
        role_wait(smem_u32(&landed[s]), (uint32_t)((it / S) & 1), failed);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint8_t* raw = smem + s * Cfg::STAGE_BYTES;
        uint32_t v[32];
        if (A_MC) {                                  // [32 rows][k][32 m], 16-byte pieces of a k-row permuted by the k
#pragma unroll
          for (int k = 0; k < 32; ++k)
            v[k] = *reinterpret_cast<const uint32_t*>(raw + quad * 4096 + k * 128 + (((lane >> 2) ^ (k & 7)) << 4) + (lane & 3) * 4);
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint4 t = *reinterpret_cast<const uint4*>(raw + row * 128 + ((c ^ (row & 7)) << 4));
            v[4 * c] = t.x; v[4 * c + 1] = t.y; v[4 * c + 2] = t.z; v[4 * c + 3] = t.w;
          }
        }
        const uint32_t taddr = tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(Cfg::A_COL0 + s * 64);
        tmem_store32(taddr, v);
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(low_part(__uint_as_float(v[k])));
        tmem_store32(taddr + 32, v);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();                                // one arrival a warp: those of a whole group on one word take turns
        if (lane == 0) mbar_arrive(smem_u32(&a_ready[s]));
      }
    }
  } else if (warp >= READ_WARP) {
    // ------------------------------ read-back ---------------------------------------------------------------------
    const int quad = warp & 3;
    int done = 0;
    for (int w = blockIdx.x; w < items; w += gridDim.x, ++done) {
      const Item i = item_of(w);
      const int b = done & 1, m = i.mt * VM + 32 * quad + lane, n0 = i.nt * BN;
      role_wait(smem_u32(&acc_full[b]), (uint32_t)((done / 2) & 1), failed);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float* rowp = nullptr;
      bool vec = false;
      if (m < p.M) {
        if (p.split > 1) { rowp = partial + (((long long)i.sp * p.G + i.g) * p.M + m) * p.N; vec = (p.N & 3) == 0; }
        else { rowp = C + c_grp[i.g] + c_row[m]; vec = p.c_vec == 2; }
      }
#pragma unroll
      for (int part = 0; part < BN / 32; ++part) {
        uint32_t v[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
            "%23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
              "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
              "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(b * BN + part * 32))
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (part == BN / 32 - 1) {                   // the accumulator is free again
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&acc_empty[b]));
        }
        const int nb = n0 + part * 32;
        if (!rowp || nb >= p.N) continue;
        if (vec && nb + 32 <= p.N) {
          float* out = rowp + (p.split > 1 ? nb : (int)c_col[nb]);
#pragma unroll
          for (int q = 0; q < 32; q += 4)
            *reinterpret_cast<float4*>(out + q) = make_float4(__uint_as_float(v[q]), __uint_as_float(v[q + 1]), __uint_as_float(v[q + 2]), __uint_as_float(v[q + 3]));
        } else {
#pragma unroll
          for (int q = 0; q < 32; ++q)
            if (nb + q < p.N) rowp[p.split > 1 ? nb + q : c_col[nb + q]] = __uint_as_float(v[q]);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && *failed) atomicAdd(error_flag, 1);
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <int BN>
cudaError_t launch(const Tile32Launch& t, const CUtensorMap& tm, const float* image, float* C, float* partial, const long long* const* ct, int* error_flag,
                   const TileParams& p, cudaStream_t stream) {
  static bool done[64];
  if (first_use_on_this_device(done)) {
    if (cudaError_t e = cudaFuncSetAttribute(tile32_kernel<BN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TileCfg<BN>::SMEM)) return e;
    if (cudaError_t e = cudaFuncSetAttribute(tile32_kernel<BN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TileCfg<BN>::SMEM)) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<long long>(148, (long long)p.G * p.split * p.tiles_n * p.tiles_m), 1, 1);
  cfg.blockDim = dim3(VTHREADS, 1, 1);
  cfg.dynamicSmemBytes = TileCfg<BN>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_programmatic ? 1 : 0;
  if (t.mode == 3) return launch_kernel(cfg, tile32_kernel<BN, true>, tm, image, C, partial, ct[0], ct[1], ct[2], error_flag, p);
  return launch_kernel(cfg, tile32_kernel<BN, false>, tm, image, C, partial, ct[0], ct[1], ct[2], error_flag, p);
}

}  // namespace

void set_tile32_programmatic_launch(bool on) { g_programmatic = on; }

cudaError_t launch_split_b(const Tile32Launch& t, bool lanes_n, const void* B, void* image, const void* const* b_tables, cudaStream_t stream, int* launches) {
  const int tiles_n = (t.N + t.bn - 1) / t.bn, ktiles = (t.K + VK - 1) / VK;
  const long long total = (long long)t.G * tiles_n * t.bn * ktiles * 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((total + 255) / 256), 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_programmatic ? 1 : 0;
  auto row = (const long long*)b_tables[0], col = (const long long*)b_tables[1], grp = (const long long*)b_tables[2];
  cudaError_t e = launch_kernel(cfg, lanes_n ? split_b_kernel<true> : split_b_kernel<false>, (const float*)B, (float*)image, row, col, grp, t.N, t.K,
                                     t.bn, tiles_n, ktiles, total);
  if (e == cudaSuccess) ++*launches;
  return e;
}

cudaError_t launch_tile32(const Tile32Launch& t, const void* A, const void* image, void* C, void* partial, const void* const* c_tables, int* error_flag,
                          cudaStream_t stream, int* launches) {
  alignas(64) CUtensorMap tm;
  unsigned long long dims[4], strides[3];
  for (int k = 0; k < 4; k++) dims[k] = (unsigned long long)t.dims[k];
  for (int k = 0; k < 3; k++) strides[k] = 4ull * (unsigned long long)t.strides[k];
  if (!encode_tensor_map(&tm, 2, 4, A, dims, strides, t.box)) return cudaErrorInvalidValue;
  TileParams p;
  p.M = t.M; p.N = t.N; p.K = t.K; p.G = t.G; p.mode = t.mode;
  p.tiles_m = (t.M + VM - 1) / VM;
  p.tiles_n = (t.N + t.bn - 1) / t.bn;
  p.ktiles = (t.K + VK - 1) / VK;
  p.kt_per_split = (p.ktiles + t.split - 1) / t.split;
  p.split = (p.ktiles + p.kt_per_split - 1) / p.kt_per_split;
  if (p.split != t.split) return cudaErrorInvalidValue;      // the plan sizes the partial sums by it
  p.ow = t.ow; p.oh = t.oh; p.kw = t.kw; p.pad_h = t.pad_h; p.pad_w = t.pad_w; p.dil_h = t.dil_h; p.dil_w = t.dil_w; p.cin = t.cin;
  p.c_vec = t.c_vec == 2 && (((uintptr_t)C) & 15) == 0 ? 2 : 0;
  const long long* ct[3] = {(const long long*)c_tables[0], (const long long*)c_tables[1], (const long long*)c_tables[2]};
  cudaError_t e = t.bn == 64 ? launch<64>(t, tm, (const float*)image, (float*)C, (float*)partial, ct, error_flag, p, stream)
                             : launch<128>(t, tm, (const float*)image, (float*)C, (float*)partial, ct, error_flag, p, stream);
  if (e != cudaSuccess) return e;
  ++*launches;
  if (t.split > 1) e = launch_splitk_reduce((const float*)partial, (float*)C, ct[0], ct[1], ct[2], t.M, t.N, t.G, t.split, t.c_vec, stream, launches);
  return e;
}

}  // namespace b200
