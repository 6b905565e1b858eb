// fp32 matrix products on the FMA pipe, for products whose time is latency and not arithmetic.
//
// C[g][m][n] = sum_k A(g, m, k) * B(g, k, n), exact fp32 multiply-adds. The 3xTF32 tensor-core kernels (kernels.cu) have
// five times the arithmetic rate, but a CTA of theirs spends about 8 us on its way through table look-ups, tensor-memory
// allocation, conversion and read-back before and after a handful of k-tiles, and their K splits need a second launch to
// be added up. A recurrent cell's products (64 x 1024 x 512: 34 M multiply-adds, 1 us of the FMA pipe of the whole chip)
// are all overhead there. Here a warp computes 32 x 64 outputs, 8 x 8 per thread, two columns per FMA instruction; the eight
// warps of a CTA share the k of a stage between two, four or eight of them (64 x 128, 64 x 64, 32 x 64 tiles; a grid of several
// waves takes 64 x 128 tiles of four warps that do not, two CTAs to an SM), and two, four or
// eight CTAs of one thread-block cluster may split K on top of that. The warps' tiles are added up in shared memory, every CTA
// sends each of the others its part of the sum (stores to distributed shared memory, behind a barrier that was begun when the
// kernel started), and adds what it was sent: one barrier to wait for, all sums in a fixed order, in the same launch. Operand
// tiles move by cp.async (16 bytes where the layout allows, single floats otherwise) through a ring of three stages and stay in
// shared memory as they lie in global memory: k-contiguous rows are read four k at a time, row-contiguous ones four rows
// at a time, so neither layout is transposed. Bound by what shared memory gives to the registers (64 bytes per thread and k, 64
// cycles of the SM's 128 bytes per cycle for the 64 cycles that the FMA instructions of four warps take: 0.87 ns per k and 64
// instructions where either alone would take 0.52) and, for the small ones, by the latency of the first loads and of the sums.
// Chains of products replayed as a graph, us a product, before (four warps, the other CTAs' tiles read behind a first and kept
// until a second barrier) and now: 64 x 1024 x 512 7.6 / 6.1, 64 x 288 x 1024 7.1 / 5.8, 6 x 256 x 512 5.4 / 4.0,
// 128 x 512 x 512 6.5 / 5.3, 250 x 784 x 1000 18.7 / 16.4; four k contiguous in B 8.1 / 7.6, 7.6 / 7.1, 5.8 / 4.2, 7.0 / 6.3, 20.8 / 19.3.
#include <cuda_runtime.h>
#include <cstdint>

#include "kernels.h"
#include "launch.h"
#include "tc_util.cuh"

namespace b200 {
namespace {

constexpr int FSTAGES = 3;

// WM x WN warps side by side, WK of them sharing the k of a stage; FK: depth of a stage.
template <int WM_, int WN_, int WK_>
struct FmaCfg {
  static constexpr int WM = WM_, WN = WN_, WK = WK_;
  static constexpr int THREADS = WM * WN * WK * 32;
  static constexpr int TM = 32 * WM, TN = 64 * WN, FK = WK >= 4 ? 64 : 32;
  static constexpr int KROW = FK + 4;                           // row stride of k-contiguous tiles: 16-byte rows, spread over banks
  static constexpr int AROW = TM + 4, BROW = TN + 4;            // the same for row-contiguous ones
  static constexpr int A_FLOATS = TM * KROW > FK * AROW ? TM * KROW : FK * AROW;
  static constexpr int B_FLOATS = TN * KROW > FK * BROW ? TN * KROW : FK * BROW;
  static constexpr int STAGE = A_FLOATS + B_FLOATS;
  static constexpr int RING = FSTAGES * STAGE, INBOX = TM * TN;  // floats; the inbox takes the sums of the cluster's other CTAs
  static constexpr int smem(int split) { return (RING + (split > 1 ? INBOX : 0)) * 4; }
  static_assert(RING >= WK * TM * BROW, "the warps' partial tiles reuse the stages");
};
// Asked for instead when every CTA can have an SM to itself: the CTAs of a cluster are otherwise packed two to an SM while
// other SMs stand idle.
constexpr int F_SMEM_ALONE = 118 * 1024;
static_assert(FmaCfg<1, 1, 8>::smem(2) <= F_SMEM_ALONE && FmaCfg<2, 1, 4>::smem(2) <= F_SMEM_ALONE && FmaCfg<2, 2, 2>::smem(2) <= F_SMEM_ALONE, "");

bool g_programmatic = true;

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

// c += a * (bx, by), each product and sum rounded as fmaf does. PAIR: in one instruction (fma.rn.f32x2), where bx and by were
// loaded side by side; packing them first costs more than it saves.
template <bool PAIR>
__device__ __forceinline__ void fma2(float2& c, float a, float bx, float by) {
  if (PAIR)
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b64 z, {%0, %1};\n\t"
        "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "+f"(c.x), "+f"(c.y) : "f"(a), "f"(bx), "f"(by));
  else { c.x = fmaf(a, bx, c.x); c.y = fmaf(a, by, c.y); }
}

// One operand's tile of T outer indices (m or n) by FK k, stage after stage. KC: k is contiguous (outer stride `ld`), else
// the outer index is (k stride `ld`). VEC: 16-byte copies. What does not change from stage to stage is worked out once.
template <int T, int FK, bool KC, bool VEC, int THREADS>
struct Loader {
  static constexpr int PER = VEC ? 4 : 1;                       // floats per copy
  static constexpr int COUNT = T * FK / PER / THREADS;
  static constexpr int LINE = (KC ? FK : T) / PER;              // copies along memory
  static constexpr int STEP = THREADS / LINE;                  // lines between a thread's copies
  static_assert(THREADS % LINE == 0, "a thread keeps its place in the line");
  const float *src, *at;                                        // a valid address; this thread's first element of the next stage
  long long step, advance;
  uint32_t dst, fine = 0;                                       // fine: which copies have their outer index inside
  int k;                                                        // k of the first copy inside the stage
  __device__ __forceinline__ Loader(const float* s, long long ld, int o0, int extent, int k0, int tid) : src(s) {
    const int line = tid / LINE, pos = (tid % LINE) * PER;
    const int o = KC ? line : pos;
    k = KC ? pos : line;
    at = s + (long long)(o0 + o) * (KC ? ld : 1) + (long long)(k0 + k) * (KC ? 1 : ld);
    step = STEP * ld;
    advance = KC ? FK : FK * ld;
    dst = 4u * (uint32_t)(KC ? o * (FK + 4) + k : k * (T + 4) + o);
#pragma unroll
    for (int q = 0; q < COUNT; ++q) fine |= (o0 + o + (KC ? q * STEP : 0) < extent ? 1u : 0u) << q;
  }
  __device__ __forceinline__ void load(uint32_t stage, int left) {      // left: k that remain from the start of this stage
    const float* from = at;
#pragma unroll
    for (int q = 0; q < COUNT; ++q) {
      const bool valid = ((fine >> q) & 1u) && k + (KC ? 0 : q * STEP) < left;
      const uint32_t d = stage + dst + 4u * (uint32_t)(q * STEP * (KC ? FK + 4 : T + 4));
      if (VEC) copy16(d, valid ? from : src, valid);
      else copy4(d, valid ? from : src, valid);
      from += step;
    }
    at += advance;
  }
};

template <class Cfg, bool AKC, bool BKC, bool AVEC, bool BVEC>
__global__ void __launch_bounds__(Cfg::THREADS) gemm32_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C,
                                                        Gemm32Launch p) {
  extern __shared__ __align__(16) float f_smem[];
  constexpr int TM = Cfg::TM, TN = Cfg::TN, FK = Cfg::FK, KROW = Cfg::KROW, THREADS = Cfg::THREADS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lx = lane & 7, ly = lane >> 3;
  const int wk = warp % Cfg::WK, wm = warp / Cfg::WK % Cfg::WM, wn = warp / (Cfg::WK * Cfg::WM);
  const int S = p.split, rank = blockIdx.x % S, tile = blockIdx.x / S;
  const int tiles_m = (p.M + TM - 1) / TM;
  const int m0 = (tile % tiles_m) * TM, n0 = (tile / tiles_m) * TN, g = blockIdx.y;
  const int chunk = ((p.K + S - 1) / S + 3) / 4 * 4;
  const int kbeg = min(p.K, rank * chunk), kend = min(p.K, kbeg + chunk);
  const int steps = (kend - kbeg + FK - 1) / FK;
  const float* Ag = A + (long long)g * p.a_gs;
  const float* Bg = B + (long long)g * p.b_gs;
  // rows and columns of a thread inside its warp's 32 x 64: four apart or eight apart where the tile's rows are k-contiguous
  // (neighbouring lanes read neighbouring rows), else two runs of four
  auto row = [&](int i) { return 32 * wm + (AKC ? ly + 4 * i : 16 * (i >> 2) + 4 * ly + (i & 3)); };
  auto col = [&](int j) { return 64 * wn + (BKC ? lx + 8 * j : 32 * (j >> 2) + 4 * lx + (j & 3)); };
  Loader<TM, FK, AKC, AVEC, THREADS> la(Ag, p.a_ld, m0, p.M, kbeg, tid);
  Loader<TN, FK, BKC, BVEC, THREADS> lb(Bg, p.b_ld, n0, p.N, kbeg, tid);
  if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");    // every CTA of the cluster is there: waited for in front of the exchange
  pdl_prologue();
  auto load = [&](int s) {
    if (s < steps) {
      const uint32_t a = smem_u32(f_smem + (s % FSTAGES) * Cfg::STAGE);
      la.load(a, kend - kbeg - s * FK);
      lb.load(a + 4u * Cfg::A_FLOATS, kend - kbeg - s * FK);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float2 acc[8][4];                                  // two columns each
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
  for (int s = 0; s < FSTAGES - 1; ++s) load(s);
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();
    load(s + FSTAGES - 1);
    const float* as = f_smem + (s % FSTAGES) * Cfg::STAGE;
    const float* bs = as + Cfg::A_FLOATS;
    const int quads = min(FK, kend - kbeg - s * FK + 3) / 4;    // k past the end read as zero
#pragma unroll 2
    for (int kq = wk; kq < quads; kq += Cfg::WK) {
      float a[8][4], b[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        // k-contiguous: outer index i, four k; else k = i / 2, outer indices 4 (i % 2) ..
        const float4 t = *reinterpret_cast<const float4*>(AKC ? as + row(i) * KROW + 4 * kq : as + (4 * kq + (i >> 1)) * Cfg::AROW + row(4 * (i & 1)));
        const float4 u = *reinterpret_cast<const float4*>(BKC ? bs + col(i) * KROW + 4 * kq : bs + (4 * kq + (i >> 1)) * Cfg::BROW + col(4 * (i & 1)));
        if (AKC) { a[i][0] = t.x; a[i][1] = t.y; a[i][2] = t.z; a[i][3] = t.w; }
        else { const int o = 4 * (i & 1), k = i >> 1; a[o][k] = t.x; a[o + 1][k] = t.y; a[o + 2][k] = t.z; a[o + 3][k] = t.w; }
        if (BKC) { b[i][0] = u.x; b[i][1] = u.y; b[i][2] = u.z; b[i][3] = u.w; }
        else { const int o = 4 * (i & 1), k = i >> 1; b[o][k] = u.x; b[o + 1][k] = u.y; b[o + 2][k] = u.z; b[o + 3][k] = u.w; }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) fma2<!BKC>(acc[i][j], a[i][k], b[2 * j][k], b[2 * j + 1][k]);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  float* Cg = C + (long long)g * p.M * p.N;
  auto store4 = [&](int m, int n, float4 v) {        // four consecutive n
    if (m >= p.M || n >= p.N) return;
    float* out = Cg + (long long)m * p.N + n;
    if ((p.N & 3) == 0) { *reinterpret_cast<float4*>(out) = v; return; }
    out[0] = v.x;
    if (n + 1 < p.N) out[1] = v.y;
    if (n + 2 < p.N) out[2] = v.z;
    if (n + 3 < p.N) out[3] = v.w;
  };
  if (Cfg::WK == 1 && S == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + row(i);
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const float2 u = acc[i][j / 2], v = acc[i][j / 2 + 1];
        if (!BKC) store4(m, n0 + col(j), make_float4(u.x, u.y, v.x, v.y));
        else {
          const float w[4] = {u.x, u.y, v.x, v.y};
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (m < p.M && n0 + col(j + q) < p.N) Cg[(long long)m * p.N + n0 + col(j + q)] = w[q];
        }
      }
    }
    return;
  }
  // the WK warps' partial tiles meet in shared memory, a thread adds up its quads of them in the order of the warps
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float* to = f_smem + (wk * TM + row(i)) * Cfg::BROW;
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      const float2 u = acc[i][j / 2], v = acc[i][j / 2 + 1];
      if (!BKC) *reinterpret_cast<float4*>(to + col(j)) = make_float4(u.x, u.y, v.x, v.y);
      else { to[col(j)] = u.x; to[col(j + 1)] = u.y; to[col(j + 2)] = v.x; to[col(j + 3)] = v.y; }
    }
  }
  __syncthreads();
  if (S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int rows = TM / S;                           // CTA r of the cluster gives out rows `rows` * r ..
  float* inbox = f_smem + Cfg::RING;                 // [sender][row][column]
#pragma unroll
  for (int e0 = 0; e0 < TM * (TN / 4); e0 += THREADS) {
    const int e = e0 + tid, r = e / (TN / 4), c = (e % (TN / 4)) * 4;
    float4 sum = *reinterpret_cast<const float4*>(f_smem + r * Cfg::BROW + c);
#pragma unroll
    for (int w = 1; w < Cfg::WK; ++w) {
      const float4 v = *reinterpret_cast<const float4*>(f_smem + (w * TM + r) * Cfg::BROW + c);
      sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    if (S == 1) { store4(m0 + r, n0 + c, sum); continue; }
    uint32_t to;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(inbox + (rank * rows + r % rows) * TN + c)), "r"(r / rows));
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(sum.x), "f"(sum.y), "f"(sum.z), "f"(sum.w) : "memory");
  }
  if (S == 1) return;
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int e = tid; e < rows * (TN / 4); e += THREADS) {
    const int r = e / (TN / 4), c = (e % (TN / 4)) * 4;
    float4 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q < S) v[q] = *reinterpret_cast<const float4*>(inbox + (q * rows + r) * TN + c);
    float4 sum = v[0];
#pragma unroll
    for (int q = 1; q < 8; ++q)
      if (q < S) { sum.x += v[q].x; sum.y += v[q].y; sum.z += v[q].z; sum.w += v[q].w; }
    store4(m0 + rank * rows + r, n0 + c, sum);
  }
}

template <class Cfg, bool AKC, bool BKC, bool AVEC, bool BVEC>
cudaError_t launch(const Gemm32Launch& p, const float* A, const float* B, float* C, cudaStream_t stream) {
  static bool done[64];
  auto* kernel = gemm32_kernel<Cfg, AKC, BKC, AVEC, BVEC>;
  if (first_use_on_this_device(done))
    if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM_ALONE)) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(((p.M + Cfg::TM - 1) / Cfg::TM) * (long long)((p.N + Cfg::TN - 1) / Cfg::TN) * p.split), (unsigned)p.G, 1);
  cfg.blockDim = dim3(Cfg::THREADS, 1, 1);
  cfg.dynamicSmemBytes = (long long)cfg.gridDim.x * p.G <= gemm32_resident(p.split) ? F_SMEM_ALONE : Cfg::smem(p.split);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (p.split > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)p.split;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (g_programmatic) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = (unsigned)n;
  return launch_kernel(cfg, kernel, A, B, C, p);
}

template <class Cfg, bool AKC, bool BKC>
cudaError_t launch_vec(const Gemm32Launch& p, const float* A, const float* B, float* C, cudaStream_t s) {
  if (p.a_vec) return p.b_vec ? launch<Cfg, AKC, BKC, true, true>(p, A, B, C, s) : launch<Cfg, AKC, BKC, true, false>(p, A, B, C, s);
  return p.b_vec ? launch<Cfg, AKC, BKC, false, true>(p, A, B, C, s) : launch<Cfg, AKC, BKC, false, false>(p, A, B, C, s);
}
template <class Cfg>
cudaError_t launch_layout(const Gemm32Launch& p, const float* A, const float* B, float* C, cudaStream_t s) {
  if (p.a_kc) return p.b_kc ? launch_vec<Cfg, true, true>(p, A, B, C, s) : launch_vec<Cfg, true, false>(p, A, B, C, s);
  return p.b_kc ? launch_vec<Cfg, false, true>(p, A, B, C, s) : launch_vec<Cfg, false, false>(p, A, B, C, s);
}

}  // namespace

void set_gemm32_programmatic_launch(bool on) { g_programmatic = on; }

cudaError_t launch_gemm32(const Gemm32Launch& p, const void* A, const void* B, void* C, cudaStream_t stream, int* launches) {
  if (p.G > 65535) return cudaErrorInvalidValue;
  const float *a = (const float*)A, *b = (const float*)B;
  cudaError_t e = p.tile == 0   ? launch_layout<FmaCfg<1, 1, 8>>(p, a, b, (float*)C, stream)
                  : p.tile == 1 ? launch_layout<FmaCfg<2, 1, 4>>(p, a, b, (float*)C, stream)
                  : p.tile == 2 ? launch_layout<FmaCfg<2, 2, 2>>(p, a, b, (float*)C, stream)
                                : launch_layout<FmaCfg<2, 2, 1>>(p, a, b, (float*)C, stream);
  if (e == cudaSuccess) ++*launches;
  return e;
}

}  // namespace b200
