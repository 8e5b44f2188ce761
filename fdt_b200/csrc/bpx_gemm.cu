// bpx_gemm.cu -- BF16 GEMM on the 5th-generation tensor cores (tcgen05), FP32 accumulation in
// tensor memory, with the fused epilogues of the learned initialiser's network.  No counterpart in
// the reference (xfibres_gpu has no learned part).
//
//   D[M][N] = sum_k A(m,k) B(n,k)      A, B bf16; D fp32 in TMEM
//
// Operands are read by TMA straight from row-major global tensors in either orientation:
//   * K-major  (the contraction index is the contiguous one): A = X[M][K], B = W[N][K];
//   * MN-major (M resp. N is the contiguous one): A stored [K][M], B stored [K][N].
// A rank-2 tensor map copies boxes whose rows are 64 elements, one 128-byte swizzle span, so the copy
// engine moves whole lines.  As 16-byte rows of an unswizzled core-matrix layout, which it also takes, the
// copies were most of a tile's time: 36.0 against 23.2 us for 32768 rows, 256 columns, K = 256 with bias
// and GELU (warps issuing 35% and 48% of the active cycles), and 333 against 215 us for the whole
// inference of 65536 rows of 288 inputs.  A chunk of 64 along K is
//   K-major tile   [rows][64]: 8-row atoms of 1024 B (SBO); the next 16 of K are 32 B further in the span
//   MN-major tile  [MN/64][64 of K][64]: atoms of 8 along K (SBO 1024 B), the next 64 of MN 8192 B on (LBO);
//                  the next 16 of K are two atoms (2048 B) further
// One thread issues TMA and MMA (M = 128, N = tile width <= 256, K = 16 per instruction) through
// an mbarrier ring of two to four stages; eight warps then read the accumulator (tcgen05.ld: warp w
// the 32 TMEM lanes w%4, every second block of 32 columns) and run the epilogue.  Every mbarrier
// wait is bounded (about a second), after which the kernel records an error code, waits (bounded) for
// its own copies and MMAs and releases its tensor memory (bpx_ring.h).
//
// The network's contractions are 2 to 5 chunks deep, so most of a CTA's time is its epilogue (256 erff per
// row of a 256-wide tile): bound by FP32 issue and by the loads that precede it, not by the tensor pipe.  Hence eight
// epilogue warps and two CTAs per SM, a tile width chosen so that the CTAs fill the device
// (choose_ntile), and for the weight gradients, whose output is a few tiles but whose contraction is
// the whole batch, a split of the contraction over CTAs (GemmArgs::split; the partial sums are added
// in split order by the caller's reduction, so a run reproduces) with all layers in one launch.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>

#include "bpx_gemm.h"
#include "bpx_internal.h"
#include "bpx_ring.h"

namespace bpx {
namespace gemm {

constexpr int kTileM = 128;
constexpr int kChunkK = 64;
constexpr int kSpan = 64;  // elements of a 128-byte swizzle span
constexpr int kThreads = 256;
constexpr int kMaxStages = 4;
constexpr long long kWaitCycles = 2000000000ll;  // ~1 s at 2 GHz
// epilogue staging per warp: a 32 x 32 fp32 block (rows padded to 36 floats) or, in the same place, a
// 32 x 32 bf16 block (rows padded to 80 bytes); both pitches keep 16-byte alignment and spread a
// quarter-warp's 16-byte accesses over distinct banks
constexpr int kPitchF = 36;
constexpr int kPitchB = 80;
constexpr int kEpiWarpBytes = 32 * kPitchF * 4;
static_assert((kThreads / 32) * kEpiWarpBytes <= 2 * (kTileM + 32) * kChunkK * 2, "epilogue tiles must fit two stages");
static_assert(kEpiWarpBytes % 16 == 0 && 32 * kPitchB <= kEpiWarpBytes, "the bf16 block shares the fp32 block's place");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try(bar, parity))
    if (clock64() - t0 > kWaitCycles) return false;
  return true;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      :
      : "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}

// shared-memory matrix descriptor: 128-byte swizzle, Blackwell descriptor version 1
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" : : "r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

__device__ __forceinline__ uint16_t to_bf16(float x) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return (uint32_t)__bfloat16_as_ushort(p.x) | ((uint32_t)__bfloat16_as_ushort(p.y) << 16);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

struct Smem {
  float bias[256];  // the tile's bias columns, staged once for the epilogue (16-byte aligned)
  uint64_t full[kMaxStages], empty[kMaxStages], done;
  uint32_t tmem_base;
};

// the problems of a launch; problem p has CTAs first[p] .. first[p+1]-1, its tiles along M fastest, then
// along N, then the splits
struct Batch {
  CUtensorMap a[kMaxProblems], b[kMaxProblems];
  GemmArgs g[kMaxProblems];
  int first[kMaxProblems + 1];
  int n, stages;
};

__host__ __device__ inline int tiles_m(const GemmArgs& g) { return (g.M + kTileM - 1) / kTileM; }
__host__ __device__ inline int tiles_n(const GemmArgs& g) { return (g.N + g.ntile - 1) / g.ntile; }

// a stage's bytes of B: an MN-major tile takes whole spans
__host__ __device__ inline uint32_t b_stage_bytes(const GemmArgs& g) {
  return (uint32_t)(g.b_mn && g.ntile < kSpan ? kSpan : g.ntile) * kChunkK * 2;
}

__global__ void __launch_bounds__(kThreads, 2) gemm_kernel(const __grid_constant__ Batch batch) {
  extern __shared__ __align__(1024) unsigned char dsmem[];
  int prob = 0;
  while (prob + 1 < batch.n && (int)blockIdx.x >= batch.first[prob + 1]) ++prob;
  const GemmArgs& g = batch.g[prob];
  const CUtensorMap &map_a = batch.a[prob], &map_b = batch.b[prob];
  const int stages = batch.stages;
  const int tile = blockIdx.x - batch.first[prob];
  const int tm = tiles_m(g), tn = tiles_n(g);
  const int bx = tile % tm, by = tile / tm % tn, bz = tile / (tm * tn);
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(dsmem) + 1023) & ~uintptr_t(1023));
  const int nt = g.ntile;
  const uint32_t a_bytes = kTileM * kChunkK * 2, b_bytes = b_stage_bytes(g);
  const uint32_t stage_bytes = a_bytes + b_bytes;
  Smem* sm = reinterpret_cast<Smem*>(base + stages * stage_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = bx * kTileM, n0 = by * nt;
  // this CTA's chunks of the contraction: [kc0, kc1)
  const int nk = (g.K + kChunkK - 1) / kChunkK, nsplit = g.split > 1 ? g.split : 1;
  const int kc0 = (int)((long long)nk * bz / nsplit), kc1 = (int)((long long)nk * (bz + 1) / nsplit);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" : : "r"(smem_u32(&sm->tmem_base)), "r"(nt));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(smem_u32(&sm->full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(smem_u32(&sm->empty[s])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(smem_u32(&sm->done)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm->tmem_base;

  if (threadIdx.x == 0) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)g.a_mn << 15) | ((uint32_t)g.b_mn << 16) |
                           ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
    struct Ops {
      const GemmArgs& g;
      const CUtensorMap &map_a, &map_b;
      Smem* sm;
      uint32_t base, a_bytes, b_bytes, tmem, idesc;
      int m0, n0, kc0;
      __device__ __forceinline__ uint32_t place(int s) const { return base + (uint32_t)s * (a_bytes + b_bytes); }
      __device__ __forceinline__ void copy(int c, int s) const {
        const uint32_t sa = place(s), sb = sa + a_bytes;
        const uint32_t bar = smem_u32(&sm->full[s]);
        const int k = (kc0 + c) * kChunkK;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" : : "r"(bar), "r"(a_bytes + b_bytes) : "memory");
        if (g.a_mn)
          for (int j = 0; j < kTileM / kSpan; ++j) tma_load_2d(sa + j * kSpan * kChunkK * 2, &map_a, m0 + j * kSpan, k, bar);
        else
          tma_load_2d(sa, &map_a, k, m0, bar);
        if (g.b_mn)
          for (uint32_t j = 0; j * kSpan * kChunkK * 2 < b_bytes; ++j)
            tma_load_2d(sb + j * kSpan * kChunkK * 2, &map_b, n0 + j * kSpan, k, bar);
        else
          tma_load_2d(sb, &map_b, k, n0, bar);
      }
      __device__ __forceinline__ bool wait_full(int s, uint32_t ph) const { return mbar_wait(smem_u32(&sm->full[s]), ph); }
      __device__ __forceinline__ bool wait_empty(int s, uint32_t ph) const { return mbar_wait(smem_u32(&sm->empty[s]), ph); }
      __device__ __forceinline__ void drain(int s, uint32_t ph) const { mbar_wait(smem_u32(&sm->full[s]), ph); }
      __device__ __forceinline__ void multiply(int c, int s) const {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = place(s), sb = sa + a_bytes;
#pragma unroll
        for (int ks = 0; ks < kChunkK / 16; ++ks) {
          const uint64_t da = g.a_mn ? smem_desc(sa + ks * 2048, kSpan * kChunkK * 2, 1024) : smem_desc(sa + ks * 32, 0, 1024);
          const uint64_t db = g.b_mn ? smem_desc(sb + ks * 2048, kSpan * kChunkK * 2, 1024) : smem_desc(sb + ks * 32, 0, 1024);
          mma_bf16(tmem, da, db, idesc, c != 0 || ks != 0);
        }
        mma_commit(smem_u32(&sm->empty[s]));
      }
      // arrives once every MMA issued has completed
      __device__ __forceinline__ void finish() const { mma_commit(smem_u32(&sm->done)); }
    };
    const Ops ops{g, map_a, map_b, sm, smem_u32(base), a_bytes, b_bytes, tmem, idesc, m0, n0, kc0};
    if (!ring_contract(ops, kc1 - kc0, stages) && g.error) atomicExch(g.error, 1);
  }
  __syncwarp();
  const bool done = mbar_wait(smem_u32(&sm->done), 0);
  if (!done && g.error) atomicExch(g.error, 2);
  // every lane of a warp adds the same bias columns: stage them in shared memory once, so the
  // epilogue reads them as broadcast 16-byte loads instead of 32 global loads per column chunk
  const bool use_bias = g.bias && (g.epi == kEpiBias || g.epi == kEpiBiasGelu);
  if (use_bias)
    for (int t = threadIdx.x; t < nt; t += kThreads) sm->bias[t] = n0 + t < g.N ? g.bias[n0 + t] : 0.f;
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  // epilogue: warp w owns accumulator rows 32(w%4) .. +31 (its TMEM lanes) of every second block of 32
  // columns.  A lane
  // holds one row of a 32x32 block, so it is turned around through a per-warp shared-memory tile:
  // lanes write their rows, then read the block back so that consecutive lanes cover consecutive
  // columns of a row, and the global stores (and the GELU-derivative's loads of z) are whole
  // 128-byte lines instead of 32 rows touched per instruction.  The tiles reuse the operand stages,
  // idle once every MMA has completed (the done barrier above).
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  float* tf = reinterpret_cast<float*>(base + warp * kEpiWarpBytes);  // [32][kPitchF] fp32 block
  unsigned char* tb = base + warp * kEpiWarpBytes;  // [32][kPitchB] bytes, bf16 block (the same place)
  const bool all_done = __all_sync(0xffffffffu, done);
  const int quad = warp & 3, half = warp >> 2;
  const int row0 = m0 + 32 * quad;
  auto aligned16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  // the block's 32 rows x 32 fp32 columns, lane = row, to out (row-major, leading dimension ld)
  auto put_f32 = [&](const float (&v)[32], float* out, int ld, int col0) {
    float4* t4 = reinterpret_cast<float4*>(tf + lane * kPitchF);
#pragma unroll
    for (int q = 0; q < 8; ++q) t4[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 4 * i + (lane >> 3), q = lane & 7;
      const int grow = row0 + r, gcol = col0 + 4 * q;
      const float4 x = reinterpret_cast<const float4*>(tf + r * kPitchF)[q];
      if (grow < g.M && gcol < g.N) {
        float* o = out + (size_t)grow * ld + gcol;
        if (gcol + 3 < g.N && aligned16(o)) {
          *reinterpret_cast<float4*>(o) = x;
        } else {
          const float e[4] = {x.x, x.y, x.z, x.w};
          for (int j = 0; j < 4 && gcol + j < g.N; ++j) o[j] = e[j];
        }
      }
    }
    __syncwarp();
  };
  // the same for bf16 values (32 per lane, packed in pairs)
  auto put_bf16 = [&](const uint32_t (&h)[16], uint16_t* out, int ld, int col0) {
    uint4* t4 = reinterpret_cast<uint4*>(tb + lane * kPitchB);
#pragma unroll
    for (int q = 0; q < 4; ++q) t4[q] = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 8 * i + (lane >> 2), q = lane & 3;
      const int grow = row0 + r, gcol = col0 + 8 * q;
      const uint4 x = reinterpret_cast<const uint4*>(tb + r * kPitchB)[q];
      if (grow < g.M && gcol < g.N) {
        uint16_t* o = out + (size_t)grow * ld + gcol;
        if (gcol + 7 < g.N && aligned16(o)) {
          *reinterpret_cast<uint4*>(o) = x;
        } else {
          const uint32_t w[4] = {x.x, x.y, x.z, x.w};
          for (int j = 0; j < 8 && gcol + j < g.N; ++j) o[j] = (uint16_t)(w[j >> 1] >> (16 * (j & 1)));
        }
      }
    }
    __syncwarp();
  };
  // z of the GELU derivative for the block's rows: coalesced loads into the fp32 tile, then each
  // lane reads its own row (columns past N read as 0)
  auto get_f32 = [&](const float* in, int ld, int col0, float (&zv)[32]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 4 * i + (lane >> 3), q = lane & 7;
      const int grow = row0 + r, gcol = col0 + 4 * q;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (grow < g.M && gcol < g.N) {
        const float* z = in + (size_t)grow * ld + gcol;
        if (gcol + 3 < g.N && aligned16(z)) {
          x = *reinterpret_cast<const float4*>(z);
        } else {
          float e[4] = {0.f, 0.f, 0.f, 0.f};
          for (int j = 0; j < 4 && gcol + j < g.N; ++j) e[j] = z[j];
          x = make_float4(e[0], e[1], e[2], e[3]);
        }
      }
      reinterpret_cast<float4*>(tf + r * kPitchF)[q] = x;
    }
    __syncwarp();
    const float4* t4 = reinterpret_cast<const float4*>(tf + lane * kPitchF);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 x = t4[q];
      zv[4 * q] = x.x;
      zv[4 * q + 1] = x.y;
      zv[4 * q + 2] = x.z;
      zv[4 * q + 3] = x.w;
    }
    __syncwarp();
  };
  float* out_f32 = g.out_f32 ? g.out_f32 + (size_t)bz * g.split_stride : nullptr;
  for (int c = half; c < nt / 32; c += 2) {
    float v[32];
    __syncwarp();
    tmem_ld32(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(c * 32), v);
    const int col0 = n0 + c * 32;
    if (!all_done || row0 >= g.M || col0 >= g.N) continue;  // warp-uniform
    const float4* sb4 = reinterpret_cast<const float4*>(sm->bias + c * 32);
    if (use_bias) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 b4 = sb4[j / 4];
        v[j] += b4.x;
        v[j + 1] += b4.y;
        v[j + 2] += b4.z;
        v[j + 3] += b4.w;
      }
    }
    if (g.epi == kEpiStoreF32 || g.epi == kEpiBias) {
      put_f32(v, out_f32, g.ld_out, col0);
    } else if (g.epi == kEpiBiasGelu) {
      if (out_f32) put_f32(v, out_f32, g.ld_out, col0);
      uint32_t h[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        h[j] = (uint32_t)to_bf16(gelu(v[2 * j])) | ((uint32_t)to_bf16(gelu(v[2 * j + 1])) << 16);
      put_bf16(h, g.out_bf16, g.ld_bf16, col0);
    } else {  // kEpiGeluGrad: dZ = (dZ_next W) * gelu'(z)
      float zv[32];
      get_f32(g.zin, g.ld_zin, col0, zv);
      uint32_t h[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        h[j] = (uint32_t)to_bf16(v[2 * j] * gelu_grad(zv[2 * j])) |
               ((uint32_t)to_bf16(v[2 * j + 1] * gelu_grad(zv[2 * j + 1])) << 16);
      put_bf16(h, g.out_bf16, g.ld_bf16, col0);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" : : "r"(tmem), "r"(nt));
  }
}

// ---------------------------------------------------------------------------------------------
// A chain of layers (network inference): every layer of 128 rows in one CTA
// ---------------------------------------------------------------------------------------------
// Bound by the FP32 issue of the epilogues (a GELU per element and hidden layer).  The rows' activations
// stay in shared memory, as the spans the next layer's products read; the weights (0.5 MB for all
// layers, L2-resident) pass through a ring of pieces of 64 along K by up to 128 output columns.  One
// CTA has an SM to itself, so that the ring holds a whole layer, which lands during the epilogue of
// the layer before, and the sums have two places in tensor memory: a layer's products of a span
// begin when the epilogue has written that span, and only the last span's are waited for.
// Inference of 65536 rows of 288 inputs: 215 us as five launches per 32768 rows (which wrote and read
// their activations, 2 x 16 MB, and waited for copies in every tile), 162 us so; 5000 rows 74 and 59 us,
// 300 rows 60 and 54 us.  Two CTAs of 128 rows to an SM with a ring of three pieces and one place for the
// sums measured 160, 74 and 70 us.  Warps issue 59% of the active cycles; what is left is layer 0's copies
// at a tile's start and the rounding of the tiles to whole rounds of the SMs.
// The products of a tile are those of gemm_kernel in the same order, so the results are too.
constexpr int kPieceN = 128;
constexpr int kRing = 10;
constexpr int kEpiWarps = 16;
constexpr int kChainThreads = 32 * kEpiWarps + 64;  // a warp that issues the copies, one for the products
constexpr int kBlockN = 16;                         // columns of a span that a warp takes
constexpr int kSpanBytes = kTileM * kSpan * 2;
constexpr int kActSpans = kChainWidth / kSpan;
static_assert(kSpanBytes == kPieceN * kChunkK * 2, "a span of activations is as large as a piece of weights");
static_assert(kEpiWarps == kTileM / 32 * (kSpan / kBlockN), "the epilogue warps cover a span");

struct Chain {
  CUtensorMap x, w[kChainLayers];
  const float* bias[kChainLayers];
  float* out;
  int* error;
  int rows, nin;
};

__device__ __forceinline__ float4 bias4(const float* b, bool vec) {
  if (vec) return __ldg(reinterpret_cast<const float4*>(b));
  return make_float4(__ldg(b), __ldg(b + 1), __ldg(b + 2), __ldg(b + 3));
}

struct ChainBars {
  uint64_t full[kRing], empty[kRing], written[kActSpans], done, drained;
  uint32_t tmem_base;
  int failed;
};

constexpr size_t kChainSmem = (size_t)(kActSpans + kRing) * kSpanBytes + sizeof(ChainBars);
static_assert(kChainSmem <= 227 * 1024, "shared memory of a CTA");

// a bounded wait that also ends when another one has given up
__device__ __forceinline__ bool chain_wait(ChainBars* sm, const uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  if (mbar_try(addr, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try(addr, parity)) {
    if (*(volatile int*)&sm->failed) return false;
    if (clock64() - t0 > kWaitCycles) {
      *(volatile int*)&sm->failed = 1;
      return false;
    }
  }
  return true;
}

// One thread copies the pieces, another multiplies: a single one, which also divided for slots and rounds,
// took 1300 cycles a piece, 3000 beside busy epilogue warps, and was the kernel's bound (205 us for the
// 65536 rows).  The last layer's pieces have kChainOut columns.
using ChainRing = RingChain<kChainLayers, kActSpans, kRing, kChainWidth / kPieceN>;

struct ChainCopy {
  const Chain& c;
  ChainBars* sm;
  uint32_t act, ring;
  int m0;
  __device__ __forceinline__ bool wait_empty(int slot, uint32_t ph) const { return chain_wait(sm, &sm->empty[slot], ph); }
  __device__ __forceinline__ void drain(int slot, uint32_t ph) const { mbar_wait(smem_u32(&sm->full[slot]), ph); }
  __device__ __forceinline__ void copy(int layer, int kc, int half, int slot) const {
    const bool with_x = layer == 0 && half == 0;
    const uint32_t w_bytes = ChainRing::halves(layer) == 1 ? kChainOut * kChunkK * 2 : kSpanBytes;
    const uint32_t bar = smem_u32(&sm->full[slot]), bytes = w_bytes + (with_x ? kSpanBytes : 0);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" : : "r"(bar), "r"(bytes) : "memory");
    if (with_x) tma_load_2d(act + (kc % kActSpans) * kSpanBytes, &c.x, kc * kChunkK, m0, bar);
    tma_load_2d(ring + slot * kSpanBytes, &c.w[layer], kc * kChunkK, half * kPieceN, bar);
  }
};

__device__ __forceinline__ bool chain_multiply(ChainBars* sm, uint32_t act, uint32_t ring, uint32_t tmem, int nk0) {
  int slot = 0;
  uint32_t ph = 0;
  const uint64_t act_desc = smem_desc(act, 0, 1024), ring_desc = smem_desc(ring, 0, 1024);
  for (int layer = 0; layer < kChainLayers; ++layer) {
    const int halves = ChainRing::halves(layer), nk = ChainRing::chunks(layer, nk0), n = halves == 1 ? kChainOut : kPieceN;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
    const uint32_t sums = tmem + (layer & 1) * kChainWidth;
    for (int kc = 0; kc < nk; ++kc) {
      if (layer > 0 && !chain_wait(sm, &sm->written[kc], (layer - 1) & 1)) return false;
      const uint64_t da = act_desc + (uint64_t)((kc % kActSpans) * (kSpanBytes >> 4));
      for (int half = 0; half < halves; ++half) {
        if (!chain_wait(sm, &sm->full[slot], ph)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t db = ring_desc + (uint64_t)(slot * (kSpanBytes >> 4));
#pragma unroll
        for (int ks = 0; ks < kChunkK / 16; ++ks)
          mma_bf16(sums + half * kPieceN, da + 2 * ks, db + 2 * ks, idesc, kc != 0 || ks != 0);
        mma_commit(smem_u32(&sm->empty[slot]));
        if (++slot == kRing) {
          slot = 0;
          ph ^= 1;
        }
      }
    }
    mma_commit(smem_u32(&sm->done));
  }
  return true;
}

__global__ void __launch_bounds__(kChainThreads, 1) chain_kernel(const __grid_constant__ Chain c) {
  extern __shared__ __align__(1024) unsigned char dsmem[];
  unsigned char* act = dsmem;
  unsigned char* ring = dsmem + kActSpans * kSpanBytes;
  ChainBars* sm = reinterpret_cast<ChainBars*>(ring + kRing * kSpanBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kTileM;
  if (smem_u32(dsmem) & 1023) {  // the swizzled spans want what the declaration asks for
    if (threadIdx.x == 0 && c.error) atomicExch(c.error, 3);
    return;
  }

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" : : "r"(smem_u32(&sm->tmem_base)), "r"(2 * kChainWidth));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    const auto init = [](const uint64_t* bar, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" : : "r"(smem_u32(bar)), "r"(count));
    };
    for (int s = 0; s < kRing; ++s) {
      init(&sm->full[s], 1);
      init(&sm->empty[s], 1);
    }
    for (int s = 0; s < kActSpans; ++s) init(&sm->written[s], kEpiWarps);
    init(&sm->done, 1);
    init(&sm->drained, 1);
    sm->failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm->tmem_base;

  const int nk0 = (c.nin + kChunkK - 1) / kChunkK;
  if (warp == kEpiWarps) {
    if (lane == 0) {
      const ChainCopy ops{c, sm, smem_u32(act), smem_u32(ring), m0};
      ChainRing::copy(ops, nk0);
    }
    __syncwarp();
  } else if (warp == kEpiWarps + 1) {
    if (lane == 0 && !chain_multiply(sm, smem_u32(act), smem_u32(ring), tmem, nk0)) {
      mma_commit(smem_u32(&sm->drained));  // the products in flight end before the shared memory goes
      mbar_wait(smem_u32(&sm->drained), 0);
    }
    __syncwarp();
  } else {
    // lane = row; a warp takes kBlockN columns of each span
    const int quad = warp & 3, part = warp >> 2, row = 32 * quad + lane;
    const uint32_t tmem_row = tmem + ((uint32_t)(32 * quad) << 16);
    bool good = true;
    for (int layer = 0; layer < kChainLayers; ++layer) {
      good = __all_sync(0xffffffffu, chain_wait(sm, &sm->done, layer & 1));
      if (!good) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sums = tmem_row + (layer & 1) * kChainWidth;
      if (layer < kChainLayers - 1) {
        for (int span = 0; span < kActSpans; ++span) {
          float v[kBlockN];
          tmem_ld16(sums + (uint32_t)(span * kSpan + part * kBlockN), v);
          const float* b = c.bias[layer] + span * kSpan + part * kBlockN;
          const bool vec = (reinterpret_cast<uintptr_t>(b) & 15) == 0;  // the parameters may lie anywhere
          unsigned char* dst = act + span * kSpanBytes + row * 128;
#pragma unroll
          for (int q = 0; q < kBlockN / 8; ++q) {
            const float4 b0 = bias4(b + 8 * q, vec), b1 = bias4(b + 8 * q + 4, vec);
            uint4 h;
            h.x = pack_bf16(gelu(v[8 * q] + b0.x), gelu(v[8 * q + 1] + b0.y));
            h.y = pack_bf16(gelu(v[8 * q + 2] + b0.z), gelu(v[8 * q + 3] + b0.w));
            h.z = pack_bf16(gelu(v[8 * q + 4] + b1.x), gelu(v[8 * q + 5] + b1.y));
            h.w = pack_bf16(gelu(v[8 * q + 6] + b1.z), gelu(v[8 * q + 7] + b1.w));
            *reinterpret_cast<uint4*>(dst + (((part * kBlockN / 8 + q) ^ (row & 7)) << 4)) = h;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads what was written here
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" : : "r"(smem_u32(&sm->written[span])) : "memory");
        }
      } else if (part == 0) {
        // the outputs: through a padded block of the (now unused) activations to whole lines
        float* tf = reinterpret_cast<float*>(act) + warp * 32 * 33;
        const float* b = c.bias[layer];
        for (int c0 = 0; c0 < kChainOut; c0 += kBlockN) {
          float v[kBlockN];
          tmem_ld16(sums + (uint32_t)c0, v);
#pragma unroll
          for (int j = 0; j < kBlockN; ++j) tf[lane * 33 + c0 + j] = v[j] + __ldg(b + c0 + j);
        }
        __syncwarp();
        for (int r = 0; r < 32; ++r) {
          const int grow = m0 + 32 * quad + r;
          if (grow < c.rows) c.out[(size_t)grow * kChainOut + lane] = tf[r * 33 + lane];
        }
      }
    }
    if (!good && lane == 0 && c.error) atomicExch(c.error, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" : : "r"(tmem), "r"(2 * kChainWidth));
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static std::once_flag once;
  static EncodeTiledFn fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// Tensor map over a row-major bf16 tensor [rows][cols] (leading dimension ld elements); box of one span
// by box_rows, 128-byte swizzle.
static bool make_map(CUtensorMap* m, const uint16_t* ptr, int rows, int cols, int ld, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {kSpan, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  std::memset(m, 0, sizeof(*m));
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// (narrower MN-major tiles of B still take a whole span)
size_t smem_bytes(int ntile, int stages) {
  return stages * (size_t)(kTileM * kChunkK * 2 + (ntile < kSpan ? kSpan : ntile) * kChunkK * 2) + 1024 + sizeof(Smem) + 64;
}

// Stages of the ring: as many as keep two CTAs on an SM (about 100 KB each) and the contraction can
// use; a wider tile's stage is larger, so 256 columns get two, 64 columns four.
int choose_stages(int ntile, int chunks) {
  const int fit = ntile >= 256 ? 2 : ntile >= 128 ? 3 : kMaxStages;
  return chunks < 2 ? 2 : chunks < fit ? chunks : fit;
}

int choose_ntile(int M, int N) {
  int nt = N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256;
  const long long tm = (M + kTileM - 1) / kTileM;
  while (nt > 64 && tm * ((N + nt - 1) / nt) < sm_count()) nt /= 2;
  return nt;
}

// The kernels' dynamic shared-memory limits are raised once per device, gemm_kernel's to what the largest ring
// needs, and never lowered: a launch with a smaller one needs less, and a CUDA graph whose nodes were
// captured with different tile widths stays launchable whatever was set last.
constexpr int kMaxDevices = 64;
cudaError_t set_smem_limits_once() {
  static std::mutex mu;
  static uint64_t done_ctx[kMaxDevices] = {0};  // context_id() the limit was set in (0: not set)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(mu);
  const uint64_t ctx = context_id();
  if (ctx != 0 && done_ctx[dev] == ctx) return cudaSuccess;
  size_t most = smem_bytes(256, 2);
  if (smem_bytes(128, 3) > most) most = smem_bytes(128, 3);
  if (smem_bytes(64, kMaxStages) > most) most = smem_bytes(64, kMaxStages);
  e = cudaFuncSetAttribute(gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChainSmem);
  if (e == cudaSuccess) done_ctx[dev] = context_id();
  return e;
}

const char* check(const GemmOperands& op, const GemmArgs& g) {
  if (g.M < 1 || g.N < 1 || g.K < 1) return "GEMM sizes must be positive";
  if (g.ntile != 32 && g.ntile != 64 && g.ntile != 128 && g.ntile != 256) return "GEMM tile width must be 32, 64, 128 or 256";
  if (((uintptr_t)op.a | (uintptr_t)op.b) & 15) return "GEMM operands must be 16-byte aligned";
  if ((op.lda | op.ldb) & 7) return "GEMM leading dimensions must be multiples of 8";
  // contiguous extents must be whole groups of 8 elements
  if ((g.a_mn ? g.M : g.K) % 8 || (g.b_mn ? g.N : g.K) % 8) return "GEMM contiguous extents must be multiples of 8";
  if (g.M > (1 << 24) || g.N > (1 << 24) || g.K > (1 << 24)) return "GEMM too large";
  if (g.split > (g.K + kChunkK - 1) / kChunkK) return "GEMM split into more parts than the contraction has chunks";
  return nullptr;
}

cudaError_t launch(const GemmOperands* op, const GemmArgs* g, int problems, cudaStream_t s, const char** why) {
  *why = nullptr;
  if (problems < 1 || problems > kMaxProblems) {
    *why = "GEMM problem count out of range";
    return cudaErrorInvalidValue;
  }
  Batch b;
  long long blocks = 0;
  int chunks = 0, nt = 0;
  for (int i = 0; i < problems; ++i) {
    *why = check(op[i], g[i]);
    if (*why) return cudaErrorInvalidValue;
    const bool ok_a = g[i].a_mn ? make_map(&b.a[i], op[i].a, g[i].K, g[i].M, op[i].lda, kChunkK)
                                : make_map(&b.a[i], op[i].a, g[i].M, g[i].K, op[i].lda, kTileM);
    const bool ok_b = g[i].b_mn ? make_map(&b.b[i], op[i].b, g[i].K, g[i].N, op[i].ldb, kChunkK)
                                : make_map(&b.b[i], op[i].b, g[i].N, g[i].K, op[i].ldb, g[i].ntile);
    if (!ok_a || !ok_b) {
      *why = "cuTensorMapEncodeTiled failed (driver entry point missing or unsupported tensor shape)";
      return cudaErrorInvalidValue;
    }
    b.g[i] = g[i];
    b.first[i] = (int)blocks;
    const int split = g[i].split > 1 ? g[i].split : 1;
    blocks += (long long)tiles_m(g[i]) * tiles_n(g[i]) * split;
    if (blocks > (1ll << 30)) {
      *why = "GEMM too large";
      return cudaErrorInvalidValue;
    }
    const int nk = ((g[i].K + kChunkK - 1) / kChunkK + split - 1) / split;
    if (nk > chunks) chunks = nk;
    if (g[i].ntile > nt) nt = g[i].ntile;
  }
  b.first[problems] = (int)blocks;
  b.n = problems;
  b.stages = choose_stages(nt, chunks);
  const cudaError_t attr = set_smem_limits_once();
  if (attr != cudaSuccess) return attr;
  gemm_kernel<<<(unsigned)blocks, kThreads, smem_bytes(nt, b.stages), s>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_chain(const ChainOperands& op, int rows, int nin, int* error, cudaStream_t s, const char** why) {
  *why = nullptr;
  Chain c;
  c.out = op.out;
  c.error = error;
  c.rows = rows;
  c.nin = nin;
  if (rows < 1 || nin < 1 || nin % 8) *why = "GEMM contiguous extents must be multiples of 8";
  if (((uintptr_t)op.x | (uintptr_t)op.w[0]) & 15) *why = "GEMM operands must be 16-byte aligned";
  if (nin > (1 << 24)) *why = "GEMM too large";
  if (*why) return cudaErrorInvalidValue;
  bool ok = make_map(&c.x, op.x, rows, nin, nin, kTileM);
  for (int l = 0; l < kChainLayers; ++l) {
    const bool last = l == kChainLayers - 1;
    const int k = l == 0 ? nin : kChainWidth, n = last ? kChainOut : kChainWidth;
    ok = ok && make_map(&c.w[l], op.w[l], n, k, k, last ? kChainOut : kPieceN);
    c.bias[l] = op.bias[l];
  }
  if (!ok) {
    *why = "cuTensorMapEncodeTiled failed (driver entry point missing or unsupported tensor shape)";
    return cudaErrorInvalidValue;
  }
  const cudaError_t attr = set_smem_limits_once();
  if (attr != cudaSuccess) return attr;
  chain_kernel<<<(unsigned)(((long long)rows + kTileM - 1) / kTileM), kChainThreads, kChainSmem, s>>>(c);
  return cudaGetLastError();
}

}  // namespace gemm
}  // namespace bpx
