// BF16 tensor-core GEMM (tcgen05 + TMA + tensor memory) with fused epilogues, and the
// small kernels of the surrogate network's training and gated inference. The surrogate
// has no reference counterpart: it maps a layer profile to channel-mean transmittance
// and is trained on spectra produced by this library's own engine.
//
// D[M, N] = A[M, K] . B[N, K]^T, A and B bf16 row-major with K contiguous ("K-major"),
// accumulated in float32 in tensor memory. The kernel is persistent (one CTA per SM,
// each looping over 128 x BN output tiles, BN = 256 or 128) and warp-specialised:
//   warp 0, lane 0   streams 128 x 64 tiles of A and BN x 64 tiles of B into a 4-stage
//                    shared-memory ring with TMA (128-byte swizzle, no multicast);
//                    each stage completes a "full" mbarrier;
//   warp 1, lane 0   issues tcgen05.mma (M = 128, N = BN, K = 16) four times per stage
//                    into one of two tensor-memory accumulators and frees the stage
//                    with tcgen05.commit on its "empty" mbarrier; a finished tile is
//                    signalled on the accumulator's "tmem_full" mbarrier;
//   warps 2-17       (the epilogue, four per SM sub-partition) each read 32 accumulator
//                    rows x a quarter of the columns with tcgen05.ld, apply the epilogue, store,
//                    and release the accumulator ("tmem_empty", one arrival per warp), so
//                    the epilogue of one tile overlaps the main loop of the next.
// Split-K (n_split > 1) is offered for the float32 mode only: split z writes its partial
// sum to out_f32 + z * split_stride and the consumer adds the partials in a fixed order
// (deterministic).
//
// Every mbarrier wait is bounded by wall-clock time (globaltimer); a wait that runs out
// marks the CTA failed, every role leaves its loop, the MMA warp drains its own
// outstanding MMAs, tensor memory is always freed and the caller's error word is raised.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <type_traits>

#include "lbl_common.cuh"

namespace lbl {

constexpr int GM = 128, GK = 64, GSTAGES = 4;
constexpr int G_A_BYTES = GM * GK * 2;                             // 16 KiB A tile per stage
// 4 per SM sub-partition; 8 warps instead: 1,426 against 1,411 us for a 4-member ensemble of
// 20,000 profiles, a training step the same
constexpr int G_EPI_WARPS = 16;
constexpr int G_EPI_GROUPS = G_EPI_WARPS / 4;                      // column groups of a tile
constexpr int G_THREADS = 64 + 32 * G_EPI_WARPS;                   // TMA warp, MMA warp, epilogue
constexpr unsigned long long G_WAIT_NS = 2000000000ull;            // 2 s per wait at most

template <int BN>
struct GemmCfg {
  static constexpr int B_BYTES = BN * GK * 2;
  static constexpr int STAGE_BYTES = G_A_BYTES + B_BYTES;
  static constexpr int TMEM_COLS = 2 * BN;                         // two float32 accumulators
  static constexpr int SMEM = GSTAGES * STAGE_BYTES + 1024 + 256;  // ring + alignment + barriers
  // kind::f16: D f32 (bits 4-5 = 1), A and B bf16 (bits 7-9, 10-12 = 1), both K-major
  // (bits 15, 16 = 0), N >> 3 at bit 17, M >> 4 at bit 24.
  static constexpr uint32_t IDESC =
      (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(GM >> 4) << 24);
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// Wait for the phase of the given parity; false when G_WAIT_NS elapsed first.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (true) {
    if (mbar_try(bar, parity)) return true;
    if (global_ns() - t0 > G_WAIT_NS) return false;
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          dst),
      "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: 128-byte
// rows (64 bf16), 8-row groups 1024 B apart (stride byte offset), descriptor version 1,
// layout type 2 (SWIZZLE_128B). The tile base is 1024-byte aligned (base offset 0);
// the K = 16 slices inside a 64-wide tile start 32 B apart.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// GELU (erf form) and its derivative.
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * __expf(-0.5f * z * z);
}

// 32 bytes of one row: one store of a whole sector where the row is 32-byte aligned (the same for
// all lanes of a warp: strides and bases decide it), else two of 16 bytes, which send every sector
// to L2 twice. The rows of a warp lie in 32 different lines, so sectors are what the stores cost:
// four members, 20,000 x 128 -> 1024 130 -> 120 us, 1024 -> 1024 204 -> 191, 1024 -> 2000 in
// float32 414 -> 352 us (the products alone 22, 115 and 213 us; the GELU and the clock, which falls
// to 1.6 GHz while tensor cores and epilogue both work, are the rest).
__device__ __forceinline__ void store32(void* dst, const uint32_t* p) {
  if (((uintptr_t)dst & 31) == 0) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(p[0]), "r"(p[1]),
                 "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7])
                 : "memory");
  } else {
    uint4* d = reinterpret_cast<uint4*>(dst);
    d[0] = make_uint4(p[0], p[1], p[2], p[3]);
    d[1] = make_uint4(p[4], p[5], p[6], p[7]);
  }
}

// 16 consecutive bf16 of one row.
__device__ __forceinline__ void store_row16(__nv_bfloat16* dst, const float* v) {
  uint32_t p[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    p[i] = *reinterpret_cast<uint32_t*>(&h);
  }
  store32(dst, p);
}

// 16 consecutive floats of one row.
__device__ __forceinline__ void store_row16(float* dst, const float* v) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t p[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = __float_as_uint(v[8 * h + i]);
    store32(dst + 8 * h, p);
  }
}

// 16 bf16 of one row from memory (z_in of the GELU' epilogue).
__device__ __forceinline__ void load_row16(const __nv_bfloat16* src, float* v) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  const uint4 a = s[0], b = s[1];
  const uint32_t p[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&p[i]);
    float2 f = __bfloat1622float2(h);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

// Epilogue of one 16-column slice of one accumulator row (row, col = first column).
__device__ __forceinline__ void epilogue16(const LblGemmEpilogue& ep, int split, int row, int col, float* v,
                                           float& loss) {
  if (ep.mode == LBL_GEMM_F32) {
    store_row16(ep.out_f32 + (long long)split * ep.split_stride + (long long)row * ep.ld_f32 + col, v);
    return;
  }
  float bias[16];
  if (ep.mode == LBL_GEMM_BIAS_GELU || ep.mode == LBL_GEMM_BIAS_SIGMOID) {   // four 16-byte loads (broadcast)
    const float4* b4 = reinterpret_cast<const float4*>(ep.bias + col);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 t = __ldg(b4 + i);
      bias[4 * i] = t.x;
      bias[4 * i + 1] = t.y;
      bias[4 * i + 2] = t.z;
      bias[4 * i + 3] = t.w;
    }
  }
  if (ep.mode == LBL_GEMM_BIAS_GELU) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += bias[i];
    if (ep.z_out) store_row16((__nv_bfloat16*)ep.z_out + (long long)row * ep.ld_z + col, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = gelu(v[i]);
  } else if (ep.mode == LBL_GEMM_BIAS_SIGMOID) {
    float p[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) p[i] = __fdividef(1.0f, 1.0f + __expf(-(v[i] + bias[i])));
    if (ep.out_f32) store_row16(ep.out_f32 + (long long)row * ep.ld_f32 + col, p);
    if (!ep.target) return;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (col + i < ep.n_valid) {
        const float d = p[i] - ep.target[(long long)row * ep.ld_target + col + i];
        loss += d * d;
        v[i] = ep.grad_scale * 2.0f * d * p[i] * (1.0f - p[i]);
      } else {
        v[i] = 0.0f;                               // padded outputs carry no gradient
      }
    }
  } else {                                         // LBL_GEMM_DGELU
    float z[16];
    load_row16((const __nv_bfloat16*)ep.z_in + (long long)row * ep.ld_zin + col, z);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] *= gelu_grad(z[i]);
  }
  if (ep.y) store_row16((__nv_bfloat16*)ep.y + (long long)row * ep.ld_y + col, v);
  if (ep.y_t) {
    __nv_bfloat16* yt = (__nv_bfloat16*)ep.y_t;
#pragma unroll
    for (int i = 0; i < 16; ++i) yt[(long long)(col + i) * ep.ld_yt + row] = __float2bfloat16(v[i]);
  }
}

// Work units of a launch: unit -> (product, split, m tile, n tile); n varies fastest so
// concurrent CTAs share A. One shape for all NB products, or two products (NB = 2) of their own
// shapes, product i's units from first[i] on (a search over the products by every role cost an
// ensemble of eight-product launches 2 to 8 %).
template <int NB>
struct GemmGrid {
  static constexpr int NS = NB == 2 ? 2 : 1;         // shapes
  int n_m[NS], n_n[NS], n_split[NS], kt_per[NS], first[NS];
  __device__ __forceinline__ int n_kt(int u) const { return kt_per[NS == 2 && u >= first[NS - 1]]; }
  __device__ __forceinline__ void unit(int u, int& op, int& split, int& m0, int& n0, int bn) const {
    const int z = NS == 2 && u >= first[NS - 1];
    if (z) u -= first[z];
    const int os = u / (n_m[z] * n_n[z]), r = u - os * n_m[z] * n_n[z];
    op = NS == 2 ? z : os / n_split[0];
    split = NS == 2 ? os : os - op * n_split[0];
    m0 = (r / n_n[z]) * GM;
    n0 = (r % n_n[z]) * bn;
  }
};

// Operands of the NB products of one launch.
template <int NB>
struct GemmOps {
  CUtensorMap a[NB], b[NB];
  LblGemmEpilogue ep[NB];
};

template <int BN, int NB>
__global__ void __launch_bounds__(G_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ GemmOps<NB> ops, const __grid_constant__ GemmGrid<NB> gg, int units, int* err) {
  using Cfg = GemmCfg<BN>;
  extern __shared__ unsigned char g_smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)g_smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + GSTAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;                       // [GSTAGES], one producer arrival + TMA bytes
  uint64_t* empty = bars + GSTAGES;            // [GSTAGES], one tcgen05.commit
  uint64_t* tfull = bars + 2 * GSTAGES;        // [2], one tcgen05.commit
  uint64_t* tempty = bars + 2 * GSTAGES + 2;   // [2], one arrival per epilogue warp
  uint64_t* drain = bars + 2 * GSTAGES + 4;    // MMA warp's final commit
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * GSTAGES + 5);
  volatile int* fail = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *fail = 0;
    for (int i = 0; i < GSTAGES; ++i) {
      mbar_init(smem_u32(&full[i]), 1);
      mbar_init(smem_u32(&empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&tfull[i]), 1);
      mbar_init(smem_u32(&tempty[i]), G_EPI_WARPS);
    }
    mbar_init(smem_u32(drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(Cfg::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  dependency_trigger();
  dependency_wait();                           // operands of the kernels before
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  float loss = 0.0f;

  if (warp == 0) {
    if (lane == 0) {                           // TMA producer
      int g = 0;
      for (int u = blockIdx.x; u < units && !*fail; u += gridDim.x) {
        int op, split, m0, n0;
        gg.unit(u, op, split, m0, n0, BN);
        const int n_kt = gg.n_kt(u), k0 = split * n_kt;
        const CUtensorMap* map_a = &ops.a[NB == 1 ? 0 : op];
        const CUtensorMap* map_b = &ops.b[NB == 1 ? 0 : op];
        for (int kt = 0; kt < n_kt; ++kt, ++g) {
          const int s = g % GSTAGES;
          if (g >= GSTAGES && !mbar_wait(smem_u32(&empty[s]), ((g / GSTAGES) - 1) & 1)) {
            *fail = 1;
            break;
          }
          if (*fail) break;
          unsigned char* st = smem + s * Cfg::STAGE_BYTES;
          const uint32_t fb = smem_u32(&full[s]);
          mbar_expect_tx(fb, Cfg::STAGE_BYTES);
          tma_load_2d(smem_u32(st), map_a, fb, (k0 + kt) * GK, m0);
#pragma unroll
          for (int h = 0; h < BN / 128; ++h)
            tma_load_2d(smem_u32(st + G_A_BYTES + h * 128 * GK * 2), map_b, fb, (k0 + kt) * GK, n0 + 128 * h);
        }
      }
      // no copy may still be writing shared memory when the CTA ends (bounded wait)
      for (int j = g > GSTAGES ? g - GSTAGES : 0; j < g; ++j)
        if (!mbar_wait(smem_u32(&full[j % GSTAGES]), (j / GSTAGES) & 1)) *fail = 1;
    }
  } else if (warp == 1) {
    if (lane == 0) {                           // MMA issuer
      // one descriptor, advanced by adds: the lane shares its scheduler with four epilogue warps
      // (1024 -> 1024 as above, built anew for each product: 191 against 188 us)
      const uint64_t desc0 = sw128_desc(smem_u32(smem));
      int g = 0, i = 0;
      for (int u = blockIdx.x; u < units && !*fail; u += gridDim.x, ++i) {
        const int b = i & 1;
        if (i >= 2 && !mbar_wait(smem_u32(&tempty[b]), ((i >> 1) - 1) & 1)) {
          *fail = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + (uint32_t)(b * BN);
        bool ok = true;
        const int n_kt = gg.n_kt(u);
        for (int kt = 0; kt < n_kt; ++kt, ++g) {
          const int s = g % GSTAGES;
          if (!mbar_wait(smem_u32(&full[s]), (g / GSTAGES) & 1)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = desc0 + (uint64_t)(s * (Cfg::STAGE_BYTES >> 4)), db = da + (G_A_BYTES >> 4);
#pragma unroll
          for (int kk = 0; kk < GK / 16; ++kk)
            umma_bf16(acc, da + 2 * kk, db + 2 * kk, Cfg::IDESC,
                      (kt > 0 || kk > 0) ? 1u : 0u);
          umma_commit(smem_u32(&empty[s]));
        }
        if (!ok) {
          *fail = 1;
          break;
        }
        umma_commit(smem_u32(&tfull[b]));
      }
      umma_commit(smem_u32(drain));            // arrives once every MMA issued above has finished
      if (!mbar_wait(smem_u32(drain), 0)) *fail = 1;
    }
  } else {  // epilogue warps: tensor-memory lanes 32 * (warp % 4), column group (warp - 2) / 4
    const int q = warp & 3;
    const int cg = (warp - 2) >> 2;
    constexpr int CW = BN / G_EPI_GROUPS;      // columns per group
    int i = 0;
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++i) {
      const int b = i & 1;
      bool ok = !*fail && mbar_wait(smem_u32(&tfull[b]), (i >> 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) *fail = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      int op, split, m0, n0;
      gg.unit(u, op, split, m0, n0, BN);
      const LblGemmEpilogue& ep = ops.ep[NB == 1 ? 0 : op];
      const int row = m0 + q * 32 + lane;
      const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN);
#pragma unroll 1
      for (int c0 = cg * CW; c0 < (cg + 1) * CW; c0 += 16) {
        uint32_t r[16];
        float v[16];
        tmem_ld16_issue(base + (uint32_t)c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
        epilogue16(ep, split, row, n0 + c0, v, loss);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty[b]));
    }
    // (several products in one launch take no loss: the host refuses it)
    const LblGemmEpilogue& ep = ops.ep[0];
    if (NB == 1 && ep.loss && ep.mode == LBL_GEMM_BIAS_SIGMOID && ep.target) {
      double l = loss;
      for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
      if (lane == 0 && l != 0.0) atomicAdd(ep.loss, l);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (threadIdx.x == 0 && *fail && err) atomicMax(err, 1);
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TMEM_COLS));
}

// ---------------------------------------------------------------------------
// Small kernels of the training step and of the gate.

// One Adam update (bias corrections c1, c2); returns the new weight.
__device__ __forceinline__ float adam_one(float w, float& m, float& v, float g, float lr, float b1, float b2, float eps,
                                          float c1, float c2) {
  m = b1 * m + (1.0f - b1) * g;
  v = b2 * v + (1.0f - b2) * g * g;
  return w - lr * (m * c1) / (sqrtf(v * c2) + eps);
}

// Adam on float32 master weights [rows, cols] (row stride ld) with the gradient summed
// over n_split partials (stride split_stride, added in order); refreshes the bf16 copy
// [rows, ld] and its transpose [cols, ld_t] when given.
__global__ void adam_kernel(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                            const float* __restrict__ g, int n_split, long long split_stride, int rows, int cols,
                            int ld, float lr, float b1, float b2, float eps, float c1, float c2,
                            __nv_bfloat16* __restrict__ w_bf, __nv_bfloat16* __restrict__ wt_bf, int ld_t) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)rows * cols) return;
  const int r = (int)(i / cols), c = (int)(i % cols);
  const long long o = (long long)r * ld + c;
  float gi = g[o];
  for (int s = 1; s < n_split; ++s) gi += g[s * split_stride + o];
  float mi = m[o], vi = v[o];
  const float wi = adam_one(w[o], mi, vi, gi, lr, b1, b2, eps, c1, c2);
  m[o] = mi;
  v[o] = vi;
  w[o] = wi;
  if (w_bf) w_bf[o] = __float2bfloat16(wi);
  if (wt_bf) wt_bf[(long long)c * ld_t + r] = __float2bfloat16(wi);
}

// The same update for up to ADAM_ITEMS tensors in one launch, a 64 x 64 tile per CTA: 16-byte
// loads and stores, and the transposed bf16 copy goes through shared memory, so it is
// written in 128-byte runs (a thread per element writes 2 bytes to a row of its own:
// 24 us for a 1024 x 1024 layer at 31 MB, and ten launches a step). Rows and columns that
// are multiples of 4 (rows = 1 for a vector), contiguous rows.
constexpr int ADAM_ITEMS = 16;
constexpr int ADAM_T = 64;
struct AdamGroup {
  LblAdamItem it[ADAM_ITEMS];
  int first[ADAM_ITEMS + 1];   // first tile of each item
};

__global__ void __launch_bounds__(256)
adam_group_kernel(const __grid_constant__ AdamGroup grp, int n, float lr, float b1, float b2, float eps, float c1,
                  float c2) {
  __shared__ __nv_bfloat16 s_t[ADAM_T][ADAM_T + 2];            // [column][row] of the tile
  dependency_trigger();
  dependency_wait();
  int k = 0;
  while (k + 1 < n && (int)blockIdx.x >= grp.first[k + 1]) ++k;
  const LblAdamItem& I = grp.it[k];
  const int tiles_c = (I.cols + ADAM_T - 1) / ADAM_T, t = blockIdx.x - grp.first[k];
  const int r0 = (t / tiles_c) * ADAM_T, c0 = (t % tiles_c) * ADAM_T;
  __nv_bfloat16* const w_bf = (__nv_bfloat16*)I.w_bf16;
  __nv_bfloat16* const wt_bf = (__nv_bfloat16*)I.wt_bf16;
  const int cl = 4 * (threadIdx.x & 15);
  for (int rl = threadIdx.x >> 4; rl < ADAM_T; rl += 16) {
    const int r = r0 + rl, c = c0 + cl;
    if (r >= I.rows || c >= I.cols) continue;
    const long long o = (long long)r * I.cols + c;
    float4 g = *(const float4*)(I.g + o);
    for (int s = 1; s < I.n_split; ++s) {
      const float4 p = *(const float4*)(I.g + s * I.split_stride + o);
      g.x += p.x; g.y += p.y; g.z += p.z; g.w += p.w;
    }
    float4 m = *(float4*)(I.m + o), v = *(float4*)(I.v + o), w = *(float4*)(I.w + o);
    w.x = adam_one(w.x, m.x, v.x, g.x, lr, b1, b2, eps, c1, c2);
    w.y = adam_one(w.y, m.y, v.y, g.y, lr, b1, b2, eps, c1, c2);
    w.z = adam_one(w.z, m.z, v.z, g.z, lr, b1, b2, eps, c1, c2);
    w.w = adam_one(w.w, m.w, v.w, g.w, lr, b1, b2, eps, c1, c2);
    *(float4*)(I.m + o) = m;
    *(float4*)(I.v + o) = v;
    *(float4*)(I.w + o) = w;
    __align__(8) const __nv_bfloat16 h[4] = {__float2bfloat16(w.x), __float2bfloat16(w.y), __float2bfloat16(w.z), __float2bfloat16(w.w)};
    if (w_bf) *(uint2*)(w_bf + o) = *(const uint2*)h;
    if (wt_bf)
#pragma unroll
      for (int i = 0; i < 4; ++i) s_t[cl + i][rl] = h[i];
  }
  if (!wt_bf) return;                                            // uniform over the CTA
  __syncthreads();
  const int rows = min(ADAM_T, I.rows - r0), cols = min(ADAM_T, I.cols - c0);
  for (int i = threadIdx.x; i < cols * (ADAM_T / 4); i += 256) {
    const int c = i / (ADAM_T / 4), r = 4 * (i % (ADAM_T / 4));
    if (r >= rows) continue;
    __align__(8) const __nv_bfloat16 h[4] = {s_t[c][r], s_t[c][r + 1], s_t[c][r + 2], s_t[c][r + 3]};
    *(uint2*)(wt_bf + (long long)(c0 + c) * I.rows + r0 + r) = *(const uint2*)h;
  }
}

// out[r] = sum_c x[r, c] over a bf16 matrix (bias gradients from dZ^T).
__global__ void rowsum_bf16_kernel(const __nv_bfloat16* __restrict__ x, int rows, int cols, int ld,
                                   float* __restrict__ out) {
  const int r = blockIdx.x;
  float s = 0.f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) s += __bfloat162float(x[(long long)r * ld + c]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ float part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    out[r] = t;
  }
}

// The same sums, bit for bit, for up to 16 matrices in one launch: a warp per row with 16-byte
// loads, lane l standing for the eight threads 8l .. 8l + 7 of the kernel above (columns
// and strides multiples of 8). HBM-bound; the five layers of a 4 x 1024 network at batch
// 4096: 9.5 us in one launch against 34 us in five.
constexpr int ROWSUM_ITEMS = 16;
struct RowsumGroup {
  LblRowsumItem it[ROWSUM_ITEMS];
  int first[ROWSUM_ITEMS + 1];   // first row of each item
};

__global__ void __launch_bounds__(256)
rowsum_group_kernel(const __grid_constant__ RowsumGroup grp, int n) {
  dependency_trigger();
  dependency_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= grp.first[n]) return;
  int k = 0;
  while (k + 1 < n && row >= grp.first[k + 1]) ++k;
  const LblRowsumItem& I = grp.it[k];
  const int r = row - grp.first[k];
  const uint4* x = (const uint4*)((const __nv_bfloat16*)I.x + (long long)r * I.ld);
  float a[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) a[e] = 0.f;
#pragma unroll 4
  for (int c = lane; c < I.cols / 8; c += 32) {
    const uint4 q = x[c];
    const uint32_t p[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&p[i]));
      a[2 * i] += f.x;
      a[2 * i + 1] += f.y;
    }
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1)                    // threads 16 and 8 apart
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] += __shfl_xor_sync(0xffffffffu, a[e], o);
  // 4, 2 and 1 apart, then the eight warps of the kernel above in order
  const float w = ((a[0] + a[4]) + (a[2] + a[6])) + ((a[1] + a[5]) + (a[3] + a[7]));
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) s += __shfl_sync(0xffffffffu, w, 4 * i);
  if (lane == 0) I.out[r] = s;
}

// x[b, c] = (raw[b, c] - mean[c]) * inv_std[c] as bf16, zero beyond cols up to ld; the
// transposed copy x_t[c, b] (row stride ld_t) when given.
__global__ void pack_inputs_kernel(const float* __restrict__ raw, int rows, int cols, const float* __restrict__ mean,
                                   const float* __restrict__ inv_std, __nv_bfloat16* __restrict__ x, int ld,
                                   __nv_bfloat16* __restrict__ x_t, int ld_t) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)rows * ld) return;
  const int r = (int)(i / ld), c = (int)(i % ld);
  const float v = c < cols ? (raw[(long long)r * cols + c] - mean[c]) * inv_std[c] : 0.0f;
  const __nv_bfloat16 b = __float2bfloat16(v);
  x[(long long)r * ld + c] = b;
  if (x_t) x_t[(long long)c * ld_t + r] = b;
}

// A training batch from the samples idx[0 .. rows): the standardised inputs x and their transpose as
// pack_inputs_kernel writes them, the targets copied row by row, the loss cleared. The first n_pack
// CTAs take 32 rows of inputs each (the transpose goes through shared memory: 64-byte runs instead
// of single values), the others a row of targets per warp. HBM- and launch-bound: at batch 4,096
// two index selections, a fill and the pack take 32 us of device time and the gaps between them, this
// 19 (four steps 1,655 -> 1,575 us). A sample outside [0, n_samples) becomes NaN.
constexpr int SB_ROWS = 32, SB_COLS = 128;
__global__ void __launch_bounds__(256)
stage_batch_kernel(const float* __restrict__ features, const float* __restrict__ targets,
                   const long long* __restrict__ idx, long long n_samples, int rows, int n_in, int n_out, int n_pack,
                   const float* __restrict__ mean, const float* __restrict__ inv_std, __nv_bfloat16* __restrict__ x,
                   int ld, __nv_bfloat16* __restrict__ x_t, int ld_t, float* __restrict__ target, double* loss,
                   int vec) {
  dependency_trigger();
  dependency_wait();                             // the step before reads what this one writes
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float nan = __int_as_float(0x7fffffff);
  if ((int)blockIdx.x < n_pack) {
    __shared__ __nv_bfloat16 tile[SB_ROWS][SB_COLS + 2];
    __shared__ long long src[SB_ROWS];
    if (blockIdx.x == 0 && tid == 0) *loss = 0.0;
    const int r0 = blockIdx.x * SB_ROWS;
    if (tid < SB_ROWS) src[tid] = r0 + tid < rows ? idx[r0 + tid] : -1;
    __syncthreads();
    for (int c0 = 0; c0 < ld; c0 += SB_COLS) {
      for (int e = tid; e < SB_ROWS * SB_COLS; e += 256) {
        const int r = e / SB_COLS, k = e % SB_COLS, c = c0 + k;
        const long long i = src[r];
        const bool in = i >= 0 && i < n_samples;
        const float v = c < n_in ? ((in ? features[i * n_in + c] : nan) - mean[c]) * inv_std[c] : 0.0f;
        const __nv_bfloat16 b = __float2bfloat16(v);
        tile[r][k] = b;
        if (r0 + r < rows && c < ld) x[(long long)(r0 + r) * ld + c] = b;
      }
      __syncthreads();
      for (int e = tid; e < SB_ROWS * SB_COLS; e += 256) {
        const int k = e / SB_ROWS, r = e % SB_ROWS;
        if (r0 + r < rows && c0 + k < ld) x_t[(long long)(c0 + k) * ld_t + r0 + r] = tile[r][k];
      }
      __syncthreads();
    }
    return;
  }
  const int r = (blockIdx.x - n_pack) * 8 + warp;
  if (r >= rows) return;
  const long long i = idx[r];
  const bool in = i >= 0 && i < n_samples;
  const float* from = targets + (in ? i : 0) * n_out;
  float* to = target + (long long)r * n_out;
  if (vec && in) {
    const float4* f4 = reinterpret_cast<const float4*>(from);
    float4* t4 = reinterpret_cast<float4*>(to);
#pragma unroll 4
    for (int c = lane; c < n_out / 4; c += 32) t4[c] = f4[c];
  } else {
    for (int c = lane; c < n_out; c += 32) to[c] = in ? from[c] : nan;
  }
}

// Standardised inputs of up to 16 networks from the same raw [rows, cols], one launch, eight
// columns per thread (ld a multiple of 8).
constexpr int PACK_ITEMS = 16;
struct PackGroup {
  LblPackItem it[PACK_ITEMS];
};

__global__ void __launch_bounds__(256)
pack_group_kernel(const __grid_constant__ PackGroup grp, const float* __restrict__ raw, int rows, int cols, int ld) {
  dependency_trigger();
  dependency_wait();
  const LblPackItem& I = grp.it[blockIdx.y];
  const int per = ld / 8;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)rows * per) return;
  const int r = (int)(i / per), c0 = 8 * (int)(i % per);
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = c0 + k;
    v[k] = c < cols ? (raw[(long long)r * cols + c] - I.mean[c]) * I.inv_std[c] : 0.0f;
  }
  uint32_t p[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    p[k] = *reinterpret_cast<const uint32_t*>(&h);
  }
  *(uint4*)((__nv_bfloat16*)I.x + (long long)r * ld + c0) = make_uint4(p[0], p[1], p[2], p[3]);
}

// Ensemble statistics of one sample per CTA: mean over the members of pred[m, b, c]
// and the error estimate est[b] = max over channels of the members' standard deviation
// (population form); flag[b] = (scale * est[b] > gate).
template <typename Load>
__device__ __forceinline__ void gate_channel(int n_mem, Load load, float& mu, float& sd) {
  float s = 0.f;
  for (int m = 0; m < n_mem; ++m) s += load(m);
  mu = s / n_mem;
  float s2 = 0.f;                                    // second pass: deviations (no cancellation)
  for (int m = 0; m < n_mem; ++m) {
    const float d = load(m) - mu;
    s2 += d * d;
  }
  sd = sqrtf(s2 / n_mem);
}

__device__ __forceinline__ void gate_finish(float worst, float scale, float gate, bool bad, float* est, int* flag) {
  for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
  __shared__ float part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = worst;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = fmaxf(t, part[w]);
    *est = bad ? __int_as_float(0x7fffffff) : t;
    *flag = (bad || scale * t > gate) ? 1 : 0;
  }
}

__global__ void ensemble_gate_kernel(const float* __restrict__ pred, int n_mem, long long member_stride, int ld,
                                     int n_ch, const float* __restrict__ ch_scale, float scale, float gate,
                                     const int* err, float* __restrict__ mean, float* __restrict__ est,
                                     int* __restrict__ flag) {
  const bool bad = err && *err != 0;
  const int b = blockIdx.x;
  float worst = 0.0f;
  for (int c = threadIdx.x; c < n_ch; c += blockDim.x) {
    const float* col = pred + (long long)b * ld + c;
    float mu, sd;
    gate_channel(n_mem, [&](int m) { return col[m * member_stride]; }, mu, sd);
    mean[(long long)b * n_ch + c] = bad ? __int_as_float(0x7fffffff) : mu;
    worst = fmaxf(worst, ch_scale ? ch_scale[c] * sd : sd);
  }
  gate_finish(worst, scale, gate, bad, est + b, flag + b);
}

// The same for NM members held in registers, four channels per thread and load (n_ch, ld and
// member_stride multiples of 4, 16-byte aligned rows): each prediction is read once, with
// NM 16-byte loads in flight per thread. HBM-bound; 20,000 samples x 2,000 channels, this and the
// scalar kernel above: 76 and 224 us for 2 members, 104 and 236 for 3, 122 and 199 for 4, 147 and
// 269 for 5, 172 and 333 for 6, 217 and 300 for 8. Seven members and more than eight are not
// compiled here (no configuration has them) and take the scalar kernel: 349 us for 7, 375 for 9.
template <int NM>
__global__ void __launch_bounds__(256)
ensemble_gate4_kernel(const float4* __restrict__ pred, long long member_stride4, int ld4, int n_ch4,
                      const float* __restrict__ ch_scale, float scale, float gate, const int* err,
                      float4* __restrict__ mean, float* __restrict__ est, int* __restrict__ flag) {
  dependency_trigger();
  dependency_wait();
  const int b = blockIdx.x;
  const bool bad = err && *err != 0;
  const float nan = __int_as_float(0x7fffffff);
  float worst = 0.0f;
  for (int c = threadIdx.x; c < n_ch4; c += blockDim.x) {
    const float4* col = pred + (long long)b * ld4 + c;
    float v[NM][4];
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      const float4 t = __ldcs(col + m * member_stride4);
      v[m][0] = t.x; v[m][1] = t.y; v[m][2] = t.z; v[m][3] = t.w;
    }
    float mu[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float sd;
      gate_channel(NM, [&](int m) { return v[m][i]; }, mu[i], sd);
      worst = fmaxf(worst, ch_scale ? ch_scale[4 * c + i] * sd : sd);
    }
    mean[(long long)b * n_ch4 + c] = bad ? make_float4(nan, nan, nan, nan) : make_float4(mu[0], mu[1], mu[2], mu[3]);
  }
  gate_finish(worst, scale, gate, bad, est + b, flag + b);
}

}  // namespace lbl

using namespace lbl;

// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

extern "C" size_t lbl_tensor_map_bytes(void) { return sizeof(CUtensorMap); }

extern "C" int lbl_tensor_map_bf16(void* map_out, const void* base, long long rows, long long cols, long long ld) {
  if (!map_out || !base || rows < GM || rows % GM || cols < GK || cols % GK || ld < cols || ld % 8 ||
      ((uintptr_t)base) % 16)
    return lbl_set_error(LBL_EINVAL,
                         "lbl_tensor_map_bf16: rows must be a multiple of 128, cols of 64, ld a multiple of 8 "
                         ">= cols and the base 16-byte aligned");
  EncodeTiledFn fn = encode_fn();
  if (!fn) return lbl_set_error(LBL_ECUDA, "lbl_tensor_map_bf16: cuTensorMapEncodeTiled unavailable");
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {GK, GM};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn((CUtensorMap*)map_out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return lbl_set_error(LBL_ECUDA, "lbl_tensor_map_bf16: encode failed (%d)", (int)r);
  return LBL_OK;
}

struct GemmSize { int M, N, K, n_split; };

template <int BN, int NB>
static int launch_gemm(const GemmOps<NB>& ops, const GemmSize* size, int count, int n_sm, int dev, int* err,
                       cudaStream_t stream) {
  static int attr_set[64] = {0};
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(gemm_bf16_kernel<BN, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             GemmCfg<BN>::SMEM) != cudaSuccess)
      return lbl_check_launch("lbl_gemm_bf16 (shared memory attribute)");
    attr_set[dev] = 1;
  }
  GemmGrid<NB> gg;
  long long units = 0;
  for (int i = 0; i < GemmGrid<NB>::NS; ++i) {
    const GemmSize& z = size[i];
    gg.n_m[i] = z.M / GM;
    gg.n_n[i] = z.N / BN;
    gg.n_split[i] = z.n_split;
    gg.kt_per[i] = z.K / GK / z.n_split;
    gg.first[i] = (int)units;
    units += (long long)gg.n_m[i] * gg.n_n[i] * z.n_split * (GemmGrid<NB>::NS == 1 ? count : 1);
    if (units > 0x7fffffffLL) return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16: too many tiles");
  }
  const int grid = (int)(units < n_sm ? units : n_sm);
  // a layer's barriers, tensor memory and first instructions overlap the layer before
  launch_dependent(gemm_bf16_kernel<BN, NB>, dim3((unsigned)grid), G_THREADS, GemmCfg<BN>::SMEM, stream, ops, gg,
                   (int)units, err);
  return lbl_check_launch("lbl_gemm_bf16");
}

// size: the shapes (one for all count products, or NB = 2 products' own).
template <int NB>
static int launch_group(const GemmOps<NB>& ops, const GemmSize* size, int count, int* err, cudaStream_t stream) {
  int dev = 0;
  cudaGetDevice(&dev);
  static int n_sm[64] = {0};
  if (dev < 0 || dev >= 64) return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16: device index out of range");
  if (!n_sm[dev]) cudaDeviceGetAttribute(&n_sm[dev], cudaDevAttrMultiProcessorCount, dev);
  // 256-wide tiles read a third less per product; 128-wide ones where 256-wide tiles would
  // leave more than a quarter of the SMs idle (4096 x 1024 x 1024, 128 wide tiles: 22.5 against
  // 24 us; four members of 256 x 2048 x 1024, 64 wide tiles: 17.2 against 12.5 us)
  long long wide = 0;
  bool fits = true;
  constexpr int NS = GemmGrid<NB>::NS;
  for (int i = 0; i < NS; ++i) {
    wide += (long long)(size[i].M / GM) * (size[i].N / 256) * size[i].n_split * (NS == 1 ? count : 1);
    fits = fits && size[i].N % 256 == 0;
  }
  if (fits && 4 * wide >= 3 * n_sm[dev]) return launch_gemm<256, NB>(ops, size, count, n_sm[dev], dev, err, stream);
  return launch_gemm<128, NB>(ops, size, count, n_sm[dev], dev, err, stream);
}

static int check_gemm(const void* map_a, const void* map_b, int M, int N, int K, int n_split,
                      const LblGemmEpilogue* ep) {
  if (!map_a || !map_b || !ep || M < GM || N < 128 || K < GK || M % GM || N % 128 || K % GK || n_split < 1 ||
      (K / GK) % n_split || ep->mode < LBL_GEMM_F32 || ep->mode > LBL_GEMM_DGELU)
    return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16: M, N must be multiples of 128, K of 64 * n_split");
  if (n_split > 1 && ep->mode != LBL_GEMM_F32)
    return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16: split-K needs the float32 epilogue");
  const bool needs_f32 = ep->mode == LBL_GEMM_F32;
  if ((needs_f32 && (!ep->out_f32 || ep->ld_f32 < N || ep->ld_f32 % 4 ||
                     (n_split > 1 && ep->split_stride < (long long)M * ep->ld_f32))) ||
      (ep->mode != LBL_GEMM_F32 && ep->mode != LBL_GEMM_DGELU && (!ep->bias || ((uintptr_t)ep->bias) % 16)) ||
      (ep->mode == LBL_GEMM_DGELU && (!ep->z_in || ep->ld_zin < N || ep->ld_zin % 8)) ||
      (ep->z_out && (ep->ld_z < N || ep->ld_z % 8)) || (ep->y && (ep->ld_y < N || ep->ld_y % 8)) ||
      (ep->y_t && ep->ld_yt < M) || (ep->mode == LBL_GEMM_BIAS_SIGMOID && ep->out_f32 && ep->ld_f32 % 4) ||
      (ep->mode == LBL_GEMM_BIAS_SIGMOID && ep->target && ep->ld_target < ep->n_valid))
    return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16: epilogue buffers missing or strides too small/unaligned");
  return LBL_OK;
}

extern "C" int lbl_gemm_bf16(const void* map_a, const void* map_b, int M, int N, int K, int n_split,
                             const LblGemmEpilogue* ep, int* err, void* stream) {
  const int st = check_gemm(map_a, map_b, M, N, K, n_split, ep);
  if (st != LBL_OK) return st;
  GemmOps<1> ops;
  memcpy(&ops.a[0], map_a, sizeof(CUtensorMap));
  memcpy(&ops.b[0], map_b, sizeof(CUtensorMap));
  ops.ep[0] = *ep;
  const GemmSize size = {M, N, K, n_split};
  return launch_group<1>(ops, &size, 1, err, (cudaStream_t)stream);
}

// Two products of their own shapes in one launch. A training step's layers are one wave of tiles
// each, so a launch of one product ends with an epilogue that nothing overlaps; a layer's weight
// gradient (split over the batch) and its input gradient need the same operand and not each other
// (four steps of a 61-1024x4-2000 network at batch 4,096: 1,740 us as two launches, 1,660 together).
extern "C" int lbl_gemm_bf16_pair(const void* const* map_a, const void* const* map_b, const int* m, const int* n,
                                  const int* k, const int* n_split, const LblGemmEpilogue* ep, int* err,
                                  void* stream) {
  if (!map_a || !map_b || !m || !n || !k || !n_split || !ep)
    return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16_pair: bad arguments");
  GemmOps<2> ops;
  GemmSize size[2];
  for (int i = 0; i < 2; ++i) {
    const int st = check_gemm(map_a[i], map_b[i], m[i], n[i], k[i], n_split[i], ep + i);
    if (st != LBL_OK) return st;
    if (ep[i].loss) return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16_pair: no loss in a pair");
    memcpy(&ops.a[i], map_a[i], sizeof(CUtensorMap));
    memcpy(&ops.b[i], map_b[i], sizeof(CUtensorMap));
    ops.ep[i] = ep[i];
    size[i] = {m[i], n[i], k[i], n_split[i]};
  }
  return launch_group<2>(ops, size, 2, err, (cudaStream_t)stream);
}

constexpr int G_GROUP = 8;   // products per launch (3.1 KB of kernel parameters)

extern "C" int lbl_gemm_bf16_group(int count, const void* const* map_a, const void* const* map_b, int M, int N, int K,
                                   const LblGemmEpilogue* ep, int* err, void* stream) {
  if (count < 1 || !map_a || !map_b || !ep) return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16_group: bad arguments");
  for (int i = 0; i < count; ++i) {
    const int st = check_gemm(map_a[i], map_b[i], M, N, K, 1, ep + i);
    if (st != LBL_OK) return st;
    if (ep[i].loss) return lbl_set_error(LBL_EINVAL, "lbl_gemm_bf16_group: no loss in a group");
  }
  for (int i0 = 0; i0 < count; i0 += G_GROUP) {
    const int n = count - i0 < G_GROUP ? count - i0 : G_GROUP;
    GemmOps<G_GROUP> ops;
    const GemmSize size = {M, N, K, 1};
    for (int i = 0; i < G_GROUP; ++i) {               // unused entries repeat the first
      const int j = i0 + (i < n ? i : 0);
      memcpy(&ops.a[i], map_a[j], sizeof(CUtensorMap));
      memcpy(&ops.b[i], map_b[j], sizeof(CUtensorMap));
      ops.ep[i] = ep[j];
    }
    const int st = launch_group<G_GROUP>(ops, &size, n, err, (cudaStream_t)stream);
    if (st != LBL_OK) return st;
  }
  return LBL_OK;
}

extern "C" int lbl_adam_step(float* w, float* m, float* v, const float* g, int n_split, long long split_stride,
                             int rows, int cols, int ld, float lr, float b1, float b2, float eps, int step,
                             void* w_bf16, void* wt_bf16, int ld_t, void* stream) {
  if (!w || !m || !v || !g || rows < 1 || cols < 1 || ld < cols || step < 1 || n_split < 1 ||
      (n_split > 1 && split_stride < (long long)rows * ld) || (wt_bf16 && ld_t < rows))
    return lbl_set_error(LBL_EINVAL, "lbl_adam_step: bad arguments");
  const float c1 = (float)(1.0 / (1.0 - pow((double)b1, step))), c2 = (float)(1.0 / (1.0 - pow((double)b2, step)));
  const long long n = (long long)rows * cols;
  adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      w, m, v, g, n_split, split_stride, rows, cols, ld, lr, b1, b2, eps, c1, c2, (__nv_bfloat16*)w_bf16,
      (__nv_bfloat16*)wt_bf16, ld_t);
  return lbl_check_launch("lbl_adam_step");
}

static bool aligned16(const void* p) { return ((uintptr_t)p) % 16 == 0; }

extern "C" int lbl_adam_group(const LblAdamItem* items, int count, float lr, float b1, float b2, float eps, int step,
                              void* stream) {
  if (!items || count < 1 || step < 1) return lbl_set_error(LBL_EINVAL, "lbl_adam_group: bad arguments");
  for (int i = 0; i < count; ++i) {
    const LblAdamItem& I = items[i];
    if (!I.w || !I.m || !I.v || !I.g || I.rows < 1 || I.cols < 1 || I.cols % 4 || I.n_split < 1 ||
        (I.n_split > 1 && (I.split_stride < (long long)I.rows * I.cols || I.split_stride % 4)) ||
        (I.wt_bf16 && I.rows % 4) || !aligned16(I.w) || !aligned16(I.m) || !aligned16(I.v) || !aligned16(I.g) ||
        !aligned16(I.w_bf16) || !aligned16(I.wt_bf16))
      return lbl_set_error(LBL_EINVAL, "lbl_adam_group: item %d: columns (and rows with a transposed copy) must be "
                                       "multiples of 4, buffers contiguous and 16-byte aligned", i);
  }
  const float c1 = (float)(1.0 / (1.0 - pow((double)b1, step))), c2 = (float)(1.0 / (1.0 - pow((double)b2, step)));
  for (int i0 = 0; i0 < count; i0 += ADAM_ITEMS) {
    const int n = count - i0 < ADAM_ITEMS ? count - i0 : ADAM_ITEMS;
    AdamGroup g = {};
    long long tiles = 0;
    for (int i = 0; i < n; ++i) {
      g.it[i] = items[i0 + i];
      g.first[i] = (int)tiles;
      tiles += (long long)((g.it[i].rows + ADAM_T - 1) / ADAM_T) * ((g.it[i].cols + ADAM_T - 1) / ADAM_T);
      if (tiles > 0x7fffffffLL) return lbl_set_error(LBL_EINVAL, "lbl_adam_group: too many tiles");
    }
    launch_dependent(adam_group_kernel, dim3((unsigned)tiles), 256, 0, (cudaStream_t)stream, g, n, lr, b1, b2, eps, c1, c2);
    const int st = lbl_check_launch("lbl_adam_group");
    if (st != LBL_OK) return st;
  }
  return LBL_OK;
}

extern "C" int lbl_rowsum_group(const LblRowsumItem* items, int count, void* stream) {
  if (!items || count < 1) return lbl_set_error(LBL_EINVAL, "lbl_rowsum_group: bad arguments");
  for (int i0 = 0; i0 < count; i0 += ROWSUM_ITEMS) {
    const int n = count - i0 < ROWSUM_ITEMS ? count - i0 : ROWSUM_ITEMS;
    RowsumGroup g = {};
    long long rows = 0;
    for (int i = 0; i < n; ++i) {
      const LblRowsumItem& I = g.it[i] = items[i0 + i];
      if (!I.x || !I.out || I.rows < 1 || I.cols < 8 || I.cols % 8 || I.ld < I.cols || I.ld % 8 || !aligned16(I.x))
        return lbl_set_error(LBL_EINVAL, "lbl_rowsum_group: item %d: columns and stride must be multiples of 8", i0 + i);
      g.first[i] = (int)rows;
      rows += I.rows;
      if (rows > 0x7fffff00LL) return lbl_set_error(LBL_EINVAL, "lbl_rowsum_group: too many rows");
    }
    for (int i = n; i <= ROWSUM_ITEMS; ++i) g.first[i] = (int)rows;
    launch_dependent(rowsum_group_kernel, dim3((unsigned)((rows + 7) / 8)), 256, 0, (cudaStream_t)stream, g, n);
    const int st = lbl_check_launch("lbl_rowsum_group");
    if (st != LBL_OK) return st;
  }
  return LBL_OK;
}

extern "C" int lbl_pack_inputs_group(const float* raw, int rows, int cols, const LblPackItem* items, int count, int ld,
                                     void* stream) {
  if (!raw || !items || rows < 1 || cols < 1 || count < 1 || ld < cols || ld % 8)
    return lbl_set_error(LBL_EINVAL, "lbl_pack_inputs_group: bad arguments");
  for (int i0 = 0; i0 < count; i0 += PACK_ITEMS) {
    const int n = count - i0 < PACK_ITEMS ? count - i0 : PACK_ITEMS;
    PackGroup g = {};
    for (int i = 0; i < n; ++i) {
      g.it[i] = items[i0 + i];
      if (!g.it[i].mean || !g.it[i].inv_std || !g.it[i].x || !aligned16(g.it[i].x))
        return lbl_set_error(LBL_EINVAL, "lbl_pack_inputs_group: item %d: missing or unaligned buffer", i0 + i);
    }
    const long long t = (long long)rows * (ld / 8);
    dim3 grid((unsigned)((t + 255) / 256), (unsigned)n);
    launch_dependent(pack_group_kernel, grid, 256, 0, (cudaStream_t)stream, g, raw, rows, cols, ld);
    const int st = lbl_check_launch("lbl_pack_inputs_group");
    if (st != LBL_OK) return st;
  }
  return LBL_OK;
}

// One host call for all launches of an ensemble's prediction: a handful of profiles is over on the
// device before six calls with their argument blocks are made from outside (four members, 200
// profiles: 100 us a pass when the host makes a call per layer, 69 us this way).
extern "C" int lbl_ensemble_forward(const float* raw, int rows, int n_in, const LblPackItem* items,
                                    const LblNetLayer* layers, int members, int n_layers, const int* widths, int M,
                                    int n_valid, float* pred, long long member_stride, int* err, void* stream) {
  if (!raw || !items || !layers || !widths || !pred || members < 1 || n_layers < 1 || rows < 1 || rows > M ||
      member_stride < (long long)M * widths[n_layers])
    return lbl_set_error(LBL_EINVAL, "lbl_ensemble_forward: bad arguments");
  int st = lbl_pack_inputs_group(raw, rows, n_in, items, members, widths[0], stream);
  for (int l = 0; l < n_layers && st == LBL_OK; ++l) {
    const int k = widths[l], n = widths[l + 1];
    for (int i0 = 0; i0 < members && st == LBL_OK; i0 += G_GROUP) {
      const int count = members - i0 < G_GROUP ? members - i0 : G_GROUP;
      const void *map_x[G_GROUP], *map_w[G_GROUP];
      LblGemmEpilogue ep[G_GROUP] = {};
      for (int i = 0; i < count; ++i) {
        const LblNetLayer& L = layers[(long long)(i0 + i) * n_layers + l];
        map_x[i] = L.map_x;
        map_w[i] = L.map_w;
        ep[i].bias = L.bias;
        if (l < n_layers - 1) {
          if (!L.y) return lbl_set_error(LBL_EINVAL, "lbl_ensemble_forward: member %d, layer %d: no output", i0 + i, l);
          ep[i].mode = LBL_GEMM_BIAS_GELU;
          ep[i].y = L.y;
          ep[i].ld_y = n;
        } else {
          ep[i].mode = LBL_GEMM_BIAS_SIGMOID;
          ep[i].n_valid = n_valid;
          ep[i].out_f32 = pred + (i0 + i) * member_stride;
          ep[i].ld_f32 = n;
        }
      }
      st = lbl_gemm_bf16_group(count, map_x, map_w, M, n, k, ep, err, stream);
    }
  }
  return st;
}

extern "C" int lbl_rowsum_bf16(const void* x, int rows, int cols, int ld, float* out, void* stream) {
  if (!x || !out || rows < 1 || cols < 1 || ld < cols)
    return lbl_set_error(LBL_EINVAL, "lbl_rowsum_bf16: bad arguments");
  rowsum_bf16_kernel<<<rows, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, rows, cols, ld, out);
  return lbl_check_launch("lbl_rowsum_bf16");
}

extern "C" int lbl_pack_inputs_bf16(const float* raw, int rows, int cols, const float* mean, const float* inv_std,
                                    void* x, int ld, void* x_t, int ld_t, void* stream) {
  if (!raw || !mean || !inv_std || !x || rows < 1 || cols < 1 || ld < cols || (x_t && ld_t < rows))
    return lbl_set_error(LBL_EINVAL, "lbl_pack_inputs_bf16: bad arguments");
  const long long n = (long long)rows * ld;
  pack_inputs_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      raw, rows, cols, mean, inv_std, (__nv_bfloat16*)x, ld, (__nv_bfloat16*)x_t, ld_t);
  return lbl_check_launch("lbl_pack_inputs_bf16");
}

extern "C" int lbl_stage_batch(const float* features, const float* targets, const long long* idx, long long n_samples,
                               int rows, int n_in, int n_out, const float* mean, const float* inv_std, void* x, int ld,
                               void* x_t, int ld_t, float* target, double* loss, void* stream) {
  if (!features || !targets || !idx || !mean || !inv_std || !x || !x_t || !target || !loss || n_samples < 1 ||
      rows < 1 || n_in < 1 || n_out < 1 || ld < n_in || ld_t < rows)
    return lbl_set_error(LBL_EINVAL, "lbl_stage_batch: bad arguments");
  const int n_pack = (rows + SB_ROWS - 1) / SB_ROWS;
  launch_dependent(stage_batch_kernel, dim3((unsigned)(n_pack + (rows + 7) / 8)), 256, 0, (cudaStream_t)stream, features,
                   targets, idx, n_samples, rows, n_in, n_out, n_pack, mean, inv_std, (__nv_bfloat16*)x, ld,
                   (__nv_bfloat16*)x_t, ld_t, target, loss,
                   (int)(n_out % 4 == 0 && aligned16(targets) && aligned16(target)));
  return lbl_check_launch("lbl_stage_batch");
}

extern "C" int lbl_ensemble_gate_checked(const float* pred, int n_mem, long long member_stride, int n_samples, int ld,
                                         int n_ch, const float* ch_scale, float scale, float gate, const int* err,
                                         float* mean, float* est, int* flag, void* stream) {
  if (!pred || !mean || !est || !flag || n_mem < 1 || n_samples < 1 || n_ch < 1 || ld < n_ch ||
      (n_mem > 1 && member_stride < (long long)n_samples * ld))
    return lbl_set_error(LBL_EINVAL, "lbl_ensemble_gate: bad arguments");
  const cudaStream_t st = (cudaStream_t)stream;
  const bool vec = n_ch % 4 == 0 && ld % 4 == 0 && member_stride % 4 == 0 && ((uintptr_t)pred | (uintptr_t)mean) % 16 == 0;
  auto vec_launch = [&](auto nm) {
    launch_dependent(ensemble_gate4_kernel<decltype(nm)::value>, dim3((unsigned)n_samples), 256, 0, st, (const float4*)pred,
                     member_stride / 4, ld / 4, n_ch / 4, ch_scale, scale, gate, err, (float4*)mean, est, flag);
  };
  if (vec && n_mem == 2) vec_launch(std::integral_constant<int, 2>());
  else if (vec && n_mem == 3) vec_launch(std::integral_constant<int, 3>());
  else if (vec && n_mem == 4) vec_launch(std::integral_constant<int, 4>());
  else if (vec && n_mem == 5) vec_launch(std::integral_constant<int, 5>());
  else if (vec && n_mem == 6) vec_launch(std::integral_constant<int, 6>());
  else if (vec && n_mem == 8) vec_launch(std::integral_constant<int, 8>());
  else
    ensemble_gate_kernel<<<n_samples, 256, 0, st>>>(pred, n_mem, member_stride, ld, n_ch, ch_scale, scale, gate, err,
                                                    mean, est, flag);
  return lbl_check_launch("lbl_ensemble_gate");
}

extern "C" int lbl_ensemble_gate(const float* pred, int n_mem, long long member_stride, int n_samples, int ld,
                                 int n_ch, const float* ch_scale, float scale, float gate, float* mean, float* est,
                                 int* flag, void* stream) {
  return lbl_ensemble_gate_checked(pred, n_mem, member_stride, n_samples, ld, n_ch, ch_scale, scale, gate, nullptr, mean,
                                   est, flag, stream);
}
