// axj_mlp.cu -- learned artificial-diffusivity sensor.
//
// An MLP (100 -> 64 -> 64 -> 2, tanh-form GELU) stands in for the evaluation of
// betastar and kappastar (ModShockCapturing.f90:18-92) between plain-sensor judge
// steps. Its inputs are 5 x 5 (z, r) windows of four channels per point: the
// dilatation, |grad rho|, the vorticity magnitude and the local grid spacing
// sqrt(deltaz*deltar). Inference runs on the 5th-generation tensor cores: BF16
// operands staged in shared memory, FP32 accumulators in tensor memory (tcgen05.mma
// issued by one thread, tcgen05.ld for the epilogues). Training runs in FP32 on the
// CUDA cores: tiled GEMMs for the forward and backward passes and Adam.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "axj_mlp.cuh"

namespace axj {

namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier (one arrival: the tcgen05.commit of the MMA-issuing thread) ----
__device__ __forceinline__ void bar_init(uint64_t* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after about 1 << 20 polls (a fraction of a second).
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
  for (int it = 0; it < (1 << 20); ++it) {
    if (bar_try(b, parity)) return true;
    if (it > 64) __nanosleep(128);
  }
  return false;
}

// ---- tcgen05 ----
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Generic-proxy shared-memory writes become visible to the tensor core (async proxy).
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Shared-memory matrix descriptor, no swizzle, K-major canonical layout: 8-row x
// 16-byte core matrices; lbo = byte distance of the two K halves of one MMA step,
// sbo = byte distance of consecutive 8-row groups; version 1 (bit 46).
__device__ __forceinline__ uint64_t mdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         (1ull << 46);
}
// Instruction descriptor of kind::f16: BF16 A and B (K-major), FP32 accumulator,
// M = 128, N = 64.
constexpr uint32_t IDESC_BF16_M128_N64 =
    (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(b))
               : "memory");
}
// 16 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Two floats to a BF16 pair (a in the low half), one packed conversion.
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

}  // namespace

// GELU, tanh form: 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))), and its derivative.
// Inference uses the hardware tanh approximation (one MUFU operation, relative error
// about 2^-11, below the BF16 rounding of the activations it feeds); training uses tanhf.
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two FP32 values in one 64-bit register pair, for the packed FP32 instructions (each half
// rounded as the scalar instruction rounds it; one issue slot for two operations).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float x, float y) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
__device__ __forceinline__ void unpk2(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// The tanh-form GELU of two values: 0.5 x (1 + tanh(x (k + 0.044715 k x^2))), k = sqrt(2/pi).
__device__ __forceinline__ f32x2 gelu_fast2(f32x2 x) {
  constexpr float k = 0.7978845608028654f;
  const f32x2 u = mul2(x, fma2(mul2(x, x), pk2(0.044715f * k, 0.044715f * k), pk2(k, k)));
  const f32x2 hx = mul2(x, pk2(0.5f, 0.5f));
  float u0, u1;
  unpk2(u, u0, u1);
  return fma2(hx, pk2(tanh_fast(u0), tanh_fast(u1)), hx);
}
__device__ __forceinline__ float gelu_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.0f + tanhf(u));
}
__device__ __forceinline__ float gelu_grad_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  const float t = tanhf(u);
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x * x);
}

// ---------------------------------------------------------------------------
// Feature channels
// ---------------------------------------------------------------------------
// Tile of 32 (z) x 16 (r) points per CTA (256 threads, two points per thread: rows
// tr and tr + 8). rho, V_r, V_z of the tile and a halo of 5 (the widest SBP boundary row
// reaches 5 points) are staged in shared memory as FP32 (zero outside the grid, the
// never-written halo), one box row per warp and pass; each thread forms its six first
// derivatives in FP32 on differences from its own value: every SBP row sums to zero, so
// sum c_m (f_m - f_0) equals sum c_m f_m, and the differences of nearby values are exact
// in FP32 (the network reads its inputs in BF16).
constexpr int FT_Z = FEAT_TILE_Z, FT_R = FEAT_TILE_R, FT_H = 5;
constexpr int FB_Z = FT_Z + 2 * FT_H, FB_R = FT_R + 2 * FT_H;

__device__ __forceinline__ float fd1s(const FeatArgs& a, const float* box, int row, int bz, int br, int dirn) {
  if (row >= 9) return 0.0f;
  const int st = dirn == 1 ? 1 : FB_Z;
  const float* p = box + br * FB_Z + bz;
  const float f0 = p[0];
  if (row == 4) {  // centred row
    float s = a.sbp1[4][0] * (p[-2 * st] - f0);
#pragma unroll
    for (int m = 1; m < 5; ++m) s = s + a.sbp1[4][m] * (p[(m - 2) * st] - f0);
    return s;
  }
  const int w0 = sbp_w0(row);
  float s = a.sbp1[row][0] * (p[w0 * st] - f0);
#pragma unroll
  for (int m = 1; m < 6; ++m) s = s + a.sbp1[row][m] * (p[(w0 + m) * st] - f0);
  return s;
}

// The four channels of point (i, j) = (i0 + tz, j0 + tr) from the staged box.
__device__ __forceinline__ void features_point(const FeatArgs& a, float (*sb)[FB_R * FB_Z], int i, int j, int tz,
                                               int tr) {
  const Grid g = a.g;
  const long long o = (long long)j * g.P + i;
  const uint32_t dsc = __ldg(a.desc + o);
  const int zr = desc_blank(dsc) ? (int)ROW_NONE : desc_zrow(dsc);
  const int rw = desc_blank(dsc) ? (int)ROW_NONE : desc_rrow(dsc);
  const int bz = tz + FT_H, br = tr + FT_H;
  const float xz = (float)__ldg(a.dxidz + i), er = (float)__ldg(a.detadr + j);
  const float drdz = fd1s(a, sb[0], zr, bz, br, 1) * xz;
  const float dVrdz = fd1s(a, sb[1], zr, bz, br, 1) * xz;
  const float dVzdz = fd1s(a, sb[2], zr, bz, br, 1) * xz;
  const float drdr = fd1s(a, sb[0], rw, bz, br, 2) * er;
  const float dVrdr = fd1s(a, sb[1], rw, bz, br, 2) * er;
  const float dVzdr = fd1s(a, sb[2], rw, bz, br, 2) * er;
  const float vr = sb[1][br * FB_Z + bz];
  const float r = (float)__ldg(a.rc + j);
  const float dil = (j == 0) ? 2.0f * dVrdr + dVzdz : dVrdr + vr / r + dVzdz;
  const float grad = sqrtf(drdz * drdz + drdr * drdr);
  const float vort = fabsf(dVrdz - dVzdr);
  const float h = sqrtf((float)(__ldg(a.dz + i) * __ldg(a.dr + j)));
  a.feat[o] = make_float4(dil, grad, vort, h);
}

template <typename SIN>
__device__ __forceinline__ void features_body(const FeatArgs& a, int i0, int j0, float (*sb)[FB_R * FB_Z]) {
  const Grid g = a.g;
  const SIN* Urho = static_cast<const SIN*>(a.U);  // planes 0 (rho), 1 (V_r), 3 (V_z)
  const SIN* Uvr = Urho + g.plane;
  const SIN* Uvz = Urho + 3 * g.plane;
  const int tz = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int br = w; br < FB_R; br += 8) {
    const int j = j0 - FT_H + br;
    const bool jin = j >= 0 && j < g.Nr;
    const long long ro = (long long)j * g.P;
    for (int bz = tz; bz < FB_Z; bz += 32) {
      const int i = i0 - FT_H + bz;
      float v0 = 0.0f, v1 = 0.0f, v2 = 0.0f;
      if (jin && i >= 0 && i < g.Nz) {
        v0 = float(Urho[ro + i]);
        v1 = float(Uvr[ro + i]);
        v2 = float(Uvz[ro + i]);
      }
      const int q = br * FB_Z + bz;
      sb[0][q] = v0;
      sb[1][q] = v1;
      sb[2][q] = v2;
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int tr = w; tr < FT_R; tr += 8) {
    const int i = i0 + tz, j = j0 + tr;
    if (i >= g.Nz || j >= g.Nr) continue;
    features_point(a, sb, i, j, tz, tr);
  }
}

template <typename SIN>
__global__ void __launch_bounds__(256) features_kernel(const FeatArgs a) {
  __shared__ float sb[3][FB_R * FB_Z];
  features_body<SIN>(a, blockIdx.x * FT_Z, blockIdx.y * FT_R, sb);
}

// Batched: persistent loop over (i0, j0, instance) tiles of 32 x 16 points.
__global__ void __launch_bounds__(256) features_kernel_batch(const FeatArgs* __restrict__ argv,
                                                             const int4* __restrict__ tiles, int ntiles) {
  __shared__ float sb[3][FB_R * FB_Z];
  __shared__ __align__(16) FeatArgs sa;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int4 tt = tiles[t];
    __syncthreads();
    for (int k = threadIdx.x; k < (int)(sizeof(FeatArgs) / 4); k += blockDim.x)
      reinterpret_cast<unsigned int*>(&sa)[k] = reinterpret_cast<const unsigned int*>(argv + tt.z)[k];
    __syncthreads();
    if (sa.f32) features_body<float>(sa, tt.x, tt.y, sb);
    else features_body<double>(sa, tt.x, tt.y, sb);
  }
}

cudaError_t launch_features(const FeatArgs& a, cudaStream_t s) {
  const dim3 grid((a.g.Nz + FT_Z - 1) / FT_Z, (a.g.Nr + FT_R - 1) / FT_R);
  if (a.f32) features_kernel<float><<<grid, 256, 0, s>>>(a);
  else features_kernel<double><<<grid, 256, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Inference on the tensor cores. A tile is 32 (z) x 4 (r) points, one point per
// thread, thread t = row t of the MMA (TMEM lane t). One CTA of 128 threads owns 64
// TMEM columns: layer 1 accumulates there, and once every thread has read its row,
// layer 2 accumulates in the same columns. Shared memory (from a 128-aligned base):
// W1 64x112 and W2 64x64 in BF16; one A operand region of 128x112 BF16 that holds the
// layer-1 inputs and then (after the layer-1 MMAs completed) the layer-2 inputs, all
// in the no-swizzle K-major layout with the K chunks outermost (chunk c of 8 K values
// at c * rows * 16, row group g at g * 128, row r of the group at r * 16); the
// normalised channel box 4 x 8 x 36 in BF16, twice (the second copy one value on); biases and
// layer 3 in FP32. The next tile's channel box is loaded into registers while this tile's MMAs
// run. About 57 KB per CTA: 4 CTAs (16 warps, 256 TMEM columns) per SM.
// The tensor pipe is idle nine tenths of the time: building the operand rows and the GELU
// epilogues bound the kernel by issue, so the epilogues use the packed FP32 instructions and the
// rows are built from 32-bit words: 271 -> 252 us at 4400 x 640 on a B200.
// ---------------------------------------------------------------------------
constexpr int MT_Z = 32, MT_R = 4, MT_THREADS = 128;
constexpr int MBOX_Z = MT_Z + 4, MBOX_R = MT_R + 4, MBOX_N = MBOX_Z * MBOX_R;  // 288 points
constexpr int MBOX_PER = (MBOX_N + MT_THREADS - 1) / MT_THREADS;              // 3
constexpr uint32_t M_OW1 = 0;
constexpr uint32_t M_OW2 = M_OW1 + MLP_HID * MLP_K1 * 2;      // 14336
constexpr uint32_t M_OA = M_OW2 + MLP_HID * MLP_HID * 2;      // 22528
constexpr uint32_t M_OBOX = M_OA + MT_THREADS * MLP_K1 * 2;   // 51200
constexpr uint32_t M_OP = M_OBOX + 2 * MLP_CH * MBOX_N * 2;   // 55808 (the box and its shifted copy)
constexpr uint32_t M_NP = MLP_HID + MLP_HID + MLP_OUT * MLP_HID + MLP_OUT;
constexpr size_t M_SMEM = M_OP + M_NP * 4 + 128;  // + alignment slack
constexpr int M_CTAS_PER_SM = 4;

// byte offset of (row, k) in a K-major operand of `rows` rows
__device__ __forceinline__ uint32_t kmaj(int row, int k, int rows) {
  return (uint32_t)((k >> 3) * rows * 16 + (row >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

// BATCH: tiles (i0, j0, instance) from a table over many instances, each with its own
// arguments in argv (the model, its normalisation and the error flag are a0's, shared by
// the batch); otherwise the tiles of a0's grid in raster order.
template <bool BATCH>
__global__ void __launch_bounds__(MT_THREADS)
    mlp_infer_kernel(const InferArgs a0, const InferArgs* __restrict__ argv, const int4* __restrict__ tiles, int ntiles) {
  const InferArgs& a = a0;
  extern __shared__ unsigned char m_raw[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  unsigned char* base = m_raw + ((128u - (smem_addr(m_raw) & 127u)) & 127u);  // 128-aligned start
  const uint32_t sb = smem_addr(base);
  __nv_bfloat16* sBox = reinterpret_cast<__nv_bfloat16*>(base + M_OBOX);  // [4][8][36]
  float* sB1 = reinterpret_cast<float*>(base + M_OP);
  float* sB2 = sB1 + MLP_HID;
  float* sW3 = sB2 + MLP_HID;  // [2][64]
  float* sB3 = sW3 + MLP_OUT * MLP_HID;
  const int tid = threadIdx.x, warp = tid >> 5;
  // weights in BF16, core-matrix layout
  for (int e = tid; e < MLP_HID * MLP_K1; e += MT_THREADS) {
    const int n = e / MLP_K1, k = e - n * MLP_K1;
    *reinterpret_cast<__nv_bfloat16*>(base + M_OW1 + kmaj(n, k, MLP_HID)) = __float2bfloat16_rn(a.params[MLP_OFF_W1 + e]);
  }
  for (int e = tid; e < MLP_HID * MLP_HID; e += MT_THREADS) {
    const int n = e / MLP_HID, k = e - n * MLP_HID;
    *reinterpret_cast<__nv_bfloat16*>(base + M_OW2 + kmaj(n, k, MLP_HID)) = __float2bfloat16_rn(a.params[MLP_OFF_W2 + e]);
  }
  for (int e = tid; e < MLP_HID; e += MT_THREADS) {
    sB1[e] = a.params[MLP_OFF_B1 + e];
    sB2[e] = a.params[MLP_OFF_B2 + e];
  }
  for (int e = tid; e < MLP_OUT * MLP_HID; e += MT_THREADS) sW3[e] = a.params[MLP_OFF_W3 + e];
  if (tid < MLP_OUT) sB3[tid] = a.params[MLP_OFF_B3 + tid];
  if (tid == 0) bar_init(&bar);
  if (warp == 0) tmem_alloc(&tmem_slot, 64);

  // channel box of a tile: raw loads (zero outside the grid) into registers ...
  // tile t: origin and instance
  auto tile_of = [&](int t, int& ti0, int& tj0, int& inst) {
    if (BATCH) {
      const int4 tt = tiles[t];
      ti0 = tt.x;
      tj0 = tt.y;
      inst = tt.z;
    } else {
      ti0 = (t % a0.ntiles_z) * MT_Z;
      tj0 = (t / a0.ntiles_z) * MT_R;
      inst = 0;
    }
  };
  auto load_box = [&](int t, float4* v) {
    int ti0, tj0, inst;
    tile_of(t, ti0, tj0, inst);
    const InferArgs& at = BATCH ? argv[inst] : a0;
    const Grid g = at.g;
    const int i0 = ti0 - 2, j0 = tj0 - 2;
#pragma unroll
    for (int q = 0; q < MBOX_PER; ++q) {
      const int e = tid + q * MT_THREADS;
      v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (e < MBOX_N) {
        const int br = e / MBOX_Z, bz = e - br * MBOX_Z;
        const int i = i0 + bz, j = j0 + br;
        if (i >= 0 && i < g.Nz && j >= 0 && j < g.Nr) v[q] = __ldg(at.feat + (long long)j * g.P + i);
      }
    }
  };
  // ... then normalised into the BF16 box
  auto store_box = [&](const float4* v) {
#pragma unroll
    for (int q = 0; q < MBOX_PER; ++q) {
      const int e = tid + q * MT_THREADS;
      if (e < MBOX_N) {
        const float f[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          const __nv_bfloat16 x = __float2bfloat16_rn((f[ch] - a.norm.feat_mean[ch]) * a.norm.feat_inv_scale[ch]);
          sBox[ch * MBOX_N + e] = x;
          if (ch * MBOX_N + e > 0) sBox[MLP_CH * MBOX_N + ch * MBOX_N + e - 1] = x;  // the shifted copy
        }
      }
    }
  };
  float4 nxt[MBOX_PER];
  if ((int)blockIdx.x < ntiles) {
    load_box(blockIdx.x, nxt);
    store_box(nxt);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);

  const int c = tid & 31, rr = tid >> 5;  // this thread's point in the tile
  uint32_t phase = 0;
  bool ok = true;
  for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
    int i0, j0, inst;
    tile_of(t, i0, j0, inst);
    const InferArgs& at = BATCH ? argv[inst] : a0;
    const Grid g = at.g;
    // A row `tid` of layer 1: feature k = ch*25 + (dr+2)*5 + (dz+2), zero for k >= 100
    // Five values from column c on per (channel, row) as three words: a second copy of the box
    // one column further makes the words of odd columns aligned too.
    const uint32_t* bw = reinterpret_cast<const uint32_t*>(sBox + (c & 1) * (MLP_CH * MBOX_N)) + rr * (MBOX_Z / 2) + (c >> 1);
    auto words = [&](int gq, uint32_t (&w)[3]) {  // group gq = ch * 5 + dr
      const uint32_t* q = bw + (gq / 5) * (MBOX_N / 2) + (gq % 5) * (MBOX_Z / 2);
      w[0] = q[0];
      w[1] = q[1];
      w[2] = q[2];
    };
    uint32_t row[MLP_K1 / 2];
#pragma unroll
    for (int gq = 0; gq < MLP_IN / 5; gq += 2) {  // ten values, five words
      uint32_t w[3], n[3];
      words(gq, w);
      words(gq + 1, n);
      uint32_t* o = row + gq / 2 * 5;
      o[0] = w[0];
      o[1] = w[1];
      o[2] = __byte_perm(w[2], n[0], 0x5410);  // low halves
      o[3] = __byte_perm(n[0], n[1], 0x5432);  // high, low
      o[4] = __byte_perm(n[1], n[2], 0x5432);
    }
#pragma unroll
    for (int e = MLP_IN / 2; e < MLP_K1 / 2; ++e) row[e] = 0u;
#pragma unroll
    for (int kc = 0; kc < MLP_K1 / 8; ++kc)
      *reinterpret_cast<uint4*>(base + M_OA + kmaj(tid, kc * 8, MT_THREADS)) =
          make_uint4(row[4 * kc], row[4 * kc + 1], row[4 * kc + 2], row[4 * kc + 3]);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int s = 0; s < MLP_K1 / 16; ++s)
        mma_bf16(tmem, mdesc(sb + M_OA + s * 2 * MT_THREADS * 16, MT_THREADS * 16, 128),
                 mdesc(sb + M_OW1 + s * 2 * MLP_HID * 16, MLP_HID * 16, 128), IDESC_BF16_M128_N64, s > 0);
      mma_commit(&bar);
    }
    __syncwarp();
    // the next tile's channel values travel while the MMAs run
    const int tn = t + gridDim.x;
    if (tn < ntiles) load_box(tn, nxt);
    ok = __syncthreads_and(bar_wait(&bar, phase));
    phase ^= 1u;
    if (!ok) break;
    tc_fence_after();
    // layer 1 epilogue: z1 + b1 -> GELU -> BF16 row of the layer-2 A operand, written
    // over the layer-1 operand (its MMAs completed)
    float z[MLP_HID];
#pragma unroll
    for (int q = 0; q < MLP_HID / 16; ++q) tmem_ld16(lane_base + q * 16, z + q * 16);
    tmem_wait_ld();
#pragma unroll
    for (int q = 0; q < MLP_HID / 8; ++q) {
      uint32_t pk[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int e = q * 8 + 2 * h;
        float g0, g1;
        unpk2(gelu_fast2(add2(pk2(z[e], z[e + 1]), *reinterpret_cast<const f32x2*>(sB1 + e))), g0, g1);
        pk[h] = pack_bf16(g0, g1);
      }
      *reinterpret_cast<uint4*>(base + M_OA + kmaj(tid, q * 8, MT_THREADS)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int s = 0; s < MLP_HID / 16; ++s)
        mma_bf16(tmem, mdesc(sb + M_OA + s * 2 * MT_THREADS * 16, MT_THREADS * 16, 128),
                 mdesc(sb + M_OW2 + s * 2 * MLP_HID * 16, MLP_HID * 16, 128), IDESC_BF16_M128_N64, s > 0);
      mma_commit(&bar);
    }
    __syncwarp();
    // the box of this tile is no longer read: the next tile's goes in while the MMAs run
    if (tn < ntiles) store_box(nxt);
    ok = __syncthreads_and(bar_wait(&bar, phase));
    phase ^= 1u;
    if (!ok) break;
    tc_fence_after();
    // layer 2 epilogue and layer 3 (64 -> 2) in FP32
#pragma unroll
    for (int q = 0; q < MLP_HID / 16; ++q) tmem_ld16(lane_base + q * 16, z + q * 16);
    tmem_wait_ld();
    f32x2 a0 = pk2(sB3[0], 0.0f), a1 = pk2(sB3[1], 0.0f);
#pragma unroll
    for (int h = 0; h < MLP_HID; h += 2) {
      const f32x2 hv = gelu_fast2(add2(pk2(z[h], z[h + 1]), *reinterpret_cast<const f32x2*>(sB2 + h)));
      a0 = fma2(*reinterpret_cast<const f32x2*>(sW3 + h), hv, a0);
      a1 = fma2(*reinterpret_cast<const f32x2*>(sW3 + MLP_HID + h), hv, a1);
    }
    float y0, y1, yo;
    unpk2(a0, y0, yo);
    y0 += yo;
    unpk2(a1, y1, yo);
    y1 += yo;
    tc_fence_before();
    const int i = i0 + c, j = j0 + rr;
    if (i < g.Nz && j < g.Nr) {
      const long long o = (long long)j * g.P + i;
      const double ramp = __ldg(at.ramp + i);
      const double p0 = (double)(y0 * a.norm.out_scale[0]) * ramp;
      const double p1 = (double)(y1 * a.norm.out_scale[1]) * ramp;
      if (at.mode == 0) {
        at.out[o] = p0;
        at.out[g.plane + o] = p1;
      } else {
        const unsigned char m = __ldg(at.mask + o);
        at.out[g.plane + o] = (m & 1) ? __ldg(at.held + o) : p0;
        at.out[2 * g.plane + o] = (m & 2) ? __ldg(at.held + g.plane + o) : p1;
      }
    }
    fence_async_smem();  // the next tile's box (generic writes) before its A operand is built
    __syncthreads();
  }
  if (!ok) {
    if (tid == 0) atomicOr(a.flags, 4);
    // let the MMA whose completion timed out finish (bounded) before the columns are
    // released (phase was already advanced past it)
    bar_wait(&bar, phase ^ 1u);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 64);
}

cudaError_t launch_mlp_infer(const InferArgs& a, cudaStream_t s) {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // at most 4 CTAs per SM (shared memory): 4 x 64 of the 512 TMEM columns
  const int grid = a.ntiles < M_CTAS_PER_SM * nsm ? a.ntiles : M_CTAS_PER_SM * nsm;
  if (grid <= 0) return cudaSuccess;
  mlp_infer_kernel<false><<<grid, MT_THREADS, M_SMEM, s>>>(a, nullptr, nullptr, a.ntiles);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Judge
// ---------------------------------------------------------------------------
__device__ __forceinline__ void judge_body(const JudgeArgs& a, long long p) {
  const Grid g = a.g;
  const long long n = (long long)g.Nz * g.Nr;
  unsigned long long fb = 0, judged = 0;
  if (p < n) {
    const int j = (int)(p / g.Nz), i = (int)(p - (long long)j * g.Nz);
    const long long o = (long long)j * g.P + i;
    unsigned char m = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double* pl = a.plain + k * g.plane;
      double lm = 0.0;
      for (int dr = -2; dr <= 2; ++dr)
        for (int dz = -2; dz <= 2; ++dz) {
          const int ii = i + dz, jj = j + dr;
          if (ii >= 0 && ii < g.Nz && jj >= 0 && jj < g.Nr) lm = fmax(lm, fabs(__ldg(pl + (long long)jj * g.P + ii)));
        }
      const double plain = __ldg(pl + o);
      const double pred = __ldg(a.pred + k * g.plane + o);
      if (fabs(pred - plain) > a.thr * lm) m |= (unsigned char)(1 << k);
      a.held[k * g.plane + o] = plain;
    }
    a.mask[o] = m;
    judged = 2;
    fb = (m & 1) + ((m >> 1) & 1);
  }
  // warp totals, one atomic per warp
  for (int off = 16; off > 0; off >>= 1) {
    fb += __shfl_down_sync(0xffffffffu, fb, off);
    judged += __shfl_down_sync(0xffffffffu, judged, off);
  }
  if ((threadIdx.x & 31) == 0 && judged) {
    atomicAdd(a.counts + 0, judged);
    atomicAdd(a.counts + 1, fb);
  }
}

__global__ void judge_kernel(const JudgeArgs a) { judge_body(a, (long long)blockIdx.x * blockDim.x + threadIdx.x); }

// Batched: blockIdx.y = instance.
__global__ void judge_kernel_batch(const JudgeArgs* __restrict__ argv) {
  judge_body(argv[blockIdx.y], (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

cudaError_t launch_judge_batch(const JudgeArgs* argv, int ninst, long long max_pts, cudaStream_t s) {
  const int bs = 256;
  judge_kernel_batch<<<dim3((unsigned)((max_pts + bs - 1) / bs), ninst), bs, 0, s>>>(argv);
  return cudaGetLastError();
}

cudaError_t launch_features_batch(const FeatArgs* argv, const int4* tiles, int ntiles, int grid, cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  features_kernel_batch<<<grid, 256, 0, s>>>(argv, tiles, ntiles);
  return cudaGetLastError();
}

cudaError_t launch_mlp_infer_batch(const InferArgs& a0, const InferArgs* argv, const int4* tiles, int ntiles,
                                   cudaStream_t s) {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int grid = ntiles < M_CTAS_PER_SM * nsm ? ntiles : M_CTAS_PER_SM * nsm;
  if (grid <= 0) return cudaSuccess;
  mlp_infer_kernel<true><<<grid, MT_THREADS, M_SMEM, s>>>(a0, argv, tiles, ntiles);
  return cudaGetLastError();
}

cudaError_t launch_judge(const JudgeArgs& a, cudaStream_t s) {
  const long long n = (long long)a.g.Nz * a.g.Nr;
  const int bs = 256;
  judge_kernel<<<(int)((n + bs - 1) / bs), bs, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Training (FP32)
// ---------------------------------------------------------------------------
__host__ __device__ inline uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Sample b of training step `step`: snapshot u % S, point (u >> 32) % (Nz*Nr).
__global__ void sample_kernel(const Dataset d, const MlpNorm norm, unsigned long long seed, const int* step, int B,
                              float* X, float* T) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)B * MLP_K1) return;
  const int b = (int)(e / MLP_K1), k = (int)(e - (long long)b * MLP_K1);
  const uint64_t u = mix64(mix64(seed + (uint64_t)(*step) * 0x9E3779B97F4A7C15ull) + (uint64_t)b);
  const int s = (int)(u % (uint64_t)d.S);
  const long long npts = (long long)d.g.Nz * d.g.Nr;
  const long long p = (long long)((u >> 32) % (uint64_t)npts);
  const int j = (int)(p / d.g.Nz), i = (int)(p - (long long)j * d.g.Nz);
  float v = 0.0f;
  if (k < MLP_IN) {
    const int ch = k / 25, w = k - ch * 25, dr = w / 5 - 2, dz = w % 5 - 2;
    const int ii = i + dz, jj = j + dr;
    float raw = 0.0f;
    if (ii >= 0 && ii < d.g.Nz && jj >= 0 && jj < d.g.Nr) {
      const float4 f = __ldg(d.feat + (long long)s * d.g.plane + (long long)jj * d.g.P + ii);
      raw = ch == 0 ? f.x : (ch == 1 ? f.y : (ch == 2 ? f.z : f.w));
    }
    v = (raw - norm.feat_mean[ch]) * norm.feat_inv_scale[ch];
  }
  X[e] = v;
  if (k < MLP_OUT) {
    const float2 t = __ldg(d.targ + (long long)s * d.g.plane + (long long)j * d.g.P + i);
    T[(long long)b * MLP_OUT + k] = (k == 0 ? t.x : t.y) / norm.out_scale[k];
  }
}

cudaError_t launch_sample(const Dataset& d, MlpNorm norm, unsigned long long seed, const int* step, int B, float* X,
                          float* T, cudaStream_t s) {
  const long long n = (long long)B * MLP_K1;
  const int bs = 256;
  sample_kernel<<<(int)((n + bs - 1) / bs), bs, 0, s>>>(d, norm, seed, step, B, X, T);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// One training step: forward and backward pass of a batch and its parameter gradients, in one
// kernel (FP32). As separate GEMM, bias, activation and column-sum kernels the batch's seven
// 64-column intermediates crossed memory once or more each (about 0.3 GB per step at 65,536
// points), and the weight-gradient GEMMs, whose reduction runs over the batch, ran as 64 CTAs
// of a serial 1024-row sum each: 0.60 of 0.98 ms per step.
//
// Here a persistent CTA per SM takes tiles of TB = 128 points: the gathered inputs, both
// hidden layers and the weights (in both orientations) stay in its shared memory, the
// pre-activations of a thread's 8 x 4 block in its registers, and the weight gradients
// accumulate in registers over up to TFLUSH of the CTA's tiles and then go to rows of `part`
// (two per CTA), which the update kernel sums in a fixed order: a step is deterministic.
// Thread blocks of 8 x 4 outputs read 3 float4 of shared memory per 32 FMA (forward and input
// gradients: points ty + 16 r, columns 4 tx..), of 8 x 7 and 8 x 4 in the weight gradients
// (half the tile's points per 128 threads), so the FP32 pipe, not shared memory, is the bound.
// Measured on a B200, a step of 65,536 points: 980 us in 20 launches -> 143 us + 7 us (update);
// a 20-step training call 25.1 -> 4.1 ms. The FP32 multiply-adds alone take 45 us at the pipe's
// rate, 52 with four rounds of tiles for 3.46 per SM; the rest is one CTA's barriers,
// the gather of a tile's windows and the activations.
// ---------------------------------------------------------------------------
constexpr int TB = 128;         // points per tile
constexpr int TT = 256;         // threads
// Tiles whose weight gradients are summed in registers before they are added to the rows of part:
// no sum runs over more than 8 * 64 points one by one. Over all of a CTA's tiles the rounding of
// 2**21 points grew to 7e-5 of an entry (sums of 1024: 2e-5).
constexpr int TFLUSH = 8;
constexpr int TXP = MLP_K1 + 4;  // row pitch of the input tile (float4 rows, banks of adjacent rows apart)
constexpr int THP = MLP_HID + 4;
struct TrainSmem {
  float X[TB][TXP];            // normalised inputs, columns past MLP_IN zero
  float H1[TB][THP];           // first hidden layer
  float D[TB][THP];            // dL/dz2, then dL/dz1
  float W1t[MLP_IN][MLP_HID];  // [k][n]
  float W2t[MLP_HID][MLP_HID];  // [k][n]
  float W2[MLP_HID][MLP_HID];   // [n][k]
  float W3[MLP_OUT][MLP_HID];
  float B1[MLP_HID], B2[MLP_HID], B3[MLP_OUT];
  float T[TB][MLP_OUT];
  long long src[TB];           // sampled point's offset in its plane of the data set (snapshot included)
  int si[TB], sj[TB];
};

__device__ __forceinline__ void fma4(float (&acc)[4], float a, const float4& w) {
  acc[0] = fmaf(a, w.x, acc[0]);
  acc[1] = fmaf(a, w.y, acc[1]);
  acc[2] = fmaf(a, w.z, acc[2]);
  acc[3] = fmaf(a, w.w, acc[3]);
}

// acc[r][c] += sum_k A[ty + 16 r][k] W[k][4 tx + c], k < K (a multiple of 4); A's row pitch in floats.
template <int K>
__device__ __forceinline__ void tile_gemm(float (&acc)[8][4], const float* A, int pitch, const float* W, int tx, int ty) {
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    float4 w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = *reinterpret_cast<const float4*>(W + (k + q) * MLP_HID + 4 * tx);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float4 a = *reinterpret_cast<const float4*>(A + (ty + 16 * r) * pitch + k);
      fma4(acc[r], a.x, w[0]);
      fma4(acc[r], a.y, w[1]);
      fma4(acc[r], a.z, w[2]);
      fma4(acc[r], a.w, w[3]);
    }
  }
}

// SAMPLED: the batch is drawn from the data set (sample_kernel's hash of (seed, step, b));
// else Xg [B x MLP_IN], Tg [B x MLP_OUT] hold it.
template <bool SAMPLED>
__global__ void __launch_bounds__(TT, 1)
    train_step_kernel(const Dataset d, const MlpNorm norm, unsigned long long seed, long long step, int B,
                      const float* __restrict__ Xg, const float* __restrict__ Tg, const float* __restrict__ P,
                      float* __restrict__ part, float* __restrict__ lpart) {
  extern __shared__ __align__(16) unsigned char train_raw[];
  TrainSmem& s = *reinterpret_cast<TrainSmem*>(train_raw);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int half = tid >> 7, ng = (tid & 127) >> 4, kg = tid & 15;  // weight-gradient blocks
  for (int e = tid; e < MLP_HID * MLP_IN; e += TT) {
    const int n = e / MLP_IN, k = e - n * MLP_IN;
    s.W1t[k][n] = P[MLP_OFF_W1 + n * MLP_K1 + k];
  }
  for (int e = tid; e < MLP_HID * MLP_HID; e += TT) {
    const int n = e / MLP_HID, k = e - n * MLP_HID;
    const float w = P[MLP_OFF_W2 + e];
    s.W2[n][k] = w;
    s.W2t[k][n] = w;
  }
  if (tid < MLP_OUT * MLP_HID) s.W3[tid / MLP_HID][tid % MLP_HID] = P[MLP_OFF_W3 + tid];
  if (tid < MLP_HID) {
    s.B1[tid] = P[MLP_OFF_B1 + tid];
    s.B2[tid] = P[MLP_OFF_B2 + tid];
  }
  if (tid < MLP_OUT) s.B3[tid] = P[MLP_OFF_B3 + tid];
  for (int e = tid; e < TB * (TXP - MLP_IN); e += TT) s.X[e / (TXP - MLP_IN)][MLP_IN + e % (TXP - MLP_IN)] = 0.0f;

  float g1[8][7], g2[8][4], g3[MLP_OUT][4], gb1[4], gb2[4], gb3[MLP_OUT], lsum = 0.0f;
#pragma unroll
  for (int x = 0; x < 8; ++x) {
#pragma unroll
    for (int y = 0; y < 7; ++y) g1[x][y] = 0.0f;
#pragma unroll
    for (int y = 0; y < 4; ++y) g2[x][y] = 0.0f;
  }
#pragma unroll
  for (int y = 0; y < 4; ++y) gb1[y] = gb2[y] = g3[0][y] = g3[1][y] = 0.0f;
  gb3[0] = gb3[1] = 0.0f;
  const float invB = 1.0f / (float)B;
  const int ntile = (B + TB - 1) / TB;
  float* row = part + (long long)(2 * blockIdx.x + half) * MLP_NPARAM;
  int held = 0;  // tiles summed in the registers
  bool first = true;
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int b0 = tile * TB;
    __syncthreads();  // the previous tile's reads of X, D and T are done
    // ---- inputs and targets (points past the batch: zeros, and no gradient below)
    if (SAMPLED) {
      if (tid < TB) {
        long long o = -1;
        int i = 0, j = 0;
        float2 t = make_float2(0.0f, 0.0f);
        if (b0 + tid < B) {
          const uint64_t u = mix64(mix64(seed + (uint64_t)step * 0x9E3779B97F4A7C15ull) + (uint64_t)(b0 + tid));
          const long long npts = (long long)d.g.Nz * d.g.Nr;
          const long long p = (long long)((u >> 32) % (uint64_t)npts);
          j = (int)(p / d.g.Nz);
          i = (int)(p - (long long)j * d.g.Nz);
          o = (long long)(u % (uint64_t)d.S) * d.g.plane + (long long)j * d.g.P + i;
          t = __ldg(d.targ + o);
          t.x /= norm.out_scale[0];
          t.y /= norm.out_scale[1];
        }
        s.src[tid] = o;
        s.si[tid] = i;
        s.sj[tid] = j;
        s.T[tid][0] = t.x;
        s.T[tid][1] = t.y;
      }
      __syncthreads();
      constexpr int NW = (TB * 25 + TT - 1) / TT;
      float4 f[NW];  // all of a thread's window values in flight
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        const int e = tid + q * TT, b = e / 25, w = e - 25 * b;
        f[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (b < TB && s.src[b] >= 0) {
          const int dr = w / 5 - 2, dz = w % 5 - 2;
          const int ii = s.si[b] + dz, jj = s.sj[b] + dr;
          if (ii >= 0 && ii < d.g.Nz && jj >= 0 && jj < d.g.Nr) f[q] = __ldg(d.feat + s.src[b] + dr * d.g.P + dz);
        }
      }
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        const int e = tid + q * TT, b = e / 25, w = e - 25 * b;
        if (b < TB) {
          const bool on = s.src[b] >= 0;
          s.X[b][w] = on ? (f[q].x - norm.feat_mean[0]) * norm.feat_inv_scale[0] : 0.0f;
          s.X[b][25 + w] = on ? (f[q].y - norm.feat_mean[1]) * norm.feat_inv_scale[1] : 0.0f;
          s.X[b][50 + w] = on ? (f[q].z - norm.feat_mean[2]) * norm.feat_inv_scale[2] : 0.0f;
          s.X[b][75 + w] = on ? (f[q].w - norm.feat_mean[3]) * norm.feat_inv_scale[3] : 0.0f;
        }
      }
    } else {
      for (int e = tid; e < TB * MLP_IN; e += TT) {
        const int b = e / MLP_IN, k = e - b * MLP_IN;
        s.X[b][k] = b0 + b < B ? Xg[(long long)(b0 + b) * MLP_IN + k] : 0.0f;
      }
      if (tid < TB * MLP_OUT) {
        const int b = tid / MLP_OUT, k = tid - b * MLP_OUT;
        s.T[b][k] = b0 + b < B ? Tg[(long long)(b0 + b) * MLP_OUT + k] : 0.0f;
      }
    }
    __syncthreads();
    // ---- layer 1
    float z1[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) z1[r][c] = 0.0f;
    tile_gemm<MLP_IN>(z1, &s.X[0][0], TXP, &s.W1t[0][0], tx, ty);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
#pragma unroll
      for (int c = 0; c < 4; ++c) z1[r][c] += s.B1[4 * tx + c];
      *reinterpret_cast<float4*>(&s.H1[ty + 16 * r][4 * tx]) =
          make_float4(gelu_f(z1[r][0]), gelu_f(z1[r][1]), gelu_f(z1[r][2]), gelu_f(z1[r][3]));
    }
    __syncthreads();
    // ---- layer 2, output layer, loss, and back to dL/dz2
    {
      float z2[8][4];
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) z2[r][c] = 0.0f;
      tile_gemm<MLP_HID>(z2, &s.H1[0][0], THP, &s.W2t[0][0], tx, ty);
      const float4 w30 = *reinterpret_cast<const float4*>(&s.W3[0][4 * tx]);
      const float4 w31 = *reinterpret_cast<const float4*>(&s.W3[1][4 * tx]);
      const float v0[4] = {w30.x, w30.y, w30.z, w30.w}, v1[4] = {w31.x, w31.y, w31.z, w31.w};
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        float h2[4], y0 = 0.0f, y1 = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          z2[r][c] += s.B2[4 * tx + c];
          h2[c] = gelu_f(z2[r][c]);
          y0 = fmaf(h2[c], v0[c], y0);
          y1 = fmaf(h2[c], v1[c], y1);
        }
        // over the 16 threads of the row
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) {
          y0 += __shfl_xor_sync(0xffffffffu, y0, off);
          y1 += __shfl_xor_sync(0xffffffffu, y1, off);
        }
        const int b = ty + 16 * r;
        const bool on = b0 + b < B;
        const float e0 = on ? (y0 + s.B3[0]) - s.T[b][0] : 0.0f, e1 = on ? (y1 + s.B3[1]) - s.T[b][1] : 0.0f;
        const float d0 = 2.0f * e0 * invB, d1 = 2.0f * e1 * invB;
        if (tx == 0) {
          lsum += e0 * e0 + e1 * e1;
          gb3[0] += d0;
          gb3[1] += d1;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          g3[0][c] = fmaf(d0, h2[c], g3[0][c]);
          g3[1][c] = fmaf(d1, h2[c], g3[1][c]);
          const float dz = fmaf(d1, v1[c], d0 * v0[c]) * gelu_grad_f(z2[r][c]);
          gb2[c] += dz;
          z2[r][c] = dz;
        }
        *reinterpret_cast<float4*>(&s.D[b][4 * tx]) = make_float4(z2[r][0], z2[r][1], z2[r][2], z2[r][3]);
      }
    }
    __syncthreads();
    // ---- dL/dz1 (kept in registers until D has been read) and the W2 gradient
    float dz1[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) dz1[r][c] = 0.0f;
    tile_gemm<MLP_HID>(dz1, &s.D[0][0], THP, &s.W2[0][0], tx, ty);
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        dz1[r][c] *= gelu_grad_f(z1[r][c]);
        gb1[c] += dz1[r][c];
      }
#pragma unroll 4
    for (int b = half * (TB / 2); b < (half + 1) * (TB / 2); ++b) {
      const float4 a0 = *reinterpret_cast<const float4*>(&s.D[b][8 * ng]);
      const float4 a1 = *reinterpret_cast<const float4*>(&s.D[b][8 * ng + 4]);
      const float4 h = *reinterpret_cast<const float4*>(&s.H1[b][4 * kg]);
      fma4(g2[0], a0.x, h);
      fma4(g2[1], a0.y, h);
      fma4(g2[2], a0.z, h);
      fma4(g2[3], a0.w, h);
      fma4(g2[4], a1.x, h);
      fma4(g2[5], a1.y, h);
      fma4(g2[6], a1.z, h);
      fma4(g2[7], a1.w, h);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; ++r)
      *reinterpret_cast<float4*>(&s.D[ty + 16 * r][4 * tx]) = make_float4(dz1[r][0], dz1[r][1], dz1[r][2], dz1[r][3]);
    __syncthreads();
    // ---- W1 gradient: columns kg + 16 t (the padding columns of X are zero)
#pragma unroll 2
    for (int b = half * (TB / 2); b < (half + 1) * (TB / 2); ++b) {
      const float4 a0 = *reinterpret_cast<const float4*>(&s.D[b][8 * ng]);
      const float4 a1 = *reinterpret_cast<const float4*>(&s.D[b][8 * ng + 4]);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int t = 0; t < 7; ++t) {
        const float x = s.X[b][kg + 16 * t];
#pragma unroll
        for (int c = 0; c < 8; ++c) g1[c][t] = fmaf(a[c], x, g1[c][t]);
      }
    }
    // ---- the weight gradients of these tiles to the half's row of part (eleven loads in flight)
    if (++held == TFLUSH || tile + gridDim.x >= ntile) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float* w1 = row + MLP_OFF_W1 + (8 * ng + c) * MLP_K1 + kg;
        float* w2 = row + MLP_OFF_W2 + (8 * ng + c) * MLP_HID + 4 * kg;
        float s1[7], s2[4];
#pragma unroll
        for (int t = 0; t < 7; ++t) s1[t] = first ? 0.0f : w1[16 * t];
#pragma unroll
        for (int q = 0; q < 4; ++q) s2[q] = first ? 0.0f : w2[q];
#pragma unroll
        for (int t = 0; t < 7; ++t) {
          w1[16 * t] = s1[t] + g1[c][t];
          g1[c][t] = 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          w2[q] = s2[q] + g2[c][q];
          g2[c][q] = 0.0f;
        }
      }
      first = false;
      held = 0;
    }
  }
  // ---- the CTA's other sums, reduced over ty into its first row
  __syncthreads();  // every thread is done with the tile buffers
  float* red = &s.X[0][0];  // [16][4 x 64 + 4]
  constexpr int RP = 4 * MLP_HID + 4;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    red[ty * RP + 4 * tx + c] = gb1[c];
    red[ty * RP + MLP_HID + 4 * tx + c] = gb2[c];
    red[ty * RP + 2 * MLP_HID + 4 * tx + c] = g3[0][c];
    red[ty * RP + 3 * MLP_HID + 4 * tx + c] = g3[1][c];
  }
  if (tx == 0) {
    red[ty * RP + 4 * MLP_HID] = gb3[0];
    red[ty * RP + 4 * MLP_HID + 1] = gb3[1];
    red[ty * RP + 4 * MLP_HID + 2] = lsum;
  }
  __syncthreads();
  float* row0 = part + (long long)(2 * blockIdx.x) * MLP_NPARAM;
  float* row1 = row0 + MLP_NPARAM;
  for (int e = tid; e < 4 * MLP_HID + 3; e += TT) {
    float v = 0.0f;
#pragma unroll
    for (int q = 0; q < 16; ++q) v += red[q * RP + e];
    if (e == 4 * MLP_HID + 2) {
      lpart[blockIdx.x] = v * invB;
    } else {
      const int o = e < MLP_HID ? MLP_OFF_B1 + e
                                : (e < 2 * MLP_HID ? MLP_OFF_B2 + e - MLP_HID
                                                   : (e < 4 * MLP_HID ? MLP_OFF_W3 + e - 2 * MLP_HID
                                                                      : MLP_OFF_B3 + e - 4 * MLP_HID));
      row0[o] = v;
      row1[o] = 0.0f;
    }
  }
}

// Sums the rows of part and the batch loss; g != null: the gradient goes there, else Adam
// updates p, m, v with it (bias corrections of step t = step + 1). Eight threads per
// parameter, consecutive parameters coalesced.
constexpr int AD_P = 32, AD_R = 8;
__global__ void __launch_bounds__(AD_P* AD_R)
    train_update_kernel(const float* __restrict__ part, int nrow, const float* __restrict__ lpart, int nl, float* p,
                        float* m, float* v, float* g, float* loss, long long step, float lr, float b1, float b2,
                        float eps) {
  __shared__ float red[AD_R][AD_P];
  const int c = threadIdx.x & (AD_P - 1), q = threadIdx.x / AD_P;
  const int e = blockIdx.x * AD_P + c;
  float sum = 0.0f;
  if (e < MLP_NPARAM) {
#pragma unroll 4
    for (int r = q; r < nrow; r += AD_R) sum += part[(long long)r * MLP_NPARAM + e];
  }
  red[q][c] = sum;
  __syncthreads();
  if (blockIdx.x == 0 && q == 1) {  // the loss of the step, by one warp
    float l = 0.0f;
    for (int k = c; k < nl; k += 32) l += lpart[k];
    for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
    if (c == 0) loss[step] = l;
  }
  if (q != 0 || e >= MLP_NPARAM) return;
  float gg = 0.0f;
#pragma unroll
  for (int k = 0; k < AD_R; ++k) gg += red[k][c];
  if (g) {
    g[e] = gg;
    return;
  }
  const float t = (float)(step + 1);
  const float mm = b1 * m[e] + (1.0f - b1) * gg;
  const float vv = b2 * v[e] + (1.0f - b2) * gg * gg;
  m[e] = mm;
  v[e] = vv;
  const float mhat = mm / (1.0f - powf(b1, t));
  const float vhat = vv / (1.0f - powf(b2, t));
  p[e] = p[e] - lr * mhat / (sqrtf(vhat) + eps);
}

int train_grid(int B) {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int nt = (B - 1) / TB + 1;
  return nt < nsm ? nt : nsm;
}

cudaError_t launch_train_pass(const Dataset* d, const MlpNorm& norm, unsigned long long seed, long long step, int B,
                              const float* X, const float* T, const float* P, float* part, float* lpart,
                              cudaStream_t s) {
  const int grid = train_grid(B);
  if (d) train_step_kernel<true><<<grid, TT, sizeof(TrainSmem), s>>>(*d, norm, seed, step, B, X, T, P, part, lpart);
  else train_step_kernel<false><<<grid, TT, sizeof(TrainSmem), s>>>(Dataset{}, norm, seed, step, B, X, T, P, part, lpart);
  return cudaGetLastError();
}

cudaError_t launch_train_update(const float* part, const float* lpart, int B, float* p, float* m, float* v, float* g,
                                float* loss, long long step, float lr, float b1, float b2, float eps, cudaStream_t s) {
  const int grid = train_grid(B);
  train_update_kernel<<<(MLP_NPARAM + AD_P - 1) / AD_P, AD_P * AD_R, 0, s>>>(part, 2 * grid, lpart, grid, p, m, v, g,
                                                                             loss, step, lr, b1, b2, eps);
  return cudaGetLastError();
}

// acc: [0..3] channel sums, [4..7] channel sums of squares, [8..9] target sums of
// squares, [10] point count.
__global__ void dataset_stats_kernel(const Dataset d, double* acc) {
  __shared__ double red[11][8];
  double loc[11];
#pragma unroll
  for (int k = 0; k < 11; ++k) loc[k] = 0.0;
  const long long npts = (long long)d.g.Nz * d.g.Nr;
  const long long n = npts * d.S;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int s = (int)(e / npts);
    const long long p = e - (long long)s * npts;
    const int j = (int)(p / d.g.Nz), i = (int)(p - (long long)j * d.g.Nz);
    const long long o = (long long)s * d.g.plane + (long long)j * d.g.P + i;
    const float4 f = __ldg(d.feat + o);
    const float2 t = __ldg(d.targ + o);
    loc[0] += f.x; loc[1] += f.y; loc[2] += f.z; loc[3] += f.w;
    loc[4] += (double)f.x * f.x; loc[5] += (double)f.y * f.y; loc[6] += (double)f.z * f.z; loc[7] += (double)f.w * f.w;
    loc[8] += (double)t.x * t.x; loc[9] += (double)t.y * t.y;
    loc[10] += 1.0;
  }
#pragma unroll
  for (int k = 0; k < 11; ++k) {
    double v = loc[k];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 11) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
    atomicAdd(acc + threadIdx.x, t);
  }
}

cudaError_t launch_dataset_stats(const Dataset& d, double* acc, cudaStream_t s) {
  dataset_stats_kernel<<<148 * 4, 256, 0, s>>>(d, acc);
  return cudaGetLastError();
}

__global__ void pack_targets_kernel(const Grid g, const double* star, float2* targ) {
  const long long n = (long long)g.Nz * g.Nr;
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int j = (int)(p / g.Nz), i = (int)(p - (long long)j * g.Nz);
  const long long o = (long long)j * g.P + i;
  targ[o] = make_float2((float)star[g.plane + o], (float)star[2 * g.plane + o]);
}

cudaError_t launch_pack_targets(const Grid& g, const double* star, float2* targ, cudaStream_t s) {
  const long long n = (long long)g.Nz * g.Nr;
  pack_targets_kernel<<<(int)((n + 255) / 256), 256, 0, s>>>(g, star, targ);
  return cudaGetLastError();
}

cudaError_t mlp_init_attributes() {
  cudaError_t e = cudaFuncSetAttribute(mlp_infer_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M_SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(mlp_infer_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M_SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(train_step_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(train_step_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem));
}

}  // namespace axj
