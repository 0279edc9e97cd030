// parmap_mlp.cu -- see parmap_mlp.cuh.
//
// The 128 x 128 layers are tcgen05.mma (kind::f16, BF16 x BF16 -> FP32,
// M = N = 128, K = 16 per instruction) on tiles of 128 batch rows, issued by
// one thread on operands staged in shared memory in the no-swizzle canonical
// layout, with the FP32 accumulators in tensor memory; a thread reads its row
// back with tcgen05.ld (32x32b: warp w owns TMEM lanes 32 (w mod 4) ..  = rows).
// Activations are rounded to BF16 where they enter a tensor-core product.
// Inference: a CTA of 512 threads holds both weight images and runs four
// tiles at a time, one on each group of four warps, so that the products of
// one overlap the activations of the others.  Training: the 512 threads share
// one tile, each a row and a quarter of its columns.
#include "parmap_mlp.cuh"

#include <cuda_bf16.h>

namespace aak {
namespace mlp {

namespace {

constexpr int kGroups = 4;                       // groups of four warps a CTA
constexpr int kThreads = kGroups * kTileRows;    // 512

// ------------------------------------------------------------------ BF16
__device__ __forceinline__ uint32_t bf16_bits(float x) { return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float bf16_val(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }

// ------------------------------------------------------------------ operand layout
// K-major, no swizzle: core matrices of 8 rows x 16 bytes (8 BF16) stored as
// 128 contiguous bytes; core (r/8, k/8) starts at byte (r/8) * 2048 + (k/8) * 128.
// In descriptor terms LBO = 128 B (K-adjacent cores), SBO = 2048 B (8-row groups).
__host__ __device__ __forceinline__ int canon(int r, int k) {
  return (((r >> 3) * 16 + (k >> 3)) << 6) + ((r & 7) << 3) + (k & 7);
}
constexpr uint32_t kLBO = 128, kSBO = 2048;
// The same image read with its columns as the M or N index (MN-major: eight
// contiguous M or N elements of eight K rows a core): cores adjacent along M or
// N are 128 B apart (SBO), those along K 2048 B (LBO), and a step of K = 16 is
// two of the latter.  So one image of activations [row][k] serves the forward
// product (K = k) and the weight gradient (K = row), and one weight image
// [out][in] the forward (K = in) and the backward product (K = out).
// Instruction descriptor (kind::f16): D F32 (bits 4-5 = 1), A BF16 (7-9 = 1),
// B BF16 (10-12 = 1), A and B K-major (bits 15, 16 = 0; 1: MN-major), N >> 3 at
// 17-22, M >> 4 at 24-28.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start >> 4 (bits 0-13), LBO >> 4 (16-29),
// SBO >> 4 (32-45), descriptor version 1 (46-47), no swizzle (61-63 = 0).
template <bool kMN>
__device__ __forceinline__ uint64_t smem_desc(uint32_t a) {
  constexpr uint32_t lbo = kMN ? kSBO : kLBO, sbo = kMN ? kLBO : kSBO;
  return (uint64_t)((a & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}

// D[128 x 128] = A[128 x 128] B[128 x 128]^T over K = 128 (8 instructions);
// kA, kB: the operand's image is read MN-major.
template <bool kA, bool kB>
__device__ __forceinline__ void mma_128(uint32_t tmem_d, uint32_t a, uint32_t b) {
  constexpr uint32_t idesc = kIdesc | (kA ? 1u << 15 : 0u) | (kB ? 1u << 16 : 0u);
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const uint64_t da = smem_desc<kA>(a + s * (kA ? 2 * kSBO : 2 * kLBO));
    const uint64_t db = smem_desc<kB>(b + s * (kB ? 2 * kSBO : 2 * kLBO));
    const uint32_t acc = (s > 0) ? 1u : 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
  }
}
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy shared-memory writes -> visible to the tensor core (async proxy)
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t mbar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Bounded wait on the phase with the given parity (about two seconds of SM clock).
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P;\n\tmbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > 4000000000ll) return false;
  }
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// 16 consecutive FP32 columns of this thread's TMEM lane (load + wait in one statement).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ------------------------------------------------------------------ activation
// Sigmoids of a pair by the library's exp and an IEEE division (training, whose
// activations and BF16 roundings do not move), and silu = z times the sigmoid.
__device__ __forceinline__ float2 sigm2(float2 z) {
  return make_float2(1.0f / (1.0f + expf(-z.x)), 1.0f / (1.0f + expf(-z.y)));
}
// silu of a pair for inference: one exponential each (ex2.approx of the FP32
// product, 2 ulp) and one reciprocal for the two, 1 / a = b / (a b).  The
// exponential is bounded at 2^90, so that a sigmoid is at least 8e-28 and silu
// within 1e-7 of 0 down to z = -1e20; where a b overflows, the reciprocal and
// both sigmoids are 0, the larger of them no more than 2^-38 before.  (Bounding z
// itself, exact to -inf, costs 3 %: the pairs of values are packed again.)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <bool kFast>
__device__ __forceinline__ float2 silu2(float2 z) {
  if constexpr (!kFast) return __fmul2_rn(z, sigm2(z));
  const float2 t = __fmul2_rn(z, make_float2(-1.44269504f, -1.44269504f));
  const float a = 1.0f + ex2(fminf(t.x, 90.0f)), b = 1.0f + ex2(fminf(t.y, 90.0f));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a * b));
  return __fmul2_rn(z, __fmul2_rn(make_float2(r, r), make_float2(b, a)));
}
// silu' = s (1 + z (1 - s))
__device__ __forceinline__ float2 dsilu2(float2 z, float2 s) {
  const float2 one = make_float2(1.0f, 1.0f);
  return __fmul2_rn(s, __ffma2_rn(z, __ffma2_rn(s, make_float2(-1.0f, -1.0f), one), one));
}
__device__ __forceinline__ uint32_t pack_bf16(float2 v) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(v.x, v.y);
  return *reinterpret_cast<const uint32_t *>(&b);
}

__device__ __forceinline__ void features(const Norm &nm, const float *xr, float f[4]) {
  const float g[4] = {rsqrtf(xr[0]), xr[1], cosf(xr[2]), xr[3]};
#pragma unroll
  for (int k = 0; k < 4; ++k) f[k] = (g[k] - nm.in_shift[k]) * nm.in_scale[k];
}

// Layer 1 of outputs 2p, 2p + 1, from their weights and biases as pairs: w[0] =
// (W[k = 0] of the two, W[1]), w[1] = (W[2], W[3]), w[2] = (bias, -).
__device__ __forceinline__ float2 layer1_pair(const float4 *w, const float f[4]) {
  const float4 u = w[0], v = w[1], c = w[2];
  float2 z = make_float2(c.x, c.y);
  z = __ffma2_rn(make_float2(u.x, u.y), make_float2(f[0], f[0]), z);
  z = __ffma2_rn(make_float2(u.z, u.w), make_float2(f[1], f[1]), z);
  z = __ffma2_rn(make_float2(v.x, v.y), make_float2(f[2], f[2]), z);
  return __ffma2_rn(make_float2(v.z, v.w), make_float2(f[3], f[3]), z);
}
// The small layers in the form the threads read them (all threads of the CTA).
struct SmallLayers {
  float4 w1[kHid / 2][3];  // layer1_pair
  float4 w4[kHid];         // W4[0..2][o], b3[o]
  float b2[kHid];
  float b4[4];
};
__device__ __forceinline__ void load_small(SmallLayers &L, const DeviceModel &md) {
  float *w1 = reinterpret_cast<float *>(L.w1), *w4 = reinterpret_cast<float *>(L.w4);
  for (int i = threadIdx.x; i < kHid / 2 * 12; i += blockDim.x) {
    const int p = i / 12, c = i % 12, o = 2 * p + (c & 1), k = c >> 1;
    w1[i] = (k < 4) ? md.wq[kOffW1 + kIn * o + k] : (k == 4) ? md.w[kOffB1 + o] : 0.f;
  }
  for (int i = threadIdx.x; i < kHid * 4; i += blockDim.x)
    w4[i] = ((i & 3) < 3) ? md.wq[kOffW4 + (i & 3) * kHid + (i >> 2)] : md.w[kOffB3 + (i >> 2)];
  for (int i = threadIdx.x; i < kHid; i += blockDim.x) L.b2[i] = md.w[kOffB2 + i];
  if (threadIdx.x < 4) L.b4[threadIdx.x] = (threadIdx.x < kOut) ? md.w[kOffB4 + threadIdx.x] : 0.f;
}

// store 8 BF16 (packed in q[4]) at row r, columns k0 .. k0 + 7 of an image
__device__ __forceinline__ void put_row8(uint16_t *img, int r, int k0, const uint32_t q[4]) {
  *reinterpret_cast<uint4 *>(img + canon(r, k0)) = make_uint4(q[0], q[1], q[2], q[3]);
}

__device__ __forceinline__ void copy_img(uint16_t *dst, const uint16_t *src, int images) {
  const uint4 *s = reinterpret_cast<const uint4 *>(src);
  uint4 *d = reinterpret_cast<uint4 *>(dst);
#pragma unroll 8
  for (int i = threadIdx.x; i < images * kImgElems / 8; i += kThreads) d[i] = s[i];
}

// Barrier of one group of 128 threads (named barrier 1 + group).
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

// One thread (of the group, or of the CTA: group -1) waits for the MMA phase; all of them learn the outcome.
__device__ __forceinline__ bool wait_mma(uint32_t mbar, uint32_t parity, volatile int *flag, int *err, int group) {
  const bool first = (group < 0) ? threadIdx.x == 0 : (threadIdx.x & 127) == 0;
  if (first && !mbar_wait(mbar, parity)) {
    *flag = 1;
    atomicExch(err, 1);
  }
  if (group < 0) __syncthreads();
  else group_sync(group);
  return *flag == 0;
}

// ------------------------------------------------------------------ publish
__device__ __forceinline__ bool is_weight(int p) {
  return p < kOffB1 || (p >= kOffW2 && p < kOffB2) || (p >= kOffW3 && p < kOffB3) || (p >= kOffW4 && p < kOffB4);
}
__device__ __forceinline__ void publish_one(const DeviceModel &md, int p, float w) {
  md.wq[p] = is_weight(p) ? bf16_round(w) : w;
  if (p >= kOffW2 && p < kOffB2) {
    const int q = p - kOffW2, o = q >> 7, i = q & 127;
    const uint16_t b = (uint16_t)bf16_bits(w);
    md.img[canon(o, i)] = b;
  } else if (p >= kOffW3 && p < kOffB3) {
    const int q = p - kOffW3, o = q >> 7, i = q & 127;
    const uint16_t b = (uint16_t)bf16_bits(w);
    md.img[kImgElems + canon(o, i)] = b;
  }
}

__global__ void k_publish(DeviceModel md) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < kParams) publish_one(md, p, md.w[p]);
}

__global__ void k_reduce_adam(DeviceModel md, int ntiles, float lr, float beta1, float beta2, float eps, float bc1,
                              float bc2, float *grad) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kParams) return;
  float g = 0.0f;
#pragma unroll 32  // the loads of a batch's tiles in flight together, added in order
  for (int t = 0; t < ntiles; ++t) g += md.partial[(int64_t)t * kPartStride + p];
  if (grad) grad[p] = g;
  if (lr > 0.0f) {
    const float m = beta1 * md.m[p] + (1.0f - beta1) * g;
    const float v = beta2 * md.v[p] + (1.0f - beta2) * g * g;
    md.m[p] = m;
    md.v[p] = v;
    const float w = md.w[p] - lr * (m / bc1) / (sqrtf(v / bc2) + eps);
    md.w[p] = w;
    publish_one(md, p, w);
  }
}

// ------------------------------------------------------------------ inference
struct FwdSmem {
  uint16_t A[kGroups][kImgElems];  // activations of each group's tile, K-major
  uint16_t W[2][kImgElems];        // W2, W3 images (B operands: N = out, K = in)
  SmallLayers L;
  unsigned long long mbar[kGroups];
  uint32_t tmem_slot;
  int flag[kGroups];
};

// The activations cost two special-function operations a value with the
// library's exp and division beside them; with silu2 they cost one and a half,
// and sixteen warps an SM on four tiles keep that pipe busy while a tile waits
// for its product.  Bound by that pipe (69 % of its rate): 1e6 points 1027 us on
// 128-thread CTAs, two an SM, 199 us here.
__global__ void __launch_bounds__(kThreads, 1) k_forward(DeviceModel md, const float *__restrict__ x,
                                                         float *__restrict__ y, int64_t n) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  FwdSmem &S = *reinterpret_cast<FwdSmem *>(smem_raw);
  const int group = threadIdx.x >> 7, t = threadIdx.x & 127, warp = (threadIdx.x >> 5) & 3;
  copy_img(S.W[0], md.img, 2);
  load_small(S.L, md);
  const uint32_t mbar = saddr(&S.mbar[group]);
  if (t == 0) {
    mbar_init(mbar);
    S.flag[group] = 0;
  }
  if (threadIdx.x < 32) tmem_alloc(saddr(&S.tmem_slot), kGroups * 128);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem_slot + 128 * group;
  const uint32_t lane = tmem + ((uint32_t)(warp * 32) << 16);
  uint16_t *A = S.A[group];
  const Norm nm = md.norm;
  uint32_t phase = 0;
  bool ok = true;
  const int64_t ntiles = (n + kTileRows - 1) / kTileRows;
  // a tile to every CTA before a second one to any
  for (int64_t g = blockIdx.x + (int64_t)gridDim.x * group; g < ntiles && ok; g += (int64_t)gridDim.x * kGroups) {
    const int64_t row = g * kTileRows + t;
    const bool valid = row < n;
    float f[4] = {0.f, 0.f, 0.f, 0.f};
    if (valid) features(nm, x + 4 * row, f);
    // layer 1 (FP32 pipe) -> A
#pragma unroll 2
    for (int c = 0; c < 16; ++c) {
      uint32_t q[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) q[j] = pack_bf16(silu2<true>(layer1_pair(S.L.w1[4 * c + j], f)));
      put_row8(A, t, 8 * c, q);
    }
    fence_async_smem();
    tc_fence_before();
    group_sync(group);
    if (t == 0) {
      tc_fence_after();
      mma_128<false, false>(tmem, saddr(A), saddr(S.W[0]));
      mma_commit(mbar);
    }
    if (!(ok = wait_mma(mbar, phase, &S.flag[group], md.error, group))) break;
    phase ^= 1;
    tc_fence_after();
    // layer 2 epilogue -> A
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
      float v[16];
      tmem_ld16(lane + 16 * c, v);
      const float4 *b4 = reinterpret_cast<const float4 *>(S.L.b2 + 16 * c);
      uint32_t q[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 b = b4[j];
        q[2 * j] = pack_bf16(silu2<true>(__fadd2_rn(make_float2(v[4 * j], v[4 * j + 1]), make_float2(b.x, b.y))));
        q[2 * j + 1] = pack_bf16(silu2<true>(__fadd2_rn(make_float2(v[4 * j + 2], v[4 * j + 3]), make_float2(b.z, b.w))));
      }
      put_row8(A, t, 16 * c, q);
      put_row8(A, t, 16 * c + 8, q + 4);
    }
    fence_async_smem();
    tc_fence_before();
    group_sync(group);
    if (t == 0) {
      tc_fence_after();
      mma_128<false, false>(tmem, saddr(A), saddr(S.W[1]));
      mma_commit(mbar);
    }
    if (!(ok = wait_mma(mbar, phase, &S.flag[group], md.error, group))) break;
    phase ^= 1;
    tc_fence_after();
    // layer 3 epilogue + output layer (FP32 pipe)
    float2 acc01 = make_float2(S.L.b4[0], S.L.b4[1]);
    float acc2 = S.L.b4[2];
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
      float v[16];
      tmem_ld16(lane + 16 * c, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 u = S.L.w4[16 * c + 2 * j], w = S.L.w4[16 * c + 2 * j + 1];
        const float2 a = silu2<true>(__fadd2_rn(make_float2(v[2 * j], v[2 * j + 1]), make_float2(u.w, w.w)));
        const uint32_t q = pack_bf16(a);
        const float a0 = __uint_as_float(q << 16), a1 = __uint_as_float(q & 0xFFFF0000u);
        acc01 = __ffma2_rn(make_float2(u.x, u.y), make_float2(a0, a0), acc01);
        acc2 = fmaf(u.z, a0, acc2);
        acc01 = __ffma2_rn(make_float2(w.x, w.y), make_float2(a1, a1), acc01);
        acc2 = fmaf(w.z, a1, acc2);
      }
    }
    if (valid) {
      y[3 * row] = acc01.x * nm.out_scale[0] + nm.out_shift[0];
      y[3 * row + 1] = acc01.y * nm.out_scale[1] + nm.out_shift[1];
      y[3 * row + 2] = acc2 * nm.out_scale[2] + nm.out_shift[2];
    }
    tc_fence_before();  // this tile's reads of the accumulators, before the next tile's product overwrites them
  }
  if (!ok && t == 0) mbar_wait(mbar, phase);  // let an MMA still in flight drain (bounded)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32) tmem_free(S.tmem_slot, kGroups * 128);
}

// ------------------------------------------------------------------ training
constexpr int kScrStride = kTileRows + 1;  // FP32 dz1 scratch, [out][row], padded against bank conflicts
struct TrainSmem {
  uint16_t D[kImgElems];     // dz3, then dz2 [row][out]
  uint16_t W[2][kImgElems];  // W2, W3
  uint16_t X1[kImgElems];    // a1 [row][in]; with X2 and A3 at the end the FP32 scratch for dz1
  uint16_t X2[kImgElems];    // a2
  uint16_t A3[kImgElems];    // a3
  SmallLayers L;
  float f[kTileRows][4];
  float dy[kTileRows][4];
  float part[kGroups][kTileRows][4];  // output layer, partial over a column quarter; then partial sums of the gradients
  float red[4];
  unsigned long long mbar;
  uint32_t tmem_slot;
  int flag;
};
static_assert(3 * kImgElems * 2 >= kHid * kScrStride * 4, "dz1 fits in three images");

// Sum over a quarter of the tile's rows (32 quarter .. ) of column o of an image.
__device__ __forceinline__ float sum_col_quarter(const uint16_t *img, int o, int quarter) {
  float s = 0.f;
#pragma unroll 8
  for (int b = 32 * quarter; b < 32 * quarter + 32; ++b) s += bf16_val(img[canon(b, o)]);
  return s;
}

// One CTA a tile, thread (row t, column quarter): 64 tiles of a minibatch of
// 8192 leave most of the chip idle, so what counts is the serial length of a
// tile.  A quarter of the columns a thread, the operand images read both ways
// by the products (no transposed copies), conflict-free scratch.  Bound by the
// latency of its eight barriers and five products: the 64 tiles 126 us on
// 128-thread CTAs, 34 us here.
__global__ void __launch_bounds__(kThreads, 1) k_gradients(DeviceModel md, const float *__restrict__ x,
                                                           const float *__restrict__ yt,
                                                           const int32_t *__restrict__ perm, int64_t n,
                                                           float inv_count) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  TrainSmem &S = *reinterpret_cast<TrainSmem *>(smem_raw);
  const int cg = threadIdx.x >> 7, t = threadIdx.x & 127, warp = (threadIdx.x >> 5) & 3;
  const int o0 = 32 * cg;  // this thread's columns
  const int64_t g = blockIdx.x;
  const int64_t row = g * kTileRows + t;
  const bool valid = row < n;
  const int64_t idx = valid ? (perm ? (int64_t)perm[row] : row) : 0;
  float *part = md.partial + g * kPartStride;
  const Norm nm = md.norm;

  copy_img(S.W[0], md.img, 2);
  load_small(S.L, md);
  const uint32_t mbar = saddr(&S.mbar);
  if (threadIdx.x == 0) {
    mbar_init(mbar);
    S.flag = 0;
  }
  if (threadIdx.x < 32) tmem_alloc(saddr(&S.tmem_slot), 512);
  float f[4] = {0.f, 0.f, 0.f, 0.f};
  if (valid) features(nm, x + 4 * idx, f);
  if (cg == 0)
    for (int k = 0; k < 4; ++k) S.f[t][k] = f[k];
  __syncthreads();  // the small layers staged
  const float on = valid ? 1.f : 0.f;  // rows past the batch contribute nothing
  const float2 on2 = make_float2(on, on);
  // layer 1 -> X1
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      q[j] = valid ? pack_bf16(silu2<false>(layer1_pair(S.L.w1[o0 / 2 + 4 * c + j], f))) : 0u;
    put_row8(S.X1, t, o0 + 8 * c, q);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem_slot;
  const uint32_t T0 = tmem, T1 = tmem + 128, T2 = tmem + 256, T3 = tmem + 384;
  const uint32_t lane = ((uint32_t)(warp * 32) << 16) + (uint32_t)o0;
  uint32_t phase = 0;
  bool ok = true;
  do {
    // ---- forward: z2 = a1 W2^T -> T0
    if (threadIdx.x == 0) {
      mma_128<false, false>(T0, saddr(S.X1), saddr(S.W[0]));
      mma_commit(mbar);
    }
    if (!(ok = wait_mma(mbar, phase, &S.flag, md.error, -1))) break;
    phase ^= 1;
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float v[16];
      tmem_ld16(T0 + lane + 16 * c, v);
      uint32_t q[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int o = o0 + 16 * c + 2 * j;
        const float2 z = __fadd2_rn(make_float2(v[2 * j], v[2 * j + 1]), make_float2(S.L.b2[o], S.L.b2[o + 1]));
        q[j] = valid ? pack_bf16(silu2<false>(z)) : 0u;
      }
      put_row8(S.X2, t, o0 + 16 * c, q);
      put_row8(S.X2, t, o0 + 16 * c + 8, q + 4);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    // ---- forward: z3 = a2 W3^T -> T1
    if (threadIdx.x == 0) {
      tc_fence_after();
      mma_128<false, false>(T1, saddr(S.X2), saddr(S.W[1]));
      mma_commit(mbar);
    }
    if (!(ok = wait_mma(mbar, phase, &S.flag, md.error, -1))) break;
    phase ^= 1;
    tc_fence_after();
    // ---- output layer over this thread's columns; a3 kept, silu' in registers
    float2 ds[16];
    {
      float2 acc01 = make_float2(0.f, 0.f);
      float acc2 = 0.f;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float v[16];
        tmem_ld16(T1 + lane + 16 * c, v);
        uint32_t q[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 u = S.L.w4[o0 + 16 * c + 2 * j], w = S.L.w4[o0 + 16 * c + 2 * j + 1];
          const float2 z = __fadd2_rn(make_float2(v[2 * j], v[2 * j + 1]), make_float2(u.w, w.w));
          const float2 sg = sigm2(z);
          ds[8 * c + j] = dsilu2(z, sg);
          q[j] = pack_bf16(__fmul2_rn(z, sg));
          const float a0 = __uint_as_float(q[j] << 16), a1 = __uint_as_float(q[j] & 0xFFFF0000u);
          acc01 = __ffma2_rn(make_float2(u.x, u.y), make_float2(a0, a0), acc01);
          acc2 = fmaf(u.z, a0, acc2);
          acc01 = __ffma2_rn(make_float2(w.x, w.y), make_float2(a1, a1), acc01);
          acc2 = fmaf(w.z, a1, acc2);
        }
        put_row8(S.A3, t, o0 + 16 * c, q);
        put_row8(S.A3, t, o0 + 16 * c + 8, q + 4);
      }
      S.part[cg][t][0] = acc01.x;
      S.part[cg][t][1] = acc01.y;
      S.part[cg][t][2] = acc2;
    }
    __syncthreads();
    // ---- loss, dy
    float dy[3], l = 0.f;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float a = S.L.b4[j] + ((S.part[0][t][j] + S.part[1][t][j]) + (S.part[2][t][j] + S.part[3][t][j]));
      const float d = valid ? a - (yt[3 * idx + j] - nm.out_shift[j]) / nm.out_scale[j] : 0.f;
      l += d * d;
      dy[j] = 2.0f * d * inv_count;
      if (cg == 0) S.dy[t][j] = dy[j];
    }
    if (cg == 0) {
      for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
      if ((t & 31) == 0) S.red[warp] = l;
    }
    // dz3 = bf16(dy W4 * silu'(z3)) -> D
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t q[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 u = S.L.w4[o0 + 8 * c + 2 * j], w = S.L.w4[o0 + 8 * c + 2 * j + 1];
        const float2 da = make_float2(dy[0] * u.x + dy[1] * u.y + dy[2] * u.z, dy[0] * w.x + dy[1] * w.y + dy[2] * w.z);
        q[j] = valid ? pack_bf16(__fmul2_rn(da, ds[4 * c + j])) : 0u;
      }
      put_row8(S.D, t, o0 + 8 * c, q);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    // ---- dW3 = dz3^T a2 -> T2 ; da2 = dz3 W3 -> T3
    if (threadIdx.x == 0) {
      tc_fence_after();
      mma_128<true, true>(T2, saddr(S.D), saddr(S.X2));
      mma_128<false, true>(T3, saddr(S.D), saddr(S.W[1]));
      mma_commit(mbar);
      md.loss_part[g] = (S.red[0] + S.red[1]) + (S.red[2] + S.red[3]);
    }
    // meanwhile: output-layer gradients and db3 (column t, a quarter of the rows a thread)
    {
      float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll 8
      for (int b = 32 * cg; b < 32 * cg + 32; ++b) {
        const float a = bf16_val(S.A3[canon(b, t)]);
        s0 += S.dy[b][0] * a;
        s1 += S.dy[b][1] * a;
        s2 += S.dy[b][2] * a;
      }
      float *p = S.part[cg][t];
      p[0] = s0;
      p[1] = s1;
      p[2] = s2;
      p[3] = sum_col_quarter(S.D, t, cg);
    }
    if (!(ok = wait_mma(mbar, phase, &S.flag, md.error, -1))) break;
    phase ^= 1;
    tc_fence_after();
    {  // thread (t, cg) writes sum cg of column t: dW4 rows 0-2, db3
      const float s = (S.part[0][t][cg] + S.part[1][t][cg]) + (S.part[2][t][cg] + S.part[3][t][cg]);
      part[cg < 3 ? kOffW4 + cg * kHid + t : kOffB3 + t] = s;
    }
    if (threadIdx.x < kOut) {
      float s = 0.f;
      for (int b = 0; b < kTileRows; ++b) s += S.dy[b][threadIdx.x];
      part[kOffB4 + threadIdx.x] = s;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {  // dW3 row t
      float v[16];
      tmem_ld16(T2 + lane + 16 * c, v);
      float4 *dst = reinterpret_cast<float4 *>(part + kOffW3 + t * kHid + o0 + 16 * c);
      for (int j = 0; j < 4; ++j) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    // dz2 = bf16(da2 * silu'(z2)) -> D
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float da[16], z[16];
      tmem_ld16(T3 + lane + 16 * c, da);
      tmem_ld16(T0 + lane + 16 * c, z);
      uint32_t q[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int o = o0 + 16 * c + 2 * j;
        const float2 zz = __fadd2_rn(make_float2(z[2 * j], z[2 * j + 1]), make_float2(S.L.b2[o], S.L.b2[o + 1]));
        q[j] = valid ? pack_bf16(__fmul2_rn(make_float2(da[2 * j], da[2 * j + 1]), dsilu2(zz, sigm2(zz)))) : 0u;
      }
      put_row8(S.D, t, o0 + 16 * c, q);
      put_row8(S.D, t, o0 + 16 * c + 8, q + 4);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    // ---- dW2 = dz2^T a1 -> T2 ; da1 = dz2 W2 -> T3
    if (threadIdx.x == 0) {
      tc_fence_after();
      mma_128<true, true>(T2, saddr(S.D), saddr(S.X1));
      mma_128<false, true>(T3, saddr(S.D), saddr(S.W[0]));
      mma_commit(mbar);
    }
    S.part[cg][t][0] = sum_col_quarter(S.D, t, cg);
    if (!(ok = wait_mma(mbar, phase, &S.flag, md.error, -1))) break;
    phase ^= 1;
    tc_fence_after();
    if (cg == 0) part[kOffB2 + t] = (S.part[0][t][0] + S.part[1][t][0]) + (S.part[2][t][0] + S.part[3][t][0]);
#pragma unroll
    for (int c = 0; c < 2; ++c) {  // dW2 row t
      float v[16];
      tmem_ld16(T2 + lane + 16 * c, v);
      float4 *dst = reinterpret_cast<float4 *>(part + kOffW2 + t * kHid + o0 + 16 * c);
      for (int j = 0; j < 4; ++j) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    // dz1 = da1 * silu'(z1) in FP32 -> scratch [out][row] (X1, X2, A3: their last readers are done)
    float *scr = reinterpret_cast<float *>(S.X1);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float v[16];
      tmem_ld16(T3 + lane + 16 * c, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int o = o0 + 16 * c + 2 * j;
        const float2 z = layer1_pair(S.L.w1[o / 2], f);
        const float2 d = __fmul2_rn(__fmul2_rn(make_float2(v[2 * j], v[2 * j + 1]), dsilu2(z, sigm2(z))), on2);
        scr[o * kScrStride + t] = d.x;
        scr[(o + 1) * kScrStride + t] = d.y;
      }
    }
    __syncthreads();
    // column t over a quarter of the rows, then the four quarters (thread (t, cg): input cg; cg = 0 the bias too)
    float s[4] = {0.f, 0.f, 0.f, 0.f}, sb = 0.f;
#pragma unroll 8
    for (int b = 32 * cg; b < 32 * cg + 32; ++b) {
      const float d = scr[t * kScrStride + b];
      sb += d;
      for (int k = 0; k < 4; ++k) s[k] += d * S.f[b][k];
    }
    float *p = S.part[cg][t];
    for (int k = 0; k < 4; ++k) p[k] = s[k];
    __syncthreads();  // the scratch is read: its first words take the bias sums
    scr[cg * kTileRows + t] = sb;
    part[kOffW1 + 4 * t + cg] = (S.part[0][t][cg] + S.part[1][t][cg]) + (S.part[2][t][cg] + S.part[3][t][cg]);
    __syncthreads();
    if (cg == 0)
      part[kOffB1 + t] = (scr[t] + scr[kTileRows + t]) + (scr[2 * kTileRows + t] + scr[3 * kTileRows + t]);
  } while (false);
  if (!ok && threadIdx.x == 0) mbar_wait(mbar, phase);  // let an MMA still in flight drain (bounded)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32) tmem_free(tmem, 512);
}

}  // namespace

void launch_publish(const DeviceModel &md, cudaStream_t st) {
  k_publish<<<(kParams + 255) / 256, 256, 0, st>>>(md);
}

void launch_forward(const DeviceModel &md, const float *x, float *y, int64_t n, int num_sms, cudaStream_t st) {
  if (n <= 0) return;
  const int smem = (int)sizeof(FwdSmem);
  cudaFuncSetAttribute(k_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const int64_t ntiles = (n + kTileRows - 1) / kTileRows;
  const int grid = (int)std::min<int64_t>(ntiles, (int64_t)num_sms);
  k_forward<<<grid, kThreads, smem, st>>>(md, x, y, n);
}

void launch_gradients(const DeviceModel &md, const float *x, const float *y_true, const int32_t *perm, int64_t n,
                      cudaStream_t st) {
  if (n <= 0 || n > kMaxTrainRows) return;
  const int smem = (int)sizeof(TrainSmem);
  cudaFuncSetAttribute(k_gradients, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const int ntiles = (int)((n + kTileRows - 1) / kTileRows);
  k_gradients<<<ntiles, kThreads, smem, st>>>(md, x, y_true, perm, n, 1.0f / (3.0f * (float)n));
}

void launch_reduce_adam(const DeviceModel &md, int ntiles, float lr, float beta1, float beta2, float eps, float bc1,
                        float bc2, float *grad, cudaStream_t st) {
  k_reduce_adam<<<(kParams + 255) / 256, 256, 0, st>>>(md, ntiles, lr, beta1, beta2, eps, bc1, bc2, grad);
}

}  // namespace mlp
}  // namespace aak
