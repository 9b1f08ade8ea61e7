// Surrogate return-map MLP (extension; the reference has no plasticity):
// 7 inputs -> 64 -> 64 -> 4 outputs, SiLU after the hidden layers, bf16
// weights and activations with f32 accumulation on the sm_100a tensor cores
// (tcgen05.mma, accumulators in tensor memory).
//
// Parameters are kept in f32 (the trainer's master copy) and packed into bf16
// tensor-core operand tiles after every change.  A CTA of 256 threads handles
// 128 samples per tile: warps w and w + 4 read rows 32 (w % 4) .. + 31 (TMEM
// lanes) back with tcgen05.ld, each one half of a hidden layer's columns.
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/agimp.h"
#include "common.cuh"
#include "umma.cuh"

namespace agimp {
namespace mlp {

constexpr int IN = 7, H = 64, OUT = 4;
constexpr int K1 = 16;  // input width padded to one MMA K step
constexpr int N3 = 16;  // output width padded to the smallest MMA N
constexpr int OW1 = 0, OB1 = OW1 + IN * H, OW2 = OB1 + H, OB2 = OW2 + H * H, OW3 = OB2 + H, OB3 = OW3 + H * OUT;
constexpr int NPARAM = OB3 + OUT;  // 4932
// packed bf16 operand tiles (K-major): forward B1 [64][16], B2 [64][64], B3 [16][64]
// (row = output unit), backward B3T [64][16] (row = hidden unit of layer 2,
// K = outputs) and B2T [64][64] (row = hidden unit of layer 1, K = layer-2 units)
constexpr int PB1 = 0, PB2 = PB1 + H * K1, PB3 = PB2 + H * H, NPACK_FWD = PB3 + N3 * H;  // 6144
constexpr int PB3T = NPACK_FWD, PB2T = PB3T + H * K1, NPACK = PB2T + H * H;           // 11264
constexpr int TILE = 128;

constexpr int THREADS = 256;

// Eight SiLU values z / (1 + exp(-z)) or, with `deriv`, SiLU derivatives.
//
// The activations are bound by the special-function unit (an exponential and a
// reciprocal each, 16 a cycle and SM) and by the instructions around it.  For
// |z| < 40 two of them share one reciprocal, 1 / d0 = d1 (1 / (d0 d1)), and the
// quotients are those of a rounded division all the same (but for less than one
// operand in 2^20, whose last bit differs): a Newton step on the
// reciprocal, then the quotient corrected by its remainder in fused
// multiply-adds (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990), two at a time.
// Other z, infinities and NaN take the plain expressions.
template <bool deriv>
__device__ __forceinline__ void silu8(const float* z, float* a) {
  bool near = true;
#pragma unroll
  for (int j = 0; j < 8; ++j) near = near && fabsf(z[j]) < 40.f;
  if (near) {
    const f2 one = f2_dup(1.f), log2e = f2_dup(-1.4426950408889634f);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const f2 zz = f2_make(z[j], z[j + 1]);
      float2 e = f2_get(f2_mul(zz, log2e));
      asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e.x));
      asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e.y));
      const f2 dd = f2_add(one, pk2(e));
      const float2 d = f2_get(dd);
      float r;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d.x * d.y));
      const f2 nd = f2_mul(dd, f2_dup(-1.f)), y0 = f2_mul(f2_dup(r), f2_make(d.y, d.x));
      const f2 y = f2_fma(y0, f2_fma(nd, y0, one), y0);
      const f2 num = deriv ? one : zz, q0 = f2_mul(num, y);
      const float2 q = f2_get(f2_fma(f2_fma(nd, q0, num), y, q0));
      a[j] = q.x;
      a[j + 1] = q.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = (deriv ? 1.f : z[j]) / (1.f + __expf(-z[j]));
  }
  if (deriv)
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = a[j] * (1.f + z[j] * (1.f - a[j]));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *(const uint32_t*)&v;
}

// eight consecutive columns of a tile row (one core-matrix row, 16 bytes)
__device__ __forceinline__ void store8(__nv_bfloat16* at, const float* v) {
  *(uint4*)at = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}

// 16-byte copies of n operand elements from global to shared memory
__device__ __forceinline__ void copy_tiles(void* dst, const __nv_bfloat16* src, int n) {
  for (int i = threadIdx.x; i < n / 8; i += THREADS) ((uint4*)dst)[i] = ((const uint4*)src)[i];
}

__global__ void k_pack(const float* __restrict__ P, __nv_bfloat16* __restrict__ packed) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NPACK; i += gridDim.x * blockDim.x) {
    float v;
    int dst;
    if (i < PB2) {
      const int n = i / K1, k = i % K1;
      v = k < IN ? P[OW1 + k * H + n] : 0.f;
      dst = PB1 + umma::tile_off(n, k, K1);
    } else if (i < PB3) {
      const int j = i - PB2, n = j / H, k = j % H;
      v = P[OW2 + k * H + n];
      dst = PB2 + umma::tile_off(n, k, H);
    } else if (i < PB3T) {
      const int j = i - PB3, n = j / H, k = j % H;
      v = n < OUT ? P[OW3 + k * OUT + n] : 0.f;
      dst = PB3 + umma::tile_off(n, k, H);
    } else if (i < PB2T) {
      const int j = i - PB3T, n = j / K1, k = j % K1;  // (n, k) = W3[n][k]
      v = k < OUT ? P[OW3 + n * OUT + k] : 0.f;
      dst = PB3T + umma::tile_off(n, k, K1);
    } else {
      const int j = i - PB2T, n = j / H, k = j % H;  // (n, k) = W2[n][k]
      v = P[OW2 + n * H + k];
      dst = PB2T + umma::tile_off(n, k, H);
    }
    packed[dst] = __float2bfloat16_rn(v);
  }
}

// shared-memory layout of the forward kernel (bytes)
struct FwdSmem {
  static constexpr int B1 = 0;
  static constexpr int B2 = B1 + 2 * H * K1;
  static constexpr int B3 = B2 + 2 * H * H;
  static constexpr int X = B3 + 2 * N3 * H;         // [128][16]
  static constexpr int A = X + 2 * TILE * K1;       // [128][64]: both hidden layers in turn
  static constexpr int BIAS = A + 2 * TILE * H;     // b1[64] b2[64] b3[4]
  static constexpr int MBAR = BIAS + 4 * (H + H + OUT);
  static constexpr int TSLOT = MBAR + 8;
  static constexpr int BYTES = TSLOT + 16;
};

// one hidden layer's epilogue: this thread's 32 columns of its row from TMEM,
// bias, SiLU, bf16, into the next layer's operand tile (column groups `groups`
// apart per 8 rows)
__device__ __forceinline__ void hidden_epilogue(uint32_t taddr, const float* bias, __nv_bfloat16* tile, int row, int col,
                                                int width, float* z) {
  umma::tmem_ld32(taddr, z);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) z[8 * g + j] += bias[col + 8 * g + j];
    silu8<false>(z + 8 * g, a);
    store8(tile + umma::tile_off(row, col + 8 * g, width), a);
  }
}

// Y[n][4] = MLP(X[n][7]) for n < N.
//
// What bounds it: the activations' special-function operations (silu8) and the
// instructions around them, each at half of its rate, and the chain of product,
// wait, epilogue and barrier, which 26 warps an SM overlap in part; the products
// are far too thin to matter (7 percent of the tensor pipe).  2M rows take 173
// us.  The activations are written as packed 16-byte
// core-matrix rows; element by element (2-byte stores with 4-way bank
// conflicts) and with general divisions 2M rows took 357 us.
__global__ void __launch_bounds__(THREADS, 4) k_forward(const float* __restrict__ X, float* __restrict__ Y, long long N,
                                                        const __nv_bfloat16* __restrict__ packed,
                                                        const float* __restrict__ P, int32_t* __restrict__ err,
                                                        const int32_t* __restrict__ n_dev, uint32_t err_bit) {
  if (n_dev) N = min((long long)*n_dev, N);  // device-side sample count, capped by the buffer size
  extern __shared__ __align__(128) unsigned char sm[];
  using S = FwdSmem;
  __nv_bfloat16* sX = (__nv_bfloat16*)(sm + S::X);
  __nv_bfloat16* sA = (__nv_bfloat16*)(sm + S::A);
  float* sb = (float*)(sm + S::BIAS);
  uint64_t* mbar = (uint64_t*)(sm + S::MBAR);
  uint32_t* tslot = (uint32_t*)(sm + S::TSLOT);
  const int tid = threadIdx.x, warp = tid >> 5, row = tid & (TILE - 1), half = tid >> 7, col = 32 * half;
  const long long ntiles = (N + TILE - 1) / TILE;
  // the first tile's samples move while the weights are copied
  float x[8];
  auto load_x = [&](long long tile) {
    const long long r = tile * TILE + row;
#pragma unroll
    for (int k = 0; k < IN; ++k) x[k] = (half == 0 && r < N) ? __ldg(&X[r * IN + k]) : 0.f;
    x[IN] = 0.f;
  };
  load_x(blockIdx.x);
  copy_tiles(sm + S::B1, packed, NPACK_FWD);
  if (tid < H) {
    sb[tid] = P[OB1 + tid];
    sb[H + tid] = P[OB2 + tid];
  }
  if (tid < OUT) sb[2 * H + tid] = P[OB3 + tid];
  if (half == 1) *(uint4*)(sX + umma::tile_off(row, 8, K1)) = make_uint4(0, 0, 0, 0);  // columns 8..15
  if (tid == 0) {
    umma::mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) umma::tmem_alloc(tslot, 64);
  auto sync_for_mma = [&]() {
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
  };
  sync_for_mma();
  const uint32_t tmem = *tslot;
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t aB1 = umma::smem_u32(sm + S::B1), aB2 = umma::smem_u32(sm + S::B2), aB3 = umma::smem_u32(sm + S::B3);
  const uint32_t aX = umma::smem_u32(sX), aA = umma::smem_u32(sA);
  uint32_t phase = 0;
  bool ok = true;
  auto wait_mma = [&]() {
    ok = umma::mbar_wait(mbar, phase) && ok;
    phase ^= 1;
    umma::fence_after_sync();
  };
  // [128 x 64] x [64 x n] from the hidden tile
  auto mma_hidden = [&](uint32_t b, int n) {
#pragma unroll
    for (int kk = 0; kk < H / 16; ++kk)
      umma::mma_bf16(tmem, umma::smem_desc(aA + kk * 256, 128, 8 * 128), umma::smem_desc(b + kk * 256, 128, 8 * 128),
                     umma::idesc_bf16_f32(TILE, n), kk > 0);
    umma::mma_commit(mbar);
  };
  // The three layers' accumulators share the 64 TMEM columns, and the hidden
  // layers one operand tile: each product starts after the barrier that
  // follows the reads of what it overwrites.
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    float z[32];
    if (half == 0) store8(sX + umma::tile_off(row, 0, K1), x);
    sync_for_mma();
    if (tid == 0) {
      umma::mma_bf16(tmem, umma::smem_desc(aX, 128, 2 * 128), umma::smem_desc(aB1, 128, 2 * 128),
                     umma::idesc_bf16_f32(TILE, H), 0);
      umma::mma_commit(mbar);
    }
    if (tile + gridDim.x < ntiles) load_x(tile + gridDim.x);
    wait_mma();
    hidden_epilogue(tmem + lanes + col, sb, sA, row, col, H, z);
    sync_for_mma();
    if (tid == 0) mma_hidden(aB2, H);
    wait_mma();
    hidden_epilogue(tmem + lanes + col, sb + H, sA, row, col, H, z);
    sync_for_mma();
    if (tid == 0) mma_hidden(aB3, N3);
    wait_mma();
    const long long r = tile * TILE + row;
    if (half == 0) {  // warps 0..3
      float y[OUT];
      umma::tmem_ld4(tmem + lanes, y);
#pragma unroll
      for (int j = 0; j < OUT; ++j) y[j] += sb[2 * H + j];
      if (r < N) {
        if (((unsigned long long)Y & 15) == 0)
          *(float4*)(Y + r * OUT) = make_float4(y[0], y[1], y[2], y[3]);
        else
          for (int j = 0; j < OUT; ++j) Y[r * OUT + j] = y[j];
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 64);
  if (!ok && tid == 0) atomicOr((unsigned*)err, err_bit);
}

// ---------------------------------------------------------------------------
// Training: loss and gradient of the mean squared error over n samples.
// Per tile of 128 samples (row = sample = TMEM lane):
//   forward  Z1 = X W1, A1 = silu(Z1 + b1), Z2 = A1 W2, A2 = silu(Z2 + b2),
//            Y = A2 W3 + b3                                  (3 products)
//   backward dY = 2 (Y - T) / n, dA2 = dY W3^T, dZ2 = dA2 silu'(.),
//            dA1 = dZ2 W2^T, dZ1 = dA1 silu'(.)              (2 products)
//   weights  G3 += [A2 1]^T dY, G2 += [A1 1]^T dZ2, G1 += [X 1]^T dZ1
// The weight gradients are products over the samples: they read the same
// tiles as MN-major operands (a column of ones beside the features yields the
// bias gradient; M is 128, and the rows beyond the features and the ones read
// whatever follows in shared memory and are not used).  They accumulate in
// TMEM over all tiles of the CTA, which then adds them to the global gradient
// with atomics.
//
// What bounds it: the chain of six products and epilogues per tile, at two CTAs
// per SM.  The activations stay in registers between forward and backward, and
// no transposed copies are written (before, one CTA of 128 threads per SM wrote
// every activation twice, element by element).  A call over 65,536 rows 124 -> 30 us.
constexpr int HW = H + 8;  // width of the activation tiles: features, ones, zeros
struct TrainSmem {
  static constexpr int B1 = 0;                       // [64][16]
  static constexpr int B2 = B1 + 2 * H * K1;         // [64][64]
  static constexpr int B3 = B2 + 2 * H * H;          // [16][64]
  static constexpr int B3T = B3 + 2 * N3 * H;        // [64][16]
  static constexpr int B2T = B3T + 2 * H * K1;       // [64][64]
  static constexpr int X = B2T + 2 * H * H;          // [128][16]: features, ones, zeros
  static constexpr int DY = X + 2 * TILE * K1;       // [128][16]
  static constexpr int A1 = DY + 2 * TILE * K1;      // [128][72]
  static constexpr int A2 = A1 + 2 * TILE * HW;      // [128][72]
  static constexpr int DZ2 = A2 + 2 * TILE * HW;     // [128][64]
  static constexpr int DZ1 = DZ2 + 2 * TILE * H;     // [128][64]
  static constexpr int BIAS = DZ1 + 2 * TILE * H;    // b1[64] b2[64] b3[4]
  static constexpr int LOSS = BIAS + 4 * (H + H + OUT);
  static constexpr int MBAR = LOSS + 8;
  static constexpr int TSLOT = MBAR + 8;
  static constexpr int BYTES = TSLOT + 16;
};
// TMEM columns: the layers' products in turn, the weight gradients
constexpr int TZ = 0, TG1 = 64, TG2 = 128, TG3 = 192, TCOLS = 256;

__global__ void k_zero(float* __restrict__ grad, float* __restrict__ loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NPARAM) grad[i] = 0.f;
  if (i == 0) *loss = 0.f;
}

// n consecutive floats added to g (16-byte atomics where the address allows)
template <int n>
__device__ __forceinline__ void add_row(float* g, const float* v) {
  if (((unsigned long long)g & 15) == 0) {
#pragma unroll
    for (int j = 0; j < n; j += 4) atomicAdd((float4*)(g + j), make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
  } else {
#pragma unroll
    for (int j = 0; j < n; ++j) atomicAdd(g + j, v[j]);
  }
}

__global__ void __launch_bounds__(THREADS, 2) k_train(const float* __restrict__ Xg, const float* __restrict__ Tg,
                                                      long long N, const __nv_bfloat16* __restrict__ packed,
                                                      const float* __restrict__ P, float* __restrict__ grad,
                                                      float* __restrict__ loss, int32_t* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char sm[];
  using S = TrainSmem;
  __nv_bfloat16* sX = (__nv_bfloat16*)(sm + S::X);
  __nv_bfloat16* sA1 = (__nv_bfloat16*)(sm + S::A1);
  __nv_bfloat16* sA2 = (__nv_bfloat16*)(sm + S::A2);
  __nv_bfloat16* sDY = (__nv_bfloat16*)(sm + S::DY);
  __nv_bfloat16* sDZ2 = (__nv_bfloat16*)(sm + S::DZ2);
  __nv_bfloat16* sDZ1 = (__nv_bfloat16*)(sm + S::DZ1);
  float* sb = (float*)(sm + S::BIAS);
  float* sloss = (float*)(sm + S::LOSS);
  uint64_t* mbar = (uint64_t*)(sm + S::MBAR);
  uint32_t* tslot = (uint32_t*)(sm + S::TSLOT);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = tid & (TILE - 1), half = tid >> 7, col = 32 * half;
  float x[8], t[OUT];
  auto load = [&](long long tile) {
    const long long r = tile * TILE + row;
    const bool live = half == 0 && r < N;
#pragma unroll
    for (int k = 0; k < IN; ++k) x[k] = live ? __ldg(&Xg[r * IN + k]) : 0.f;
    x[IN] = 1.f;
#pragma unroll
    for (int j = 0; j < OUT; ++j) t[j] = live ? __ldg(&Tg[r * OUT + j]) : 0.f;
  };
  load(blockIdx.x);
  copy_tiles(sm + S::B1, packed, NPACK);
  if (tid < H) {
    sb[tid] = P[OB1 + tid];
    sb[H + tid] = P[OB2 + tid];
  }
  if (tid < OUT) sb[2 * H + tid] = P[OB3 + tid];
  // constant parts of the operand tiles: ones and zero padding
  const uint4 zero4 = make_uint4(0, 0, 0, 0), ones = make_uint4(pack_bf16(1.f, 0.f), 0, 0, 0);
  if (half == 0) {
    *(uint4*)(sA1 + umma::tile_off(row, H, HW)) = ones;
    *(uint4*)(sX + umma::tile_off(row, 8, K1)) = zero4;
  } else {
    *(uint4*)(sA2 + umma::tile_off(row, H, HW)) = ones;
    *(uint4*)(sDY + umma::tile_off(row, 8, K1)) = zero4;
  }
  if (tid == 0) {
    *sloss = 0.f;
    umma::mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) umma::tmem_alloc(tslot, TCOLS);
  auto sync_for_mma = [&]() {
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
  };
  sync_for_mma();
  const uint32_t tmem = *tslot;
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  auto addr = [&](int off) { return umma::smem_u32(sm + off); };
  uint32_t phase = 0;
  bool ok = true;
  auto wait_mma = [&]() {
    ok = umma::mbar_wait(mbar, phase) && ok;
    phase ^= 1;
    umma::fence_after_sync();
  };
  // D[TZ, n columns] = A[128][K] (tile of width wa) x B[n][K]
  auto layer = [&](int a, int wa, int b, int K, int n) {
    for (int kk = 0; kk < K / 16; ++kk)
      umma::mma_bf16(tmem + TZ, umma::smem_desc(addr(a) + kk * 256, 128, wa * 16),
                     umma::smem_desc(addr(b) + kk * 256, 128, K * 16), umma::idesc_bf16_f32(TILE, n), kk > 0);
  };
  // D[d, n columns] += A[128][wa]^T B[128][n] over the 128 samples
  auto weight = [&](int d, int a, int wa, int b, int n, bool first) {
    for (int kk = 0; kk < TILE / 16; ++kk)
      umma::mma_bf16(tmem + d, umma::smem_desc(addr(a) + kk * 2 * wa * 16, wa * 16, 128),
                     umma::smem_desc(addr(b) + kk * 2 * n * 16, n * 16, 128), umma::idesc_bf16_f32(TILE, n, true),
                     (!first || kk > 0) ? 1u : 0u);
  };
  // this thread's 32 columns of dA times silu'(z), bf16, into a gradient tile
  auto backward = [&](const float* z, __nv_bfloat16* tile) {
    float d[32];
    umma::tmem_ld32(tmem + TZ + lanes + col, d);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float ds[8];
      silu8<true>(z + 8 * g, ds);
#pragma unroll
      for (int j = 0; j < 8; ++j) d[8 * g + j] *= ds[j];
      store8(tile + umma::tile_off(row, col + 8 * g, H), d + 8 * g);
    }
  };
  float my_loss = 0.f;
  const float inv_n = 1.f / (float)N;
  const long long ntiles = (N + TILE - 1) / TILE;
  bool first = true;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const bool live = tile * TILE + row < N;
    float z1[32], z2[32], tt[OUT];
    if (half == 0) store8(sX + umma::tile_off(row, 0, K1), x);
#pragma unroll
    for (int j = 0; j < OUT; ++j) tt[j] = t[j];
    sync_for_mma();
    if (tid == 0) {
      layer(S::X, K1, S::B1, K1, H);
      umma::mma_commit(mbar);
    }
    if (tile + gridDim.x < ntiles) load(tile + gridDim.x);
    wait_mma();
    hidden_epilogue(tmem + TZ + lanes + col, sb, sA1, row, col, HW, z1);
    sync_for_mma();
    if (tid == 0) {
      layer(S::A1, HW, S::B2, H, H);
      umma::mma_commit(mbar);
    }
    wait_mma();
    hidden_epilogue(tmem + TZ + lanes + col, sb + H, sA2, row, col, HW, z2);
    sync_for_mma();
    if (tid == 0) {
      layer(S::A2, HW, S::B3, H, N3);
      umma::mma_commit(mbar);
    }
    wait_mma();
    if (half == 0) {  // warps 0..3
      float d[8];
      umma::tmem_ld4(tmem + TZ + lanes, d);
#pragma unroll
      for (int j = 0; j < OUT; ++j) {
        const float e = live ? d[j] + sb[2 * H + j] - tt[j] : 0.f;
        my_loss += e * e;
        d[j] = 2.f * e * inv_n;
        d[OUT + j] = 0.f;
      }
      store8(sDY + umma::tile_off(row, 0, K1), d);
    }
    sync_for_mma();
    if (tid == 0) {
      layer(S::DY, K1, S::B3T, K1, H);  // dA2
      weight(TG3, S::A2, HW, S::DY, N3, first);
      umma::mma_commit(mbar);
    }
    wait_mma();
    backward(z2, sDZ2);
    sync_for_mma();
    if (tid == 0) {
      layer(S::DZ2, H, S::B2T, H, H);  // dA1
      weight(TG2, S::A1, HW, S::DZ2, H, first);
      umma::mma_commit(mbar);
    }
    wait_mma();
    backward(z1, sDZ1);
    sync_for_mma();
    if (tid == 0) {
      weight(TG1, S::X, K1, S::DZ1, H, first);
      umma::mma_commit(mbar);
    }
    wait_mma();
    first = false;
  }
  // loss
#pragma unroll
  for (int o = 16; o; o >>= 1) my_loss += __shfl_xor_sync(0xffffffffu, my_loss, o);
  if (lane == 0) atomicAdd(sloss, my_loss);
  // weight gradients: this thread holds 32 columns of row `row` of G1 and G2
  if (!first) {
    float g[32];
    if ((warp & 3) == 0) {
      umma::tmem_ld32(tmem + TG1 + lanes + col, g);
      if (row < IN)
        add_row<32>(&grad[OW1 + row * H + col], g);
      else if (row == IN)
        add_row<32>(&grad[OB1 + col], g);
    }
    if ((warp & 3) < 3) {
      umma::tmem_ld32(tmem + TG2 + lanes + col, g);
      if (row < H)
        add_row<32>(&grad[OW2 + row * H + col], g);
      else if (row == H)
        add_row<32>(&grad[OB2 + col], g);
    }
    if (warp < 3) {
      umma::tmem_ld4(tmem + TG3 + lanes, g);
      if (row < H)
        add_row<OUT>(&grad[OW3 + row * OUT], g);
      else if (row == H)
        add_row<OUT>(&grad[OB3], g);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (tid == 0) atomicAdd(loss, *sloss * inv_n);
  if (warp == 0) umma::tmem_dealloc(tmem, TCOLS);
  if (!ok && tid == 0) atomicOr((unsigned*)err, 1u);
}

// Adam (Kingma & Ba 2015) on the f32 parameters; step >= 1
__global__ void k_adam(float* __restrict__ P, const float* __restrict__ g, float* __restrict__ m1,
                       float* __restrict__ m2, float lr, float b1, float b2, float eps, int step) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NPARAM) return;
  const float gi = g[i];
  const float a = b1 * m1[i] + (1.f - b1) * gi, b = b2 * m2[i] + (1.f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = b;
  const float ah = a / (1.f - powf(b1, (float)step)), bh = b / (1.f - powf(b2, (float)step));
  P[i] -= lr * ah / (sqrtf(bh) + eps);
}

}  // namespace mlp

void launch_mlp_forward_dev(const void* packed, const float* P, const float* X, float* Y, const int32_t* n_dev,
                            long long cap, int32_t* err, int sms, cudaStream_t s) {
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(mlp::k_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, mlp::FwdSmem::BYTES);
    attr = true;
  }
  const long long ntiles = (cap + mlp::TILE - 1) / mlp::TILE;
  const int grid = (int)std::min<long long>(ntiles, (long long)sms * 4);
  mlp::k_forward<<<grid, mlp::THREADS, mlp::FwdSmem::BYTES, s>>>(X, Y, cap, (const __nv_bfloat16*)packed, P, err, n_dev,
                                                             ERR_MLP);
}

// Self-test of the bounded completion wait of the tensor-core kernels
// (umma::mbar_wait): one CTA waits on an mbarrier of one expected arrival.
// With arrive = 1 a thread arrives first and the wait succeeds; with
// arrive = 0 nothing ever arrives, the wait gives up after max_polls polls,
// the kernel records ERR_MLP in *err and returns normally, so the context
// stays usable.  This is how a lost tensor-core completion surfaces.
__global__ void k_wait_selftest(uint32_t* err, uint32_t max_polls, int arrive) {
  __shared__ uint64_t mbar;
  if (threadIdx.x == 0) {
    umma::mbar_init(&mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (arrive && threadIdx.x == 0)
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(&mbar)) : "memory");
  const bool ok = umma::mbar_wait(&mbar, 0, max_polls);
  if (!ok && threadIdx.x == 0) atomicOr(err, ERR_MLP);
}

}  // namespace agimp

using namespace agimp;

struct agimp_mlp {
  int device = 0;
  float* P = nullptr;               // f32 parameters
  __nv_bfloat16* packed = nullptr;  // bf16 operand tiles
  float* grad = nullptr;            // gradient, Adam moments, loss
  float* m1 = nullptr;
  float* m2 = nullptr;
  float* loss = nullptr;
  int step = 0;
  int32_t* err = nullptr;
  int sms = 148;
  std::string msg;
};

namespace agimp {
void mlp_buffers(const agimp_mlp* m, const void** packed, const float** P) {
  *packed = m->packed;
  *P = m->P;
}
}  // namespace agimp

extern "C" {

agimp_status agimp_mlp_create(int32_t device, agimp_mlp** out) {
  if (!out) return AGIMP_INVALID_ARG;
  *out = nullptr;
  if (cudaSetDevice(device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  agimp_mlp* m = new agimp_mlp();
  m->device = device;
  cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device);
  if (cudaMalloc(&m->P, mlp::NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->packed, mlp::NPACK * sizeof(__nv_bfloat16)) != cudaSuccess ||
      cudaMalloc(&m->grad, mlp::NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->m1, mlp::NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->m2, mlp::NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->loss, sizeof(float)) != cudaSuccess || cudaMalloc(&m->err, sizeof(int32_t)) != cudaSuccess) {
    cudaFree(m->P);
    cudaFree(m->packed);
    cudaFree(m->grad);
    cudaFree(m->m1);
    cudaFree(m->m2);
    cudaFree(m->loss);
    cudaFree(m->err);
    delete m;
    return AGIMP_OUT_OF_MEMORY;
  }
  cudaMemset(m->m1, 0, mlp::NPARAM * sizeof(float));
  cudaMemset(m->m2, 0, mlp::NPARAM * sizeof(float));
  cudaMemset(m->P, 0, mlp::NPARAM * sizeof(float));
  cudaMemset(m->packed, 0, mlp::NPACK * sizeof(__nv_bfloat16));
  cudaMemset(m->err, 0, sizeof(int32_t));
  cudaFuncSetAttribute(mlp::k_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, mlp::FwdSmem::BYTES);
  cudaFuncSetAttribute(mlp::k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, mlp::TrainSmem::BYTES);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    delete m;
    return AGIMP_CUDA_ERROR;
  }
  *out = m;
  return AGIMP_OK;
}

agimp_status agimp_mlp_destroy(agimp_mlp* m) {
  if (!m) return AGIMP_INVALID_ARG;
  cudaSetDevice(m->device);
  cudaDeviceSynchronize();
  cudaFree(m->P);
  cudaFree(m->packed);
  cudaFree(m->grad);
  cudaFree(m->m1);
  cudaFree(m->m2);
  cudaFree(m->loss);
  cudaFree(m->err);
  delete m;
  return AGIMP_OK;
}

int32_t agimp_mlp_num_params(void) { return mlp::NPARAM; }

agimp_status agimp_mlp_set_params(agimp_mlp* m, const float* params, int32_t memory, void* stream) {
  if (!m || !params) return AGIMP_INVALID_ARG;
  if (cudaSetDevice(m->device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  cudaStream_t s = (cudaStream_t)stream;
  const cudaMemcpyKind k = memory == AGIMP_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  if (cudaMemcpyAsync(m->P, params, mlp::NPARAM * sizeof(float), k, s) != cudaSuccess) return AGIMP_CUDA_ERROR;
  mlp::k_pack<<<(mlp::NPACK + 255) / 256, 256, 0, s>>>(m->P, m->packed);
  if (memory == AGIMP_MEM_HOST && cudaStreamSynchronize(s) != cudaSuccess) return AGIMP_CUDA_ERROR;
  return cudaGetLastError() == cudaSuccess ? AGIMP_OK : AGIMP_CUDA_ERROR;
}

agimp_status agimp_mlp_get_params(agimp_mlp* m, float* params, int32_t memory, void* stream) {
  if (!m || !params) return AGIMP_INVALID_ARG;
  if (cudaSetDevice(m->device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  cudaStream_t s = (cudaStream_t)stream;
  const cudaMemcpyKind k = memory == AGIMP_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  if (cudaMemcpyAsync(params, m->P, mlp::NPARAM * sizeof(float), k, s) != cudaSuccess) return AGIMP_CUDA_ERROR;
  if (memory == AGIMP_MEM_HOST && cudaStreamSynchronize(s) != cudaSuccess) return AGIMP_CUDA_ERROR;
  return AGIMP_OK;
}

agimp_status agimp_mlp_forward(agimp_mlp* m, const float* X, float* Y, int64_t n, void* stream) {
  if (!m || n < 0 || (n > 0 && (!X || !Y))) return AGIMP_INVALID_ARG;
  if (n == 0) return AGIMP_OK;
  if (cudaSetDevice(m->device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  const long long ntiles = (n + mlp::TILE - 1) / mlp::TILE;
  const int grid = (int)std::min<long long>(ntiles, (long long)m->sms * 4);
  mlp::k_forward<<<grid, mlp::THREADS, mlp::FwdSmem::BYTES, (cudaStream_t)stream>>>(X, Y, n, m->packed, m->P, m->err,
                                                                                 nullptr, 1u);
  return cudaGetLastError() == cudaSuccess ? AGIMP_OK : AGIMP_CUDA_ERROR;
}

// loss and gradient into the given device buffers
static agimp_status mlp_grad(agimp_mlp* m, const float* X, const float* T, int64_t n, float* grad, float* loss,
                             cudaStream_t s) {
  mlp::k_zero<<<(mlp::NPARAM + 255) / 256, 256, 0, s>>>(grad, loss);
  if (n > 0) {
    const long long ntiles = (n + mlp::TILE - 1) / mlp::TILE;
    const int grid = (int)std::min<long long>(ntiles, 2ll * m->sms);
    mlp::k_train<<<grid, mlp::THREADS, mlp::TrainSmem::BYTES, s>>>(X, T, n, m->packed, m->P, grad, loss, m->err);
  }
  return cudaGetLastError() == cudaSuccess ? AGIMP_OK : AGIMP_CUDA_ERROR;
}

agimp_status agimp_mlp_grad(agimp_mlp* m, const float* X, const float* T, int64_t n, float* grad, float* loss,
                            void* stream) {
  if (!m || n < 0 || (n > 0 && (!X || !T))) return AGIMP_INVALID_ARG;
  if (cudaSetDevice(m->device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  return mlp_grad(m, X, T, n, grad ? grad : m->grad, loss ? loss : m->loss, (cudaStream_t)stream);
}

agimp_status agimp_mlp_train_step(agimp_mlp* m, const float* X, const float* T, int64_t n, float lr, float* loss,
                                  void* stream) {
  if (!m || n <= 0 || !X || !T || !(lr > 0.f)) return AGIMP_INVALID_ARG;
  if (cudaSetDevice(m->device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  cudaStream_t s = (cudaStream_t)stream;
  agimp_status r = mlp_grad(m, X, T, n, m->grad, m->loss, s);
  if (r) return r;
  m->step += 1;
  mlp::k_adam<<<(mlp::NPARAM + 255) / 256, 256, 0, s>>>(m->P, m->grad, m->m1, m->m2, lr, 0.9f, 0.999f, 1e-8f,
                                                         m->step);
  mlp::k_pack<<<(mlp::NPACK + 255) / 256, 256, 0, s>>>(m->P, m->packed);
  if (loss && cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return AGIMP_CUDA_ERROR;
  return cudaGetLastError() == cudaSuccess ? AGIMP_OK : AGIMP_CUDA_ERROR;
}

agimp_status agimp_mlp_reset_optimizer(agimp_mlp* m) {
  if (!m) return AGIMP_INVALID_ARG;
  if (cudaSetDevice(m->device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  cudaMemset(m->m1, 0, mlp::NPARAM * sizeof(float));
  cudaMemset(m->m2, 0, mlp::NPARAM * sizeof(float));
  m->step = 0;
  return AGIMP_OK;
}

agimp_status agimp_mlp_errors(agimp_mlp* m, uint32_t* bits, int32_t clear) {
  if (!m || !bits) return AGIMP_INVALID_ARG;
  if (cudaSetDevice(m->device) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return AGIMP_CUDA_ERROR;
  int32_t v = 0;
  if (cudaMemcpy(&v, m->err, sizeof(v), cudaMemcpyDeviceToHost) != cudaSuccess) return AGIMP_CUDA_ERROR;
  *bits = (uint32_t)v;
  if (clear) cudaMemset(m->err, 0, sizeof(int32_t));
  return AGIMP_OK;
}

agimp_status agimp_wait_selftest(int32_t device, int32_t arrive, uint32_t max_polls, uint32_t* bits) {
  if (!bits || max_polls == 0) return AGIMP_INVALID_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return AGIMP_CUDA_ERROR;
  uint32_t* d = nullptr;
  if (cudaMalloc(&d, sizeof(uint32_t)) != cudaSuccess) return AGIMP_OUT_OF_MEMORY;
  uint32_t v = 0;
  bool good = cudaMemset(d, 0, sizeof(uint32_t)) == cudaSuccess;
  if (good) {
    k_wait_selftest<<<1, 128>>>(d, max_polls, arrive);
    good = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess &&
           cudaMemcpy(&v, d, sizeof(v), cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  cudaFree(d);
  if (!good) return AGIMP_CUDA_ERROR;
  *bits = v ? AGIMP_ERR_WAIT : 0u;
  return v ? AGIMP_DEVICE_TIMEOUT : AGIMP_OK;
}

}  // extern "C"
