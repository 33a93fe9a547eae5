// Share network: a small MLP that predicts, for every corner vertex coincident with a
// coarser corner, its coefficient in the minimum-norm solution of the shell system (the
// solution Eigen's CGLS reaches from zero). Those coefficients are exactly the free "shares"
// of the exact start, so a good prediction puts the exact solution close to the reference's.
//
// Network: 64 features -> 128 GELU -> 128 GELU -> 128 GELU -> 1, BF16 weights and
// activations, FP32 accumulation; FP32 master weights trained with Adam on a mean squared
// error. Inference and the training step are one persistent kernel each (kMlpForwardFused,
// kMlpGradientFused): tcgen05 products of 128 rows, operands in shared memory in the
// 128-byte-swizzled layout, accumulators in TMEM, everything between two products in the epilogue.
// Partial sums are added in a fixed order, so a training step is deterministic. The forward pass
// also runs layer by layer (kUmmaGemm), the same bits.
//
// Parameters (flat FP32): W1[128x64] b1[128] W2[128x128] b2[128] W3[128x128] b3[128]
// w4[128] b4[1] (W[o][i]: output o, input i).
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "its_ctx.cuh"
#include "its_umma.cuh"

namespace its {

constexpr int kIn = 64, kHid = 128;
constexpr int64_t kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
                  kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kHid, kOffW4 = kOffB3 + kHid,
                  kOffB4 = kOffW4 + kHid, kNumParams = kOffB4 + 1;

using bf16 = __nv_bfloat16;

// GELU in its tanh form (Hendrycks & Gimpel, "Gaussian Error Linear Units", 2016):
//   gelu(z) = z/2 (1 + tanh(u)),  u = sqrt(2/pi) (z + 0.044715 z^3),
// with the tanh from the hardware's approximate unit: a handful of instructions where the
// erf form costs a few dozen, in the epilogues that bound the network's kernels.
constexpr float kGeluK0 = 0.7978845608028654f;  // sqrt(2 / pi)
constexpr float kGeluK1 = 0.044715f;
__device__ __forceinline__ float tanhApprox(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float geluF(float z) {
  const float u = z * fmaf(kGeluK0 * kGeluK1, z * z, kGeluK0);
  const float h = 0.5f * z;
  return fmaf(h, tanhApprox(u), h);
}
// Two lanes of geluF with the packed FP32 instructions (each lane one IEEE FP32 operation of
// geluF's, in geluF's order: the same bits at half the instructions).
__device__ __forceinline__ float2 geluF2(float2 z) {
  const float2 p = __ffma2_rn(make_float2(kGeluK0 * kGeluK1, kGeluK0 * kGeluK1), __fmul2_rn(z, z),
                              make_float2(kGeluK0, kGeluK0));
  const float2 u = __fmul2_rn(z, p);
  const float2 h = __fmul2_rn(make_float2(0.5f, 0.5f), z);
  return __ffma2_rn(h, make_float2(tanhApprox(u.x), tanhApprox(u.y)), h);
}
// d gelu / dz = (1 + t)/2 + z/2 (1 - t^2) sqrt(2/pi) (1 + 3 * 0.044715 z^2), t = tanh(u); two lanes
__device__ __forceinline__ float2 geluGrad2(float2 z) {
  const float2 k0 = make_float2(kGeluK0, kGeluK0), half = make_float2(0.5f, 0.5f), one = make_float2(1.0f, 1.0f);
  const float2 z2 = __fmul2_rn(z, z);
  const float2 u = __fmul2_rn(z, __ffma2_rn(make_float2(kGeluK0 * kGeluK1, kGeluK0 * kGeluK1), z2, k0));
  const float2 t = make_float2(tanhApprox(u.x), tanhApprox(u.y));
  const float2 du = __ffma2_rn(make_float2(3.0f * kGeluK0 * kGeluK1, 3.0f * kGeluK0 * kGeluK1), z2, k0);
  return __ffma2_rn(__fmul2_rn(__fmul2_rn(half, z), du), __ffma2_rn(make_float2(-t.x, -t.y), t, one),
                    __fmul2_rn(half, __fadd2_rn(one, t)));
}

// ---- one tcgen05 GEMM: C[m][n] = sum_k A[m][k] B[n][k], n < 128 -----------------------------
// 128 rows per CTA and four warp groups: 64-wide K chunks are fetched by all 512 threads with
// cp.async into one of two stages while the tensor core multiplies the other; the accumulator
// (TMEM) is read back by each warp group for a quarter of the columns (thread = row, the TMEM
// lane of its warp) and handed to the epilogue functor with that quarter. K is a multiple of 64.
constexpr int kGemmGroups = 4;
constexpr int kGemmThreads = 128 * kGemmGroups;
constexpr int kGemmStage = 2 * 128 * 128;  // a chunk of A and one of B
// two stages, the epilogue's per-group row partials, mbarriers, TMEM slot
constexpr int kGemmSmem = 2 * kGemmStage + kGemmGroups * 128 * 4 + 64 + 1024;

// 16 bytes global -> shared without staging through registers; bytes < 16 zero-fills the rest.
__device__ __forceinline__ void cpAsync16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int Pending>
__device__ __forceinline__ void cpAsyncWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(Pending) : "memory");
}

template <class Epi>
__global__ void __launch_bounds__(kGemmThreads, 2) kUmmaGemm(const bf16* __restrict__ A, int64_t M,
                                                             const bf16* __restrict__ B, int K, Epi epi,
                                                             int* __restrict__ err) {
  using namespace umma;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  float* sPart = (float*)(smem + 2 * kGemmStage);          // [group][row]
  uint64_t* mbar = (uint64_t*)(sPart + kGemmGroups * 128);  // one per stage
  uint32_t* slot = (uint32_t*)(mbar + 2);
  const int tid = threadIdx.x, warp = tid >> 5, grp = tid >> 7, row = tid & 127;
  const int64_t m0 = (int64_t)blockIdx.x * 128;
  if (warp == 0) tmemAlloc(smemAddr(slot), 128);
  if (tid == 0) {
    mbarInit(smemAddr(mbar), 1);
    mbarInit(smemAddr(mbar + 1), 1);
  }
  fenceBefore();
  __syncthreads();
  fenceAfter();
  const uint32_t tmem = *slot;
  constexpr uint32_t idesc = idescBf16(128, 128);
  // chunk kc into stage st; rows past M read as zeros
  auto load = [&](int st, int kc) {
    uint8_t* sA = smem + st * kGemmStage;
    uint8_t* sB = sA + kGemmStage / 2;
    for (int i = tid; i < 128 * 8; i += kGemmThreads) {
      const int r = i >> 3, c = i & 7, col = kc + c * 8;
      const bool in = m0 + r < M;
      cpAsync16(smemAddr(sA + swizzledChunk(r, c)), in ? (const void*)(A + (m0 + r) * K + col) : (const void*)A,
                in ? 16u : 0u);
      cpAsync16(smemAddr(sB + swizzledChunk(r, c)), B + (int64_t)r * K + col, 16u);
    }
    cpAsyncCommit();
  };
  const int nk = K / 64;
  uint32_t ph[2] = {0u, 0u};
  bool ok = true;
  load(0, 0);
  for (int c = 0; c < nk; ++c) {
    const int st = c & 1;
    if (c + 1 < nk) {
      if (c >= 1) {  // the products of chunk c - 1 have read the stage chunk c + 1 goes into
        ok = mbarWait(smemAddr(mbar + (st ^ 1)), ph[st ^ 1]) && ok;
        ph[st ^ 1] ^= 1u;
      }
      load(st ^ 1, (c + 1) * 64);
      cpAsyncWait<1>();  // this chunk's copies (the next chunk's may still be in flight)
    } else {
      cpAsyncWait<0>();
    }
    fenceProxyAsync();
    __syncthreads();
    if (tid == 0) {
      fenceAfter();
      const uint8_t* sA = smem + st * kGemmStage;
      const uint64_t da = descSw128(smemAddr(sA)), db = descSw128(smemAddr(sA + kGemmStage / 2));
#pragma unroll
      for (int k = 0; k < 4; ++k) mma(tmem, da + 2 * k, db + 2 * k, idesc, (c > 0 || k > 0) ? 1u : 0u);
      commit(smemAddr(mbar + st));
    }
  }
  const int last = (nk - 1) & 1;  // the last chunk's products (and with them every earlier one)
  ok = mbarWait(smemAddr(mbar + last), ph[last]) && ok;
  fenceAfter();
  constexpr int C = 128 / kGemmGroups;
  static_assert(C == 32, "a quarter of the columns per warp group");
  float v[C];
  const uint32_t lane = (uint32_t)((warp & 3) * 32) << 16;
  tmemLoad32(tmem + lane + (uint32_t)(grp * C), v);
  const int64_t m = m0 + row;
  epi(m, ok && m < M, grp * C, v, sPart, grp, smem, m0, M);  // the stages are free: the products are done
  fenceBefore();
  __syncthreads();
  if (warp == 0) tmemFree(tmem, 128);
  if (!ok && tid == 0) atomicExch(err, 1);
}

// ---- epilogues ----------------------------------------------------------------------------
// Each is called by every thread with its row m, whether the row is written (valid), the first
// column j0 of its warp group's quarter and that quarter's accumulators.
__device__ __forceinline__ uint4 packBf16x8(const float* v) {
  uint4 r;
  __nv_bfloat162* q = (__nv_bfloat162*)&r;
#pragma unroll
  for (int e = 0; e < 4; ++e) q[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
  return r;
}
// A row-major 128-row tile goes out through shared memory: each thread stages its row's 16-byte
// pieces (piece c of row r at slot c ^ (r mod pieces per row): no bank conflicts either way),
// then consecutive threads write consecutive pieces of whole rows.
template <int RowBytes>
__device__ __forceinline__ void stageRow(uint8_t* sR, int row, int byteCol, const uint4& v) {
  constexpr int kPieces = RowBytes / 16;
  *(uint4*)(sR + row * RowBytes + (((byteCol >> 4) ^ (row % kPieces)) << 4)) = v;
}
template <int RowBytes>
__device__ __forceinline__ uint4 rowPiece(const uint8_t* sR, int row, int byteCol) {
  constexpr int kPieces = RowBytes / 16;
  return *(const uint4*)(sR + row * RowBytes + (((byteCol >> 4) ^ (row % kPieces)) << 4));
}
template <int RowBytes>
__device__ __forceinline__ void storeRows(const uint8_t* sR, void* dst, int64_t m0, int64_t M) {
  constexpr int kPieces = RowBytes / 16;
  for (int p = threadIdx.x; p < 128 * kPieces; p += blockDim.x) {
    const int row = p / kPieces, c = p % kPieces;
    if (m0 + row < M)
      *(uint4*)((uint8_t*)dst + (m0 + row) * RowBytes + c * 16) = rowPiece<RowBytes>(sR, row, c * 16);
  }
}
// Hidden layer: h = gelu(acc + b), out through the first half of the stage area.
struct EpiHidden {
  const float* bias;
  bf16* H;
  template <int C>
  __device__ void operator()(int64_t m, bool valid, int j0, float (&v)[C], float*, int, uint8_t* stage,
                             int64_t m0, int64_t M) const {
    const int row = threadIdx.x & 127;
    if (valid) {
#pragma unroll
      for (int jb = 0; jb < C; jb += 8) {
        const int j = j0 + jb;
        float h[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) h[e] = geluF(v[jb + e] + bias[j + e]);
        stageRow<kHid * 2>(stage, row, j * 2, packBf16x8(h));
      }
    }
    __syncthreads();
    storeRows<kHid * 2>(stage, H, m0, M);
  }
};

constexpr int kOutParts = 4;  // partial sums of the output unit (one per quarter of the columns)
static_assert(kOutParts == kGemmGroups, "the output unit's partial sums follow the warp groups");

// Last hidden layer plus the output unit: out = sum_j h_j w4_j + b4. The output unit sums each quarter
// of the columns in order (one per warp group), then the four partial sums in order -- the fused
// kernels' split, so all give the same bits.
struct EpiOutput {
  const float* bias;
  const float* w4;  // BF16-rounded values
  const float* b4;
  float* out;
  template <int C>
  __device__ void operator()(int64_t m, bool valid, int j0, float (&v)[C], float* sPart, int grp, uint8_t*,
                             int64_t, int64_t) const {
    const int row = threadIdx.x & 127;
    float o = 0.0f;
    if (valid) {
#pragma unroll
      for (int e = 0; e < C; ++e)
        o += __bfloat162float(__float2bfloat16_rn(geluF(v[e] + bias[j0 + e]))) * w4[j0 + e];
    }
    sPart[grp * 128 + row] = o;
    __syncthreads();
    if (grp == 0 && valid) {
      float oo = sPart[row];
#pragma unroll
      for (int g = 1; g < kOutParts; ++g) oo += sPart[g * 128 + row];
      out[m] = oo + b4[0];
    }
  }
};

// ---- fused inference ------------------------------------------------------------------------
// The whole network for 128-row tiles in one persistent kernel: the three weight matrices
// stay in shared memory (80 KB, loaded once per CTA), the features of a tile are converted to
// BF16 into shared memory, and each layer's activations go from TMEM through the epilogue
// straight back into shared memory as the next layer's A operand -- nothing but the features
// and the outputs touches global memory. The MMA sequence and the epilogue arithmetic are
// those of the layer-by-layer kernels, so the outputs are identical.
constexpr int kFusedSlots = 2;                                 // 128-row tiles in flight per CTA
constexpr int kFusedGroups = 4;                                // warp groups per tile, one per quarter of the columns
constexpr int kSlotThreads = 128 * kFusedGroups;
constexpr int kFusedThreads = kSlotThreads * kFusedSlots;
constexpr int kGroupCols = 128 / kFusedGroups;
static_assert(kFusedGroups == kOutParts, "the output unit's partial sums follow the warp groups in both kernels");
constexpr int kFusedSmem = 16384 /*W1*/ + 32768 /*W2*/ + 32768 /*W3*/ + kFusedSlots * (16384 /*X*/ + 32768 /*H*/) +
                           4 * 128 * 4 /*b1 b2 b3 w4*/ + kFusedSlots * kFusedGroups * 128 * 4 /*partial sums*/ + 64 +
                           1024;

// The fused kernel's shared-memory image of the weights, built once per parameter update:
// W1 (16 KB), W2 and W3 (32 KB each) as 128 x K bf16 K-major B operands in 128-byte-swizzled
// blocks of 128 x 64, then b1, b2, b3 and the BF16-rounded w4 (512 floats). A CTA fetches it
// with a few bulk copies.
constexpr int kImgWeights = 16384 + 32768 + 32768, kImgBytes = kImgWeights + 4 * 128 * 4;
__global__ void kPackFusedImage(const float* __restrict__ P, const bf16* __restrict__ W1, const bf16* __restrict__ W2,
                                const bf16* __restrict__ W3, const float* __restrict__ w4r, uint8_t* __restrict__ img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // one 16-byte chunk of a weight row
  if (i < 128 * 8 + 2 * 128 * 16) {
    const bf16* W = i < 1024 ? W1 : (i < 1024 + 2048 ? W2 : W3);
    const int K = i < 1024 ? kIn : kHid;
    const int j = i < 1024 ? i : (i - 1024) % 2048;
    const int r = j / (K / 8), c = j % (K / 8);
    uint8_t* dst = img + (i < 1024 ? 0 : (i < 1024 + 2048 ? 16384 : 16384 + 32768));
    *(uint4*)(dst + (c >> 3) * 16384 + umma::swizzledChunk(r, c & 7)) = *(const uint4*)(W + (int64_t)r * K + c * 8);
  }
  if (i < 512) {
    float* b = (float*)(img + kImgWeights);
    b[i] = i < 384 ? P[(i < 128 ? kOffB1 : (i < 256 ? kOffB2 : kOffB3)) + (i & 127)] : w4r[i - 384];
  }
}

// Barrier of one tile slot (256 threads), ids 1 and 2 (0 is __syncthreads').
__device__ __forceinline__ void slotSync(int s) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + s), "n"(kSlotThreads) : "memory");
}

// Share-network inference: persistent, one CTA per SM, two 128-row tiles in flight. A tile's
// 512 threads load its features, one of them issues each layer's MMAs, and the four warp
// groups run the epilogue of a quarter of the 128 columns each (thread = row, the TMEM lane of
// its warp). Biases and output weights sit in shared memory. The output unit sums each
// group's quarter of the columns in order and the first group adds the four partial sums in
// order, as the layer-by-layer kernels do, so the result is theirs bit for bit.
__global__ void __launch_bounds__(kFusedThreads, 1)
    kMlpForwardFused(const float* __restrict__ X, int64_t n, const uint8_t* __restrict__ img,
                     const float* __restrict__ P, float* __restrict__ out, int* __restrict__ err, const int64_t* __restrict__ shareIds,
                     double* __restrict__ shares, float shareScale, float shareMean, const bf16* __restrict__ Xt) {
  using namespace umma;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t* sW1 = smem;
  uint8_t* sW2 = sW1 + 16384;
  uint8_t* sW3 = sW2 + 32768;
  const int tid = threadIdx.x, s = tid / kSlotThreads, st = tid % kSlotThreads, grp = st >> 7, row = tid & 127,
            warp = tid >> 5;
  uint8_t* sX = sW3 + 32768 + s * (16384 + 32768);
  uint8_t* sH = sX + 16384;
  float* sBias = (float*)(sW3 + 32768 + kFusedSlots * (16384 + 32768));  // b1, b2, b3, w4 (128 each)
  float* sPart = sBias + 4 * 128 + s * kFusedGroups * 128;               // [group][row] partial sums
  uint64_t* mbar = (uint64_t*)(sBias + 4 * 128 + kFusedSlots * kFusedGroups * 128);  // MMA, input loads, weights
  uint32_t* tslot = (uint32_t*)(mbar + 2 * kFusedSlots + 1);
  volatile uint32_t* slot0Started = tslot + 1;  // set once slot 0's first layer-1 product is done
  const uint32_t barW = smemAddr(mbar + 2 * kFusedSlots);
  if (warp == 0) tmemAlloc(smemAddr(tslot), 128 * kFusedSlots);
  if (tid == 0) {
    *slot0Started = 0;
    for (int k = 0; k < 2 * kFusedSlots + 1; ++k) mbarInit(smemAddr(mbar + k), 1);
    // the weight image in five 16 KB bulk copies and the biases in one; the image was written
    // before the previous kernel started (only the features are its output)
    mbarArriveExpectTx(barW, kImgBytes);
#pragma unroll
    for (int k = 0; k < kImgWeights / 16384; ++k) bulkLoad(smemAddr(sW1 + k * 16384), img + k * 16384, 16384, barW);
    bulkLoad(smemAddr(sBias), img + kImgWeights, kImgBytes - kImgWeights, barW);
  }
  gridDependencyWait();
  gridDependents();
  const int64_t tiles = (n + 127) / 128;
  if (tid == 0 && Xt)  // each slot's first input tile (the previous kernel's output), beside the weights
    for (int s2 = 0; s2 < kFusedSlots; ++s2) {
      const int64_t t0 = (int64_t)blockIdx.x * kFusedSlots + s2;
      if (t0 >= tiles) break;
      const uint32_t b2 = smemAddr(mbar + kFusedSlots + s2);
      mbarArriveExpectTx(b2, 16384);
      bulkLoad(smemAddr(sW3 + 32768 + s2 * (16384 + 32768)), (const uint8_t*)Xt + t0 * 16384, 16384, b2);
    }
  fenceBefore();
  __syncthreads();
  fenceAfter();
  bool ok = mbarWait(barW, 0);
  const uint32_t tmem = *tslot + 128u * s;                 // this tile slot's 128 columns
  const uint32_t lane = (uint32_t)((warp & 3) * 32) << 16;  // the warp's TMEM lanes
  constexpr uint32_t idesc = idescBf16(128, kHid);
  const uint32_t bar = smemAddr(mbar + s), barX = smemAddr(mbar + kFusedSlots + s);
  uint32_t phase = 0, phaseX = 0;
  const float* b1 = sBias;
  const float* b2 = sBias + 128;
  const float* b3 = sBias + 256;
  const float* w4 = sBias + 384;
  const bool xVec = ((uintptr_t)X & 15) == 0;  // rows are 256 B apart: 16-byte loads when the base allows
  for (int64_t t = (int64_t)blockIdx.x * kFusedSlots + s; t < tiles; t += (int64_t)gridDim.x * kFusedSlots) {
    const int64_t m = t * 128 + row;
    if (Xt) {  // the tile already in BF16 and swizzled: one bulk copy by the TMA engine
      if (st == 0 && t != (int64_t)blockIdx.x * kFusedSlots + s) {  // (the first was issued above)
        mbarArriveExpectTx(barX, 16384);
        bulkLoad(smemAddr(sX), (const uint8_t*)Xt + t * 16384, 16384, barX);
      }
      ok = mbarWait(barX, phaseX) && ok;
      phaseX ^= 1u;
    }
    // features -> BF16: the tile's 128 rows x 256 B read in coalesced 32-byte pieces, each one
    // 16-byte chunk of a row in the swizzled A tile
#pragma unroll 2
    for (int p = st; p < (Xt ? 0 : 128 * 8); p += kSlotThreads) {
      const int pr = p >> 3, pc = p & 7;
      const int64_t mr = t * 128 + pr;
      float4 f0 = make_float4(0.f, 0.f, 0.f, 0.f), f1 = f0;
      if (mr < n) {
        const float* src = X + mr * kIn + pc * 8;
        if (xVec) {
          f0 = ((const float4*)src)[0];
          f1 = ((const float4*)src)[1];
        } else {
          f0 = make_float4(src[0], src[1], src[2], src[3]);
          f1 = make_float4(src[4], src[5], src[6], src[7]);
        }
      }
      __align__(16) bf16 v[8] = {__float2bfloat16_rn(f0.x), __float2bfloat16_rn(f0.y), __float2bfloat16_rn(f0.z),
                                 __float2bfloat16_rn(f0.w), __float2bfloat16_rn(f1.x), __float2bfloat16_rn(f1.y),
                                 __float2bfloat16_rn(f1.z), __float2bfloat16_rn(f1.w)};
      *(uint4*)(sX + swizzledChunk(pr, pc)) = *(const uint4*)v;
    }
    // The two slots start half a layer apart: slot 1 begins once slot 0's first product is
    // done, so that one slot's epilogue (bound by the tanh unit and the issue rate) runs while
    // the other's MMA does. A bounded wait: past the bound slot 1 simply goes on.
    if (s == 1 && t == (int64_t)blockIdx.x * kFusedSlots + s)
      for (int spin = 0; spin < 20000 && *slot0Started == 0; ++spin) __nanosleep(32);
    float o = 0.0f;
    for (int layer = 0; layer < 3; ++layer) {
      fenceProxyAsync();
      fenceBefore();
      slotSync(s);
      if (st == 0) {
        fenceAfter();
        if (layer == 0) {
          const uint64_t da = descSw128(smemAddr(sX)), db = descSw128(smemAddr(sW1));
#pragma unroll
          for (int k = 0; k < 4; ++k) mma(tmem, da + 2 * k, db + 2 * k, idesc, k > 0 ? 1u : 0u);
        } else {
          const uint8_t* sW = layer == 1 ? sW2 : sW3;
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
            const uint64_t da = descSw128(smemAddr(sH + kb * 16384)), db = descSw128(smemAddr(sW + kb * 16384));
#pragma unroll
            for (int k = 0; k < 4; ++k) mma(tmem, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
        }
        commit(bar);
      }
      ok = mbarWait(bar, phase) && ok;
      phase ^= 1u;
      fenceAfter();
      if (s == 0 && st == 0 && layer == 0) *slot0Started = 1;
      // epilogue of this group's 32 columns: one TMEM load, one wait
      const float* bias = layer == 0 ? b1 : (layer == 1 ? b2 : b3);
      const int n0 = kGroupCols * grp;
      float v[kGroupCols];
      tmemLoad32(tmem + lane + (uint32_t)n0, v);
      // two columns per packed FP32 instruction; the output unit's sum stays in column order
      if (layer < 2) {  // hidden layer: the next layer's A operand
#pragma unroll
        for (int h = 0; h < kGroupCols / 8; ++h) {
          __align__(16) __nv_bfloat162 q[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int j = h * 8 + 2 * e;
            const float2 b = *(const float2*)(bias + n0 + j);
            q[e] = __float22bfloat162_rn(geluF2(__fadd2_rn(make_float2(v[j], v[j + 1]), b)));
          }
          const int c = (n0 >> 3) + h;
          *(uint4*)(sH + (c >> 3) * 16384 + swizzledChunk(row, c & 7)) = *(const uint4*)q;
        }
      } else {  // output unit: this group's quarter of the columns, in order
#pragma unroll
        for (int j = 0; j < kGroupCols; j += 2) {
          const float2 b = *(const float2*)(bias + n0 + j);
          const float2 g = __bfloat1622float2(__float22bfloat162_rn(geluF2(__fadd2_rn(make_float2(v[j], v[j + 1]), b))));
          const float2 t = __fmul2_rn(g, *(const float2*)(w4 + n0 + j));
          o += t.x;
          o += t.y;
        }
      }
    }
    if (grp > 0) sPart[grp * 128 + row] = o;
    slotSync(s);
    if (grp == 0) {
#pragma unroll
      for (int g = 1; g < kFusedGroups; ++g) o += sPart[g * 128 + row];
      if (m < n && ok) {
        const float pred = o + P[kOffB4];
        if (shares)  // the learned start's share of coincident vertex shareIds[m], de-normalised
          shares[shareIds[m]] = (double)pred * (double)shareScale + (double)shareMean;
        else
          out[m] = pred;
      }
    }
    fenceBefore();
    slotSync(s);  // TMEM read and sH free before the next tile
  }
  fenceBefore();
  __syncthreads();
  if (warp == 0) tmemFree(*tslot, 128 * kFusedSlots);
  if (!ok) atomicExch(err, 1);
}

// ---- small kernels ----------------------------------------------------------------------
// Features (FP32, n x 64, already normalised) to BF16 rows.
__global__ void kFeaturesBf16(const float* __restrict__ X, int64_t n, bf16* __restrict__ Xb) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n * kIn) Xb[i] = __float2bfloat16_rn(X[i]);
}

// BF16 weight copies and the BF16-rounded output weights.
__global__ void kCastWeights(const float* __restrict__ P, bf16* __restrict__ W1, bf16* __restrict__ W2,
                             bf16* __restrict__ W3, float* __restrict__ w4r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kHid * kIn) W1[i] = __float2bfloat16_rn(P[kOffW1 + i]);
  if (i < kHid * kHid) {
    W2[i] = __float2bfloat16_rn(P[kOffW2 + i]);
    W3[i] = __float2bfloat16_rn(P[kOffW3 + i]);
  }
  if (i < kHid) w4r[i] = __bfloat162float(__float2bfloat16_rn(P[kOffW4 + i]));
}

// ---- fused training step ------------------------------------------------------------------
// Loss and gradient of a batch in one persistent kernel, a CTA per SM: a 128-row tile goes forward
// and back without leaving the SM. Shared memory holds the weights (80 KB) and the tile's features,
// H1, H2 and dZ (112 KB), each once, row by row: the transposed products (dH = dZ W, dW = dZ^T H)
// read the same blocks MN-major. TMEM holds one 128-column accumulator for the layers and, across
// the CTA's tiles, the weight and bias gradients (320 + 48 columns). gelu' needs the pre-activations in
// FP32: they are formed again by the same products just before they are used, instead of being
// kept. The bias gradients are products with a tile of ones; the output weights' are summed over a
// warp's rows by exchanges, a column per lane, in FP32. Every CTA leaves its sums in a slot of its own, which kSumPartials adds in CTA order, so a
// step is deterministic. The forward values, the loss gradient and every dZ are those of a pass
// layer by layer, bit for bit; the weight gradients are grouped by CTA. (Layer by layer, with the
// activations, their transposes and FP32 pre-activations through memory, 75-84 MB a layer: 253 us in
// 11 launches at 65,536 rows; now 66 + 8 us.)
constexpr int kTrainThreads = 512;
constexpr int64_t kPartStride = (kNumParams + 1 + 3) / 4 * 4;  // the parameters' order, then the squared errors
constexpr int kTrainSmem = 16384 + 32768 + 32768 /*W1 W2 W3*/ + 2 * 16384 /*X, this tile's and the next's*/ + 3 * 32768 /*H1 H2 dZ*/ +
                           4096 /*ones*/ + 4 * 128 * 4 /*b1 b2 b3 w4*/ + kOutParts * 128 * 4 /*partial sums*/ + 128 * 4 /*d*/ +
                           64 + 1024;

// Where a batch's row m lies in the dataset: itself, or a random row (splitmix64 of seed, step and m).
struct BatchRows {
  int64_t n;  // rows of the dataset to draw from; 0: row m itself
  uint64_t seed, first;
  __device__ __forceinline__ int64_t operator()(int64_t m) const {
    if (n == 0) return m;
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (first + (uint64_t)m + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (int64_t)(z % (uint64_t)n);
  }
};

// Column l of the warp's 32 x 32 block (v: a lane's row) summed over its rows, in lane l.
__device__ __forceinline__ float columnSum(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + o], o);
      v[i] = (up ? v[i + o] : v[i]) + other;
    }
  }
  return v[0];
}

__global__ void __launch_bounds__(kTrainThreads, 1)
    kMlpGradientFused(const float* __restrict__ X, const float* __restrict__ y, const BatchRows rows, int64_t n,
                      float scale, const uint8_t* __restrict__ img, const float* __restrict__ P,
                      float* __restrict__ part, int* __restrict__ err) {
  using namespace umma;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t* sW1 = smem;
  uint8_t* sW2 = sW1 + 16384;
  uint8_t* sW3 = sW2 + 32768;
  uint8_t* sX = sW3 + 32768;
  uint8_t* sH1 = sX + 2 * 16384;
  uint8_t* sH2 = sH1 + 32768;
  uint8_t* sD = sH2 + 32768;
  uint8_t* sOne = sD + 32768;              // 16 rows of 128 ones: dZ^T 1 is the bias gradient
  float* sBias = (float*)(sOne + 4096);    // b1, b2, b3, w4 (128 each)
  float* sPart = sBias + 4 * 128;          // [group][row] partial sums
  float* sRow = sPart + kOutParts * 128;   // the loss gradient of each row
  uint64_t* mbar = (uint64_t*)(sRow + 128);
  uint32_t* tslot = (uint32_t*)(mbar + 3);
  const int tid = threadIdx.x, grp = tid >> 7, row = tid & 127, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar = smemAddr(mbar), barW = smemAddr(mbar + 1), barD = smemAddr(mbar + 2);
  if (warp == 0) tmemAlloc(smemAddr(tslot), 512);
  if (tid == 0) {
    mbarInit(bar, 1);
    mbarInit(barW, 1);
    mbarInit(barD, 1);
    mbarArriveExpectTx(barW, kImgBytes);
#pragma unroll
    for (int k = 0; k < kImgWeights / 16384; ++k) bulkLoad(smemAddr(sW1 + k * 16384), img + k * 16384, 16384, barW);
    bulkLoad(smemAddr(sBias), img + kImgWeights, kImgBytes - kImgWeights, barW);
  }
  if (tid < 256) *(uint4*)(sOne + 16 * tid) = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
  fenceBefore();
  __syncthreads();
  fenceAfter();
  bool ok = mbarWait(barW, 0);
  const uint32_t acc = *tslot, dW3 = acc + 128, dW2 = acc + 256, dW1 = acc + 384, dB = acc + 448;
  const uint32_t tl = (uint32_t)((warp & 3) * 32) << 16;  // the warp's TMEM lanes
  const int n0 = 32 * grp;                                // the group's columns
  const uint32_t myAcc = acc + tl + (uint32_t)n0;
  const float *b1 = sBias + n0, *b2 = b1 + 128, *b3 = b1 + 256, *w4 = b1 + 384;
  const float b4 = P[kOffB4];
  constexpr uint32_t idKK = idescBf16(128, 128), idKM = idKK | kMnB, idMM = idKK | kMnA | kMnB,
                     idMM64 = idescBf16(128, 64) | kMnA | kMnB, idMK16 = idescBf16(128, 16) | kMnA;
  const bool xVec = ((uintptr_t)X & 15) == 0;
  uint32_t phase = 0, phaseD = 0;
  float gW4 = 0.f, gB4 = 0.f, sq = 0.f;
  __align__(8) float v[32];
  float2* v2 = (float2*)v;

  // operands written by every thread -> one thread's products -> its barrier
  auto begin = [&] {
    fenceProxyAsync();
    fenceBefore();
    __syncthreads();
    if (tid == 0) fenceAfter();
  };
  auto wait = [&] {
    ok = mbarWait(bar, phase) && ok;
    phase ^= 1u;
    fenceAfter();
  };
  // ... and the products that read dZ's tile, committed to a barrier of their own
  auto waitD = [&] {
    ok = mbarWait(barD, phaseD) && ok;
    phaseD ^= 1u;
    fenceAfter();
  };
  // acc = A B^T, A and B K-major, kBlocks blocks of 64 along K
  auto layer = [&](const uint8_t* A, const uint8_t* B, int kBlocks) {
    for (int kb = 0; kb < kBlocks; ++kb) {
      const uint64_t da = descSw128(smemAddr(A + kb * 16384)), db = descSw128(smemAddr(B + kb * 16384));
#pragma unroll
      for (int k = 0; k < 4; ++k) mma(acc, da + 2 * k, db + 2 * k, idKK, (kb > 0 || k > 0) ? 1u : 0u);
    }
  };
  // acc = dZ W (dZ K-major, W's rows are K)
  auto back = [&](const uint8_t* W) {
    const uint64_t db = descSw128Mn(smemAddr(W));
#pragma unroll
    for (int s = 0; s < 8; ++s)
      mma(acc, descSw128(smemAddr(sD + (s >> 2) * 16384)) + 2 * (s & 3), db + 128 * s, idKM, s > 0 ? 1u : 0u);
  };
  // dW += dZ^T H over the tile's rows, and db += dZ^T 1
  auto weights = [&](uint32_t d, const uint8_t* H, uint32_t id, uint32_t db, bool more) {
    const uint64_t da = descSw128Mn(smemAddr(sD)), dh = descSw128Mn(smemAddr(H));
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      mma(d, da + 128 * s, dh + 128 * s, id, (more || s > 0) ? 1u : 0u);
      mma(db, da + 128 * s, descSw128(smemAddr(sOne + (s >> 2) * 2048)) + 2 * (s & 3), idMK16, (more || s > 0) ? 1u : 0u);
    }
  };
  // this thread's 32 columns of its row, BF16, into a K-major tile
  auto store = [&](uint8_t* T) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int c = (n0 >> 3) + h;
      *(uint4*)(T + (c >> 3) * 16384 + swizzledChunk(row, c & 7)) = packBf16x8(v + 8 * h);
    }
  };
  // v = gelu(v + b), and v *= gelu'(the accumulator + b)
  auto activate = [&](const float* b) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v2[j] = geluF2(__fadd2_rn(v2[j], ((const float2*)b)[j]));
  };
  auto derive = [&](const float* b) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      __align__(8) float z[16];
      tmemLoad16(myAcc + 16 * half, z);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 g = geluGrad2(__fadd2_rn(((const float2*)z)[j], ((const float2*)b)[8 * half + j]));
        v2[8 * half + j] = __fmul2_rn(v2[8 * half + j], g);
      }
    }
  };

  // features -> BF16, 16-byte chunks of the swizzled tile (rows past the batch: zeros)
  auto features = [&](int64_t t, uint8_t* T) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int p = tid + q * kTrainThreads, pr = p >> 3, pc = p & 7;
      const int64_t mr = t * 128 + pr;
      __align__(16) float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (mr < n) {
        const float* src = X + rows(mr) * kIn + pc * 8;
        if (xVec) {
          *(float4*)f = __ldg((const float4*)src);
          *(float4*)(f + 4) = __ldg((const float4*)src + 1);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = src[e];
        }
      }
      *(uint4*)(T + swizzledChunk(pr, pc)) = packBf16x8(f);
    }
  };

  const int64_t tiles = (n + 127) / 128;
  bool more = false;
  features(blockIdx.x, sX);
  begin();
  if (tid == 0) {
    layer(sX, sW1, 1);
    commit(bar);
  }
  int cur = 0;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t m = t * 128 + row;
    const uint8_t* sXt = sX + cur * 16384;
    uint8_t* sXn = sX + (cur ^ 1) * 16384;
    const bool next = t + gridDim.x < tiles;
    const float target = grp == 0 && m < n ? y[rows(m)] : 0.0f;
    // forward (the first layer's product is under way)
    wait();
    tmemLoad32(myAcc, v);
    activate(b1);
    store(sH1);
    begin();
    if (tid == 0) {
      layer(sH1, sW2, 2);
      commit(bar);
    }
    wait();
    tmemLoad32(myAcc, v);
    activate(b2);
    store(sH2);
    begin();
    if (tid == 0) {
      layer(sH2, sW3, 2);
      commit(bar);
    }
    wait();  // with it the previous tile's dW1: its features and dZ1 have been read
    if (next) features(t + gridDim.x, sXn);
    tmemLoad32(myAcc, v);
    float o = 0.0f;
    __nv_bfloat162 h3[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v2[j] = __fadd2_rn(v2[j], ((const float2*)b3)[j]);
      h3[j] = __float22bfloat162_rn(geluF2(v2[j]));
      const float2 p = __fmul2_rn(__bfloat1622float2(h3[j]), ((const float2*)w4)[j]);
      o += p.x;
      o += p.y;
    }
    sPart[grp * 128 + row] = o;
    __syncthreads();
    if (grp == 0) {
      float d = 0.0f;
      if (m < n) {
        float oo = sPart[row];
#pragma unroll
        for (int g = 1; g < kOutParts; ++g) oo += sPart[g * 128 + row];
        oo += b4;
        const float e = oo - target;
        d = scale * e;
        gB4 += d;
        sq += e * e;
      }
      sRow[row] = d;
    }
    __syncthreads();
    const float d = sRow[row];
    const float2 d2 = make_float2(d, d);
    // backward: dZ3 and dH2; Z2 again, with dW3 behind it, dZ2 and dH1; Z1 again, with dW2 behind it,
    // dZ1; dW1, with the next tile's first layer behind it
#pragma unroll
    for (int j = 0; j < 16; ++j)
      v2[j] = __fmul2_rn(__fmul2_rn(d2, ((const float2*)w4)[j]), geluGrad2(v2[j]));
    store(sD);
    begin();
    if (tid == 0) {
      back(sW3);
      commit(bar);
    }
    // the output weights' gradient while the product runs
#pragma unroll
    for (int j = 0; j < 16; ++j) v2[j] = __fmul2_rn(__bfloat1622float2(h3[j]), d2);
    gW4 += columnSum(v, lane);
    wait();
    tmemLoad32(myAcc, v);
    begin();
    if (tid == 0) {
      layer(sH1, sW2, 2);
      commit(bar);
      weights(dW3, sH2, idMM, dB + 32, more);
      commit(barD);
    }
    wait();
    derive(b2);
    waitD();
    store(sD);
    begin();
    if (tid == 0) {
      back(sW2);
      commit(bar);
    }
    wait();
    tmemLoad32(myAcc, v);
    begin();
    if (tid == 0) {
      layer(sXt, sW1, 1);
      commit(bar);
      weights(dW2, sH1, idMM, dB + 16, more);
      commit(barD);
    }
    wait();
    derive(b1);
    waitD();
    store(sD);
    begin();
    if (tid == 0) {
      weights(dW1, sXt, idMM64, dB, more);
      if (next) layer(sXn, sW1, 1);
      commit(bar);
    }
    more = true;
    cur ^= 1;
  }
  wait();  // the last tile's dW1
  // the CTA's sums: weight gradients (row o of this thread), then the columns' and rows' sums
  float* out = part + (int64_t)blockIdx.x * kPartStride;
  // (four columns of all rows after one another, so that a warp's stores are contiguous)
  tmemLoad32(dW3 + tl + (uint32_t)n0, v);
#pragma unroll
  for (int j = 0; j < 32; j += 4)
    *(float4*)(out + kOffW3 + (n0 + j) * 128 + row * 4) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  tmemLoad32(dW2 + tl + (uint32_t)n0, v);
#pragma unroll
  for (int j = 0; j < 32; j += 4)
    *(float4*)(out + kOffW2 + (n0 + j) * 128 + row * 4) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  {
    float u[16];
    tmemLoad16(dW1 + tl + (uint32_t)(16 * grp), u);
#pragma unroll
    for (int j = 0; j < 16; j += 4)
      *(float4*)(out + kOffW1 + (16 * grp + j) * 128 + row * 4) = make_float4(u[j], u[j + 1], u[j + 2], u[j + 3]);
  }
  if (grp < 3) {  // the bias gradients: each of the 16 columns holds them
    float u[16];
    tmemLoad16(dB + tl + (uint32_t)(16 * grp), u);
    out[(grp == 0 ? kOffB1 : grp == 1 ? kOffB2 : kOffB3) + row] = u[0];
  }
  float* sums = (float*)sX;  // [quarter of the rows][128 columns], then two per warp of group 0
  sums[(warp & 3) * 128 + n0 + lane] = gW4;
  if (grp == 0) {
    for (int o = 16; o > 0; o >>= 1) {
      gB4 += __shfl_down_sync(0xffffffffu, gB4, o);
      sq += __shfl_down_sync(0xffffffffu, sq, o);
    }
    if (lane == 0) {
      sums[4 * 128 + 2 * warp] = gB4;
      sums[4 * 128 + 2 * warp + 1] = sq;
    }
  }
  fenceBefore();
  __syncthreads();
  if (warp == 0) tmemFree(*tslot, 512);
  if (grp == 0) out[kOffW4 + row] = ((sums[row] + sums[128 + row]) + sums[256 + row]) + sums[384 + row];
  if (tid < 2) {
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) s += sums[4 * 128 + 2 * q + tid];
    out[tid == 0 ? kOffB4 : kNumParams] = s;
  }
  if (!ok) atomicExch(err, 1);
}

// The CTAs' sums added in CTA order, in four runs that are then added in order: the gradient, and the
// mean squared error behind it. A block takes 64 values of the slots, a quarter of the CTAs per warp pair.
__global__ void __launch_bounds__(256) kSumPartials(const float* __restrict__ part, int ctas, int64_t n,
                                                    float* __restrict__ grad) {
  __shared__ float sRun[4][64];
  const int64_t i = blockIdx.x * 64ll + (threadIdx.x & 63);
  const int run = threadIdx.x >> 6, per = (ctas + 3) / 4, c1 = min(ctas, (run + 1) * per);
  float s = 0.0f;
  if (i <= kNumParams) {
    int c = run * per;
    for (; c + 16 <= c1; c += 16) {
      float p[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) p[k] = part[(int64_t)(c + k) * kPartStride + i];
#pragma unroll
      for (int k = 0; k < 16; ++k) s += p[k];
    }
    for (; c < c1; ++c) s += part[(int64_t)c * kPartStride + i];
  }
  sRun[run][threadIdx.x & 63] = s;
  __syncthreads();
  if (run > 0 || i > kNumParams) return;
  s = ((sRun[0][threadIdx.x] + sRun[1][threadIdx.x]) + sRun[2][threadIdx.x]) + sRun[3][threadIdx.x];
  int64_t to = i;
  for (int l = 0; l < 3; ++l) {  // the weights' slots run four columns at a time: back to row-major
    const int64_t off = l == 0 ? kOffW1 : l == 1 ? kOffW2 : kOffW3, cols = l == 0 ? kIn : kHid, e = i - off;
    if (e >= 0 && e < kHid * cols) to = off + ((e & 511) >> 2) * cols + (e >> 9) * 4 + (e & 3);
  }
  grad[to] = i < kNumParams ? s : s / (float)n;
}

// Adam (Kingma & Ba): m = b1 m + (1-b1) g; v = b2 v + (1-b2) g^2; p -= lr mhat / (sqrt(vhat) + eps).
__global__ void kAdam(float* __restrict__ P, float* __restrict__ Mo, float* __restrict__ Ve,
                      const float* __restrict__ G, int64_t n, float lr, float b1, float b2, float eps, float c1,
                      float c2) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = G[i];
  const float m = b1 * Mo[i] + (1.0f - b1) * g;
  const float v = b2 * Ve[i] + (1.0f - b2) * g * g;
  Mo[i] = m;
  Ve[i] = v;
  P[i] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

template <class Epi>
static its_status gemm(its_ctx* ctx, const bf16* A, int64_t M, const bf16* B, int K, const Epi& epi, int* err) {
  ITS_CU(ctx, cudaFuncSetAttribute(kUmmaGemm<Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
  kUmmaGemm<Epi><<<gridFor(M, 128), kGemmThreads, kGemmSmem, ctx->stream>>>(A, M, B, K, epi, err);
  ITS_LAUNCHED(ctx);
  return ITS_OK;
}

}  // namespace its

using namespace its;

struct its_mlp {
  its_ctx* ctx = nullptr;
  uint64_t uid = 0;  // distinct for every network made (a later one may reuse a freed address)
  int64_t cap = 0;  // rows per batch
  float* P = nullptr;
  float* Mo = nullptr;
  float* Ve = nullptr;
  float* G = nullptr;     // the gradient; behind it the mean squared error and the error flag
  float* loss = nullptr;  // behind the gradient
  float* host = nullptr;  // page-locked: the gradient and the two words behind it
  int64_t step = 0;
  bf16 *W1, *W2, *W3;
  float* w4r;
  uint8_t* img;  // the fused inference kernel's shared-memory image of the parameters
  // batch buffers
  bf16 *Xb, *H1, *H2;
  float* part;  // the gradient's sums, a slot per CTA
  int* err;
  std::vector<void*> allocs;
  template <typename T>
  its_status alloc(T** p, int64_t count) {
    its_status s = devAlloc(ctx, (void**)p, (size_t)count * sizeof(T));
    if (s == ITS_OK) allocs.push_back((void*)*p);
    return s;
  }
};

namespace its {

static its_status mlpCast(its_mlp* h) {
  kCastWeights<<<gridFor(kHid * kHid, 256), 256, 0, h->ctx->stream>>>(h->P, h->W1, h->W2, h->W3, h->w4r);
  ITS_LAUNCHED(h->ctx);
  kPackFusedImage<<<gridFor(128 * 8 + 2 * 128 * 16, 256), 256, 0, h->ctx->stream>>>(h->P, h->W1, h->W2, h->W3, h->w4r,
                                                                                    h->img);
  ITS_LAUNCHED(h->ctx);
  return ITS_OK;
}

// Forward of n <= cap rows already in h->Xb, layer by layer.
static its_status mlpForward(its_mlp* h, int64_t n, float* out) {
  its_ctx* ctx = h->ctx;
  its_status st;
  if ((st = gemm(ctx, h->Xb, n, h->W1, kIn, EpiHidden{h->P + kOffB1, h->H1}, h->err)) != ITS_OK ||
      (st = gemm(ctx, h->H1, n, h->W2, kHid, EpiHidden{h->P + kOffB2, h->H2}, h->err)) != ITS_OK)
    return st;
  const EpiOutput e3{h->P + kOffB3, h->w4r, h->P + kOffB4, out};
  return gemm(ctx, h->H2, n, h->W3, kHid, e3, h->err);
}

// Gradient of the mean squared error over n rows of X (targets y), drawn as rows says, into h->G.
static its_status mlpGradient(its_mlp* h, const float* X, const float* y, const BatchRows& rows, int64_t n) {
  its_ctx* ctx = h->ctx;
  const int64_t tiles = (n + 127) / 128;
  const int ctas = (int)(tiles < ctx->numSMs ? tiles : ctx->numSMs);
  kMlpGradientFused<<<ctas, kTrainThreads, kTrainSmem, ctx->stream>>>(X, y, rows, n, 2.0f / (float)n, h->img, h->P,
                                                                     h->part, h->err);
  ITS_LAUNCHED(ctx);
  kSumPartials<<<gridFor(kNumParams + 1, 64), 256, 0, ctx->stream>>>(h->part, ctas, n, h->G);
  ITS_LAUNCHED(ctx);
  return ITS_OK;
}

static its_status mlpAdam(its_mlp* h, float lr) {
  ++h->step;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - powf(b1, (float)h->step), c2 = 1.0f - powf(b2, (float)h->step);
  kAdam<<<gridFor(kNumParams, 256), 256, 0, h->ctx->stream>>>(h->P, h->Mo, h->Ve, h->G, kNumParams, lr, b1, b2, 1e-8f,
                                                              c1, c2);
  ITS_LAUNCHED(h->ctx);
  return mlpCast(h);
}

static its_status checkErr(its_mlp* h) {
  int e = 0;
  ITS_CU(h->ctx, cudaMemcpyAsync(&e, h->err, 4, cudaMemcpyDeviceToHost, h->ctx->stream));
  ITS_CU(h->ctx, cudaStreamSynchronize(h->ctx->stream));
  if (e) return setError(h->ctx, ITS_ERR_TIMEOUT, "share network: a tensor-core wait ran out");
  return ITS_OK;
}

// Predictions for n device rows into device out, launched on the context's stream without
// waiting (the caller checks the error flag at its next synchronisation).
static its_status launchFused(its_mlp* h, const float* X, int64_t n, float* out, const int64_t* ids, double* shares,
                              float scale, float mean, bool afterKernel, const bf16* Xt = nullptr) {
  its_ctx* ctx = h->ctx;
  if (n <= 0) return ITS_OK;
  const int64_t tiles = (n + 127) / 128, ctas = (tiles + kFusedSlots - 1) / kFusedSlots;
  const unsigned grid = (unsigned)(ctas < ctx->numSMs ? ctas : ctx->numSMs);
  return launchDependent(ctx, afterKernel, kMlpForwardFused, grid, kFusedThreads, kFusedSmem, ctx->stream, X, n,
                         (const uint8_t*)h->img, (const float*)h->P, out, h->err, ids, shares, scale, mean, Xt);
}
its_status mlpInfer(its_mlp* h, const float* X, int64_t n, float* out, bool afterKernel) {
  return launchFused(h, X, n, out, nullptr, nullptr, 0.0f, 0.0f, afterKernel);
}
// The same predictions written as shares: shares[ids[m]] = pred[m] * scale + mean (in FP64,
// as the share scatter of the learned start computes it).
// Predictions from input tiles that are already BF16 and swizzled (128 rows x 128 B each,
// whole tiles): into out, or, with shares set, as shares[ids[m]] = pred[m] * scale + mean (in
// FP64, as the share scatter of the learned start computes it).
its_status mlpInferTiles(its_mlp* h, const bf16* tiles, int64_t n, float* out, const int64_t* ids, float scale,
                         float mean, double* shares, bool afterKernel) {
  return launchFused(h, nullptr, n, out, ids, shares, scale, mean, afterKernel, tiles);
}

its_status mlpCheck(its_mlp* h) { return checkErr(h); }
// The network's (sticky) error flag in device memory, for callers that read it with their own copy.
const int* mlpErrFlag(its_mlp* h) { return h->err; }
uint64_t mlpUid(const its_mlp* h) { return h->uid; }

}  // namespace its

extern "C" {

its_status its_mlp_create(its_ctx* ctx, int64_t batch, its_mlp** out) {
  if (!ctx || !out || batch <= 0 || batch % 128) return ITS_ERR_INVALID;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  its_mlp* h = new its_mlp;
  h->ctx = ctx;
  static std::atomic<uint64_t> made{0};
  h->uid = ++made;
  h->cap = batch;
  const int64_t B = batch;
  its_status s = ITS_OK;
  auto A = [&](auto** p, int64_t c) {
    if (s == ITS_OK) s = h->alloc(p, c);
  };
  A(&h->P, kNumParams); A(&h->Mo, kNumParams); A(&h->Ve, kNumParams); A(&h->G, kNumParams + 2);
  A(&h->W1, kHid * kIn); A(&h->W2, kHid * kHid); A(&h->W3, kHid * kHid); A(&h->w4r, kHid); A(&h->img, kImgBytes);
  A(&h->Xb, B * kIn); A(&h->H1, B * kHid); A(&h->H2, B * kHid); A(&h->part, ctx->numSMs * kPartStride);
  if (s != ITS_OK) {
    for (void* p : h->allocs) devFree(ctx, p);
    delete h;
    return s;
  }
  h->loss = h->G + kNumParams;
  h->err = (int*)(h->G + kNumParams + 1);
  if (cudaMallocHost((void**)&h->host, (kNumParams + 2) * 4) != cudaSuccess) {
    cudaGetLastError();
    h->host = nullptr;  // gradients then go to the caller's memory directly
  }
  cudaMemsetAsync(h->P, 0, kNumParams * 4, ctx->stream);
  cudaMemsetAsync(h->Mo, 0, kNumParams * 4, ctx->stream);
  cudaMemsetAsync(h->Ve, 0, kNumParams * 4, ctx->stream);
  cudaMemsetAsync(h->err, 0, 4, ctx->stream);
  cudaMemsetAsync(h->img, 0, kImgBytes, ctx->stream);
  // the fused kernels' shared memory, set here once (not inside a graph capture)
  ITS_CU(ctx, cudaFuncSetAttribute(kMlpForwardFused, cudaFuncAttributeMaxDynamicSharedMemorySize, kFusedSmem));
  ITS_CU(ctx, cudaFuncSetAttribute(kMlpGradientFused, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem));
  *out = h;
  return ITS_OK;
}

its_status its_mlp_free(its_mlp* h) {
  if (!h) return ITS_ERR_INVALID;
  cudaStreamSynchronize(h->ctx->stream);
  for (void* p : h->allocs) devFree(h->ctx, p);
  if (h->host) cudaFreeHost(h->host);
  delete h;
  return ITS_OK;
}

int64_t its_mlp_num_params(void) { return kNumParams; }

its_status its_mlp_set_params(its_mlp* h, const float* params) {
  if (!h || !params) return ITS_ERR_INVALID;
  ITS_CU(h->ctx, cudaMemcpyAsync(h->P, params, kNumParams * 4, cudaMemcpyDefault, h->ctx->stream));
  ITS_CU(h->ctx, cudaMemsetAsync(h->Mo, 0, kNumParams * 4, h->ctx->stream));
  ITS_CU(h->ctx, cudaMemsetAsync(h->Ve, 0, kNumParams * 4, h->ctx->stream));
  h->step = 0;
  its_status s = mlpCast(h);
  if (s != ITS_OK) return s;
  ITS_CU(h->ctx, cudaStreamSynchronize(h->ctx->stream));
  return ITS_OK;
}

its_status its_mlp_get_params(its_mlp* h, float* params) {
  if (!h || !params) return ITS_ERR_INVALID;
  ITS_CU(h->ctx, cudaMemcpyAsync(params, h->P, kNumParams * 4, cudaMemcpyDefault, h->ctx->stream));
  ITS_CU(h->ctx, cudaStreamSynchronize(h->ctx->stream));
  return ITS_OK;
}

// Predictions for n rows of features (n x 64 FP32, normalised), host or device memory.
its_status its_mlp_forward(its_mlp* h, const float* X, int64_t n, float* out) {
  if (!h || (n > 0 && (!X || !out)) || n < 0) return ITS_ERR_INVALID;
  its_ctx* ctx = h->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<float> x;
  OutArg<float> o;
  its_status st;
  if ((st = x.stage(ctx, X, n * kIn)) != ITS_OK) return st;
  if ((st = o.stage(ctx, out, n)) != ITS_OK) return st;
  if ((st = mlpInfer(h, x.d, n, o.d, false)) != ITS_OK) return st;
  if ((st = o.finish(ctx)) != ITS_OK) return st;
  return checkErr(h);
}

// The same predictions for device rows, queued on the context's stream without waiting; a
// tensor-core wait that ran out is reported by the next its_mlp_check (the flag is sticky).
its_status its_mlp_forward_async(its_mlp* h, const float* X, int64_t n, float* out) {
  if (!h || (n > 0 && (!X || !out)) || n < 0) return ITS_ERR_INVALID;
  its_ctx* ctx = h->ctx;
  if (n > 0 && (!isDevicePtr(ctx, X) || !isDevicePtr(ctx, out)))
    return setError(ctx, ITS_ERR_INVALID, "its_mlp_forward_async: features and output must be device memory");
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  return mlpInfer(h, X, n, out, false);
}

its_status its_mlp_forward_tiles_async(its_mlp* h, const void* tiles, int64_t n, float* out, int after_kernel) {
  if (!h || (n > 0 && (!tiles || !out)) || n < 0) return ITS_ERR_INVALID;
  its_ctx* ctx = h->ctx;
  if (n > 0 && (!isDevicePtr(ctx, tiles) || !isDevicePtr(ctx, out) || ((uintptr_t)tiles & 15)))
    return setError(ctx, ITS_ERR_INVALID,
                    "its_mlp_forward_tiles_async: tiles (16-byte aligned) and output must be device memory");
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  return mlpInferTiles(h, (const bf16*)tiles, n, out, nullptr, 0.0f, 0.0f, nullptr, after_kernel != 0);
}

// Waits for the context's stream and reports the network's error flag.
its_status its_mlp_check(its_mlp* h) {
  if (!h) return ITS_ERR_INVALID;
  ITS_CU(h->ctx, cudaSetDevice(h->ctx->device));
  return checkErr(h);
}

// The same predictions layer by layer; identical to
// its_mlp_forward bit for bit (a test hook).
its_status its_mlp_forward_layers(its_mlp* h, const float* X, int64_t n, float* out) {
  if (!h || (n > 0 && (!X || !out)) || n < 0) return ITS_ERR_INVALID;
  its_ctx* ctx = h->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<float> x;
  OutArg<float> o;
  its_status st;
  if ((st = x.stage(ctx, X, n * kIn)) != ITS_OK) return st;
  if ((st = o.stage(ctx, out, n)) != ITS_OK) return st;
  for (int64_t r0 = 0; r0 < n; r0 += h->cap) {
    const int64_t rows = n - r0 < h->cap ? n - r0 : h->cap;
    kFeaturesBf16<<<gridFor(rows * kIn, 256), 256, 0, ctx->stream>>>(x.d + r0 * kIn, rows, h->Xb);
    ITS_LAUNCHED(ctx);
    if ((st = mlpForward(h, rows, o.d + r0)) != ITS_OK) return st;
  }
  if ((st = o.finish(ctx)) != ITS_OK) return st;
  return checkErr(h);
}

// Gradient of the mean squared error over n rows (n <= batch, a multiple of 64; no update):
// grad has its_mlp_num_params() entries; loss may be NULL.
its_status its_mlp_gradient(its_mlp* h, const float* X, const float* y, int64_t n, float* grad, float* loss) {
  if (!h || !X || !y || !grad || n <= 0 || n > h->cap || n % 64) return ITS_ERR_INVALID;
  its_ctx* ctx = h->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<float> x, yy;
  its_status st;
  if ((st = x.stage(ctx, X, n * kIn)) != ITS_OK) return st;
  if ((st = yy.stage(ctx, y, n)) != ITS_OK) return st;
  if ((st = mlpGradient(h, x.d, yy.d, BatchRows{0, 0, 0}, n)) != ITS_OK) return st;
  if (h->host && ptrClass(grad, ctx->device) == PtrClass::Pageable &&
      (!loss || ptrClass(loss, ctx->device) == PtrClass::Pageable)) {
    // one copy for the gradient, the loss and the flag (three to pageable memory took 40 us)
    ITS_CU(ctx, cudaMemcpyAsync(h->host, h->G, (kNumParams + 2) * 4, cudaMemcpyDeviceToHost, ctx->stream));
    ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
    std::memcpy(grad, h->host, kNumParams * 4);
    if (loss) *loss = h->host[kNumParams];
    int e;
    std::memcpy(&e, h->host + kNumParams + 1, 4);
    return e ? setError(ctx, ITS_ERR_TIMEOUT, "share network: a tensor-core wait ran out") : ITS_OK;
  }
  ITS_CU(ctx, cudaMemcpyAsync(grad, h->G, kNumParams * 4, cudaMemcpyDefault, ctx->stream));
  if (loss) ITS_CU(ctx, cudaMemcpyAsync(loss, h->loss, 4, cudaMemcpyDefault, ctx->stream));
  return checkErr(h);
}

// steps Adam steps on random batches (batch = capacity) of a resident dataset (n x 64
// normalised features, n targets; host or device). loss_curve (may be NULL) gets the
// mean squared error of every step.
its_status its_mlp_train(its_mlp* h, const float* X, const float* y, int64_t n, int64_t steps, float lr,
                         uint64_t seed, float* loss_curve) {
  if (!h || !X || !y || n <= 0 || steps < 0) return ITS_ERR_INVALID;
  its_ctx* ctx = h->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<float> x, yy;
  its_status st;
  if ((st = x.stage(ctx, X, n * kIn)) != ITS_OK) return st;
  if ((st = yy.stage(ctx, y, n)) != ITS_OK) return st;
  DevBuf<float> curve;
  if ((st = curve.alloc(ctx, steps > 0 ? steps : 1)) != ITS_OK) return st;
  for (int64_t s = 0; s < steps; ++s) {
    const BatchRows rows{n, seed, (uint64_t)s * (uint64_t)h->cap};
    if ((st = mlpGradient(h, x.d, yy.d, rows, h->cap)) != ITS_OK) return st;
    if ((st = mlpAdam(h, lr)) != ITS_OK) return st;
    ITS_CU(ctx, cudaMemcpyAsync(curve.p + s, h->loss, 4, cudaMemcpyDeviceToDevice, ctx->stream));
  }
  if (loss_curve && steps > 0)
    ITS_CU(ctx, cudaMemcpyAsync(loss_curve, curve.p, steps * 4, cudaMemcpyDefault, ctx->stream));
  return checkErr(h);
}

}  // extern "C"
