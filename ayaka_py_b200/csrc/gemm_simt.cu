// C[M,N] = act(A[M,K] * W[N,K]^T + bias[N]) (+ residual[M,N]) on the FP32 FMA
// pipes: the matrix product of the true 32-bit path (no TF32, no tensor cores),
// also usable with bfloat16 operands.  The reference's linear layers are
// F.linear (layers/linear/methods.py:73-76); the activation formulas are those
// of kernel/triton/activation.py:145-154, applied in 32-bit in the epilogue.
//
// float32 operands: gemm_f32_kernel below.  bfloat16 operands (K no multiple of 8): gemm_simt_kernel, tile
// 64x64x16, 256 threads, 4x4 outputs per thread, products accumulated in ascending k in one float per output.
// In both a row's result does not depend on which other rows are in the batch.
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16;

// ---------------------------------------------------------------- float32 --
// A tile of TM x 64 outputs: of every slab of 32 k each of the block's eight warps takes its own four, so that a tile keeps
// eight warps busy whatever its height.  A thread holds TM / 4 x 8 sums and reads TM / 4 + 8 float4 from shared memory for
// 32 * (TM / 4) products.  Slabs arrive by cp.async, three ahead; the next is asked for behind the first of a slab's products.
// At the end the eight warps' sums meet in shared memory and are added in one order, ((0 + 1) + (2 + 3)) + ((4 + 5) + (6 + 7)),
// the same for every TM: the height is chosen by the row count, a row's result is not.
//
// Bound by the FP32 pipes (128 FMA a clock and multiprocessor) and by what shared memory hands out, 128 bytes a clock: a
// thread's 8 x 8 sums need four clocks for each of 16 float4 where the products need 64; and, per tile, by how many
// multiprocessors have one.  Four groups of two warps and tiles of up to 64 rows gave a thread of 32 rows 4 x 8 sums, 12 float4
// for 128 products.  Measured, weights cold, in a row (us; before, now): K 768, N 2304: 1 row 12.5, 9.9; 32 rows 13.1, 10.4;
// 300 rows 49.8, 40.8; 377 rows 53.9, 40.8; 600 rows 74.9, 65.0; 1,200 rows 120, 125; N 3072: 377 rows 49.2, 52.4; 600 rows
// 93.4, 88.6; K 3072, N 768: 1 row 42.5, 30.7; 130 rows 47.1, 36.5; 377 rows 62.0, 55.5; 1,200 rows 183, 187.  Tried beside it:
// 16 x 8 sums a thread in tiles of 64 rows, one block to a multiprocessor (2,048 rows, N 4096, K 1024: 496 against 450);
// fma.rn.f32x2 on pairs of k, which takes twice the registers and so 4 x 8 sums (526); slabs of 64 (526).
constexpr int FN = 64, FK = 32, FLD = FK + 4, FSTAGES = 4, FWARPS = 8;       // rows of 36 floats: eight neighbours' 16-byte pieces lie on different banks
constexpr int FSUM = FN + 8;             // floats per row of the warps' sums: a warp's four rows of eight lie on different banks
constexpr int f32_stage_floats(int tm) { return (tm + FN) * FLD; }
constexpr size_t f32_smem(int tm) {
  const size_t ring = (size_t)FSTAGES * f32_stage_floats(tm), sums = (size_t)FWARPS * tm * FSUM;
  return (ring > sums ? ring : sums) * sizeof(float);
}

__device__ __forceinline__ void f32_copy16(float* dst, const float* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void f32_copy4(float* dst, const float* src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 4 : 0) : "memory");
}

template <int TM, bool VEC>
__global__ void __launch_bounds__(256, 2)
gemm_f32_kernel(float* C, const float* A, const float* __restrict__ W, const float* __restrict__ bias,
                const float* residual,               // C and residual may be one buffer (the residual stream in place)
                int M, int N, int K, int act) {
  constexpr int RM = TM / 4;
  extern __shared__ __align__(16) float f32_tiles[];
  if (gridDim.x * gridDim.y <= AYK_FEW_BLOCKS) pdl_trigger();
  const int tid = threadIdx.x, warp = tid >> 5, tn = tid & 7, tm = (tid >> 3) & 3;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * FN;
  const int slabs = (K + FK - 1) / FK;
  // One slab into buffer b; rows past the matrices' ends and k past K are zeros.  In 16-byte pieces a thread always brings
  // the same piece of the same rows, whose addresses it works out once.
  constexpr int COPIES = ((TM + FN) * (FK / 4) + 255) / 256;
  const float* src[COPIES];
  bool there[COPIES];
  if (VEC) {
#pragma unroll
    for (int j = 0; j < COPIES; ++j) {
      const int row = (tid >> 3) + 32 * j;
      const bool of_a = row < TM;
      const int at = of_a ? m0 + row : n0 + row - TM;
      there[j] = at < (of_a ? M : N);
      src[j] = (there[j] ? (of_a ? A : W) + (size_t)at * K : A) + (tid & 7) * 4;
    }
  }
  auto fetch = [&](int slab, int b) {
    float* to = f32_tiles + b * f32_stage_floats(TM);
    if (VEC) {
      const int k = slab * FK + (tid & 7) * 4;
#pragma unroll
      for (int j = 0; j < COPIES; ++j) {
        const int row = (tid >> 3) + 32 * j;
        const bool on = there[j] && k < K;
        if (row < TM + FN) f32_copy16(to + row * FLD + (tid & 7) * 4, on ? src[j] + slab * FK : A, on);
      }
    } else {
      for (int i = tid; i < (TM + FN) * FK; i += 256) {
        const int row = i / FK, c = i % FK, k = slab * FK + c;
        const bool of_a = row < TM;
        const int at = of_a ? m0 + row : n0 + row - TM;
        const bool on = at < (of_a ? M : N) && k < K;
        f32_copy4(to + row * FLD + c, on ? (of_a ? A : W) + (size_t)at * K + k : A, on);
      }
    }
  };
  float acc[RM][8];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  pdl_wait();
#pragma unroll
  for (int st = 0; st < FSTAGES - 1; ++st) {
    if (st < slabs) fetch(st, st);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int slab = 0; slab < slabs; ++slab) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();                                 // this slab is there for everybody; the one before has been read
    const float* as = f32_tiles + (slab % FSTAGES) * f32_stage_floats(TM) + tm * FLD + warp * 4;
    const float* ws = f32_tiles + (slab % FSTAGES) * f32_stage_floats(TM) + (TM + tn) * FLD + warp * 4;
    float4 a[RM];
#pragma unroll
    for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * 4 * FLD);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 w = *reinterpret_cast<const float4*>(ws + j * 8 * FLD);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        acc[i][j] = fmaf(a[i].x, w.x, acc[i][j]);
        acc[i][j] = fmaf(a[i].y, w.y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, w.z, acc[i][j]);
        acc[i][j] = fmaf(a[i].w, w.w, acc[i][j]);
      }
      if (j == 0) {
        if (slab + FSTAGES - 1 < slabs) fetch(slab + FSTAGES - 1, (slab + FSTAGES - 1) % FSTAGES);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                   // the ring is free for the sums
  float* mine = f32_tiles + warp * TM * FSUM;
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) mine[(tm + 4 * i) * FSUM + tn + 8 * j] = acc[i][j];
  __syncthreads();
  const int col = tid & (FN - 1), n = n0 + col;
  if (n >= N) return;
  const float b = bias ? bias[n] : 0.f;
#pragma unroll
  for (int r = tid / FN; r < TM; r += 256 / FN) {
    const int m = m0 + r;
    if (m >= M) break;
    const float* at = f32_tiles + r * FSUM + col;
    auto sum = [&](int g) { return at[g * TM * FSUM]; };
    float v = (((sum(0) + sum(1)) + (sum(2) + sum(3))) + ((sum(4) + sum(5)) + (sum(6) + sum(7)))) + b;
    v = apply_activation(v, act);
    if (residual) v += residual[(size_t)m * N + n];
    C[(size_t)m * N + n] = v;
  }
}

// Rows per tile: the least work on the fullest multiprocessor, a multiprocessor taking whole tiles one after the other
// (two at a time do not make it faster: the pipes are the bound).  Lower tiles read more of shared memory per product and
// pay the same for a slab's barrier, which is what the factors say: 377 rows, K 768, N 3072 by tiles of 32, 16 and 8 rows take
// 52, 63 and 90 us; 130 rows, N 2304 (180, 324 and 612 tiles) 26.8, 25.8 and 31.2; 32 rows 16.4, 12.3 and 10.4.
int f32_rows(int M, int N, int sms) {
  const int heights[3] = {32, 16, 8};
  const double factor[3] = {1.0, 1.25, 1.9};
  int best = 32;
  double least = -1.0;
  for (int i = 0; i < 3; ++i) {
    const long tiles = (long)((M + heights[i] - 1) / heights[i]) * ((N + FN - 1) / FN);
    const double work = (double)((tiles + sms - 1) / sms) * heights[i] * factor[i];
    if (least < 0 || work < least) { least = work; best = heights[i]; }
  }
  return best;
}

template <int TM, bool VEC>
int launch_f32(float* C, const float* A, const float* W, const float* bias, const float* residual, int M, int N, int K, int act,
               cudaStream_t stream) {
  static AykPerDevice configured;
  bool& done = configured.here();
  if (!done) {
    cudaError_t err = cudaFuncSetAttribute(gemm_f32_kernel<TM, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f32_smem(TM));
    if (err != cudaSuccess) return ayk_fail("ayk_gemm_simt: shared memory %zu: %s", f32_smem(TM), cudaGetErrorString(err));
    done = true;
  }
  constexpr int MOST = 65535 * TM;                   // rows of one launch
  for (int m = 0;; m += MOST) {
    const int rows = M - m < MOST ? M - m : MOST;
    dim3 grid((N + FN - 1) / FN, (rows + TM - 1) / TM);
    ayk_launch_as(grid.x * grid.y <= AYK_FEW_BLOCKS, gemm_f32_kernel<TM, VEC>, grid, dim3(256), f32_smem(TM), stream, C + (size_t)m * N,
                  A + (size_t)m * K, W, bias, residual ? residual + (size_t)m * N : nullptr, rows, N, K, act);
    if (M - m <= MOST) break;
  }
  return ayk_check_launch("ayk_gemm_simt");
}

template <bool VEC>
int launch_f32_rows(float* C, const float* A, const float* W, const float* bias, const float* residual, int M, int N, int K, int act,
                    cudaStream_t stream) {
  switch (f32_rows(M, N, ayk_sm_count())) {
    case 32: return launch_f32<32, VEC>(C, A, W, bias, residual, M, N, K, act, stream);
    case 16: return launch_f32<16, VEC>(C, A, W, bias, residual, M, N, K, act, stream);
    default: return launch_f32<8, VEC>(C, A, W, bias, residual, M, N, K, act, stream);
  }
}

// --------------------------------------------------------------- bfloat16 --

__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
  uint2 x = *reinterpret_cast<const uint2*>(p);
  __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&x.x);
  __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&x.y);
  v[0] = __bfloat162float(a.x); v[1] = __bfloat162float(a.y);
  v[2] = __bfloat162float(b.x); v[3] = __bfloat162float(b.y);
}

template <typename TA, typename TW, typename TO, bool VEC>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(TO* C, const TA* A, const TW* __restrict__ W,
                 const float* __restrict__ bias, const float* residual,      // C and residual may be one buffer (the residual stream in place)
                 int M, int N, int K, int act) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  if (gridDim.x * gridDim.y <= AYK_FEW_BLOCKS) pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int lr = tid >> 2, lk = (tid & 3) * 4;       // loader: row of the tile, k offset
  const int tm = (tid >> 4) * 4, tn = (tid & 15) * 4;  // this thread's 4x4 outputs
  float acc[4][4] = {};

  for (int k0 = 0; k0 < K; k0 += BK) {
    float a[4] = {0.f, 0.f, 0.f, 0.f}, w[4] = {0.f, 0.f, 0.f, 0.f};
    const int gm = m0 + lr, gn = n0 + lr, gk = k0 + lk;
    if (VEC) {
      if (gm < M && gk < K) load4(A + (size_t)gm * K + gk, a);
      if (gn < N && gk < K) load4(W + (size_t)gn * K + gk, w);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (gm < M && gk + j < K) a[j] = to_float<TA>(A[(size_t)gm * K + gk + j]);
        if (gn < N && gk + j < K) w[j] = to_float<TW>(W[(size_t)gn * K + gk + j]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      As[lk + j][lr] = a[j];
      Ws[lk + j][lr] = w[j];
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float4 av = *reinterpret_cast<const float4*>(&As[kk][tm]);
      float4 wv = *reinterpret_cast<const float4*>(&Ws[kk][tn]);
      float ar[4] = {av.x, av.y, av.z, av.w}, wr[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], wr[j], acc[i][j]);
    }
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int m = m0 + tm + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int n = n0 + tn + j;
      if (n >= N) continue;
      float v = acc[i][j] + (bias ? bias[n] : 0.f);
      v = apply_activation(v, act);
      if (residual) v += residual[(size_t)m * N + n];
      C[(size_t)m * N + n] = from_float<TO>(v);
    }
  }
}

template <typename TA, typename TW, typename TO>
int launch(void* C, const void* A, const void* W, const float* bias, const float* residual, int M,
           int N, int K, int act, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  bool vec = (K % 4 == 0) && ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0);
  if (vec)
    ayk_launch_as(grid.x * grid.y <= AYK_FEW_BLOCKS, gemm_simt_kernel<TA, TW, TO, true>, grid, dim3(256), 0, stream, (TO*)C, (const TA*)A, (const TW*)W, bias,
               residual, M, N, K, act);
  else
    ayk_launch_as(grid.x * grid.y <= AYK_FEW_BLOCKS, gemm_simt_kernel<TA, TW, TO, false>, grid, dim3(256), 0, stream, (TO*)C, (const TA*)A, (const TW*)W, bias,
               residual, M, N, K, act);
  return ayk_check_launch("ayk_gemm_simt");
}

}  // namespace

// in_dtype: dtype of A and W; out_dtype: dtype of C.  bias and residual are
// float32 or null; residual may alias C when out_dtype is float32.
AYK_EXPORT int ayk_gemm_simt(void* C, const void* A, const void* W, const float* bias,
                             const float* residual, int M, int N, int K, int act, int in_dtype,
                             int out_dtype, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  AYK_REQUIRE(K >= 1, "ayk_gemm_simt: K must be positive");
  AYK_REQUIRE((M + BM - 1) / BM <= 65535, "ayk_gemm_simt: M = %d exceeds %d rows", M, 65535 * BM);
  if (in_dtype == AYK_DTYPE_F32 && out_dtype == AYK_DTYPE_F32) {
    const bool vec = K % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
    return vec ? launch_f32_rows<true>((float*)C, (const float*)A, (const float*)W, bias, residual, M, N, K, act, stream)
               : launch_f32_rows<false>((float*)C, (const float*)A, (const float*)W, bias, residual, M, N, K, act, stream);
  }
  if (in_dtype == AYK_DTYPE_BF16 && out_dtype == AYK_DTYPE_F32)
    return launch<__nv_bfloat16, __nv_bfloat16, float>(C, A, W, bias, residual, M, N, K, act, stream);
  if (in_dtype == AYK_DTYPE_BF16 && out_dtype == AYK_DTYPE_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(C, A, W, bias, residual, M, N, K, act, stream);
  return ayk_fail("ayk_gemm_simt: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
}
