// The per-head products around the latent attention, for many rows, on tcgen05:
//   out[t, h, n] = sum_k a[t, h, k] w[h, n, k]   (* sigmoid(gate))      bfloat16 weights, float32 operand
// The float32 operand enters as two bfloat16 parts, its rounding and what the rounding left over, each multiplied with
// the weights into one 32-bit sum, so that it keeps 16 bits of mantissa (as in latent_mma.cu's mma.sync form).
//
// A CTA takes 128 rows x 128 columns of one head.  K goes through a ring of two stages of 64: eight warps load the
// operand's rows into registers a chunk ahead, split them and store both parts in the MMA's swizzled layout; the weights
// come by TMA; one lane issues eight MMAs per chunk (M = 128, N = 128, both parts).  The sums leave through the idle ring,
// a warp storing 128 bytes of a row at a time.  Two CTAs share a multiprocessor, so that one loads while the other
// stores: the product is bound by the operand's and the result's bytes, not by the tensor pipe.
// Measured, a latent attention layer over 1,801 rows of 16 heads (K 128 N 512 in front, K 512 N 128 behind): 356 -> 288 us, the
// two products together 125 before (mma.sync, the operand read and split again for every 64 columns), 57 now.
#include <cuda.h>
#include <math.h>

#include <mutex>

#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int HM = 128, HN = 128, HK = 64, HSTAGES = 2;
constexpr int PART_BYTES = HM * 128, STAGE_BYTES = 3 * PART_BYTES;      // upper parts, lower parts, weights
constexpr int WORKERS = 8, HTHREADS = (WORKERS + 1) * 32;
constexpr size_t HSMEM = (size_t)HSTAGES * STAGE_BYTES + 128;
constexpr int OUT_LD = 36;                                               // floats per row of a warp's 32 x 32 block on its way out

struct HeadArgs {
  void* out;
  const float* a;
  const float* gate;
  int* error;
  long long out_row, a_row, gate_row;
  int out_head, a_head, gate_head, gate_col, T, N, K, out_vec;
};

__device__ __forceinline__ uint32_t pack2(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ float sigmoid_of(float x) { return 1.0f / (1.0f + expf(-x)); }

template <typename O>
__global__ void __launch_bounds__(HTHREADS, 2)
head_tc_kernel(const __grid_constant__ CUtensorMap map_w, const HeadArgs args) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  if (base & 1023u) {                                  // the swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) atomicExch(args.error, 68);
    return;
  }
  const uint32_t bars = base + (uint32_t)HSTAGES * STAGE_BYTES;
  const uint32_t a_full = bars, w_full = bars + 16, empty = bars + 32, done = bars + 48, tmem_slot = bars + 56;
  volatile uint32_t* tmem_slot_ptr = (volatile uint32_t*)(smem_raw + (tmem_slot - base));
  const int warp = warp_number(), lane = threadIdx.x & 31;
  const int h = blockIdx.y, t0 = blockIdx.x * HM, n0 = blockIdx.z * HN;
  const int chunks = (args.K + HK - 1) / HK;
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    for (int s = 0; s < HSTAGES; ++s) { mbar_init(a_full + 8 * s, WORKERS); mbar_init(w_full + 8 * s, 1); mbar_init(empty + 8 * s, 1); }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == WORKERS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(HN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot_ptr);
  pdl_wait();

  if (warp == WORKERS) {
    if (elect_one()) {
      constexpr uint32_t IDESC = make_idesc(HM, HN);
      auto weights = [&](int c) {
        const int s = c & 1;
        mbar_expect_tx(w_full + 8 * s, PART_BYTES);
        tma_load_2d(base + s * STAGE_BYTES + 2 * PART_BYTES, &map_w, c * HK, h * args.N + n0, w_full + 8 * s);
      };
      int asked = 0;
      for (; asked < chunks && asked < HSTAGES; ++asked) weights(asked);
      bool ok = true;
      for (int c = 0; c < chunks; ++c) {
        const int s = c & 1;
        const uint32_t parity = (uint32_t)(c >> 1) & 1u;
        ok = mbar_wait(w_full + 8 * s, parity, args.error, 61) && mbar_wait(a_full + 8 * s, parity, args.error, 62);
        if (!ok) break;
        tc_fence_after();
        const uint32_t at = base + s * STAGE_BYTES;
        const uint64_t hi = make_desc(at), lo = make_desc(at + PART_BYTES), w = make_desc(at + 2 * PART_BYTES);
#pragma unroll
        for (int k = 0; k < HK / 16; ++k) {
          umma(tmem, lo + (uint64_t)(2 * k), w + (uint64_t)(2 * k), IDESC, (c > 0 || k > 0) ? 1u : 0u);
          umma(tmem, hi + (uint64_t)(2 * k), w + (uint64_t)(2 * k), IDESC, 1u);
        }
        umma_commit(empty + 8 * s);
        if (asked < chunks) {                          // this stage's next weights, once these products have read it
          ok = mbar_wait(empty + 8 * s, parity, args.error, 63);
          if (!ok) break;
          weights(asked++);
        }
      }
      umma_commit(done);
      if (!ok)                                         // nobody consumes any more: wait for the copies in flight
        for (int i = max(0, asked - HSTAGES); i < asked; ++i) mbar_wait(w_full + 8 * (i & 1), (uint32_t)(i >> 1) & 1u, args.error, 64);
    }
    __syncwarp();
  } else {
    // A worker's share of a chunk: four times four rows, eight lanes to a row, eight numbers to a lane.
    const int piece = lane & 7, sub = lane >> 3;       // 16-byte piece of bfloat16 (8 numbers), row within the warp's group of 4
    const float* rows_at = args.a + (size_t)h * args.a_head;
    float4 x[4][2];
    auto load = [&](int c) {
      const int k = c * HK + piece * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = t0 + i * 32 + warp * 4 + sub;
        x[i][0] = x[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < args.T && k < args.K) {                // K is a multiple of 8: a piece is whole
          const float4* src = reinterpret_cast<const float4*>(rows_at + (size_t)t * args.a_row + k);
          x[i][0] = src[0];
          x[i][1] = src[1];
        }
      }
    };
    load(0);
    bool ok = true;
    for (int c = 0; c < chunks && ok; ++c) {
      const int s = c & 1;
      if (c >= HSTAGES) {
        if (lane == 0) ok = mbar_wait(empty + 8 * s, (uint32_t)((c >> 1) & 1) ^ 1u, args.error, 65);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) break;
      }
      uint8_t* at = smem_raw + s * STAGE_BYTES;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = i * 32 + warp * 4 + sub;
        const float v[8] = {x[i][0].x, x[i][0].y, x[i][0].z, x[i][0].w, x[i][1].x, x[i][1].y, x[i][1].z, x[i][1].w};
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 up = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
          hi[e] = pack2(up);
          lo[e] = pack2(__floats2bfloat162_rn(v[2 * e] - __bfloat162float(up.x), v[2 * e + 1] - __bfloat162float(up.y)));
        }
        const int to = r * 128 + ((piece ^ (r & 7)) << 4);               // the 128-byte swizzle
        *reinterpret_cast<uint4*>(at + to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(at + PART_BYTES + to) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      if (c + 1 < chunks) load(c + 1);                 // on its way under the products
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full + 8 * s);
    }
    if (lane == 0) ok = ok && mbar_wait(done, 0u, args.error, 66);
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    if (ok) {
      tc_fence_after();
      const int quarter = warp & 3, half = warp >> 2;  // rows 32 quarter ..., columns 64 half ...
      float* stage = reinterpret_cast<float*>(smem_raw) + warp * 32 * OUT_LD;
      for (int c = half * 64; c < half * 64 + 64; c += 32) {
        uint32_t o[32];
        tmem_ld32(tmem + (uint32_t)c + ((uint32_t)(quarter * 32) << 16), o);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(stage + lane * OUT_LD + j) =
              make_float4(__uint_as_float(o[j]), __uint_as_float(o[j + 1]), __uint_as_float(o[j + 2]), __uint_as_float(o[j + 3]));
        __syncwarp();
#pragma unroll 2
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + sub, t = t0 + quarter * 32 + r, n = n0 + c + piece * 4;
          const float4 v4 = *reinterpret_cast<const float4*>(stage + r * OUT_LD + piece * 4);
          if (t >= args.T || n >= args.N) continue;
          float v[4] = {v4.x, v4.y, v4.z, v4.w};
          if (args.gate) {
            const float* g = args.gate + (size_t)t * args.gate_row + (size_t)h * args.gate_head;
            if (args.gate_col == 0) {
              const float f = sigmoid_of(g[0]);
#pragma unroll
              for (int e = 0; e < 4; ++e) v[e] *= f;
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (n + e < args.N) v[e] *= sigmoid_of(g[(size_t)(n + e) * args.gate_col]);
            }
          }
          O* dst = reinterpret_cast<O*>(args.out) + (size_t)t * args.out_row + (size_t)h * args.out_head + n;
          if (args.out_vec && n + 4 <= args.N) {
            if constexpr (sizeof(O) == 4) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            else *reinterpret_cast<uint2*>(dst) = make_uint2(pack2(__floats2bfloat162_rn(v[0], v[1])), pack2(__floats2bfloat162_rn(v[2], v[3])));
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n + e < args.N) dst[e] = from_float<O>(v[e]);
          }
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == WORKERS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(HN) : "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
int* g_error_host = nullptr;
int* g_error_dev = nullptr;
std::mutex g_mutex;
AykPerDevice g_configured;

int setup() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t err = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (err != cudaSuccess || fn == nullptr || q != cudaDriverEntryPointSuccess)
      return ayk_fail("ayk_head_matmul_tc: cuTensorMapEncodeTiled is not available from this driver");
    g_encode = (EncodeTiledFn)fn;
  }
  if (!g_error_host) {
    cudaError_t err = cudaHostAlloc((void**)&g_error_host, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
    if (err != cudaSuccess) return ayk_fail("ayk_head_matmul_tc: cudaHostAlloc: %s", cudaGetErrorString(err));
    *g_error_host = 0;
    err = cudaHostGetDevicePointer((void**)&g_error_dev, g_error_host, 0);
    if (err != cudaSuccess) return ayk_fail("ayk_head_matmul_tc: cudaHostGetDevicePointer: %s", cudaGetErrorString(err));
  }
  if (!g_configured.here()) {
    cudaError_t err = cudaFuncSetAttribute(head_tc_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HSMEM);
    if (err == cudaSuccess) err = cudaFuncSetAttribute(head_tc_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HSMEM);
    if (err != cudaSuccess) return ayk_fail("ayk_head_matmul_tc: shared memory %zu: %s", HSMEM, cudaGetErrorString(err));
    g_configured.here() = true;
  }
  return 0;
}

}  // namespace

AYK_EXPORT int ayk_head_tc_error() { return g_error_host ? *g_error_host : 0; }

// The operand's rows and heads on 16-byte boundaries, the weights' too; 64 rows and more, half a tile.  Measured against the
// mma.sync form at 64 to 1,024 rows of 12 shapes (1 to 128 heads, N 32 to 512, K 40 to 512), it is never behind: (us, mma.sync
// and this; 64 rows, 128, 512) 16 heads, N 512, K 128: 7.7 4.9, 8.9 5.3, 14.9 7.6; 16 heads, N 128, K 512: 25.9 9.5, 26.0 9.9, 28.5
// 10.1; 128 heads, N 512, K 128: 17.1 12.5, 31.4 14.5, 119 56.7; the least, 2 heads, N 72, K 40: 4.6 4.2, 4.6 4.5, 4.6 4.5.
AYK_EXPORT int ayk_head_matmul_tc_takes(const void* a, long long a_row, int a_head, const void* w, int T, int H, int N, int K) {
  return T >= 64 && K % 8 == 0 && a_row % 4 == 0 && a_head % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)w % 16 == 0 &&
         (long long)H * N < (1ll << 31);
}

// As ayk_head_matmul for bfloat16 weights.
AYK_EXPORT int ayk_head_matmul_tc(void* out, long long out_row, int out_head, const float* a, long long a_row, int a_head, const void* w,
                                  const float* gate, long long gate_row, int gate_head, int gate_col, int T, int H, int N, int K,
                                  int out_dtype, cudaStream_t stream) {
  if (T == 0 || H == 0 || N == 0) return 0;
  AYK_REQUIRE(ayk_head_matmul_tc_takes(a, a_row, a_head, w, T, H, N, K), "ayk_head_matmul_tc: %d rows, K %d, or the operands' layout, are not taken", T, K);
  AYK_REQUIRE(out_dtype == AYK_DTYPE_F32 || out_dtype == AYK_DTYPE_BF16, "ayk_head_matmul_tc: unknown dtype %d", out_dtype);
  dim3 grid((T + HM - 1) / HM, H, (N + HN - 1) / HN);
  AYK_REQUIRE(H <= 65535 && grid.z <= 65535, "ayk_head_matmul_tc: too many heads or columns");
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (setup() != 0) return -1;
  }
  CUtensorMap mw;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)H * N};
  cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)HK, (cuuint32_t)HN};
  cuuint32_t elem[2] = {1, 1};
  CUresult r = g_encode(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return ayk_fail("ayk_head_matmul_tc: cuTensorMapEncodeTiled failed with %d", (int)r);
  const int bytes = out_dtype == AYK_DTYPE_F32 ? 4 : 2;
  const int out_vec = (uintptr_t)out % (4 * bytes) == 0 && out_row % 4 == 0 && out_head % 4 == 0;
  HeadArgs args{out, a, gate, g_error_dev, out_row, a_row, gate_row, out_head, a_head, gate_head, gate_col, T, N, K, out_vec};
  if (out_dtype == AYK_DTYPE_F32) ayk_launch(head_tc_kernel<float>, grid, dim3(HTHREADS), HSMEM, stream, mw, args);
  else ayk_launch(head_tc_kernel<__nv_bfloat16>, grid, dim3(HTHREADS), HSMEM, stream, mw, args);
  return ayk_check_launch("ayk_head_matmul_tc");
}
