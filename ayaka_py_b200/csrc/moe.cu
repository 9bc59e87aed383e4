// Mixture of experts: routing, the plan of a step's (token, choice) pairs sorted by expert, the
// grouped products over the sorted rows, the gated activation and the weighted sum.
//
// Routing: the ``top`` largest of a token's router logits (the lower index wins a tie), weights =
// softmax over the chosen logits only; all 32-bit.  Nothing of the routing goes to the host: the
// plan kernel counts the pairs of every expert, lays them out expert by expert (``sorted``: place
// -> pair), and cuts them into tiles of TILE_ROWS rows of one expert each; the grouped product is
// launched with the largest number of tiles that the pair count allows and its surplus blocks leave.
//
// An expert's activation: g = min(gate, limit), u = clamp(up, -limit, limit),
// y = g * sigmoid(slope * g) * (u + plus).  An infinite limit clamps nothing; slope 1 and plus 0 make it
// silu(gate) * up.  Experts without a gate (a plain product with an activation of common.cuh in its epilogue) run
// through the same kernels.
//
// Routing by sigmoid scores in groups (moe_route_scored_kernel): s = sigmoid(z); experts are ranked by
// s + correction[e]; the experts are ``groups`` equal runs of consecutive experts, a run's score is the sum of its
// two largest ranking scores, and only experts of the ``keep`` best runs can be chosen; the weights are
// the chosen s divided by their sum, times a factor.
//
// The same kernel with softmax scores: s = softmax(z) over all experts; with a correction experts are ranked by
// s + correction[e], without one by z itself (the same order, also where s underflows).  Sigmoid scores without a
// correction rank by z too unless groups count by their two best.  Two more things are
// parameters of both: a run's score may be its largest ranking score alone, and the weights may be the chosen s as they are,
// times the factor.
#include <math.h>

#include "common.cuh"

namespace {

__device__ __forceinline__ float sigmoidf(float z) { return 1.0f / (1.0f + expf(-z)); }

__device__ __forceinline__ float glu_limited(float g, float u, float limit, float slope, float plus) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g * sigmoidf(slope * g) * (u + plus);
}

constexpr int MAX_TOP = 16;
constexpr int TILE_ROWS = 32;

// ------------------------------------------------------------------- route --
// A warp per token.
__global__ void __launch_bounds__(128)
moe_route_kernel(int* __restrict__ ids, float* __restrict__ weights, const float* logits, long long stride,
                 int T, int E, int top) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  const float* z = logits + (size_t)t * stride;
  int chosen[MAX_TOP];
  float value[MAX_TOP];
#pragma unroll
  for (int k = 0; k < MAX_TOP; ++k) {
    if (k >= top) break;
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      bool taken = false;
#pragma unroll
      for (int j = 0; j < MAX_TOP; ++j) taken |= (j < k && chosen[j] == e);
      const float v = z[e];
      if (!taken && (v > best || (v == best && e < at) || at == 0x7fffffff)) { best = v; at = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (oa != 0x7fffffff && (at == 0x7fffffff || ob > best || (ob == best && oa < at))) { best = ob; at = oa; }
    }
    chosen[k] = at;
    value[k] = best;
  }
  if (lane == 0) {
    float sum = 0.f, w[MAX_TOP];
#pragma unroll
    for (int k = 0; k < MAX_TOP; ++k) {
      if (k >= top) break;
      w[k] = expf(value[k] - value[0]);          // value[0] is the largest
      sum += w[k];
    }
#pragma unroll
    for (int k = 0; k < MAX_TOP; ++k) {
      if (k >= top) break;
      ids[(size_t)t * top + k] = chosen[k];
      weights[(size_t)t * top + k] = w[k] / sum;
    }
  }
}

// A warp per token.  Lane g holds the score of run g (at most 32 runs); the runs that may be chosen are a
// bit mask that every lane holds; then the same repeated arg-max as above over the allowed experts' ranking
// scores (the lower index wins a tie).
template <bool SOFTMAX>
__global__ void __launch_bounds__(128)
moe_route_scored_kernel(int* __restrict__ ids, float* __restrict__ weights, const float* logits, long long stride,
                        const float* __restrict__ correction, int T, int E, int top, int groups, int keep, int group_best,
                        int normalize, float factor) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  const float* z = logits + (size_t)t * stride;
  const int per = E / groups;
  float zmax = 0.f, inv_sum = 1.f;
  if (SOFTMAX) {
    float m = -INFINITY, sum = 0.f;
    for (int e = lane; e < E; e += 32) m = fmaxf(m, z[e]);
    zmax = warp_max(m);
    for (int e = lane; e < E; e += 32) sum += expf(z[e] - zmax);
    inv_sum = 1.0f / warp_sum(sum);
  }
  auto score = [&](int e) { return SOFTMAX ? expf(z[e] - zmax) * inv_sum : sigmoidf(z[e]); };
  // without a correction the logits rank alike, also where scores underflow or saturate (sums of two scores need the scores)
  const bool by_logit = !correction && (SOFTMAX || keep >= groups || group_best == 1);
  auto ranking = [&](int e) {
    if (by_logit) return z[e];
    return score(e) + (correction ? correction[e] : 0.f);
  };
  unsigned allowed = 0xffffffffu;
  if (keep < groups) {
    float mine = -INFINITY;                    // lane g: run g's largest ranking score, or the sum of its two largest
    for (int g = 0; g < groups; ++g) {
      float best = -INFINITY, second = -INFINITY;
      for (int e = g * per + lane; e < (g + 1) * per; e += 32) {
        const float v = ranking(e);
        if (v > best) { second = best; best = v; } else if (v > second) second = v;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o), os = __shfl_xor_sync(0xffffffffu, second, o);
        const float hi = fmaxf(best, ob), lo = fminf(best, ob);
        second = fmaxf(lo, fmaxf(second, os));
        best = hi;
      }
      const float total = (group_best == 2 && per > 1) ? best + second : best;
      if (lane == g) mine = total;
    }
    int rank = 0;                              // runs that come before mine: a larger score, or the same and a lower index
    for (int g = 0; g < groups; ++g) {
      const float other = __shfl_sync(0xffffffffu, mine, g);
      rank += (other > mine || (other == mine && g < lane)) ? 1 : 0;
    }
    allowed = __ballot_sync(0xffffffffu, lane < groups && rank < keep);
  }
  int chosen[MAX_TOP];
  float value[MAX_TOP];
#pragma unroll
  for (int k = 0; k < MAX_TOP; ++k) {
    if (k >= top) break;
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      bool taken = !((allowed >> (e / per)) & 1u);
#pragma unroll
      for (int j = 0; j < MAX_TOP; ++j) taken |= (j < k && chosen[j] == e);
      const float v = ranking(e);
      if (!taken && (v > best || (v == best && e < at) || at == 0x7fffffff)) { best = v; at = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (oa != 0x7fffffff && (at == 0x7fffffff || ob > best || (ob == best && oa < at))) { best = ob; at = oa; }
    }
    chosen[k] = at;
    value[k] = score(at);
  }
  if (lane == 0) {
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < MAX_TOP; ++k) {
      if (k >= top) break;
      sum += value[k];
    }
    const float inv = normalize ? factor / (sum + 1e-20f) : factor;
#pragma unroll
    for (int k = 0; k < MAX_TOP; ++k) {
      if (k >= top) break;
      ids[(size_t)t * top + k] = chosen[k];
      weights[(size_t)t * top + k] = value[k] * inv;
    }
  }
}

// -------------------------------------------------------------------- plan --
// One block.  tiles[0] = number of tiles; tile i: expert tiles[1 + 3 i], first sorted row
// tiles[2 + 3 i], rows tiles[3 + 3 i].
__global__ void __launch_bounds__(1024)
moe_plan_kernel(int* __restrict__ sorted, int* __restrict__ tiles, const int* ids, int P, int E) {
  extern __shared__ int sh[];
  int* count = sh;          // [E]
  int* start = sh + E;      // [E]
  int* cursor = sh + 2 * E; // [E]
  pdl_trigger();
  for (int e = threadIdx.x; e < E; e += blockDim.x) { count[e] = 0; cursor[e] = 0; }
  pdl_wait();
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) atomicAdd(&count[ids[p]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int off = 0, n = 0;
    for (int e = 0; e < E; ++e) {
      const int c = count[e];
      start[e] = off;
      for (int r = 0; r < c; r += TILE_ROWS) {
        tiles[1 + 3 * n] = e;
        tiles[2 + 3 * n] = off + r;
        tiles[3 + 3 * n] = min(TILE_ROWS, c - r);
        ++n;
      }
      off += c;
    }
    tiles[0] = n;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int e = ids[p];
    sorted[start[e] + atomicAdd(&cursor[e], 1)] = p;     // a row's result does not depend on its place
  }
}

// The plan for the product that runs on tcgen05 (gemm_tc_prefill, grouped form): every expert's pairs
// start at a multiple of PAD_ROWS rows, so that each 128-row tile of the gathered rows belongs to one
// expert.  row_of_pair[p]: the pair's row in that layout; w_rows1 / w_rows2 [max_tiles]: per tile the first
// weight row of its expert in the two stacked weights (n1 and n2 rows per expert; 0 for tiles past the end).
constexpr int PAD_ROWS = 128;

__global__ void __launch_bounds__(1024)
moe_plan_padded_kernel(int* __restrict__ row_of_pair, int* __restrict__ w_rows1, int* __restrict__ w_rows2,
                       const int* ids, int P, int E, int n1, int n2, int max_tiles) {
  extern __shared__ int sh[];
  int* count = sh;          // [E]
  int* start = sh + E;      // [E]
  int* cursor = sh + 2 * E; // [E]
  pdl_trigger();
  for (int e = threadIdx.x; e < E; e += blockDim.x) { count[e] = 0; cursor[e] = 0; }
  pdl_wait();
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) atomicAdd(&count[ids[p]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int e = 0; e < E; ++e) {
      start[e] = n * PAD_ROWS;
      for (int r = 0; r < count[e]; r += PAD_ROWS) {
        if (n < max_tiles) { w_rows1[n] = e * n1; w_rows2[n] = e * n2; }
        ++n;
      }
    }
    w_rows1[max_tiles] = w_rows2[max_tiles] = min(n, max_tiles);       // tiles that hold rows: the products stop there
    for (; n < max_tiles; ++n) { w_rows1[n] = 0; w_rows2[n] = 0; }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int e = ids[p];
    row_of_pair[p] = start[e] + atomicAdd(&cursor[e], 1);     // a row's result does not depend on its place
  }
}

// out[row_of_pair[p], :] = in[p / top, :], bfloat16 rows of d elements (d a multiple of 8); a warp per pair.  With
// row_scale: row_scale[row_of_pair[p]] = weights[p].
__global__ void __launch_bounds__(256)
moe_gather_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* in, long long in_stride,
                  const int* row_of_pair, float* __restrict__ row_scale, const float* weights, int P,
                  int top, int d) {
  pdl_trigger();
  pdl_wait();
  const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (p >= P) return;
  const uint4* src = reinterpret_cast<const uint4*>(in + (size_t)(p / top) * in_stride);
  const int to = row_of_pair[p];
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)to * d);
  if (row_scale && lane == 0) row_scale[to] = weights[p];
  for (int i = lane; i < d / 8; i += 32) dst[i] = src[i];
}

// --------------------------------------------------------- grouped product --
// out[o(s), n] = sum_k a[r(s), k] * w[expert, n, k] over the sorted rows s of a tile; w holds N_w
// rows per expert.  GLU: w rows [0, N) are the gate, [N, 2N) the up projection, and the output is
// the activation of the pair.  gather: r(s) = sorted[s] / top (rows of tokens), else s.  scatter:
// o(s) = sorted[s] (the pair's own row), else s.  early: the pair's weight multiplies its products ahead of the
// activation (null: nothing does).  On the FP32 pipes with 32-bit sums.
constexpr int BN = 64, BK = 32;

template <typename T, typename O, bool GLU>
__global__ void __launch_bounds__(256)
moe_gemm_kernel(O* __restrict__ out, const T* a, long long a_stride, const T* __restrict__ w,
                const int* sorted, const int* tiles, int top, int gather, int scatter, int N,
                int N_w, int Kd, float limit, float slope, float plus, int act, const float* early) {
  __shared__ float factor[TILE_ROWS];
  __shared__ float As[BK][TILE_ROWS + 1];
  __shared__ float Bs[GLU ? 2 : 1][BK][BN + 1];
  __shared__ int a_row[TILE_ROWS], o_row[TILE_ROWS];
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= tiles[0]) return;
  const int e = tiles[1 + 3 * blockIdx.x], s0 = tiles[2 + 3 * blockIdx.x], rows = tiles[3 + 3 * blockIdx.x];
  const int n0 = blockIdx.y * BN;
  const int tid = threadIdx.x;
  if (tid < TILE_ROWS) {
    const int pair = tid < rows ? sorted[s0 + tid] : -1;
    a_row[tid] = tid < rows ? (gather ? pair / top : s0 + tid) : -1;
    factor[tid] = early && tid < rows ? early[pair] : 1.f;
    o_row[tid] = tid < rows ? (scatter ? pair : s0 + tid) : -1;
  }
  __syncthreads();
  const T* we = w + (size_t)e * N_w * Kd;
  const int ty = tid >> 4, tx = tid & 15;        // rows ty * 2 + {0, 1}; columns tx + 16 * {0 .. 3}
  float acc[GLU ? 2 : 1][2][4];
#pragma unroll
  for (int g = 0; g < (GLU ? 2 : 1); ++g)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[g][i][j] = 0.f;

  for (int k0 = 0; k0 < Kd; k0 += BK) {
    {   // A: 32 rows x 32 k
      const int kk = tid & 31;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = (tid >> 5) + 8 * i;
        const int src = a_row[r];
        As[kk][r] = (src >= 0 && k0 + kk < Kd) ? to_float<T>(a[(size_t)src * a_stride + k0 + kk]) : 0.f;
      }
    }
#pragma unroll
    for (int g = 0; g < (GLU ? 2 : 1); ++g) {   // B: 64 n x 32 k
      const int kk = tid & 31;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int n = (tid >> 5) + 8 * i;
        Bs[g][kk][n] = (n0 + n < N && k0 + kk < Kd) ? to_float<T>(we[(size_t)(g * N + n0 + n) * Kd + k0 + kk]) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < BK; ++kk) {
      const float a0 = As[kk][ty * 2], a1 = As[kk][ty * 2 + 1];
#pragma unroll
      for (int g = 0; g < (GLU ? 2 : 1); ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float b = Bs[g][kk][tx + 16 * j];
          acc[g][0][j] = fmaf(a0, b, acc[g][0][j]);
          acc[g][1][j] = fmaf(a1, b, acc[g][1][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int dst = o_row[ty * 2 + i];
    if (dst < 0) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= N) continue;
      const float f = factor[ty * 2 + i];
      const float v = GLU ? glu_limited(f * acc[0][i][j], f * acc[GLU ? 1 : 0][i][j], limit, slope, plus) : apply_activation(f * acc[0][i][j], act);
      out[(size_t)dst * N + n] = from_float<O>(v);
    }
  }
}

// ------------------------------------- grouped product on the tensor cores --
// The same for bfloat16 operands: a tile of 32 sorted rows x 64 columns per block of four warps, each
// warp 32 rows x 16 columns as 2 x 2 fragments of mma.sync m16n8k16 with float32 sums; operands pass
// through shared memory as they lie in global memory (k innermost, rows padded by 8 elements so that
// a fragment's loads fall into different banks).
constexpr int TK = 64;                 // k per stage
constexpr int TLD = TK + 8;

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <typename O, bool GLU>
__global__ void __launch_bounds__(128)
moe_gemm_mma_kernel(O* __restrict__ out, const __nv_bfloat16* a, long long a_stride,
                    const __nv_bfloat16* __restrict__ w, const int* sorted, const int* tiles,
                    int top, int gather, int scatter, int N, int N_w, int Kd, float limit, float slope, float plus, int act,
                    const float* early) {
  __shared__ float factor[TILE_ROWS];
  __shared__ __align__(16) __nv_bfloat16 As[TILE_ROWS][TLD];
  __shared__ __align__(16) __nv_bfloat16 Bs[GLU ? 2 : 1][BN][TLD];
  __shared__ int a_row[TILE_ROWS], o_row[TILE_ROWS];
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= tiles[0]) return;
  const int e = tiles[1 + 3 * blockIdx.x], s0 = tiles[2 + 3 * blockIdx.x], rows = tiles[3 + 3 * blockIdx.x];
  const int n0 = blockIdx.y * BN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < TILE_ROWS) {
    const int pair = tid < rows ? sorted[s0 + tid] : -1;
    a_row[tid] = tid < rows ? (gather ? pair / top : s0 + tid) : -1;
    factor[tid] = early && tid < rows ? early[pair] : 1.f;
    o_row[tid] = tid < rows ? (scatter ? pair : s0 + tid) : -1;
  }
  __syncthreads();
  const __nv_bfloat16* we = w + (size_t)e * N_w * Kd;
  float acc[GLU ? 2 : 1][2][2][4];
#pragma unroll
  for (int g = 0; g < (GLU ? 2 : 1); ++g)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[g][i][j][c] = 0.f;
  const int gid = lane >> 2, tig = lane & 3;
  const uint4 zero = make_uint4(0, 0, 0, 0);

  for (int k0 = 0; k0 < Kd; k0 += TK) {
    // 16-byte pieces: a row of TK elements is 8 pieces (Kd is a multiple of 8)
    for (int i = tid; i < TILE_ROWS * (TK / 8); i += 128) {
      const int r = i >> 3, piece = i & 7;
      const int src = a_row[r], k = k0 + piece * 8;
      uint4 v = zero;
      if (src >= 0 && k < Kd) v = *reinterpret_cast<const uint4*>(a + (size_t)src * a_stride + k);
      *reinterpret_cast<uint4*>(&As[r][piece * 8]) = v;
    }
#pragma unroll
    for (int g = 0; g < (GLU ? 2 : 1); ++g)
      for (int i = tid; i < BN * (TK / 8); i += 128) {
        const int n = i >> 3, piece = i & 7;
        const int k = k0 + piece * 8;
        uint4 v = zero;
        if (n0 + n < N && k < Kd) v = *reinterpret_cast<const uint4*>(we + (size_t)(g * N + n0 + n) * Kd + k);
        *reinterpret_cast<uint4*>(&Bs[g][n][piece * 8]) = v;
      }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; kk += 16) {
      uint32_t af[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const __nv_bfloat16* base = &As[i * 16 + gid][kk + tig * 2];
        af[i][0] = *reinterpret_cast<const uint32_t*>(base);
        af[i][1] = *reinterpret_cast<const uint32_t*>(base + 8 * TLD);
        af[i][2] = *reinterpret_cast<const uint32_t*>(base + 8);
        af[i][3] = *reinterpret_cast<const uint32_t*>(base + 8 * TLD + 8);
      }
#pragma unroll
      for (int g = 0; g < (GLU ? 2 : 1); ++g)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const __nv_bfloat16* base = &Bs[g][warp * 16 + j * 8 + gid][kk + tig * 2];
          uint32_t bf[2];
          bf[0] = *reinterpret_cast<const uint32_t*>(base);
          bf[1] = *reinterpret_cast<const uint32_t*>(base + 8);
#pragma unroll
          for (int i = 0; i < 2; ++i) mma_bf16(acc[g][i][j], af[i], bf);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int dst = o_row[i * 16 + gid + half * 8];
      const float f = factor[i * 16 + gid + half * 8];
      if (dst < 0) continue;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int n = n0 + warp * 16 + j * 8 + tig * 2 + c;
          if (n >= N) continue;
          const float v0 = f * acc[0][i][j][half * 2 + c];
          const float v = GLU ? glu_limited(v0, f * acc[GLU ? 1 : 0][i][j][half * 2 + c], limit, slope, plus) : apply_activation(v0, act);
          out[(size_t)dst * N + n] = from_float<O>(v);
        }
    }
}

// --------------------------------------------- few pairs: matrix times vector --
// A step of single tokens has a handful of (token, choice) pairs, most on experts of their own: each pair
// then streams its expert's matrix once, and little else happens (moe_gemv_kernel below takes over where the matrices are many).  A block takes one pair and
// 64 output features (32 with the activation); the pair's activation row waits in shared memory as float32; a warp takes 8 (4)
// features, two at a time, its lanes striding along K in 16-byte pieces of the weight rows (with the activation, both the gate
// row and the up row of a feature), sixteen pieces (eight without the activation, by twice as
// many blocks) asked for before the first is used; the first are on their way while the activation row is laid out.  No sorting: pair p reads row p / top (gather) or p, and writes row p.
// Measured, the routed layer of width 2,048 (us; before: 64 features a block, four pieces at a time): 1 row 65 -> 33, 3 rows
// 92 -> 62, 8 rows 99 -> 92; of width 1,024 1 row 33 -> 25, 8 rows 44 -> 34.  The first product of the 8 rows 56 -> 37; the second
// 20 -> 24 with sixteen pieces, and the layer 89 -> 85 with eight and four blocks to a multiprocessor.
constexpr int pv_cols(bool glu) { return glu ? 32 : 64; }

__device__ __forceinline__ float dot8(const uint4& w, const float4& x0, const float4& x1) {
  // a bfloat16 is the upper half of a float
  float s = __uint_as_float(w.x << 16) * x0.x;
  s = fmaf(__uint_as_float(w.x & 0xffff0000u), x0.y, s);
  s = fmaf(__uint_as_float(w.y << 16), x0.z, s);
  s = fmaf(__uint_as_float(w.y & 0xffff0000u), x0.w, s);
  s = fmaf(__uint_as_float(w.z << 16), x1.x, s);
  s = fmaf(__uint_as_float(w.z & 0xffff0000u), x1.y, s);
  s = fmaf(__uint_as_float(w.w << 16), x1.z, s);
  return fmaf(__uint_as_float(w.w & 0xffff0000u), x1.w, s);
}

template <typename O, bool GLU>
__global__ void __launch_bounds__(256, GLU ? 2 : 4)
moe_pair_gemv_kernel(O* __restrict__ out, const __nv_bfloat16* a, long long a_stride,
                const __nv_bfloat16* __restrict__ w, const int* ids, int top, int gather, int N, int N_w,
                int Kd, float limit, float slope, float plus, int act, const float* early) {
  constexpr int STREAMS = GLU ? 4 : 2, STEPS = 4, PER_WARP = pv_cols(GLU) / 8;
  extern __shared__ __align__(16) float xs[];          // [Kd]
  pdl_wait();
  const int pair = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const __nv_bfloat16* arow = a + (size_t)(gather ? pair / top : pair) * a_stride;
  const __nv_bfloat16* we = w + (size_t)ids[pair] * N_w * Kd;
  const int first = (blockIdx.y * 8 + warp) * PER_WARP;
  // the rows of two neighbouring features from n0 on (of their up halves too); past the last feature the last one's again
  const __nv_bfloat16* rows[STREAMS];
  auto rows_of = [&](int n0) {
    const int m0 = min(n0, N - 1), m1 = min(n0 + 1, N - 1);
    rows[0] = we + (size_t)m0 * Kd;
    rows[1] = we + (size_t)m1 * Kd;
    if (GLU) {
      rows[2] = rows[0] + (size_t)N * Kd;
      rows[3] = rows[1] + (size_t)N * Kd;
    }
  };
  uint4 piece[STREAMS][STEPS];
  auto ask = [&](int k) {                              // this lane's pieces at k, k + 256, ...
#pragma unroll
    for (int i = 0; i < STEPS; ++i)
#pragma unroll
      for (int st = 0; st < STREAMS; ++st) {
        piece[st][i] = make_uint4(0u, 0u, 0u, 0u);
        if (k + 256 * i < Kd) piece[st][i] = __ldg(reinterpret_cast<const uint4*>(rows[st] + k + 256 * i));
      }
  };
  rows_of(first);
  ask(lane * 8);
  for (int i = tid; i < Kd / 8; i += 256) {
    const uint4 v = *reinterpret_cast<const uint4*>(arow + i * 8);
    float4 lo, hi;
    lo.x = __uint_as_float(v.x << 16); lo.y = __uint_as_float(v.x & 0xffff0000u);
    lo.z = __uint_as_float(v.y << 16); lo.w = __uint_as_float(v.y & 0xffff0000u);
    hi.x = __uint_as_float(v.z << 16); hi.y = __uint_as_float(v.z & 0xffff0000u);
    hi.z = __uint_as_float(v.w << 16); hi.w = __uint_as_float(v.w & 0xffff0000u);
    *reinterpret_cast<float4*>(xs + i * 8) = lo;
    *reinterpret_cast<float4*>(xs + i * 8 + 4) = hi;
  }
  __syncthreads();
  const float factor = early ? early[pair] : 1.f;
#pragma unroll 1
  for (int j = 0; j < PER_WARP; j += 2) {
    const int n0 = first + j, n1 = n0 + 1;               // warp-uniform
    if (n0 >= N) break;
    if (j > 0) {
      rows_of(n0);
      ask(lane * 8);
    }
    float sum[STREAMS];
#pragma unroll
    for (int st = 0; st < STREAMS; ++st) sum[st] = 0.f;
    for (int k = lane * 8; k < Kd; k += 256 * STEPS) {
      if (k != lane * 8) ask(k);
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        const int at = k + 256 * i;
        if (at < Kd) {
          const float4 x0 = *reinterpret_cast<const float4*>(xs + at), x1 = *reinterpret_cast<const float4*>(xs + at + 4);
#pragma unroll
          for (int st = 0; st < STREAMS; ++st) sum[st] += dot8(piece[st][i], x0, x1);
        }
      }
    }
#pragma unroll
    for (int st = 0; st < STREAMS; ++st) sum[st] = factor * warp_sum(sum[st]);
    if (lane == 0) {
      out[(size_t)pair * N + n0] = from_float<O>(GLU ? glu_limited(sum[0], sum[STREAMS - 2], limit, slope, plus) : apply_activation(sum[0], act));
      if (n1 < N)
        out[(size_t)pair * N + n1] = from_float<O>(GLU ? glu_limited(sum[1], sum[STREAMS - 1], limit, slope, plus) : apply_activation(sum[1], act));
    }
  }
}

// ----------------------------------------------- few pairs: a stream of weights --
// A step of single tokens has a handful of (token, choice) pairs, and the product is bound by the stream of their experts'
// matrices.  The pairs are grouped by expert, up to eight to a group, so that an expert that several rows chose is streamed once
// for them (8 rows of 2 of 16 experts choose 10.5 experts on average, in 16 pairs).  The work is cut into (group, 16 weight rows): with the
// activation the gate and up rows of eight features, else the rows of sixteen; in equal runs to the blocks, one block of eight warps to a
// multiprocessor, and a run's K in steps of 32 to the warps in turn.  A lane copies the 16-byte pieces that it multiplies itself into its own places of shared
// memory, GV_STAGES stages of two steps deep and across the ends of the units, and waits for nothing but its own copies:
// no registers are held for pieces on their way, and 128 KB of a multiprocessor's share are always asked for.  The weight rows are the rows of
// m16n8k16, the group's activation rows its columns; which of the K numbers of a step sits at which place of the product does not matter, so
// a piece of eight numbers goes into two products as it lies.  A unit's sums of the eight warps meet in shared memory.  What the loop reads besides lies in
// shared memory too: a load from global memory is answered behind the copies asked for before it, even when it hits the L1.  No
// sorting of rows: pair p reads row p / top (gather) or p, and writes row p; a pair's sum does not depend on its group.
// Where the line to moe_pair_gemv_kernel lies: this kernel needs the list of groups and most of a multiprocessor's shared memory before its
// first copy, about 2 us a launch.  Measured, the routed layer, 2 of 16 experts (us; pair by pair, grouped): width 2,048 2 rows 39.0, 41.5, 3 rows
// 57.1, 54.2, 8 rows 83.2, 68.8, 31 rows 210, 99; width 1,024 8 rows 30.8, 32.8, 12 rows 40.9, 38.6, 31 rows 74.3, 50.0; width 512 24 rows 32.8,
// 34.9.  Summing on the FP32 pipes in place of the tensor cores took 82 at 8 rows: the blocks whose experts had three and four rows were late.
constexpr long long GV_LINE = 20LL << 20;                // pairs times the numbers of a result's matrix, from which on the grouped kernel is the faster
constexpr int GV_WARPS = 8, GV_STAGES = 9, GV_STEP = 32, GV_GROUP = 8;
constexpr int GV_MOST = 128;                             // pairs of one launch
constexpr int GV_PAD = 32;                               // numbers between two activation rows: eight lanes' pieces of two rows lie in different banks
constexpr size_t GV_RING = (size_t)GV_WARPS * GV_STAGES * 4 * 32 * sizeof(uint4);        // two steps of two rows a lane
constexpr size_t GV_SUMS = (size_t)2 * GV_WARPS * 128 * sizeof(float);
constexpr int gv_group(int Kd) { return Kd <= 4096 ? 8 : Kd <= 8192 ? 4 : 2; }            // pairs of a group: as many rows as fit
constexpr int gv_held(int Kd) { return Kd <= 2048 ? 2 : 1; }      // groups whose rows are held: a block's run rarely meets more than two
constexpr size_t gv_smem(int Kd) {
  return GV_RING + GV_SUMS + 4 * GV_MOST * sizeof(int) + (size_t)gv_held(Kd) * gv_group(Kd) * (Kd + GV_PAD) * sizeof(__nv_bfloat16);
}
static_assert(gv_smem(2048) <= 227 * 1024 && gv_smem(4096) <= 227 * 1024 && gv_smem(8192) <= 227 * 1024 && gv_smem(12288) <= 227 * 1024,
              "the places of the copies and the activation rows share a multiprocessor");

__device__ __forceinline__ void gv_copy(void* dst, const __nv_bfloat16* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void gv_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <typename O, bool GLU>
__global__ void __launch_bounds__(GV_WARPS * 32, 1)
moe_gemv_kernel(O* __restrict__ out, const __nv_bfloat16* a, long long a_stride,
                const __nv_bfloat16* __restrict__ w, const int* ids, int pairs, int top, int gather, int N, int N_w,
                int Kd, int held, int most, float limit, float slope, float plus, int act, const float* early) {
  constexpr int COLS = GLU ? 8 : 16;                     // features of a unit
  extern __shared__ __align__(16) unsigned char gv_shared[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  uint4* ring = reinterpret_cast<uint4*>(gv_shared) + (size_t)warp * GV_STAGES * 4 * 32 + lane;      // [stage][step, row][lane]
  float* sums = reinterpret_cast<float*>(gv_shared + GV_RING);    // [2][warp][16 rows][8 pairs]
  int* id_of = reinterpret_cast<int*>(gv_shared + GV_RING + GV_SUMS);      // [pairs]
  int* sorted = id_of + GV_MOST;                                  // the pairs, by expert
  int* start = sorted + GV_MOST;                                  // place in ``sorted`` at which a group starts
  float* factor = reinterpret_cast<float*>(start + GV_MOST);      // [pairs]
  __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(factor + GV_MOST);      // [held][most][Kd + GV_PAD]
  pdl_wait();
  if (tid < GV_MOST) {
    id_of[tid] = tid < pairs ? ids[tid] : 0x7fffffff;
    factor[tid] = early && tid < pairs ? early[tid] : 1.f;
    sorted[tid] = -1;
  }
  __syncthreads();
  if (tid < pairs) {                                              // place of a pair: those of lower experts, then those before it
    const int id = id_of[tid];
    int lower = 0, same = 0;
    for (int q = 0; q < pairs; q += 4) {
      const int4 v = *reinterpret_cast<const int4*>(id_of + q);
      lower += (v.x < id) + (v.y < id) + (v.z < id) + (v.w < id);
      same += (v.x == id && q < tid) + (v.y == id && q + 1 < tid) + (v.z == id && q + 2 < tid) + (v.w == id && q + 3 < tid);
    }
    sorted[lower + same] = same % most == 0 ? tid : ~tid;         // a group's first pair as it is, the others inverted
  }
  __syncthreads();
  const bool starts = tid < pairs && sorted[tid] >= 0;
  if (starts) {
    int at = 0;
    for (int j = 0; j < tid; j += 4) {
      const int4 v = *reinterpret_cast<const int4*>(sorted + j);
      at += (v.x >= 0) + (v.y >= 0 && j + 1 < tid) + (v.z >= 0 && j + 2 < tid) + (v.w >= 0 && j + 3 < tid);
    }
    start[at] = tid;
  }
  const int groups = __syncthreads_count(starts);

  const int units = (N + COLS - 1) / COLS;               // of a group
  const long long total = (long long)groups * units;
  const int begin = (int)(total * blockIdx.x / gridDim.x), end = (int)(total * (blockIdx.x + 1) / gridDim.x);
  if (begin == end) return;
  auto pair_at = [&](int i) { const int p = sorted[i]; return p < 0 ? ~p : p; };
  auto members_of = [&](int g) { return (g + 1 < groups ? start[g + 1] : pairs) - start[g]; };
  const int g_first = begin / units, g_last = (end - 1) / units;
  auto bring_rows = [&](int g_from) {                    // the activation rows of the next ``held`` groups
    for (int g = g_from; g <= g_last && g < g_from + held; ++g)
      for (int m = 0; m < members_of(g); ++m) {
        const int p = pair_at(start[g] + m);
        const __nv_bfloat16* from = a + (size_t)(gather ? p / top : p) * a_stride;
        __nv_bfloat16* to = rows + (size_t)((g - g_from) * most + m) * (Kd + GV_PAD);
        for (int i = tid * 8; i < Kd; i += GV_WARPS * 32 * 8) gv_copy(to + i, from + i);
      }
    gv_commit();
  };
  bring_rows(g_first);
  // the copies of the weights run ahead of the products: their own unit, first K number and rows
  const int k_mine = warp * GV_STEP + tig * 8;           // of a stage: this lane's piece of the first step; the second step lies 8 warps on
  constexpr int STAGE_K = 2 * GV_WARPS * GV_STEP;
  int ask_unit = begin, ask_k = 0, ask_slot = 0, ask_g = g_first, ask_f = (begin - g_first * units) * COLS;
  const __nv_bfloat16 *ask0 = w, *ask1 = w;
  auto ask_rows = [&]() {
    const __nv_bfloat16* we = w + (size_t)id_of[sorted[start[ask_g]]] * N_w * Kd + k_mine;
    const int f0 = min(ask_f + gid, N - 1), f1 = GLU ? f0 + N : min(ask_f + 8 + gid, N - 1);       // past the last feature the last one's again
    ask0 = we + (size_t)f0 * Kd;
    ask1 = we + (size_t)f1 * Kd;
  };
  auto ask = [&]() {
    if (ask_unit < end) {
      uint4* to = ring + ask_slot * 4 * 32;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (ask_k + i * (STAGE_K / 2) + k_mine < Kd) {
          gv_copy(to + i * 64, ask0 + ask_k + i * (STAGE_K / 2));
          gv_copy(to + i * 64 + 32, ask1 + ask_k + i * (STAGE_K / 2));
        }
      ask_k += STAGE_K;
      if (ask_k >= Kd) {
        ask_k = 0;
        ask_f += COLS;
        if (ask_f >= N) {
          ask_f = 0;
          ++ask_g;
        }
        if (++ask_unit < end) ask_rows();
      }
    }
    gv_commit();                                         // one group a stage, so that "all but the last ones" means the oldest stage
    ask_slot = ask_slot + 1 == GV_STAGES ? 0 : ask_slot + 1;
  };
  ask_rows();
#pragma unroll
  for (int i = 0; i < GV_STAGES - 1; ++i) ask();
  asm volatile("cp.async.wait_group %0;" ::"n"(GV_STAGES - 1) : "memory");        // the activation rows
  __syncthreads();

  int slot = 0, g_from = g_first, g = g_first, f = (begin - g_first * units) * COLS;
#pragma unroll 1
  for (int unit = begin; unit < end; ++unit) {
    const int members = members_of(g);
    const __nv_bfloat16* x = rows + (size_t)((g - g_from) * most + gid) * (Kd + GV_PAD) + k_mine;
    float acc[2][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[0][c] = acc[1][c] = 0.f;
#pragma unroll 1
    for (int k = 0; k < Kd; k += STAGE_K) {
      ask();
      asm volatile("cp.async.wait_group %0;" ::"n"(GV_STAGES - 1) : "memory");
      const uint4* from = ring + slot * 4 * 32;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int at = k + i * (STAGE_K / 2);
        if (at + warp * GV_STEP >= Kd) break;            // warp-uniform
        uint4 w0 = make_uint4(0u, 0u, 0u, 0u), w1 = w0, v = w0;
        if (at + k_mine < Kd) {
          w0 = from[i * 64];
          w1 = from[i * 64 + 32];
          if (gid < members) v = *reinterpret_cast<const uint4*>(x + at);
        }
        const uint32_t a0[4] = {w0.x, w1.x, w0.y, w1.y}, a1[4] = {w0.z, w1.z, w0.w, w1.w};
        const uint32_t b0[2] = {v.x, v.y}, b1[2] = {v.z, v.w};
        mma_bf16(acc[0], a0, b0);
        mma_bf16(acc[1], a1, b1);
      }
      slot = slot + 1 == GV_STAGES ? 0 : slot + 1;
    }
    float* meet = sums + (unit & 1) * (GV_WARPS * 128);  // in turns: a unit's readers are through at the next unit's barrier
    float* to = meet + warp * 128 + gid * 8 + tig * 2;
    *reinterpret_cast<float2*>(to) = make_float2(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1]);
    *reinterpret_cast<float2*>(to + 64) = make_float2(acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
    __syncthreads();
    const int m = tid / COLS, j = tid % COLS;            // a pair and a feature to a thread
    if (m < members && f + j < N) {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int i = 0; i < GV_WARPS; ++i) {
        s0 += meet[i * 128 + j * 8 + m];
        if (GLU) s1 += meet[i * 128 + 64 + j * 8 + m];
      }
      const int p = pair_at(start[g] + m);
      const float by = factor[p];
      out[(size_t)p * N + f + j] = from_float<O>(GLU ? glu_limited(by * s0, by * s1, limit, slope, plus) : apply_activation(by * s0, act));
    }
    f += COLS;
    if (f >= N) {
      f = 0;
      ++g;
      if (g - g_from == held && unit + 1 < end) {        // a run over more groups than are held
        g_from = g;
        __syncthreads();
        bring_rows(g_from);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
      }
    }
  }
}

// ------------------------------------------------- activation and weighted sum --
// out[t, c] = act(f in[t, c], f in[t, n + c]) for the dense (shared) expert, f = row_scale[t] (null: 1).
template <typename I, typename O>
__global__ void __launch_bounds__(256)
glu_limited_kernel(O* __restrict__ out, const I* in, long long stride, int n, float limit, float slope, float plus,
                   const float* row_scale) {
  pdl_trigger();
  pdl_wait();
  const I* row = in + (size_t)blockIdx.x * stride;
  const float f = row_scale ? row_scale[blockIdx.x] : 1.f;
  for (int c = threadIdx.x; c < n; c += blockDim.x)
    out[(size_t)blockIdx.x * n + c] = from_float<O>(glu_limited(f * to_float<I>(row[c]), f * to_float<I>(row[n + c]), limit, slope, plus));
}

// The same from 32-bit or bfloat16 rows, four columns to a thread; grid (rows, column chunks).  bfloat16 results take the
// sigmoid from the fast exponential (a few ulp in 32-bit before the rounding).
__device__ __forceinline__ void load_four(const float* p, float (&v)[4]) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
__device__ __forceinline__ void load_four(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xffff0000u);
  v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xffff0000u);
}

template <typename I, typename O>
__global__ void __launch_bounds__(256)
glu_limited_vec_kernel(O* __restrict__ out, const I* in, long long stride, int n, float limit, float slope, float plus,
                       const float* row_scale) {
  pdl_trigger();
  pdl_wait();
  const int c = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (c >= n) return;
  const I* row = in + (size_t)blockIdx.x * stride;
  float g[4], u[4];
  load_four(row + c, g);
  load_four(row + n + c, u);
  if (row_scale) {
    const float f = row_scale[blockIdx.x];
#pragma unroll
    for (int i = 0; i < 4; ++i) { g[i] *= f; u[i] *= f; }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = fminf(g[i], limit), b = fminf(fmaxf(u[i], -limit), limit) + plus;
    g[i] = sizeof(O) == 2 ? __fdividef(a, 1.0f + fast_exp2(-1.4426950408889634f * slope * a)) * b : a * sigmoidf(slope * a) * b;
  }
  O* dst = out + (size_t)blockIdx.x * n + c;
  if (sizeof(O) == 2) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(g[0], g[1]), hi = __floats2bfloat162_rn(g[2], g[3]);
    uint2 packed;
    packed.x = *reinterpret_cast<uint32_t*>(&lo);
    packed.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(dst) = packed;
  } else {
    *reinterpret_cast<float4*>(dst) = make_float4(g[0], g[1], g[2], g[3]);
  }
}

// shared[t, :] = sum_k weights[t, k] * picked[row of pair t * top + k, :] + sigmoid(mix[t]) * shared[t, :], the
// chosen experts in the order of their choice; row_of_pair null: the pair's own number; weights null: 1.
// A thread takes four columns (one where rows are no whole 16-byte pieces), grid (tokens, runs of 256 threads): a step of a
// few rows spreads over as many blocks as it has columns for, and four choices' loads are on their way together.  Bound by
// the rows' bytes.  Measured, width 2,048, two choices (us; before: a column a thread, one block to a token): 8 rows 11.7 -> 3.7, 2,048 rows 23.7 -> 14.1.
template <int V>
__global__ void __launch_bounds__(256)
moe_combine_kernel(float* shared, const float* picked, const int* row_of_pair, const float* weights, const float* mix, long long mix_stride,
                   int top, int d) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, c = (blockIdx.y * 256 + threadIdx.x) * V;
  if (c >= d) return;
  float own[V], s[V];
  float* at = shared + (size_t)t * d + c;
#pragma unroll
  for (int i = 0; i < V; ++i) s[i] = 0.f;
  if constexpr (V == 4) {
    const float4 x = *reinterpret_cast<const float4*>(at);
    own[0] = x.x; own[1] = x.y; own[2] = x.z; own[3] = x.w;
  } else {
    own[0] = at[0];
  }
  const float gate = mix ? sigmoidf(mix[(size_t)t * mix_stride]) : 1.0f;
  for (int k0 = 0; k0 < top; k0 += 4) {
    float x[4][V], w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (k0 + u >= top) continue;
      const size_t pair = (size_t)t * top + k0 + u;
      const float* from = picked + (size_t)(row_of_pair ? row_of_pair[pair] : pair) * d + c;
      w[u] = weights ? weights[pair] : 1.f;
      if constexpr (V == 4) {
        const float4 f = *reinterpret_cast<const float4*>(from);
        x[u][0] = f.x; x[u][1] = f.y; x[u][2] = f.z; x[u][3] = f.w;
      } else {
        x[u][0] = from[0];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (k0 + u >= top) continue;
#pragma unroll
      for (int i = 0; i < V; ++i) s[i] = fmaf(w[u], x[u][i], s[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) s[i] = fmaf(gate, own[i], s[i]);
  if constexpr (V == 4) *reinterpret_cast<float4*>(at) = make_float4(s[0], s[1], s[2], s[3]);
  else at[0] = s[0];
}

}  // namespace

AYK_EXPORT int ayk_moe_tile_rows() { return TILE_ROWS; }

// ids, weights [T, top]; sorted [T * top]; tiles [1 + 3 * (T * top / TILE_ROWS + E)].  Two launches; with sorted null
// only the routing (the plan is for the products over sorted rows).
AYK_EXPORT int ayk_moe_route(int* ids, float* weights, int* sorted, int* tiles, const float* logits, long long stride,
                             int T, int E, int top, cudaStream_t stream) {
  if (T == 0) return 0;
  AYK_REQUIRE(top >= 1 && top <= MAX_TOP && top <= E, "ayk_moe_route: top %d of %d experts (at most %d)", top, E, MAX_TOP);
  AYK_REQUIRE(E <= 4096, "ayk_moe_route: %d experts (at most 4096)", E);
  ayk_launch(moe_route_kernel, dim3((T + 3) / 4), dim3(128), 0, stream, ids, weights, logits, stride, T, E, top);
  if (sorted) ayk_launch(moe_plan_kernel, dim3(1), dim3(1024), (size_t)3 * E * sizeof(int), stream, sorted, tiles, (const int*)ids,
             T * top, E);
  return ayk_check_launch("ayk_moe_route");
}

// The same plan after routing by sigmoid (or, with ``softmax``, softmax) scores in groups (see the head of the file).
// correction [E] float32 or null; groups equal runs of consecutive experts (at most 32) of which keep may be chosen from;
// group_best: 1 or 2 scores of a run make its own; normalize: the weights are divided by their sum.
AYK_EXPORT int ayk_moe_route_scored(int* ids, float* weights, int* sorted, int* tiles, const float* logits, long long stride,
                                    const float* correction, int T, int E, int top, int groups, int keep, float factor,
                                    int softmax, int group_best, int normalize, cudaStream_t stream) {
  if (T == 0) return 0;
  AYK_REQUIRE(top >= 1 && top <= MAX_TOP && top <= E, "ayk_moe_route_scored: top %d of %d experts (at most %d)", top, E, MAX_TOP);
  AYK_REQUIRE(E <= 4096, "ayk_moe_route_scored: %d experts (at most 4096)", E);
  AYK_REQUIRE(groups >= 1 && groups <= 32 && E % groups == 0 && keep >= 1 && keep <= groups && keep * (E / groups) >= top,
              "ayk_moe_route_scored: %d experts in %d groups of which %d are kept cannot give %d choices", E, groups, keep, top);
  AYK_REQUIRE(group_best == 1 || group_best == 2, "ayk_moe_route_scored: a group's score is its best or its two best");
  ayk_launch(softmax ? moe_route_scored_kernel<true> : moe_route_scored_kernel<false>, dim3((T + 3) / 4), dim3(128), 0, stream, ids,
             weights, logits, stride, correction, T, E, top, groups, keep, group_best, normalize, factor);
  if (sorted) ayk_launch(moe_plan_kernel, dim3(1), dim3(1024), (size_t)3 * E * sizeof(int), stream, sorted, tiles, (const int*)ids,
             T * top, E);
  return ayk_check_launch("ayk_moe_route_scored");
}

// See moe_gemm_kernel.  dtype: of a and w; out_dtype: of out (gated rows are of the operands' dtype, plain
// products, with the activation ``act``, of that or float32).  early [pairs] or null: see moe_gemm_kernel.  max_tiles: the grid's first dimension.
AYK_EXPORT int ayk_moe_gemm(void* out, const void* a, long long a_stride, const void* w, const int* sorted,
                            const int* tiles, int max_tiles, int top, int gather, int scatter, int N, int N_w, int Kd,
                            int glu, float limit, float slope, float plus, int act, const float* early, int dtype, int out_dtype,
                            cudaStream_t stream) {
  if (max_tiles == 0 || N == 0) return 0;
  dim3 grid(max_tiles, (N + BN - 1) / BN);
#define AYK_MOE(T, O, G)                                                                                              \
  ayk_launch(moe_gemm_kernel<T, O, G>, grid, dim3(256), 0, stream, (O*)out, (const T*)a, a_stride, (const T*)w, sorted, \
             tiles, top, gather, scatter, N, N_w, Kd, limit, slope, plus, act, early)
#define AYK_MOE_MMA(O, G)                                                                                        \
  ayk_launch(moe_gemm_mma_kernel<O, G>, grid, dim3(128), 0, stream, (O*)out, (const __nv_bfloat16*)a, a_stride, \
             (const __nv_bfloat16*)w, sorted, tiles, top, gather, scatter, N, N_w, Kd, limit, slope, plus, act, early)
  if (dtype == AYK_DTYPE_F32) {
    AYK_REQUIRE(out_dtype == AYK_DTYPE_F32, "ayk_moe_gemm: float32 operands give float32 rows");
    if (glu) AYK_MOE(float, float, true); else AYK_MOE(float, float, false);
  } else if (dtype == AYK_DTYPE_BF16) {
    const bool tensor = Kd % 8 == 0 && a_stride % 8 == 0 && ((uintptr_t)a % 16 == 0) && ((uintptr_t)w % 16 == 0);
    if (glu) {
      AYK_REQUIRE(out_dtype == AYK_DTYPE_BF16, "ayk_moe_gemm: the activation's rows are bfloat16 here");
      if (tensor) AYK_MOE_MMA(__nv_bfloat16, true); else AYK_MOE(__nv_bfloat16, __nv_bfloat16, true);
    } else if (out_dtype == AYK_DTYPE_BF16) {
      if (tensor) AYK_MOE_MMA(__nv_bfloat16, false); else AYK_MOE(__nv_bfloat16, __nv_bfloat16, false);
    } else {
      AYK_REQUIRE(out_dtype == AYK_DTYPE_F32, "ayk_moe_gemm: unknown dtype %d", out_dtype);
      if (tensor) AYK_MOE_MMA(float, false); else AYK_MOE(__nv_bfloat16, float, false);
    }
  } else {
    return ayk_fail("ayk_moe_gemm: unknown dtype %d", dtype);
  }
#undef AYK_MOE
#undef AYK_MOE_MMA
  return ayk_check_launch("ayk_moe_gemm");
}

AYK_EXPORT int ayk_glu_limited(void* out, const void* in, long long stride, int T, int n, float limit, float slope, float plus,
                               const float* row_scale, int in_dtype, int out_dtype, cudaStream_t stream) {
  if (T == 0 || n == 0) return 0;
  if (n % 4 == 0 && stride % 4 == 0 && (((uintptr_t)in | (uintptr_t)out) & 15) == 0 && (n + 1023) / 1024 <= 65535) {
    const dim3 grid(T, (n + 1023) / 1024);
#define AYK_GLU(I, O) ayk_launch(glu_limited_vec_kernel<I, O>, grid, dim3(256), 0, stream, (O*)out, (const I*)in, stride, n, limit, slope, plus, row_scale)
    if (in_dtype == AYK_DTYPE_F32 && out_dtype == AYK_DTYPE_F32) AYK_GLU(float, float);
    else if (in_dtype == AYK_DTYPE_F32 && out_dtype == AYK_DTYPE_BF16) AYK_GLU(float, __nv_bfloat16);
    else if (in_dtype == AYK_DTYPE_BF16 && out_dtype == AYK_DTYPE_BF16) AYK_GLU(__nv_bfloat16, __nv_bfloat16);
    else return ayk_fail("ayk_glu_limited: dtypes %d -> %d", in_dtype, out_dtype);
#undef AYK_GLU
    return ayk_check_launch("ayk_glu_limited");
  }
  if (in_dtype == AYK_DTYPE_F32 && out_dtype == AYK_DTYPE_F32)
    ayk_launch(glu_limited_kernel<float, float>, dim3(T), dim3(256), 0, stream, (float*)out, (const float*)in, stride, n, limit, slope, plus, row_scale);
  else if (in_dtype == AYK_DTYPE_F32 && out_dtype == AYK_DTYPE_BF16)
    ayk_launch(glu_limited_kernel<float, __nv_bfloat16>, dim3(T), dim3(256), 0, stream, (__nv_bfloat16*)out, (const float*)in,
               stride, n, limit, slope, plus, row_scale);
  else if (in_dtype == AYK_DTYPE_BF16 && out_dtype == AYK_DTYPE_BF16)
    ayk_launch(glu_limited_kernel<__nv_bfloat16, __nv_bfloat16>, dim3(T), dim3(256), 0, stream, (__nv_bfloat16*)out,
               (const __nv_bfloat16*)in, stride, n, limit, slope, plus, row_scale);
  else
    return ayk_fail("ayk_glu_limited: dtypes %d -> %d", in_dtype, out_dtype);
  return ayk_check_launch("ayk_glu_limited");
}

AYK_EXPORT int ayk_moe_pad_rows() { return PAD_ROWS; }

// The padded plan (see moe_plan_padded_kernel) and the gathered rows: gathered [max_tiles * 128, d] bfloat16 gets
// row p / top of ``in`` at row_of_pair[p], row_scale [max_tiles * 128] (or null) weights[p].  Two launches.
AYK_EXPORT int ayk_moe_plan_padded(int* row_of_pair, int* w_rows1, int* w_rows2, void* gathered, float* row_scale,
                                   const float* weights, const int* ids,
                                   const void* in, long long in_stride, int T, int E, int top, int d, int n1, int n2,
                                   int max_tiles, cudaStream_t stream) {
  if (T == 0) return 0;
  AYK_REQUIRE(E <= 4096 && d % 8 == 0 && in_stride % 8 == 0, "ayk_moe_plan_padded: %d experts, rows of %d", E, d);
  ayk_launch(moe_plan_padded_kernel, dim3(1), dim3(1024), (size_t)3 * E * sizeof(int), stream, row_of_pair, w_rows1, w_rows2, ids,
             T * top, E, n1, n2, max_tiles);
  ayk_launch(moe_gather_kernel, dim3((T * top + 7) / 8), dim3(256), 0, stream, (__nv_bfloat16*)gathered, (const __nv_bfloat16*)in,
             in_stride, (const int*)row_of_pair, row_scale, weights, T * top, top, d);
  return ayk_check_launch("ayk_moe_plan_padded");
}

AYK_EXPORT int ayk_moe_combine(float* shared, const float* picked, const int* row_of_pair, const float* weights,
                               const float* mix, long long mix_stride, int T, int top, int d, cudaStream_t stream) {
  if (T == 0 || d == 0) return 0;
  const bool vec = d % 4 == 0 && ((uintptr_t)shared | (uintptr_t)picked) % 16 == 0;
  dim3 grid(T, (d + (vec ? 1024 : 256) - 1) / (vec ? 1024 : 256));
  AYK_REQUIRE(grid.y <= 65535, "ayk_moe_combine: rows of %d", d);
  if (vec) ayk_launch(moe_combine_kernel<4>, grid, dim3(256), 0, stream, shared, picked, row_of_pair, weights, mix, mix_stride, top, d);
  else ayk_launch(moe_combine_kernel<1>, grid, dim3(256), 0, stream, shared, picked, row_of_pair, weights, mix, mix_stride, top, d);
  return ayk_check_launch("ayk_moe_combine");
}

// The products of a few pairs (see moe_gemv_kernel): bfloat16 a and w, K a multiple of 8 and at most
// 12,288.  gather: pair p reads row p / top of a, else row p.  glu: out [pairs, N] bfloat16 = activation of (gate, up)
// rows of w [E, 2 N, K]; else out [pairs, N] (out_dtype) = act(row times w [E, N, K]).
AYK_EXPORT int ayk_moe_gemv_takes(int Kd, long long a_stride) { return Kd % 8 == 0 && a_stride % 8 == 0 && Kd <= 12288; }

namespace {
template <typename O, bool GLU>
int gemv(O* out, const __nv_bfloat16* a, long long a_stride, const __nv_bfloat16* w, const int* ids, int pairs, int top, int gather, int N,
         int N_w, int Kd, float limit, float slope, float plus, int act, const float* early, cudaStream_t stream) {
  if ((long long)pairs * N * Kd < GV_LINE || top > GV_MOST) {       // a launch below holds whole tokens
    ayk_launch(moe_pair_gemv_kernel<O, GLU>, dim3(pairs, (N + pv_cols(GLU) - 1) / pv_cols(GLU)), dim3(256), (size_t)Kd * sizeof(float), stream,
               out, a, a_stride, w, ids, top, gather, N, N_w, Kd, limit, slope, plus, act, early);
    return ayk_check_launch("ayk_moe_gemv");
  }
  static AykPerDevice granted;
  if (!granted.here()) {
    cudaError_t e = cudaFuncSetAttribute(moe_gemv_kernel<O, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return ayk_fail("ayk_moe_gemv: shared memory: %s", cudaGetErrorString(e));
    granted.here() = true;
  }
  const int units = (N + (GLU ? 7 : 15)) / (GLU ? 8 : 16);
  const int most = GV_MOST / top * top;                  // whole tokens a launch
  for (int p = 0; p < pairs; p += most) {
    const int n = pairs - p < most ? pairs - p : most;
    const long long blocks = (long long)n * units;
    const int sms = ayk_sm_count();
    ayk_launch(moe_gemv_kernel<O, GLU>, dim3((unsigned)(blocks < sms ? blocks : sms)), dim3(GV_WARPS * 32), gv_smem(Kd), stream, out + (size_t)p * N,
               a + (size_t)(gather ? p / top : p) * a_stride, a_stride, w, ids + p, n, top, gather, N, N_w, Kd, gv_held(Kd), gv_group(Kd), limit, slope, plus, act,
               early ? early + p : nullptr);
  }
  return ayk_check_launch("ayk_moe_gemv");
}
}  // namespace

AYK_EXPORT int ayk_moe_gemv(void* out, const void* a, long long a_stride, const void* w, const int* ids, int pairs, int top,
                            int N, int N_w, int Kd, int gather, int glu, float limit, float slope, float plus, int act, const float* early,
                            int out_dtype,
                            cudaStream_t stream) {
  if (pairs == 0 || N == 0) return 0;
  AYK_REQUIRE(ayk_moe_gemv_takes(Kd, a_stride), "ayk_moe_gemv: rows of %d elements (stride %lld)", Kd, a_stride);
  AYK_REQUIRE(top >= 1, "ayk_moe_gemv: %d choices a row", top);
  const __nv_bfloat16 *rows = (const __nv_bfloat16*)a, *weights = (const __nv_bfloat16*)w;
  if (glu)
    return gemv<__nv_bfloat16, true>((__nv_bfloat16*)out, rows, a_stride, weights, ids, pairs, top, gather, N, N_w, Kd, limit, slope, plus, act, early, stream);
  if (out_dtype == AYK_DTYPE_BF16)
    return gemv<__nv_bfloat16, false>((__nv_bfloat16*)out, rows, a_stride, weights, ids, pairs, top, gather, N, N_w, Kd, limit, slope, plus, act, early, stream);
  return gemv<float, false>((float*)out, rows, a_stride, weights, ids, pairs, top, gather, N, N_w, Kd, limit, slope, plus, act, early, stream);
}
