// Latent attention of prompt portions with keys and values expanded: what comes in front of the attention (attention_wide_tc.cu).
//
// With U_k^T applied to the queries (latent.cu) a (query, key) pair costs rank + rot + rank products per head, with keys U_k c and values
// U_v c made once per cached token dim + rot + vdim: 1,088 against 320 for 512, 64, 128 and 128.  So where a step's rows are many
// for the tokens that they read, the step's latents lie side by side (a request's from its first visible 64 tokens on, request
// after request), one product with [U_k; U_v] makes their keys and values, and the rows attend to those.
//
// The kernel below does the rest, a block to a row.  For a row of the step, from the float32 projection row [q (H x (128 + 64)) | down (rank + 64) | ...]:
//   latent = rmsnorm(down[:rank]) * w  -> its page and its place among the rows side by side
//   k_r    = turn(down[rank:])         -> the rotated-key page
//   q      -> per head times a power of two that brings its largest unrotated number to [128, 256), unrotated part float16,
//             turn(rotated part) bfloat16; the factor that undoes it goes to the scores (q_scale)
// For a token that earlier steps cached: its latent from its page to its place.
// float16 keeps three more bits than bfloat16: with queries, keys, weights and values in bfloat16 the layer's error against 64 bits was 15 %
// larger than with U_k^T applied to 32-bit queries.  It has three bits of exponent less, so everything comes into its range by powers of
// two: queries as above; a head's keys and its values by `up_scale` (LatentAttention.bind), which brings the largest number that they
// can hold to [2^14, 2^15), 28 powers of two above float16's smallest of full precision.  The keys' factor is also on the rotated
// query parts, whose keys have none, and q_scale takes both out; the values' is taken out with the softmax's sum.
// Bound by the projection's 32-bit rows (14.6 KB a row at 16 heads): 11 us for 1,801 rows, 41 MB.
// Measured, the layer of width 2,048 (16 heads, latent 512 + 64), 1,024 + 777 rows: 280 -> 104 us (absorbed attention 176, its two products per
// head 52, preparation 19; now preparation 11, keys and values 13, attention 28); error against 64 bits 3.2e-3 -> 2.8e-3, and over 23
// drawn steps 0.69 to 1.00 of what it was.
#include <cuda_fp16.h>
#include <math.h>

#include "common.cuh"

namespace {

constexpr int DIM = 128, ROT = 64, THREADS = 128, WARPS = THREADS / 32;

// The first token of a request whose latent lies among the rows side by side: the start of the 64 that hold the first visible key of its first row.
__device__ __forceinline__ int first_token(int pos0, int window) { return window > 0 ? max(0, pos0 - window + 1) / 64 * 64 : 0; }

__global__ void __launch_bounds__(THREADS)
latent_expand_prepare_kernel(__nv_bfloat16* latent_pages, __nv_bfloat16* __restrict__ rope_pages, __half* q16, __nv_bfloat16* q_rot, float* q_scale,
                             __nv_bfloat16* side, const float* proj, long long proj_stride, const float* __restrict__ norm_w, const float* up_scale,
                             const float* __restrict__ freq, float gain, int rot_dims, int halves, const int* __restrict__ row_req,
                             const int* __restrict__ positions, const int* __restrict__ table, int table_stride, int page_size,
                             const int* __restrict__ req_q_start, const int* __restrict__ req_pos0, int num_req, int T, int H, int rank, float eps,
                             int window) {
  __shared__ float turn[ROT];                              // cos [rot_dims / 2], sin [rot_dims / 2]
  __shared__ float red[WARPS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_trigger();
  if ((int)blockIdx.x >= T) {
    // a cached token's latent: which request's?
    int j = blockIdx.x - T, base = 0, req = -1, first = 0;
    for (int r0 = 0; r0 < num_req && req < 0; r0 += 32) {
      const int r = r0 + lane;
      const int pos0 = r < num_req ? req_pos0[r] : 0, f = first_token(pos0, window);
      int cached = pos0 - f, held = r < num_req ? cached + req_q_start[r + 1] - req_q_start[r] : 0;       // tokens side by side
      int cached_to = cached, held_to = held;              // sums up to this lane
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int c = __shfl_up_sync(0xffffffffu, cached_to, o), h = __shfl_up_sync(0xffffffffu, held_to, o);
        if (lane >= o) { cached_to += c; held_to += h; }
      }
      const unsigned behind = __ballot_sync(0xffffffffu, j < cached_to);
      if (behind) {
        const int src = __ffs(behind) - 1;
        req = r0 + src;
        first = __shfl_sync(0xffffffffu, f, src);
        j -= __shfl_sync(0xffffffffu, cached_to - cached, src);
        base += __shfl_sync(0xffffffffu, held_to - held, src);
      } else {
        j -= __shfl_sync(0xffffffffu, cached_to, 31);
        base += __shfl_sync(0xffffffffu, held_to, 31);
      }
    }
    if (req < 0) return;
    const int p = first + j;
    const int page = table[(size_t)req * table_stride + p / page_size];
    pdl_wait();
    const __nv_bfloat16* from = latent_pages + ((size_t)page * page_size + p % page_size) * rank;
    __nv_bfloat16* to = side + (size_t)(base + j) * rank;
    for (int i = tid * 8; i < rank; i += THREADS * 8)      // a token on no page: zeros
      *reinterpret_cast<uint4*>(to + i) = page > 0 ? *reinterpret_cast<const uint4*>(from + i) : make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const int t = blockIdx.x, p = positions[t], my_req = row_req[t];
  const int page = table[(size_t)my_req * table_stride + p / page_size];
  const int half = rot_dims >> 1;
  if (tid < half) {
    float s, c;
    sincosf((float)p * freq[tid], &s, &c);
    turn[tid] = c * gain;
    turn[half + tid] = s * gain;
  }
  int base = 0;                                            // rows side by side of the requests before this one
  for (int r = lane; r < my_req; r += 32) base += req_pos0[r] - first_token(req_pos0[r], window) + req_q_start[r + 1] - req_q_start[r];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
  base += p - first_token(req_pos0[my_req], window);
  __syncthreads();
  float up_next = up_scale[min(warp, H - 1)];              // asked for a head ahead
  pdl_wait();
  const float* row = proj + (size_t)t * proj_stride;
  const float* down = row + (size_t)H * (DIM + ROT);
  // number e of a rotated part: u cos - v sin for the first of a pair (u, v), v cos + u sin for the second
  auto turned = [&](const float* src, int e, float x) {
    if (e >= rot_dims) return x;
    const bool second = halves ? e >= half : (e & 1) != 0;
    const int i = halves ? (second ? e - half : e) : e >> 1, other = halves ? (second ? i : e + half) : e ^ 1;
    const float s = turn[half + i];
    return fmaf(src[other], second ? s : -s, x * turn[i]);
  };
  for (int h = warp; h < H; h += WARPS) {
    const float* src = row + (size_t)h * (DIM + ROT);
    const int up = ((int)__float_as_uint(up_next) >> 23) - 127;          // the keys' factor is 2^up, 0 <= up <= 40
    up_next = up_scale[min(h + WARPS, H - 1)];
    const float4 v = *reinterpret_cast<const float4*>(src + lane * 4);
    const float2 w = *reinterpret_cast<const float2*>(src + DIM + lane * 2);
    const float r0 = turned(src + DIM, lane * 2, w.x), r1 = turned(src + DIM, lane * 2 + 1, w.y);
    const float top = warp_max(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    // 2^k with top 2^k in [128, 256); 1 for zeros, infinities and not-a-numbers.  At most 2^(60 - up): queries that would need more are so
    // small that, with keys of at most 2^(15 - up), what they lose moves a score by less than 2^-40.
    const int e = ((int)__float_as_uint(top) >> 23) & 0xff;              // of 2^(e - 127) <= top
    const int k = e > 0 && e < 255 ? min(max(134 - e, -120), 60 - up) : 0;
    const float by = __uint_as_float((uint32_t)(k + 127) << 23), by_rot = __uint_as_float((uint32_t)(k + up + 127) << 23);
    const size_t at = (size_t)t * H + h;
    const __half2 a = __floats2half2_rn(v.x * by, v.y * by), b = __floats2half2_rn(v.z * by, v.w * by);
    *reinterpret_cast<uint2*>(q16 + at * DIM + lane * 4) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    *reinterpret_cast<__nv_bfloat162*>(q_rot + at * ROT + lane * 2) = __floats2bfloat162_rn(r0 * by_rot, r1 * by_rot);
    if (lane == 0) q_scale[at] = __uint_as_float((uint32_t)(127 - k - up) << 23);
  }
  const size_t cell = (size_t)max(page, 0) * page_size + p % page_size;
  if (page > 0 && tid < ROT) rope_pages[cell * ROT + tid] = __float2bfloat16_rn(turned(down + rank, tid, down[rank + tid]));
  float s = 0.f;
  for (int i = tid * 4; i < rank; i += THREADS * 4) {
    const float4 v = *reinterpret_cast<const float4*>(down + i);
    s = fmaf(v.x, v.x, s); s = fmaf(v.y, v.y, s); s = fmaf(v.z, v.z, s); s = fmaf(v.w, v.w, s);
  }
  s = warp_sum(s);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  const float inv = 1.0f / sqrtf(((red[0] + red[1]) + (red[2] + red[3])) / (float)rank + eps);
  for (int i = tid * 4; i < rank; i += THREADS * 4) {
    const float4 v = *reinterpret_cast<const float4*>(down + i), w = *reinterpret_cast<const float4*>(norm_w + i);
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x * inv * w.x, v.y * inv * w.y), b = __floats2bfloat162_rn(v.z * inv * w.z, v.w * inv * w.w);
    const uint2 c = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    if (page > 0) *reinterpret_cast<uint2*>(latent_pages + cell * rank + i) = c;
    *reinterpret_cast<uint2*>(side + (size_t)base * rank + i) = c;
  }
}

}  // namespace

// See above.  q16 [T, H, 128] float16, q_rot [T, H, 64] bfloat16, q_scale [T, H] float32, side [rows, rank] bfloat16: T rows and `cached` tokens
// of earlier steps, request after request.  up_scale [H or more]: the heads' factors on the keys.  rank a multiple of 8, proj_stride of 4, all tensors 16-byte aligned.
AYK_EXPORT int ayk_latent_expand_prepare(void* latent_pages, void* rope_pages, void* q16, void* q_rot, float* q_scale, void* side, const float* proj,
                                         long long proj_stride, const float* norm_w, const float* up_scale, const float* freq, float gain, int rot_dims, int halves,
                                         const int* row_req, const int* positions, const int* table, int table_stride, int page_size,
                                         const int* req_q_start, const int* req_pos0, int num_req, int T, int cached, int H, int rank, float eps,
                                         int window, cudaStream_t stream) {
  if (T == 0) return 0;
  AYK_REQUIRE(rot_dims % 2 == 0 && rot_dims >= 0 && rot_dims <= ROT, "ayk_latent_expand_prepare: %d rotated dimensions of %d", rot_dims, ROT);
  AYK_REQUIRE(rank % 8 == 0 && proj_stride % 4 == 0 && cached >= 0, "ayk_latent_expand_prepare: latents of %d, rows of %lld", rank, proj_stride);
  AYK_REQUIRE((((uintptr_t)latent_pages | (uintptr_t)q16 | (uintptr_t)q_rot | (uintptr_t)side | (uintptr_t)proj | (uintptr_t)norm_w) & 15) == 0,
              "ayk_latent_expand_prepare: operands must be 16-byte aligned");
  ayk_launch(latent_expand_prepare_kernel, dim3((unsigned)(T + cached)), dim3(THREADS), 0, stream, (__nv_bfloat16*)latent_pages, (__nv_bfloat16*)rope_pages,
             (__half*)q16, (__nv_bfloat16*)q_rot, q_scale, (__nv_bfloat16*)side, proj, proj_stride, norm_w, up_scale, freq, gain, rot_dims, halves, row_req,
             positions, table, table_stride, page_size, req_q_start, req_pos0, num_req, T, H, rank, eps, window);
  return ayk_check_launch("ayk_latent_expand_prepare");
}
