// Layer norm with weight and bias, fused with the residual add in front of it.
//
//   residual += delta;  out = (residual - mean) / sqrt(var + eps) * w + b,  var = mean((residual - mean)^2)
//
// `delta` is a 32-bit tensor [rows, hidden], or `parts` partial sums [parts, rows, hidden] of a product split along k
// that are added in order. Mean and variance are taken in two passes over the row held in registers (rows of a length that
// 16-byte pieces do not divide: in shared memory), in 32-bit, with a fixed order of additions, so a row's result never
// depends on the batch. With `gather` output row i is made
// from row gather[i] and the residual stays as it was (the last norm, for the rows whose logits are wanted).
#include "common.cuh"

namespace tl {

// Rows whose length is a multiple of four, VPT 16-byte pieces a thread. A decode step has a block or a few, whose time is the
// chain of round trips: the row and its sources are asked for together, up to eight partial sums at a time, and the norm's own
// numbers before the first reduction. Measured at four rows of 2048 in a decode step with ten partial sums every other time:
// 11.3 us with a number a load and a load a round trip, 3.3 us here; 1997 rows without partial sums 19.2 and 17.4 us.
//
// PLAIN: one source at most and more rows than the other form lets stand on the GPU at once (1024 threads an SM with a piece a thread;
// with more pieces the line lies at two rounds of rows): with no loads to send ahead of others, an instantiation without their registers keeps more rows on an SM and
// reads the norm's numbers where they are used. One source, 2000 and 6000 rows: of 2048 15.8 and 52.1 -> 10.7 and 36.1 us (a number a load
// 16.8 and 57.1), of 2560 24.7 and 100.6 -> 11.0 and 39.6 (20.0 and 69.2; the 640 pieces of a row also went to 512 threads, 384 of which idled
// through the second).
template <typename T, int VPT, bool PLAIN>
__global__ void __launch_bounds__(512, PLAIN ? (VPT == 1 ? 3 : VPT == 2 ? 2 : 1) : 0) add_layernorm_vec_kernel(float* __restrict__ residual, const float* __restrict__ delta,
                                                                int parts, long long part_stride,
                                                                const float* __restrict__ weight, const float* __restrict__ bias,
                                                                float eps, T* __restrict__ out, const int* __restrict__ gather,
                                                                int hidden) {
  __shared__ float red[64];
  const int i = blockIdx.x;
  const int r = gather ? gather[i] : i;
  float* res = residual + (size_t)r * hidden;
  const float* src = delta + (size_t)r * hidden;
  float4 x[VPT], w[VPT], b[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * blockDim.x) * 4;
    x[v] = w[v] = b[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < hidden) x[v] = load4_now(res + c);
  }
  constexpr int AT_ONCE = PLAIN ? 1 : VPT == 1 ? 8 : VPT == 2 ? 4 : 1;
  for (int p0 = 0; p0 < parts; p0 += AT_ONCE) {
    float4 d[AT_ONCE][VPT];
#pragma unroll
    for (int p = 0; p < AT_ONCE; ++p)
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (threadIdx.x + v * blockDim.x) * 4;
        if (p0 + p < parts && c < hidden) d[p][v] = load4_now(src + (size_t)(p0 + p) * part_stride + c);
        else d[p][v] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    if (!PLAIN && p0 == 0)
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (threadIdx.x + v * blockDim.x) * 4;
        if (c < hidden) {
          w[v] = load4_now(weight + c);
          b[v] = load4_now(bias + c);
        }
      }
#pragma unroll
    for (int p = 0; p < AT_ONCE; ++p)
      if (p0 + p < parts)
#pragma unroll
        for (int v = 0; v < VPT; ++v) add4(x[v], d[p][v]);
  }
  if (!PLAIN && parts == 0)
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (threadIdx.x + v * blockDim.x) * 4;
      if (c < hidden) {
        w[v] = load4_now(weight + c);
        b[v] = load4_now(bias + c);
      }
    }
  float sum = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * blockDim.x) * 4;
    if (!gather && parts && c < hidden) store4(res + c, x[v].x, x[v].y, x[v].z, x[v].w);
    sum += x[v].x + x[v].y + x[v].z + x[v].w;
  }
  const float mean = block_sum_once(sum, red) / (float)hidden;
  float sq = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * blockDim.x) * 4;
    if (c < hidden) {
      x[v].x -= mean; x[v].y -= mean; x[v].z -= mean; x[v].w -= mean;
      sq = dot4(x[v], x[v], sq);
    }
  }
  const float var = block_sum_once(sq, red + 32) / (float)hidden;
  const float inv = 1.f / sqrtf(var + eps);
  T* o = out + (size_t)i * hidden;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * blockDim.x) * 4;
    if (PLAIN && c < hidden) {
      w[v] = *reinterpret_cast<const float4*>(weight + c);
      b[v] = *reinterpret_cast<const float4*>(bias + c);
    }
    if (c < hidden)
      store4(o + c, fmaf(x[v].x * inv, w[v].x, b[v].x), fmaf(x[v].y * inv, w[v].y, b[v].y), fmaf(x[v].z * inv, w[v].z, b[v].z),
             fmaf(x[v].w * inv, w[v].w, b[v].w));
  }
}

template <typename T>
void launch_layernorm_vec(float* residual, const float* delta, int parts, long long part_stride, const float* weight,
                          const float* bias, float eps, T* out, const int* gather, int rows, int hidden, cudaStream_t stream) {
  // (as few pieces a thread as 512 threads allow, and then as few threads as those need: 640 pieces are two for each of 320)
  const int pieces = hidden / 4, vpt = ceil_div(pieces, 512), threads = ceil_div(ceil_div(pieces, vpt), 32) * 32;
  const bool plain = parts <= 1 && rows * (long long)threads > 1024LL * sm_count();
#define TL_LN_(V_, P_) add_layernorm_vec_kernel<T, V_, P_><<<rows, threads, 0, stream>>>(residual, delta, parts, part_stride, weight, bias, eps, out, gather, hidden)
#define TL_LN(V_)               \
  do {                          \
    if (plain) TL_LN_(V_, true); \
    else TL_LN_(V_, false);     \
  } while (0)
  if (vpt == 1) TL_LN(1);
  else if (vpt == 2) TL_LN(2);
  else if (vpt <= 4) TL_LN(4);
  else TL_LN(6);
#undef TL_LN_
#undef TL_LN
}

template <typename T>
__global__ void __launch_bounds__(256) add_layernorm_kernel(float* __restrict__ residual, const float* __restrict__ delta,
                                                            int parts, long long part_stride, const float* __restrict__ weight,
                                                            const float* __restrict__ bias, float eps, T* __restrict__ out,
                                                            const int* __restrict__ gather, int hidden) {
  extern __shared__ float row[];            // [hidden] + 33 for the reductions
  float* red = row + hidden;
  const int i = blockIdx.x;
  const int r = gather ? gather[i] : i;
  float* res = residual + (size_t)r * hidden;
  float sum = 0.f;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    float x = res[c];
    for (int p = 0; p < parts; ++p) x += delta[(size_t)p * part_stride + (size_t)r * hidden + c];
    if (!gather && parts) res[c] = x;
    row[c] = x;
    sum += x;
  }
  const float mean = block_sum(sum, red) / (float)hidden;
  float sq = 0.f;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    const float d = row[c] - mean;
    sq = fmaf(d, d, sq);
  }
  const float var = block_sum(sq, red) / (float)hidden;
  const float inv = 1.f / sqrtf(var + eps);
  T* o = out + (size_t)i * hidden;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) o[c] = from_f32<T>(fmaf((row[c] - mean) * inv, weight[c], bias[c]));
}

}  // namespace tl

using namespace tl;

extern "C" int tl_add_layernorm(float* residual, const float* delta, int parts, long long part_stride, const float* weight,
                                const float* bias, float eps, void* out, const int* gather, int out_rows, int hidden,
                                int dtype, cudaStream_t stream) {
  if (out_rows == 0) return 0;
  TL_REQUIRE(hidden > 0 && hidden <= 11264 && parts >= 0 && (parts == 0 || delta), "add_layernorm: hidden %d (up to 11264), %d parts",
             hidden, parts);
  const uintptr_t all = (uintptr_t)residual | (uintptr_t)delta | (uintptr_t)weight | (uintptr_t)bias | (uintptr_t)out;
  if (hidden % 4 == 0 && (all & 15) == 0 && (parts <= 1 || part_stride % 4 == 0)) {
    if (dtype == TL_FP32)
      launch_layernorm_vec(residual, delta, parts, part_stride, weight, bias, eps, (float*)out, gather, out_rows, hidden, stream);
    else
      launch_layernorm_vec(residual, delta, parts, part_stride, weight, bias, eps, (bf16*)out, gather, out_rows, hidden, stream);
    TL_LAUNCH_CHECK();
    return 0;
  }
  const int threads = hidden >= 1024 ? 256 : 128;
  const size_t smem = (size_t)(hidden + 40) * sizeof(float);
  if (dtype == TL_FP32)
    add_layernorm_kernel<float><<<out_rows, threads, smem, stream>>>(residual, delta, parts, part_stride, weight, bias, eps,
                                                                     (float*)out, gather, hidden);
  else
    add_layernorm_kernel<bf16><<<out_rows, threads, smem, stream>>>(residual, delta, parts, part_stride, weight, bias, eps,
                                                                    (bf16*)out, gather, hidden);
  TL_LAUNCH_CHECK();
  return 0;
}
