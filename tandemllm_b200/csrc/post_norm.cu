// A norm behind a branch (the second norm of a layer whose sublayers are normed before and after), fused with the
// residual add, and a vector added to every row of the residual stream.
//
//   d[r] = (sum of the dense parts)[r] * (gate ? sigmoid(gate[r]) : 1) + sum_j wts[r, j] * expert_rows[pos_of_pair[r k + j]]
//   residual[r] += weight * d[r] * rsqrt(mean(d[r]^2) + eps)
//   with `pre_weight`: normed[i] = pre_weight * residual[r] * rsqrt(mean(residual[r]^2) + eps)  (the norm in front of the next
//   sublayer in the same pass; with `gather`, output row i reads row gather[i] and the residual stays as it was)
//
// The branch output comes in the forms the products leave it in: a 32-bit tensor or partial sums of a product split along
// k (added in order), the rows of a routed expert layer (weighed and added in ascending expert id), or both (a shared
// feed-forward beside the routed one, times a gate a row). Everything is 32-bit; one block a row, fixed orders of addition.
#include "route.cuh"

namespace tl {

struct PostNormParams {
  float* residual;
  const float* delta;
  int parts;
  long long part_stride;
  const float* delta_gate;   // [rows] logits or nullptr: the dense parts times sigmoid(logit)
  const float* expert_rows;
  int expert_parts;
  long long expert_part_stride;
  const int* pos_of_pair;
  const int* ids;
  const float* wts;
  int top_k;
  const float* weight;
  float eps;
  int hidden;
  const float* pre_weight;   // the next norm's weight, or nullptr: only the add
  float pre_eps;
  void* normed;
  const int* gather;
  int few_rows;              // rows with a load a number: a step of few rows (few blocks), the form whose loads of a source are all in flight together
  const void* gate_x;        // or the gate's rows and its vector: logit = gate_x[r] . gate_w (delta_gate is then nullptr)
  const void* gate_w;
  long long gate_ld;
  int gate_bf16;
};

// Rows whose length is a multiple of four, VPT 16-byte pieces a thread, held in registers from the first load to the last store.
// A decode step has a block or a few and their time is the chain of round trips, so what does not depend on another load (the
// residual, both norms' weights, the gate's row and vector, the dense parts) is asked for before the experts' rows, which are asked
// for four slots at a time; every warp orders the row's slots itself and no barrier stands in front of them. The gate's logit is
// taken here because a kernel of its own cost 5.5 us and a launch for one number a row. Measured at two rows of 2048 in a decode
// step, six slots beside a shared part in ten partial sums: 13.8 us with a number a load, 4.5 us here (with the gate's logit); 1000
// rows 30.9 and 19.8 us.
//
// PLAIN: one dense source, no slots, no gate's rows, and more rows than the other form lets stand on the GPU at once (1024
// threads an SM with a piece a thread; with more, two rounds of rows): with no loads to send ahead, an instantiation without their registers keeps more
// rows on an SM and reads the norms' weights where they are used. 2000 and 6000 rows of 1536 13.1 and 39.1 -> 6.5 and 16.0 us (a
// number a load 11.6 and 29.8), of 2048 15.4 and 53.9 -> 8.3 and 27.6 (13.5 and 50.4), of 2560 20.3 and 88.8 -> 8.5 and 33.0 (16.3 and 73.6).
template <typename T, int VPT, bool PLAIN>
__global__ void __launch_bounds__(512, PLAIN ? (VPT == 1 ? 3 : VPT == 2 ? 2 : 1) : VPT == 1 ? 2 : 1) add_normed_vec_kernel(PostNormParams p) {
  __shared__ float red[96];
  const int hidden = p.hidden, lane = threadIdx.x & 31;
  const int r = p.gather ? p.gather[blockIdx.x] : (int)blockIdx.x;
  // the row's slots in ascending expert id (the slot index breaks ties)
  int slot_src = 0, rank = -1;
  float slot_w = 0.f;
  if (!PLAIN && p.expert_rows) {
    const int k = p.top_k, j = lane;
    const bool mine = j < k;
    const int e = mine ? p.ids[(long long)r * k + j] : 0x7fffffff;
    slot_src = mine ? p.pos_of_pair[(long long)r * k + j] : 0;
    slot_w = mine ? (p.wts ? p.wts[(long long)r * k + j] : 1.f) : 0.f;
    int before = 0;
    for (int i = 0; i < k; ++i) {
      const int ei = __shfl_sync(0xffffffffu, e, i);
      before += (ei < e) || (ei == e && i < j);
    }
    if (mine) rank = before;
  }
  float* res = p.residual + (size_t)r * hidden;
  float4 d[VPT], x[VPT], w[VPT], pw[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * blockDim.x) * 4;
    d[v] = x[v] = w[v] = pw[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < hidden) {
      x[v] = load4_now(res + c);
      if (!PLAIN) {
        w[v] = load4_now(p.weight + c);
        if (p.pre_weight) pw[v] = load4_now(p.pre_weight + c);
      }
    }
  }
  float g = 1.f;
  if (!PLAIN && p.gate_x) {
    float dot = 0.f;
    if (p.gate_bf16) {
      const bf16* gx = reinterpret_cast<const bf16*>(p.gate_x) + (long long)r * p.gate_ld;
      const bf16* gw = reinterpret_cast<const bf16*>(p.gate_w);
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (threadIdx.x + v * blockDim.x) * 4;
        if (c < hidden) {
          const uint2 a = *reinterpret_cast<const uint2*>(gx + c), b = *reinterpret_cast<const uint2*>(gw + c);
          const float2 a0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.x));
          const float2 a1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.y));
          const float2 b0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&b.x));
          const float2 b1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&b.y));
          dot = dot4(make_float4(a0.x, a0.y, a1.x, a1.y), make_float4(b0.x, b0.y, b1.x, b1.y), dot);
        }
      }
    } else {
      const float* gx = reinterpret_cast<const float*>(p.gate_x) + (long long)r * p.gate_ld;
      const float* gw = reinterpret_cast<const float*>(p.gate_w);
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (threadIdx.x + v * blockDim.x) * 4;
        if (c < hidden) dot = dot4(load4_now(gx + c), load4_now(gw + c), dot);
      }
    }
    g = 1.f / (1.f + expf(-block_sum_once(dot, red + 64)));
  } else if (p.delta_gate) {
    g = 1.f / (1.f + expf(-p.delta_gate[r]));
  }
  constexpr int AT_ONCE = PLAIN ? 1 : VPT == 1 ? 4 : VPT == 2 ? 2 : 1;
  if (p.delta) {
    const float* src = p.delta + (size_t)r * hidden;
    for (int s0 = 0; s0 < p.parts; s0 += AT_ONCE) {
      float4 y[AT_ONCE][VPT];
#pragma unroll
      for (int s = 0; s < AT_ONCE; ++s)
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
          const int c = (threadIdx.x + v * blockDim.x) * 4;
          if (s0 + s < p.parts && c < hidden) y[s][v] = load4_now(src + (long long)(s0 + s) * p.part_stride + c);
          else y[s][v] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
      for (int s = 0; s < AT_ONCE; ++s)
        if (s0 + s < p.parts)
#pragma unroll
          for (int v = 0; v < VPT; ++v) add4(d[v], y[s][v]);
    }
#pragma unroll
    for (int v = 0; v < VPT; ++v) { d[v].x *= g; d[v].y *= g; d[v].z *= g; d[v].w *= g; }
  }
  if (!PLAIN && p.expert_rows) {
    float4 routed[VPT];
#pragma unroll
    for (int v = 0; v < VPT; ++v) routed[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = 0; j0 < p.top_k; j0 += AT_ONCE) {
      float4 y[AT_ONCE][VPT];
      float ws[AT_ONCE];
      const float* from[AT_ONCE];
#pragma unroll
      for (int j = 0; j < AT_ONCE; ++j) {
        const unsigned who = __ballot_sync(0xffffffffu, rank == j0 + j);
        const int at = who ? __ffs(who) - 1 : 0;
        ws[j] = __shfl_sync(0xffffffffu, slot_w, at);
        from[j] = p.expert_rows + (long long)__shfl_sync(0xffffffffu, slot_src, at) * hidden;
#pragma unroll
        for (int v = 0; v < VPT; ++v) y[j][v] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      for (int s = 0; s < p.expert_parts; ++s) {
        float4 t[AT_ONCE][VPT];
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j)
#pragma unroll
          for (int v = 0; v < VPT; ++v) {
            const int c = (threadIdx.x + v * blockDim.x) * 4;
            if (j0 + j < p.top_k && c < hidden) t[j][v] = load4_now(from[j] + (long long)s * p.expert_part_stride + c);
            else t[j][v] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j)
#pragma unroll
          for (int v = 0; v < VPT; ++v) add4(y[j][v], t[j][v]);
      }
#pragma unroll
      for (int j = 0; j < AT_ONCE; ++j)
        if (j0 + j < p.top_k)
#pragma unroll
          for (int v = 0; v < VPT; ++v) {
            routed[v].x = fmaf(ws[j], y[j][v].x, routed[v].x);
            routed[v].y = fmaf(ws[j], y[j][v].y, routed[v].y);
            routed[v].z = fmaf(ws[j], y[j][v].z, routed[v].z);
            routed[v].w = fmaf(ws[j], y[j][v].w, routed[v].w);
          }
    }
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      add4(routed[v], d[v]);
      d[v] = routed[v];
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) ss = dot4(d[v], d[v], ss);
  const float inv = rsqrtf(block_sum_once(ss, red) / (float)hidden + p.eps);
  float ss2 = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * blockDim.x) * 4;
    if (PLAIN && c < hidden) w[v] = *reinterpret_cast<const float4*>(p.weight + c);
    x[v].x += d[v].x * inv * w[v].x;
    x[v].y += d[v].y * inv * w[v].y;
    x[v].z += d[v].z * inv * w[v].z;
    x[v].w += d[v].w * inv * w[v].w;
    if (!p.gather && c < hidden) store4(res + c, x[v].x, x[v].y, x[v].z, x[v].w);
    ss2 = dot4(x[v], x[v], ss2);
  }
  if (!p.pre_weight) return;
  const float inv2 = rsqrtf(block_sum_once(ss2, red + 32) / (float)hidden + p.pre_eps);
  T* out = reinterpret_cast<T*>(p.normed) + (size_t)blockIdx.x * hidden;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (threadIdx.x + v * blockDim.x) * 4;
    if (PLAIN && c < hidden) pw[v] = *reinterpret_cast<const float4*>(p.pre_weight + c);
    if (c < hidden)
      store4(out + c, x[v].x * inv2 * pw[v].x, x[v].y * inv2 * pw[v].y, x[v].z * inv2 * pw[v].z, x[v].w * inv2 * pw[v].w);
  }
}

// Rows of any other length, or that do not begin at 16 bytes: a number a load, the row in shared memory. FEW: the form for a step of
// few rows (see `few_rows`), a kernel of its own so that the other keeps its few registers (rows of 2050, six slots beside a dense part:
// one row 26.1 us without, 10.9 with it; 296 rows 27.8 and 12.3).
template <typename T, bool FEW>
__global__ void __launch_bounds__(256) add_normed_kernel(PostNormParams p) {
  extern __shared__ __align__(16) float row[];          // hidden floats, then 33 for the reductions
  float* scratch = row + p.hidden;
  __shared__ int s_src[MAX_TOP_K];
  __shared__ float s_w[MAX_TOP_K];
  const int hidden = p.hidden;
  const int r = p.gather ? p.gather[blockIdx.x] : (int)blockIdx.x;
  if (p.expert_rows) {
    if (threadIdx.x < 32) {
      // the row's slots in ascending expert id (the slot index breaks ties)
      const int k = p.top_k, j = threadIdx.x;
      const bool mine = j < k;
      const int e = mine ? p.ids[(long long)r * k + j] : 0x7fffffff;
      const int src = mine ? p.pos_of_pair[(long long)r * k + j] : 0;
      const float w = mine ? (p.wts ? p.wts[(long long)r * k + j] : 1.f) : 0.f;
      int rank = 0;
      for (int i = 0; i < k; ++i) {
        const int ei = __shfl_sync(0xffffffffu, e, i);
        rank += (ei < e) || (ei == e && i < j);
      }
      if (mine) {
        s_src[rank] = src;
        s_w[rank] = w;
      }
    }
    __syncthreads();
  }
  const float g = p.delta_gate ? 1.f / (1.f + expf(-p.delta_gate[r])) : 1.f;
  float ss = 0.f;
  constexpr int CPT = 16;           // columns a thread holds in registers in the form for rows of up to 16 x 256 numbers
  if (FEW && hidden <= CPT * (int)blockDim.x) {
    // Source by source, a thread's loads of one source all sent before the first is used: a decode step has a handful of
    // blocks, and their time is the chain of round trips to L2, one a source instead of one a source and column.
    float d[CPT], routed[CPT];
#pragma unroll
    for (int i = 0; i < CPT; ++i) d[i] = routed[i] = 0.f;
    if (p.delta) {
      for (int s = 0; s < p.parts; ++s) {
        const float* src = p.delta + (long long)s * p.part_stride + (size_t)r * hidden;
#pragma unroll
        for (int i = 0; i < CPT; ++i) {
          const int c = threadIdx.x + i * blockDim.x;
          if (c < hidden) d[i] += src[c];
        }
      }
#pragma unroll
      for (int i = 0; i < CPT; ++i) d[i] *= g;
    }
    if (p.expert_rows) {
      for (int j = 0; j < p.top_k; ++j) {
        float v[CPT];
#pragma unroll
        for (int i = 0; i < CPT; ++i) v[i] = 0.f;
        for (int s = 0; s < p.expert_parts; ++s) {
          const float* src = p.expert_rows + (long long)s * p.expert_part_stride + (long long)s_src[j] * hidden;
#pragma unroll
          for (int i = 0; i < CPT; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
            if (c < hidden) v[i] += src[c];
          }
        }
#pragma unroll
        for (int i = 0; i < CPT; ++i) routed[i] = fmaf(s_w[j], v[i], routed[i]);
      }
#pragma unroll
      for (int i = 0; i < CPT; ++i) d[i] = routed[i] + d[i];
    }
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      const int c = threadIdx.x + i * blockDim.x;
      if (c < hidden) {
        row[c] = d[i];
        ss += d[i] * d[i];
      }
    }
  } else
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    float d = 0.f;
    if (p.delta) {
      for (int s = 0; s < p.parts; ++s) d += p.delta[(long long)s * p.part_stride + (size_t)r * hidden + c];
      d *= g;
    }
    if (p.expert_rows) {
      float routed = 0.f;
      for (int j = 0; j < p.top_k; ++j) {
        float v = 0.f;
        for (int s = 0; s < p.expert_parts; ++s)
          v += p.expert_rows[(long long)s * p.expert_part_stride + (long long)s_src[j] * hidden + c];
        routed = fmaf(s_w[j], v, routed);
      }
      d = routed + d;
    }
    row[c] = d;
    ss += d * d;
  }
  ss = block_sum(ss, scratch);
  const float inv = rsqrtf(ss / (float)hidden + p.eps);
  float* res = p.residual + (size_t)r * hidden;
  float ss2 = 0.f;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    const float x = res[c] + row[c] * inv * p.weight[c];
    if (!p.gather) res[c] = x;
    row[c] = x;
    ss2 += x * x;
  }
  if (!p.pre_weight) return;
  ss2 = block_sum(ss2, scratch);
  const float inv2 = rsqrtf(ss2 / (float)hidden + p.pre_eps);
  T* out = reinterpret_cast<T*>(p.normed) + (size_t)blockIdx.x * hidden;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) out[c] = from_f32<T>(row[c] * inv2 * p.pre_weight[c]);
}

// out[r] = scale * (weight_a * a[r] / rms(a[r]) + weight_b * b[r] / rms(b[r])): two branches' rows, each normed on its own (a tensor or
// partial sums each, added in order). One block a row.
struct NormedSumParams {
  const float *a, *b;
  int a_parts, b_parts;
  long long part_stride;
  const float *weight_a, *weight_b;
  float eps, scale;
  float* out;
  int hidden;
};
template <int CPT>
__global__ void __launch_bounds__(256) normed_sum_kernel(NormedSumParams p) {
  __shared__ float scratch[33];
  const int hidden = p.hidden;
  const size_t at = (size_t)blockIdx.x * hidden;
  float a[CPT], b[CPT];
  float sa = 0.f, sb = 0.f;
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    a[i] = c < hidden ? p.a[at + c] : 0.f;
    b[i] = c < hidden ? p.b[at + c] : 0.f;
  }
  for (int s = 1; s < p.a_parts; ++s) {
    const float* src = p.a + (long long)s * p.part_stride + at;
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      const int c = threadIdx.x + i * blockDim.x;
      if (c < hidden) a[i] += src[c];
    }
  }
  for (int s = 1; s < p.b_parts; ++s) {
    const float* src = p.b + (long long)s * p.part_stride + at;
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      const int c = threadIdx.x + i * blockDim.x;
      if (c < hidden) b[i] += src[c];
    }
  }
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    sa = fmaf(a[i], a[i], sa);
    sb = fmaf(b[i], b[i], sb);
  }
  sa = block_sum(sa, scratch);
  __syncthreads();
  sb = block_sum(sb, scratch);
  const float ia = rsqrtf(sa / (float)hidden + p.eps), ib = rsqrtf(sb / (float)hidden + p.eps);
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < hidden) p.out[at + c] = p.scale * (a[i] * ia * p.weight_a[c] + b[i] * ib * p.weight_b[c]);
  }
}

// out[r] = x[r, :] . w: a warp a row (a projection onto one number a row, such as the logit of a gate)
template <typename T>
__global__ void __launch_bounds__(256) row_dot_kernel(const T* __restrict__ x, long long ld_x, const T* __restrict__ w,
                                                      float* __restrict__ out, int rows, int hidden) {
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  const T* xr = x + (long long)r * ld_x;
  float acc = 0.f;
#pragma unroll 8
  for (int c = lane; c < hidden; c += 32) acc = fmaf(to_f32(xr[c]), to_f32(w[c]), acc);
  acc = warp_sum(acc);
  if (lane == 0) out[r] = acc;
}

// residual[r, :] += vec
__global__ void add_vector_kernel(float* __restrict__ residual, const float* __restrict__ vec, long long n, int hidden) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    residual[i] += vec[i % hidden];
}

}  // namespace tl

using namespace tl;

// Whether everything add_normed_vec_kernel reads and writes begins at 16 bytes, row by row.
static bool add_normed_aligned(const PostNormParams& p) {
  const uintptr_t all = (uintptr_t)p.residual | (uintptr_t)p.delta | (uintptr_t)p.expert_rows | (uintptr_t)p.weight |
                        (uintptr_t)p.pre_weight | (uintptr_t)p.normed | (uintptr_t)p.gate_x | (uintptr_t)p.gate_w;
  return (all & 15) == 0 && (!p.delta || p.parts <= 1 || p.part_stride % 4 == 0) &&
         (!p.expert_rows || p.expert_parts <= 1 || p.expert_part_stride % 4 == 0) && (!p.gate_x || p.gate_ld % 4 == 0);
}

extern "C" int tl_add_normed(float* residual, const float* delta, int parts, long long part_stride, const float* delta_gate,
                             const float* expert_rows, int expert_parts, long long expert_part_stride, const int* pos_of_pair,
                             const int* ids, const float* wts, int top_k, const float* weight, float eps,
                             const float* pre_weight, float pre_eps, void* normed, const int* gather, const void* gate_x,
                             long long gate_ld, const void* gate_w, int gate_dtype, int rows, int hidden, int dtype,
                             cudaStream_t stream) {
  if (rows == 0) return 0;
  TL_REQUIRE(rows > 0 && hidden > 0 && hidden <= 16384, "add_normed: %d rows of %d", rows, hidden);
  TL_REQUIRE(residual && weight && (delta || expert_rows), "add_normed: a residual, a weight and a branch output are needed");
  TL_REQUIRE(!delta || parts >= 1, "add_normed: %d parts", parts);
  TL_REQUIRE(!expert_rows || (pos_of_pair && ids && top_k > 0 && top_k <= MAX_TOP_K && expert_parts >= 1),
             "add_normed: expert rows with top-%d in %d parts", top_k, expert_parts);
  TL_REQUIRE(!pre_weight || normed, "add_normed: the following norm needs a place for its rows");
  TL_REQUIRE(!gather || pre_weight, "add_normed: chosen rows are only read for the following norm");
  PostNormParams p;
  p.residual = residual; p.delta = delta; p.parts = parts; p.part_stride = part_stride; p.delta_gate = delta_gate;
  p.expert_rows = expert_rows; p.expert_parts = expert_parts; p.expert_part_stride = expert_part_stride;
  p.pos_of_pair = pos_of_pair; p.ids = ids; p.wts = wts; p.top_k = top_k; p.weight = weight; p.eps = eps; p.hidden = hidden;
  p.pre_weight = pre_weight; p.pre_eps = pre_eps; p.normed = normed; p.gather = gather;
  p.gate_x = gate_x; p.gate_w = gate_w; p.gate_ld = gate_ld; p.gate_bf16 = gate_dtype == TL_BF16;
  if (hidden % 4 == 0 && hidden <= 8192 && add_normed_aligned(p)) {
    // (as few pieces a thread as 512 threads allow, and then as few threads as those need: 640 pieces are two for each of 320)
    const int pieces = hidden / 4, vpt = ceil_div(pieces, 512), threads = ceil_div(ceil_div(pieces, vpt), 32) * 32;
    const bool plain = !expert_rows && parts <= 1 && !gate_x && rows * (long long)threads > 1024LL * sm_count();
#define TL_ADD_NORMED_VEC_(T_, V_, P_) add_normed_vec_kernel<T_, V_, P_><<<rows, threads, 0, stream>>>(p)
#define TL_ADD_NORMED_VEC(V_)                               \
  do {                                                      \
    if (dtype == TL_FP32) {                                 \
      if (plain) TL_ADD_NORMED_VEC_(float, V_, true);       \
      else TL_ADD_NORMED_VEC_(float, V_, false);            \
    } else {                                                \
      if (plain) TL_ADD_NORMED_VEC_(bf16, V_, true);        \
      else TL_ADD_NORMED_VEC_(bf16, V_, false);             \
    }                                                       \
  } while (0)
    if (vpt == 1) TL_ADD_NORMED_VEC(1);
    else if (vpt == 2) TL_ADD_NORMED_VEC(2);
    else TL_ADD_NORMED_VEC(4);
#undef TL_ADD_NORMED_VEC_
#undef TL_ADD_NORMED_VEC
    TL_LAUNCH_CHECK();
    return 0;
  }
  TL_REQUIRE(!gate_x, "add_normed: rows of %d that are not laid out for 16-byte loads take the gate's logits, not its rows", hidden);
  p.few_rows = rows <= 2 * sm_count() ? 1 : 0;
  const size_t smem = (size_t)(hidden + 33) * sizeof(float);
#define TL_ADD_NORMED(T_, FEW_)                                                                                         \
  do {                                                                                                                  \
    if (smem > 48 * 1024)                                                                                               \
      cudaFuncSetAttribute(add_normed_kernel<T_, FEW_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);        \
    add_normed_kernel<T_, FEW_><<<rows, 256, smem, stream>>>(p);                                                        \
  } while (0)
  if (dtype == TL_FP32) {
    if (p.few_rows) TL_ADD_NORMED(float, true);
    else TL_ADD_NORMED(float, false);
  } else {
    if (p.few_rows) TL_ADD_NORMED(bf16, true);
    else TL_ADD_NORMED(bf16, false);
  }
#undef TL_ADD_NORMED
  TL_LAUNCH_CHECK();
  return 0;
}

extern "C" int tl_normed_sum(const float* a, int a_parts, const float* b, int b_parts, long long part_stride, const float* weight_a,
                             const float* weight_b, float eps, float scale, float* out, int rows, int hidden, cudaStream_t stream) {
  if (rows == 0) return 0;
  TL_REQUIRE(rows > 0 && hidden > 0 && hidden <= 16384 && a && b && a_parts >= 1 && b_parts >= 1, "normed_sum: %d rows of %d", rows,
             hidden);
  NormedSumParams p{a, b, a_parts, b_parts, part_stride, weight_a, weight_b, eps, scale, out, hidden};
  const int threads = hidden <= 512 ? 64 : (hidden <= 1024 ? 128 : 256);
  const int cpt = ceil_div(hidden, threads);
  if (cpt <= 8) normed_sum_kernel<8><<<rows, threads, 0, stream>>>(p);
  else if (cpt <= 16) normed_sum_kernel<16><<<rows, threads, 0, stream>>>(p);
  else if (cpt <= 32) normed_sum_kernel<32><<<rows, threads, 0, stream>>>(p);
  else normed_sum_kernel<64><<<rows, threads, 0, stream>>>(p);
  TL_LAUNCH_CHECK();
  return 0;
}

extern "C" int tl_row_dot(const void* x, long long ld_x, const void* w, float* out, int rows, int hidden, int dtype,
                          cudaStream_t stream) {
  if (rows == 0) return 0;
  TL_REQUIRE(rows > 0 && hidden > 0 && x && w && out, "row dot: %d rows of %d", rows, hidden);
  if (dtype == TL_FP32) row_dot_kernel<float><<<ceil_div(rows, 8), 256, 0, stream>>>((const float*)x, ld_x, (const float*)w, out, rows, hidden);
  else row_dot_kernel<bf16><<<ceil_div(rows, 8), 256, 0, stream>>>((const bf16*)x, ld_x, (const bf16*)w, out, rows, hidden);
  TL_LAUNCH_CHECK();
  return 0;
}

extern "C" int tl_add_vector(float* residual, const float* vec, int rows, int hidden, cudaStream_t stream) {
  if (rows == 0) return 0;
  TL_REQUIRE(rows > 0 && hidden > 0 && residual && vec, "add_vector: %d rows of %d", rows, hidden);
  const long long n = (long long)rows * hidden;
  const long long most = (long long)sm_count() * 8;
  const int blocks = (int)(ceil_div64(n, 256) < most ? ceil_div64(n, 256) : most);
  add_vector_kernel<<<blocks, 256, 0, stream>>>(residual, vec, n, hidden);
  TL_LAUNCH_CHECK();
  return 0;
}
