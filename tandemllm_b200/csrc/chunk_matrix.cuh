// Long portions of a linear recurrence whose state decays by one number a head and token, in matrix form:
//
//   S_t = a_t S_(t-1) + w_t k_t v_t^T,   o_t = S_t^T q_t      (S [N keys, P values] a head, 32-bit)
//
// over a chunk of 64 tokens that starts from S_0, with d(t, s) = a_(s+1) .. a_t:
//
//   o_t = d(t, 0) S_0^T q_t + sum over s <= t of d(t, s) w_s (q_t . k_s) v_s
//   S_64 = d(64, 0) S_0 + sum over s of d(64, s) w_s k_s v_s^T
//
// so a chunk is four small products instead of 64 dependent steps over the state. Chunks run side by side: first what every chunk adds
// to a zero state and the product of its decays (`chunk_end_kernel`), then the states the chunks start from (the caller walks a
// request's chunks), then the outputs (`chunk_out_kernel`), with the scores q . k in front (`chunk_score_kernel`: heads that
// share q and k share them). Every product of decays is multiplied up token by token, never taken as a quotient or as a
// difference of logarithms, so it has the error that the scan's repeated multiplication has. All arithmetic is 32-bit, and a chunk
// starts at the first row of a request's portion whatever else is in the step.
//
// What bounds it: a token costs a head N P multiply-adds for the state it adds, N P for the state it reads and 64 P for its
// neighbours, as register tiles of 8 x 8 that read 16 bytes of shared memory for every 16 multiply-adds; the scan wanted three to five
// instructions an entry of the state and a 16-byte read for four of them.
#pragma once

#include "common.cuh"

namespace tl {

constexpr int CM_TOKENS = 64;        // tokens a chunk
constexpr int CM_KEYS = 128;         // keys staged at a time
constexpr int CM_COLS = 64;          // value columns a block
constexpr int CM_THREADS = 128;

struct ChunkMatrix {
  const float* q;            // q of head h, row r: q + r * ld_q + group(h) * group_q
  const float* k;            // the same with k
  const float* v;            // v + r * ld_v + h * P
  long long ld_qk, group_qk, ld_v;
  int heads_per_group;       // heads that share q and k
  const float* decay;        // a_t of (row, head) at r * H + h
  const float* weight;       // w_t of (row, head)
  const float* skip;         // o_t += skip[h] v_t
  const int* row_start;
  float* scores;             // [places][groups][64][64]
  float* chunk_state;        // [places][H][P][N]
  float* chunk_decay;        // [places][H]
  float* y;                  // [rows, H P]
  int H, P, N, max_chunks;
};

// A request's chunks lie at row_start / 64 + request and on: no two requests' overlap (one of n rows has at most n / 64 + 1 chunks),
// and the step's chunks need `chunk_places` places, however unequal its portions are.
static inline long long chunk_places(long long rows, int requests) { return rows / CM_TOKENS + requests + 1; }
__device__ __forceinline__ int cm_place(const int* row_start, int req) { return row_start[req] / CM_TOKENS + req; }

// The chunk of block (request, chunk of it): its place, first row and rows; false where the request has fewer.
__device__ __forceinline__ bool cm_chunk(const ChunkMatrix& m, int b, int& place, int& first, int& n) {
  const int req = b / m.max_chunks, c = b - req * m.max_chunks;
  place = cm_place(m.row_start, req) + c;
  first = m.row_start[req] + c * CM_TOKENS;
  n = min(CM_TOKENS, m.row_start[req + 1] - first);
  return n > 0;
}

// rows [0, n) of `src` (`ld` apart), `cols` of their numbers, to `dst` [64][`pitch`]; what lies past them is zero. 16-byte pieces.
__device__ __forceinline__ void cm_stage(float* dst, int pitch, int width, const float* src, long long ld, int n, int cols) {
  const int pieces = width >> 2;
  for (int i = threadIdx.x; i < CM_TOKENS * pieces; i += CM_THREADS) {
    const int r = i / pieces, c = (i - r * pieces) * 4;
    const float4 v = (r < n && c < cols) ? *reinterpret_cast<const float4*>(src + r * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(dst + r * pitch + c) = v;
  }
}

// The 64 x 64 products of a block: two halves of 64 threads take a half of the sum each, a thread rows ti + 8 i of `a` against rows tj
// + 8 j of `b` (i, j < 8), so that 16 reads of 16 bytes feed 256 multiply-adds. Sixteen products are added up in a row before their
// sum joins the others (CM_RUN pieces): chains as long as the keys lost half as much again as the scan token by token does.
struct CmPlace {
  int half, ti, tj;
  __device__ __forceinline__ CmPlace() : half(threadIdx.x >> 6), ti((threadIdx.x & 63) >> 3), tj(threadIdx.x & 7) {}
};
constexpr int CM_RUN = 4;
__device__ __forceinline__ void cm_dots(float (&sum)[8][8], const CmPlace& at, const float* a, const float* b, int pitch, int pieces) {
  const int mid = (pieces + 1) >> 1, e1 = at.half ? pieces : mid;
  a += at.ti * pitch;
  b += at.tj * pitch;
#pragma unroll 1
  for (int e0 = at.half ? mid : 0; e0 < e1; e0 += CM_RUN) {
    float acc[8][8] = {};
#pragma unroll 1
    for (int e = e0; e < min(e0 + CM_RUN, e1); ++e) {
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4*>(a + i * 8 * pitch + 4 * e);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 z = *reinterpret_cast<const float4*>(b + j * 8 * pitch + 4 * e);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][j] = dot4(x[i], z, acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[i][j] += acc[i][j];
  }
}
// Adds the halves: the first half's threads keep rows i < 4, the second's i >= 4, in r[i & 3][j]. `buf`: 4096 floats nobody reads.
__device__ __forceinline__ void cm_join(const float (&acc)[8][8], float (&r)[4][8], const CmPlace& at, float* buf) {
  const int thread = threadIdx.x & 63;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) buf[(at.half * 32 + i * 8 + j) * 64 + thread] = at.half ? acc[i][j] : acc[i + 4][j];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float other = buf[((at.half ^ 1) * 32 + i * 8 + j) * 64 + thread];
      r[i][j] = at.half ? other + acc[i + 4][j] : acc[i][j] + other;
    }
}

// grid (groups, chunks): scores[t][s] = q_t . k_s.
__global__ void __launch_bounds__(CM_THREADS) chunk_score_kernel(ChunkMatrix m) {
  extern __shared__ __align__(16) float sm[];
  constexpr int PITCH = CM_KEYS + 4;
  float* sq = sm;
  float* sk = sq + CM_TOKENS * PITCH;
  int b, first, n;
  if (!cm_chunk(m, blockIdx.y, b, first, n)) return;
  const CmPlace place;
  float acc[8][8] = {};
  for (int n0 = 0; n0 < m.N; n0 += CM_KEYS) {
    const int cols = min(CM_KEYS, m.N - n0);
    const long long at = (long long)first * m.ld_qk + (long long)blockIdx.x * m.group_qk + n0;
    __syncthreads();
    cm_stage(sq, PITCH, CM_KEYS, m.q + at, m.ld_qk, n, cols);
    cm_stage(sk, PITCH, CM_KEYS, m.k + at, m.ld_qk, n, cols);
    __syncthreads();
    cm_dots(acc, place, sq, sk, PITCH, cols >> 2);
  }
  float* out = m.scores + ((long long)b * gridDim.x + blockIdx.x) * (CM_TOKENS * CM_TOKENS);
  __syncthreads();
  float r[4][8];
  cm_join(acc, r, place, sq);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) out[(place.ti + 8 * (i + 4 * place.half)) * CM_TOKENS + place.tj + 8 * j] = r[i][j];
}

// grid (H, chunks, tiles of 64 columns x tiles of 128 keys): what the chunk adds to a zero state. A thread holds 8 columns and 8 keys.
static __global__ void __launch_bounds__(CM_THREADS) chunk_end_kernel(ChunkMatrix m) {
  extern __shared__ __align__(16) float sm[];
  float* sk = sm;                                    // [64][128]
  float* sv = sk + CM_TOKENS * CM_KEYS;              // [64][64], weighed
  float* sa = sv + CM_TOKENS * CM_COLS;              // a_t, then what a token's share still is at the chunk's end
  const int h = blockIdx.x, tid = threadIdx.x;
  int b, first, n;
  if (!cm_chunk(m, blockIdx.y, b, first, n)) return;
  const int key_tiles = ceil_div(m.N, CM_KEYS);
  const int p0 = (blockIdx.z / key_tiles) * CM_COLS, n0 = (blockIdx.z % key_tiles) * CM_KEYS;
  const int keys = min(CM_KEYS, m.N - n0), cols = min(CM_COLS, m.P - p0);
  const int group = h / m.heads_per_group;
  if (tid < CM_TOKENS) sa[tid] = tid < n ? m.decay[(long long)(first + tid) * m.H + h] : 1.f;
  cm_stage(sk, CM_KEYS, CM_KEYS, m.k + (long long)first * m.ld_qk + (long long)group * m.group_qk + n0, m.ld_qk, n, keys);
  cm_stage(sv, CM_COLS, CM_COLS, m.v + (long long)first * m.ld_v + (long long)h * m.P + p0, m.ld_v, n, cols);
  __syncthreads();
  float left = 0.f;
  if (tid < CM_TOKENS) {
    left = 1.f;
    for (int u = tid + 1; u < n; ++u) left *= sa[u];
    if (tid == 0 && blockIdx.z == 0) m.chunk_decay[(long long)b * m.H + h] = left * sa[0];
    if (tid < n) left *= m.weight[(long long)(first + tid) * m.H + h];
  }
  __syncthreads();
  if (tid < CM_TOKENS) sa[tid] = tid < n ? left : 0.f;
  __syncthreads();
  for (int i = tid; i < CM_TOKENS * CM_COLS; i += CM_THREADS) sv[i] *= sa[i / CM_COLS];
  __syncthreads();
  // columns 4 tp + 32 i + c, keys 4 tn + 64 j + c
  const int tp = tid >> 4, tn = tid & 15;
  float acc[8][8] = {};
#pragma unroll 2
  for (int s = 0; s < n; ++s) {
    float x[8], z[8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(sv + s * CM_COLS + 4 * tp + 32 * i);
      const float4 k = *reinterpret_cast<const float4*>(sk + s * CM_KEYS + 4 * tn + 64 * i);
      x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
      z[4 * i] = k.x; z[4 * i + 1] = k.y; z[4 * i + 2] = k.z; z[4 * i + 3] = k.w;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(x[i], z[j], acc[i][j]);
  }
  float* out = m.chunk_state + ((long long)b * m.H + h) * ((long long)m.N * m.P);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int p = p0 + 4 * tp + 32 * (i >> 2) + (i & 3);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int key = n0 + 4 * tn + 64 * j;
      if (p < m.P && key < m.N)
        *reinterpret_cast<float4*>(out + (long long)p * m.N + key) =
            make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
    }
  }
}

constexpr int CM_OUT_FLOATS = 2 * CM_TOKENS * (CM_KEYS + 4) + CM_TOKENS * (CM_TOKENS + 4) + CM_COLS * (CM_TOKENS + 4) + 2 * CM_TOKENS;

// grid (H, chunks, tiles of 64 columns): the chunk's outputs from the state it starts from.
static __global__ void __launch_bounds__(CM_THREADS) chunk_out_kernel(ChunkMatrix m) {
  extern __shared__ __align__(16) float sm[];
  constexpr int PITCH = CM_KEYS + 4, SHORT = CM_TOKENS + 4;
  float* sq = sm;                                    // [64 tokens][128]
  float* ss = sq + CM_TOKENS * PITCH;                // [64 columns][128]: the state, keys last
  float* sg = ss + CM_COLS * PITCH;                  // [64 tokens][64]: d(t, s) w_s (q_t . k_s)
  float* sv = sg + CM_TOKENS * SHORT;                // [64 columns][64 tokens]
  float* sa = sv + CM_COLS * SHORT;                  // a_t
  float* sd = sa + CM_TOKENS;                        // d(t, 0)
  const int h = blockIdx.x, p0 = blockIdx.z * CM_COLS, tid = threadIdx.x;
  int b, first, n;
  if (!cm_chunk(m, blockIdx.y, b, first, n)) return;
  const int cols = min(CM_COLS, m.P - p0), group = h / m.heads_per_group, groups = m.H / m.heads_per_group;
  if (tid < CM_TOKENS) sa[tid] = tid < n ? m.decay[(long long)(first + tid) * m.H + h] : 1.f;
  cm_stage(sg, SHORT, CM_TOKENS, m.scores + ((long long)b * groups + group) * (CM_TOKENS * CM_TOKENS), CM_TOKENS, n, CM_TOKENS);
  const float* v = m.v + (long long)first * m.ld_v + (long long)h * m.P + p0;
  bool wild = false;
  for (int i = tid; i < CM_TOKENS * CM_COLS; i += CM_THREADS) {
    const int t = i / CM_COLS, c = i - t * CM_COLS;
    const float x = (t < n && c < cols) ? v[t * m.ld_v + c] : 0.f;
    wild |= !isfinite(x);
    sv[c * SHORT + t] = x;
  }
  wild = __syncthreads_or(wild);     // then a token's zero share of a later one would not be nothing
  if (tid < CM_TOKENS) {             // a thread a token s: its share of every later token's output
    const int s = tid;
    float d = s < n ? m.weight[(long long)(first + s) * m.H + h] : 1.f;
    for (int t = 0; t < n; ++t) {
      if (t > s) d *= sa[t];
      sg[t * SHORT + s] = t >= s ? d * sg[t * SHORT + s] : 0.f;
    }
  } else {                           // and a thread a token t: what is left of the state there
    const int t = tid - CM_TOKENS;
    float d = 1.f;
    for (int u = 0; u <= t && u < n; ++u) d *= sa[u];
    sd[t] = d;
  }
  const CmPlace place;
  const float* state = m.chunk_state + ((long long)b * m.H + h) * ((long long)m.N * m.P);
  float acc[8][8] = {};
  for (int n0 = 0; n0 < m.N; n0 += CM_KEYS) {
    const int keys = min(CM_KEYS, m.N - n0);
    if (n0) __syncthreads();
    cm_stage(sq, PITCH, CM_KEYS, m.q + (long long)first * m.ld_qk + (long long)group * m.group_qk + n0, m.ld_qk, n, keys);
    cm_stage(ss, PITCH, CM_KEYS, state + (long long)p0 * m.N + n0, m.N, cols, keys);
    __syncthreads();
    cm_dots(acc, place, sq, ss, PITCH, keys >> 2);
  }
  // The two sums are joined one after the other and meet in one multiply-add: every addition less at the size of the result is felt in
  // its last bits.
  float r0[4][8], r[4][8];
  __syncthreads();                   // sq has been read
  cm_join(acc, r0, place, sq);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  if (!wild) cm_dots(acc, place, sg, sv, SHORT, ceil_div(n, 4));
  __syncthreads();                   // the first sums have been read
  cm_join(acc, r, place, sq);
  const float skip = m.skip[h];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = place.ti + 8 * (i + 4 * place.half);
    if (t >= n) continue;
    const float d = sd[t];
    float* out = m.y + (long long)(first + t) * ((long long)m.H * m.P) + (long long)h * m.P + p0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = place.tj + 8 * j;
      if (wild)
        for (int s = 0; s <= t; ++s) r[i][j] = fmaf(sg[t * SHORT + s], sv[c * SHORT + s], r[i][j]);
      if (c < cols) out[c] = fmaf(skip, sv[c * SHORT + t], fmaf(d, r0[i][j], r[i][j]));
    }
  }
}

// grid (ceil(H PN / (256 V)), requests), V the numbers a thread takes (float: 1, float4: 4): an entry of the state walks the
// request's chunks in order (`packed`: at their places, else max_chunks a request apart); four chunks' numbers are on their way at a time. Every chunk's place receives the state it starts
// from, the slot the state after the last chunk.
__device__ __forceinline__ float cm_step(float d, float s, float add) { return fmaf(d, s, add); }
__device__ __forceinline__ float4 cm_step(float d, const float4& s, const float4& add) {
  return make_float4(fmaf(d, s.x, add.x), fmaf(d, s.y, add.y), fmaf(d, s.z, add.z), fmaf(d, s.w, add.w));
}
template <typename V>
__global__ void __launch_bounds__(256) chunk_walk_kernel(float* __restrict__ chunk_state, const float* __restrict__ chunk_decay,
                                                         float* __restrict__ state, long long state_stride,
                                                         const int* __restrict__ state_slot, const int* __restrict__ row_start, int H,
                                                         int PN, int chunk_tokens, int max_chunks, int write_state, int packed) {
  constexpr int EACH = sizeof(V) / 4, AHEAD = 4;
  const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * EACH;
  const int b = blockIdx.y;
  const long long per = (long long)H * PN;
  if (e >= per) return;
  const int h = (int)(e / PN);
  const int chunks = ceil_div(row_start[b + 1] - row_start[b], chunk_tokens);
  if (chunks <= 0) return;
  V* slot = reinterpret_cast<V*>(state + (long long)state_slot[b] * state_stride + e);
  const long long place = packed ? cm_place(row_start, b) : (long long)b * max_chunks;
  float* at = chunk_state + place * per + e;
  const float* decay = chunk_decay + place * H + h;
  V S = *slot;
  for (int c = 0; c < chunks; c += AHEAD) {
    V add[AHEAD];
    float d[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c + i < chunks) {
        add[i] = *reinterpret_cast<const V*>(at + (c + i) * per);
        d[i] = decay[(long long)(c + i) * H];
      }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c + i < chunks) {
        *reinterpret_cast<V*>(at + (c + i) * per) = S;
        S = cm_step(d[i], S, add[i]);
      }
  }
  if (write_state) *slot = S;
}
static int chunk_walk(float* chunk_state, const float* chunk_decay, float* state, long long state_stride, const int* state_slot,
                      const int* row_start, int requests, int H, int PN, int chunk_tokens, int max_chunks, int write_state, int packed,
                      cudaStream_t stream) {
  const long long per = (long long)H * PN;
  const bool pieces = PN % 4 == 0 && state_stride % 4 == 0 && (((uintptr_t)chunk_state | (uintptr_t)state) & 15) == 0;
  if (pieces)
    chunk_walk_kernel<float4><<<dim3((unsigned)ceil_div64(per, 1024), requests), 256, 0, stream>>>(
        chunk_state, chunk_decay, state, state_stride, state_slot, row_start, H, PN, chunk_tokens, max_chunks, write_state, packed);
  else
    chunk_walk_kernel<float><<<dim3((unsigned)ceil_div64(per, 256), requests), 256, 0, stream>>>(
        chunk_state, chunk_decay, state, state_stride, state_slot, row_start, H, PN, chunk_tokens, max_chunks, write_state, packed);
  TL_LAUNCH_CHECK();
  return 0;
}

// The three kernels' sizes and launches; `walk` puts the states the chunks start from in the place of what they add.
template <typename Walk>
static int chunk_matrix_run(const ChunkMatrix& m, int chunks, Walk walk, cudaStream_t stream) {
  const int groups = m.H / m.heads_per_group, key_tiles = ceil_div(m.N, CM_KEYS), col_tiles = ceil_div(m.P, CM_COLS);
  constexpr int score_bytes = 2 * CM_TOKENS * (CM_KEYS + 4) * 4;
  constexpr int end_bytes = (CM_TOKENS * (CM_KEYS + CM_COLS) + CM_TOKENS) * 4, out_bytes = CM_OUT_FLOATS * 4;
  cudaError_t e = cudaFuncSetAttribute(chunk_score_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, score_bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_end_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, end_bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, out_bytes);
  if (e != cudaSuccess) return (int)e;
  chunk_score_kernel<<<dim3(groups, chunks), CM_THREADS, score_bytes, stream>>>(m);
  TL_LAUNCH_CHECK();
  chunk_end_kernel<<<dim3(m.H, chunks, col_tiles * key_tiles), CM_THREADS, end_bytes, stream>>>(m);
  TL_LAUNCH_CHECK();
  if (int err = walk()) return err;
  chunk_out_kernel<<<dim3(m.H, chunks, col_tiles), CM_THREADS, out_bytes, stream>>>(m);
  TL_LAUNCH_CHECK();
  return 0;
}

// Whether the pieces fit: keys and values in 16-byte pieces, rows and bases aligned.
static inline bool chunk_matrix_fits(const ChunkMatrix& m) {
  const uintptr_t all = (uintptr_t)m.q | (uintptr_t)m.k | (uintptr_t)m.v | (uintptr_t)m.scores | (uintptr_t)m.chunk_state;
  return m.N % 4 == 0 && m.P % 4 == 0 && m.ld_qk % 4 == 0 && m.group_qk % 4 == 0 && m.ld_v % 4 == 0 && (all & 15) == 0;
}

}  // namespace tl
