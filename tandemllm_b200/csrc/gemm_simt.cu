// Matrix products on the CUDA cores with 32-bit accumulation: the true 32-bit path of every projection
// (no tensor-core and no reduced-precision mode is involved), and a plain fallback for bfloat16 inputs.
//
//   C[m, n] = sum_k A[m, k] * W[n, k] (+ bias[n])            both operands row-major with k contiguous
//
// The order in which an output's products are added depends on k alone in each kernel: ascending, by one thread, in the tiled kernels;
// in those for 32-bit operands of whole 16-byte pieces the eight chains described there. So in every grouped product, and with 32-bit
// operands of whole pieces, more than 64 outputs and a k of up to 256, a row's result
// does not depend on how many other rows the call has (the reference's row invariance,
// engine/models/lfm2_moe/kernels.py:290-306). Up to 8 rows of a longer k are added more exactly, and plain products of up to 64 outputs,
// of bfloat16 operands and of rows that are not whole pieces have kernels of their own for up to 8 rows, with a warp's or a CTA's lanes
// along k: there a row's last bits differ between
// a call of up to 8 rows and one of more. The same kernel runs the experts: a tile map built on the
// device (moe_route.cu) names, per row tile, the expert whose weights it multiplies by and the rows of
// the expert-sorted pair list it covers; with `swiglu` the epilogue is silu(gate) * up over the two
// halves of the expert's fused [2 I, H] matrix (engine/models/lfm2_moe/ref.py:199-205).
#include "common.cuh"

namespace tl {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

struct GemmParams {
  const void* A;
  const void* W;
  const float* bias;
  void* C;
  long long lda, ldw, ldc, w_group_stride;
  int M, N, K;
  // grouped (nullptr tile_group: plain)
  const int* tile_group;   // [max_tiles] expert of the tile
  const int* tile_row0;    // [max_tiles] first row of the tile in the sorted list
  const int* tile_rows;    // [max_tiles] rows of the tile
  const int* n_tiles;      // [1]
  const int* a_gather;     // [M] or nullptr: A row of sorted row i is a_gather[i] / a_div
  int a_div;
  const float* pair_weight;   // [pairs] or nullptr: the row's weight, applied in front of the activation (gated products)
  const int* weight_index;    // [M] or nullptr: the pair of sorted row i
  float ga0, ga1;          // the constants of a gate form that has some
  int swiglu;              // a gate activation TL_ACT_* (1: SiLU): W holds 2 N rows per group; C = act(A W[0:N]^T) * (A W[N:2N]^T)
                           // (negative: N rows per group, C = act(A W^T) with the code's activation; grouped products only)
  int k_run;                  // > 0: k is cut into runs of so many elements, a CTA each; run z's result begins part_stride floats behind
  long long part_stride;      // the one before it
};

template <typename TIn, typename TOut, bool SWIGLU>
__global__ void __launch_bounds__(256) gemm_tiled_kernel(GemmParams p) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[SWIGLU ? 2 : 1][BK][BN + 4];

  int row0 = blockIdx.y * BM, rows = BM;
  const TIn* W = (const TIn*)p.W;
  if (p.tile_group) {
    const int t = blockIdx.y;
    if (t >= *p.n_tiles) return;
    row0 = p.tile_row0[t];
    rows = p.tile_rows[t];
    W += (long long)p.tile_group[t] * p.w_group_stride;
  } else {
    rows = min(BM, p.M - row0);
  }
  const int col0 = blockIdx.x * BN;
  const TIn* A = (const TIn*)p.A;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;          // thread's 4 columns start at tx*4, 4 rows at ty*4
  const int lr = tid >> 2, lk = (tid & 3) * 4;     // loader: row lr of the tile, k offset lk..lk+3

  // the A row this loader thread reads (-1: out of the tile)
  long long a_row = -1;
  if (lr < rows) {
    const int i = row0 + lr;
    a_row = p.a_gather ? (long long)(p.a_gather[i] / p.a_div) : (long long)i;
  }
  const int w_row = col0 + lr;                      // weight row (output column) this loader thread reads

  float acc[TM][TN];
  float acc2[SWIGLU ? TM : 1][SWIGLU ? TN : 1];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      acc[i][j] = 0.f;
      if constexpr (SWIGLU) acc2[i][j] = 0.f;
    }

  for (int k0 = 0; k0 < p.K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + lk + j;
      float a = 0.f, w = 0.f, w2 = 0.f;
      if (k < p.K) {
        if (a_row >= 0) a = to_f32(A[a_row * p.lda + k]);
        if (w_row < p.N) {
          w = to_f32(W[(long long)w_row * p.ldw + k]);
          if constexpr (SWIGLU) w2 = to_f32(W[(long long)(w_row + p.N) * p.ldw + k]);
        }
      }
      As[lk + j][lr] = a;
      Ws[0][lk + j][lr] = w;
      if constexpr (SWIGLU) Ws[1][lk + j][lr] = w2;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN], b2[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        b[j] = Ws[0][kk][tx * TN + j];
        if constexpr (SWIGLU) b2[j] = Ws[1][kk][tx * TN + j];
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
          if constexpr (SWIGLU) acc2[i][j] = fmaf(a[i], b2[j], acc2[i][j]);
        }
    }
    __syncthreads();
  }

  TOut* C = (TOut*)p.C;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int lr_out = ty * TM + i;
    if (lr_out >= rows) continue;
    const long long r = row0 + lr_out;
    const float rw = SWIGLU ? pair_weight(p.pair_weight, p.weight_index, r) : 1.f;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = col0 + tx * TN + j;
      if (n >= p.N) continue;
      float v = acc[i][j];
      if constexpr (SWIGLU) {
        v = gated(rw * v, rw * acc2[i][j], p.swiglu, p.ga0, p.ga1);
      } else {
        if (p.bias) v += p.bias[n];
        if (p.swiglu < 0) v = gate_activation(v, -p.swiglu);
      }
      C[r * p.ldc + n] = from_f32<TOut>(v);
    }
  }
}

// Few rows (M <= 8): one warp per output column, lanes stride over k. Weight rows are read once, coalesced.
template <typename TIn, typename TOut, int MAXM>
__global__ void __launch_bounds__(256) gemm_skinny_kernel(GemmParams p) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= p.N) return;
  const TIn* A = (const TIn*)p.A;
  const TIn* w = (const TIn*)p.W + (long long)warp * p.ldw;
  float acc[MAXM];
#pragma unroll
  for (int m = 0; m < MAXM; ++m) acc[m] = 0.f;
  for (int k = lane; k < p.K; k += 32) {
    const float wv = to_f32(w[k]);
#pragma unroll
    for (int m = 0; m < MAXM; ++m)
      if (m < p.M) acc[m] = fmaf(to_f32(A[(long long)m * p.lda + k]), wv, acc[m]);
  }
  TOut* C = (TOut*)p.C;
#pragma unroll
  for (int m = 0; m < MAXM; ++m) {
    if (m >= p.M) break;
    float v = warp_sum(acc[m]);
    if (lane == 0) {
      if (p.bias) v += p.bias[warp];
      C[(long long)m * p.ldc + warp] = from_f32<TOut>(v);
    }
  }
}

// Few rows and few output columns (a router's E x H product): one CTA per output column, its 256 threads stride
// over k and their sums are joined in a fixed order (lanes by shuffles, then the 8 warps in order).
template <typename TIn, typename TOut, int MAXM>
__global__ void __launch_bounds__(256) gemm_skinny_narrow_kernel(GemmParams p) {
  __shared__ float part[8][MAXM];
  const int n = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const TIn* A = (const TIn*)p.A;
  const TIn* w = (const TIn*)p.W + (long long)n * p.ldw;
  float acc[MAXM];
#pragma unroll
  for (int m = 0; m < MAXM; ++m) acc[m] = 0.f;
  for (int k = tid; k < p.K; k += 256) {
    const float wv = to_f32(w[k]);
#pragma unroll
    for (int m = 0; m < MAXM; ++m)
      if (m < p.M) acc[m] = fmaf(to_f32(A[(long long)m * p.lda + k]), wv, acc[m]);
  }
#pragma unroll
  for (int m = 0; m < MAXM; ++m) {
    const float v = warp_sum(acc[m]);
    if (lane == 0) part[warp][m] = v;
  }
  __syncthreads();
  if (tid < p.M) {
    float v = 0.f;
#pragma unroll
    for (int wi = 0; wi < 8; ++wi) v += part[wi][tid];
    if (p.bias) v += p.bias[n];
    ((TOut*)p.C)[(long long)tid * p.ldc + n] = from_f32<TOut>(v);
  }
}

// Many rows and few output columns (a router over a prompt portion): a CTA takes 16 rows and all of up to 64
// columns, so that the grid has M / 16 CTAs instead of one column of 64-row tiles. k is walked in order.
template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256) gemm_tall_narrow_kernel(GemmParams p) {
  constexpr int RM = 16, RN = 64, RK = 32;
  __shared__ float As[RK][RM + 1];
  __shared__ float Ws[RK][RN + 1];
  const int tid = threadIdx.x;
  const int row0 = blockIdx.x * RM;
  const int r = tid >> 4, cg = (tid & 15) * 4;
  const TIn* A = (const TIn*)p.A;
  const TIn* W = (const TIn*)p.W;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < p.K; k0 += RK) {
    for (int i = tid; i < RM * RK; i += 256) {
      const int rr = i / RK, kk = i % RK;
      As[kk][rr] = (row0 + rr < p.M && k0 + kk < p.K) ? to_f32(A[(long long)(row0 + rr) * p.lda + k0 + kk]) : 0.f;
    }
    for (int i = tid; i < RN * RK; i += 256) {
      const int nn = i / RK, kk = i % RK;
      Ws[kk][nn] = (nn < p.N && k0 + kk < p.K) ? to_f32(W[(long long)nn * p.ldw + k0 + kk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < RK; ++kk) {
      const float a = As[kk][r];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = fmaf(a, Ws[kk][cg + j], acc[j]);
    }
    __syncthreads();
  }
  if (row0 + r < p.M) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = cg + j;
      if (n < p.N) ((TOut*)p.C)[(long long)(row0 + r) * p.ldc + n] = from_f32<TOut>(acc[j] + (p.bias ? p.bias[n] : 0.f));
    }
  }
}

// ---- 32-bit operands whose rows are whole 16-byte pieces ----
//
// The kernels above fetch a number at a time, wait for a tile before they multiply it and were what a 32-bit prompt
// consisted of. These take 16 bytes a load and keep four stages of 32 k-elements in flight (cp.async).
//
// CTA: BM rows by 64 outputs (gated: 32 gate rows and the 32 up rows of the same outputs), four warps that all hold the whole
// tile and take two of a stage's eight k-quads each; their sums meet in shared memory at the end. What bounds such a
// kernel is the multiply-adds and what shared memory hands to the registers, 128 bytes a clock. The multiply-adds go two an
// instruction (fma.rn.f32x2) on neighbouring k of one output, so both operands lie in registers as they were loaded, and an output
// is two sums, of the even k and of the odd. A 16-byte load feeds 16 multiply-adds with 8 x 8 outputs a thread, as many as the SM
// does meanwhile, and a warp on a tile of its own is what makes 8 x 8 possible with tiles small enough to fill the GPU. Two CTAs of
// four warps share an SM (240 registers a thread); the multiply-add pipe is then 58 % busy, what is lost is two warps a scheduler
// waiting for shared memory and for one another. Measured at 150 rows, eight warps of single multiply-adds -> this: 14336 outputs of
// 2048 281 -> 252 us, 6144 of 2048 144 -> 130 us, 2048 of 2048 and of 7168 140 -> 128 us on average, the experts' gate/up of
// 600 pairs 448 -> 403 us. A thread's rows lie 4 and its columns 8 apart, so a quarter of a warp reads one row or eight neighbouring ones:
// with 36 floats a row the eight meet no bank twice.
//
// A product of few tiles (150 rows against 2048 outputs are 160 CTAs on 148 SMs: twelve SMs with two, and the others wait for them)
// whose sums may stay in parts is cut into runs of k, a CTA each (`simt_runs` in kernels/ops.py).
//
// An output is the sum of eight chains, a warp's even and odd k in ascending order over the quads q = warp (mod 4), added in
// order: which k a chain has depends on k alone, whatever the tile's height, so a row does not depend on the others as long as the
// product is whole; in runs of k, and with up to eight rows of a long k (below), it has other chains. Eight short chains lose less than
// one long one.
//
// Up to 8 rows are bound by the weights' bytes: tiles of 1, 2, 4 or 8 rows and so few outputs (8, 16 or 32) that the weights come
// through as many SMs as there are, a lane an output where it goes (a weight is then read from shared memory once, by one lane), and
// stages of 128 k-elements, eight of them for the narrow tiles, so that enough is in flight. Up to a k of WHOLE the chains and their order are
// the same, and a row's bits do not depend on the rows beside it. Of a longer k the chains are folded into one sum with its rounding
// errors kept beside it, at WHOLE and at every 128 behind, which loses a quarter of what whole chains lose (a head of k 2048); the taller tiles
// have no registers for that, and folding in shared memory cost them 9 % (512 rows against 6144 x 2048 338 -> 370 us).
// 1 and 8 rows, outputs x k: 512 x 256 2.2 and 2.3 us (a warp an output, lanes along k: 3.1 and 4.4), 512 x 1024 3.5 and 4.1 (a CTA an
// output: 3.3 and 3.7), 2048 x 2048 6.9 and 9.1 (a warp for two outputs: 6.8 and 26.5), 65536 x 2048 87 and 126 (81 and 186). Still faster are a CTA an output for some hundred
// outputs of a long k (128 x 1024 2.5 and 2.9 us, 3.4 and 4.0 here) and, for one row alone, a warp for two outputs of many (6144 x 2048 10.6 us, 12.0).
constexpr int FWARPS = 4;
constexpr int FEW_ROWS = 8;
constexpr int WHOLE = 256;              // k up to which a few rows' chains are not folded

template <int BM_, int FN_>
struct F32Tile {
  static constexpr bool FEW = BM_ <= FEW_ROWS;
  static constexpr int FK = FEW ? 128 : 32, PITCH = FK + 4, STAGES = FEW && FN_ <= 16 ? 8 : 4;
  static constexpr int TX = FEW ? FN_ : 8, TY = 32 / TX;              // lanes across outputs and across rows
  static constexpr int TM = BM_ < TY ? 1 : BM_ / TY, TN = FN_ / TX;   // outputs a thread
  static constexpr int STAGE = (BM_ + FN_) * PITCH;                   // floats
  static constexpr int RED = FWARPS * TM * TN * 32;                   // the warps' sums
  static constexpr int SMEM = (STAGES * STAGE > RED ? STAGES * STAGE : RED) * 4;
  static constexpr int PIECES = FK / 4;                               // 16-byte pieces of a staged row
  static constexpr int ROWS_A_PASS = FWARPS * 32 / PIECES;            // rows of [A tile; W tile] that the CTA's threads load at a time
  static constexpr int LOADS = (BM_ + FN_ + ROWS_A_PASS - 1) / ROWS_A_PASS;    // pieces a thread and stage
  static constexpr int CTAS = BM_ == 32 ? 2 : BM_ == 16 ? 3 : 2;      // an SM
};

__device__ __forceinline__ void cp16(uint32_t dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
// two multiply-adds on neighbouring numbers
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float both(unsigned long long v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

// `sub`: how many CTA tiles a tile of the plan is cut into (grouped)
template <int BM_, int FN, bool GATED>
__global__ void __launch_bounds__(FWARPS * 32, F32Tile<BM_, FN>::CTAS) gemm_f32_kernel(GemmParams p, int sub) {
  using T = F32Tile<BM_, FN>;
  constexpr int TM_ = T::TM, TN_ = T::TN, TX = T::TX, TY = T::TY, FK = T::FK, FPITCH = T::PITCH, FSTAGES = T::STAGES;
  extern __shared__ float4 f32_smem[];
  float* tiles = reinterpret_cast<float*>(f32_smem);
  int row0 = blockIdx.y * BM_, rows;
  const float* W = (const float*)p.W;
  if (p.tile_group) {
    const int t = blockIdx.y / sub, off = (blockIdx.y - t * sub) * BM_;
    if (t >= *p.n_tiles) return;
    rows = min(BM_, p.tile_rows[t] - off);
    if (rows <= 0) return;
    row0 = p.tile_row0[t] + off;
    W += (long long)p.tile_group[t] * p.w_group_stride;
  } else {
    rows = min(BM_, p.M - row0);
  }
  constexpr int OUTS = GATED ? FN / 2 : FN;          // outputs a CTA
  const int col0 = blockIdx.x * OUTS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = lane / TX, tx = lane % TX;

  // what this thread loads: a piece of row tid / PIECES and of every ROWS_A_PASS-th behind it of [A tile; W tile]
  const int lrow = tid / T::PIECES, lk = (tid % T::PIECES) * 4;
  const float* src[T::LOADS];
  bool ok[T::LOADS];
#pragma unroll
  for (int i = 0; i < T::LOADS; ++i) {
    const int r = lrow + T::ROWS_A_PASS * i;
    src[i] = W;
    ok[i] = false;
    if (r < BM_) {
      if (r < rows) {
        const int m = row0 + r;
        src[i] = (const float*)p.A + (p.a_gather ? (long long)(p.a_gather[m] / p.a_div) : (long long)m) * p.lda;
        ok[i] = true;
      }
    } else if (r < BM_ + FN) {
      const int j = r - BM_;
      const int n = col0 + (GATED && j >= OUTS ? j - OUTS : j);
      if (n < p.N) {
        src[i] = W + (long long)(GATED && j >= OUTS ? n + p.N : n) * p.ldw;
        ok[i] = true;
      }
    }
  }
  // (a run of k: its sums go to a result of their own, the bias into the first's)
  const int k0 = p.k_run ? (int)blockIdx.z * p.k_run : 0, k_len = p.k_run ? min(p.k_run, p.K - k0) : p.K;
#pragma unroll
  for (int i = 0; i < T::LOADS; ++i)
    if (ok[i]) src[i] += k0;
  const int steps = (k_len + FK - 1) / FK;
  const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(tiles) + (uint32_t)((lrow * FPITCH + lk) * 4);
  auto load = [&](int step) {
    if (step < steps) {
      const int k = step * FK + lk;
      const uint32_t at = smem0 + (uint32_t)((step % FSTAGES) * T::STAGE * 4);
#pragma unroll
      for (int i = 0; i < T::LOADS; ++i)
        if (lrow + T::ROWS_A_PASS * i < BM_ + FN) {
          const bool in = ok[i] && k < k_len;        // (K and a run are multiples of 4)
          cp16(at + (uint32_t)(T::ROWS_A_PASS * i * FPITCH * 4), in ? src[i] + k : W, in);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  unsigned long long acc[TM_][TN_];                   // (sum over even k, sum over odd k)
#pragma unroll
  for (int i = 0; i < TM_; ++i)
#pragma unroll
    for (int j = 0; j < TN_; ++j) acc[i][j] = 0ull;

  // (few rows: what the chains have been folded to, and what the folding lost)
  float high[T::FEW ? TM_ : 1][T::FEW ? TN_ : 1], low[T::FEW ? TM_ : 1][T::FEW ? TN_ : 1];
  auto fold = [&](int m, int j) {
    const float v = both(acc[m][j]), sum = high[m][j] + v, part = sum - high[m][j];
    low[m][j] += (high[m][j] - (sum - part)) + (v - part);
    high[m][j] = sum;
    acc[m][j] = 0ull;
  };
  if constexpr (T::FEW) {
#pragma unroll
    for (int i = 0; i < TM_; ++i)
#pragma unroll
      for (int j = 0; j < TN_; ++j) high[i][j] = low[i][j] = 0.f;
  }

  for (int s = 0; s < FSTAGES - 1; ++s) load(s);
  for (int step = 0; step < steps; ++step) {
    if constexpr (T::FEW) {
      if (step >= WHOLE / FK) {
#pragma unroll
        for (int m = 0; m < TM_; ++m)
#pragma unroll
          for (int j = 0; j < TN_; ++j) fold(m, j);
      }
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();                                  // the stage is here, and everybody is done with the one before
    load(step + FSTAGES - 1);
#pragma unroll
    for (int part = 0; part < FK / 16; ++part) {
      const float* st = tiles + (step % FSTAGES) * T::STAGE + (warp + FWARPS * part) * 4;
      const float* a_at = st + (BM_ < TY ? ty % BM_ : ty) * FPITCH, * w_at = st + (BM_ + tx) * FPITCH;
      ulonglong2 w[TN_];
#pragma unroll
      for (int j = 0; j < TN_; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(w_at + j * TX * FPITCH);
#pragma unroll
      for (int m = 0; m < TM_; ++m) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_at + m * TY * FPITCH);
#pragma unroll
        for (int j = 0; j < TN_; ++j) fma2(acc[m][j], a.x, w[j].x);
#pragma unroll
        for (int j = 0; j < TN_; ++j) fma2(acc[m][j], a.y, w[j].y);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* red = tiles;                                // [warps][TM][TN][32]
#pragma unroll
  for (int m = 0; m < TM_; ++m)
#pragma unroll
    for (int j = 0; j < TN_; ++j) {
      float v = both(acc[m][j]);
      if constexpr (T::FEW) {
        if (steps > WHOLE / FK) {
          fold(m, j);
          v = fabsf(high[m][j]) < INFINITY ? high[m][j] + low[m][j] : high[m][j];      // (an infinity loses no finite rest)
        }
      }
      red[((warp * TM_ + m) * TN_ + j) * 32 + lane] = v;
    }
  __syncthreads();
  auto sum = [&](int m, int j) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < FWARPS; ++w) v += red[((w * TM_ + m) * TN_ + j) * 32 + lane];
    return v;
  };
  float* C = (float*)p.C + (long long)blockIdx.z * p.part_stride;
  const float* bias = blockIdx.z == 0 ? p.bias : nullptr;
  // a warp stores every fourth of the TM x TN blocks of outputs (gated: the gate's column blocks are the first four)
  constexpr int BLOCKS = GATED ? 4 : TN_;
#pragma unroll
  for (int i = 0; i < (TM_ * BLOCKS + FWARPS - 1) / FWARPS; ++i) {
    const int m = (warp + FWARPS * i) / BLOCKS, j = (warp + FWARPS * i) % BLOCKS;
    if (m >= TM_) break;
    const int lr = ty + TY * m, n = col0 + tx + TX * j;
    const float v = sum(m, j), u = GATED ? sum(m, j + 4) : 0.f;
    if (lr >= rows || n >= p.N) continue;
    const long long r = row0 + lr;
    if constexpr (GATED) {
      const float rw = pair_weight(p.pair_weight, p.weight_index, r);
      C[r * p.ldc + n] = gated(rw * v, rw * u, p.swiglu, p.ga0, p.ga1);
    } else {
      const float x = v + (bias ? bias[n] : 0.f);
      C[r * p.ldc + n] = p.swiglu < 0 ? gate_activation(x, -p.swiglu) : x;
    }
  }
}

template <int BM_, int FN, bool GATED>
static int launch_f32(const GemmParams& p, int max_tiles, cudaStream_t stream) {
  const int sub = p.tile_group ? BM / BM_ : 1;       // (a plan's tiles hold at most BM rows)
  constexpr int SMEM = F32Tile<BM_, FN>::SMEM;
  auto kernel = gemm_f32_kernel<BM_, FN, GATED>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const unsigned y = p.tile_group ? (unsigned)(max_tiles * sub) : (unsigned)ceil_div(p.M, BM_);
  kernel<<<dim3(ceil_div(p.N, GATED ? FN / 2 : FN), y, p.k_run ? ceil_div(p.K, p.k_run) : 1), FWARPS * 32, SMEM, stream>>>(p, sub);
  return 0;
}

// Tiles of 8, 16 or 32 outputs: the widest of which there is one for every SM (16 in place of 32: 6144 x 2048 14.3 us for a row, 11.8 so;
// 64 in place of 32: 65536 x 2048 93 us, 88 so).
template <int BM_>
static int launch_f32_few(const GemmParams& p, cudaStream_t stream) {
  if (p.N <= 8 * sm_count()) return launch_f32<BM_, 8, false>(p, 0, stream);
  if (p.N <= 32 * sm_count()) return launch_f32<BM_, 16, false>(p, 0, stream);
  return launch_f32<BM_, 32, false>(p, 0, stream);
}

// Whether the 16-byte kernels take these operands: rows that are whole pieces, a grid within its limit, and not a product of so few
// outputs (a router's) that it has kernels of its own.
static bool f32_pieces(const GemmParams& p, int max_tiles) {
  if (p.K % 4 || p.lda % 4 || p.ldw % 4 || p.w_group_stride % 4 || ((uintptr_t)p.A & 15) || ((uintptr_t)p.W & 15)) return false;
  if (p.tile_group) return (long long)max_tiles * (BM / 16) <= 65535;
  return p.N > 64 && ceil_div(p.M, 16) <= 65535;
}

static int launch_f32_any(const GemmParams& p, int max_tiles, cudaStream_t stream) {
  if (!p.tile_group && p.M <= FEW_ROWS) {
    if (p.M == 1) return launch_f32_few<1>(p, stream);
    if (p.M == 2) return launch_f32_few<2>(p, stream);
    return p.M <= 4 ? launch_f32_few<4>(p, stream) : launch_f32_few<8>(p, stream);
  }
  // tiles of 16 rows for what fits one; grouped, where an expert has as few on average (max_tiles: the experts or more)
  const bool low = p.tile_group ? p.M <= 10 * max_tiles : p.M <= 16;
  if (p.swiglu > 0) return low ? launch_f32<16, 64, true>(p, max_tiles, stream) : launch_f32<32, 64, true>(p, max_tiles, stream);
  return low ? launch_f32<16, 64, false>(p, max_tiles, stream) : launch_f32<32, 64, false>(p, max_tiles, stream);
}

template <typename TIn, typename TOut>
static int launch(const GemmParams& p, int max_tiles, cudaStream_t stream) {
  if constexpr (sizeof(TIn) == 4) {
    if (f32_pieces(p, max_tiles)) return launch_f32_any(p, max_tiles, stream);
  }
  if (!p.tile_group && !p.swiglu && p.N <= 64 && p.M > 64) {
    gemm_tall_narrow_kernel<TIn, TOut><<<ceil_div(p.M, 16), 256, 0, stream>>>(p);
    return 0;
  }
  if (!p.tile_group && !p.swiglu && p.M <= 8) {
    if (p.N <= 512 && p.K >= 512) {
      gemm_skinny_narrow_kernel<TIn, TOut, 8><<<p.N, 256, 0, stream>>>(p);
      return 0;
    }
    const int blocks = ceil_div(p.N, 8);
    gemm_skinny_kernel<TIn, TOut, 8><<<blocks, 256, 0, stream>>>(p);
    return 0;
  }
  dim3 grid(ceil_div(p.N, BN), p.tile_group ? max_tiles : ceil_div(p.M, BM));
  if (p.swiglu > 0)
    gemm_tiled_kernel<TIn, TOut, true><<<grid, 256, 0, stream>>>(p);
  else
    gemm_tiled_kernel<TIn, TOut, false><<<grid, 256, 0, stream>>>(p);
  return 0;
}

}  // namespace tl

using namespace tl;

// in_dtype / out_dtype: TL_FP32 or TL_BF16 (an fp32 input with a bf16 output is refused).
extern "C" int tl_gemm_simt(const void* A, long long lda, const void* W, long long ldw, const float* bias, void* C,
                            long long ldc, int M, int N, int K, int in_dtype, int out_dtype, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  TL_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: M %d N %d K %d", M, N, K);
  TL_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm: strides lda %lld ldw %lld ldc %lld for M %d N %d K %d", lda, ldw,
             ldc, M, N, K);
  TL_REQUIRE(ceil_div(M, BM) <= 65535, "gemm: %d rows exceed the grid limit of %d", M, 65535 * BM);
  GemmParams p = {};
  p.A = A; p.W = W; p.bias = bias; p.C = C; p.lda = lda; p.ldw = ldw; p.ldc = ldc;
  p.M = M; p.N = N; p.K = K; p.a_div = 1;
  int e = 0;
  if (in_dtype == TL_FP32 && out_dtype == TL_FP32) e = launch<float, float>(p, 0, stream);
  else if (in_dtype == TL_BF16 && out_dtype == TL_BF16) e = launch<bf16, bf16>(p, 0, stream);
  else if (in_dtype == TL_BF16 && out_dtype == TL_FP32) e = launch<bf16, float>(p, 0, stream);
  else TL_REQUIRE(false, "gemm: input dtype %d with output dtype %d is not implemented", in_dtype, out_dtype);
  if (e) return e;
  TL_LAUNCH_CHECK();
  return 0;
}

// The 32-bit product in runs of `run` k-elements (a multiple of 32; 32-bit operands whose rows are whole 16-byte pieces, more than 64
// outputs): C receives every run's sums, [runs][M][ldc], for the caller to add in order; the bias is in the first.
extern "C" int tl_gemm_simt_runs(const float* A, long long lda, const float* W, long long ldw, const float* bias, float* C, long long ldc,
                                 int M, int N, int K, int run, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  TL_REQUIRE(M > 0 && N > 0 && K > 0 && run > 0 && run % 32 == 0, "gemm in runs: M %d N %d K %d, runs of %d", M, N, K, run);
  TL_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm in runs: strides lda %lld ldw %lld ldc %lld for M %d N %d K %d", lda, ldw, ldc, M, N, K);
  GemmParams p = {};
  p.A = A; p.W = W; p.bias = bias; p.C = C; p.lda = lda; p.ldw = ldw; p.ldc = ldc;
  p.M = M; p.N = N; p.K = K; p.a_div = 1; p.k_run = run; p.part_stride = (long long)M * ldc;
  TL_REQUIRE(f32_pieces(p, 0) && M > FEW_ROWS && ceil_div(K, run) <= 65535, "gemm in runs: %d rows of %d against %d outputs", M, K, N);
  if (int e = launch_f32_any(p, 0, stream)) return e;
  TL_LAUNCH_CHECK();
  return 0;
}

// Grouped product over the expert-sorted pair list. Sorted row i multiplies A row (a_gather ? a_gather[i] / a_div : i)
// by the weights of its tile's expert and writes C row i. `row_weight` and `weight_index` (gated form only): see `pair_weight`.
extern "C" int tl_gemm_simt_grouped(const void* A, long long lda, const int* a_gather, int a_div, const void* W,
                                    long long ldw, long long w_group_stride, void* C, long long ldc, int n_sorted_rows,
                                    int N, int K, const int* tile_group, const int* tile_row0, const int* tile_rows,
                                    const int* n_tiles, int max_tiles, int swiglu, int in_dtype, int out_dtype,
                                    const float* row_weight, const int* weight_index, cudaStream_t stream) {
  if (n_sorted_rows == 0 || N == 0) return 0;
  TL_REQUIRE(n_sorted_rows > 0 && N > 0 && K > 0 && max_tiles > 0, "grouped gemm: rows %d N %d K %d tiles %d",
             n_sorted_rows, N, K, max_tiles);
  TL_REQUIRE(max_tiles <= 65535, "grouped gemm: %d row tiles exceed the grid limit", max_tiles);
  TL_REQUIRE(a_div >= 1, "grouped gemm: a_div %d", a_div);
  TL_REQUIRE(!row_weight || swiglu > 0, "grouped gemm: row weights need the gated form (activation %d)", swiglu);
  GemmParams p = {};
  p.A = A; p.W = W; p.bias = nullptr; p.C = C; p.lda = lda; p.ldw = ldw; p.ldc = ldc;
  p.w_group_stride = w_group_stride; p.M = n_sorted_rows; p.N = N; p.K = K;
  p.tile_group = tile_group; p.tile_row0 = tile_row0; p.tile_rows = tile_rows; p.n_tiles = n_tiles;
  p.a_gather = a_gather; p.a_div = a_div; p.swiglu = swiglu; p.pair_weight = row_weight; p.weight_index = weight_index;
  p.ga0 = tl_gate_constants[0]; p.ga1 = tl_gate_constants[1];
  int e = 0;
  if (in_dtype == TL_FP32 && out_dtype == TL_FP32) e = launch<float, float>(p, max_tiles, stream);
  else if (in_dtype == TL_BF16 && out_dtype == TL_BF16) e = launch<bf16, bf16>(p, max_tiles, stream);
  else if (in_dtype == TL_BF16 && out_dtype == TL_FP32) e = launch<bf16, float>(p, max_tiles, stream);
  else TL_REQUIRE(false, "grouped gemm: input dtype %d with output dtype %d is not implemented", in_dtype, out_dtype);
  if (e) return e;
  TL_LAUNCH_CHECK();
  return 0;
}

extern "C" int tl_gemm_simt_tile_rows() { return BM; }
