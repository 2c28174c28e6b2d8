// Dense policy-network path: forward chain, backward (cross-entropy on a masked
// softmax head), split-K weight gradients and the fused SGD update.
//
// Forward replaces the per-node device functions the reference's graph
// interpreter emits (BlockMatmul -> BlockMap relu -> BlockRowMap head,
// ml/layers.spi:181-252, one global-memory pass per node): here every layer is
// one tensor-core GEMM whose epilogue applies bias, ReLU, the storage rounding
// of the next layer's input and, on the last layer, the row head.
//
// The reference has no backward pass, loss or optimiser (its training is CEM /
// tabular CFR, ml/cem.spi:99-146); dgrad (NN), wgrad (TN) and SGD below follow
// the benchmark's training configurations and are pinned by the NumPy oracle.
//
// Memory model (caller-owned, as in ml/layers.spi:127-172): a flat fp32 master
// parameter buffer [W0 | b0 | W1 | b1 | ...] with 64-element aligned segments,
// a compute copy of the same layout in the storage type of the arithmetic class,
// a flat fp32 gradient buffer of the same layout (the unit of the data-parallel
// all-reduce), per-layer activation buffers and one scratch buffer.
#include "common.cuh"

#include <mutex>
#include <type_traits>

namespace {

constexpr int MLP_MAX_LAYERS = 16;
constexpr long long SEG_ALIGN = 64;  // elements; 256 B in fp32, 128 B in 16-bit storage

long long align_up(long long x, long long a) { return (x + a - 1) / a * a; }

int storage_dtype(int in_dtype) { return in_dtype == SB_TF32 ? SB_TF32 : in_dtype; }

int check_layout(const char* who, int n_layers, const int* sizes, int batch, int in_dtype) {
  if (n_layers < 1 || n_layers > MLP_MAX_LAYERS) return sb_fail(SB_ERR_BAD_ARG, "%s: n_layers must be in [1, %d]", who, MLP_MAX_LAYERS);
  if (!sizes) return sb_fail(SB_ERR_BAD_ARG, "%s: sizes is null", who);
  for (int i = 0; i <= n_layers; ++i)
    if (sizes[i] < 1) return sb_fail(SB_ERR_BAD_ARG, "%s: sizes[%d] = %d", who, i, sizes[i]);
  if (batch < 0) return sb_fail(SB_ERR_BAD_ARG, "%s: negative batch", who);
  if (in_dtype != SB_TF32 && in_dtype != SB_BF16 && in_dtype != SB_F16)
    return sb_fail(SB_ERR_UNSUPPORTED, "%s: arithmetic class must be SB_TF32, SB_BF16 or SB_F16", who);
  return SB_OK;
}

// Rows of a weight segment: the fan-out padded to a multiple of 8 so that the
// transposed uses of dY (wgrad A operand, dgrad inner dimension) have 16-byte
// row pitches.  Padding rows stay zero: their gradients are zero.
int padded_out(int fan_out) { return (fan_out + 7) / 8 * 8; }

void param_offsets(int n_layers, const int* sizes, long long* off) {
  long long cur = 0;
  for (int i = 0; i < n_layers; ++i) {
    off[2 * i] = cur;
    cur = align_up(cur + (long long)padded_out(sizes[i + 1]) * sizes[i], SEG_ALIGN);
    off[2 * i + 1] = cur;
    cur = align_up(cur + sizes[i + 1], SEG_ALIGN);
  }
  off[2 * n_layers] = cur;
}

// d logits of cross-entropy(masked softmax): (p * sum(t) - t) / global_batch on
// legal entries, 0 elsewhere; also accumulates the loss.  One thread per row.
// LD > 0: the padded row width is the compile-time LD and the column sums of
// d logits -- the head layer's bias gradient -- are added to db here (a CTA-wide
// reduction, then LD atomics per CTA) instead of in a pass of their own over dY.
template <typename DyT, bool ROUND_TF32, int LD>
__global__ void ce_grad_kernel(const float* __restrict__ probs, const float* __restrict__ target,
                               const uint8_t* __restrict__ mask, DyT* __restrict__ dy, int rows, int n,
                               int ld, float inv_batch, float* __restrict__ loss, float* __restrict__ db) {
  constexpr int NACC = LD > 0 ? LD : 1;
  __shared__ float colpart[8][NACC];
  sb_grid_dependency_wait();
  sb_grid_dependents_launch();
  float local = 0.f;
  float colacc[NACC];
#pragma unroll
  for (int j = 0; j < NACC; ++j) colacc[j] = 0.f;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
       r += (long long)gridDim.x * blockDim.x) {
    const float* pr = probs + r * n;
    const float* tr = target + r * n;
    const uint8_t* mr = mask ? mask + r * n : nullptr;
    if (LD > 0 && sizeof(DyT) == 2) {
      // The whole row in registers first (an even row length keeps every row 8-byte aligned:
      // probabilities and targets then come as two-float loads); then one or two 16-byte stores of
      // the padded 16-bit row instead of LD two-byte ones 2 * LD bytes apart.
      float pv[NACC], tv[NACC];
      if ((n & 1) == 0) {
#pragma unroll
        for (int j = 0; j < NACC; j += 2) {
          float2 a = make_float2(0.f, 0.f), b = a;
          if (j < n) {
            a = __ldg(reinterpret_cast<const float2*>(pr + j));
            b = __ldg(reinterpret_cast<const float2*>(tr + j));
          }
          pv[j] = a.x; pv[j + 1] = a.y;
          tv[j] = b.x; tv[j + 1] = b.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < NACC; ++j) {
          pv[j] = j < n ? __ldg(pr + j) : 0.f;
          tv[j] = j < n ? __ldg(tr + j) : 0.f;
        }
      }
      bool legal[NACC];
      float ts = 0.f;
#pragma unroll
      for (int j = 0; j < NACC; ++j) {
        legal[j] = j < n && (!mr || mr[j]);
        if (legal[j]) ts += tv[j];
      }
      __align__(16) DyT packed[NACC];
#pragma unroll
      for (int j = 0; j < NACC; ++j) {
        float g = 0.f;
        if (legal[j]) {
          g = (pv[j] * ts - tv[j]) * inv_batch;
          local -= tv[j] * __logf(fmaxf(pv[j], 1e-38f));
        }
        colacc[j] += g;
        packed[j] = (DyT)g;
      }
      uint4* dst = reinterpret_cast<uint4*>(dy + r * ld);
#pragma unroll
      for (int q = 0; q < NACC / 8; ++q) dst[q] = reinterpret_cast<const uint4*>(packed)[q];
      continue;
    }
    float tsum = 0.f;
    for (int j = 0; j < n; ++j)
      if (!mr || mr[j]) tsum += tr[j];
    auto one = [&](int j) {
      const bool lg = j < n && (!mr || mr[j]);
      float g = 0.f;
      if (lg) {
        const float pj = pr[j], tj = tr[j];
        g = (pj * tsum - tj) * inv_batch;
        local -= tj * __logf(fmaxf(pj, 1e-38f));
      }
      if (ROUND_TF32) {
        uint32_t u = __float_as_uint(g);
        u += 0x0fffu + ((u >> 13) & 1u);
        g = __uint_as_float(u & 0xffffe000u);
      }
      if (sizeof(DyT) == 4) reinterpret_cast<float*>(dy)[r * ld + j] = g;
      else if (sizeof(DyT) == 2) dy[r * ld + j] = (DyT)g;
      return g;
    };
    if (LD > 0) {
#pragma unroll
      for (int j = 0; j < NACC; ++j) colacc[j] += one(j);
    } else {
      for (int j = 0; j < ld; ++j) one(j);
    }
  }
  if (loss) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local != 0.f) atomicAdd(loss, local * inv_batch);
  }
  if (LD > 0 && db) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < NACC; ++j) {
      float v = colacc[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) colpart[warp][j] = v;
    }
    __syncthreads();
    if (threadIdx.x < NACC && (int)threadIdx.x < n) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) t += colpart[w][threadIdx.x];
      if (t != 0.f) atomicAdd(db + threadIdx.x, t);
    }
  }
}

// Column sums of dY [rows, n] -> db[n] (bias gradient).  A block owns a slab of
// rows and a strip of 32 * VEC columns; each thread reads 16-byte pieces (VEC
// elements) so that a warp covers 512 contiguous bytes of a row, the 8 warps
// take alternate rows, and the block's partial sums are combined with atomics
// into a zeroed output (fp32, run-dependent order over a few hundred terms).
template <typename DyT>
__global__ void __launch_bounds__(256)
colsum_kernel(const DyT* __restrict__ dy, float* __restrict__ db, int rows, int n, int rows_per_block) {
  constexpr int VEC = 16 / sizeof(DyT);
  __shared__ float part[8][32 * VEC + 1];
  sb_grid_dependency_wait();
  sb_grid_dependents_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col0 = (blockIdx.x * 32 + lane) * VEC;
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(rows, r0 + rows_per_block);
  float s[VEC];
#pragma unroll
  for (int t = 0; t < VEC; ++t) s[t] = 0.f;
  const bool vec_ok = (n % VEC == 0) && ((reinterpret_cast<uintptr_t>(dy) & 15) == 0) && col0 + VEC <= n;
  if (vec_ok) {
    for (int r = r0 + warp; r < r1; r += 8) {
      const uint4 raw = *reinterpret_cast<const uint4*>(dy + (long long)r * n + col0);
      const DyT* e = reinterpret_cast<const DyT*>(&raw);
#pragma unroll
      for (int t = 0; t < VEC; ++t) s[t] += (float)e[t];
    }
  } else {
    for (int r = r0 + warp; r < r1; r += 8)
#pragma unroll
      for (int t = 0; t < VEC; ++t)
        if (col0 + t < n) s[t] += (float)dy[(long long)r * n + col0 + t];
  }
#pragma unroll
  for (int t = 0; t < VEC; ++t) part[warp][lane * VEC + t] = s[t];
  __syncthreads();
  for (int j = threadIdx.x; j < 32 * VEC; j += 256) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w][j];
    const int col = blockIdx.x * 32 * VEC + j;
    if (col < n && t != 0.f) atomicAdd(db + col, t);
  }
}

// dgrad of a layer with at most 16 outputs (the head): dX[r, n] = gate(r, n) * sum_k dY[r, k] * W[k, n].
// With so short an inner dimension there is nothing to pipeline: warp-level MMAs have all of K for 16 rows
// and 8 columns, and what bounds the kernel is the output it writes.  A warp keeps the W fragments of NG x 32
// columns and goes down the rows 16 at a time, the next step's dY and sign words (stored [N / 32, rows]) on their way.
// The columns of four MMAs are dealt so that a thread ends up with 8 neighbouring ones of a row: column c of MMA j
// is column 8 (c / 2) + 2 j + c % 2 of the 32, a 16-byte store per row.  Column sums of the output (the bias gradient of
// the layer below) stay in registers over all the rows of a warp, fold over the row warps of a block and are added once.
// The form before this one did the multiply-adds on the CUDA cores: 110 instructions for 8 outputs of 10 terms on twelve
// warps of an SM, issue-bound at half of the slots.  Here it is some 35 on sixteen.  ce_grad, the head's wgrad and this, us, then
// and now: 32 columns, 3 outputs, 65536 rows 24.8 / 18.4; 64 columns 22.7 / 16.3; 256 columns 26.9 / 22.9, 2048 rows 15.1 / 10.9; 1024
// columns, 10 outputs, 65536 rows 92.6 / 74.4.  Rows leave in 128-byte pieces (NG = 2): with 64-byte ones 15 % more (fp16 with more than
// 8 outputs, whose fragments take twice the registers, has them: 512 columns, 10 outputs, 262144 rows 174 / 169); three blocks to
// an SM with 80 registers spill, two steps of 16 rows at a time are the same.

// The products of 16 rows and 8 columns.  KP: registers that hold a thread's part of W per MMA.  bf16: one m16n8k16 on the
// values as they are.  fp16: its subnormals (gradients of a large batch) would be summed with the exponent of the smallest
// normal value, bits of the sum below it lost; as TF32 every fp16 value is a normal one, exactly.  One m16n8k8 has eight k's,
// slot t the even and slot t + 4 the odd one of a thread's pair.
template <typename T, int KP>
struct NarrowMma;
template <int KP>
struct NarrowMma<__nv_bfloat16, KP> {
  static_assert(KP == 2, "all of K in one product");
  uint32_t a[4];
  __device__ __forceinline__ void load(const uint32_t* words) {
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = words[i];
  }
  __device__ __forceinline__ static void weights(uint32_t* b, const uint32_t* words) { b[0] = words[0]; b[1] = words[1]; }
  __device__ __forceinline__ void run(float* c, const uint32_t* b) const {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
  }
};
template <int KP>
struct NarrowMma<__half, KP> {
  static_assert(KP == 2 || KP == 4, "eight or sixteen k's");
  uint32_t a[2 * KP];
  __device__ __forceinline__ static void unpack(uint32_t word, uint32_t& even, uint32_t& odd) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&word));
    even = __float_as_uint(f.x);
    odd = __float_as_uint(f.y);
  }
  __device__ __forceinline__ void load(const uint32_t* words) {
#pragma unroll
    for (int p = 0; p < KP / 2; ++p)
#pragma unroll
      for (int i = 0; i < 2; ++i) unpack(words[2 * p + i], a[4 * p + i], a[4 * p + 2 + i]);
  }
  __device__ __forceinline__ static void weights(uint32_t* b, const uint32_t* words) {
#pragma unroll
    for (int p = 0; p < KP / 2; ++p) unpack(words[p], b[2 * p], b[2 * p + 1]);
  }
  __device__ __forceinline__ void run(float* c, const uint32_t* b) const {
#pragma unroll
    for (int p = 0; p < KP / 2; ++p)
      asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                   : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                   : "r"(a[4 * p]), "r"(a[4 * p + 1]), "r"(a[4 * p + 2]), "r"(a[4 * p + 3]), "r"(b[2 * p]), "r"(b[2 * p + 1]));
  }
};
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// dy [rows, ldy] with ldy 8 or 16 (zero beyond the real outputs), w [.., n] of which k_real rows are read, n a multiple of
// 32 NG, bits [n / 32, rows].  A block's warps: col_warps side by side, the others further down the rows.  FOLD: a single strip
// of blocks, which add once per column; otherwise every row warp does.
template <typename T, int NG, int KP, int THREADS, bool FOLD>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
narrow_dgrad_kernel(const T* __restrict__ dy, int ldy, const T* __restrict__ w, int k_real, int n, const uint32_t* __restrict__ bits,
                    T* __restrict__ dx, float* __restrict__ colsum, int rows, int col_warps) {
  sb_grid_dependency_wait();
  sb_grid_dependents_launch();
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int row_warps = (THREADS / 32) / col_warps;
  const int group = (int)blockIdx.x * col_warps + warp % col_warps, row_warp = warp / col_warps;
  const int col0 = group * 32 * NG;
  const bool active = row_warp < row_warps && col0 < n;
  if (!FOLD && !active) return;
  uint32_t b[NG][4][KP];
#pragma unroll
  for (int h = 0; h < NG; ++h)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 + 32 * h + 8 * (g >> 1) + 2 * j + (g & 1);
      uint32_t words[2];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int k = 2 * t + 8 * p;
        const uint16_t lo = k < k_real ? *reinterpret_cast<const uint16_t*>(w + (long long)k * n + col) : (uint16_t)0;
        const uint16_t hi = k + 1 < k_real ? *reinterpret_cast<const uint16_t*>(w + (long long)(k + 1) * n + col) : (uint16_t)0;
        words[p] = (uint32_t)lo | (uint32_t)hi << 16;
      }
      NarrowMma<T, KP>::weights(b[h][j], words);
    }
  float cs[NG][8];
#pragma unroll
  for (int h = 0; h < NG; ++h)
#pragma unroll
    for (int j = 0; j < 8; ++j) cs[h][j] = 0.f;
  const uint32_t* words = bits + (long long)(col0 >> 5) * rows;
  // Row r of the step (g, g + 8): this thread's pieces of the dY row and the sign words of its columns.
  auto fetch = [&](long long r0, uint32_t* a, uint32_t* gate) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const long long r = r0 + g + 8 * i;
      const bool ok = r < rows;
      a[i] = ok ? __ldg(reinterpret_cast<const uint32_t*>(dy + r * ldy + 2 * t)) : 0u;
      a[2 + i] = ok && ldy > 8 ? __ldg(reinterpret_cast<const uint32_t*>(dy + r * ldy + 2 * t + 8)) : 0u;
#pragma unroll
      for (int h = 0; h < NG; ++h) gate[2 * h + i] = ok ? __ldg(words + (long long)h * rows + r) : 0u;
    }
  };
  const long long stride = 16LL * gridDim.y * row_warps;
  long long r0 = 16LL * ((long long)blockIdx.y * row_warps + row_warp);
  uint32_t a[4], gate[2 * NG], a_next[4], gate_next[2 * NG];
  if (FOLD && !active) r0 = rows;
  fetch(r0, a, gate);
  for (; r0 < rows; r0 += stride) {
    fetch(r0 + stride, a_next, gate_next);
    NarrowMma<T, KP> mma;
    mma.load(a);
#pragma unroll
    for (int h = 0; h < NG; ++h) {
      float c[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
        mma.run(c[j], b[h][j]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {              // rows g and g + 8
        const uint32_t mine = gate[2 * h + i] >> (8 * t);
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = (mine >> j) & 1u ? c[j >> 1][2 * i + (j & 1)] : 0.f;
          cs[h][j] += v[j];
        }
        if (r0 + g + 8 * i < rows)
          *reinterpret_cast<uint4*>(dx + (r0 + g + 8 * i) * n + col0 + 32 * h + 8 * t) =
              make_uint4(pack_pair<T>(v[0], v[1]), pack_pair<T>(v[2], v[3]), pack_pair<T>(v[4], v[5]), pack_pair<T>(v[6], v[7]));
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = a_next[i];
#pragma unroll
    for (int i = 0; i < 2 * NG; ++i) gate[i] = gate_next[i];
  }
  if (!colsum) return;
  // The eight row slots g fold together; lane (g, t) then has column 8 t + g of each 32.  The row warps of a block add up
  // before they add to memory.
  __shared__ float part[FOLD ? THREADS / 32 : 1][32 * NG];
#pragma unroll
  for (int h = 0; h < NG; ++h) {
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v = cs[h][j];
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if (g == j) sum = v;
    }
    if (!FOLD) atomicAdd(colsum + col0 + 32 * h + 8 * t + g, sum);
    else part[warp][32 * h + 8 * t + g] = sum;
  }
  if (!FOLD) return;
  __syncthreads();
  for (int c = (int)threadIdx.x; c < n; c += THREADS) {
    float sum = 0.f;
#pragma unroll 4
    for (int w = c / (32 * NG); w < row_warps * col_warps; w += col_warps) sum += part[w][c % (32 * NG)];
    atomicAdd(colsum + c, sum);
  }
}

// Whether the narrow dgrad kernel serves a layer: a 16-bit storage type, at most 16 (real) outputs,
// whole sign words per row.
bool narrow_dgrad_ok(int fan_out_real, int fan_in, int in_dtype) {
  static int off = -1;
  if (off < 0) {
    const char* e = getenv("SB_NARROW_DGRAD");          // SB_NARROW_DGRAD=0: the tensor-core kernel for every layer
    off = (e && e[0] == '0') ? 1 : 0;
  }
  return !off && (in_dtype == SB_BF16 || in_dtype == SB_F16) && fan_out_real >= 1 && fan_out_real <= 16 && fan_in % 32 == 0;
}

template <typename T>
int narrow_dgrad_launch(const void* dy, int ldy, const void* w, int fan_out_real, int n, const uint32_t* bits, void* dx,
                        float* colsum, int rows, cudaStream_t s) {
  constexpr bool HALF = std::is_same<T, __half>::value;
  const bool long_k = HALF && fan_out_real > 8;
  const int ng = n % 64 == 0 && !long_k ? 2 : 1, groups = n / (32 * ng);
  // A column gets an addition to memory per row warp (`direct`), or one per block of sixteen warps.  Up to 512 columns a row
  // warp is one of two to sixteen of its block: their additions at the end of a launch, up to 2368 to an address, cost up to 4 us
  // (64 columns, 65536 rows: 20.5, folded 16.3) and the accuracy of the sum (relative error 5.0e-7, folded 1.6e-7; 262144 rows
  // 6.8e-7 and 1.7e-7).  Wider ones have a row warp per block, 148 additions at most.  Few rows are done sooner without the
  // meeting: 64 rows of 256 columns 8.3 / 9.0, 256 rows of 32 10.4 / 12.1, but 1024 of 256 10.7 / 10.6, 4096 of 256 11.6 / 11.1.
  const bool direct = groups > 8 || rows <= 512;
  const int threads = direct ? 256 : 512, warps = threads / 32;
  const int col_warps = groups < 8 ? groups : 8, row_warps = warps / col_warps;
  const int strips = (groups + col_warps - 1) / col_warps;
  const int least = direct ? 64 : 16;             // rows of a warp, to pay for its W fragments and its additions
  long long want = ((long long)rows + (long long)least * row_warps - 1) / ((long long)least * row_warps);
  long long most = ((direct ? 2LL : 1LL) * sb_sm_count() + strips - 1) / strips;
  if (most > 65535) most = 65535;
  const dim3 grid((unsigned)strips, (unsigned)(want < 1 ? 1 : want < most ? want : most));
  const T* dyp = reinterpret_cast<const T*>(dy);
  const T* wp = reinterpret_cast<const T*>(w);
  T* dxp = reinterpret_cast<T*>(dx);
#define SB_ND_LAUNCH(NG, KP, THREADS, FOLD) \
  SB_CUDA(sb_launch(narrow_dgrad_kernel<T, NG, KP, THREADS, FOLD>, grid, dim3(THREADS), 0, s, 1, dyp, ldy, wp, fan_out_real, n, bits, dxp, colsum, rows, col_warps))
#define SB_ND_BY_FOLD(NG, KP)                       \
  do {                                              \
    if (direct) SB_ND_LAUNCH(NG, KP, 256, false);   \
    else SB_ND_LAUNCH(NG, KP, 512, true);           \
  } while (0)
  if (long_k) SB_ND_BY_FOLD(1, HALF ? 4 : 2);
  else if (ng == 2) SB_ND_BY_FOLD(2, 2);
  else SB_ND_BY_FOLD(1, 2);
#undef SB_ND_BY_FOLD
#undef SB_ND_LAUNCH
  SB_COUNT_LAUNCH();
  SB_CUDA(cudaGetLastError());
  return SB_OK;
}

// grads[i] = sum over splits of partial[s][i]; deterministic order.
__global__ void splitk_reduce_kernel(const float* __restrict__ partial, float* __restrict__ out,
                                     long long n, int splits) {
  sb_grid_dependency_wait();
  sb_grid_dependents_launch();
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    float s = 0.f;
    for (int k = 0; k < splits; ++k) s += partial[(long long)k * n + i];
    out[i] = s;
  }
}

// params -= lr * grads ; compute copy = params rounded to the storage type.
__global__ void sgd_kernel(float* __restrict__ params, const float* __restrict__ grads,
                           void* __restrict__ compute, long long n, float lr, int dt) {
  sb_grid_dependency_wait();
  sb_grid_dependents_launch();
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    const float w = params[i] - lr * grads[i];
    params[i] = w;
    if (!compute) continue;
    if (dt == SB_BF16) reinterpret_cast<__nv_bfloat16*>(compute)[i] = __float2bfloat16_rn(w);
    else if (dt == SB_F16) reinterpret_cast<__half*>(compute)[i] = __float2half_rn(w);
    else if (dt == SB_TF32) {
      uint32_t u = __float_as_uint(w);
      if ((u & 0x7f800000u) != 0x7f800000u) { u += 0x0fffu + ((u >> 13) & 1u); u &= 0xffffe000u; }
      reinterpret_cast<float*>(compute)[i] = __uint_as_float(u);
    } else reinterpret_cast<float*>(compute)[i] = w;
  }
}

int blocks_for(long long n, int per_block, int cap = 0) {
  if (cap <= 0) cap = sb_sm_count() * 8;
  long long b = (n + per_block - 1) / per_block;
  if (b < 1) b = 1;
  return (int)(b > cap ? cap : b);
}

// Split factor of a wgrad GEMM [out, in] with inner dimension = batch.  A GEMM with more than
// 128 output rows runs on CTA pairs (256 x 256 tiles, 74 pairs).  Model of its time, in k-blocks:
// (waves of work items over the pairs) x (k-blocks per item + a fixed part per item for pipeline
// fill and the tile's reduce-add).  For a 1024 x 1024 layer at a batch of 262144 that picks 9 splits
// (144 items, two full waves) instead of 4 (64 items on 74 pairs, 14 % of the GPU idle), at 32768
// rows still 4; a 256 x 256 layer (one tile) is cut into as many items as there are pairs, which
// measured 23 us against 37 us with 11.  Narrow outputs run on single CTAs, one item each.
int wgrad_splits(int out, int in, int batch, int in_dtype) {
  static int forced = -1;                  // SB_WGRAD_SPLITS=n in the environment fixes the factor (tuning runs)
  if (forced < 0) {
    const char* e = getenv("SB_WGRAD_SPLITS");
    forced = e ? atoi(e) : 0;
    if (forced < 0 || forced > 128) forced = 0;
  }
  const int es = sb_dtype_size(in_dtype);
  const int block_k = 128 / es;
  const int k_blocks = (batch + block_k - 1) / block_k;
  const int max_by_k = k_blocks / 8 > 0 ? k_blocks / 8 : 1;  // keep >= 8 k-blocks per split
  if (forced > 0) return forced < max_by_k ? forced : max_by_k;
  if (out > 128) {
    const int tiles = ((out + 255) / 256) * ((in + 255) / 256);
    const int workers = sb_sm_count() / 2;
    // The fixed part of an item, in k-blocks (about 6 us against 0.55 us per k-block of a pair tile).
    const int item_fixed = 10;
    int best = 1;
    long long best_cost = -1;
    for (int s = 1; s <= 128 && s <= max_by_k; ++s) {
      const long long waves = ((long long)tiles * s + workers - 1) / workers;
      const long long cost = waves * ((k_blocks + s - 1) / s + item_fixed);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best = s;
      }
    }
    return best;
  }
  const int tiles = ((out + 127) / 128) * ((in + 255) / 256);
  int s = sb_sm_count() / (tiles > 0 ? tiles : 1);
  if (s < 1) s = 1;
  if (s > max_by_k) s = max_by_k;
  if (s > 128) s = 128;
  return s;
}

bool wgrad_partials_forced() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("SB_WGRAD_PARTIALS");
    v = (e && e[0] == '1') ? 1 : 0;
  }
  return v == 1;
}

size_t backward_scratch_bytes(int n_layers, const int* sizes, int batch, int in_dtype) {
  const int es = sb_dtype_size(in_dtype);
  int max_w = 0;
  long long max_partial = 0;
  for (int i = 0; i < n_layers; ++i) {
    const int op = padded_out(sizes[i + 1]);
    if (op > max_w) max_w = op;
    const long long p = (long long)wgrad_splits(op, sizes[i], batch, in_dtype) * op * sizes[i];
    if (p > max_partial) max_partial = p;
  }
  const size_t dy = (size_t)align_up((long long)batch * max_w * es, 256);
  return 2 * dy + (size_t)max_partial * 4 + 256;
}

}  // namespace

extern "C" {

int sb_mlp_param_offsets(int n_layers, const int* sizes, long long* offsets) {
  if (!offsets) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_param_offsets: null output");
  int rc = check_layout("sb_mlp_param_offsets", n_layers, sizes, 0, SB_BF16);
  if (rc != SB_OK) return rc;
  param_offsets(n_layers, sizes, offsets);
  return SB_OK;
}

int sb_mlp_forward(int n_layers, const int* sizes, int batch, int in_dtype, const void* x,
                   const void* w_compute, const float* params, void* const* activations,
                   void* const* relu_bits, int head, const uint8_t* mask, float* out, int32_t* actions,
                   void* stream) {
  int rc = check_layout("sb_mlp_forward", n_layers, sizes, batch, in_dtype);
  if (rc != SB_OK) return rc;
  if (batch == 0) return SB_OK;
  if (!x || !w_compute || !out) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward: null pointer");
  if (n_layers > 1 && !activations) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward: activations is null");
  if (head & ~(SB_EPI_MASKED_SOFTMAX | SB_EPI_REGRET_MATCHING | SB_EPI_ARGMAX))
    return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward: head may hold only row-head flags");
  if ((head & SB_EPI_ARGMAX) && !actions) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward: SB_EPI_ARGMAX without an actions buffer");
  long long off[2 * MLP_MAX_LAYERS + 1];
  param_offsets(n_layers, sizes, off);
  const int es = sb_dtype_size(in_dtype);
  const int st = storage_dtype(in_dtype);
  const void* h = x;
  for (int i = 0; i < n_layers; ++i) {
    const bool last = i == n_layers - 1;
    const void* w = reinterpret_cast<const char*>(w_compute) + off[2 * i] * es;
    const float* b = params ? params + off[2 * i + 1] : nullptr;
    int epi = b ? SB_EPI_BIAS : 0;
    void* dst;
    int odt;
    if (last) {
      epi |= head;
      dst = out;
      odt = SB_F32;
    } else {
      if (!activations[i]) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_forward: activations[%d] is null", i);
      epi |= SB_EPI_RELU;
      dst = activations[i];
      odt = st;
      if (relu_bits && relu_bits[i] && sizes[i + 1] % 32 == 0) epi |= SB_EPI_RELU_MASK_OUT;
    }
    void* aux_out = last ? (void*)actions : ((epi & SB_EPI_RELU_MASK_OUT) ? relu_bits[i] : nullptr);
    rc = sb_matmul_ex(0, 1, 1.0f, h, w, 0.0f, dst, batch, sizes[i + 1], sizes[i], in_dtype, odt, epi, b,
                      last ? mask : nullptr, nullptr, aux_out, stream);
    if (rc != SB_OK) return rc;
    h = dst;
  }
  return SB_OK;
}

// ---------------------------------------------------------------------------
// Forward pass for hosts that cannot allocate device memory.
//
// Some callers of this library have no way to obtain the hidden-activation
// workspace that sb_mlp_forward wants: a per-decision game loop that only
// holds the reference's three arenas, a plugin running inside someone else's
// CUDA context with allocation forbidden, or code between cudaStreamBeginCapture
// and EndCapture, where cudaMalloc is illegal.  For them the hidden activations
// live in the fixed array below, which is part of the library image: every GPU
// that loads the library holds these SB_STATIC_WORKSPACE_BYTES until the
// process exits.
//
// In host code the name `g_static_workspace` is only a host-side stand-in for
// the symbol, not a device address; the real address is looked up once per
// device with cudaGetSymbolAddress and that pointer is what the kernels get.
//
// All calls on a device use the one array, so a call waits on the GPU for the
// call before it, whatever streams and host threads the two come from: its
// stream waits for the event that the call before recorded behind its last
// launch.  A stream under capture takes no part in this (its launches run when
// the graph does, and an event of a capture may not be waited for outside it).
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_workspace[SB_STATIC_WORKSPACE_BYTES];

namespace {
struct StaticWorkspace {
  std::mutex lock;                 // held while a call is issued: wait, launches, record
  unsigned char* addr = nullptr;   // device address, looked up on the device's first call
  cudaEvent_t done = nullptr;      // behind the last launch of the last call that was not captured
};
StaticWorkspace g_static_ws[64];

// Looks up what the current device's first call needs; `ws->lock` is held.
int static_workspace_init(StaticWorkspace* ws) {
  if (ws->addr) return SB_OK;
  if (!ws->done) SB_CUDA(cudaEventCreateWithFlags(&ws->done, cudaEventDisableTiming));
  void* p = nullptr;
  SB_CUDA(cudaGetSymbolAddress(&p, g_static_workspace));
  if (!p) return sb_fail(SB_ERR_CUDA, "sb_mlp_forward_static: cudaGetSymbolAddress returned a null address");
  ws->addr = reinterpret_cast<unsigned char*>(p);
  return SB_OK;
}
}  // namespace

int sb_mlp_forward_static(int n_layers, const int* sizes, int batch, int in_dtype, const void* x,
                          const void* w_compute, const float* params, int head, const uint8_t* mask,
                          float* out, int32_t* actions, void* stream) {
  int rc = check_layout("sb_mlp_forward_static", n_layers, sizes, batch, in_dtype);
  if (rc != SB_OK) return rc;
  // Carve one 256-byte aligned slab per hidden layer out of the fixed array.
  const int es = sb_dtype_size(in_dtype);
  void* acts[MLP_MAX_LAYERS];
  size_t offset = 0;
  size_t offsets[MLP_MAX_LAYERS];
  for (int i = 0; i + 1 < n_layers; ++i) {
    offsets[i] = offset;
    offset += (size_t)align_up((long long)batch * sizes[i + 1] * es, 256);
  }
  if (offset > (size_t)SB_STATIC_WORKSPACE_BYTES)
    return sb_fail(SB_ERR_TOO_LARGE,
                   "sb_mlp_forward_static: hidden activations need %zu bytes, the built-in workspace holds %zu; "
                   "use sb_mlp_forward with caller memory for this batch", offset, (size_t)SB_STATIC_WORKSPACE_BYTES);
  int dev = 0;
  SB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return sb_fail(SB_ERR_UNSUPPORTED, "sb_mlp_forward_static: device index %d out of range", dev);
  StaticWorkspace& ws = g_static_ws[dev];
  std::lock_guard<std::mutex> guard(ws.lock);
  rc = static_workspace_init(&ws);
  if (rc != SB_OK) return rc;
  for (int i = 0; i + 1 < n_layers; ++i) acts[i] = ws.addr + offsets[i];
  cudaStream_t s = (cudaStream_t)stream;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  SB_CUDA(cudaStreamIsCapturing(s, &capture));
  const bool ordered = n_layers > 1 && capture == cudaStreamCaptureStatusNone;
  if (ordered) SB_CUDA(cudaStreamWaitEvent(s, ws.done, 0));     // returns at once for an event never recorded
  // Every slab is completely overwritten by its layer before the next layer
  // reads it, so nothing left behind by an earlier call needs clearing.
  rc = sb_mlp_forward(n_layers, sizes, batch, in_dtype, x, w_compute, params, n_layers > 1 ? acts : nullptr,
                      nullptr, head, mask, out, actions, stream);
  // Also behind a call that failed: some of its layers may have been launched.
  if (ordered) SB_CUDA(cudaEventRecord(ws.done, s));
  return rc;
}

int sb_mlp_backward_scratch_bytes(int n_layers, const int* sizes, int batch, int in_dtype, size_t* bytes) {
  if (!bytes) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward_scratch_bytes: null output");
  int rc = check_layout("sb_mlp_backward_scratch_bytes", n_layers, sizes, batch, in_dtype);
  if (rc != SB_OK) return rc;
  *bytes = backward_scratch_bytes(n_layers, sizes, batch, in_dtype);
  return SB_OK;
}

int sb_mlp_backward_dy_offset(int n_layers, const int* sizes, int batch, int in_dtype, int layer, size_t* offset) {
  if (!offset) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward_dy_offset: null output");
  int rc = check_layout("sb_mlp_backward_dy_offset", n_layers, sizes, batch, in_dtype);
  if (rc != SB_OK) return rc;
  if (layer < 0 || layer >= n_layers) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward_dy_offset: layer %d of %d", layer, n_layers);
  int max_w = 0;
  for (int i = 0; i < n_layers; ++i) max_w = max(max_w, padded_out(sizes[i + 1]));
  const size_t dy_bytes = (size_t)align_up((long long)batch * max_w * sb_dtype_size(in_dtype), 256);
  *offset = ((n_layers - 1 - layer) & 1) ? dy_bytes : 0;
  return SB_OK;
}

// Which layers' weight gradients a data-parallel backward pass adds straight into the owners' copies.
static bool layer_grads_go_to_peers(int fan_out_padded, int fan_in, int world) {
  return world > 1 && sb_umma_peer_out_ok(fan_out_padded, fan_in, world);
}

int sb_mlp_dp_fused_layers(int n_layers, const int* sizes, int world_size, int* fused) {
  if (!fused) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_dp_fused_layers: null output");
  int rc = check_layout("sb_mlp_dp_fused_layers", n_layers, sizes, 0, SB_BF16);
  if (rc != SB_OK) return rc;
  for (int i = 0; i < n_layers; ++i) fused[i] = layer_grads_go_to_peers(padded_out(sizes[i + 1]), sizes[i], world_size) ? 1 : 0;
  return SB_OK;
}

static int backward_impl(int n_layers, const int* sizes, int batch, float inv_global_batch, int in_dtype,
                         const void* x, const void* w_compute, void* const* activations,
                         void* const* relu_bits, const float* probs, const uint8_t* mask,
                         const float* target, float* grads, int with_bias, void* scratch,
                         size_t scratch_bytes, float* loss, int first_layer, int last_layer, void* stream,
                         float* const* grads_peers, int world);

int sb_mlp_backward_range(int n_layers, const int* sizes, int batch, float inv_global_batch, int in_dtype,
                          const void* x, const void* w_compute, void* const* activations,
                          void* const* relu_bits, const float* probs, const uint8_t* mask,
                          const float* target, float* grads, int with_bias, void* scratch,
                          size_t scratch_bytes, float* loss, int first_layer, int last_layer, void* stream) {
  return backward_impl(n_layers, sizes, batch, inv_global_batch, in_dtype, x, w_compute, activations, relu_bits, probs,
                       mask, target, grads, with_bias, scratch, scratch_bytes, loss, first_layer, last_layer, stream,
                       nullptr, 1);
}

int sb_mlp_backward_dp(int n_layers, const int* sizes, int batch, float inv_global_batch, int in_dtype,
                       const void* x, const void* w_compute, void* const* activations,
                       void* const* relu_bits, const float* probs, const uint8_t* mask, const float* target,
                       float* const* grads_peers, int world_size, int rank, int with_bias, void* scratch,
                       size_t scratch_bytes, float* loss, void* stream) {
  if (world_size < 1 || world_size > 16 || rank < 0 || rank >= world_size || !grads_peers)
    return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward_dp: rank %d of world size %d, or no table of gradient buffers", rank, world_size);
  for (int r = 0; r < world_size; ++r)
    if (!grads_peers[r]) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward_dp: gradient buffer of rank %d is null", r);
  // This rank's own buffer comes first in the peers table handed down: the launcher's C.
  return backward_impl(n_layers, sizes, batch, inv_global_batch, in_dtype, x, w_compute, activations, relu_bits, probs,
                       mask, target, grads_peers[rank], with_bias, scratch, scratch_bytes, loss, n_layers - 1, 0, stream,
                       grads_peers, world_size);
}

static int backward_impl(int n_layers, const int* sizes, int batch, float inv_global_batch, int in_dtype,
                         const void* x, const void* w_compute, void* const* activations,
                         void* const* relu_bits, const float* probs, const uint8_t* mask,
                         const float* target, float* grads, int with_bias, void* scratch,
                         size_t scratch_bytes, float* loss, int first_layer, int last_layer, void* stream,
                         float* const* grads_peers, int world) {
  int rc = check_layout("sb_mlp_backward", n_layers, sizes, batch, in_dtype);
  if (rc != SB_OK) return rc;
  if (!grads) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward: grads is null");
  if (first_layer < last_layer || first_layer >= n_layers || last_layer < 0)
    return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward: layer range [%d, %d] of %d layers", last_layer, first_layer, n_layers);
  const bool from_top = first_layer == n_layers - 1;
  long long off[2 * MLP_MAX_LAYERS + 1];
  param_offsets(n_layers, sizes, off);
  cudaStream_t s = (cudaStream_t)stream;
  // Zeroes the gradient vector before a pass.  Weight segments that peers add into (data-parallel
  // pass) are left alone: their owner slices are zeroed by the update kernel that consumed them, and a
  // faster rank may already be adding this step's tiles.
  auto zero_grads = [&]() -> int {
    if (!grads_peers || world <= 1) {
      SB_CUDA(cudaMemsetAsync(grads, 0, (size_t)off[2 * n_layers] * 4, s));
      return SB_OK;
    }
    for (int i = 0; i < n_layers; ++i) {
      const bool fused = layer_grads_go_to_peers(padded_out(sizes[i + 1]), sizes[i], world);
      const long long begin = fused ? off[2 * i + 1] : off[2 * i];
      SB_CUDA(cudaMemsetAsync(grads + begin, 0, (size_t)(off[2 * i + 2] - begin) * 4, s));
    }
    return SB_OK;
  };
  if (batch == 0) {
    if (from_top) return zero_grads();
    return SB_OK;
  }
  if (!x || !w_compute || !probs || !target || !scratch)
    return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward: null pointer");
  if (n_layers > 1 && !activations) return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward: activations is null");
  for (int i = 1; i < n_layers; ++i)
    if (sizes[i] % 8 != 0)
      return sb_fail(SB_ERR_UNSUPPORTED, "sb_mlp_backward: hidden width %d is not a multiple of 8", sizes[i]);
  const size_t need = backward_scratch_bytes(n_layers, sizes, batch, in_dtype);
  if (scratch_bytes < need)
    return sb_fail(SB_ERR_BAD_ARG, "sb_mlp_backward: scratch of %zu bytes, %zu needed", scratch_bytes, need);
  if (reinterpret_cast<uintptr_t>(scratch) & 255) return sb_fail(SB_ERR_MISALIGNED, "sb_mlp_backward: scratch must be 256-byte aligned");
  const int es = sb_dtype_size(in_dtype);
  const int st = storage_dtype(in_dtype);
  int max_w = 0;
  for (int i = 0; i < n_layers; ++i) max_w = max(max_w, padded_out(sizes[i + 1]));
  const size_t dy_bytes = (size_t)align_up((long long)batch * max_w * es, 256);
  char* sc = reinterpret_cast<char*>(scratch);
  // The two dY buffers alternate once per dgrad: layer i reads the buffer chosen by the number of
  // dgrads above it, so a pass split into several calls finds its input where the last call left it.
  const bool odd = ((n_layers - 1 - first_layer) & 1) != 0;
  void* dy_cur = odd ? sc + dy_bytes : sc;
  void* dy_next = odd ? sc : sc + dy_bytes;
  float* partial = reinterpret_cast<float*>(sc + 2 * dy_bytes);

  // Bias gradients and split-K weight gradients are accumulated into zeroed memory.  Zero the whole buffer (padding included) so that
  // the all-reduce and the SGD update can treat it as one flat vector.
  if (from_top) {
    rc = zero_grads();
    if (rc != SB_OK) return rc;
  }

  const int n_out = sizes[n_layers];
  const int ld_out = padded_out(n_out);
  bool head_bias_done = false;
  if (from_top) {
    const int blocks = blocks_for(batch, 256);
    // The head layer's bias gradient is summed by this kernel when its padded width is 8 or 16.
    head_bias_done = with_bias && first_layer == n_layers - 1 && (ld_out == 8 || ld_out == 16);
    float* db_head = head_bias_done ? grads + off[2 * (n_layers - 1) + 1] : nullptr;
#define SB_CE_LAUNCH(T, R, L)                                                                                     \
  SB_CUDA(sb_launch(ce_grad_kernel<T, R, L>, dim3(blocks), dim3(256), 0, s, 1, probs, target, mask, (T*)dy_cur, \
                    batch, n_out, ld_out, inv_global_batch, loss, db_head))
#define SB_CE_BY_LD(T, R)                                     \
  do {                                                        \
    if (head_bias_done && ld_out == 8) SB_CE_LAUNCH(T, R, 8); \
    else if (head_bias_done) SB_CE_LAUNCH(T, R, 16);          \
    else SB_CE_LAUNCH(T, R, 0);                               \
  } while (0)
    if (in_dtype == SB_BF16) SB_CE_BY_LD(__nv_bfloat16, false);
    else if (in_dtype == SB_F16) SB_CE_BY_LD(__half, false);
    else SB_CE_BY_LD(float, true);
#undef SB_CE_BY_LD
#undef SB_CE_LAUNCH
    SB_COUNT_LAUNCH();
    SB_CUDA(cudaGetLastError());
  }

  // True when dY of the current layer came out of a dgrad whose epilogue already added its column
  // sums to the bias gradient, so that the stand-alone column-sum pass (a second read of dY) is skipped.
  // A pass split into several calls: the dgrad of the layer above ran in an earlier call.
  bool bias_done = from_top ? head_bias_done
                            : (with_bias && relu_bits && relu_bits[first_layer] && sizes[first_layer + 1] % 32 == 0);
  for (int i = first_layer; i >= last_layer; --i) {
    const int fan_out = padded_out(sizes[i + 1]), fan_in = sizes[i];
    const void* h_in = i == 0 ? x : activations[i - 1];
    if (with_bias && !bias_done) {
      // Enough blocks to fill the GPU a few times over, each with a long row slab.
      const int strip = 32 * (16 / es);
      const int strips = (fan_out + strip - 1) / strip;
      int slabs = (sb_sm_count() * 4 + strips - 1) / strips;
      int rows_per_block = (batch + slabs - 1) / slabs;
      if (rows_per_block < 64) rows_per_block = 64;
      dim3 grid(strips, (batch + rows_per_block - 1) / rows_per_block);
      float* db = grads + off[2 * i + 1];
      if (in_dtype == SB_BF16) SB_CUDA(sb_launch(colsum_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, s, 1, (const __nv_bfloat16*)dy_cur, db, batch, fan_out, rows_per_block));
      else if (in_dtype == SB_F16) SB_CUDA(sb_launch(colsum_kernel<__half>, dim3(grid), dim3(256), 0, s, 1, (const __half*)dy_cur, db, batch, fan_out, rows_per_block));
      else SB_CUDA(sb_launch(colsum_kernel<float>, dim3(grid), dim3(256), 0, s, 1, (const float*)dy_cur, db, batch, fan_out, rows_per_block));
      SB_COUNT_LAUNCH();
  SB_CUDA(cudaGetLastError());
    }
    // wgrad (TN): dW[out, in] = dY^T [out, B] * H_in [B, in]
    float* dw = grads + off[2 * i];
    const int want = wgrad_splits(fan_out, fan_in, batch, in_dtype);
    int used = 1;
    // The splits add their tiles straight into dW (zeroed above) through TMA reduce-add stores: no
    // partial matrices, no reduction kernel.  The order of those fp32 additions is not fixed, so the
    // last bits of dW can differ between runs; SB_WGRAD_PARTIALS=1 in the environment selects the
    // older form, partials reduced in a fixed order by a kernel of their own.
    const bool may_accumulate = want > 1 && !wgrad_partials_forced();
    if (grads_peers && layer_grads_go_to_peers(fan_out, fan_in, world)) {
      // Data-parallel pass: every tile is added to the copy of dW on the rank that owns its rows (the
      // reduce-scatter of the gradient all-reduce, done by the GEMM's own stores over peer memory).
      SbPeerOut po;
      po.n = world;
      for (int r = 0; r < world; ++r) po.c[r] = grads_peers[r] + off[2 * i];
      rc = sb_umma_gemm_launch(1, 0, 1.0f, dy_cur, h_in, 0.0f, nullptr, fan_out, fan_in, batch, in_dtype, SB_F32, 0, nullptr,
                               nullptr, nullptr, nullptr, s, want, &used, nullptr, nullptr, &po);
    } else {
      rc = sb_umma_gemm_launch(1, 0, 1.0f, dy_cur, h_in, 0.0f, (want > 1 && !may_accumulate) ? (void*)partial : (void*)dw,
                               fan_out, fan_in, batch, in_dtype, SB_F32, 0, nullptr, nullptr, nullptr, nullptr, s, want,
                               &used, nullptr, may_accumulate ? (void*)partial : nullptr);
    }
    if (rc != SB_OK) return rc;
    if (used > 1) {
      const long long n = (long long)fan_out * fan_in;
      SB_CUDA(sb_launch(splitk_reduce_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, s, 1, partial, dw, n, used));
      SB_COUNT_LAUNCH();
  SB_CUDA(cudaGetLastError());
    }
    // dgrad (NN): dH[B, in] = dY [B, out] * W [out, in], gated by ReLU'(H_in)
    if (i > 0) {
      const void* w = reinterpret_cast<const char*>(w_compute) + off[2 * i] * es;
      // The gate is ReLU'(H_in): read from the sign bits the forward pass recorded
      // when they exist (4 bytes per row and 32 columns), else from H_in itself.
      const bool bits = relu_bits && relu_bits[i - 1] && fan_in % 32 == 0;
      // The output is dY of layer i-1, whose column sums are that layer's bias gradient
      // (fan_in = sizes[i] is its unpadded width: hidden widths are multiples of 8 and, here, of 32).
      const bool sum_cols = bits && with_bias;
      float* db_below = grads + off[2 * (i - 1) + 1];
      if (bits && narrow_dgrad_ok(sizes[i + 1], fan_in, in_dtype) && st == in_dtype) {
        // A head layer: the inner dimension is at most 16, a single warp-level product.
        const uint32_t* gate = reinterpret_cast<const uint32_t*>(relu_bits[i - 1]);
        rc = in_dtype == SB_BF16
                 ? narrow_dgrad_launch<__nv_bfloat16>(dy_cur, fan_out, w, sizes[i + 1], fan_in, gate, dy_next, sum_cols ? db_below : nullptr, batch, s)
                 : narrow_dgrad_launch<__half>(dy_cur, fan_out, w, sizes[i + 1], fan_in, gate, dy_next, sum_cols ? db_below : nullptr, batch, s);
      } else
      rc = sb_umma_gemm_launch(0, 0, 1.0f, dy_cur, w, 0.0f, dy_next, batch, fan_in, fan_out, in_dtype, st,
                               bits ? (SB_EPI_RELU_GRAD_MASK | (sum_cols ? SB_EPI_COLSUM_OUT : 0)) : SB_EPI_RELU_GRAD,
                               nullptr, nullptr, bits ? (const void*)relu_bits[i - 1] : h_in,
                               sum_cols ? (void*)db_below : nullptr, s, 1, nullptr);
      if (rc != SB_OK) return rc;
      bias_done = sum_cols;
      void* t = dy_cur; dy_cur = dy_next; dy_next = t;
    }
  }
  return SB_OK;
}

int sb_mlp_backward(int n_layers, const int* sizes, int batch, float inv_global_batch, int in_dtype,
                    const void* x, const void* w_compute, void* const* activations,
                    void* const* relu_bits, const float* probs, const uint8_t* mask, const float* target,
                    float* grads, int with_bias, void* scratch, size_t scratch_bytes, float* loss,
                    void* stream) {
  return sb_mlp_backward_range(n_layers, sizes, batch, inv_global_batch, in_dtype, x, w_compute, activations,
                               relu_bits, probs, mask, target, grads, with_bias, scratch, scratch_bytes, loss,
                               n_layers - 1, 0, stream);
}

int sb_sgd_update(float* params, const float* grads, void* w_compute, long long n, float lr,
                  int compute_dtype, void* stream) {
  if (n < 0) return sb_fail(SB_ERR_BAD_ARG, "sb_sgd_update: negative length");
  if (n == 0) return SB_OK;
  if (!params || !grads) return sb_fail(SB_ERR_BAD_ARG, "sb_sgd_update: null pointer");
  SB_CUDA(sb_launch(sgd_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, (cudaStream_t)stream, 1, params, grads, w_compute, n, lr, compute_dtype));
  SB_COUNT_LAUNCH();
  SB_CUDA(cudaGetLastError());
  return SB_OK;
}

int sb_mlp_train_step(int n_layers, const int* sizes, int batch, int in_dtype, const void* x,
                      float* params, void* w_compute, void* const* activations, void* const* relu_bits,
                      const uint8_t* mask,
                      const float* target, float* probs, float* grads, int with_bias, float lr,
                      void* scratch, size_t scratch_bytes, float* loss, void* stream) {
  // Narrow nets run the whole forward pass as one fused launch that also writes what backward needs.
  int rc;
  if (sb_mlp_fused_supported(n_layers, sizes, in_dtype) && batch > 0)
    rc = sb_mlp_forward_fused_train(n_layers, sizes, batch, in_dtype, x, w_compute, with_bias ? params : nullptr,
                                    activations, relu_bits, SB_EPI_MASKED_SOFTMAX, mask, probs, nullptr, stream);
  else
    rc = sb_mlp_forward(n_layers, sizes, batch, in_dtype, x, w_compute, with_bias ? params : nullptr,
                        activations, relu_bits, SB_EPI_MASKED_SOFTMAX, mask, probs, nullptr, stream);
  if (rc != SB_OK) return rc;
  rc = sb_mlp_backward(n_layers, sizes, batch, batch > 0 ? 1.0f / (float)batch : 0.f, in_dtype, x, w_compute,
                       activations, relu_bits, probs, mask, target, grads, with_bias, scratch, scratch_bytes, loss,
                       stream);
  if (rc != SB_OK) return rc;
  long long off[2 * MLP_MAX_LAYERS + 1];
  param_offsets(n_layers, sizes, off);
  return sb_sgd_update(params, grads, w_compute, off[2 * n_layers], lr, storage_dtype(in_dtype), stream);
}

}  // extern "C"
