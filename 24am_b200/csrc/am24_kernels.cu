// Device kernels of one AM step and their launchers.
//
// One step for a batch of k starting points (reference:
// perform_one_iteration_for_{constrained,penalized}_pca,
// c++/src/gpower/gpower_commons.h:68-177):
//
//   1. gemm1     Z = B V            tcgen05 3xTF32, split-K partial tiles
//   2. z_reduce  sum the split partials; L1 variance: ||z||_1 and z <- sgn(z);
//                L2 variance: ||z||_2 (constrained) or z <- z/||z|| (penalized);
//                writes Z as TF32 hi/lo planes for gemm2
//   3. gemm2     V = B^T Z          tcgen05 3xTF32; penalized forms apply the
//                threshold, the per-start objective and non-zero count in the
//                epilogue; constrained forms store raw V
//   4. select    constrained only: per-start radix select of the s-th largest
//                |v| (L0) or the L1-ball level w (L1), normalisation
//   5. finalize  per-start objective, relative change, logs, batch maximum
//
// Every reduction has a fixed order, so a step is bitwise reproducible.
#include <cfloat>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <climits>
#include <cstdio>
#include <map>
#include <mutex>
#include <utility>

#include "am24_internal.h"
#include "gemm_tf32x3.cuh"
#include "gemm_pair.cuh"

namespace am24 {

namespace {

constexpr unsigned FULL = 0xffffffffu;
// K elements accumulated in TMEM before promotion to registers
constexpr int GEMM_PROMO_K = 128;

// x rounded to the nearest TF32 value (low 13 mantissa bits zero).  With
// lo = x - hi exact in FP32, x = hi + lo bit for bit, and lo takes either sign,
// so whatever the tensor core does with lo's low bits is unbiased.
__device__ __forceinline__ float tf32_hi(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
__device__ __forceinline__ void split_store(float x, float *hi, float *lo) {
  const float h = tf32_hi(x);
  *hi = h;
  *lo = x - h;
}
// sgn with sgn(0) = 0 (c++/src/utils/various.h:44-46)
__device__ __forceinline__ float sgnf(float v) { return (float)((v > 0.f) - (v < 0.f)); }
// x rounded to the nearest BF16, as bits.
__device__ __forceinline__ uint16_t bf16_bits(float x) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}
// sgn(v) as BF16 bits: +1 0x3F80, -1 0xBF80, 0 (and NaN) 0.
__device__ __forceinline__ uint16_t bf16_sign(float v) {
  return v > 0.f ? (uint16_t)0x3F80u : (v < 0.f ? (uint16_t)0xBF80u : (uint16_t)0u);
}
__device__ __forceinline__ uint32_t abs_key(float v) { return __float_as_uint(v) & 0x7FFFFFFFu; }
// sgn(v) as FP16 bits: +1 0x3C00, -1 0xBC00, 0 (and NaN) 0.
__device__ __forceinline__ uint16_t f16_sign(float v) {
  return v > 0.f ? (uint16_t)0x3C00u : (v < 0.f ? (uint16_t)0xBC00u : (uint16_t)0u);
}
// 2^e for e in [-126, 127], exactly.
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }
// The shift s in [-113, 126] that puts a positive bound on |x| into
// [2^14, 2^15) (bounds below 2^-112 stay below that range); 0 for zero, NaN or
// infinite bounds.  x * 2^s then splits into FP16 planes without overflow
// (FP16's largest finite value is 65504).
__device__ __forceinline__ int fp16_shift(float bound) {
  const uint32_t eb = (__float_as_uint(bound) >> 23) & 0xFFu;
  if (!(bound > 0.f) || eb == 0xFFu) return 0;
  const int e = max((int)eb, 1) - 127;  // floor(log2(bound)) for normal bounds
  return min(14 - e, 126);
}
// x = h0 + h1 + r: h0 = fp16_rn(x), h1 = fp16_rn(x - h0) (the difference is
// exact in FP32), |r| <= 2^-11 |x - h0| for FP16-normal x - h0, else <= 2^-25.
__device__ __forceinline__ void fp16_split(float x, uint16_t *h0, uint16_t *h1) {
  const __half a = __float2half_rn(x);
  *h0 = __half_as_ushort(a);
  *h1 = __half_as_ushort(__float2half_rn(x - __half2float(a)));
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// Block-wide sum, result valid in every thread.  `red` holds >= 32 T.
template <typename T>
__device__ T block_sum(T v, T *red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  T r = (lane < nw) ? red[lane] : T(0);
  if (w == 0) r = warp_sum(r);
  if (threadIdx.x == 0) red[0] = r;
  __syncthreads();
  r = red[0];
  __syncthreads();
  return r;
}

// Transposes the 32 x 32 bit matrix held by a warp: lane L passes bit j of
// x = A[L][j]; lane j gets the word whose bit L is A[L][j].  Five butterfly
// stages, each swapping the off-diagonal s x s blocks of every 2s x 2s block.
__device__ __forceinline__ uint32_t bit_transpose32(uint32_t x, int lane) {
  const uint32_t masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const int sft = 16 >> k;
    const uint32_t m = masks[k];
    const uint32_t y = __shfl_xor_sync(FULL, x, sft);
    x = (lane & sft) ? ((x & ~m) | ((y >> sft) & m)) : ((x & m) | ((y << sft) & ~m));
  }
  return x;
}

// 32 lanes each hold v[0..31] (one per column); afterwards lane L returns the
// sum over all lanes of v[L].  31 shuffles instead of 32 x 5.
__device__ __forceinline__ float transpose_reduce32(float (&v)[32], int lane) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < off; i++) {
      const float send = upper ? v[i] : v[i + off];
      const float keep = upper ? v[i + off] : v[i];
      v[i] = keep + __shfl_xor_sync(FULL, send, off);
    }
  }
  return v[0];
}

// fraction of the previous level used as the gather bound of the hinted searches
constexpr float HINT_FRACTION = 0.9f;
// The hinted bound on |v| keys of a column whose previous level was `hint` (> 0).
__device__ __forceinline__ uint32_t hinted_bound(float hint) {
  return max(1u, abs_key(HINT_FRACTION * hint));
}

// ------------------------------------------------------------ GEMM epilogues
// Z = B V split-K partial tile: ws[unit][col][row], whole 128 x bn tile.
struct EpiPartial {
  float *ws;
  int bn, m_tiles, n_tiles;  // m_tiles: 128-row blocks of C
  __device__ void setup() {}
  __device__ void unit_begin(const Unit &, int, int) {}
  __device__ void chunk(const Unit &t, int, int, int row, int col0, float (&r)[32]) {
    if (t.m0 >= m_tiles * BM) return;  // a 2-CTA tile's second half can lie past the last block
    const size_t slot = ((size_t)t.split * m_tiles + t.m0 / BM) * n_tiles + t.nt;
    float *base = ws + slot * ((size_t)bn * BM) + row;
#pragma unroll
    for (int j = 0; j < 32; j++) base[(size_t)(col0 + j) * BM] = r[j];
  }
};

// V = B^T Z raw output (constrained forms): out[col * ld + row].  With a
// candidate mask (cmask != null) it also does the selects' hinted gather: bit
// r of column col's mask (ld / 32 words per column, like vmask) is set when
// the column has a previous level hint[col] > 0 and |V[r, col]|'s key is at
// least hinted_bound(hint).  Every launch rewrites every word of rows < ld, so
// nothing needs clearing; the select kernels list the set bits instead of
// streaming the column.
struct EpiRaw {
  float *out;
  int ld, M, N, bn;
  const float *hint = nullptr;
  uint32_t *cmask = nullptr;
  // per unit: lane L holds the bound of column col_base + 32 c + L in bl[c]
  // (0xFFFFFFFF: the column has no level and lists nothing)
  int col_base = 0;
  uint32_t bl[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
  __device__ void setup() {}
  __device__ void unit_begin(const Unit &t, int lane, int cb) {
    if (!cmask) return;
    col_base = cb;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int col = t.nt * bn + cb + c * 32 + lane;
      const float h = col < N ? __ldg(hint + col) : 0.f;
      bl[c] = h > 0.f ? hinted_bound(h) : 0xFFFFFFFFu;
    }
  }
  __device__ void chunk(const Unit &t, int q, int lane, int row, int col0, float (&r)[32]) {
    if (t.m0 >= M) return;  // uniform: a 2-CTA tile's second half past the last row
    const int gi = t.m0 + row;
    const bool rv = gi < M;
    const int c0 = t.nt * bn + col0;
    if (rv) {
#pragma unroll
      for (int j = 0; j < 32; j++)
        if (c0 + j < N) out[(size_t)(c0 + j) * ld + gi] = r[j];
    }
    if (!cmask) return;
    // lane L: the rows of column c0 + L at or above its bound, as one mask word
    const int cl = c0 + lane;
    const int ci = ((col0 - col_base) >> 5) & 3;  // selects, not a local-memory index
    const uint32_t bound = ci == 0 ? bl[0] : ci == 1 ? bl[1] : ci == 2 ? bl[2] : bl[3];
    uint32_t mine = 0u;
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const uint32_t bj = __shfl_sync(FULL, bound, j);
      const uint32_t bal = __ballot_sync(FULL, rv && bj != 0xFFFFFFFFu && abs_key(r[j]) >= bj);
      if (lane == j) mine = bal;
    }
    const int w = (t.m0 >> 5) + q;
    if (cl < N && w < (ld >> 5)) cmask[(size_t)cl * (ld >> 5) + w] = mine;
  }
};

// *p = x where d > 0, as one predicated store.
__device__ __forceinline__ void store_if_positive(float *p, float x, float d) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.gt.f32 q, %2, 0f00000000;\n\t@q st.global.f32 [%0], %1;\n\t}"
      ::"l"(p), "f"(x), "f"(d)
      : "memory");
}

// V = B^T Z with the penalty threshold fused (penalized forms).
//   L1 (c++/src/gpower/sparse_PCA_thresholding.h:26-47): d = |v| - gamma,
//      x = sgn(v) d if d > 0, objective term d^2.
//   L0 (:68-87): d = v^2 - gamma, x = v if d > 0, objective term d.
// The reference subtracts a double gamma; here d is the FP32 difference with
// gamma rounded to FP32 (they differ only where |v| or v^2 is within an ulp
// of gamma, a decision that the FP32 products feeding it already leave open).
// Writes the non-zero x and the non-zero bitmask and, per start and per
// (128-row block, warp), the partial objective and non-zero count, summed in
// fixed order by the finalize kernel.  When the previous step was dense
// (*max_nnz > cap), the next step most likely is too, so the epilogue also
// writes x as the TF32 hi/lo planes the tensor-core Z = B V reads (zeros
// included), which spares that step the densify pass.
template <bool L1>
struct EpiPenalty {
  float *Vx;
  float *obj_part, *nnz_part;
  int ld, M, N, bn, parts;  // parts = m_tiles * 4
  float gamma;
  uint32_t *vmask;  // non-zero bitmask words, ld / 32 per column
  float *V_hi, *V_lo;
  const uint32_t *max_nnz;  // the previous step's largest non-zero count
  uint32_t cap;             // ... above which Z = B V runs dense
  bool planes = false;      // this launch writes V_hi / V_lo (set by setup)
  __device__ void setup() { planes = V_hi != nullptr && *max_nnz > cap; }
  __device__ void unit_begin(const Unit &, int, int) {}
  // r holds this thread's 32 values (row `row`, columns col0..col0+31) and is
  // overwritten with the objective terms.
  __device__ void chunk(const Unit &t, int q, int lane, int row, int col0, float (&r)[32]) {
    if (planes)
      body<true>(t, q, lane, row, col0, r);
    else
      body<false>(t, q, lane, row, col0, r);
  }
  template <bool PLANES>
  __device__ void body(const Unit &t, int q, int lane, int row, int col0, float (&r)[32]) {
    if (t.m0 >= M) return;  // a 2-CTA tile's second half can lie past the last row
    const int gi = t.m0 + row;
    const bool rv = gi < M;
    const int mb = t.m0 / BM;  // 128-row block
    const int c0 = t.nt * bn + col0;
    const int ncols = rv ? min(32, N - c0) : 0;  // valid columns of this row
    uint32_t bits = 0u;  // bit j: (row, column c0 + j) is a non-zero
    if (!PLANES && gamma >= 0.f && __all_sync(FULL, ncols == 32)) {
      // whole chunks of a tile's interior (d > 0 then means v != 0): no test per
      // entry but the threshold's, which predicates the store.  The epilogue is
      // bound by its instructions, and a short K leaves it nothing to hide
      // behind: 202 x 33654, 1005 starts 130 -> 122 us
      float *px = Vx + (size_t)c0 * ld + gi;
#pragma unroll
      for (int j = 0; j < 32; j++) {
        const float v = r[j];
        const float d = L1 ? __fsub_rn(fabsf(v), gamma) : __fsub_rn(__fmul_rn(v, v), gamma);
        store_if_positive(px, L1 ? copysignf(d, v) : v, d);
        px += ld;
        r[j] = d > 0.f ? (L1 ? __fmul_rn(d, d) : d) : 0.f;
        bits |= d > 0.f ? 1u << j : 0u;
      }
    } else
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const float v = r[j];
      const bool valid = j < ncols;
      float d, o, x;
      if (L1) {
        d = __fsub_rn(fabsf(v), gamma);
        o = __fmul_rn(d, d);
        x = v > 0.f ? d : -d;
      } else {
        d = __fsub_rn(__fmul_rn(v, v), gamma);
        o = d;
        x = v;
      }
      const bool keep = valid && d > 0.f;
      r[j] = keep ? o : 0.f;
      const bool nz = keep && v != 0.f;
      bits |= (uint32_t)nz << j;
      if (nz) Vx[(size_t)(c0 + j) * ld + gi] = x;  // zeros live in the mask
      if (PLANES && valid) {
        const size_t o = (size_t)(c0 + j) * ld + gi;
        split_store(nz ? x : 0.f, V_hi + o, V_lo + o);
      }
    }
    const uint32_t word = bit_transpose32(bits, lane);  // lane j: column c0 + j, bit = row
    const float so = transpose_reduce32(r, lane);
    const int col = c0 + lane;
    if (col < N) {
      obj_part[(size_t)col * parts + mb * 4 + q] = so;
      nnz_part[(size_t)col * parts + mb * 4 + q] = (float)__popc(word);
      if (mb * 4 + q < (ld >> 5)) vmask[(size_t)col * (ld >> 5) + mb * 4 + q] = word;
    }
  }
};

// ------------------------------------------------------------ operand prep
// Bc[c * ldm + r] = split(B[c * ldB + r]): one block per feature column.
__global__ void prep_copy_kernel(const float *__restrict__ B, int ldB, int m, float *__restrict__ hi,
                                 float *__restrict__ lo, float *__restrict__ full, int ldm) {
  const size_t c = blockIdx.x;
  for (int r = threadIdx.x; r < m; r += blockDim.x) {
    const float v = B[c * ldB + r];
    split_store(v, hi + c * ldm + r, lo + c * ldm + r);
    if (full) full[c * ldm + r] = v;
  }
}

// Three BF16 planes with x = b0 + b1 + b2 exactly: b0 = bf16_rn(x),
// b1 = bf16_rn(x - b0), b2 = x - b0 - b1.  Each difference is exact in FP32
// (its operands are within a factor of two), the first remainder has at most
// 16 significant bits and the second at most 8, so b2 is a BF16 value.  (FP32
// subnormals below 2^-126 aside, where a tensor core may flush b2.)
__global__ void prep_bf16x3_kernel(const float *__restrict__ Bc, int ldm, int m, size_t plane,
                                   int planes, uint16_t *__restrict__ out) {
  const size_t c = blockIdx.x;
  for (int r = threadIdx.x; r < m; r += blockDim.x) {
    const size_t o = c * ldm + r;
    const float x = Bc[o];
    const __nv_bfloat16 b0 = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(b0);
    const __nv_bfloat16 b1 = __float2bfloat16_rn(r1);
    const __nv_bfloat16 b2 = __float2bfloat16_rn(r1 - __bfloat162float(b1));
    out[o] = __bfloat16_as_ushort(b0);
    if (planes == 3) {
      out[plane + o] = __bfloat16_as_ushort(b1);
      out[2 * plane + o] = __bfloat16_as_ushort(b2);
    }
  }
}

// B (column-major, leading dimension ldB) into Bc's layout, pad rows zeroed;
// 16 bytes at a time where the source allows it (`vec`).
__global__ void __launch_bounds__(256) copy_matrix_kernel(const float *__restrict__ B, int ldB,
                                                          int m, bool vec, float *__restrict__ Bc,
                                                          int ldm) {
  const float *src = B + (size_t)blockIdx.x * ldB;
  float *dst = Bc + (size_t)blockIdx.x * ldm;
  for (int q = threadIdx.x; q < (ldm >> 2); q += blockDim.x) {
    const int r = 4 * q;
    float4 v;
    if (vec && r + 3 < m) {
      v = __ldg(reinterpret_cast<const float4 *>(src) + q);
    } else {
      v.x = r < m ? src[r] : 0.f;
      v.y = r + 1 < m ? src[r + 1] : 0.f;
      v.z = r + 2 < m ? src[r + 2] : 0.f;
      v.w = r + 3 < m ? src[r + 3] : 0.f;
    }
    reinterpret_cast<float4 *>(dst)[q] = v;
  }
}

// The largest |B[i, c]| as keys, per feature (row_key) and per sample (key),
// both zeroed before: blocks of 1024 samples x MAX_CHUNK features, four samples
// per thread.
constexpr int MAX_CHUNK = 64;
__global__ void __launch_bounds__(256) matrix_max_kernel(const float *__restrict__ Bc, int ldm,
                                                         int m, int n,
                                                         uint32_t *__restrict__ row_key,
                                                         uint32_t *__restrict__ key) {
  __shared__ uint32_t fmax[8][MAX_CHUNK];  // per warp
  const int warp = threadIdx.x >> 5;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = q < (ldm >> 2);
  const size_t ld4 = (size_t)ldm >> 2;
  const int c0 = blockIdx.y * MAX_CHUNK, cn = min(n - c0, MAX_CHUNK);
  const float4 *B4 = reinterpret_cast<const float4 *>(Bc) + (size_t)c0 * ld4 + (on ? q : 0);
  uint32_t mx[4] = {0u, 0u, 0u, 0u};
#pragma unroll 8
  for (int c = 0; c < cn; c++) {
    const float4 v = __ldg(B4 + c * ld4);  // off threads repeat the first quad
    const uint32_t k[4] = {abs_key(v.x), abs_key(v.y), abs_key(v.z), abs_key(v.w)};
#pragma unroll
    for (int e = 0; e < 4; e++) mx[e] = max(mx[e], k[e]);
    const uint32_t f = __reduce_max_sync(FULL, max(max(k[0], k[1]), max(k[2], k[3])));
    if ((threadIdx.x & 31) == 0) fmax[warp][c] = f;
  }
  if (on)
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (4 * q + e < m) atomicMax(key + 4 * q + e, mx[e]);
  __syncthreads();
  if (threadIdx.x < cn) {
    uint32_t f = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) f = max(f, fmax[w][threadIdx.x]);
    atomicMax(row_key + c0 + threadIdx.x, f);
  }
}

// The FP16 operand planes of B (rows = features) and of B^T (rows = samples),
// each row with its power-of-two scale from its largest |x|:
// x * 2^s = h0 + h1 (fp16_split), second plane at + plane; scale[row] = 2^-s
// undoes it in the GEMM epilogue.  64 x 64 tiles through shared memory, B read
// once for both, 8-byte stores.  HBM bound: 1000 x 20000 in 40 us (240 MB), with
// matrix_max_kernel 66; a pass per orientation and one for the samples' maxima
// took 180.
__global__ void __launch_bounds__(256) split_matrix_kernel(
    const float *__restrict__ Bc, int ldm, int m, int n, int ldn,
    const uint32_t *__restrict__ row_key, const uint32_t *__restrict__ key,
    uint16_t *__restrict__ Ch, size_t cplane, float *__restrict__ row_scale,
    uint16_t *__restrict__ Th, size_t tplane, float *__restrict__ bt_row_scale) {
  __shared__ float tile[64][65];
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;  // features, samples
  const int q = threadIdx.x & 15, row = threadIdx.x >> 4;
  auto put = [](const float (&v)[4], float sc, uint16_t *out, size_t plane) {
    uint16_t a[4], b[4];
#pragma unroll
    for (int e = 0; e < 4; e++) fp16_split(v[e] * sc, &a[e], &b[e]);
    *reinterpret_cast<uint2 *>(out) =
        make_uint2(a[0] | ((uint32_t)a[1] << 16), a[2] | ((uint32_t)a[3] << 16));
    *reinterpret_cast<uint2 *>(out + plane) =
        make_uint2(b[0] | ((uint32_t)b[1] << 16), b[2] | ((uint32_t)b[3] << 16));
  };
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int f = row + 16 * i, c = c0 + f, r = r0 + 4 * q;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (c < n && r < ldm) {  // rows in [m, ldm) are zeros
      const float4 x = __ldg(reinterpret_cast<const float4 *>(Bc + (size_t)c * ldm + r));
      v[0] = x.x;
      v[1] = x.y;
      v[2] = x.z;
      v[3] = x.w;
      const int s = fp16_shift(__uint_as_float(row_key[c]));
      put(v, pow2f(s), Ch + (size_t)c * ldm + r, cplane);
      if (r == 0) row_scale[c] = pow2f(-s);
    }
#pragma unroll
    for (int e = 0; e < 4; e++) tile[f][4 * q + e] = v[e];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int t = row + 16 * i, r = r0 + t, c = c0 + 4 * q;
    if (r >= m || c >= ldn) continue;  // columns in [n, ldn) take zeros
    const float v[4] = {tile[4 * q][t], tile[4 * q + 1][t], tile[4 * q + 2][t], tile[4 * q + 3][t]};
    const int s = fp16_shift(__uint_as_float(key[r]));
    put(v, pow2f(s), Th + (size_t)r * ldn + c, tplane);
    if (c == 0) bt_row_scale[r] = pow2f(-s);
  }
}

// Bt[r * ldn + c] = split(B[c * ldB + r]): 32 x 32 tiles through shared memory.
__global__ void prep_transpose_kernel(const float *__restrict__ B, int ldB, int m, int n,
                                      float *__restrict__ hi, float *__restrict__ lo, int ldn) {
  __shared__ float tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    const int c = c0 + y, r = r0 + threadIdx.x;
    tile[y][threadIdx.x] = (c < n && r < m) ? B[(size_t)c * ldB + r] : 0.f;
  }
  __syncthreads();
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    const int r = r0 + y, c = c0 + threadIdx.x;
    if (r < m && c < n) {
      const size_t off = (size_t)r * ldn + c;
      split_store(tile[threadIdx.x][y], hi + off, lo + off);
    }
  }
}

// dst = src (rows entries, zero up to ld_dst) and the column's non-zero bitmask
// (ld_dst / 32 words); whole warps.
__device__ __forceinline__ void load_column(const float *__restrict__ src, int rows,
                                            float *__restrict__ dst, int ld_dst,
                                            uint32_t *__restrict__ mask) {
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int base = threadIdx.x & ~31; base < ld_dst; base += blockDim.x) {
    const int r = base + lane;
    const float v = (r < rows) ? src[r] : 0.f;
    dst[r] = v;
    const unsigned nz = __ballot_sync(FULL, v != 0.f);
    if (lane == 0) mask[base >> 5] = nz;
  }
}
// One block per column.
__global__ void load_columns_kernel(const float *__restrict__ src, int ld_src, int rows,
                                    float *__restrict__ dst, int ld_dst,
                                    uint32_t *__restrict__ mask) {
  const size_t c = blockIdx.x;
  load_column(src + c * ld_src, rows, dst + c * ld_dst, ld_dst, mask + c * (ld_dst >> 5));
}
// Column c into column slots[c], a start that begins anew (launch_load_slots).
__global__ void load_slots_kernel(const float *__restrict__ src, int ld_src, int rows,
                                  const int *__restrict__ slots, float *__restrict__ dst,
                                  int ld_dst, uint32_t *__restrict__ mask, float *sel_hint,
                                  float *val, uint32_t *max_nnz, uint32_t *planes_nnz) {
  const size_t c = blockIdx.x, to = slots[c];
  load_column(src + c * ld_src, rows, dst + to * ld_dst, ld_dst, mask + to * (ld_dst >> 5));
  if (threadIdx.x == 0) {
    sel_hint[to] = 0.f;
    val[to] = 0.f;
    if (c == 0) {
      *max_nnz = 0xFFFFFFFFu;
      *planes_nnz = 0u;
    }
  }
}

// dst = the column's values where its mask is set, zero elsewhere; blockIdx.y
// walks pieces of COPY_ROWS rows (a single column is most calls' whole work: one
// block for it took 45 us at 50000 rows).
constexpr int COPY_ROWS = 2048;
__global__ void masked_copy_kernel(const float *__restrict__ Vx, const uint32_t *__restrict__ mask,
                                   int ld, int rows, float *__restrict__ dst, int ld_dst) {
  const size_t c = blockIdx.x;
  for (int r0 = blockIdx.y * COPY_ROWS; r0 < rows; r0 += gridDim.y * COPY_ROWS) {
    const int r1 = min(rows, r0 + COPY_ROWS);
#pragma unroll 8
    for (int r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
      const bool on = (mask[c * (ld >> 5) + (r >> 5)] >> (r & 31)) & 1u;
      dst[c * ld_dst + r] = on ? Vx[c * ld + r] : 0.f;
    }
  }
}

// Dense TF32 hi/lo planes of V for the tensor-core Z = B V; does nothing on
// steps where the gather kernel takes Z = B V (*gate <= gate_max), and on
// dense steps whose planes the previous step's penalty epilogue already wrote
// (*planes > gate_max: the count that epilogue saw).
__global__ void densify_kernel(const float *__restrict__ Vx, const uint32_t *__restrict__ mask,
                               int ld, int rows, float *__restrict__ V_hi,
                               float *__restrict__ V_lo, const uint32_t *gate,
                               const uint32_t *planes, uint32_t gate_max,
                               const uint32_t *stop) {
  pdl_enter();
  if (*stop || *gate <= gate_max || *planes > gate_max) return;
  const size_t c = blockIdx.x;
  for (int r = threadIdx.x; r < ld; r += blockDim.x) {
    const bool on = r < rows && ((mask[c * (ld >> 5) + (r >> 5)] >> (r & 31)) & 1u);
    split_store(on ? Vx[c * ld + r] : 0.f, V_hi + c * ld + r, V_lo + c * ld + r);
  }
}

// Dense FP16 planes of V for the CTA-pair Z = B V (split FP16 operands): on
// dense steps only (*gate > gate_max), one block per start, v * 2^s = h0 + h1
// with s from the column's largest |v|, v_scale[c] = 2^-s.
// The body for start c (one 256-thread block); densify_fp16_kernel runs it for
// blockIdx.x, the grouped steps for every start of their dense problems.
__device__ __forceinline__ void densify_fp16_body(const float *__restrict__ Vx,
                                                  const uint32_t *__restrict__ mask, int ld,
                                                  int rows, uint16_t *__restrict__ Vh,
                                                  size_t plane, float *__restrict__ v_scale,
                                                  const uint32_t *gate, uint32_t gate_max,
                                                  const uint32_t *stop, size_t c) {
  __shared__ uint32_t red[32];
  if (*stop || *gate <= gate_max) return;
  const uint32_t *mk = mask + c * (ld >> 5);
  const float4 *vx4 = reinterpret_cast<const float4 *>(Vx + c * ld);
  // four consecutive rows per thread and pass (ld is a multiple of 32)
  auto quad = [&](int q, float (&v)[4]) {
    const float4 x = vx4[q];
    const uint32_t bits = mk[q >> 3] >> ((4 * q) & 31);
    v[0] = ((bits & 1u) && 4 * q < rows) ? x.x : 0.f;
    v[1] = ((bits & 2u) && 4 * q + 1 < rows) ? x.y : 0.f;
    v[2] = ((bits & 4u) && 4 * q + 2 < rows) ? x.z : 0.f;
    v[3] = ((bits & 8u) && 4 * q + 3 < rows) ? x.w : 0.f;
  };
  const int quads = ld >> 2;
  uint32_t mx = 0;
#pragma unroll 8
  for (int q = threadIdx.x; q < quads; q += blockDim.x) {
    float v[4];
    quad(q, v);
    mx = max(mx, max(max(abs_key(v[0]), abs_key(v[1])), max(abs_key(v[2]), abs_key(v[3]))));
  }
  mx = __reduce_max_sync(FULL, mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); w++) mx = max(mx, red[w]);
  const int s = fp16_shift(__uint_as_float(mx));
  const float sc = pow2f(s);
  if (threadIdx.x == 0) v_scale[c] = pow2f(-s);
  uint2 *h0 = reinterpret_cast<uint2 *>(Vh + c * ld);
  uint2 *h1 = reinterpret_cast<uint2 *>(Vh + plane + c * ld);
#pragma unroll 4
  for (int q = threadIdx.x; q < quads; q += blockDim.x) {
    float v[4];
    quad(q, v);
    uint16_t a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) fp16_split(v[i] * sc, &a[i], &b[i]);
    h0[q] = make_uint2(a[0] | ((uint32_t)a[1] << 16), a[2] | ((uint32_t)a[3] << 16));
    h1[q] = make_uint2(b[0] | ((uint32_t)b[1] << 16), b[2] | ((uint32_t)b[3] << 16));
  }
}
// Persistent over the k columns with DENSIFY_BLOCKS_PER_SM blocks of 512
// threads per SM: a column's first pass (its largest |v|) streams it from HBM,
// and with this few columns in flight (2 x 148 x 4 B x p, 59 MB at p = 50000)
// the second pass finds it in L2, so V crosses HBM once.
constexpr int DENSIFY_THREADS = 512, DENSIFY_BLOCKS_PER_SM = 2;
__global__ void __launch_bounds__(DENSIFY_THREADS, DENSIFY_BLOCKS_PER_SM) densify_fp16_kernel(
    const float *__restrict__ Vx, const uint32_t *__restrict__ mask, int ld, int rows,
    uint16_t *__restrict__ Vh, size_t plane, float *__restrict__ v_scale, const uint32_t *gate,
    uint32_t gate_max, const uint32_t *stop, int k) {
  pdl_enter();
  for (int c = blockIdx.x; c < k; c += gridDim.x) {
    densify_fp16_body(Vx, mask, ld, rows, Vh, plane, v_scale, gate, gate_max, stop, c);
    __syncthreads();  // red[] is reused by the next column
  }
}

// ------------------------------------------------------------ Z reduction
// What becomes of y = B v, by mode:
// 0: L2 variance, constrained  -> z = y, fz = ||y||_2  (gpower_commons.h:100)
// 1: L1 variance               -> z = sgn(y), fz = ||y||_1 (:85-86, :156)
// 2: L2 variance, penalized    -> z = y * (1/||y||_2)     (:163-164)
struct ZOut {
  float *hi, *lo;     // one start's FP32 planes, ldm each: hi + lo = z when lo is
                      // wanted (the TF32 operands); else hi holds y between passes
  uint16_t *b;        // its BF16 z (null: not wanted)
  uint16_t *h;        // its FP16 z (null: not wanted); second plane at h + plane
  size_t plane;
  float *scale, *fz;  // the start's words
};
__device__ __forceinline__ ZOut z_out(int j, int ldm, float *Z_hi, float *Z_lo, uint16_t *Zb,
                                      uint16_t *Zh, size_t zplane, float *zscale, float *fz) {
  const size_t o = (size_t)j * ldm;
  return ZOut{Z_hi + o, Z_lo ? Z_lo + o : nullptr, Zb ? Zb + o : nullptr, Zh ? Zh + o : nullptr,
              zplane, zscale ? zscale + j : nullptr, fz + j};
}
// C consecutive values of T at p (aligned to them) in one store.
template <int C, class T>
__device__ __forceinline__ void store_run(T *p, const T (&v)[C]) {
  if (C == 1) {
    *p = v[0];
  } else if (sizeof(T) == 4) {
    *reinterpret_cast<uint4 *>(p) = *reinterpret_cast<const uint4 *>(v);
  } else {
    *reinterpret_cast<uint2 *>(p) = *reinterpret_cast<const uint2 *>(v);
  }
}
template <int C>
__device__ __forceinline__ void z_store_split(const ZOut &z, int i, const float (&y)[C]) {
  alignas(16) float hi[C], lo[C];
#pragma unroll
  for (int c = 0; c < C; c++) split_store(y[c], hi + c, lo + c);
  store_run(z.hi + i, hi);
  store_run(z.lo + i, lo);
}
__device__ __forceinline__ bool z_second_pass(const ZOut &z, int mode) {
  return mode == 2 || (mode == 0 && z.h);
}
// Samples i .. i + C - 1 (C = 1 or 4) before the norm is known: their share of it
// into acc, and what can be stored already.  Those beyond m are padding: stored,
// but not of the norm (zero only while the loadings are finite: 0 x inf is NaN).
// KEEP: y is stored for a second pass, which reads it back.
template <int C, bool KEEP>
__device__ __forceinline__ void z_emit(const ZOut &z, int mode, int m, int i, const float (&y)[C],
                                       double &acc) {
  if (mode == 1) {
    alignas(16) uint16_t b[C], h[C];
    alignas(16) float sg[C], zero[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      if (C == 1 || i + c < m) acc += (double)fabsf(y[c]);
      sg[c] = sgnf(y[c]);
      zero[c] = 0.f;
      b[c] = bf16_sign(y[c]);
      h[c] = f16_sign(y[c]);
    }
    if (z.lo) {
      store_run(z.hi + i, sg);
      store_run(z.lo + i, zero);
    }
    if (z.b) store_run(z.b + i, b);
    if (z.h) store_run(z.h + i, h);
  } else {
    alignas(16) uint16_t b[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      if (C == 1 || i + c < m) acc += (double)y[c] * (double)y[c];
      b[c] = bf16_bits(y[c]);
    }
    if (z.lo) {
      if (mode == 0 || KEEP) z_store_split(z, i, y);
    } else if (KEEP && C == 1 && z_second_pass(z, mode)) {
      z.hi[i] = y[0];
    }
    if (mode == 0 && z.b) store_run(z.b + i, b);
  }
}
// Second pass over them: mode 2 normalises; both write the FP16 planes of
// z * 2^s, s from a bound on |z| (||y||_2, or 1 for the normalised z).
struct ZScale {
  float inv, sc;
  int s;
};
__device__ __forceinline__ ZScale z_scales(int mode, double tot) {
  ZScale r;
  r.inv = mode == 2 ? 1.0f / (float)sqrt(tot) : 1.0f;
  r.s = fp16_shift(mode == 2 ? 1.0f : (float)sqrt(tot));
  r.sc = pow2f(r.s);
  return r;
}
template <int C>
__device__ __forceinline__ void z_emit2(const ZOut &z, int mode, const ZScale &c, int i,
                                        const float (&y)[C]) {
  float v[C];
  alignas(16) uint16_t b[C], h0[C], h1[C];
#pragma unroll
  for (int q = 0; q < C; q++) {
    v[q] = mode == 2 ? y[q] * c.inv : y[q];
    b[q] = bf16_bits(v[q]);
    fp16_split(v[q] * c.sc, h0 + q, h1 + q);
  }
  if (mode == 2) {
    if (z.lo) z_store_split(z, i, v);
    if (z.b) store_run(z.b + i, b);
  }
  if (z.h) {
    store_run(z.h + i, h0);
    store_run(z.h + z.plane + i, h1);
  }
}
__device__ __forceinline__ void z_close(const ZOut &z, int mode, double tot) {  // one thread
  if (z_second_pass(z, mode) && z.h) *z.scale = pow2f(-z_scales(mode, tot).s);
  if (mode != 2) *z.fz = (mode == 1) ? (float)tot : (float)sqrt(tot);
}

// Dense steps: y from the split-K partial tiles of Z = B V.
__device__ __forceinline__ void z_reduce_body(int mode, const float *__restrict__ ws, int splits,
                                              int m_tiles, int n_tiles, int bn, int m,
                                              const ZOut &z, int j) {
  __shared__ double red[32];
  const int nt = j / bn, c = j - nt * bn;
  const size_t unit_stride = (size_t)bn * BM;
  double acc = 0.0;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const int mt = i >> 7, r = i & 127;
    float y = 0.f;
    for (int s = 0; s < splits; s++) {
      const size_t u = ((size_t)s * m_tiles + mt) * n_tiles + nt;
      y += ws[u * unit_stride + (size_t)c * BM + r];
    }
    z_emit<1, true>(z, mode, m, i, {y}, acc);
  }
  const double tot = block_sum(acc, red);
  if (z_second_pass(z, mode)) {
    const ZScale sc = z_scales(mode, tot);
    for (int i = threadIdx.x; i < m; i += blockDim.x)  // exact: this thread wrote the planes
      z_emit2<1>(z, mode, sc, i, {z.lo ? z.hi[i] + z.lo[i] : z.hi[i]});
  }
  if (threadIdx.x == 0) z_close(z, mode, tot);
}

// Sparse steps of matrices with more than GATHER_NARROW samples: y from the
// plane gather_tile_body left it in (z.hi, zeros in its padding).  256 threads,
// 4 consecutive samples each (16- and 8-byte stores: 1024 starts of 2000 samples
// in 7 us, 19 with a store per sample).
__device__ __forceinline__ void z_finish_body(int mode, int m, const ZOut &z) {
  __shared__ double red[32];
  double acc = 0.0;
  for (int i = 4 * threadIdx.x; i < m; i += 4 * blockDim.x) {
    const float4 y = *reinterpret_cast<const float4 *>(z.hi + i);
    z_emit<4, true>(z, mode, m, i, {y.x, y.y, y.z, y.w}, acc);
  }
  const double tot = block_sum(acc, red);
  if (z_second_pass(z, mode)) {
    const ZScale sc = z_scales(mode, tot);
    for (int i = 4 * threadIdx.x; i < m; i += 4 * blockDim.x) {
      float4 y = *reinterpret_cast<const float4 *>(z.hi + i);
      if (z.lo) {
        const float4 l = *reinterpret_cast<const float4 *>(z.lo + i);
        y = make_float4(y.x + l.x, y.y + l.y, y.z + l.z, y.w + l.w);
      }
      z_emit2<4>(z, mode, sc, i, {y.x, y.y, y.z, y.w});
    }
  }
  if (threadIdx.x == 0) z_close(z, mode, tot);
}

// One block per start: the dense step's reduction, or the end of a sparse
// step's tiled gather (`wide`).
__global__ void __launch_bounds__(256) z_reduce_kernel(int mode, const float *__restrict__ ws,
                                                       int splits, int m_tiles, int n_tiles,
                                                       int bn, int m, float *__restrict__ Z_hi,
                                                       float *__restrict__ Z_lo, int ldm,
                                                       float *__restrict__ fz,
                                                       const uint32_t *gate, uint32_t gate_max,
                                                       uint16_t *__restrict__ Zb,
                                                       uint16_t *__restrict__ Zh, size_t zplane,
                                                       float *__restrict__ zscale, bool wide,
                                                       const uint32_t *stop) {
  pdl_enter();
  if (*stop) return;
  const bool dense = *gate > gate_max;
  if (!dense && !wide) return;  // gather_narrow_kernel produced Z this step
  const ZOut z = z_out(blockIdx.x, ldm, Z_hi, Z_lo, Zb, Zh, zplane, zscale, fz);
  if (dense)
    z_reduce_body(mode, ws, splits, m_tiles, n_tiles, bn, m, z, blockIdx.x);
  else
    z_finish_body(mode, m, z);
}

// ------------------------------------------------------------ sparse Z = B V
constexpr int GATHER_THREADS = 256;

// MIXED phase word after a step: the lead-in counts down to the single-pass
// phase 0, which switches to refinement (1, sticky) once enough starts are stable.
__device__ __forceinline__ uint32_t mixed_next_phase(uint32_t ph, bool stable_enough) {
  if (ph >= 2u) return ph == 2u ? 0u : ph - 1u;
  return (ph == 0u && stable_enough) ? 1u : ph;
}
constexpr int GATHER_CAP = 4096;

// MIXED precision bookkeeping, after the step's non-zero masks are written:
// per start, the number of consecutive steps whose support (non-zero mask)
// equals the previous step's.  When at least `need` starts of the batch have
// kept their support for k_stable steps, phase[0] switches to refinement for
// good; the last block to finish decides, keeps the phase the step ran in as
// phase[3] and resets the step's scratch words.  phase[0] >= 2 is the FP32
// lead-in (phase[0] - 1 accurate steps left, no start counted stable); its
// last step hands over to the single-pass phase 0.
__global__ void __launch_bounds__(256) support_kernel(const uint32_t *__restrict__ vmask,
                                                      const uint32_t *__restrict__ prev, int words,
                                                      uint32_t *stable, uint32_t *phase,
                                                      uint32_t k_stable, uint32_t need,
                                                      const uint32_t *stop) {
  pdl_enter();
  if (*stop) return;
  const int j = blockIdx.x;
  const uint32_t *a = vmask + (size_t)j * words, *b = prev + (size_t)j * words;
  int diff = 0;
  for (int w = threadIdx.x; w < words; w += blockDim.x) diff |= (a[w] != b[w]);
  diff = __syncthreads_or(diff);
  if (threadIdx.x == 0) {
    // read before this block's arrival: the last block rewrites phase[0] only
    // after every block has arrived
    const bool lead = *reinterpret_cast<volatile uint32_t *>(phase) >= 2u;
    const uint32_t st = (diff || lead) ? 0u : min(stable[j] + 1u, 0x7FFFFFFFu);
    stable[j] = st;
    if (st >= k_stable) atomicAdd(&phase[1], 1u);
    __threadfence();
    if (atomicAdd(&phase[2], 1u) == gridDim.x - 1) {
      __threadfence();
      const uint32_t count = atomicExch(&phase[1], 0u);
      const uint32_t ph = phase[0];
      phase[3] = ph;
      phase[0] = mixed_next_phase(ph, count >= need);
      phase[2] = 0u;
    }
  }
}

// The sparse Z = B V: z = sum_q v_q B[:, q] over the column's non-zeros, in index
// order with FP32 FMAs (deterministic), on steps whose previous step left at
// most gate_max non-zeros in every column (*gate); the FP32 rows of Bc are read.
// Two forms, by the matrix's number of samples:
//   up to GATHER_NARROW   one block per start and one launch: the list of
//       non-zeros in shared memory, four samples per thread, the norm and the
//       output planes from registers.  A chain of loads bounds it.
//   above                 gather_list_kernel writes every start's list to
//       memory once; gather_tile_kernel gives each (start, 128 samples) a warp
//       that reads one 512-byte row segment per non-zero, the tiles of 128
//       samples one after another over all starts, so that the segments in use
//       (512 bytes per feature) stay in L2; z_finish_body closes the columns.
//       L2 reads bound it (12.5 TB/s at 8192 samples, 4096 starts).
// Measured against one kernel of four starts per block walking whole rows:
// 8192 x 65536, 4096 starts of 128 non-zeros 2.47 -> 1.38 ms; 2000 x 50000, 1024
// starts of 240 to 400: 204..302 -> 155..243 us (beyond 1024 non-zeros, 638 ->
// 360); 400 samples, 64 starts of 16: 14 -> 5.4 us; 1000 samples, 256 starts of
// 40 to 100: 54..100 -> 14..23 us, where the listed form takes 6 + 20..36.
// The list of start j: a header {count, 0}, then (row, value bits) pairs.

// The non-zeros of a column (its mask words) in index order through
// put(position, row); returns their number.  Each thread of the block
// owns a contiguous run of words, so an exclusive scan of their counts places
// the entries.  wsum: a word per warp.
template <class Put>
__device__ __forceinline__ uint32_t list_column(const uint32_t *__restrict__ mk, int words,
                                                uint32_t *wsum, Put put) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per = (words + GATHER_THREADS - 1) / GATHER_THREADS;
  const int w0 = min(words, (int)threadIdx.x * per), w1 = min(words, w0 + per);
  uint32_t cnt = 0;
  for (int q = w0; q < w1; q++) cnt += __popc(mk[q]);
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  uint32_t off = incl - cnt, total = 0;
#pragma unroll
  for (int i = 0; i < GATHER_THREADS / 32; i++) {
    if (i < w) off += wsum[i];
    total += wsum[i];
  }
  for (int q = w0; q < w1; q++)
    for (uint32_t bits = mk[q]; bits; bits &= bits - 1) put(off++, q * 32 + __ffs(bits) - 1);
  __syncthreads();
  return total;
}

__device__ __forceinline__ void fma4(float v, const float4 &b, float4 &acc) {
  acc.x = fmaf(v, b.x, acc.x);
  acc.y = fmaf(v, b.y, acc.y);
  acc.z = fmaf(v, b.z, acc.z);
  acc.w = fmaf(v, b.w, acc.w);
}

constexpr int GATHER_NARROW = 4 * GATHER_THREADS;  // samples one block holds in registers
__device__ __forceinline__ void gather_narrow_body(int mode, const float *__restrict__ Bc, int ldm,
                                                   int m, int ldn, const float *__restrict__ Vx,
                                                   const uint32_t *__restrict__ vmask,
                                                   const ZOut &z, int j) {
  __shared__ int list[GATHER_CAP];
  __shared__ float val[GATHER_CAP];
  __shared__ uint32_t wsum[GATHER_THREADS / 32];
  __shared__ double red[32];
  const int words = ldn >> 5;
  const float *vx = Vx + (size_t)j * ldn;
  uint32_t total = list_column(vmask + (size_t)j * words, words, wsum, [&](uint32_t at, int r) {
    if (at < (uint32_t)GATHER_CAP) list[at] = r;
  });
  total = min(total, (uint32_t)GATHER_CAP);  // more cannot happen below the gate
  // a batch of rows is loaded before its FMAs (a short list's values with them);
  // samples in [m, ldm) read B's zeros
  constexpr uint32_t SHORT = 16, U = 8;
  const int i4 = threadIdx.x;
  const bool on = i4 < (ldm >> 2);
  const float4 *B4 = reinterpret_cast<const float4 *>(Bc) + (on ? i4 : 0);
  const size_t ld4 = (size_t)ldm >> 2;
  float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
  if (total <= SHORT) {
    float4 b[SHORT];
    float v[SHORT];
#pragma unroll
    for (uint32_t u = 0; u < SHORT; u++)
      if (on && u < total) {
        b[u] = __ldg(B4 + list[u] * ld4);
        v[u] = vx[list[u]];
      }
#pragma unroll
    for (uint32_t u = 0; u < SHORT; u++)
      if (on && u < total) fma4(v[u], b[u], y);
  } else {
    for (uint32_t q = threadIdx.x; q < total; q += GATHER_THREADS) val[q] = vx[list[q]];
    __syncthreads();
    uint32_t q = 0;
    for (; on && q + U <= total; q += U) {
      float4 b[U];
#pragma unroll
      for (uint32_t u = 0; u < U; u++) b[u] = __ldg(B4 + list[q + u] * ld4);
#pragma unroll
      for (uint32_t u = 0; u < U; u++) fma4(val[q + u], b[u], y);
    }
    float4 b[U];
#pragma unroll
    for (uint32_t u = 0; u < U; u++)
      if (on && q + u < total) b[u] = __ldg(B4 + list[q + u] * ld4);
#pragma unroll
    for (uint32_t u = 0; u < U; u++)
      if (on && q + u < total) fma4(val[q + u], b[u], y);
  }
  const float e[4] = {y.x, y.y, y.z, y.w};
  double acc = 0.0;
  if (on) z_emit<4, false>(z, mode, m, 4 * i4, e, acc);
  const double tot = block_sum(acc, red);
  if (on && z_second_pass(z, mode)) z_emit2<4>(z, mode, z_scales(mode, tot), 4 * i4, e);
  if (threadIdx.x == 0) z_close(z, mode, tot);
}
__global__ void __launch_bounds__(GATHER_THREADS) gather_narrow_kernel(
    int mode, const float *__restrict__ Bc, int ldm, int m, int ldn, const float *__restrict__ Vx,
    const uint32_t *__restrict__ vmask, float *__restrict__ Z_hi, float *__restrict__ Z_lo,
    float *__restrict__ fz, const uint32_t *gate, uint32_t gate_max, uint16_t *__restrict__ Zb,
    uint16_t *__restrict__ Zh, size_t zplane, float *__restrict__ zscale, float *max_err,
    const uint32_t *stop) {
  pdl_enter();
  if (*stop) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) *max_err = 0.f;  // the step begins here
  if (*gate > gate_max) return;  // dense V: gemm1 + z_reduce
  gather_narrow_body(mode, Bc, ldm, m, ldn, Vx, vmask,
                     z_out(blockIdx.x, ldm, Z_hi, Z_lo, Zb, Zh, zplane, zscale, fz), blockIdx.x);
}

// int2 entries between the lists of consecutive starts: the plane they live in
// holds ldn floats per start, and a list at most n / 32 + 1 pairs.
__device__ __forceinline__ size_t list_stride(int ldn) { return (size_t)ldn / 2; }
__device__ __forceinline__ void gather_list_body(int ldn, const float *__restrict__ Vx,
                                                 const uint32_t *__restrict__ vmask, uint32_t cap,
                                                 int2 *__restrict__ lists, int j) {
  __shared__ uint32_t wsum[GATHER_THREADS / 32];
  const int words = ldn >> 5;
  int2 *list = lists + (size_t)j * list_stride(ldn);
  const float *vx = Vx + (size_t)j * ldn;
  const uint32_t total =
      list_column(vmask + (size_t)j * words, words, wsum, [&](uint32_t at, int r) {
        if (at < cap) list[1 + at] = make_int2(r, __float_as_int(vx[r]));
      });
  if (threadIdx.x == 0) list[0] = make_int2((int)min(total, cap), 0);
}
__global__ void __launch_bounds__(GATHER_THREADS) gather_list_kernel(
    int ldn, const float *__restrict__ Vx, const uint32_t *__restrict__ vmask, const uint32_t *gate,
    uint32_t gate_max, int2 *__restrict__ lists, float *max_err, const uint32_t *stop) {
  pdl_enter();
  if (*stop) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) *max_err = 0.f;  // the step begins here
  if (*gate > gate_max) return;
  gather_list_body(ldn, Vx, vmask, gate_max, lists, blockIdx.x);
}

constexpr int GATHER_STARTS = GATHER_THREADS / 32;  // starts per block, a warp each
__host__ __device__ __forceinline__ int gather_groups(int k) {
  return (k + GATHER_STARTS - 1) / GATHER_STARTS;
}
__host__ __device__ __forceinline__ int gather_tiles(int ldm) { return (ldm + 127) / 128; }
// Item: tile * gather_groups(k) + group of starts.  No block barrier: warps of
// starts past k return.
__device__ __forceinline__ void gather_tile_body(const float *__restrict__ Bc, int ldm, int ldn,
                                                 int k, const int2 *__restrict__ lists,
                                                 float *__restrict__ Z_hi, int item) {
  const int groups = gather_groups(k);
  const int tile = item / groups;
  const int j = (item - tile * groups) * GATHER_STARTS + ((int)threadIdx.x >> 5);
  if (j >= k) return;
  const int lane = threadIdx.x & 31;
  const int i4 = tile * 32 + lane;
  const bool on = i4 < (ldm >> 2);
  const float4 *B4 = reinterpret_cast<const float4 *>(Bc) + (on ? i4 : tile * 32);
  const size_t ld4 = (size_t)ldm >> 2;
  const int2 *list = lists + (size_t)j * list_stride(ldn);
  const int total = list[0].x;
  float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
  auto pair = [&](int e) { return e < total ? list[1 + e] : make_int2(0, 0); };
  int2 next = pair(lane);
  for (int base = 0; base < total; base += 32) {
    const int2 mine = next;
    next = pair(base + 32 + lane);  // in flight while this chunk's rows are read
    const int cnt = min(32, total - base);
#pragma unroll 16
    for (int t = 0; t < cnt; t++) {
      const int q = __shfl_sync(FULL, mine.x, t);
      const float v = __int_as_float(__shfl_sync(FULL, mine.y, t));
      fma4(v, __ldg(B4 + q * ld4), y);
    }
  }
  if (on) reinterpret_cast<float4 *>(Z_hi + (size_t)j * ldm)[i4] = y;
}
__global__ void __launch_bounds__(GATHER_THREADS) gather_tile_kernel(
    const float *__restrict__ Bc, int ldm, int ldn, int k, const int2 *__restrict__ lists,
    float *__restrict__ Z_hi, const uint32_t *gate, uint32_t gate_max, const uint32_t *stop) {
  pdl_enter();
  if (*stop || *gate > gate_max) return;
  gather_tile_body(Bc, ldm, ldn, k, lists, Z_hi, blockIdx.x);
}

// ------------------------------------------------------------ radix select
struct SelResult {
  uint32_t key;  // bit pattern of |v| at the requested descending rank
  uint32_t gt;   // number of keys strictly greater
  uint32_t eq;   // number of keys equal
};


// Key of descending rank `rank` (1 = largest) among |col[0..n)|, by three
// histogram passes over 11, 11 and 9 key bits.  All threads of the block
// call it; hist has 2048 entries, res 4.
// Readers of the values a selection walks: a column of V (read-only in the
// kernel) or a list of keys the kernel wrote itself (read through L2, never the
// non-coherent path).
struct ColumnSrc {
  const float *__restrict__ p;
  __device__ __forceinline__ float operator()(int i) const { return p[i]; }
};
struct ListSrc {
  const float *p;
  __device__ __forceinline__ float operator()(int i) const { return __ldcg(p + i); }
};

template <class Src>
__device__ SelResult block_select_src(Src colg, int n, uint32_t rank, uint32_t *hist,
                                      uint32_t *res);
__device__ __forceinline__ SelResult block_select(const float *__restrict__ colg, int n,
                                                  uint32_t rank, uint32_t *hist, uint32_t *res) {
  return block_select_src(ColumnSrc{colg}, n, rank, hist, res);
}
template <class Src>
__device__ SelResult block_select_src(Src colg, int n, uint32_t rank, uint32_t *hist,
                                      uint32_t *res) {
  uint32_t prefix = 0, pmask = 0, gt = 0, need = rank, eq = 0;
#pragma unroll 1
  for (int lvl = 0; lvl < 3; lvl++) {
    const int sh = (lvl == 0) ? 20 : (lvl == 1) ? 9 : 0;
    const uint32_t nb = (lvl == 2) ? 512u : 2048u;
    const uint32_t bmask = nb - 1;
    for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) hist[b] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const uint32_t key = abs_key(colg(i));
      if ((key & pmask) == prefix) {
        const uint32_t bin = (key >> sh) & bmask;
        const unsigned peers = __match_any_sync(__activemask(), bin);
        if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[bin], __popc(peers));
      }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      uint32_t running = 0, fbin = 0, fcum = 0, feq = 0;
      bool found = false;
      for (int base = (int)nb - 32; base >= 0 && !found; base -= 32) {
        const uint32_t b = base + 31 - lane;
        const uint32_t c = hist[b];
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(FULL, incl, o);
          if (lane >= o) incl += t;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        if (running + total >= need) {
          const unsigned ballot = __ballot_sync(FULL, running + incl >= need);
          const int f = __ffs(ballot) - 1;
          const uint32_t inc_f = __shfl_sync(FULL, incl, f);
          const uint32_t c_f = __shfl_sync(FULL, c, f);
          fbin = base + 31 - f;
          fcum = running + inc_f - c_f;
          feq = c_f;
          found = true;
        } else {
          running += total;
        }
      }
      if (lane == 0) {
        res[0] = fbin;
        res[1] = fcum;
        res[2] = feq;
      }
    }
    __syncthreads();
    const uint32_t bin = res[0];
    gt += res[1];
    need -= res[1];
    eq = res[2];
    prefix |= bin << sh;
    pmask |= bmask << sh;
    __syncthreads();
  }
  return SelResult{prefix, gt, eq};
}

// x_i = f(v_i) for a column in global memory: the non-zero x_i are stored
// (only they are defined; the bitmask says which) and the column's non-zero
// bitmask is written.
template <class Fn>
__device__ __forceinline__ void write_column_global(const float *__restrict__ colg, int n,
                                                    float *vx, uint32_t *mask, Fn fn) {
  const int lane = threadIdx.x & 31;
  const int n32 = (n + 31) & ~31;
  for (int base = threadIdx.x & ~31; base < n32; base += blockDim.x) {
    const int i = base + lane;
    const float y = fn(colg[i]);  // every column has room for the last whole warp
    const float x = i < n ? y : 0.f;
    if (x != 0.f) vx[i] = x;
    const unsigned nz = __ballot_sync(FULL, x != 0.f);
    if (lane == 0) mask[base >> 5] = nz;
  }
}

// Warp 0 walks the histogram from the top bin down and finds the bin holding
// descending rank `need` (1-based): res[0] = bin, res[1] = count of keys in
// higher bins, res[2] = count in the bin.  All threads call; result after the
// trailing barrier.
__device__ void find_rank_bin(const uint32_t *hist, int nb, uint32_t need, uint32_t *res) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    uint32_t running = 0, fbin = 0, fcum = running, feq = 0;
    bool found = false;
    for (int base = nb - 32; base >= 0 && !found; base -= 32) {
      const uint32_t c = hist[base + 31 - lane];
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
      }
      const uint32_t total = __shfl_sync(FULL, incl, 31);
      if (running + total >= need) {
        const unsigned ballot = __ballot_sync(FULL, running + incl >= need);
        const int f = __ffs(ballot) - 1;
        const uint32_t inc_f = __shfl_sync(FULL, incl, f);
        const uint32_t c_f = __shfl_sync(FULL, c, f);
        fbin = base + 31 - f;
        fcum = running + inc_f - c_f;
        feq = c_f;
        found = true;
      } else {
        running += total;
      }
    }
    if (!found) {  // fewer than `need` keys: every bin lies above
      fbin = 0;
      fcum = running;
      feq = 0;
    }
    if (lane == 0) {
      res[0] = fbin;
      res[1] = fcum;
      res[2] = feq;
    }
  }
  __syncthreads();
}

// Top-11-bit histogram of |col| keys into hist[2048] (warp-aggregated adds).
__device__ void key_histogram(const float *__restrict__ colg, int n, uint32_t *hist) {
  for (int b = threadIdx.x; b < 2048; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const uint32_t bin = abs_key(colg[i]) >> 20;
    const unsigned peers = __match_any_sync(__activemask(), bin);
    if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[bin], __popc(peers));
  }
  __syncthreads();
}

// Descending bitonic sort of a[0..len), len a power of two.
template <typename T>
__device__ void bitonic_desc(T *a, int len) {
  for (int k = 2; k <= len; k <<= 1) {
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int i = threadIdx.x; i < len; i += blockDim.x) {
        const int ixj = i ^ jj;
        if (ixj > i) {
          const T x = a[i], y = a[ixj];
          const bool first_block = (i & k) == 0;
          if (first_block ? (x < y) : (x > y)) {
            a[i] = y;
            a[ixj] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

constexpr int SELECT_THREADS = 256;  // block size of both selects

// Descending sort of a[0..c) (zeros taken beyond, up to the next power of two),
// E = 1, 2, 4, 8 or 16 elements per thread of a SELECT_THREADS block in
// registers: a bitonic network whose exchanges run inside a thread (distances
// below E), by shuffles (below 32 E) and only beyond that through shared memory.
// Bound by instruction issue: the same network on shared memory pays a block
// barrier and two round trips for every one of its stages.
template <int E>
__device__ __noinline__ void sort_desc_regs(uint64_t *a, int c, int len) {
  const int t = threadIdx.x;
  uint64_t v[E];
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int i = e * SELECT_THREADS + t;
    v[e] = i < c ? a[i] : 0ull;
  }
  auto pick = [](uint64_t x, uint64_t y, bool larger) { return (x > y) == larger ? x : y; };
  // element t * E + e; the one at distance j is in this thread, lane or warp
  for (int k = 2; k <= len; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32 * E) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) a[e * SELECT_THREADS + t] = v[e];
        __syncthreads();
        const int o = t ^ (j / E);
        const bool larger = ((t * E & k) == 0) == ((t * E & j) == 0);
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = pick(v[e], a[e * SELECT_THREADS + o], larger);
      } else if (j >= E) {
        const bool larger = (((t * E) & k) == 0) == (((t * E) & j) == 0);
#pragma unroll
        for (int e = 0; e < E; e++)
          v[e] = pick(v[e], __shfl_xor_sync(FULL, v[e], j / E), larger);
      } else {
#pragma unroll
        for (int q = 1; q < E; q <<= 1) {
          if (j != q) continue;
#pragma unroll
          for (int e = 0; e < E; e++) {
            if (e & q) continue;
            const bool desc = ((t * E + e) & k) == 0;
            const uint64_t x = v[e], y = v[e | q];
            v[e] = pick(x, y, desc);
            v[e | q] = pick(x, y, !desc);
          }
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < E; e++) a[t * E + e] = v[e];
  __syncthreads();
}
// a[0..c) descending, c <= cap (a power of two, at most 16 * SELECT_THREADS; a
// has room for max(cap, SELECT_THREADS)).
__device__ __forceinline__ void sort_pairs_desc(uint64_t *a, int c, int cap) {
  int len = 1;
  while (len < c) len <<= 1;
  if (len <= SELECT_THREADS) sort_desc_regs<1>(a, c, len);
  else if (len == 2 * SELECT_THREADS) sort_desc_regs<2>(a, c, len);
  else if (len == 4 * SELECT_THREADS) sort_desc_regs<4>(a, c, len);
  else if (len == 8 * SELECT_THREADS || cap <= 8 * SELECT_THREADS) sort_desc_regs<8>(a, c, len);
  else sort_desc_regs<16>(a, c, len);
}

// The (|v| key << 32 | ~index) pairs of the entries whose bit is set in a
// column's mask (words 32-bit words) in index order into out, when there are at
// most `cap`; returns how many bits are set.  Each thread owns a contiguous run
// of words, so an exclusive scan of their counts places the entries in order.
// scratch: one word of shared memory per warp of the block.
__device__ uint32_t pairs_from_mask(const uint32_t *__restrict__ mk, int words,
                                    const float *__restrict__ colg, uint64_t *out, uint32_t cap,
                                    uint32_t *scratch) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int per = (words + blockDim.x - 1) / blockDim.x;
  const int w0 = min(words, (int)threadIdx.x * per), w1 = min(words, w0 + per);
  uint32_t cnt = 0;
  for (int q = w0; q < w1; q++) cnt += __popc(mk[q]);
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();  // scratch may still be read by the caller's previous use
  if (lane == 31) scratch[w] = incl;
  __syncthreads();
  uint32_t off = incl - cnt, total = 0;
  for (int i = 0; i < nw; i++) {
    if (i < w) off += scratch[i];
    total += scratch[i];
  }
  if (total > cap) return total;  // not listed: nobody reads a part of the set
  for (int q = w0; q < w1; q++) {
    uint32_t bits = mk[q];
    while (bits) {
      const int b = __ffs(bits) - 1;
      bits &= bits - 1;
      const uint32_t i = (uint32_t)(q * 32 + b);
      if (off < cap) out[off] = ((uint64_t)abs_key(__ldg(colg + i)) << 32) | (uint32_t)~i;
      off++;
    }
  }
  __syncthreads();
  return total;
}

// ------------------------------------------------------------ end of a step
// Per start: objective f, relative change |f - f0| / f0
// (c++/src/utils/termination_criteria.h:30-36), the storeIterationsForAllPoints
// logs (c++/src/gpower/gpower_commons.h:120-130), and the batch maximum that
// ignores NaN changes (:132-133).  Runs at the end of the select kernels, or as
// finalize_kernel where a step has no select (the penalties) or another pass
// after it (MIXED).
struct FinalizeArgs {
  int k, formulation, parts, it, store_all, log_shift, log_capacity;
  double tolerance;
  const float *fz;
  const float *obj_part, *nnz_part;
  const uint32_t *nnz_sel;
  float *val, *err, *max_err;
  uint32_t *next_nnz;    // the step's largest non-zero count is formed here ...
  uint32_t *max_nnz;     // ... and becomes the next step's gate as the step closes
  uint32_t *planes_nnz;  // takes the closing step's own gate (null: not wanted)
  int *iters, *cards;
  // run-ahead control (StepCtl words); stop_check: this step may stop the batch
  uint32_t *ctl;
  uint32_t *host_stop;    // pinned host word that takes the stop word (or null)
  const uint32_t *phase;  // MIXED: phase[3] is the phase the step ran in; else null
  const int *status;
  int stop_check;
};

// Whether the batch had stopped before this step (tells the host so).
__device__ __forceinline__ bool step_stopped(const FinalizeArgs &a) {
  if (!a.ctl[CTL_STOP]) return false;
  if (a.host_stop && blockIdx.x == 0 && threadIdx.x == 0)
    *reinterpret_cast<volatile uint32_t *>(a.host_stop) = 1u;
  return true;
}

// One start's objective f and non-zero count (one thread).  The batch maximum
// is an atomicMax on the bit pattern of the (non-negative, non-NaN) changes,
// zeroed as the step begins -- max is order-independent, so the result is
// deterministic.
__device__ void finalize_value(const FinalizeArgs &a, int j, float f, uint32_t nz) {
  atomicMax(a.next_nnz, nz);
  const float f0 = a.val[j];
  const float e = fabsf(f - f0) / f0;
  a.err[j] = e;
  a.val[j] = f;
  // the reference's `if (max < e) max = e`: NaN never wins
  if (e > 0.f) atomicMax(reinterpret_cast<unsigned int *>(a.max_err), __float_as_uint(e));
  if (a.store_all) {
    // the penalized thresholding calls log into slot j of every batch
    // (gpower_commons.h:170,173 leave the batch shift at 0)
    const int slot = a.formulation <= 3 ? a.log_shift + j : j;
    if (slot < a.log_capacity) {
      const bool done = a.it > 0 && (double)e < a.tolerance;
      if (done && a.iters[slot] == -1) {
        a.iters[slot] = a.it;
        a.cards[slot] = (int)nz;
      } else if (!done && a.iters[slot] != -1) {
        a.iters[slot] = -1;
      }
    }
  }
}

// One start, by a warp (lane 0 writes): the constraints' values as they stand,
// the penalties' from the epilogue's partials.
__device__ void finalize_start(const FinalizeArgs &a, int j, int lane) {
  float f;
  uint32_t nz;
  if (a.formulation <= 3) {
    f = a.fz[j];
    nz = a.nnz_sel[j];
  } else {
    // fixed order: lane-strided partial sums, then a butterfly
    double acc = 0.0, c = 0.0;
    for (int q = lane; q < a.parts; q += 32) {
      acc += (double)a.obj_part[(size_t)j * a.parts + q];
      c += (double)a.nnz_part[(size_t)j * a.parts + q];
    }
    acc = warp_sum(acc);
    c = warp_sum(c);
    f = a.formulation >= 6 ? (float)sqrt(acc) : (float)acc;
    nz = (uint32_t)c;
  }
  if (lane == 0) finalize_value(a, j, f, nz);
}

// Called by one thread of every block once its starts are done.  The last block
// closes the step for the run-ahead driver: it counts the step (and, MIXED,
// whether it ran in the BF16 phase), keeps the batch's largest change, hands the
// non-zero count to the next step, and sets the stop word when the reference's
// batch loop would end here (it > 0, a refinement step, max change < tolerance)
// or a device-side wait gave up.
__device__ void close_step(const FinalizeArgs &a) {
  __threadfence();
  if (atomicAdd(&a.ctl[CTL_BLOCKS], 1u) != gridDim.x - 1) return;
  __threadfence();
  const float me = *reinterpret_cast<volatile float *>(a.max_err);
  const bool refined = a.phase == nullptr || a.phase[3] != 0u;
  a.ctl[CTL_STEPS] += 1u;
  if (!refined) a.ctl[CTL_LOW_STEPS] += 1u;
  a.ctl[CTL_MAX_ERR] = __float_as_uint(me);
  if (a.planes_nnz) *a.planes_nnz = *a.max_nnz;
  *a.max_nnz = atomicExch(a.next_nnz, 0u);
  const bool stop =
      (a.stop_check && a.it > 0 && refined && (double)me < a.tolerance) ||
      *reinterpret_cast<const volatile int *>(a.status) != 0;
  if (stop) a.ctl[CTL_STOP] = 1u;
  if (a.host_stop) *reinterpret_cast<volatile uint32_t *>(a.host_stop) = stop ? 1u : 0u;
  a.ctl[CTL_BLOCKS] = 0u;
}

// ------------------------------------------------------------ L0 constraint
constexpr int HARD_THREADS = 256;
constexpr int HARD_CAND = 2048;  // hinted (key, index) candidates resolved in shared memory

// One streaming pass over a column in global memory (16-byte loads, four in
// flight per thread): the entries with |v| key >= bound (>= 1) go to cand as
// (key << 32 | ~index), the first `cap` of them in any order; returns how many
// there are (it may exceed cap) and, BELOW, leaves in counter[1] the largest
// key below the bound (0 if none).  Entries past n (the padding read with the
// last 16 bytes) are not taken.  The bound leaves a few hundred entries
// of a column, so a quad of them is tested by its largest key and the taken
// ones placed by single shared-memory atomics.
template <bool BELOW>
__device__ uint32_t gather_pairs_above(const float *__restrict__ colg, int n, uint32_t bound,
                                       uint64_t *cand, uint32_t cap, uint32_t *counter) {
  if (threadIdx.x == 0) {
    counter[0] = 0;
    counter[1] = 0;
  }
  __syncthreads();
  uint32_t below = 0;
  const int n4 = (n + 3) >> 2;
  const float4 *c4 = reinterpret_cast<const float4 *>(colg);
  constexpr int U = 4;
  for (int base = threadIdx.x; base < n4; base += U * blockDim.x) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = base + u * blockDim.x;
      v[u] = (i < n4) ? __ldg(c4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t k[4] = {abs_key(v[u].x), abs_key(v[u].y), abs_key(v[u].z), abs_key(v[u].w)};
      const int e0 = 4 * (base + u * (int)blockDim.x);
      if (BELOW) {
#pragma unroll
        for (int q = 0; q < 4; q++) below = max(below, k[q] < bound && e0 + q < n ? k[q] : 0u);
      }
      if (max(max(k[0], k[1]), max(k[2], k[3])) < bound) continue;
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (k[q] >= bound && e0 + q < n) {
          const uint32_t pos = atomicAdd(&counter[0], 1u);
          if (pos < cap) cand[pos] = ((uint64_t)k[q] << 32) | (uint32_t)~(uint32_t)(e0 + q);
        }
    }
  }
  if (BELOW) {
    below = __reduce_max_sync(FULL, below);
    if ((threadIdx.x & 31) == 0) atomicMax(&counter[1], below);
  }
  __syncthreads();
  return counter[0];
}

// A bound on |v| keys that about `target` to a few times as many of a column's
// entries reach, from a sample of SAMPLE_KEYS evenly spaced ones (twice as
// many from long columns; every entry of a short one): the sample's r-th
// largest key to 8 significant bits, r the sample's share of `target` plus
// 2.5 standard deviations of that count and 3, and at most 0.85 of its share of
// `most` (0 when that is none).  For columns whose level has no usable
// hint; reading 8 KB of a column in place of a histogram pass over all of it.
// smp: room for 2 * SAMPLE_KEYS keys; cnt: 16 words.  The bound only decides how many
// candidates are looked at, not the result.
constexpr int SAMPLE_KEYS = 2048, SAMPLE_LONG = 65536;
__device__ uint32_t sampled_bound(const float *__restrict__ colg, int n, uint32_t target,
                                  uint32_t most, uint32_t *smp, uint32_t *cnt) {
  const int n4 = n >> 2;  // whole quads
  const int s4 = min(n4, (n > SAMPLE_LONG ? 2 : 1) * SAMPLE_KEYS / 4);
  if (s4 == 0) return 1u;
  const float f = (float)(4 * s4) / (float)n;
  const float x = (float)target * f;
  const float rf = fminf(s4 == n4 ? (float)target : x + 2.5f * sqrtf(x) + 3.f,
                         fminf(0.85f * f * (float)most, (float)(4 * s4)));
  const uint32_t r = (uint32_t)rf;
  if (r == 0u) return 0u;
  __syncthreads();  // smp and cnt may still be read by their previous users
  if (threadIdx.x < 16) cnt[threadIdx.x] = 0u;
  const float4 *c4 = reinterpret_cast<const float4 *>(colg);
  for (int i = threadIdx.x; i < s4; i += blockDim.x) {
    const float4 v = __ldg(c4 + (s4 == n4 ? i : (int)(((int64_t)i * n4) / s4)));
    reinterpret_cast<uint4 *>(smp)[i] =
        make_uint4(abs_key(v.x), abs_key(v.y), abs_key(v.z), abs_key(v.w));
  }
  __syncthreads();
  uint32_t bound = 0u;
  for (int bit = 30; bit >= 15; bit--) {
    const uint32_t t = bound | (1u << bit);
    uint32_t c = 0;
    for (int i = threadIdx.x; i < s4; i += blockDim.x) {
      const uint4 k = reinterpret_cast<const uint4 *>(smp)[i];
      c += (k.x >= t) + (k.y >= t) + (k.z >= t) + (k.w >= t);
    }
    c = __reduce_add_sync(FULL, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&cnt[30 - bit], c);
    __syncthreads();
    if (cnt[30 - bit] >= r) bound = t;
  }
  __syncthreads();
  return max(bound, 1u);
}

// The hint for the next step's candidate bound from this step's c sorted candidates,
// `need` of which the level keeps: at most HINT_FRACTION of the level, and the key
// of rank `want` (a little below the last candidate when there are fewer), so that
// columns which change fast do not outrun it.  A set beyond `cap` is worth nothing,
// though, so where `want` is a large share of it the bound goes below the level's
// only as far as this step's candidates show that there is room (half of what is left).
// 128 columns of 200000, top 1700: 61 us a select, 755 when the bound went 15 %
// below the last candidate whatever the capacity; exact L1 ball, s = 2048: 110, 1150.
__device__ __forceinline__ float next_hint(const uint64_t *sorted, uint32_t c, uint32_t need,
                                           uint32_t want, uint32_t cap, float level) {
  auto key = [&](uint32_t rank) {
    return __uint_as_float((uint32_t)(sorted[min(c - 1, rank)] >> 32));
  };
  const float by_level = HINT_FRACTION * level;
  float b = key(want);
  if (want <= cap / 4u)
    b = c <= want ? 0.85f * b : b;
  else if (c > want)
    b = fminf(b, fmaxf(by_level, key((need + cap) / 2u)));
  return fminf(level, b / HINT_FRACTION);
}

// One streaming pass over a column: every |v| with key >= bound goes to
// list[] (global memory, room for n) as a float, in any order; returns how
// many, and leaves in counter[1] the largest key below the bound (0 if none).
__device__ uint32_t gather_keys_above(const float *__restrict__ colg, int n, uint32_t bound,
                                      float *list, uint32_t *counter) {
  if (threadIdx.x == 0) {
    counter[0] = 0;
    counter[1] = 0;
  }
  __syncthreads();
  uint32_t below = 0;
  const int lane = threadIdx.x & 31;
  for (int base = (threadIdx.x & ~31); base < n; base += blockDim.x) {
    const int i = base + lane;
    const uint32_t key = i < n ? abs_key(colg[i]) : 0u;
    const bool take = i < n && key >= bound;
    if (i < n && !take) below = max(below, key);
    const unsigned bal = __ballot_sync(FULL, take);
    if (!bal) continue;
    uint32_t wbase = 0;
    if (lane == 0) wbase = atomicAdd(&counter[0], (uint32_t)__popc(bal));
    wbase = __shfl_sync(FULL, wbase, 0);
    if (take) list[wbase + __popc(bal & ((1u << lane) - 1u))] = __uint_as_float(key);
  }
  below = __reduce_max_sync(FULL, below);
  if (lane == 0) atomicMax(&counter[1], below);
  __syncthreads();
  return counter[0];
}

// k_hard_thresholding (c++/src/utils/thresh_functions.h:121-145): level = the
// s-th largest |v| (with multiplicity, as the sorting variant :92-98 defines
// it), keep |v| >= level, then x <- x / ||x|| (c++/src/gpower/gpower_commons.h:111).
//
// One block per column, reading it from global memory.  (a) The entries with
// |v| at or above a bound, with their indices: the previous step's hint, whose
// entries V = B^T Z's epilogue marked (or a streaming pass gathers), or, when
// the hinted set is short of s or too large, or there is no hint, a bound from
// a sample of the column.  When that gives s to HARD_CAND entries, sorting them
// gives the exact level, the norm and the kept entries, and the column is
// written sparsely (its mask words cleared, then the kept entries' bits and
// values set).  Otherwise (b) a histogram of the top 11 bits of |v| finds the
// bin holding rank s, keys above it are kept for sure, keys in it are gathered
// and sorted; a bin too full for shared memory falls back to (c) the exact
// three-level radix select; the column is then written by a full pass.
// What bounds it: with a hint, the latency of the candidates' loads and sort;
// without, one read of V (205 MB at 1024 columns of 50000, 31 us at the copy
// rate).  Measured there: 84 us unhinted (704 with the histogram of every
// column), 31 us hinted with a few columns falling back (265 when a hint that
// came up short streamed the column twice).
__device__ __forceinline__ void hard_select_body(
    const float *__restrict__ Vraw, int ldv, int n, unsigned s, float *__restrict__ Vx,
    uint32_t *__restrict__ nnz_out, uint32_t *__restrict__ vmask, float *__restrict__ hints,
    const uint32_t *__restrict__ cmask, int j) {
  // also 2 * HARD_CAND keys for (b), and the sample, read 16 bytes at a time
  __shared__ __align__(16) uint64_t cand[HARD_CAND];
  __shared__ uint32_t hist[2048];
  __shared__ uint32_t res[8];
  __shared__ double red[32];
  uint32_t *cand32 = reinterpret_cast<uint32_t *>(cand);
  const float *colg = Vraw + (size_t)j * ldv;
  float *vx = Vx + (size_t)j * ldv;
  uint32_t *mk = vmask + (size_t)j * (ldv >> 5);
  uint32_t thr = 0;
  double ss = 0.0, cnt = 0.0;
  bool done = false;
  const float hint = hints[j];
  float new_hint = 0.f;
  // the bound that is wanted next time: about twice s entries reach it (many more
  // cost every step more in listing and sorting than the columns that outrun their
  // hint: 64 starts of 96 x 640, s = 8, 835 us a solve, 918 with 176 beyond s)
  const uint32_t want = s + min(s + 32u, 192u);
  uint32_t c = 0;
  if (hint > 0.f)
    c = cmask ? pairs_from_mask(cmask + (size_t)j * (ldv >> 5), ldv >> 5, colg, cand, HARD_CAND,
                                &res[0])
              : gather_pairs_above<false>(colg, n, hinted_bound(hint), cand, HARD_CAND, &res[0]);
  // (a sampled bound aims at 0.85 of the capacity, so a set between s and the whole of
  // it is luck for the largest s: 128 columns of 200000, a select at s = 1900 takes
  // 1.10 to 1.28 ms with the attempt and 1.28 without, at 2048 1.35 and 1.30)
  if ((c < s || c > (uint32_t)HARD_CAND) && s <= (uint32_t)HARD_CAND * 15u / 16u) {
    const uint32_t bound = sampled_bound(colg, n, want, HARD_CAND, cand32, hist);
    c = bound ? gather_pairs_above<false>(colg, n, bound, cand, HARD_CAND, &res[0]) : 0u;
  }
  if (c >= s && c <= (uint32_t)HARD_CAND) {
    __syncthreads();
    sort_pairs_desc(cand, (int)c, HARD_CAND);
    thr = (uint32_t)(cand[s - 1] >> 32);
    // kept: the sorted prefix with key >= thr (ties with the s-th included)
    for (int q = threadIdx.x; q < (int)c; q += blockDim.x) {
      const uint32_t key = (uint32_t)(cand[q] >> 32);
      if (key >= thr && (q + 1 == (int)c || (uint32_t)(cand[q + 1] >> 32) < thr))
        res[1] = q + 1;
      if (key >= thr) {
        const double v = (double)__uint_as_float(key);
        ss += v * v;
      }
    }
    new_hint = next_hint(cand, c, s, want, HARD_CAND, __uint_as_float(thr));
    done = true;
    __syncthreads();
  }
  if (done) {
    const uint32_t kept = res[1];
    ss = block_sum(ss, red);
    const float inv = 1.0f / (float)sqrt(ss);
    for (int w = threadIdx.x; w < (ldv >> 5); w += blockDim.x) mk[w] = 0u;
    __syncthreads();
    for (int q = threadIdx.x; q < (int)kept; q += blockDim.x) {
      const uint32_t i = ~(uint32_t)cand[q];
      const float x = __ldg(colg + i) * inv;
      if (x != 0.f) {
        vx[i] = x;
        atomicOr(&mk[i >> 5], 1u << (i & 31));
      }
    }
    cnt = (double)kept;
  } else {
    // (b) histogram of the top 11 key bits, then the bin holding rank s
    key_histogram(colg, n, hist);
    find_rank_bin(hist, 2048, s, res);
    const uint32_t b1 = res[0], above = res[1], in_bin = res[2];
    __syncthreads();
    if (in_bin <= (uint32_t)(2 * HARD_CAND)) {
      if (threadIdx.x == 0) res[3] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t key = abs_key(colg[i]);
        const uint32_t bin = key >> 20;
        if (bin > b1) {
          const double v = (double)__uint_as_float(key);
          ss += v * v;
          cnt += 1.0;
        } else if (bin == b1) {
          cand32[atomicAdd(&res[3], 1u)] = key;
        }
      }
      __syncthreads();
      const int nc = (int)res[3];
      int len = 1;
      while (len < nc) len <<= 1;
      for (int q = nc + threadIdx.x; q < len; q += blockDim.x) cand32[q] = 0u;
      __syncthreads();
      bitonic_desc(cand32, len);
      thr = cand32[s - above - 1];
      for (int q = threadIdx.x; q < nc; q += blockDim.x)
        if (cand32[q] >= thr) {
          const double v = (double)__uint_as_float(cand32[q]);
          ss += v * v;
          cnt += 1.0;
        }
    } else {
      // (c) exact radix select
      thr = block_select(colg, n, s, hist, res).key;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float v = colg[i];
        if (abs_key(v) >= thr) {
          ss += (double)v * (double)v;
          cnt += 1.0;
        }
      }
    }
    ss = block_sum(ss, red);
    cnt = block_sum(cnt, red);
    const float inv = 1.0f / (float)sqrt(ss);
    write_column_global(colg, n, vx, mk,
                        [=](float v) { return (abs_key(v) >= thr) ? v * inv : 0.f; });
  }
  if (threadIdx.x == 0) {
    hints[j] = done ? new_hint : __uint_as_float(thr);
    nnz_out[j] = (uint32_t)cnt;
  }
}
// `finish`: the step ends here (FinalizeArgs), one start per block.
__global__ void __launch_bounds__(HARD_THREADS) hard_select_kernel(
    const float *__restrict__ Vraw, int ldv, int n, unsigned s, float *__restrict__ Vx,
    uint32_t *__restrict__ nnz_out, uint32_t *__restrict__ vmask, float *__restrict__ hints,
    const uint32_t *__restrict__ cmask, FinalizeArgs a, bool finish) {
  pdl_enter();
  if (step_stopped(a)) return;
  hard_select_body(Vraw, ldv, n, s, Vx, nnz_out, vmask, hints, cmask, blockIdx.x);
  if (finish && threadIdx.x == 0) {
    finalize_value(a, blockIdx.x, a.fz[blockIdx.x], nnz_out[blockIdx.x]);
    close_step(a);
  }
}

// ------------------------------------------------------------ L1 constraint
constexpr int SOFT_C = 1024;  // sorted-candidate chunk (power of two for the bitonic sort)
constexpr int SOFT_THREADS = 256;
// hinted candidates sorted at once (then scanned a chunk at a time)
constexpr int SOFT_HINT_CAP = 4096;
constexpr int SOFT_SMEM = 8 * SOFT_HINT_CAP + 4 * SOFT_C + 2 * 8 * SOFT_C;

// Unfused double arithmetic (no FMA contraction), as host C++ evaluates it.
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
// (S1 - t l) / sqrt(S2 - 2 l S1 + t l^2): ||(|v| - l)_+||_1 / ||(|v| - l)_+||_2 over the
// top t entries, in the reference's operation order (thresh_functions.h:193-204).
__device__ __forceinline__ double ratio_at(double S1, double S2, double t, double l) {
  const double num = dsub(S1, dmul(t, l));
  const double den = __dadd_rn(dsub(S2, dmul(dmul(2.0, l), S1)), dmul(dmul(t, l), l));
  return __ddiv_rn(num, __dsqrt_rn(den));
}

// Inclusive prefix sums of cand[0..total) (0 beyond), in double, offset by
// (o1, o2) for the values and their squares.  4 items per thread.
__device__ void block_scan2(const float *cand, int total, double o1, double o2, double *p1,
                            double *p2, double *red) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int base = t * (SOFT_C / SOFT_THREADS);
  double a[SOFT_C / SOFT_THREADS], b[SOFT_C / SOFT_THREADS];
  double s1 = 0, s2 = 0;
#pragma unroll
  for (int q = 0; q < SOFT_C / SOFT_THREADS; q++) {
    const double v = (base + q < total) ? (double)cand[base + q] : 0.0;
    s1 += v;
    s2 += v * v;
    a[q] = s1;
    b[q] = s2;
  }
  // exclusive scan of (s1, s2) over threads
  double x1 = s1, x2 = s2;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y1 = __shfl_up_sync(FULL, x1, o), y2 = __shfl_up_sync(FULL, x2, o);
    if (lane >= o) {
      x1 += y1;
      x2 += y2;
    }
  }
  __syncthreads();
  if (lane == 31) {
    red[w] = x1;
    red[16 + w] = x2;
  }
  __syncthreads();
  double w1 = 0, w2 = 0;
  for (int i = 0; i < w; i++) {
    w1 += red[i];
    w2 += red[16 + i];
  }
  const double e1 = o1 + w1 + x1 - s1, e2 = o2 + w2 + x2 - s2;
#pragma unroll
  for (int q = 0; q < SOFT_C / SOFT_THREADS; q++) {
    p1[base + q] = e1 + a[q];
    p2[base + q] = e2 + b[q];
  }
  __syncthreads();
}

__device__ void bitonic_sort_desc(float *a) {
  for (int k = 2; k <= SOFT_C; k <<= 1) {
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int i = threadIdx.x; i < SOFT_C; i += blockDim.x) {
        const int ixj = i ^ jj;
        if (ixj > i) {
          const float x = a[i], y = a[ixj];
          const bool first_block = (i & k) == 0;
          if (first_block ? (x < y) : (x > y)) {
            a[i] = y;
            a[ixj] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Evaluates the reference scan's stopping predicates (or, EXACT, the exact
// projection's segment test) at chunk positions q in [0, E) of a descending
// sorted chunk; global rank index g = base + q.  p1/p2 are inclusive prefix
// sums including everything before the chunk (S1, S2).  The value below
// position q is cand[q + 1], or lo_after for the chunk's last position.
// Per thread: the smallest stopping g found and its level; w_last gets the
// '+' root at g = n - 1 (the reference's level when it never stops).
template <bool EXACT>
__device__ void eval_chunk(const float *cand, const double *p1, const double *p2, uint32_t total,
                           uint32_t E, uint32_t base, uint32_t n, double S1, double S2,
                           double lo_after, double sq, double sq2, double lim, uint32_t &best,
                           double &bw, double &w_last) {
  for (uint32_t q = threadIdx.x; q < E; q += blockDim.x) {
    const uint32_t g = base + q;
    const double t = (double)(g + 1);
    const double hi = (double)cand[q];
    const double lov = (q + 1 < total) ? (double)cand[q + 1] : lo_after;
    const double S1i = p1[q], S2i = p2[q];
    // Ranks that cannot stop are passed over without the predicates' roots and
    // quotients.  With R(l) = num / sqrt(den) at the segment's lower end below
    // sqrt(s) by 5e-6 relative, the segment lies strictly between the roots of
    // the stopping quadratic (or, t < s, its discriminant -4 (s - t) s D is
    // negative), at a distance of 5e-6 of their spacing or more; den and D, the
    // spreads that rounding is measured against, are large enough here that the
    // predicates' own rounding moves a root by less than a tenth of that.  Equal
    // or nearly equal leading values (den, D near 0), where the last bit
    // decides, and NaN all fail these tests and are evaluated.
    {
      const double num = S1i - t * lov, den = S2i - 2.0 * lov * S1i + t * lov * lov;
      const double lead = S2i - 2.0 * hi * S1i + t * hi * hi;  // sum (v_i - v_t)^2
      if (num >= 0.0 && num * num < 0.99999 * sq2 * den && lead > 1e-6 * S2i && g + 1 != n &&
          (EXACT || sq2 * (t * S2i - S1i * S1i) > 1e-8 * S1i * S1i * fmax(t, sq2)))
        continue;
    }
    if (!EXACT) {
      // Same operations, order and (unfused) rounding as the reference's
      // expressions at thresh_functions.h:193-213; several of its stops are
      // decided by the last bit (e.g. a zero discriminant at the first step).
      const double S1p = q ? p1[q - 1] : S1, S2p = q ? p2[q - 1] : S2;
      const double left = ratio_at(S1i, S2i, t, hi);
      const double rprev = (g == 0) ? sq : ratio_at(S1p, S2p, t - 1.0, hi);
      const double a = dmul(t, dsub(t, sq2));
      const double b = dsub(dmul(dmul(2.0, S1i), sq2), dmul(dmul(2.0, t), S1i));
      const double c = dsub(dmul(S1i, S1i), dmul(sq2, S2i));
      const double disc = __dsqrt_rn(dsub(dmul(b, b), dmul(dmul(4.0, a), c)));
      const double wm = __ddiv_rn(dsub(-b, disc), dmul(2.0, a));
      const double wp = __ddiv_rn(__dadd_rn(-b, disc), dmul(2.0, a));
      if (g + 1 == n) w_last = wp;
      double cw = 0.0;
      bool hit = false;
      if (left > sq && rprev < sq) {
        hit = true;
        cw = hi;
      } else if (wm > lov && wm < hi) {
        hit = true;
        cw = wm;
      } else if (wp > lov && wp < hi && wp < lim) {
        hit = true;
        cw = wp;
      }
      if (hit && g < best) {
        best = g;
        bw = cw;
      }
    } else {
      const double rlo = (S1i - t * lov) / sqrt(S2i - 2.0 * lov * S1i + t * lov * lov);
      if (rlo >= sq && g < best) {
        const double a = t * (t - sq2);
        const double b = 2.0 * S1i * sq2 - 2.0 * t * S1i;
        const double c = S1i * S1i - sq2 * S2i;
        double lam;
        if (a == 0.0) {
          lam = -c / b;
        } else {
          const double disc = sqrt(fmax(b * b - 4.0 * a * c, 0.0));
          const double r1 = (-b - disc) / (2.0 * a), r2 = (-b + disc) / (2.0 * a);
          // the genuine root keeps every one of the t entries above it
          const bool ok1 = r1 >= lov && r1 <= hi, ok2 = r2 >= lov && r2 <= hi;
          lam = ok1 ? r1 : ok2 ? r2 : fmin(fmax(r1, lov), hi);
        }
        best = g;
        bw = lam;
      }
    }
  }
}

// Block minimum of the per-thread stopping rank; the owning thread publishes
// its level.  Returns the rank (0xFFFFFFFF when nobody stopped) and sets *w.
__device__ uint32_t resolve_stop(uint32_t best, double bw, uint32_t *res,
                                 volatile uint32_t *misc, double *w_sh, double *w) {
  uint32_t mb = best;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mb = min(mb, __shfl_xor_sync(FULL, mb, o));
  if ((threadIdx.x & 31) == 0) res[4 + (threadIdx.x >> 5)] = mb;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t m2 = 0xFFFFFFFFu;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) m2 = min(m2, res[4 + i]);
    misc[1] = m2;
  }
  __syncthreads();
  const uint32_t brk = misc[1];
  if (brk != 0xFFFFFFFFu && best == brk) *w_sh = bw;
  __syncthreads();
  if (brk != 0xFFFFFFFFu) *w = *w_sh;
  __syncthreads();
  return brk;
}

// soft_thresholding (c++/src/utils/thresh_functions.h:162-254): the level w
// and x = sgn(v)(|v| - w)_+, then x <- x / ||x||.
//
// The reference sorts |v| and scans it from the top, stopping at the first
// index i where one of three predicates holds (:197-216).  Common case, three
// passes over the column: a histogram of the top 11 bits of |v| picks the
// highest bins holding at most SOFT_C values; one pass gathers them (and the
// largest value below them); they are sorted in shared memory, prefix sums
// in double give S1 and S2 at every rank, and all ranks' predicates are
// evaluated at once -- the smallest stopping rank wins, and the norm comes
// from the gathered values; a last pass writes the loadings.  When the stop
// lies deeper, the column is walked exactly a chunk of SOFT_C ranks at a time
// (radix select of each chunk boundary, ties by count); a column that never
// stops is walked to its end as in the reference (w is then the '+' root of
// the last step).
// EXACT: stop at the first segment whose lower knot already gives
// ||.||_1/||.||_2 >= sqrt(s) and take the root inside it -- the exact
// L1-ball / unit-sphere projection.
// The reference scan's exact walk over the values src(0..len) (all of a
// column's entries above some bound, or the whole column when len == n), a
// chunk of SOFT_C ranks at a time: each chunk's keys are found by a radix
// select of its lowest rank, gathered, sorted and scanned, and the stopping
// predicates evaluated rank by rank.  lo_end is the largest value below the
// set (0 for the whole column).  Returns the stopping rank and sets *w; NONE
// when the set ran out first (len < n), and the caller walks the column.
// It begins behind the ranks that a sorted candidate set has shown not to stop:
// misc[SEEN] of them (0: none; below len), all the entries with keys of at least
// misc[SEEN_KEY], their S1 and S2 at w_sh[1] and w_sh[2].
enum { SEEN = 4, SEEN_KEY = 5, SET_KEY = 6 };  // words of misc
template <bool EXACT, class Src>
__device__ __noinline__ uint32_t exact_walk(Src src, uint32_t len, uint32_t n, double lo_end, float *cand,
                               double *p1, double *p2, uint32_t *hist, uint32_t *res,
                               double *red, volatile uint32_t *misc, double *w_sh, double sq,
                               double sq2, double *w) {
  const uint32_t NONE = 0xFFFFFFFFu;
  if (len == 0) return NONE;
  uint32_t brk = NONE;
  const SelResult top = block_select_src(src, (int)len, 1u, hist, res);
  const double lim = __dsub_rn((double)__uint_as_float(top.key), 0.000001);
  uint32_t consumed = misc[SEEN], khi = consumed ? misc[SEEN_KEY] : NONE, ge_hi = consumed;
  double S1 = w_sh[1], S2 = w_sh[2];
  while (true) {
    const uint32_t R = min(consumed + (uint32_t)SOFT_C, len);
    const uint32_t total = R - consumed;
    const SelResult lo = block_select_src(src, (int)len, R, hist, res);
    if (threadIdx.x == 0) misc[0] = 0;
    __syncthreads();
    if (lo.key == khi) {
      const float v = __uint_as_float(khi);
      for (uint32_t q = threadIdx.x; q < total; q += blockDim.x) cand[q] = v;
    } else {
      for (int i = threadIdx.x; i < (int)len; i += blockDim.x) {
        const uint32_t key = abs_key(src(i));
        if (key > lo.key && key < khi)
          cand[atomicAdd((uint32_t *)&misc[0], 1u)] = __uint_as_float(key);
      }
      __syncthreads();
      const uint32_t nb = misc[0];
      const uint32_t c_hi = ge_hi - consumed;
      const uint32_t c_lo = R - lo.gt;
      const float vhi = __uint_as_float(khi), vlo = __uint_as_float(lo.key);
      for (uint32_t q = threadIdx.x; q < c_hi + c_lo; q += blockDim.x)
        cand[nb + q] = (q < c_hi) ? vhi : vlo;
    }
    for (uint32_t q = total + threadIdx.x; q < (uint32_t)SOFT_C; q += blockDim.x) cand[q] = -1.f;
    __syncthreads();
    bitonic_sort_desc(cand);
    block_scan2(cand, (int)total, S1, S2, p1, p2, red);
    // the last position of a chunk waits for the next chunk's first value,
    // except at the end of the set, where the value below it is lo_end
    const uint32_t E = (R == len) ? total : total - 1;
    uint32_t best = NONE;
    double bw = 0.0, w_last = 0.0;
    eval_chunk<EXACT>(cand, p1, p2, total, E, consumed, n, S1, S2, lo_end, sq, sq2, lim, best, bw,
                      w_last);
    brk = resolve_stop(best, bw, res, misc, w_sh, w);
    if (brk != NONE) break;
    if (R == len) {
      if (len == n) {
        // never stopped: the reference keeps the '+' root of its last step;
        // the exact projection with ratio < sqrt(s) everywhere is lambda = 0
        if (!EXACT && consumed + E - 1 == n - 1 && threadIdx.x == (E - 1) % blockDim.x)
          *w_sh = w_last;
        if (EXACT && threadIdx.x == 0) *w_sh = 0.0;
        __syncthreads();
        *w = *w_sh;
        __syncthreads();
      }
      break;
    }
    consumed += E;
    S1 = p1[E - 1];
    S2 = p2[E - 1];
    khi = lo.key;
    ge_hi = lo.gt + lo.eq;
    __syncthreads();
  }
  return brk;
}

template <bool EXACT>
__device__ __forceinline__ void soft_select_body(
    const float *__restrict__ Vraw, int ldv, int n, unsigned s, float *__restrict__ Vx,
    uint32_t *__restrict__ nnz_out, uint32_t *__restrict__ vmask, float *__restrict__ hints,
    const uint32_t *__restrict__ cmask, int j) {
  // dynamic shared memory (SOFT_SMEM bytes): the hinted (key, index)
  // candidates, a chunk of sorted values and its prefix sums; the histogram
  // of the slower paths reuses the candidates' space (those paths run only
  // when the hinted one found no stop, and then its pairs are not needed)
  extern __shared__ __align__(16) uint8_t soft_smem[];
  uint64_t *pairs = reinterpret_cast<uint64_t *>(soft_smem);        // SOFT_HINT_CAP
  float *cand = reinterpret_cast<float *>(soft_smem + 8 * SOFT_HINT_CAP);  // SOFT_C
  double *p1 = reinterpret_cast<double *>(soft_smem + 8 * SOFT_HINT_CAP + 4 * SOFT_C);
  double *p2 = p1 + SOFT_C;
  uint32_t *hist = reinterpret_cast<uint32_t *>(soft_smem);           // 2048, over pairs
  __shared__ uint32_t res[32];
  __shared__ double red[32];
  __shared__ uint32_t misc_raw[16];
  __shared__ double w_shared[3];
  volatile uint32_t *misc = misc_raw;
  double *w_sh = w_shared;

  const float *colg = Vraw + (size_t)j * ldv;
  // sqrt(s), sqrt(s)^2 as the double-precision reference forms them
  const double sq = __dsqrt_rn((double)s);
  const double sq2 = __dmul_rn(sq, sq);
  const uint32_t NONE = 0xFFFFFFFFu;

  double w = 0.0;
  uint32_t brk = NONE;
  bool have_norm = false;  // ss and cnt already summed over the gathered values
  bool sparse = false;     // ... and the gathered pairs hold every kept entry
  uint32_t c_pairs = 0;
  double ss = 0.0, cnt = 0.0;
  // ---- candidate sets (1024 columns of 50000, s = 128: 186 us on the first
  // step where the histogram and the chunked walk took 780; 90 to 190 later,
  // where columns that outran the hint took 690): the (key, index) pairs with
  // |v| at or above a bound,
  // sorted and scanned a chunk of SOFT_C ranks at a time.  Attempt 0 takes the
  // hinted set; when that is empty, too large or ends before the stop, attempts
  // 1 and 2 take bounds from a sample of the column (4 s + 64 entries or twice
  // the set that was too small; then as many as fit)
  // A set of attempts 1 and 2 that ends before the stop is not lost: the walks below
  // begin behind it (256 columns of 9000, exact, supports of 4650: 317 us a select,
  // 504 when they began at the first rank, 424 without the attempts)
  constexpr uint32_t MOST = SOFT_HINT_CAP;
  const float hint = hints[j];
  uint32_t c_hint = 0;  // entries at or above the hinted bound
  if (threadIdx.x == 0) {
    misc[SEEN] = 0;
    w_sh[1] = w_sh[2] = 0.0;
  }
  uint32_t want = s < MOST / 4u ? 4u * s + 64u : MOST;
  for (int attempt = hint > 0.f ? 0 : 1; attempt < 3 && brk == NONE; attempt++) {
    uint32_t c = 0, below_key = 0;
    const bool listed = attempt == 0 && cmask != nullptr;
    if (listed) {  // marked by V = B^T Z's epilogue, with the same bound
      c = pairs_from_mask(cmask + (size_t)j * (ldv >> 5), ldv >> 5, colg, pairs, SOFT_HINT_CAP,
                          res);
    } else {
      uint32_t bound = 0;
      if (attempt == 0) {
        bound = hinted_bound(hint);
      } else if (attempt == 2 || want < MOST / 2u) {
        if (attempt == 2) want = MOST;
        bound = sampled_bound(colg, n, want, SOFT_HINT_CAP, reinterpret_cast<uint32_t *>(pairs),
                              res);
      }
      if (bound) {
        c = gather_pairs_above<true>(colg, n, bound, pairs, SOFT_HINT_CAP, res);
        below_key = res[1];
        if (threadIdx.x == 0) misc[SET_KEY] = bound;
      }
    }
    if (attempt == 0) c_hint = c;
    __syncthreads();
    if (c > 0 && c <= (uint32_t)SOFT_HINT_CAP) {
      sort_pairs_desc(pairs, (int)c, SOFT_HINT_CAP);
      // the sorted set, a chunk of SOFT_C ranks at a time; every position sees
      // its next value in the set, except the set's last: for a listed set
      // (no largest value below it) that one is left to the paths below
      const double lim =
          __dsub_rn((double)__uint_as_float((uint32_t)(pairs[0] >> 32)), 0.000001);
      const double lo_after = (c == (uint32_t)n) ? 0.0 : (double)__uint_as_float(below_key);
      double S1 = 0.0, S2 = 0.0, w_last = 0.0;
      uint32_t q0 = 0;
      for (;;) {
        const uint32_t total = min((uint32_t)SOFT_C, c - q0);
        const bool last = q0 + total == c;
        for (uint32_t q = threadIdx.x; q < (uint32_t)SOFT_C; q += blockDim.x)
          cand[q] = (q < total) ? __uint_as_float((uint32_t)(pairs[q0 + q] >> 32)) : -1.f;
        __syncthreads();
        const double next =
            last ? lo_after : (double)__uint_as_float((uint32_t)(pairs[q0 + total] >> 32));
        const uint32_t E = (last && listed && c < (uint32_t)n) ? total - 1 : total;
        block_scan2(cand, (int)total, S1, S2, p1, p2, red);
        uint32_t best = NONE;
        double bw = 0.0;
        eval_chunk<EXACT>(cand, p1, p2, total, E, q0, (uint32_t)n, S1, S2, next, sq, sq2, lim,
                          best, bw, w_last);
        brk = resolve_stop(best, bw, res, misc, w_sh, &w);
        if (brk != NONE || last) break;
        S1 = p1[total - 1];
        S2 = p2[total - 1];
        q0 += total;
        __syncthreads();
      }
      if (brk == NONE && c == (uint32_t)n) {
        // never stopped: the '+' root at the column's last rank (evaluated by
        // the thread holding that position of the last chunk)
        if (!EXACT && threadIdx.x == (c - 1 - q0) % blockDim.x) *w_sh = w_last;
        if (EXACT && threadIdx.x == 0) *w_sh = 0.0;
        __syncthreads();
        w = *w_sh;
        brk = (uint32_t)n;
        __syncthreads();
      }
      if (brk != NONE) {
        // the level lies at or above every value outside the gathered set
        for (uint32_t q = threadIdx.x; q < c; q += blockDim.x) {
          const double d = (double)__uint_as_float((uint32_t)(pairs[q] >> 32)) - w;
          if (d > 0.0) {
            const double x = (double)(float)d;
            ss += x * x;
            cnt += 1.0;
          }
        }
        have_norm = true;
        sparse = true;
        c_pairs = c;
        if (threadIdx.x == 0)
          hints[j] = next_hint(pairs, c, brk + 1u, brk + brk / 2u + 32u, SOFT_HINT_CAP, (float)w);
      } else {
        want = max(want, 2u * c);
        if (!listed && threadIdx.x == 0) {
          misc[SEEN] = c;
          misc[SEEN_KEY] = misc[SET_KEY];
          w_sh[1] = p1[c - 1 - q0];
          w_sh[2] = p2[c - 1 - q0];
        }
      }
    }
    __syncthreads();
  }

  // ---- more than SOFT_HINT_CAP entries above the hinted bound: the exact
  // walk over them alone (a compact list in this column of Vx, which the
  // writes below overwrite); it gives up if the stop lies below the bound
  if (brk == NONE && c_hint > (uint32_t)SOFT_HINT_CAP && c_hint < (uint32_t)n) {
    float *list = Vx + (size_t)j * ldv;
    const uint32_t cl = gather_keys_above(colg, n, hinted_bound(hint), list, res);
    const double lo_end = (double)__uint_as_float(res[1]);
    brk = exact_walk<EXACT>(ListSrc{list}, cl, (uint32_t)n, lo_end, cand, p1, p2, hist, res, red,
                            misc, w_sh, sq, sq2, &w);
  }

  // ---- fast path: the highest bins holding at most SOFT_C values (unless as many
  // ranks are seen already)
  uint32_t c = 0, bstar = 0;
  bool hist_ok = false;  // hist holds the column's top-bit histogram
  if (brk == NONE && (misc[SEEN] < (uint32_t)SOFT_C || n > 8 * SOFT_C)) {
    key_histogram(colg, n, hist);
    hist_ok = true;
  }
  if (brk == NONE && misc[SEEN] < (uint32_t)SOFT_C) {
    find_rank_bin(hist, 2048, (uint32_t)SOFT_C + 1u, res);
    const bool whole = (uint32_t)n <= (uint32_t)SOFT_C;
    bstar = whole ? 0u : res[0] + 1u;  // gather bins >= bstar
    c = whole ? (uint32_t)n : res[1];
    __syncthreads();
  }
  if (brk == NONE && c > 0) {
    if (threadIdx.x == 0) {
      misc[0] = 0;
      misc[2] = 0;
    }
    __syncthreads();
    uint32_t below = 0;  // largest key under the gathered bins
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const uint32_t key = abs_key(colg[i]);
      if ((key >> 20) >= bstar) cand[atomicAdd((uint32_t *)&misc[0], 1u)] = __uint_as_float(key);
      else below = max(below, key);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) below = max(below, __shfl_xor_sync(FULL, below, o));
    if ((threadIdx.x & 31) == 0) atomicMax((uint32_t *)&misc[2], below);
    for (uint32_t q = c + threadIdx.x; q < (uint32_t)SOFT_C; q += blockDim.x) cand[q] = -1.f;
    __syncthreads();
    const double lo_after = (c == (uint32_t)n) ? 0.0 : (double)__uint_as_float(misc[2]);
    bitonic_sort_desc(cand);
    block_scan2(cand, (int)c, 0.0, 0.0, p1, p2, red);
    const double lim = __dsub_rn((double)cand[0], 0.000001);  // ||v||_inf - 1e-6
    uint32_t best = NONE;
    double bw = 0.0, w_last = 0.0;
    eval_chunk<EXACT>(cand, p1, p2, c, c, 0, (uint32_t)n, 0.0, 0.0, lo_after, sq, sq2, lim, best,
                      bw, w_last);
    brk = resolve_stop(best, bw, res, misc, w_sh, &w);
    if (brk == NONE && c == (uint32_t)n) {
      // never stopped: the reference keeps the '+' root of its last step;
      // the exact projection with ratio < sqrt(s) everywhere is lambda = 0
      if (!EXACT && threadIdx.x == (c - 1) % blockDim.x) *w_sh = w_last;
      if (EXACT && threadIdx.x == 0) *w_sh = 0.0;
      __syncthreads();
      w = *w_sh;
      brk = (uint32_t)n;
      __syncthreads();
    }
    if (brk != NONE) {
      // every value above w sits in the gathered chunk
      for (uint32_t q = threadIdx.x; q < c; q += blockDim.x) {
        const double d = (double)cand[q] - w;
        if (d > 0.0) {
          const double x = (double)(float)d;
          ss += x * x;
          cnt += 1.0;
        }
      }
      have_norm = true;
    }
  }

  // ---- exact walk, a chunk of SOFT_C ranks at a time: over the entries in
  // the histogram's bins holding the top 8 * SOFT_C ranks first (a compact
  // list in this column of Vx), then, if the stop lies below them, over the
  // column
  if (brk == NONE && hist_ok && n > 8 * SOFT_C) {
    // the fast path's histogram: the bins holding the top 8 * SOFT_C ranks
    find_rank_bin(hist, 2048, 8u * (uint32_t)SOFT_C, res);
    const uint32_t bound = res[0] << 20;
    __syncthreads();
    float *list = Vx + (size_t)j * ldv;
    const uint32_t cl = gather_keys_above(colg, n, bound, list, res);
    if (cl < (uint32_t)n) {
      const double lo_end = (double)__uint_as_float(res[1]);
      brk = exact_walk<EXACT>(ListSrc{list}, cl, (uint32_t)n, lo_end, cand, p1, p2, hist, res,
                              red, misc, w_sh, sq, sq2, &w);
    }
  }
  if (brk == NONE)
    brk = exact_walk<EXACT>(ColumnSrc{colg}, (uint32_t)n, (uint32_t)n, 0.0, cand, p1, p2, hist,
                            res, red, misc, w_sh, sq, sq2, &w);

  if (threadIdx.x == 0 && !sparse) hints[j] = (float)w;
  // x = sgn(v)(|v| - w)_+ with w kept in double: a level that lands within
  // rounding of the largest |v| still leaves that entry non-zero, as in the
  // reference's double arithmetic.
  if (!have_norm) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const float v = colg[i];
      const double d = (double)fabsf(v) - w;
      if (d > 0.0) {
        const double x = (double)(float)d;
        ss += x * x;
        cnt += 1.0;
      }
    }
  }
  ss = block_sum(ss, red);
  cnt = block_sum(cnt, red);
  const float inv = 1.0f / (float)sqrt(ss);
  float *vx = Vx + (size_t)j * ldv;
  auto soft = [=](float v) {
    const double d = (double)fabsf(v) - w;
    return ((d > 0.0) ? (float)d * sgnf(v) : 0.f) * inv;
  };
  uint32_t *mk = vmask + (size_t)j * (ldv >> 5);
  if (sparse) {
    // every kept entry is a gathered pair: clear the mask, then set the kept
    for (int wd = threadIdx.x; wd < (ldv >> 5); wd += blockDim.x) mk[wd] = 0u;
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < c_pairs; q += blockDim.x) {
      const uint32_t i = ~(uint32_t)pairs[q];
      const float x = soft(__ldg(colg + i));
      if (x != 0.f) {
        vx[i] = x;
        atomicOr(&mk[i >> 5], 1u << (i & 31));
      }
    }
  } else {
    write_column_global(colg, n, vx, mk, soft);
  }
  if (threadIdx.x == 0) {
    nnz_out[j] = (uint32_t)cnt;
  }
}
template <bool EXACT>
__global__ void __launch_bounds__(SOFT_THREADS, 4) soft_select_kernel(
    const float *__restrict__ Vraw, int ldv, int n, unsigned s, float *__restrict__ Vx,
    uint32_t *__restrict__ nnz_out, uint32_t *__restrict__ vmask, float *__restrict__ hints,
    const uint32_t *__restrict__ cmask, FinalizeArgs a, bool finish) {
  pdl_enter();
  if (step_stopped(a)) return;
  soft_select_body<EXACT>(Vraw, ldv, n, s, Vx, nnz_out, vmask, hints, cmask, blockIdx.x);
  if (finish && threadIdx.x == 0) {
    finalize_value(a, blockIdx.x, a.fz[blockIdx.x], nnz_out[blockIdx.x]);
    close_step(a);
  }
}

// ------------------------------------------------------------ finalize
// Penalized and MIXED steps: one warp per start, after the step's other passes.
__global__ void __launch_bounds__(256) finalize_kernel(FinalizeArgs a) {
  pdl_enter();
  if (step_stopped(a)) return;
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j < a.k) finalize_start(a, j, lane);
  __syncthreads();
  if (threadIdx.x == 0) close_step(a);
}

// x = v / ||v|| (c++/src/gpower/sparse_PCA_solver.h:236-237).
__global__ void __launch_bounds__(1024) finalize_x_kernel(const float *__restrict__ v, int n,
                                                          float *__restrict__ x) {
  __shared__ double red[32];
  const int n4 = n >> 2;
  const float4 *v4 = reinterpret_cast<const float4 *>(v);
  float4 *x4 = reinterpret_cast<float4 *>(x);
  double ss = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < n4; i += blockDim.x) {
    const float4 a = v4[i];
    ss += (double)a.x * a.x + (double)a.y * a.y + (double)a.z * a.z + (double)a.w * a.w;
  }
  const int tail = 4 * n4 + threadIdx.x;
  if (tail < n) ss += (double)v[tail] * (double)v[tail];
  ss = block_sum(ss, red);
  const float inv = 1.0f / (float)sqrt(ss);
#pragma unroll 4
  for (int i = threadIdx.x; i < n4; i += blockDim.x) {
    const float4 a = v4[i];
    x4[i] = make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv);
  }
  if (tail < n) x[tail] = v[tail] * inv;
}

// Partial sums of y_i = sum_c B[i, c] x_c in FP64 over chunks of EV_CHUNK
// features: partial[chunk * m + i], threads over samples (coalesced reads of
// B's columns), features with x_c = 0 skipped, a fixed order per chunk.  The
// block lists the chunk's non-zeros first, so that their columns' loads do not
// wait for a test of every feature (2000 x 50000, 16 non-zeros: 3 us, 62 with
// the test).
__global__ void __launch_bounds__(256) ev_partial_kernel(const float *__restrict__ Bc, int ldm,
                                                         int m, int n, const float *__restrict__ x,
                                                         double *__restrict__ partial) {
  __shared__ int list[EV_CHUNK];
  __shared__ float val[EV_CHUNK];
  __shared__ int wsum[EV_CHUNK / 32];
  const int lane = threadIdx.x & 31;
  const int c0 = blockIdx.y * EV_CHUNK, c1 = min(n, c0 + EV_CHUNK);
  constexpr int PER = EV_CHUNK / 256;
  float xc[PER];
  uint32_t bits[PER];
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const int c = c0 + r * 256 + threadIdx.x;
    xc[r] = c < c1 ? x[c] : 0.f;
    bits[r] = __ballot_sync(FULL, xc[r] != 0.f);
    if (lane == 0) wsum[r * 8 + (threadIdx.x >> 5)] = __popc(bits[r]);
  }
  __syncthreads();
  int total = 0, before[PER];
#pragma unroll
  for (int q = 0; q < EV_CHUNK / 32; q++) {
#pragma unroll
    for (int r = 0; r < PER; r++)
      if (q == r * 8 + (int)(threadIdx.x >> 5)) before[r] = total;
    total += wsum[q];
  }
#pragma unroll
  for (int r = 0; r < PER; r++)
    if (xc[r] != 0.f) {
      const int at = before[r] + __popc(bits[r] & ((1u << lane) - 1u));
      list[at] = c0 + r * 256 + threadIdx.x;
      val[at] = xc[r];
    }
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double acc = 0.0;
#pragma unroll 8
  for (int q = 0; q < total; q++) acc += (double)Bc[(size_t)list[q] * ldm + i] * (double)val[q];
  partial[(size_t)blockIdx.y * m + i] = acc;
}

// ||y||^2 (one block).
__global__ void __launch_bounds__(1024) ev_norm_kernel(const double *__restrict__ y, int m,
                                                       double *__restrict__ out) {
  __shared__ double red[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < m; i += blockDim.x) acc += y[i] * y[i];
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) *out = acc;
}

// Compressed sparse columns into B's dense layout (zeroed before): one block
// per column.
__global__ void csc_scatter_kernel(const float *__restrict__ vals,
                                   const int32_t *__restrict__ row_ind,
                                   const int32_t *__restrict__ col_ptr, float *__restrict__ Bc,
                                   int ldm) {
  const size_t c = blockIdx.x;
  for (int q = col_ptr[c] + threadIdx.x; q < col_ptr[c + 1]; q += blockDim.x)
    Bc[c * ldm + row_ind[q]] = vals[q];
}

// The sparse solver's implicit centring made explicit:
// b <- (b - means[c]) - row_means[i] in FP32, either correction optional.
__global__ void center_kernel(float *__restrict__ Bc, int ldm, int m,
                              const float *__restrict__ means,
                              const float *__restrict__ row_means) {
  const size_t c = blockIdx.x;
  const float mc = means ? means[c] : 0.f;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    float b = Bc[c * ldm + i];
    if (means) b = b - mc;
    if (row_means) b = b - row_means[i];
    Bc[c * ldm + i] = b;
  }
}

// y_i = the sum of its chunks' partials (in chunk order), FP64.
// *bad (may be null) is set when some y_i is not finite.
__global__ void rowsum_kernel(const double *__restrict__ partial, int chunks, int m,
                              double *__restrict__ y, int *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double acc = 0.0;
#pragma unroll 8
  for (int c = 0; c < chunks; c++) acc += partial[(size_t)c * m + i];
  y[i] = acc;
  if (bad && !isfinite(acc)) *bad = 1;
}

// Deflation B <- B (I - x x^T) = B - y x^T with y = B x: every entry in FP64,
// rounded to FP32 once.  One block per feature, threads over samples.  Features
// with x_c = 0 keep their values (unless y is not finite: 0 y_i is NaN then), and
// a sparse component leaves most of them: 1000 x 20000 in 13 us, 52 with every
// feature rewritten.
__global__ void deflate_kernel(float *__restrict__ Bc, int ldm, int m,
                               const double *__restrict__ y, const float *__restrict__ x,
                               const int *__restrict__ bad) {
  const size_t c = blockIdx.x;
  const double xc = (double)x[c];
  if (xc == 0.0 && !*bad) return;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const size_t o = c * ldm + i;
    Bc[o] = (float)((double)Bc[o] - y[i] * xc);
  }
}

// ------------------------------------------------------------ GEMM launch
// Co-resident clusters of two CTAs for a pair kernel.
template <class K>
cudaError_t pair_clusters(K kern, int threads, int smem, int *out) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * num_sms());
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  int n = 0;
  cudaError_t e = cudaOccupancyMaxActiveClusters(&n, (void *)kern, &cfg);
  if (e != cudaSuccess) return e;
  if (n < 1) return cudaErrorInvalidConfiguration;
  *out = n;
  return cudaSuccess;
}

// Launch set-up of a kernel on the current device, done once per (kernel,
// device) under a lock (serving runs several host threads, and a process may
// drive several devices): the dynamic shared-memory limit raised to smem and,
// for pair kernels, the number of co-resident clusters of two.
struct LaunchSetup {
  cudaError_t err;
  int clusters;
};
std::mutex g_setup_mu;
std::map<std::pair<const void *, int>, LaunchSetup> g_setup;

template <class K>
cudaError_t kernel_setup(K kern, int smem, int pair_threads = 0, int *clusters = nullptr) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_setup_mu);
  const auto key = std::make_pair(reinterpret_cast<const void *>(kern), dev);
  auto it = g_setup.find(key);
  if (it == g_setup.end()) {
    LaunchSetup c{cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                  0};
    if (c.err == cudaSuccess && pair_threads)
      c.err = pair_clusters(kern, pair_threads, smem, &c.clusters);
    it = g_setup.emplace(key, c).first;
  }
  if (clusters) *clusters = it->second.clusters;
  return it->second.err;
}

// Launches a kernel of a step so that it may start while the one before it
// still runs (programmatic stream serialization): every step kernel begins with
// pdl_enter(), which waits for that one to complete, so only launch latency and
// set-up overlap.  A small batch's step is a chain of short kernels: 20 steps of 64
// starts of 96 x 640 took 1323 us with 2 us and a memset or copy between kernels,
// 849 with this and none.
template <class... P, class... A>
cudaError_t launch_step(void (*kern)(P...), int grid, int threads, int smem, cudaStream_t st,
                        A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

template <int BN, int BKT, int ST, class Epi>
cudaError_t run_gemm(const CUtensorMap &a_hi, const CUtensorMap &a_lo, const CUtensorMap &b_hi,
                     const CUtensorMap &b_lo, const GemmShape &sh, const Epi &epi,
                     cudaStream_t st) {
  using L = GemmSmem<BN, BKT, ST>;
  auto kern = gemm_tf32x3_kernel<BN, BKT, ST, GEMM_PROMO_K / BKT, Epi>;
  const cudaError_t e = kernel_setup(kern, L::TOTAL);
  if (e != cudaSuccess) return e;
  const int grid = sh.num_units < num_sms() ? sh.num_units : num_sms();
  return launch_step(kern, grid, GEMM_THREADS, L::TOTAL, st, a_hi, a_lo, b_hi, b_lo, sh, epi);
}

// Stages per (N tile, K slab) fill ~192 KB of shared memory.
template <class S, int BN, int ST, class Epi>
cudaError_t run_gemm_pair(const CUtensorMap &m0, const CUtensorMap &m1, const CUtensorMap &m2,
                          const CUtensorMap &m3, const GemmShape &sh, const Epi &epi,
                          cudaStream_t st, int splits = 1) {
  using L = PairSmem<S, BN, ST>;
  auto kern = gemm_pair_kernel<S, BN, ST, S::PROMO_K / S::BK, Epi>;
  int clusters = 0;
  const cudaError_t e = kernel_setup(kern, L::TOTAL, PairEpi<BN>::THREADS, &clusters);
  if (e != cudaSuccess) return e;
  GemmShape s2 = sh;  // K blocks of this scheme's BK; units are pair tiles x splits
  s2.kb_total = (sh.K + S::BK - 1) / S::BK;
  s2.kb_per_split = (s2.kb_total + splits - 1) / splits;
  s2.splits = (s2.kb_total + s2.kb_per_split - 1) / s2.kb_per_split;
  s2.num_units = s2.splits * ((sh.m_tiles + 1) / 2) * sh.n_tiles;
  const int pairs = s2.num_units < clusters ? s2.num_units : clusters;
  return launch_step(kern, 2 * pairs, PairEpi<BN>::THREADS, L::TOTAL, st, m0, m1, m2, m3, s2, epi);
}

template <class Epi>
cudaError_t dispatch_gemm(int bn, int bk, const CUtensorMap &a_hi, const CUtensorMap &a_lo,
                          const CUtensorMap &b_hi, const CUtensorMap &b_lo, const GemmShape &sh,
                          const Epi &epi, cudaStream_t st) {
  if (bk == 32) {
    switch (bn) {
      case 256: return run_gemm<256, 32, 2>(a_hi, a_lo, b_hi, b_lo, sh, epi, st);
      case 128: return run_gemm<128, 32, 3>(a_hi, a_lo, b_hi, b_lo, sh, epi, st);
      case 64: return run_gemm<64, 32, 4>(a_hi, a_lo, b_hi, b_lo, sh, epi, st);
    }
  } else if (bk == 16) {
    switch (bn) {
      case 256: return run_gemm<256, 16, 4>(a_hi, a_lo, b_hi, b_lo, sh, epi, st);
      case 128: return run_gemm<128, 16, 6>(a_hi, a_lo, b_hi, b_lo, sh, epi, st);
      case 64: return run_gemm<64, 16, 8>(a_hi, a_lo, b_hi, b_lo, sh, epi, st);
    }
  }
  return cudaErrorInvalidValue;
}

// V = B^T Z: CTA pairs when the N tile is 256 (BF16 operands for the
// L1-variance forms when prepared), else the one-CTA kernel.
template <class Epi>
cudaError_t dispatch_gemm2(const BatchDev &b, const TensorMaps &tm, const GemmShape &sh,
                           const Epi &epi, bool l1_variance, cudaStream_t st) {
  if (b.pair2) {
    if (b.fp16_2) {
      GemmShape s2 = sh;
      s2.row_scale = b.row_scale;
      if (l1_variance)  // B = sgn(z), exact
        return run_gemm_pair<PairFP16x2A, 256, 4>(tm.a2_h0, tm.a2_h1, tm.b2_h0, tm.b2_h0, s2, epi,
                                                  st);
      s2.col_scale = b.z_scale;
      return run_gemm_pair<PairFP16x3, 256, 3>(tm.a2_h0, tm.a2_h1, tm.b2_h0, tm.b2_h1, s2, epi,
                                               st);
    }
    if (b.bf16_2 && l1_variance)
      return run_gemm_pair<PairBF16x3A, 256, 3>(tm.a2_b0, tm.a2_b1, tm.a2_b2, tm.b2_b, sh, epi,
                                                st);
    return run_gemm_pair<PairTF32x3, 256, 3>(tm.a2_hi, tm.a2_lo, tm.b2_hi, tm.b2_lo, sh, epi, st);
  }
  return dispatch_gemm(b.bn2, b.bk, tm.a2_hi, tm.a2_lo, tm.b2_hi, tm.b2_lo, sh, epi, st);
}


}  // namespace

int num_sms() {
  // SMs of the first device that asks (every device of a B200 node has 148);
  // a function-local static, initialised once however many threads ask
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  return sms;
}

bool gather_is_wide(int m) { return m > GATHER_NARROW; }

int pick_bn(int k) { return k > 128 ? 256 : (k > 64 ? 128 : 64); }

size_t ws_floats(int splits, int m_tiles, int n_tiles, int bn) {
  return (size_t)splits * m_tiles * n_tiles * bn * BM;
}

cudaError_t launch_prep_bf16x3(const MatrixDev &M, cudaStream_t st) {
  prep_bf16x3_kernel<<<M.n, 256, 0, st>>>(M.Bc, M.ldm, M.m, (size_t)M.n * M.ldm, M.bf16_planes,
                                          M.Bc_b3);
  return cudaGetLastError();
}

cudaError_t launch_copy_matrix(const MatrixDev &M, const float *B, int ldB, cudaStream_t st) {
  const bool vec = ldB % 4 == 0 && reinterpret_cast<uintptr_t>(B) % 16 == 0;
  copy_matrix_kernel<<<M.n, 256, 0, st>>>(B, ldB, M.m, vec, M.Bc, M.ldm);
  return cudaGetLastError();
}

cudaError_t launch_prep_fp16(const MatrixDev &M, cudaStream_t st) {
  uint32_t *row_key = M.fp16_keys, *key = M.fp16_keys + M.n;
  cudaError_t e = cudaMemsetAsync(M.fp16_keys, 0, sizeof(uint32_t) * ((size_t)M.n + M.m), st);
  if (e != cudaSuccess) return e;
  matrix_max_kernel<<<dim3((M.ldm / 4 + 255) / 256, (M.n + MAX_CHUNK - 1) / MAX_CHUNK), 256, 0,
                      st>>>(M.Bc, M.ldm, M.m, M.n, row_key, key);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  split_matrix_kernel<<<dim3((M.n + 63) / 64, (M.ldm + 63) / 64), 256, 0, st>>>(
      M.Bc, M.ldm, M.m, M.n, M.ldn, row_key, key, M.Bc_h2, (size_t)M.n * M.ldm, M.row_scale,
      M.Bt_h2, (size_t)M.m * M.ldn, M.bt_row_scale);
  return cudaGetLastError();
}

cudaError_t launch_prep_tf32_planes(MatrixDev &M, cudaStream_t st) {
  prep_copy_kernel<<<M.n, 256, 0, st>>>(M.Bc, M.ldm, M.m, M.Bc_hi, M.Bc_lo, nullptr, M.ldm);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  dim3 grid((M.n + 31) / 32, (M.m + 31) / 32);
  prep_transpose_kernel<<<grid, dim3(32, 8), 0, st>>>(M.Bc, M.ldm, M.m, M.n, M.Bt_hi, M.Bt_lo,
                                                      M.ldn);
  return cudaGetLastError();
}

cudaError_t launch_load_columns(const float *src, int ld_src, int rows, int cols, float *dst,
                                int ld_dst, uint32_t *mask, cudaStream_t st) {
  if (cols <= 0) return cudaSuccess;
  load_columns_kernel<<<cols, 256, 0, st>>>(src, ld_src, rows, dst, ld_dst, mask);
  return cudaGetLastError();
}

cudaError_t launch_load_slots(const float *src, int ld_src, int rows, int cols, const int *slots,
                              float *dst, int ld_dst, uint32_t *mask, float *sel_hint, float *val,
                              uint32_t *max_nnz, uint32_t *planes_nnz, cudaStream_t st) {
  if (cols <= 0) return cudaSuccess;
  load_slots_kernel<<<cols, 1024, 0, st>>>(src, ld_src, rows, slots, dst, ld_dst, mask, sel_hint,
                                           val, max_nnz, planes_nnz);
  return cudaGetLastError();
}

// splitmix64's output mixer (Steele, Lea and Flood, "Fast splittable
// pseudorandom number generators", OOPSLA 2014): a bijection on 64-bit words.
__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Column c of the loadings: U[-1, 1) from the top 24 bits of splitmix64((first +
// c) << 32 | i) for row i < rows, scaled to unit 2-norm, zero up to ld, and its
// non-zero mask.  u = t 2^-23 with t a 24-bit integer, so the squares add up
// exactly in integers.  Persistent at two blocks per SM: the second pass, which
// scales, finds the column in L2.  Bound by the mixer's integer instructions:
// 1024 columns of 50000 take 108 us (310 with 256-thread blocks and a pass of
// load_columns_kernel for the values and masks).
constexpr int STARTS_THREADS = 1024;
__global__ void __launch_bounds__(STARTS_THREADS, 2) uniform_starts_kernel(
    float *__restrict__ V, int ld, int rows, int cols, uint32_t first,
    uint32_t *__restrict__ mask) {
  __shared__ double red[32];
  for (int c = blockIdx.x; c < cols; c += gridDim.x) {
    float *v = V + (size_t)c * ld;
    const uint64_t key = (uint64_t)(first + (uint32_t)c) << 32;
    double ss = 0.0;
    uint64_t part = 0;
    int run = 0;  // squares in `part`: each at most 2^46
    float4 *v4 = reinterpret_cast<float4 *>(v);
    for (int q = threadIdx.x; q < (ld >> 2); q += STARTS_THREADS) {
      float u[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int i = 4 * q + e;
        int t = (int)(uint32_t)(splitmix64(key | (uint32_t)i) >> 40) - (1 << 23);
        if (i >= rows) t = 0;
        u[e] = (float)t * (1.0f / 8388608.0f);
        part += (uint64_t)((int64_t)t * t);
      }
      v4[q] = make_float4(u[0], u[1], u[2], u[3]);
      if ((run += 4) == 1 << 17) {
        ss += (double)part;
        part = 0;
        run = 0;
      }
    }
    ss = block_sum((ss + (double)part) * (1.0 / 70368744177664.0), red);
    const float inv = (float)(1.0 / sqrt(ss));
    for (int q = threadIdx.x; q < (ld >> 2); q += STARTS_THREADS) {
      float4 x = v4[q];
      x = make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
      v4[q] = x;
      uint32_t nz = (x.x != 0.f) | (x.y != 0.f) << 1 | (x.z != 0.f) << 2 | (x.w != 0.f) << 3;
      // eight lanes hold a word (ld is a multiple of 32, so they are all here)
      nz <<= 4 * (threadIdx.x & 7);
      const uint32_t eight = 0xFFu << (threadIdx.x & 24);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) nz |= __shfl_xor_sync(eight, nz, o);
      if ((threadIdx.x & 7) == 0) mask[(size_t)c * (ld >> 5) + (q >> 3)] = nz;
    }
  }
}

cudaError_t launch_uniform_starts(float *V, int ld, int rows, int cols, uint32_t first,
                                  uint32_t *mask, cudaStream_t st) {
  if (cols <= 0) return cudaSuccess;
  uniform_starts_kernel<<<std::min(cols, 2 * num_sms()), STARTS_THREADS, 0, st>>>(
      V, ld, rows, cols, first, mask);
  return cudaGetLastError();
}

// ValueCoordinateHolder::reset (c++/src/utils/various.h:33-38) and a batch's
// other words for newly loaded starts: no hints, a dense first step, no planes,
// the run-ahead words cleared.
__global__ void reset_batch_kernel(int k, float *sel_hint, float *val, float *err,
                                   uint32_t *max_nnz, uint32_t *planes_nnz, uint32_t *ctl) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < k) {
    sel_hint[j] = 0.f;
    val[j] = 0.f;
    err[j] = 0.f;
  }
  if (j < CTL_WORDS) ctl[j] = 0u;
  if (j == 0) {
    *max_nnz = 0xFFFFFFFFu;
    if (planes_nnz) *planes_nnz = 0u;
  }
}
cudaError_t launch_reset_batch(int k, float *sel_hint, float *val, float *err, uint32_t *max_nnz,
                               uint32_t *planes_nnz, uint32_t *ctl, cudaStream_t st) {
  reset_batch_kernel<<<(std::max(k, (int)CTL_WORDS) + 255) / 256, 256, 0, st>>>(
      k, sel_hint, val, err, max_nnz, planes_nnz, ctl);
  return cudaGetLastError();
}

cudaError_t launch_masked_copy(const float *Vx, const uint32_t *mask, int ld, int rows, int cols,
                               float *dst, int ld_dst, cudaStream_t st) {
  if (cols <= 0) return cudaSuccess;
  const int pieces = std::min(65535, (rows + COPY_ROWS - 1) / COPY_ROWS);
  masked_copy_kernel<<<dim3(cols, pieces), 256, 0, st>>>(Vx, mask, ld, rows, dst, ld_dst);
  return cudaGetLastError();
}

// One warp waits, bounded by timeout_ns, on an mbarrier that nothing arrives
// on: the wait gives up, records DEV_ERR_TIMEOUT_PROBE in *status and the
// kernel returns, as every kernel's waits do when a partner never comes.
__global__ void bounded_wait_probe_kernel(unsigned long long timeout_ns, int *status) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();
  mbar_wait_bounded(&bar, 0, &abort_flag, status, DEV_ERR_TIMEOUT_PROBE, timeout_ns);
  __syncwarp();
}

cudaError_t launch_bounded_wait_probe(unsigned long long timeout_ns, int *status,
                                      cudaStream_t st) {
  bounded_wait_probe_kernel<<<1, 32, 0, st>>>(timeout_ns, status);
  return cudaGetLastError();
}

cudaError_t launch_finalize_x(const float *v, int n, float *x, cudaStream_t st) {
  finalize_x_kernel<<<1, 1024, 0, st>>>(v, n, x);
  return cudaGetLastError();
}

cudaError_t launch_explained_variance(const MatrixDev &M, const float *x, double *partial,
                                      double *out, cudaStream_t st) {
  const int chunks = (M.n + EV_CHUNK - 1) / EV_CHUNK;
  ev_partial_kernel<<<dim3((M.m + 255) / 256, chunks), 256, 0, st>>>(M.Bc, M.ldm, M.m, M.n, x,
                                                                     partial);
  double *y = partial + (size_t)chunks * M.m;
  rowsum_kernel<<<(M.m + 127) / 128, 128, 0, st>>>(partial, chunks, M.m, y, nullptr);
  ev_norm_kernel<<<1, 1024, 0, st>>>(y, M.m, out);
  return cudaGetLastError();
}

cudaError_t launch_csc_to_dense(MatrixDev &M, const float *vals, const int32_t *row_ind,
                               const int32_t *col_ptr, const float *means,
                               const float *row_means, cudaStream_t st) {
  csc_scatter_kernel<<<M.n, 256, 0, st>>>(vals, row_ind, col_ptr, M.Bc, M.ldm);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || (!means && !row_means)) return e;
  center_kernel<<<M.n, 256, 0, st>>>(M.Bc, M.ldm, M.m, means, row_means);
  return cudaGetLastError();
}

cudaError_t launch_deflate(MatrixDev &M, const float *x, double *partial, double *y, int *bad,
                           cudaStream_t st) {
  const int chunks = (M.n + EV_CHUNK - 1) / EV_CHUNK;
  ev_partial_kernel<<<dim3((M.m + 255) / 256, chunks), 256, 0, st>>>(M.Bc, M.ldm, M.m, M.n, x,
                                                                     partial);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(bad, 0, sizeof(int), st)) != cudaSuccess) return e;
  rowsum_kernel<<<(M.m + 255) / 256, 256, 0, st>>>(partial, chunks, M.m, y, bad);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  deflate_kernel<<<M.n, 256, 0, st>>>(M.Bc, M.ldm, M.m, y, x, bad);
  return cudaGetLastError();
}

// The select of a constrained form (the L1 ball in p's mode); see the kernels.
static cudaError_t launch_select(int f, const StepParams &p, int k, const float *Vraw, int ldn,
                                 int n, float *Vx, uint32_t *nnz, uint32_t *vmask, float *hints,
                                 const uint32_t *cmask, const FinalizeArgs &fa, bool finish,
                                 cudaStream_t st) {
  if (!is_l1_constrained(f))
    return launch_step(hard_select_kernel, k, HARD_THREADS, 0, st, Vraw, ldn, n, p.constraint, Vx,
                       nnz, vmask, hints, cmask, fa, finish);
  auto kern = p.l1_mode == 0 ? soft_select_kernel<false> : soft_select_kernel<true>;
  const cudaError_t e = kernel_setup(kern, SOFT_SMEM);
  if (e != cudaSuccess) return e;
  return launch_step(kern, k, SOFT_THREADS, SOFT_SMEM, st, Vraw, ldn, n, p.constraint, Vx, nnz,
                     vmask, hints, cmask, fa, finish);
}

cudaError_t launch_am_step(const MatrixDev &M, BatchDev &b, const TensorMaps &tm,
                           const StepParams &p, cudaStream_t st, int *launches, cudaEvent_t *ev,
                           int *kinds) {
  cudaError_t e;
  int nl = 0;
  const int f = p.formulation;
  auto mark = [&](int kind) -> cudaError_t {
    if (kinds) kinds[nl] = kind;
    return ev ? cudaEventRecord(ev[nl], st) : cudaSuccess;
  };
  if (b.mixed &&  // the support this step starts from, for the stability count
      (e = cudaMemcpyAsync(b.vmask_prev, b.vmask, sizeof(uint32_t) * (size_t)b.k * (M.ldn / 32),
                           cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
    return e;
  // 1. Z = B V (split-K partials)
  GemmShape g1;
  g1.M = M.m;
  g1.N = b.k;
  g1.K = M.n;
  g1.m_tiles = b.m_tiles1;
  g1.n_tiles = b.n_tiles1;
  g1.kb_total = (M.n + b.bk - 1) / b.bk;
  g1.kb_per_split = b.kbps1;
  g1.splits = b.splits1;
  g1.num_units = g1.splits * g1.m_tiles * g1.n_tiles;
  g1.timeout_ns = p.timeout_ns;
  g1.status = b.status;
  g1.stop = b.ctl;
  g1.gate = b.max_nnz;  // dense steps only
  g1.gate_min = b.sparse_cap + 1;
  g1.gate_max = 0xFFFFFFFFu;
  const int mode = is_l1_variance(f) ? 1 : (is_constrained(f) ? 0 : 2);
  const size_t zplane = (size_t)b.k * M.ldm;  // second FP16 plane of Z
  float *z_lo = b.fp16_2 ? nullptr : b.Z_lo;  // FP16 operands read no TF32 planes
  // 1a. sparse V (every column <= sparse_cap non-zeros last step): gather
  const bool wide = gather_is_wide(M.m);
  if ((e = mark(9)) != cudaSuccess) return e;
  if (wide) {
    // the lists take the dense planes' place (not read on sparse steps)
    int2 *lists = reinterpret_cast<int2 *>(b.fp16_1 ? (void *)b.V_h : (void *)b.V_hi);
    if ((e = launch_step(gather_list_kernel, b.k, GATHER_THREADS, 0, st, M.ldn, b.Vx, b.vmask,
                         b.max_nnz, b.sparse_cap, lists, b.max_err, b.ctl)) != cudaSuccess)
      return e;
    nl++;
    if ((e = mark(5)) != cudaSuccess) return e;
    if ((e = launch_step(gather_tile_kernel, gather_tiles(M.ldm) * gather_groups(b.k),
                         GATHER_THREADS, 0, st, M.Bc, M.ldm, M.ldn, b.k, lists, b.Z_hi,
                         b.max_nnz, b.sparse_cap, b.ctl)) != cudaSuccess)
      return e;
    nl++;
  } else {
    if ((e = launch_step(gather_narrow_kernel, b.k, GATHER_THREADS, 0, st, mode, M.Bc, M.ldm, M.m,
                         M.ldn, b.Vx, b.vmask, b.Z_hi, z_lo, b.fz, b.max_nnz, b.sparse_cap, b.Z_b,
                         b.Z_h, zplane, b.z_scale, b.max_err, b.ctl)) != cudaSuccess)
      return e;
    nl++;
    if (ev) {  // one launch serves both kinds: am24_batch_step_timed names it by the counts
      if ((e = mark(5)) != cudaSuccess) return e;
      nl++;
    }
  }
  // 1b. dense V: TF32 hi/lo planes, tensor-core Z = B V (split-K partials) ...
  if ((e = mark(6)) != cudaSuccess) return e;
  if (b.fp16_1)
    e = launch_step(densify_fp16_kernel, std::min(b.k, DENSIFY_BLOCKS_PER_SM * num_sms()),
                    DENSIFY_THREADS, 0, st, b.Vx, b.vmask, M.ldn, M.n, b.V_h, (size_t)b.k * M.ldn,
                    b.v_scale, b.max_nnz, b.sparse_cap, b.ctl, b.k);
  else
    e = launch_step(densify_kernel, b.k, 256, 0, st, b.Vx, b.vmask, M.ldn, M.n, b.V_hi, b.V_lo,
                    b.max_nnz, b.planes_nnz, b.sparse_cap, b.ctl);
  if (e != cudaSuccess) return e;
  nl++;
  EpiPartial ep{b.ws, b.bn1, b.m_tiles1, b.n_tiles1};
  if ((e = mark(0)) != cudaSuccess) return e;
  if (b.fp16_1) {
    GemmShape gp = g1;
    gp.row_scale = b.bt_row_scale;
    gp.col_scale = b.v_scale;
    e = run_gemm_pair<PairFP16x3, 256, 3>(tm.a1_h0, tm.a1_h1, tm.b1_h0, tm.b1_h1, gp, ep, st,
                                          b.splits1p);
  } else {
    e = dispatch_gemm(b.bn1, b.bk, tm.a1_hi, tm.a1_lo, tm.b1_hi, tm.b1_lo, g1, ep, st);
  }
  if (e != cudaSuccess) return e;
  nl++;
  // 2. ... then reduce + sign / normalise
  const int splits1 = b.fp16_1 ? b.splits1p : b.splits1;
  if ((e = mark(1)) != cudaSuccess) return e;
  if ((e = launch_step(z_reduce_kernel, b.k, 256, 0, st, mode, b.ws, splits1, b.m_tiles1,
                       b.n_tiles1, b.bn1, M.m, b.Z_hi, z_lo, M.ldm, b.fz, b.max_nnz, b.sparse_cap,
                       b.Z_b, b.Z_h, zplane, b.z_scale, wide, b.ctl)) != cudaSuccess)
    return e;
  nl++;
  // 3. V = B^T Z
  GemmShape g2;
  g2.M = M.n;
  g2.N = b.k;
  g2.K = M.m;
  g2.m_tiles = b.m_tiles2;
  g2.n_tiles = b.n_tiles2;
  g2.kb_total = (M.m + b.bk - 1) / b.bk;
  g2.kb_per_split = g2.kb_total;
  g2.splits = 1;
  g2.num_units = g2.m_tiles * g2.n_tiles;
  g2.timeout_ns = p.timeout_ns;
  g2.status = b.status;
  g2.stop = b.ctl;
  g2.gate = nullptr;
  g2.gate_min = 0;
  g2.gate_max = 0;
  const int parts = b.m_tiles2 * 4;
  // MIXED: the single-pass BF16 product runs while phase[0] == 0, the
  // FP32-accurate one from then on; each launch returns at once in the other phase
  auto gemm2 = [&](const auto &epi) -> cudaError_t {
    cudaError_t e2;
    if (b.mixed) {
      GemmShape gl = g2;
      gl.gate = b.phase;
      gl.gate_min = 0;
      gl.gate_max = 0;
      if ((e2 = mark(7)) != cudaSuccess) return e2;
      if (b.mixed_fp16) {
        gl.row_scale = b.row_scale;
        gl.col_scale = is_l1_variance(f) ? nullptr : b.z_scale;  // sgn(z) is exact
        e2 = run_gemm_pair<PairFP16x1, 256, 6>(tm.a2_h0, tm.b2_h0, tm.a2_h0, tm.b2_h0, gl, epi,
                                                st);
      } else {
        e2 = run_gemm_pair<PairBF16x1, 256, 6>(tm.a2_b0, tm.b2_b, tm.a2_b0, tm.b2_b, gl, epi,
                                                st);
      }
      if (e2 != cudaSuccess) return e2;
      nl++;
      g2.gate = b.phase;
      g2.gate_min = 1;
      g2.gate_max = 0xFFFFFFFFu;
    }
    if ((e2 = mark(2)) != cudaSuccess) return e2;
    if ((e2 = dispatch_gemm2(b, tm, g2, epi, is_l1_variance(f), st)) != cudaSuccess) return e2;
    nl++;
    return cudaSuccess;
  };
  // the penalty epilogue writes the next dense step's TF32 planes of V
  // (unless that step's Z = B V takes FP16 planes from densify_fp16_kernel)
  float *vhi = b.fp16_1 ? nullptr : b.V_hi;
  if (is_constrained(f)) {
    EpiRaw er{b.Vraw, M.ldn, M.n, b.k, b.bn2};
    if (b.cmask) {  // the selects' hinted gather, done while V is in registers
      er.hint = b.sel_hint;
      er.cmask = b.cmask;
    }
    e = gemm2(er);
  } else if (is_l1_penalized(f)) {
    EpiPenalty<true> pe{b.Vx,       b.obj_part, b.nnz_part, M.ldn,    M.n,
                        b.k,        b.bn2,      parts,      (float)p.penalty,
                        b.vmask,    vhi,        b.V_lo,     b.max_nnz, b.sparse_cap};
    e = gemm2(pe);
  } else {
    EpiPenalty<false> pe{b.Vx,       b.obj_part, b.nnz_part, M.ldn,    M.n,
                         b.k,        b.bn2,      parts,      (float)p.penalty,
                         b.vmask,    vhi,        b.V_lo,     b.max_nnz, b.sparse_cap};
    e = gemm2(pe);
  }
  if (e != cudaSuccess) return e;
  FinalizeArgs fa;
  fa.k = b.k;
  fa.formulation = f;
  fa.parts = parts;
  fa.it = p.it;
  fa.store_all = p.store_all;
  fa.log_shift = p.log_shift;
  fa.log_capacity = b.log_capacity;
  fa.tolerance = p.tolerance;
  fa.fz = b.fz;
  fa.obj_part = b.obj_part;
  fa.nnz_part = b.nnz_part;
  fa.nnz_sel = b.nnz;
  fa.val = b.val;
  fa.err = b.err;
  fa.max_err = b.max_err;
  fa.iters = b.iters;
  fa.cards = b.cards;
  fa.next_nnz = b.ctl + CTL_NEXT_NNZ;
  fa.max_nnz = b.max_nnz;
  // penalized forms: the count this step's epilogue saw (whether it wrote the
  // dense planes), for the next step's densify gate
  fa.planes_nnz = !is_constrained(f) && !b.fp16_1 ? b.planes_nnz : nullptr;
  fa.ctl = b.ctl;
  fa.host_stop = p.host_stop;
  fa.phase = b.mixed ? b.phase : nullptr;
  fa.status = b.status;
  fa.stop_check = p.stop_check;
  // 4. constrained: selection / projection + normalisation, and the step's end
  const bool finish = is_constrained(f) && !b.mixed;
  if (is_constrained(f)) {
    if ((e = mark(3)) != cudaSuccess) return e;
    if ((e = launch_select(f, p, b.k, b.Vraw, M.ldn, M.n, b.Vx, b.nnz, b.vmask, b.sel_hint, b.cmask,
                           fa, finish, st)) != cudaSuccess)
      return e;
    nl++;
  }
  // 4b. MIXED: support stability and the phase switch
  if (b.mixed) {
    if ((e = mark(8)) != cudaSuccess) return e;
    if ((e = launch_step(support_kernel, b.k, 256, 0, st, b.vmask, b.vmask_prev, M.ldn / 32,
                         b.stable, b.phase, b.k_stable, b.need_stable, b.ctl)) != cudaSuccess)
      return e;
    nl++;
  }
  // 5. finalize
  if (!finish) {
    if ((e = mark(4)) != cudaSuccess) return e;
    if ((e = launch_step(finalize_kernel, (b.k + 7) / 8, 256, 0, st, fa)) != cudaSuccess) return e;
    nl++;
  }
  if (ev && (e = cudaEventRecord(ev[nl], st)) != cudaSuccess) return e;
  if (launches) *launches = nl;
  return cudaSuccess;
}

// ------------------------------------------------------------ grouped steps
#include "gemm_pair_grouped.cuh"
#include "am24_group_kernels.cuh"

namespace {

template <class K>
cudaError_t persistent_grid(K kern, int threads, int smem, int *grid) {
  int per = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (void *)kern, threads, smem);
  if (e != cudaSuccess) return e;
  *grid = num_sms() * (per > 0 ? per : 1);
  return cudaSuccess;
}

template <int BN, int EPI>
cudaError_t grouped_gemm_setup(int *clusters) {
  return kernel_setup(gemm_pair_grouped_kernel<BN, EPI>, GPairSmem<BN>::TOTAL,
                      PairEpi<BN>::THREADS, clusters);
}

template <int BN, int EPI>
cudaError_t launch_grouped_gemm(const GroupDev &g, int list, cudaStream_t st) {
  int clusters = 0;
  const cudaError_t e = grouped_gemm_setup<BN, EPI>(&clusters);
  if (e != cudaSuccess) return e;
  gemm_pair_grouped_kernel<BN, EPI>
      <<<2 * clusters, PairEpi<BN>::THREADS, GPairSmem<BN>::TOTAL, st>>>(g, list);
  return cudaGetLastError();
}

// The three N tiles of one epilogue, lists l64, l64 + 1, l64 + 2; the widest first.
template <int EPI>
cudaError_t launch_grouped_gemms(const GroupDev &g, int l64, cudaStream_t st) {
  cudaError_t e;
  if ((e = launch_grouped_gemm<256, EPI>(g, l64 + 2, st)) ||
      (e = launch_grouped_gemm<128, EPI>(g, l64 + 1, st)) ||
      (e = launch_grouped_gemm<64, EPI>(g, l64, st)))
    return e;
  return cudaSuccess;
}

template <int EPI>
cudaError_t grouped_gemms_setup(int *c) {
  cudaError_t e;
  if ((e = grouped_gemm_setup<64, EPI>(c)) || (e = grouped_gemm_setup<128, EPI>(c)) ||
      (e = grouped_gemm_setup<256, EPI>(c)))
    return e;
  return cudaSuccess;
}

}  // namespace

cudaError_t grouped_grids(GroupGrids *gr) {
  cudaError_t e;
  int c = 0;
  if ((e = grouped_gemms_setup<GE_PARTIAL>(&c)) || (e = grouped_gemms_setup<GE_RAW>(&c)) ||
      (e = grouped_gemms_setup<GE_PL1>(&c)) || (e = grouped_gemms_setup<GE_PL0>(&c)))
    return e;
  if ((e = persistent_grid(g_z_reduce_kernel, 256, 0, &gr->col)) ||
      (e = persistent_grid(g_hard_select_kernel, HARD_THREADS, 0, &gr->select_hard)) ||
      (e = kernel_setup(g_soft_select_kernel<false>, SOFT_SMEM)) ||
      (e = kernel_setup(g_soft_select_kernel<true>, SOFT_SMEM)) ||
      (e = persistent_grid(g_soft_select_kernel<false>, SOFT_THREADS, SOFT_SMEM,
                           &gr->select_soft)) ||
      (e = persistent_grid(g_gather_narrow_kernel, GATHER_THREADS, 0, &gr->gather)) ||
      (e = persistent_grid(g_gather_tile_kernel, GATHER_THREADS, 0, &gr->gather_tile)) ||
      (e = persistent_grid(g_finalize_kernel, 256, 0, &gr->fin)))
    return e;
  return cudaSuccess;
}

// The parts of a step that do not depend on one another run as branches (side
// streams of the capture): the sparse gathers beside the dense product, the three
// epilogues of V = B^T Z beside each other, the selects beside the penalties'
// products.  Every one is persistent and ends with a tail of its last units, which
// the next branch's blocks fill: a queue of 16 requests on 4 matrices took 12.8 ms
// one after another, 11.7 so.
cudaError_t launch_grouped_step(const GroupDev &g, const GroupGrids &gr, const GroupStreams &q,
                                cudaStream_t st) {
  cudaError_t e;
  auto after = [&](cudaStream_t to, int ev, cudaStream_t from) -> cudaError_t {
    const cudaError_t r = cudaEventRecord(q.ev[ev], from);
    return r ? r : cudaStreamWaitEvent(to, q.ev[ev], 0);
  };
  group_plan_kernel<<<1, PLAN_THREADS, 0, st>>>(g);
  if ((e = cudaGetLastError())) return e;
  // Z = B V: the sparse gathers, and the dense path
  if ((e = after(q.side[0], 0, st))) return e;
  g_gather_list_kernel<<<gr.col, GATHER_THREADS, 0, q.side[0]>>>(g);
  g_gather_tile_kernel<<<gr.gather_tile, GATHER_THREADS, 0, q.side[0]>>>(g);
  g_gather_narrow_kernel<<<gr.gather, GATHER_THREADS, 0, q.side[0]>>>(g);
  g_densify_kernel<<<DENSIFY_BLOCKS_PER_SM * num_sms(), DENSIFY_THREADS, 0, st>>>(g);
  if ((e = cudaGetLastError())) return e;
  if ((e = launch_grouped_gemms<GE_PARTIAL>(g, GL_GEMM1_64, st))) return e;
  if ((e = after(st, 1, q.side[0]))) return e;
  g_z_reduce_kernel<<<gr.col, 256, 0, st>>>(g);
  if ((e = cudaGetLastError())) return e;
  // V = B^T Z with the raw output marked for the selects or the penalty fused
  if ((e = after(q.side[0], 2, st)) || (e = cudaStreamWaitEvent(q.side[1], q.ev[2], 0)) ||
      (e = launch_grouped_gemms<GE_RAW>(g, GL_RAW_64, st)) ||
      (e = launch_grouped_gemms<GE_PL0>(g, GL_PL0_64, q.side[0])) ||
      (e = launch_grouped_gemms<GE_PL1>(g, GL_PL1_64, q.side[1])) ||
      (e = after(q.side[2], 3, st)))
    return e;
  g_soft_select_kernel<false><<<gr.select_soft, SOFT_THREADS, SOFT_SMEM, st>>>(g);
  g_soft_select_kernel<true><<<gr.select_soft, SOFT_THREADS, SOFT_SMEM, st>>>(g);
  g_hard_select_kernel<<<gr.select_hard, HARD_THREADS, 0, q.side[2]>>>(g);
  if ((e = cudaGetLastError()) || (e = after(st, 4, q.side[0])) || (e = after(st, 5, q.side[1])) ||
      (e = after(st, 6, q.side[2])))
    return e;
  g_support_kernel<<<gr.col, 256, 0, st>>>(g);
  g_finalize_kernel<<<gr.fin, 256, 0, st>>>(g);
  return cudaGetLastError();
}

cudaError_t launch_grouped_condition(const GroupDev &g, unsigned long long handle,
                                     cudaStream_t st, bool in_graph) {
  g_condition_kernel<<<1, 256, 0, st>>>(g, (cudaGraphConditionalHandle)handle, in_graph);
  return cudaGetLastError();
}

// ------------------------------------------------------------ sparse steps
#include "am24_sparse_kernels.cuh"

namespace {
// One product on the compressed arrays: the tile kernel for the outer entries
// and the segments of the long ones, the combine kernel for the long ones' sums.
// gate (may be null): the launches do their work only when *gate >= gate_min.
// xmask (may be null): the rows of X that are not zero, per tile of starts.
template <bool SKIP, bool ROWS>
void sparse_product(const int32_t *ptr, const int32_t *idx, const float *val, int ncols,
                    const SparseLong &L, const float *X, float *part, const SparseBatchDev &b,
                    float *out, int ld_out, const float *cvec, const double *a, const double *bv,
                    const uint32_t *gate, uint32_t gate_min, const uint32_t *xmask,
                    cudaStream_t st) {
  const int tiles = (b.kp + SP_WIDE - 1) / SP_WIDE;
  const int seg_blocks = L.count ? (L.segs + SP_OUTER - 1) / SP_OUTER : 0;
  sp_spmm_kernel<SKIP, ROWS>
      <<<dim3(seg_blocks + (ncols + SP_OUTER - 1) / SP_OUTER, tiles), SP_THREADS, 0, st>>>(
          ptr, idx, val, ncols, X, b.kp, b.k, out, ld_out, cvec, a, bv, b.ctl, gate, gate_min,
          xmask, b.ldn / 32, L.seg_e0, L.seg_e1, L.segs, seg_blocks, part);
  if (L.count == 0) return;
  sp_spmm_long_kernel<ROWS><<<dim3(L.count, b.kp / SP_TILE), SP_TILE, 0, st>>>(
      L.outer, L.seg_first, part, b.kp, b.k, out, ld_out, cvec, a, bv, b.ctl, gate, gate_min);
}

}  // namespace

// Blocks a tile of starts for the pass over Z: over all tiles as many as run at once
// (three a multiprocessor), each warp with at least four rows.
int sparse_zblocks(int m, int kp) {
  const int tiles = (kp + SP_WIDE - 1) / SP_WIDE;
  const int most = std::max(1, 3 * num_sms() / tiles);
  const int per = 4 * SP_THREADS / 32;
  return std::max(1, std::min(most, (m + per - 1) / per));
}

cudaError_t launch_sparse_step(const SparseDev &S, const SparseBatchDev &b, const StepParams &p,
                               cudaStream_t st) {
  cudaError_t e;
  const int f = p.formulation;
  const bool centred = S.means || S.row_means;
  // 1. Z = (B - 1 mu^T - r 1^T) V: CSR rows against V transposed
  // the centring's sums, and the entries a scatter of the supports would touch
  sp_vstats_kernel<<<b.k, SP_THREADS, 0, st>>>(b.Vx, b.vmask, b.ldn, S.n, S.means,
                                               centred ? b.sum_v : nullptr, b.dot_mu, S.col_ptr,
                                               b.work, b.ctl);
  // the scatter of each support when the previous step left at most
  // SP_SCATTER_CAP loadings in every start and the scatter touches fewer
  // entries than the CSR product steps through; else the CSR product
  // deflated: the projected loadings P v are dense, so the CSR product runs
  if (S.comps > 0)
    sp_defl_coef_kernel<<<b.k, SP_THREADS, 0, st>>>(
        b.Vx, b.vmask, b.ldn, S.n, S.defl, S.comps, S.gram, S.defl_sum, S.defl_mu, b.defl_a,
        centred ? b.sum_v : nullptr, b.dot_mu, b.ctl);
  sp_zgate_kernel<<<1, 1, 0, st>>>(
      b.max_nnz, (uint32_t)SP_SCATTER_CAP, b.work,
      S.comps > 0 ? -1.0 : SP_SCATTER_PER_STEP * (double)S.nnz * (double)(b.kp / 32), b.zgate,
      b.max_err, b.ctl);
  sp_transpose_v_kernel<<<dim3((S.n + SP_TILE - 1) / SP_TILE, (b.kp + SP_WIDE - 1) / SP_WIDE),
                          SP_THREADS, 0, st>>>(b.Vx, b.vmask, b.ldn, S.n, b.k, b.Vt, b.kp,
                                               b.xmask, b.ctl, b.zgate, 1u, S.defl, S.comps,
                                               b.defl_a);
  sparse_product<true, true>(S.row_ptr, S.col_ind, S.rvals, S.m, S.long_rows, b.Vt, b.part_rows,
                             b, b.Zt, b.kp, S.row_means, S.row_means ? b.sum_v : nullptr,
                             S.means ? b.dot_mu : nullptr, b.zgate, 1u, b.xmask, st);
  sp_scatter_z_kernel<<<b.k, SP_THREADS, 0, st>>>(
      S.col_ptr, S.row_ind, S.cvals, b.Vx, b.vmask, b.ldn, b.Zs, b.ldm, S.m, S.row_means,
      S.row_means ? b.sum_v : nullptr, S.means ? b.dot_mu : nullptr, b.zgate, 0u, b.ctl);
  // eight blocks a multiprocessor, so that a step without the scatter passes quickly
  const int zt_blocks = std::max(1, 8 * num_sms() / (b.kp / SP_TILE));
  sp_transpose_z_kernel<<<dim3(std::min((S.m + SP_TILE - 1) / SP_TILE, zt_blocks),
                               b.kp / SP_TILE),
                          SP_THREADS, 0, st>>>(b.Zs, b.ldm, S.m, b.k, b.Zt, b.kp, b.zgate, b.ctl);
  // 2. the formulation's sign / norm of z, and the sums V's correction needs
  const dim3 zp(sparse_zblocks(S.m, b.kp), (b.kp + SP_WIDE - 1) / SP_WIDE);
  const int rows = (S.m + zp.x - 1) / zp.x;
  const bool l1var = f & 1, norm = f <= 3 || !l1var, twice = f > 3 && !l1var;
  sp_zpass_kernel<<<zp, SP_THREADS, 0, st>>>(b.Zt, b.kp, S.m, rows, f, nullptr, centred,
                                             S.row_means, b.zpart, b.ctl);
  if (norm || centred)
    sp_zsum_kernel<<<b.kp / 32, SP_THREADS, 0, st>>>(b.zpart, zp.x, b.kp, b.k, f, norm,
                                                     centred && !twice, b.fz, b.zinv, b.zsum,
                                                     b.zdot, b.ctl);
  if (twice) {
    sp_zpass_kernel<<<zp, SP_THREADS, 0, st>>>(b.Zt, b.kp, S.m, rows, f, b.zinv, centred,
                                               S.row_means, b.zpart, b.ctl);
    if (centred)
      sp_zsum_kernel<<<b.kp / 32, SP_THREADS, 0, st>>>(b.zpart, zp.x, b.kp, b.k, f, false, true,
                                                       b.fz, b.zinv, b.zsum, b.zdot, b.ctl);
  }
  // 3. V = (B - 1 mu^T - r 1^T)^T Z: CSC columns against Z transposed
  sparse_product<false, false>(S.col_ptr, S.row_ind, S.cvals, S.n, S.long_cols, b.Zt,
                               b.part_cols, b, b.Vraw, b.ldn, S.means,
                               S.means ? b.zsum : nullptr, S.row_means ? b.zdot : nullptr,
                               nullptr, 0, nullptr, st);
  if (S.comps > 0)
    sp_defl_vraw_kernel<<<b.k, SP_THREADS, 0, st>>>(b.Vraw, b.ldn, S.n, S.defl, S.comps, S.gram,
                                                    b.ctl);
  if ((e = cudaGetLastError())) return e;
  // 4. thresholds: the dense path's selects (own candidate gather), or the penalties
  FinalizeArgs fa;
  fa.k = b.k;
  fa.formulation = f;
  fa.parts = 1;
  fa.it = p.it;
  fa.store_all = p.store_all;
  fa.log_shift = p.log_shift;
  fa.log_capacity = b.log_capacity;
  fa.tolerance = p.tolerance;
  fa.fz = b.fz;
  fa.obj_part = b.obj_part;
  fa.nnz_part = b.nnz_part;
  fa.nnz_sel = b.nnz;
  fa.val = b.val;
  fa.err = b.err;
  fa.max_err = b.max_err;
  fa.iters = b.iters;
  fa.cards = b.cards;
  fa.next_nnz = b.ctl + CTL_NEXT_NNZ;
  fa.max_nnz = b.max_nnz;
  fa.planes_nnz = nullptr;
  fa.ctl = b.ctl;
  fa.host_stop = p.host_stop;
  fa.phase = nullptr;
  fa.status = b.status;
  fa.stop_check = p.stop_check;
  if (is_constrained(f)) {
    return launch_select(f, p, b.k, b.Vraw, b.ldn, S.n, b.Vx, b.nnz, b.vmask, b.sel_hint, nullptr,
                         fa, true, st);
  } else if (is_l1_penalized(f)) {
    sp_penalty_kernel<true><<<b.k, SP_THREADS, 0, st>>>(b.Vraw, b.ldn, S.n, (float)p.penalty,
                                                        b.Vx, b.vmask, b.obj_part, b.nnz_part,
                                                        b.ctl);
  } else {
    sp_penalty_kernel<false><<<b.k, SP_THREADS, 0, st>>>(b.Vraw, b.ldn, S.n, (float)p.penalty,
                                                         b.Vx, b.vmask, b.obj_part, b.nnz_part,
                                                         b.ctl);
  }
  if ((e = cudaGetLastError())) return e;
  // 5. objective, change, logs and the batch loop's termination test
  finalize_kernel<<<(b.k + 7) / 8, 256, 0, st>>>(fa);
  return cudaGetLastError();
}

cudaError_t launch_sparse_ev(const SparseDev &S, const float *x, double *scratch, double *out,
                             cudaStream_t st) {
  const int blocks = (S.m + SP_THREADS - 1) / SP_THREADS;
  double *xs = scratch, *partial = scratch + 2;
  sp_ev_xstats_kernel<<<1, SP_THREADS, 0, st>>>(x, S.n, S.means, xs);
  sp_ev_rows_kernel<<<blocks, SP_THREADS, 0, st>>>(S.row_ptr, S.col_ind, S.rvals, S.m, x,
                                                   S.row_means, xs, partial);
  sp_ev_sum_kernel<<<1, SP_THREADS, 0, st>>>(partial, blocks, out);
  return cudaGetLastError();
}

}  // namespace am24
