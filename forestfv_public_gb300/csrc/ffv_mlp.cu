// Learned refinement indicator: a 135-64-64-1 perceptron (GELU, GELU, sigmoid) over the
// 27-cell stencil of five per-cell fields, trained on the GPU with AdamW.
//
// Inputs: for every cell, the fields log rho, log p, alpha_0, |u| and the von Mises stress
// of the 27 cells reached by steps of -1/0/+1 along x, then y, then z across faces (a
// boundary face keeps the cell, a face with four finer neighbours takes the first of them),
// normalised per field by a stored mean and standard deviation: 135 BF16 values, padded to
// 144 with zeros.  Output: the probability that the plain criterion will ask for a finer
// level within the prediction horizon.
//
// Arithmetic: BF16 operands, FP32 accumulation on the tensor cores.  Inference (features,
// both layers and the marks in one kernel, mlp_infer_tc): a CTA builds the feature rows of
// 128 cells in shared memory and one thread issues tcgen05.mma (M = 128, N = 64) for each
// layer, the accumulators in tensor memory.  Training: warp-level mma.sync m16n8k16 over
// 64-sample tiles, the weight gradients accumulated in registers and summed over blocks in a
// fixed order.
// Where a tensor-core product needs an operand the forward pass holds in FP32 (the hidden
// activations, the pre-activation gradients) it is rounded to BF16; the CPU restatement
// (oracle/mlp.py) rounds at the same points.
#include <cuda_bf16.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "ffv.h"
#include "ffv_device.cuh"
#include "ffv_m5.cuh"
#include "ffv_tc.cuh"

namespace {

constexpr int NIN = 135, KIN = 144, NH = 64;
constexpr int OFF_W1 = 0, OFF_B1 = NH * NIN, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH;
constexpr int OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NH, NPARAM = OFF_B3 + 1;
static_assert(NPARAM == FFV_MLP_NPARAM, "parameter count");
constexpr int SX = 152;  // shared row stride (bf16) of 144-wide tiles: conflict-free fragments
constexpr int SH = 72;   // shared row stride (bf16) of 64-wide tiles

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ uint32_t ld32(const bf16 *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ uint32_t pack2(bf16 lo, bf16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}
__device__ __forceinline__ void mma16816(float c[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// GELU (exact, erf form)
__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

// ------------------------------------------------------------------------- features
// the cells across faces fneg and fpos of cell e: a boundary face keeps the cell, a face
// with four finer neighbours takes the first of them
__device__ __forceinline__ void face_steps(const ffv_dmesh &m, int32_t e, int fneg, int fpos,
                                           int32_t &en, int32_t &ep) {
  const uint32_t info = m.info[e];
  const uint32_t kn = ffv_face_kind(info, fneg), kp = ffv_face_kind(info, fpos);
  en = e;
  ep = e;
  if (!(kn & FFV_FK_BC)) {
    const int32_t s = m.nbr[(int64_t)fneg * m.n + e];
    en = kn == FFV_FK_FINER ? m.sub[4 * (int64_t)s] : s;
  }
  if (!(kp & FFV_FK_BC)) {
    const int32_t s = m.nbr[(int64_t)fpos * m.n + e];
    ep = kp == FFV_FK_FINER ? m.sub[4 * (int64_t)s] : s;
  }
}

// the 27 stencil cells of c, o = (dx + 1) + 3 (dy + 1) + 9 (dz + 1): the step along x, then
// along y, then along z.  The walks share their prefixes: 2 + 6 + 18 independent face steps
// in three dependent rounds.
__device__ __forceinline__ void stencil27(const ffv_dmesh &m, int32_t c, int32_t e[27]) {
  int32_t x[3], y[9];
  x[1] = c;
  face_steps(m, c, 0, 2, x[0], x[2]);
#pragma unroll
  for (int ix = 0; ix < 3; ix++) {
    y[ix + 3] = x[ix];
    face_steps(m, x[ix], 3, 1, y[ix], y[ix + 6]);
  }
#pragma unroll
  for (int j = 0; j < 9; j++) {
    e[j + 9] = y[j];
    face_steps(m, y[j], 4, 5, e[j], e[j + 18]);
  }
}

// the 135 normalised features of a cell as BF16, eight per 16-byte chunk (chunk 16 holds
// features 128-134 and a zero, chunk 17 zeros), handed to put(chunk, uint4).  A stencil cell's five
// come as one record: a value is normalised and rounded once, where its cell's fields are formed,
// and not by each of the 27 rows that take it, and a row's gather is 27 loads instead of 135.
template <typename Put>
__device__ __forceinline__ void cell_features(const ffv_dmesh &m, const uint4 *__restrict__ R,
                                              int32_t c, Put put) {
  int32_t e[27];
  stencil27(m, c, e);
  uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int o = 0; o < 27; o++) {
    const uint4 r = R[e[o]];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      const int k = 5 * o + q;
      const uint32_t pair = q < 2 ? r.x : (q < 4 ? r.y : r.z);
      const uint32_t u = (q & 1) ? pair >> 16 : pair & 0xFFFFu;
      if ((k & 1) == 0) w[(k & 7) >> 1] = u;
      else w[(k & 7) >> 1] |= u << 16;
      if ((k & 7) == 7) put(k >> 3, make_uint4(w[0], w[1], w[2], w[3]));
    }
  }
  put(NIN >> 3, make_uint4(w[0], w[1], w[2], w[3] & 0xFFFFu));
  put(KIN / 8 - 1, make_uint4(0u, 0u, 0u, 0u));
}

// A block builds its 128 feature rows in shared memory (row stride 146 BF16 = 73 words,
// odd, so that the threads' 4-byte accesses to their own rows fall in distinct banks) and
// then writes them out as one contiguous run of 4-byte words: a thread writing its own
// 288-byte row directly would touch 32 cache lines per warp store.
constexpr int GATHER_TPB = 128, GATHER_SW = 73;  // shared words per row (KIN / 2 = 72, +1)
__global__ void __launch_bounds__(GATHER_TPB) mlp_gather(ffv_dmesh m, const uint4 *__restrict__ R,
                                                         bf16 *__restrict__ X) {
  __shared__ uint32_t tile[GATHER_TPB * GATHER_SW];
  const int64_t c0 = (int64_t)blockIdx.x * GATHER_TPB;
  const int64_t c = c0 + threadIdx.x;
  if (c < m.n) {
    uint32_t *row = tile + threadIdx.x * GATHER_SW;
    cell_features(m, R, (int32_t)c, [&](int ch, uint4 v) {
      row[4 * ch] = v.x;
      row[4 * ch + 1] = v.y;
      row[4 * ch + 2] = v.z;
      row[4 * ch + 3] = v.w;
    });
  }
  __syncthreads();
  const int64_t rows = m.n - c0 < GATHER_TPB ? m.n - c0 : GATHER_TPB;
  const int words = (int)rows * (KIN / 2);
  uint32_t *dst = reinterpret_cast<uint32_t *>(X + c0 * KIN);
  for (int w = threadIdx.x; w < words; w += GATHER_TPB)
    dst[w] = tile[(w / (KIN / 2)) * GATHER_SW + w % (KIN / 2)];
}

// ------------------------------------------------------------------------- weights
__global__ void mlp_pack(const float *__restrict__ P, bf16 *__restrict__ W1, bf16 *__restrict__ W2,
                         bf16 *__restrict__ W2T) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NH * KIN; i += gridDim.x * blockDim.x) {
    const int r = i / KIN, k = i % KIN;
    W1[i] = __float2bfloat16_rn(k < NIN ? P[OFF_W1 + r * NIN + k] : 0.0f);
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NH * NH; i += gridDim.x * blockDim.x) {
    const int r = i / NH, k = i % NH;
    const bf16 w = __float2bfloat16_rn(P[OFF_W2 + i]);
    W2[i] = w;
    W2T[k * NH + r] = w;
  }
}

// ------------------------------------------------------------------ inference (tcgen05)
// One CTA of 128 threads per 128-cell tile (persistent over tiles), thread r owning cell
// row r.  Shared memory, canonical K-major BF16 tiles (ffv_tc.cuh): the feature tile X
// [128][144] (later the first hidden layer H [128][64] over it), W1 [64][144], W2 [64][64],
// then b1, b2, w3 in FP32.  Tensor memory: 64 FP32 columns x 128 lanes, the accumulator of
// either layer (lane r = row r).  Per tile: rows built (stencil gather or copied feature
// rows) -> 9 MMAs (K = 16) of layer 1 -> GELU + BF16 of row r into H -> 4 MMAs of layer 2 ->
// GELU, the w3 dot product and the sigmoid of row r.  The MMAs take ~1 us of a tile's time:
// the gather dominates, and three CTAs per SM overlap one another's phases.
constexpr int TC_ROWS = 128;
constexpr int TC_SBO_X = (KIN / 8) * 128, TC_SBO_H = (NH / 8) * 128;
constexpr int TC_W1 = TC_ROWS * KIN * 2;     // byte offsets in the dynamic shared memory
constexpr int TC_W2 = TC_W1 + NH * KIN * 2;
constexpr int TC_VEC = TC_W2 + NH * NH * 2;
constexpr int TC_SMEM = TC_VEC + 3 * NH * 4;
constexpr int TC_CTAS_PER_SM = 3;
constexpr int TC_TMEM_COLS = 64;
constexpr int TC_WAIT_POLLS = 1 << 22;  // an MMA group takes ~1 us; this is far beyond it
static_assert(TC_SMEM * TC_CTAS_PER_SM <= 227 * 1024, "shared memory of three CTAs per SM");
static_assert(TC_TMEM_COLS * TC_CTAS_PER_SM <= 512, "tensor memory of three CTAs per SM");

template <bool GATHER>
__global__ void __launch_bounds__(TC_ROWS, TC_CTAS_PER_SM)
    mlp_infer_tc(ffv_dmesh m, const uint4 *__restrict__ R, const bf16 *__restrict__ X, int64_t n, const bf16 *__restrict__ W1,
                 const bf16 *__restrict__ W2, const float *__restrict__ P, float *__restrict__ prob,
                 uint8_t *__restrict__ marks, float threshold, int accumulate,
                 unsigned *__restrict__ err) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ uint32_t tmem_holder;
  __shared__ __align__(8) uint64_t bar;
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int i = tid; i < NH * (KIN / 8); i += TC_ROWS) {
    const int r = i / (KIN / 8), ch = i % (KIN / 8);
    *reinterpret_cast<uint4 *>(sm + TC_W1 + tc::kmajor_offset(r, 8 * ch, KIN)) =
        *reinterpret_cast<const uint4 *>(W1 + r * KIN + 8 * ch);
  }
  for (int i = tid; i < NH * (NH / 8); i += TC_ROWS) {
    const int r = i / (NH / 8), ch = i % (NH / 8);
    *reinterpret_cast<uint4 *>(sm + TC_W2 + tc::kmajor_offset(r, 8 * ch, NH)) =
        *reinterpret_cast<const uint4 *>(W2 + r * NH + 8 * ch);
  }
  float *b1s = reinterpret_cast<float *>(sm + TC_VEC), *b2s = b1s + NH, *w3s = b2s + NH;
  for (int i = tid; i < NH; i += TC_ROWS) {
    b1s[i] = P[OFF_B1 + i];
    b2s[i] = P[OFF_B2 + i];
    w3s[i] = P[OFF_W3 + i];
  }
  if (warp == 0) tc::tmem_alloc(&tmem_holder, TC_TMEM_COLS);
  if (tid == 0) tc::mbar_init(&bar, 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_holder;
  const uint32_t row_tmem = tmem + ((uint32_t)(warp * 32) << 16);  // this warp's 32 lanes
  const uint32_t xs = tc::smem_addr(sm), w1s = tc::smem_addr(sm + TC_W1),
                 w2s = tc::smem_addr(sm + TC_W2);
  constexpr uint32_t idesc = tc::idesc_bf16_f32(TC_ROWS, NH);
  const float b3 = P[OFF_B3];
  const int64_t ntiles = (n + TC_ROWS - 1) / TC_ROWS;
  int failed_parity = -1;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t c = t * TC_ROWS + tid;
    const bool valid = c < n;
    auto put = [&](int ch, uint4 v) {
      *reinterpret_cast<uint4 *>(sm + tc::kmajor_offset(tid, 8 * ch, KIN)) = v;
    };
    if (!valid) {
#pragma unroll 1
      for (int ch = 0; ch < KIN / 8; ch++) put(ch, make_uint4(0u, 0u, 0u, 0u));
    } else if (GATHER) {
      cell_features(m, R, (int32_t)c, put);
    } else {
#pragma unroll
      for (int ch = 0; ch < KIN / 8; ch++) put(ch, *reinterpret_cast<const uint4 *>(X + c * KIN + 8 * ch));
    }
    // layer 1: pre-activations of the 128 rows into tensor memory
    tc::fence_async_shared();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0) {
#pragma unroll
      for (int kk = 0; kk < KIN / 16; kk++)
        tc::mma_bf16(tmem, tc::sdesc(xs + 256 * kk, 128, TC_SBO_X), tc::sdesc(w1s + 256 * kk, 128, TC_SBO_X),
                     idesc, kk > 0);
      tc::commit(&bar);
    }
    if (__syncthreads_or(!tc::mbar_wait(&bar, 0, TC_WAIT_POLLS))) {
      failed_parity = 0;
      break;
    }
    tc::fence_after_sync();
    // rolled, like the loop of layer 2: 128 erff in line are 80 KB of code, which every warp then
    // waited for (1.7 M cells: 696 -> 531 us)
#pragma unroll 1
    for (int c0 = 0; c0 < NH; c0 += 16) {
      float a[16];
      tc::tmem_ld16(row_tmem + c0, a);
      uint32_t pk[8];
#pragma unroll
      for (int j = 0; j < 8; j++)
        pk[j] = pack2(__float2bfloat16_rn(gelu(a[2 * j] + b1s[c0 + 2 * j])),
                      __float2bfloat16_rn(gelu(a[2 * j + 1] + b1s[c0 + 2 * j + 1])));
      *reinterpret_cast<uint4 *>(sm + tc::kmajor_offset(tid, c0, NH)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      *reinterpret_cast<uint4 *>(sm + tc::kmajor_offset(tid, c0 + 8, NH)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
    // layer 2 over H (the feature tile's first 16 KB: layer 1 has finished reading it)
    tc::fence_async_shared();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0) {
#pragma unroll
      for (int kk = 0; kk < NH / 16; kk++)
        tc::mma_bf16(tmem, tc::sdesc(xs + 256 * kk, 128, TC_SBO_H), tc::sdesc(w2s + 256 * kk, 128, TC_SBO_H),
                     idesc, kk > 0);
      tc::commit(&bar);
    }
    if (__syncthreads_or(!tc::mbar_wait(&bar, 1, TC_WAIT_POLLS))) {
      failed_parity = 1;
      break;
    }
    tc::fence_after_sync();
    float z = 0.0f;
#pragma unroll 1
    for (int c0 = 0; c0 < NH; c0 += 16) {
      float a[16];
      tc::tmem_ld16(row_tmem + c0, a);
#pragma unroll
      for (int j = 0; j < 16; j++) z += gelu(a[j] + b2s[c0 + j]) * w3s[c0 + j];
    }
    if (valid) {
      const float p = 1.0f / (1.0f + expf(-(z + b3)));
      if (prob) prob[c] = p;
      if (marks) {
        const uint8_t hit = p > threshold ? 1 : 0;
        marks[c] = accumulate ? (uint8_t)(marks[c] | hit) : hit;
      }
    }
    // the next tile's MMAs (after its barrier) overwrite the accumulator these loads read
    tc::fence_before_sync();
  }
  if (failed_parity >= 0) {
    // a wait ran out: report it, give the MMAs in flight one more bounded wait, free the
    // tensor memory and leave (the tiles not finished keep their outputs)
    if (tid == 0) atomicOr(err, 1u);
    tc::mbar_wait(&bar, (uint32_t)failed_parity, TC_WAIT_POLLS);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, TC_TMEM_COLS);
}

// row index of sample i of a training step: identity (seed 0) or a hashed draw
__device__ __forceinline__ int64_t sample_row(uint64_t seed, int64_t step, int64_t i, int64_t N) {
  if (seed == 0) return i;
  uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(step * 1315423911ll + i + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (int64_t)(z % (uint64_t)N);
}

// reduce a per-lane column partial over the eight row groups (lanes with the same q)
__device__ __forceinline__ float rows_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  return v;
}

// ------------------------------------------------------------------ training (mma.sync)
// The gradient of one batch, in two launches.
//
// mlp_grad_tiles: a block of eight warps takes 64 samples at a time.  Warp w holds rows 16 (w & 3) ..
// of the tile and the output columns 32 (w >> 2) .. of either hidden layer, forms its activations
// and their derivatives from one erf and one exponential each, and the pre-activation gradients;
// the weight gradients are products over the tile's 64 samples (dW = dA^T X, both operands read
// transposed by ldmatrix), accumulated in registers over the block's tiles: warp w owns rows
// 16 (w & 3) .. and half of the columns of dW1 and dW2.  Every block then writes its own gradient.
// mlp_update: the blocks' gradients summed in a fixed order (the result does not depend on the order
// of execution), and AdamW and the BF16 copies of the weights in the same launch.
//
// What bounds it: at 8192 samples the grid is 128 blocks of one tile each, so the time is one
// tile's chain of loads, products and activations.  With one warp per 16 samples, shared-memory
// atomics for every outer product and global ones per block the gradient took 64 us and a step, with
// its two clears, AdamW, packing and loss copy, 82 us; now 18 us of a step of 24, and 18 with each
// kernel's launch overlapping the one before (the next batch's rows load during the update).
constexpr int TG = 64, TG_TPB = 256;               // samples per tile, threads
constexpr int PART = NPARAM + 1;                   // a block's gradient and loss
struct TrainSmem {
  bf16 W1[NH * SX], W2[NH * SH], W2T[NH * SH];
  bf16 X[TG * SX], H1[TG * SH], DA2[TG * SH], DA1[TG * SH];
  float b1[NH], b2[NH], w3[NH], y[TG], cols[3][4][NH], last[2][4];
  float logit[NH / 8][TG][4];  // the logits' terms: column tile, sample, lane of its quad
  int64_t row[TG];
};

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t r[4], const bf16 *p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

// GELU (exact, erf form) and its derivative from one erf.  Every product and sum that BF16 rounding or
// AdamW's m / sqrt(v) could carry on is rounded as in the kernel that took one warp per 16 samples
// (explicit forms here, in the logits' terms and in the column sums): the gradient of one 16-sample tile
// has that kernel's bits.
__device__ __forceinline__ void gelu_both(float x, float &h, float &d) {
  const float half_cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  h = x * half_cdf;
  d = __fadd_rn(half_cdf, __fmul_rn(__fmul_rn(x, 0.39894228040143268f), expf(-0.5f * x * x)));
}

// acc[nt] += A^T B over the tile's 64 samples for rows m0 .. m0 + 15 of A^T and NT column tiles from
// n0 of B; A [64][SH], B [64][sb].  Sixteen samples at a time from zero, the products added in FP32:
// the tensor core's accumulator does not round to nearest, and a chain of products through it grows
// with the batch (a million samples: entries off by up to 230 * 2^-24 of their terms' magnitudes with
// the chain, 26 now).  Rolled: four copies of the loop cost more in instruction fetches (40 steps of
// 8192: 762 us unrolled, 693 rolled, 671 with the chain).
template <int NT>
__device__ __forceinline__ void outer_tile(const bf16 *A, int m0, const bf16 *B, int sb, int n0,
                                           float acc[NT][4]) {
  const int lane = threadIdx.x & 31, j = lane >> 3, r = lane & 7;
#pragma unroll 1
  for (int kk = 0; kk < TG / 16; kk++) {
    uint32_t a[4];  // the 8 x 8 blocks (m, k): (0, 0), (8, 0), (0, 8), (8, 8)
    ldmatrix_x4_trans(a, A + (kk * 16 + (j >> 1) * 8 + r) * SH + m0 + (j & 1) * 8);
#pragma unroll
    for (int nt = 0; nt < NT; nt += 2) {
      // blocks (k, n): (0, 0), (8, 0) and the next column tile's; a last odd tile loads itself twice
      const int n = n0 + 8 * (nt + 1 < NT ? nt + (j >> 1) : nt);
      uint32_t b[4];
      ldmatrix_x4_trans(b, B + (kk * 16 + (j & 1) * 8 + r) * sb + n);
#pragma unroll
      for (int t = 0; t < (nt + 1 < NT ? 2 : 1); t++) {
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        mma16816(c, a[0], a[1], a[2], a[3], b[2 * t], b[2 * t + 1]);
#pragma unroll
        for (int e = 0; e < 4; e++) acc[nt + t][e] += c[e];
      }
    }
  }
}

// c[nt] = A B^T for the 16 rows of A from row0 (stride sa) and four column tiles from n0 of B [n][k]
// (stride sb), K the contraction length
template <int K>
__device__ __forceinline__ void rows_times(const bf16 *A, int row0, int sa, const bf16 *B, int n0,
                                           int sb, float c[4][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 4; nt++) c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.0f;
#pragma unroll
  for (int kk = 0; kk < K / 16; kk++) {
    const int k0 = kk * 16 + 2 * q;
    const bf16 *x = A + (row0 + g) * sa + k0;
    const uint32_t x0 = ld32(x), x1 = ld32(x + 8 * sa), x2 = ld32(x + 8), x3 = ld32(x + 8 * sa + 8);
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const bf16 *w = B + (n0 + nt * 8 + g) * sb + k0;
      mma16816(c[nt], x0, x1, x2, x3, ld32(w), ld32(w + 8));
    }
  }
}

// gradient of the mean binary cross-entropy over B samples (rows drawn by sample_row): the
// block's share and its sum of the loss into part[blockIdx.x]
__global__ void __launch_bounds__(TG_TPB) mlp_grad_tiles(const bf16 *__restrict__ X,
                                                         const float *__restrict__ y, int64_t N,
                                                         int64_t B, uint64_t seed, int64_t step,
                                                         const bf16 *W1, const bf16 *W2,
                                                         const bf16 *W2T, const float *P, float *part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainSmem &s = *reinterpret_cast<TrainSmem *>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int row0 = 16 * (warp & 3), n0 = 32 * (warp >> 2);
  const int64_t ntiles = (B + TG - 1) / TG;
  const auto load_tile = [&](int64_t t) {
    const int64_t i0 = t * TG;
    const int valid = (int)((B - i0) < TG ? (B - i0) : TG);
    if (tid < TG) {
      const int64_t r = tid < valid ? sample_row(seed, step, i0 + tid, N) : 0;
      s.row[tid] = r;
      s.y[tid] = tid < valid ? y[r] : 0.0f;
    }
    __syncthreads();
    for (int i = tid; i < TG * (KIN / 8); i += TG_TPB) {
      const int r = i / (KIN / 8), ch = i % (KIN / 8);
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < valid) v = *reinterpret_cast<const uint4 *>(X + s.row[r] * KIN + ch * 8);
      *reinterpret_cast<uint4 *>(s.X + r * SX + ch * 8) = v;
    }
  };
  // the samples do not depend on the step before: they load while its update still runs
  cudaTriggerProgrammaticLaunchCompletion();
  load_tile(blockIdx.x);
  cudaGridDependencySynchronize();
  for (int i = tid; i < NH * (KIN / 8); i += TG_TPB) {
    const int r = i / (KIN / 8), ch = i % (KIN / 8);
    *reinterpret_cast<uint4 *>(s.W1 + r * SX + ch * 8) = *reinterpret_cast<const uint4 *>(W1 + r * KIN + ch * 8);
  }
  for (int i = tid; i < NH * (NH / 8); i += TG_TPB) {
    const int r = i / (NH / 8), ch = i % (NH / 8);
    *reinterpret_cast<uint4 *>(s.W2 + r * SH + ch * 8) = *reinterpret_cast<const uint4 *>(W2 + r * NH + ch * 8);
    *reinterpret_cast<uint4 *>(s.W2T + r * SH + ch * 8) = *reinterpret_cast<const uint4 *>(W2T + r * NH + ch * 8);
  }
  if (tid < NH) {
    s.b1[tid] = P[OFF_B1 + tid];
    s.b2[tid] = P[OFF_B2 + tid];
    s.w3[tid] = P[OFF_W3 + tid];
  }
  const float b3 = P[OFF_B3], invB = 1.0f / (float)B;
  float dW1[9][4], dW2[4][4], db1[4][2], db2[4][2], dw3[4][2], db3 = 0.0f, loss = 0.0f;
#pragma unroll
  for (int i = 0; i < 9; i++) dW1[i][0] = dW1[i][1] = dW1[i][2] = dW1[i][3] = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    dW2[i][0] = dW2[i][1] = dW2[i][2] = dW2[i][3] = 0.0f;
    db1[i][0] = db1[i][1] = db2[i][0] = db2[i][1] = dw3[i][0] = dw3[i][1] = 0.0f;
  }
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int valid = (int)((B - t * TG) < TG ? (B - t * TG) : TG);
    __syncthreads();
    // first hidden layer: H1 in BF16, the derivatives kept
    float a[4][4], g1[4][4];
    rows_times<KIN>(s.X, row0, SX, s.W1, n0, SX, a);
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const int col = n0 + nt * 8 + 2 * q;
      float h[4];
#pragma unroll
      for (int e = 0; e < 4; e++) gelu_both(a[nt][e] + s.b1[col + (e & 1)], h[e], g1[nt][e]);
      *reinterpret_cast<__nv_bfloat162 *>(s.H1 + (row0 + g) * SH + col) = __floats2bfloat162_rn(h[0], h[1]);
      *reinterpret_cast<__nv_bfloat162 *>(s.H1 + (row0 + g + 8) * SH + col) = __floats2bfloat162_rn(h[2], h[3]);
    }
    __syncthreads();
    // second hidden layer and this warp's terms of the logits
    float h2[4][4], g2[4][4];
    rows_times<NH>(s.H1, row0, SH, s.W2, n0, SH, a);
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const int col = n0 + nt * 8 + 2 * q;
#pragma unroll
      for (int e = 0; e < 4; e++) gelu_both(a[nt][e] + s.b2[col + (e & 1)], h2[nt][e], g2[nt][e]);
      s.logit[(n0 >> 3) + nt][row0 + g][q] =
          __fmaf_rn(h2[nt][0], s.w3[col], __fmul_rn(h2[nt][1], s.w3[col + 1]));
      s.logit[(n0 >> 3) + nt][row0 + g + 8][q] =
          __fmaf_rn(h2[nt][3], s.w3[col + 1], __fmul_rn(h2[nt][2], s.w3[col]));
    }
    __syncthreads();
    // the logits, formed alike by both warps of a row: a chain over the column tiles, then the quad
    float z[2] = {0.0f, 0.0f};
#pragma unroll
    for (int e = 0; e < 2; e++) {
#pragma unroll
      for (int nt = 0; nt < NH / 8; nt++) z[e] += s.logit[nt][row0 + g + 8 * e][q];
      z[e] += __shfl_xor_sync(0xffffffffu, z[e], 1);
      z[e] += __shfl_xor_sync(0xffffffffu, z[e], 2);
    }
    // output layer: d loss / d z = (p - y) / B
    float dz[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int r = row0 + g + 8 * e;
      dz[e] = 0.0f;
      if (r < valid) {
        const float p = 1.0f / (1.0f + expf(-(z[e] + b3))), yy = s.y[r];
        dz[e] = (p - yy) * invB;
        if (q == 0 && n0 == 0) {
          db3 += dz[e];
          loss -= yy * logf(fmaxf(p, 1e-12f)) + (1.0f - yy) * logf(fmaxf(1.0f - p, 1e-12f));
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const int col = n0 + nt * 8 + 2 * q;
      float d[4];
#pragma unroll
      for (int e = 0; e < 4; e++) d[e] = __fmul_rn(dz[e >> 1] * s.w3[col + (e & 1)], g2[nt][e]);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        dw3[nt][e] += __fmaf_rn(dz[0], h2[nt][e], __fmul_rn(dz[1], h2[nt][e + 2]));
        db2[nt][e] += __fadd_rn(d[e], d[e + 2]);
      }
      *reinterpret_cast<__nv_bfloat162 *>(s.DA2 + (row0 + g) * SH + col) = __floats2bfloat162_rn(d[0], d[1]);
      *reinterpret_cast<__nv_bfloat162 *>(s.DA2 + (row0 + g + 8) * SH + col) = __floats2bfloat162_rn(d[2], d[3]);
    }
    __syncthreads();
    // dh1 = da2 W2, da1 = dh1 gelu'(a1)
    rows_times<NH>(s.DA2, row0, SH, s.W2T, n0, SH, a);
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const int col = n0 + nt * 8 + 2 * q;
#pragma unroll
      for (int e = 0; e < 4; e++) a[nt][e] = __fmul_rn(a[nt][e], g1[nt][e]);
#pragma unroll
      for (int e = 0; e < 2; e++) db1[nt][e] += __fadd_rn(a[nt][e], a[nt][e + 2]);
      *reinterpret_cast<__nv_bfloat162 *>(s.DA1 + (row0 + g) * SH + col) = __floats2bfloat162_rn(a[nt][0], a[nt][1]);
      *reinterpret_cast<__nv_bfloat162 *>(s.DA1 + (row0 + g + 8) * SH + col) = __floats2bfloat162_rn(a[nt][2], a[nt][3]);
    }
    outer_tile<4>(s.DA2, row0, s.H1, SH, n0, dW2);
    __syncthreads();
    outer_tile<9>(s.DA1, row0, s.X, SX, 72 * (warp >> 2), dW1);
    if (t + gridDim.x < ntiles) {
      __syncthreads();  // the next tile overwrites what these read
      load_tile(t + gridDim.x);
    }
  }
  // the block's gradient
  float *G = part + (size_t)blockIdx.x * PART;
#pragma unroll
  for (int nt = 0; nt < 9; nt++) {
    const int col = 72 * (warp >> 2) + nt * 8 + 2 * q;
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (col + (e & 1) < NIN) G[OFF_W1 + (row0 + g + 8 * (e >> 1)) * NIN + col + (e & 1)] = dW1[nt][e];
  }
#pragma unroll
  for (int nt = 0; nt < 4; nt++) {
    const int col = n0 + nt * 8 + 2 * q;
#pragma unroll
    for (int e = 0; e < 4; e++) G[OFF_W2 + (row0 + g + 8 * (e >> 1)) * NH + col + (e & 1)] = dW2[nt][e];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const float v[3] = {db1[nt][e], db2[nt][e], dw3[nt][e]};
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const float sum = rows_sum(v[j]);
        if (g == 0) s.cols[j][warp & 3][col + e] = sum;
      }
    }
  }
  db3 = rows_sum(db3);
  loss = rows_sum(loss);
  if (lane == 0 && n0 == 0) {
    s.last[0][warp] = db3;
    s.last[1][warp] = loss;
  }
  __syncthreads();
  if (tid < 3 * NH) {
    const int j = tid / NH, c = tid % NH;
    const float v = (s.cols[j][0][c] + s.cols[j][1][c]) + (s.cols[j][2][c] + s.cols[j][3][c]);
    G[(j == 0 ? OFF_B1 : j == 1 ? OFF_B2 : OFF_W3) + c] = v;
  } else if (tid < 3 * NH + 2) {
    const int j = tid - 3 * NH;
    G[j == 0 ? OFF_B3 : NPARAM] = (s.last[j][0] + s.last[j][1]) + (s.last[j][2] + s.last[j][3]);
  }
}

// the sum of the blocks' gradients (four lanes per entry, each every fourth block), into G and the
// loss sum into *loss; with STEP then AdamW (decoupled weight decay on W1, W2, w3; none on the
// biases) and the weights' BF16 copies
template <bool STEP>
__global__ void __launch_bounds__(256) mlp_update(const float *part, int nblocks,
                                                  float *__restrict__ G, float *__restrict__ loss,
                                                  float *__restrict__ P, float *__restrict__ M,
                                                  float *__restrict__ V, bf16 *__restrict__ W1,
                                                  bf16 *__restrict__ W2, bf16 *__restrict__ W2T,
                                                  float lr, float wd, float b1, float b2, float eps,
                                                  float c1, float c2) {
  const int i = (int)(blockIdx.x * 256 + threadIdx.x) >> 2, j = threadIdx.x & 3;
  float gr = 0.0f;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  if (i < PART) {
#pragma unroll 8
    for (int b = j; b < nblocks; b += 4) gr += part[(size_t)b * PART + i];
  }
  gr += __shfl_xor_sync(0xffffffffu, gr, 1);
  gr += __shfl_xor_sync(0xffffffffu, gr, 2);
  if (i >= PART || j) return;
  if (i == NPARAM) {
    *loss = gr;
    return;
  }
  if (!STEP) {
    G[i] = gr;
    return;
  }
  const float m = b1 * M[i] + (1.0f - b1) * gr;
  const float v = b2 * V[i] + (1.0f - b2) * gr * gr;
  M[i] = m;
  V[i] = v;
  const bool decay = (i < OFF_B1) || (i >= OFF_W2 && i < OFF_B2) || (i >= OFF_W3 && i < OFF_B3);
  float p = P[i];
  if (decay) p -= lr * wd * p;
  p -= lr * (m / c1) / (sqrtf(v / c2) + eps);
  P[i] = p;
  if (i < OFF_B1) {
    W1[(i / NIN) * KIN + i % NIN] = __float2bfloat16_rn(p);
  } else if (i >= OFF_W2 && i < OFF_B2) {
    const int r = (i - OFF_W2) / NH, k = (i - OFF_W2) % NH;
    const bf16 w = __float2bfloat16_rn(p);
    W2[i - OFF_W2] = w;
    W2T[k * NH + r] = w;
  }
}

}  // namespace

struct ffv_mlp {
  int device, nsm;
  cudaStream_t stream;
  float *d_P, *d_G, *d_M, *d_V, *d_norm, *d_loss;
  bf16 *d_W1, *d_W2, *d_W2T;
  int64_t t;  // AdamW step count
  // training: the blocks' gradients [nsm][PART] and the steps' losses, made by the first call
  float *d_part, *d_losses;
  int64_t cap_losses;
  // predict buffers
  int64_t cap;
  uint4 *d_R;  // records of the mesh's cells
  float *d_prob;
  // inference wait timeouts: mapped pinned word, set by the device, read by the host
  unsigned *h_err, *d_err;
};

namespace {
int mlp_cuda(cudaError_t e) { return e == cudaSuccess ? FFV_OK : FFV_ERR_CUDA; }
#define MCK(x)                                  \
  do {                                          \
    int _r = mlp_cuda(x);                       \
    if (_r != FFV_OK) return _r;                \
  } while (0)

int repack(ffv_mlp *m) {
  mlp_pack<<<64, 256, 0, m->stream>>>(m->d_P, m->d_W1, m->d_W2, m->d_W2T);
  return mlp_cuda(cudaGetLastError());
}

int ensure_cap(ffv_mlp *m, int64_t n) {
  if (m->cap >= n) return FFV_OK;
  cudaFree(m->d_R);
  cudaFree(m->d_prob);
  m->d_R = nullptr;
  m->d_prob = nullptr;
  m->cap = 0;
  if (cudaMalloc(&m->d_R, sizeof(uint4) * n) != cudaSuccess ||
      cudaMalloc(&m->d_prob, sizeof(float) * n) != cudaSuccess)
    return FFV_ERR_NOMEM;
  m->cap = n;
  return FFV_OK;
}

// the fused inference kernel over n rows: feature rows X (dm unused), or the stencil gather
// of the cells' records R on mesh dm (X unused); probabilities and/or marks out
int infer(ffv_mlp *m, bool gather, const ffv_dmesh &dm, const uint4 *R, const bf16 *X, int64_t n,
          float *prob, uint8_t *marks, float threshold, int accumulate, cudaStream_t st) {
  if (n <= 0) return FFV_OK;
  const int64_t tiles = (n + TC_ROWS - 1) / TC_ROWS;
  int64_t blocks = (int64_t)m->nsm * TC_CTAS_PER_SM;
  if (blocks > tiles) blocks = tiles;
  if (gather) {
    MCK(cudaFuncSetAttribute(mlp_infer_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM));
    mlp_infer_tc<true><<<(unsigned)blocks, TC_ROWS, TC_SMEM, st>>>(
        dm, R, nullptr, n, m->d_W1, m->d_W2, m->d_P, prob, marks, threshold, accumulate, m->d_err);
  } else {
    MCK(cudaFuncSetAttribute(mlp_infer_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM));
    mlp_infer_tc<false><<<(unsigned)blocks, TC_ROWS, TC_SMEM, st>>>(
        dm, nullptr, X, n, m->d_W1, m->d_W2, m->d_P, prob, marks, threshold, accumulate, m->d_err);
  }
  return mlp_cuda(cudaGetLastError());
}

// a timeout recorded by an inference kernel that has finished (the word is cleared)
int take_timeout(ffv_mlp *m) {
  const unsigned e = *(volatile unsigned *)m->h_err;
  if (!e) return FFV_OK;
  *(volatile unsigned *)m->h_err = 0u;
  return FFV_ERR_TIMEOUT;
}

// a launch that may begin before the stream's previous kernel has ended: the kernel itself waits
// for it (cudaGridDependencySynchronize) before it reads or writes what the two share
template <typename... Params, typename... Args>
int launch_early(ffv_mlp *m, void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t smem,
                 Args... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = m->stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return mlp_cuda(cudaLaunchKernelEx(&cfg, kernel, Params(args)...));
}

// the blocks' gradients of one batch into d_part; *blocks receives their number
int grad(ffv_mlp *m, const bf16 *X, const float *y, int64_t N, int64_t B, uint64_t seed,
         int64_t step, int *blocks) {
  if (!m->d_part && cudaMalloc(&m->d_part, sizeof(float) * PART * (size_t)m->nsm) != cudaSuccess) {
    m->d_part = nullptr;
    return FFV_ERR_NOMEM;
  }
  MCK(cudaFuncSetAttribute(mlp_grad_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem)));
  const int64_t tiles = (B + TG - 1) / TG;
  *blocks = (int)(tiles < m->nsm ? tiles : m->nsm);
  return launch_early(m, mlp_grad_tiles, (unsigned)*blocks, TG_TPB, sizeof(TrainSmem), X, y, N, B, seed, step,
                      (const bf16 *)m->d_W1, (const bf16 *)m->d_W2, (const bf16 *)m->d_W2T,
                      (const float *)m->d_P, m->d_part);
}
constexpr unsigned UPDATE_BLOCKS = (4 * PART + 255) / 256;

// seeded host initialisation: weights uniform in +-1/sqrt(fan_in), biases zero
void init_params(float *P, uint64_t seed) {
  uint64_t s = seed ? seed : 1;
  auto next = [&]() {
    s += 0x9E3779B97F4A7C15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  memset(P, 0, sizeof(float) * NPARAM);
  for (int i = 0; i < NH * NIN; i++) P[OFF_W1 + i] = (float)((2.0 * next() - 1.0) / sqrt((double)NIN));
  for (int i = 0; i < NH * NH; i++) P[OFF_W2 + i] = (float)((2.0 * next() - 1.0) / sqrt((double)NH));
  for (int i = 0; i < NH; i++) P[OFF_W3 + i] = (float)((2.0 * next() - 1.0) / sqrt((double)NH));
}
}  // namespace

// defined in ffv_api.cu
int ffv_ctx_view(ffv_ctx *ctx, int *device, cudaStream_t *st, ffv_dmesh *dm, const double **S,
                 const M5Consts **k, int *model, double *gamma0, double *pinf0);

namespace {
struct CtxView {
  int device, model;
  cudaStream_t st;
  ffv_dmesh dm;
  const double *S;
  const M5Consts *k;
  double gamma0, pinf0;
};
int view(ffv_ctx *ctx, CtxView &v) {
  return ffv_ctx_view(ctx, &v.device, &v.st, &v.dm, &v.S, &v.k, &v.model, &v.gamma0, &v.pinf0);
}
void launch_fields(const CtxView &v, const ffv_field_out &out) {
  if (v.model == 5) ffv_m5f_indicator_fields(v.dm.n, *v.k, v.S, out, v.st);
  else ffv_m0_indicator_fields(v.dm.n, v.gamma0, v.pinf0, v.S, out, v.st);
}
void launch_records(const CtxView &v, ffv_mlp *m) { launch_fields(v, {nullptr, m->d_R, m->d_norm}); }
}  // namespace

extern "C" {

int ffv_mlp_create(ffv_mlp **out, int device, uint64_t seed) {
  if (!out) return FFV_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return FFV_ERR_CUDA;
  MCK(cudaSetDevice(device));
  ffv_mlp *m = (ffv_mlp *)calloc(1, sizeof(ffv_mlp));
  if (!m) return FFV_ERR_NOMEM;
  m->device = device;
  if (cudaDeviceGetAttribute(&m->nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      m->nsm < 1)
    m->nsm = 1;
  float *h = (float *)malloc(sizeof(float) * NPARAM);
  const float norm[10] = {0, 0, 0, 0, 0, 1, 1, 1, 1, 1};
  int rc = FFV_OK;
  if (!h || cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&m->d_P, sizeof(float) * NPARAM) != cudaSuccess ||
      cudaMalloc(&m->d_G, sizeof(float) * NPARAM) != cudaSuccess ||
      cudaMalloc(&m->d_M, sizeof(float) * NPARAM) != cudaSuccess ||
      cudaMalloc(&m->d_V, sizeof(float) * NPARAM) != cudaSuccess ||
      cudaMalloc(&m->d_norm, sizeof(float) * 10) != cudaSuccess ||
      cudaMalloc(&m->d_loss, sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->d_W1, sizeof(bf16) * NH * KIN) != cudaSuccess ||
      cudaMalloc(&m->d_W2, sizeof(bf16) * NH * NH) != cudaSuccess ||
      cudaMalloc(&m->d_W2T, sizeof(bf16) * NH * NH) != cudaSuccess ||
      cudaHostAlloc(&m->h_err, sizeof(unsigned), cudaHostAllocMapped) != cudaSuccess ||
      cudaHostGetDevicePointer(&m->d_err, m->h_err, 0) != cudaSuccess) {
    rc = FFV_ERR_NOMEM;
  }
  if (rc == FFV_OK) *m->h_err = 0u;
  if (rc == FFV_OK) {
    init_params(h, seed);
    if (cudaMemcpy(m->d_P, h, sizeof(float) * NPARAM, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(m->d_norm, norm, sizeof(norm), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(m->d_M, 0, sizeof(float) * NPARAM) != cudaSuccess ||
        cudaMemset(m->d_V, 0, sizeof(float) * NPARAM) != cudaSuccess)
      rc = FFV_ERR_CUDA;
  }
  if (rc == FFV_OK) rc = repack(m);
  if (rc == FFV_OK && cudaStreamSynchronize(m->stream) != cudaSuccess) rc = FFV_ERR_CUDA;
  free(h);
  if (rc != FFV_OK) {
    ffv_mlp_destroy(m);
    return rc;
  }
  *out = m;
  return FFV_OK;
}

int ffv_mlp_destroy(ffv_mlp *m) {
  if (!m) return FFV_OK;
  cudaSetDevice(m->device);
  if (m->stream) cudaStreamSynchronize(m->stream);
  cudaFree(m->d_P);
  cudaFree(m->d_G);
  cudaFree(m->d_M);
  cudaFree(m->d_V);
  cudaFree(m->d_norm);
  cudaFree(m->d_loss);
  cudaFree(m->d_W1);
  cudaFree(m->d_W2);
  cudaFree(m->d_W2T);
  cudaFree(m->d_R);
  cudaFree(m->d_prob);
  cudaFree(m->d_part);
  cudaFree(m->d_losses);
  cudaFreeHost(m->h_err);
  if (m->stream) cudaStreamDestroy(m->stream);
  free(m);
  return FFV_OK;
}

int ffv_mlp_get_params(ffv_mlp *m, float *params) {
  if (!m || !params) return FFV_ERR_ARG;
  MCK(cudaSetDevice(m->device));
  MCK(cudaMemcpyAsync(params, m->d_P, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  return FFV_OK;
}

int ffv_mlp_set_params(ffv_mlp *m, const float *params) {
  if (!m || !params) return FFV_ERR_ARG;
  MCK(cudaSetDevice(m->device));
  MCK(cudaMemcpyAsync(m->d_P, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice, m->stream));
  MCK(cudaMemsetAsync(m->d_M, 0, sizeof(float) * NPARAM, m->stream));
  MCK(cudaMemsetAsync(m->d_V, 0, sizeof(float) * NPARAM, m->stream));
  m->t = 0;
  int rc = repack(m);
  if (rc != FFV_OK) return rc;
  MCK(cudaStreamSynchronize(m->stream));
  return FFV_OK;
}

int ffv_mlp_set_norm(ffv_mlp *m, const float *mean, const float *stdev) {
  if (!m || !mean || !stdev) return FFV_ERR_ARG;
  float h[10];
  for (int q = 0; q < 5; q++) {
    if (!(stdev[q] > 0.0f)) return FFV_ERR_ARG;
    h[q] = mean[q];
    h[5 + q] = stdev[q];
  }
  MCK(cudaSetDevice(m->device));
  MCK(cudaMemcpyAsync(m->d_norm, h, sizeof(h), cudaMemcpyHostToDevice, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  return FFV_OK;
}

int ffv_mlp_fields(ffv_ctx *ctx, float *F_dev) {
  CtxView v;
  int rc = view(ctx, v);
  if (rc != FFV_OK) return rc;
  if (!F_dev) return FFV_ERR_ARG;
  MCK(cudaSetDevice(v.device));
  launch_fields(v, {F_dev, nullptr, nullptr});
  MCK(cudaGetLastError());
  MCK(cudaStreamSynchronize(v.st));
  return FFV_OK;
}

int ffv_mlp_features(ffv_ctx *ctx, ffv_mlp *m, void *X_dev) {
  if (!m || !X_dev) return FFV_ERR_ARG;
  CtxView v;
  int rc = view(ctx, v);
  if (rc != FFV_OK) return rc;
  if (v.device != m->device) return FFV_ERR_ARG;
  MCK(cudaSetDevice(v.device));
  rc = ensure_cap(m, v.dm.n);
  if (rc != FFV_OK) return rc;
  launch_records(v, m);
  mlp_gather<<<(unsigned)((v.dm.n + 127) / 128), 128, 0, v.st>>>(v.dm, m->d_R, (bf16 *)X_dev);
  MCK(cudaGetLastError());
  MCK(cudaStreamSynchronize(v.st));
  return FFV_OK;
}

int ffv_mlp_forward(ffv_mlp *m, const void *X_dev, int64_t n, float *prob_dev) {
  if (!m || !X_dev || !prob_dev || n < 0) return FFV_ERR_ARG;
  MCK(cudaSetDevice(m->device));
  if (n == 0) return FFV_OK;
  int rc = infer(m, false, ffv_dmesh{}, nullptr, (const bf16 *)X_dev, n, prob_dev, nullptr, 0.0f, 0,
                 m->stream);
  if (rc != FFV_OK) return rc;
  MCK(cudaStreamSynchronize(m->stream));
  return take_timeout(m);
}

int ffv_mlp_predict(ffv_ctx *ctx, ffv_mlp *m, float *prob_host) {
  if (!m || !prob_host) return FFV_ERR_ARG;
  CtxView v;
  int rc = view(ctx, v);
  if (rc != FFV_OK) return rc;
  if (v.device != m->device) return FFV_ERR_ARG;
  MCK(cudaSetDevice(v.device));
  rc = ensure_cap(m, v.dm.n);
  if (rc != FFV_OK) return rc;
  launch_records(v, m);
  rc = infer(m, true, v.dm, m->d_R, nullptr, v.dm.n, m->d_prob, nullptr, 0.0f, 0, v.st);
  if (rc != FFV_OK) return rc;
  MCK(cudaMemcpyAsync(prob_host, m->d_prob, sizeof(float) * v.dm.n, cudaMemcpyDeviceToHost, v.st));
  MCK(cudaStreamSynchronize(v.st));
  return take_timeout(m);
}

int ffv_mlp_mark(ffv_ctx *ctx, ffv_mlp *m, float threshold, uint8_t *marks_dev,
                 int32_t accumulate) {
  if (!m || !marks_dev) return FFV_ERR_ARG;
  CtxView v;
  int rc = view(ctx, v);
  if (rc != FFV_OK) return rc;
  if (v.device != m->device) return FFV_ERR_ARG;
  MCK(cudaSetDevice(v.device));
  rc = ensure_cap(m, v.dm.n);
  if (rc != FFV_OK) return rc;
  // a timeout of an earlier call (this call is not waited for)
  rc = take_timeout(m);
  if (rc != FFV_OK) return rc;
  launch_records(v, m);
  return infer(m, true, v.dm, m->d_R, nullptr, v.dm.n, nullptr, marks_dev, threshold, accumulate, v.st);
}

int ffv_mlp_grad(ffv_mlp *m, const void *X_dev, const float *y_dev, int64_t B, float *grad_host,
                 float *loss_host) {
  if (!m || !X_dev || !y_dev || !grad_host || B < 1) return FFV_ERR_ARG;
  MCK(cudaSetDevice(m->device));
  int blocks;
  int rc = grad(m, (const bf16 *)X_dev, y_dev, B, B, 0, 0, &blocks);
  if (rc != FFV_OK) return rc;
  rc = launch_early(m, mlp_update<false>, UPDATE_BLOCKS, 256, 0, m->d_part, blocks, m->d_G, m->d_loss, m->d_P,
                    m->d_M, m->d_V, m->d_W1, m->d_W2, m->d_W2T, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f, 1.0f);
  if (rc != FFV_OK) return rc;
  MCK(cudaMemcpyAsync(grad_host, m->d_G, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, m->stream));
  float l = 0.0f;
  MCK(cudaMemcpyAsync(&l, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  if (loss_host) *loss_host = l / (float)B;
  return FFV_OK;
}

int ffv_mlp_train(ffv_mlp *m, const void *X_dev, const float *y_dev, int64_t N, int32_t batch,
                  int32_t steps, float lr, float wd, uint64_t seed, float *loss_host) {
  if (!m || !X_dev || !y_dev || N < 1 || batch < 1 || steps < 0 || seed == 0) return FFV_ERR_ARG;
  MCK(cudaSetDevice(m->device));
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  if (steps > m->cap_losses) {
    cudaFree(m->d_losses);
    m->d_losses = nullptr;
    m->cap_losses = 0;
    if (cudaMalloc(&m->d_losses, sizeof(float) * (size_t)steps) != cudaSuccess) return FFV_ERR_NOMEM;
    m->cap_losses = steps;
  }
  for (int32_t i = 0; i < steps; i++) {
    int blocks;
    int rc = grad(m, (const bf16 *)X_dev, y_dev, N, batch, seed, m->t, &blocks);
    if (rc != FFV_OK) return rc;
    m->t++;
    const float c1 = 1.0f - powf(b1, (float)m->t), c2 = 1.0f - powf(b2, (float)m->t);
    rc = launch_early(m, mlp_update<true>, UPDATE_BLOCKS, 256, 0, m->d_part, blocks, m->d_G, m->d_losses + i,
                      m->d_P, m->d_M, m->d_V, m->d_W1, m->d_W2, m->d_W2T, lr, wd, b1, b2, eps, c1, c2);
    if (rc != FFV_OK) return rc;
  }
  if (loss_host && steps > 0)
    MCK(cudaMemcpyAsync(loss_host, m->d_losses, sizeof(float) * (size_t)steps, cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  if (loss_host)
    for (int32_t i = 0; i < steps; i++) loss_host[i] /= (float)batch;
  return FFV_OK;
}

}  // extern "C"
