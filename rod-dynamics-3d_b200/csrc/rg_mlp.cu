// rg_mlp.cu - training and batch inference of the learned PSOR warm start.
//
// No reference counterpart: the reference warm-starts PSOR from a hash map of
// last-step impulses only (src/physics/nsc_contact.cpp:305-317, :646-654).
// The network (rg_mlp_dev.cuh) is trained on records of converged impulses
// that the plain PSOR path itself produces (rg_mlp_record), with this file's
// own kernels: one fused forward + loss + backward + weight-gradient kernel
// per minibatch on tensor cores (mma.sync m16n8k16, BF16 operands, FP32
// accumulation) and one kernel that sums the blocks' partial gradients and
// applies Adam to the FP32 master weights.  BF16 copies of the weights feed
// both training and the in-step inference.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "rg_internal.cuh"
#include "rg_mlp_dev.cuh"

namespace rg {

// ---------------------------------------------------------------------------
// Training: one fused kernel per minibatch.  A block takes tiles of kTrainRows
// rows and runs, for its rows, the forward pass (pre-activations Z kept in
// shared memory), the loss, the backward pass (dH = dZ W with W read
// transposed from shared memory, dZ = dH * silu'(Z)) and the block's share of
// the weight gradients dW = dZ^T H as block-level mma.sync products over the
// tile's rows.  A row group of 16 rows belongs to kTrainCols warps, each with
// its share of a layer's output columns; the BF16 activations pass between
// them through the dZ buffers, which are free during the forward pass.  Each
// block writes its partial gradient (and loss) to its own slice of a partial
// buffer, summing over its tiles in a fixed order; one reduction kernel then
// adds the slices in block order (deterministic) and applies Adam and the BF16
// weight copies.
//
// Bound by the instructions of a minibatch's 64 blocks (a tile's chain of
// products and its activations; the tensor pipe is idle most of the time).
// One warp a row group recomputed silu(Z) for every m-tile of a weight
// gradient and gathered transposed fragments by 16-bit loads: 157 us for 4096
// rows from a cold L2.  Now silu is taken once more, in place of Z, fragments
// come by ldmatrix, and four warps share a row group: 33 us; 65536 records, 4
// epochs: 7.43 -> 4.29 ms (two warps a row group 4.7).
// ---------------------------------------------------------------------------
constexpr int kTrainGroups = 4;                   // row groups of 16 rows
constexpr int kTrainCols = 4;                     // warps a row group
constexpr int kTrainWarps = kTrainGroups * kTrainCols;
constexpr int kTrainThreads = 32 * kTrainWarps;
constexpr int kTrainRows = 16 * kTrainGroups;     // 64 rows per tile
constexpr int kTrainNt = 16 / kTrainCols;         // n-tiles (8 columns) a warp
constexpr int kZLd = kMlpH + 4;                   // FP32 pre-activation rows (132)
constexpr int kHLd = 2 * kZLd;                    // BF16 activations in the place of Z
constexpr int kXLd = kW1Pad + 8;                  // BF16 input rows (24)
constexpr int kDyLd = 16;                         // BF16 output-gradient rows
constexpr int kGradParams = kOffInMean;           // trained parameters
constexpr int kTrainMaxBlocks = 296;

// Shared-memory carve-up of the training kernel (byte offsets, 16-aligned).
constexpr int kTsW2 = 0;
constexpr int kTsW3 = kTsW2 + 2 * kStageWh;
constexpr int kTsSmall = kTsW3 + 2 * kStageWh;                         // W1, W4, floats (MlpStage)
constexpr int kTsX = kTsSmall + ((kStageSmallBytes + 15) / 16) * 16;
constexpr int kTsZ = kTsX + 2 * kTrainRows * kXLd;                     // Z1, Z2, Z3
constexpr int kTsDzA = kTsZ + 3 * 4 * kTrainRows * kZLd;
constexpr int kTsDzB = kTsDzA + 2 * kTrainRows * kWhLd;
constexpr int kTsDy = kTsDzB + 2 * kTrainRows * kWhLd;
constexpr int kTsBias = kTsDy + 2 * kTrainRows * kDyLd;                // [row group][b1|b2|b3|b4(8)]
constexpr int kTsLoss = kTsBias + 4 * kTrainGroups * (3 * kMlpH + 8);
constexpr int kTrainSmem = kTsLoss + 16 * kTrainGroups;
static_assert(kTrainSmem <= 227 * 1024, "training kernel shared memory");
static_assert(kTsSmall % 16 == 0 && kTsX % 16 == 0 && kTsZ % 16 == 0 && kTsDzA % 16 == 0 && kTsDzB % 16 == 0 &&
                  kTsDy % 16 == 0 && kTsBias % 16 == 0,
              "16-byte aligned regions");

struct TrainSmem {
  __nv_bfloat16 *w2, *w3;  // [128][kWhLd]
  MlpStage st;             // W1 [128][kW1Ld], W4 [8][kWhLd], biases and scales
  __nv_bfloat16* x;        // [64][kXLd] normalised inputs (columns 0..7)
  float* z[3];             // [64][kZLd] pre-activations of layers 1..3; then [64][kHLd] BF16 activations
  __nv_bfloat16 *dza, *dzb;  // [64][kWhLd] BF16 dZ of two layers (forward: activations)
  __nv_bfloat16* dy;       // [64][kDyLd] BF16 dY (columns 3..15 zero)
  float* bias;             // [row group][3 * 128 + 8] bias-gradient partial sums
  float* loss;             // [row group]
};
__device__ inline TrainSmem train_smem(unsigned char* b) {
  TrainSmem s;
  s.w2 = reinterpret_cast<__nv_bfloat16*>(b + kTsW2);
  s.w3 = reinterpret_cast<__nv_bfloat16*>(b + kTsW3);
  s.st = mlp_stage_at(b + kTsSmall);
  s.x = reinterpret_cast<__nv_bfloat16*>(b + kTsX);
  for (int l = 0; l < 3; ++l) s.z[l] = reinterpret_cast<float*>(b + kTsZ) + (size_t)l * kTrainRows * kZLd;
  s.dza = reinterpret_cast<__nv_bfloat16*>(b + kTsDzA);
  s.dzb = reinterpret_cast<__nv_bfloat16*>(b + kTsDzB);
  s.dy = reinterpret_cast<__nv_bfloat16*>(b + kTsDy);
  s.bias = reinterpret_cast<float*>(b + kTsBias);
  s.loss = reinterpret_cast<float*>(b + kTsLoss);
  return s;
}

__device__ inline unsigned short bf16_bits(__nv_bfloat16 v) { return *reinterpret_cast<unsigned short*>(&v); }
// Two BF16 values from different rows packed into one fragment register.
__device__ inline unsigned pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (unsigned)bf16_bits(lo) | ((unsigned)bf16_bits(hi) << 16);
}
// Four (two) 8 x 8 BF16 matrices from shared memory, lane l giving the address
// of row l % 8 of matrix l / 8; trans: the transposed matrices' fragments.
__device__ inline void ldm4(const __nv_bfloat16* row, unsigned (&f)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3])
               : "r"((unsigned)__cvta_generic_to_shared(row)) : "memory");
}
__device__ inline void ldm4t(const __nv_bfloat16* row, unsigned (&f)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3])
               : "r"((unsigned)__cvta_generic_to_shared(row)) : "memory");
}
__device__ inline void ldm2t(const __nv_bfloat16* row, unsigned& f0, unsigned& f1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];"
               : "=r"(f0), "=r"(f1)
               : "r"((unsigned)__cvta_generic_to_shared(row)) : "memory");
}
// Barrier of the warps of one row group.
__device__ inline void group_sync(int rg) {
  asm volatile("bar.sync %0, %1;" ::"r"(rg + 1), "r"(32 * kTrainCols) : "memory");
}
__device__ inline float silu_grad(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}
// A warp's accumulator block (16 rows from lr0, columns from c0) as FP32 rows
// of Z, and its BF16 activations as rows of h.
__device__ inline void store_zh(float* z, __nv_bfloat16* h, int lr0, int c0, const float (&c)[kTrainNt][4], int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < kTrainNt; ++nt) {
    const int col = c0 + nt * 8 + 2 * t;
    *reinterpret_cast<float2*>(&z[(lr0 + g) * kZLd + col]) = make_float2(c[nt][0], c[nt][1]);
    *reinterpret_cast<float2*>(&z[(lr0 + g + 8) * kZLd + col]) = make_float2(c[nt][2], c[nt][3]);
    *reinterpret_cast<unsigned*>(&h[(lr0 + g) * kWhLd + col]) = pack_bf16(silu(c[nt][0]), silu(c[nt][1]));
    *reinterpret_cast<unsigned*>(&h[(lr0 + g + 8) * kWhLd + col]) = pack_bf16(silu(c[nt][2]), silu(c[nt][3]));
  }
}
// A fragment of rows lr0.. of x (BF16 [64][kWhLd]), k-tile kt.
__device__ inline void load_a(const __nv_bfloat16* x, int lr0, int kt, int lane, unsigned (&a)[4]) {
  ldm4(x + (lr0 + (lane & 15)) * kWhLd + kt * 16 + (lane >> 4) * 8, a);
}

__device__ inline float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Partial gradient slice of a block: '=' on its first tile, '+=' after.
__device__ inline void part_put(float* p, int i, float v, bool first) { p[i] = first ? v : p[i] + v; }

// Block-level weight gradient dW[o][i] = Σ_r dZ[r][o] H[r][i] over the
// tile's 64 rows: output rows o in m-tiles [0, mtiles), input columns in
// ngroups groups of NTN n-tiles; the warps take the (m-tile, group) products
// in turn.  dZ, H: BF16 rows of leading dimensions ldz and ldh.  Rows
// o < nrows and columns i < ncols go to part[off + o * ncols + i].
template <int NTN>
__device__ inline void block_dw(const __nv_bfloat16* dz, int ldz, int mtiles, int nrows, const __nv_bfloat16* h,
                                int ldh, int ngroups, int ncols, float* part, int off, bool first, int warp,
                                int lane) {
  const int g = lane >> 2, t = lane & 3;
  for (int u = warp; u < mtiles * ngroups; u += kTrainWarps) {
    const int m0 = (u / ngroups) * 16, n0 = (u % ngroups) * NTN * 8;
    float c[NTN][4];
#pragma unroll
    for (int j = 0; j < NTN; ++j) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < kTrainRows / 16; ++ks) {
      unsigned a[4];
      ldm4t(dz + (ks * 16 + (lane & 7) + (lane >> 4) * 8) * ldz + m0 + ((lane >> 3) & 1) * 8, a);
      const __nv_bfloat16* hr = h + (ks * 16 + (lane & 15)) * ldh + n0;
      if constexpr (NTN == 1) {
        unsigned b0, b1;
        ldm2t(hr, b0, b1);
        mma_bf16(c[0], a[0], a[1], a[2], a[3], b0, b1);
      } else {
#pragma unroll
        for (int j = 0; j < NTN; j += 2) {
          unsigned b[4];
          ldm4t(hr + j * 8 + (lane >> 4) * 8, b);
          mma_bf16(c[j], a[0], a[1], a[2], a[3], b[0], b[1]);
          mma_bf16(c[j + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NTN; ++j) {
      const int col = n0 + j * 8 + 2 * t;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int o = m0 + g + (e >= 2 ? 8 : 0), i = col + (e & 1);
        if (o < nrows && i < ncols) part_put(part, off + o * ncols + i, c[j][e], first);
      }
    }
  }
}

// Column sums over a warp's 16 rows of its FP32 fragment block, added to
// sums[c0..] ('=' on the block's first tile); lanes with g = 0 write.
__device__ inline void warp_colsum_acc(const float (&c)[kTrainNt][4], float* sums, int c0, int lane, bool first) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < kTrainNt; ++nt) {
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      float v = c[nt][cc] + c[nt][2 + cc];
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if (g == 0) {
        float* s = &sums[c0 + nt * 8 + 2 * t + cc];
        *s = first ? v : *s + v;
      }
    }
  }
}

// dZ = dH * silu'(Z) in place on the accumulator block (Z rows lr0..), its
// BF16 copy into dzs, and, once the whole row group has read its Z, the BF16
// activations silu(Z) in Z's place.
__device__ inline void dz_from_dh(float (&c)[kTrainNt][4], float* z, __nv_bfloat16* dzs, int rg, int c0, int lane) {
  const int g = lane >> 2, t = lane & 3, lr0 = 16 * rg;
  unsigned h[kTrainNt][2];
#pragma unroll
  for (int nt = 0; nt < kTrainNt; ++nt) {
    const int col = c0 + nt * 8 + 2 * t;
    const float2 z0 = *reinterpret_cast<const float2*>(&z[(lr0 + g) * kZLd + col]);
    const float2 z1 = *reinterpret_cast<const float2*>(&z[(lr0 + g + 8) * kZLd + col]);
    c[nt][0] *= silu_grad(z0.x);
    c[nt][1] *= silu_grad(z0.y);
    c[nt][2] *= silu_grad(z1.x);
    c[nt][3] *= silu_grad(z1.y);
    h[nt][0] = pack_bf16(silu(z0.x), silu(z0.y));
    h[nt][1] = pack_bf16(silu(z1.x), silu(z1.y));
    *reinterpret_cast<unsigned*>(&dzs[(lr0 + g) * kWhLd + col]) = pack_bf16(c[nt][0], c[nt][1]);
    *reinterpret_cast<unsigned*>(&dzs[(lr0 + g + 8) * kWhLd + col]) = pack_bf16(c[nt][2], c[nt][3]);
  }
  group_sync(rg);
  __nv_bfloat16* hz = reinterpret_cast<__nv_bfloat16*>(z);
#pragma unroll
  for (int nt = 0; nt < kTrainNt; ++nt) {
    const int col = c0 + nt * 8 + 2 * t;
    *reinterpret_cast<unsigned*>(&hz[(lr0 + g) * kHLd + col]) = h[nt][0];
    *reinterpret_cast<unsigned*>(&hz[(lr0 + g + 8) * kHLd + col]) = h[nt][1];
  }
}
// dH = dZ W for a warp's 16 rows and columns c0..: dZ A fragments from dzs
// (BF16 rows lr0..), W staged [out][kWhLd].
__device__ inline void dh_product(const __nv_bfloat16* dzs, int lr0, const __nv_bfloat16* W, int c0,
                                  float (&c)[kTrainNt][4], int lane) {
#pragma unroll
  for (int nt = 0; nt < kTrainNt; ++nt) c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.0f;
#pragma unroll
  for (int kt = 0; kt < 8; ++kt) {
    unsigned a[4];
    load_a(dzs, lr0, kt, lane, a);
#pragma unroll
    for (int nt = 0; nt < kTrainNt; nt += 2) {
      unsigned b[4];  // k = out, n = in: the transposed fragments of two n-tiles
      ldm4t(W + (kt * 16 + (lane & 15)) * kWhLd + c0 + nt * 8 + (lane >> 4) * 8, b);
      mma_bf16(c[nt], a[0], a[1], a[2], a[3], b[0], b[1]);
      mma_bf16(c[nt + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
    }
  }
}
// Forward through one hidden layer from BF16 rows h (lr0..), columns c0..,
// with W staged [out][kWhLd]: c = h W^T + bias (FP32).
__device__ inline void fwd_product(const __nv_bfloat16* h, int lr0, const __nv_bfloat16* W, const float* bias, int c0,
                                   float (&c)[kTrainNt][4], int lane) {
  const int t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < kTrainNt; ++nt) {
    const float bl = bias[c0 + nt * 8 + 2 * t], bh = bias[c0 + nt * 8 + 2 * t + 1];
    c[nt][0] = bl; c[nt][1] = bh; c[nt][2] = bl; c[nt][3] = bh;
  }
#pragma unroll
  for (int kt = 0; kt < 8; ++kt) {
    unsigned a[4];
    load_a(h, lr0, kt, lane, a);
#pragma unroll
    for (int nt = 0; nt < kTrainNt; nt += 2) {
      unsigned b[4];  // two n-tiles
      ldm4(W + (c0 + nt * 8 + (lane & 7) + (lane >> 4) * 8) * kWhLd + kt * 16 + ((lane >> 3) & 1) * 8, b);
      mma_bf16(c[nt], a[0], a[1], a[2], a[3], b[0], b[1]);
      mma_bf16(c[nt + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
    }
  }
}

// One minibatch: rows [0, n) of feat/tgt (row-major [n][8] / [n][3]),
// gathered by idx when given.  Block b handles tiles b, b + gridDim.x, ...
// and leaves its partial gradient in part[b * kGradParams ...] and its
// partial loss (Σ squared error) in loss_part[b].
__global__ void __launch_bounds__(kTrainThreads, 1)
    k_mlp_train_fb(MlpDev M, const float* feat, const float* tgt, const int* idx, int n, float* part,
                   float* loss_part) {
  extern __shared__ __align__(16) unsigned char tsm[];
  const TrainSmem S = train_smem(tsm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  stage_bf16(S.w2, kWhLd, M.w2, kMlpH, kMlpH);
  stage_bf16(S.w3, kWhLd, M.w3, kMlpH, kMlpH);
  stage_small(S.st, M);
  stage_wait();
  __syncthreads();
  const MlpSmall q = S.st.small();
  float* mypart = part + (size_t)blockIdx.x * kGradParams;
  const int ntiles = (n + kTrainRows - 1) / kTrainRows;
  const float inv_n3 = 1.0f / (float)(n * kMlpOut);
  const int rg = warp & (kTrainGroups - 1), lr0 = 16 * rg;           // row group
  const int cg = warp / kTrainGroups, c0 = cg * kTrainNt * 8;        // column group
  float* bsum = S.bias + rg * (3 * kMlpH + 8);
  float lsum = 0.0f;
  bool first = true;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, first = false) {
    const int row0 = tile * kTrainRows;
    // ---- forward (rows lr0..lr0+15 of the tile, columns c0..) ----
    unsigned x0, x1;
    {
      float v[4];
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int lr = lr0 + g + 8 * rr, r = row0 + lr;
        const int rid = r < n ? (idx ? idx[r] : r) : 0;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const int k = 2 * t + cc;
          v[rr * 2 + cc] = r < n ? (feat[(size_t)rid * kMlpIn + k] - q.in_mean[k]) * q.in_scale[k] : 0.0f;
        }
        if (cg == 0) *reinterpret_cast<unsigned*>(&S.x[(size_t)lr * kXLd + 2 * t]) = pack_bf16(v[rr * 2], v[rr * 2 + 1]);
      }
      x0 = pack_bf16(v[0], v[1]);
      x1 = pack_bf16(v[2], v[3]);
    }
    float c[kTrainNt][4];
#pragma unroll
    for (int nt = 0; nt < kTrainNt; ++nt) {
      const int col = c0 + nt * 8 + 2 * t;
      const float bl = q.b1[col], bh = q.b1[col + 1];
      c[nt][0] = bl; c[nt][1] = bh; c[nt][2] = bl; c[nt][3] = bh;
      unsigned b0, b1;
      load_b(S.st.w1, kW1Ld, cg * kTrainNt + nt, 0, lane, b0, b1);
      mma_bf16(c[nt], x0, x1, 0u, 0u, b0, b1);
    }
    store_zh(S.z[0], S.dza, lr0, c0, c, lane);
    group_sync(rg);
    fwd_product(S.dza, lr0, S.w2, q.b2, c0, c, lane);
    store_zh(S.z[1], S.dzb, lr0, c0, c, lane);
    group_sync(rg);  // (and no warp of the group reads dza any more)
    fwd_product(S.dzb, lr0, S.w3, q.b3, c0, c, lane);
    store_zh(S.z[2], S.dza, lr0, c0, c, lane);
    group_sync(rg);
    // output layer, loss and dY (outputs 2t, 2t + 1 of rows g, g + 8), by every
    // warp of the row group; the first one keeps them
    float dy[4];
    {
      float y[4];
      const float bl = 2 * t < kMlpOut ? q.b4[2 * t] : 0.0f, bh = 2 * t + 1 < kMlpOut ? q.b4[2 * t + 1] : 0.0f;
      y[0] = bl; y[1] = bh; y[2] = bl; y[3] = bh;
#pragma unroll
      for (int kt = 0; kt < 8; ++kt) {
        unsigned a[4], b0, b1;
        load_a(S.dza, lr0, kt, lane, a);
        load_b(S.st.w4, kWhLd, 0, kt, lane, b0, b1);
        mma_bf16(y, a[0], a[1], a[2], a[3], b0, b1);
      }
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int lr = lr0 + g + 8 * rr, r = row0 + lr;
        const int rid = r < n ? (idx ? idx[r] : r) : 0;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const int o = 2 * t + cc;
          float d = 0.0f;
          if (o < kMlpOut && r < n) {
            const float tn = (tgt[(size_t)rid * kMlpOut + o] - feat[(size_t)rid * kMlpIn + 4 + o]) / q.out_scale[o];
            const float diff = y[rr * 2 + cc] - tn;
            if (cg == 0) lsum += diff * diff;
            d = 2.0f * diff * inv_n3;
          }
          dy[rr * 2 + cc] = d;
        }
        if (cg == 0) {
          *reinterpret_cast<unsigned*>(&S.dy[(size_t)lr * kDyLd + 2 * t]) = pack_bf16(dy[rr * 2], dy[rr * 2 + 1]);
          *reinterpret_cast<unsigned*>(&S.dy[(size_t)lr * kDyLd + 8 + 2 * t]) = 0u;
        }
      }
    }
    // ---- backward through the output layer: db4, dH3 = dY W4 ----
    {
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        float v = dy[cc] + dy[2 + cc];
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (g == 0 && cg == 0) {
          float* s = &bsum[3 * kMlpH + 2 * t + cc];
          *s = first ? v : *s + v;
        }
      }
      const unsigned ya0 = pack_bf16(dy[0], dy[1]), ya1 = pack_bf16(dy[2], dy[3]);
#pragma unroll
      for (int nt = 0; nt < kTrainNt; ++nt) {
        c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.0f;
        const int nn = c0 + nt * 8 + g;
        const unsigned b0 = pack2(S.st.w4[(size_t)(2 * t) * kWhLd + nn], S.st.w4[(size_t)(2 * t + 1) * kWhLd + nn]);
        mma_bf16(c[nt], ya0, ya1, 0u, 0u, b0, 0u);
      }
    }
    group_sync(rg);  // every warp of the group has read H3 in dza
    // layer 3: dZ3 -> dza, db3; dH2 = dZ3 W3
    dz_from_dh(c, S.z[2], S.dza, rg, c0, lane);
    warp_colsum_acc(c, bsum + 2 * kMlpH, c0, lane, first);
    dh_product(S.dza, lr0, S.w3, c0, c, lane);
    // layer 2: dZ2 -> dzb, db2
    dz_from_dh(c, S.z[1], S.dzb, rg, c0, lane);
    warp_colsum_acc(c, bsum + kMlpH, c0, lane, first);
    __syncthreads();  // every warp's dZ3, dZ2, dY, H3 and H2 are in shared memory
    const __nv_bfloat16* h1 = reinterpret_cast<const __nv_bfloat16*>(S.z[0]);
    const __nv_bfloat16* h2 = reinterpret_cast<const __nv_bfloat16*>(S.z[1]);
    const __nv_bfloat16* h3 = reinterpret_cast<const __nv_bfloat16*>(S.z[2]);
    block_dw<8>(S.dza, kWhLd, kMlpH / 16, kMlpH, h2, kHLd, 2, kMlpH, mypart, kOffW3, first, warp, lane);
    block_dw<1>(S.dy, kDyLd, 1, kMlpOut, h3, kHLd, 16, kMlpH, mypart, kOffW4, first, warp, lane);
    __syncthreads();  // dza is free again
    // layer 1: dH1 = dZ2 W2, dZ1 -> dza, db1
    dh_product(S.dzb, lr0, S.w2, c0, c, lane);
    dz_from_dh(c, S.z[0], S.dza, rg, c0, lane);
    warp_colsum_acc(c, bsum, c0, lane, first);
    __syncthreads();
    block_dw<8>(S.dzb, kWhLd, kMlpH / 16, kMlpH, h1, kHLd, 2, kMlpH, mypart, kOffW2, first, warp, lane);
    block_dw<1>(S.dza, kWhLd, kMlpH / 16, kMlpH, S.x, kXLd, 1, kMlpIn, mypart, kOffW1, first, warp, lane);
    __syncthreads();  // shared tiles are reused by the next tile
  }
  // bias gradients and loss: sum the row groups' partial sums in order
  lsum = warp_sum_f(lsum);
  if (lane == 0 && cg == 0) S.loss[rg] = lsum;
  __syncthreads();
  const bool any = blockIdx.x < ntiles;
  for (int i = threadIdx.x; i < 3 * kMlpH + kMlpOut; i += blockDim.x) {
    float v = 0.0f;
    if (any)
      for (int w = 0; w < kTrainGroups; ++w) v += S.bias[w * (3 * kMlpH + 8) + i];
    const int off = i < kMlpH ? kOffB1 + i : i < 2 * kMlpH ? kOffB2 + i - kMlpH
                  : i < 3 * kMlpH ? kOffB3 + i - 2 * kMlpH : kOffB4 + i - 3 * kMlpH;
    mypart[off] = v;
  }
  if (threadIdx.x == 0) {
    float l = 0.0f;
    for (int w = 0; w < kTrainGroups; ++w) l += S.loss[w];
    loss_part[blockIdx.x] = any ? l : 0.0f;
  }
  if (!any) {  // a block without a tile contributes zero weight gradients
    for (int i = threadIdx.x; i < kGradParams; i += blockDim.x) {
      const bool bias = (i >= kOffB1 && i < kOffW2) || (i >= kOffB2 && i < kOffW3) || (i >= kOffB3 && i < kOffW4) ||
                        i >= kOffB4;
      if (!bias) mypart[i] = 0.0f;
    }
  }
}

// g_i = Σ_b part[b][i] in block order (deterministic), i < kGradParams.
__device__ inline float grad_sum(const float* part, int nblk, int i) {
  float g = 0.0f;
#pragma unroll 16
  for (int b = 0; b < nblk; ++b) g += part[(size_t)b * kGradParams + i];
  return g;
}
__global__ void k_mlp_grad_sum(const float* part, int nblk, float* G) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kGradParams; i += gridDim.x * blockDim.x)
    G[i] = grad_sum(part, nblk, i);
}
// Adam on the trained parameters from the summed partial gradients, then
// the BF16 weight copies the next minibatch and the in-step inference read
// (their padding stays zero from the full copy).
__global__ void k_mlp_adam(const float* part, int nblk, float* P, float* m, float* v, float lr, float b1, float b2,
                           float eps, float bc1, float bc2, __nv_bfloat16* w1, __nv_bfloat16* w2,
                           __nv_bfloat16* w3, __nv_bfloat16* w4) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kGradParams; i += gridDim.x * blockDim.x) {
    const float g = grad_sum(part, nblk, i);
    const float mi = b1 * m[i] + (1.0f - b1) * g;
    const float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float p = P[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    P[i] = p;
    const __nv_bfloat16 pb = __float2bfloat16(p);
    if (i < kOffB1) {
      w1[(i / kMlpIn) * kW1Pad + i % kMlpIn] = pb;
    } else if (i >= kOffW2 && i < kOffB2) {
      w2[i - kOffW2] = pb;
    } else if (i >= kOffW3 && i < kOffB3) {
      w3[i - kOffW3] = pb;
    } else if (i >= kOffW4 && i < kOffB4) {
      w4[i - kOffW4] = pb;
    }
  }
}

// BF16 padded weight copies from the FP32 parameter vector.
__global__ void k_weights_bf16(const float* P, __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3,
                               __nv_bfloat16* w4) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, str = gridDim.x * blockDim.x;
  for (int e = tid; e < kMlpH * kW1Pad; e += str) {
    int n = e / kW1Pad, k = e % kW1Pad;
    w1[e] = __float2bfloat16(k < kMlpIn ? P[kOffW1 + n * kMlpIn + k] : 0.0f);
  }
  for (int e = tid; e < kMlpH * kMlpH; e += str) {
    w2[e] = __float2bfloat16(P[kOffW2 + e]);
    w3[e] = __float2bfloat16(P[kOffW3 + e]);
  }
  for (int e = tid; e < kW4Pad * kMlpH; e += str) {
    int n = e / kMlpH;
    w4[e] = __float2bfloat16(n < kMlpOut ? P[kOffW4 + e] : 0.0f);
  }
}
// Batch inference with the in-step warp routine (feature-major input):
// predicted impulse = previous impulse (features 4-6) + network output.
__global__ void k_mlp_infer(MlpDev M, const float* featT, int n, float* outT) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int row0 = warp * 16; row0 < n; row0 += nw * 16) {
    mlp_warp(M, featT, n, row0, n, outT, lane);
    __syncwarp();
    if (lane < 16 && row0 + lane < n)
      for (int o = 0; o < kMlpOut; ++o) outT[(size_t)o * n + row0 + lane] += featT[(size_t)(4 + o) * n + row0 + lane];
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Host-side network state.
// ---------------------------------------------------------------------------
struct MlpHost {
  float* P = nullptr;              // FP32 parameters (kMlpParams)
  __nv_bfloat16* wb = nullptr;     // w1 | w2 | w3 | w4 (padded)
  // training workspace
  float *part = nullptr, *loss = nullptr;  // per-block partial gradients / losses
  float *G = nullptr, *Am = nullptr, *Av = nullptr;
  int* idx = nullptr;              // minibatch order of an epoch (n)
  size_t nidx = 0;
  float *feat = nullptr, *tgt = nullptr;  // dataset on the device
  size_t nfeat = 0;
};

static MlpHost& host_of(rg_system* s) { return *reinterpret_cast<MlpHost*>(s->mlp_host); }

static cudaError_t ensure_net(rg_system* s) {
  if (!s->mlp_host) s->mlp_host = new MlpHost();
  MlpHost& H = host_of(s);
  cudaError_t e = cudaSuccess;
  if (!H.P) {
    if ((e = cudaMalloc(&H.P, sizeof(float) * kMlpParams))) return e;
    if ((e = cudaMemset(H.P, 0, sizeof(float) * kMlpParams))) return e;
    size_t nb = kMlpH * kW1Pad + 2 * kMlpH * kMlpH + kW4Pad * kMlpH;
    if ((e = cudaMalloc(&H.wb, sizeof(__nv_bfloat16) * nb))) return e;
  }
  return e;
}

MlpDev mlp_dev(rg_system* s) {
  MlpHost& H = host_of(s);
  MlpDev M;
  M.w1 = H.wb;
  M.w2 = M.w1 + kMlpH * kW1Pad;
  M.w3 = M.w2 + kMlpH * kMlpH;
  M.w4 = M.w3 + kMlpH * kMlpH;
  M.p = H.P;
  return M;
}

static void refresh_bf16(rg_system* s) {
  MlpHost& H = host_of(s);
  MlpDev M = mlp_dev(s);
  RGL k_weights_bf16<<<64, 256, 0, s->stream>>>(H.P, const_cast<__nv_bfloat16*>(M.w1),
                                                 const_cast<__nv_bfloat16*>(M.w2),
                                                 const_cast<__nv_bfloat16*>(M.w3),
                                                 const_cast<__nv_bfloat16*>(M.w4));
}

static cudaError_t ensure_workspace(rg_system* s) {
  MlpHost& H = host_of(s);
  if (H.part) return cudaSuccess;
  cudaError_t e;
  if ((e = cudaMalloc(&H.part, sizeof(float) * (size_t)kTrainMaxBlocks * kGradParams))) return e;
  if ((e = cudaMalloc(&H.loss, sizeof(float) * kTrainMaxBlocks))) return e;
  if ((e = cudaMalloc(&H.G, sizeof(float) * kMlpParams))) return e;
  if ((e = cudaMalloc(&H.Am, sizeof(float) * kMlpParams))) return e;
  if ((e = cudaMalloc(&H.Av, sizeof(float) * kMlpParams))) return e;
  return cudaFuncSetAttribute(k_mlp_train_fb, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem);
}

// Forward + backward of rows [0, n) (feat/tgt row-major, gathered by idx
// when given) into the per-block partial gradients and losses; returns the
// number of blocks (partial slices) used.
static int forward_backward(rg_system* s, const float* feat, const float* tgt, const int* idx, int n) {
  MlpHost& H = host_of(s);
  const int tiles = (n + kTrainRows - 1) / kTrainRows;
  const int nblk = tiles < kTrainMaxBlocks ? tiles : kTrainMaxBlocks;
  RGL k_mlp_train_fb<<<nblk, kTrainThreads, kTrainSmem, s->stream>>>(mlp_dev(s), feat, tgt, idx, n, H.part,
                                                                     H.loss);
  return nblk;
}

static double read_loss(rg_system* s, int n, int nblk) {
  MlpHost& H = host_of(s);
  std::vector<float> part(nblk);
  cudaMemcpyAsync(part.data(), H.loss, sizeof(float) * nblk, cudaMemcpyDeviceToHost, s->stream);
  cudaStreamSynchronize(s->stream);
  double l = 0;
  for (int i = 0; i < nblk; ++i) l += part[i];
  return l / ((double)n * kMlpOut);
}

static void init_params(std::vector<float>& P, const float* feat, const float* tgt, size_t n, uint64_t seed) {
  P.assign(kMlpParams, 0.0f);
  for (int k = 0; k < kMlpIn; ++k) {
    double m = 0, v = 0;
    for (size_t i = 0; i < n; ++i) m += feat[i * kMlpIn + k];
    m /= (double)n;
    for (size_t i = 0; i < n; ++i) { double d = feat[i * kMlpIn + k] - m; v += d * d; }
    double sd = std::sqrt(v / (double)n);
    P[kOffInMean + k] = (float)m;
    P[kOffInScale + k] = sd > 1e-30 ? (float)(1.0 / sd) : 1.0f;
  }
  for (int o = 0; o < kMlpOut; ++o) {
    double v = 0;
    for (size_t i = 0; i < n; ++i) {
      double d = (double)tgt[i * kMlpOut + o] - feat[i * kMlpIn + 4 + o];
      v += d * d;
    }
    double rms = std::sqrt(v / (double)n);
    P[kOffOutScale + o] = rms > 1e-30 ? (float)rms : 1.0f;
  }
  std::mt19937_64 rng(seed);
  auto fill = [&](int off, int fan_in, int count) {
    double lim = std::sqrt(6.0 / fan_in);
    std::uniform_real_distribution<double> U(-lim, lim);
    for (int i = 0; i < count; ++i) P[off + i] = (float)U(rng);
  };
  fill(kOffW1, kMlpIn, kMlpH * kMlpIn);
  fill(kOffW2, kMlpH, kMlpH * kMlpH);
  fill(kOffW3, kMlpH, kMlpH * kMlpH);
  fill(kOffW4, kMlpH, kMlpOut * kMlpH);
  for (int i = 0; i < kMlpOut * kMlpH; ++i) P[kOffW4 + i] *= 0.1f;
}

void mlp_free(rg_system* s) {
  if (!s->mlp_host) return;
  MlpHost& H = host_of(s);
  cudaFree(H.P); cudaFree(H.wb);
  cudaFree(H.part); cudaFree(H.loss); cudaFree(H.G); cudaFree(H.Am); cudaFree(H.Av);
  cudaFree(H.idx); cudaFree(H.feat); cudaFree(H.tgt);
  delete &H;
  s->mlp_host = nullptr;
}

}  // namespace rg

using namespace rg;

extern "C" {

size_t rg_mlp_param_count(void) { return (size_t)kMlpParams; }

int rg_mlp_set_params(rg_system* s, const float* params, size_t n) {
  if (!s || !params || n != (size_t)kMlpParams) return RG_ERR_ARG;
  if (ensure_net(s)) return RG_ERR_CUDA;
  // on the system's stream: a default-stream copy from pageable memory may
  // still be on its way when the conversion starts on the non-blocking stream
  cudaMemcpyAsync(host_of(s).P, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, s->stream);
  refresh_bf16(s);
  if (cudaStreamSynchronize(s->stream)) return RG_ERR_CUDA;
  s->mlp_ready = true;
  return RG_OK;
}

int rg_mlp_get_params(const rg_system* s, float* params, size_t n) {
  if (!s || !params || n != (size_t)kMlpParams || !s->mlp_host) return RG_ERR_ARG;
  cudaMemcpy(params, reinterpret_cast<MlpHost*>(s->mlp_host)->P, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost);
  return RG_OK;
}

int rg_mlp_record(rg_system* s, int enable, size_t cap) {
  if (!s) return RG_ERR_ARG;
  if (!enable) {
    s->recording = false;
    return RG_OK;
  }
  if (cap == 0 || cap > (size_t)1 << 30) return RG_ERR_ARG;
  cudaFree(s->d_rec_x);
  cudaFree(s->d_rec_y);
  if (cudaMalloc(&s->d_rec_x, sizeof(float) * kMlpIn * cap) || cudaMalloc(&s->d_rec_y, sizeof(float) * kMlpOut * cap))
    return RG_ERR_CUDA;
  s->rec_cap = (int)cap;
  s->recording = true;
  int zero = 0;
  cudaMemcpy(&s->d_ctl->rec_n, &zero, sizeof(int), cudaMemcpyHostToDevice);
  return RG_OK;
}

int rg_mlp_records(const rg_system* s, float* features, float* targets, size_t cap, size_t* n) {
  if (!s || !n) return RG_ERR_ARG;
  int rn = 0;
  cudaMemcpy(&rn, &s->d_ctl->rec_n, sizeof(int), cudaMemcpyDeviceToHost);
  if (rn > s->rec_cap) rn = s->rec_cap;
  *n = (size_t)rn;
  size_t m = cap < (size_t)rn ? cap : (size_t)rn;
  if (m && features) cudaMemcpy(features, s->d_rec_x, sizeof(float) * kMlpIn * m, cudaMemcpyDeviceToHost);
  if (m && targets) cudaMemcpy(targets, s->d_rec_y, sizeof(float) * kMlpOut * m, cudaMemcpyDeviceToHost);
  return (size_t)rn > cap ? RG_ERR_CAPACITY : RG_OK;
}

// Loss and gradient (parameter layout) of one batch at the current weights.
int rg_mlp_grad(rg_system* s, const float* features, const float* targets, size_t n, float* grad, float* loss) {
  if (!s || !features || !targets || n == 0 || n > (1u << 24)) return RG_ERR_ARG;
  if (!s->mlp_host || !reinterpret_cast<MlpHost*>(s->mlp_host)->P) return RG_ERR_STATE;
  MlpHost& H = host_of(s);
  if (ensure_workspace(s)) return RG_ERR_CUDA;
  float *df = nullptr, *dt = nullptr;
  if (cudaMalloc(&df, sizeof(float) * kMlpIn * n) || cudaMalloc(&dt, sizeof(float) * kMlpOut * n)) return RG_ERR_CUDA;
  cudaMemcpyAsync(df, features, sizeof(float) * kMlpIn * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(dt, targets, sizeof(float) * kMlpOut * n, cudaMemcpyHostToDevice, s->stream);
  const int nblk = forward_backward(s, df, dt, nullptr, (int)n);
  cudaMemsetAsync(H.G, 0, sizeof(float) * kMlpParams, s->stream);
  RGL k_mlp_grad_sum<<<grid_for(kGradParams, 256), 256, 0, s->stream>>>(H.part, nblk, H.G);
  double l = read_loss(s, (int)n, nblk);
  if (grad) cudaMemcpy(grad, H.G, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost);
  if (loss) *loss = (float)l;
  cudaFree(df);
  cudaFree(dt);
  return cudaGetLastError() == cudaSuccess ? RG_OK : RG_ERR_CUDA;
}

int rg_mlp_train(rg_system* s, const float* features, const float* targets, size_t n, int epochs, int batch,
                 float lr, uint64_t seed, float* final_loss) {
  if (!s || !features || !targets || n < 16 || epochs <= 0 || batch < 16 || !(lr > 0)) return RG_ERR_ARG;
  if (ensure_net(s)) return RG_ERR_CUDA;
  MlpHost& H = host_of(s);
  std::vector<float> P;
  init_params(P, features, targets, n, seed);
  cudaMemcpyAsync(H.P, P.data(), sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, s->stream);
  refresh_bf16(s);
  if (batch > (int)n) batch = (int)n;
  if (ensure_workspace(s)) return RG_ERR_CUDA;
  if (H.nfeat < n) {
    cudaFree(H.feat);
    cudaFree(H.tgt);
    if (cudaMalloc(&H.feat, sizeof(float) * kMlpIn * n) || cudaMalloc(&H.tgt, sizeof(float) * kMlpOut * n))
      return RG_ERR_CUDA;
    H.nfeat = n;
  }
  cudaMemcpyAsync(H.feat, features, sizeof(float) * kMlpIn * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(H.tgt, targets, sizeof(float) * kMlpOut * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemsetAsync(H.Am, 0, sizeof(float) * kMlpParams, s->stream);
  cudaMemsetAsync(H.Av, 0, sizeof(float) * kMlpParams, s->stream);
  if (H.nidx < n) {
    cudaFree(H.idx);
    if (cudaMalloc(&H.idx, sizeof(int) * n)) return RG_ERR_CUDA;
    H.nidx = n;
  }
  std::mt19937_64 rng(seed ^ 0xA5A5A5A5ull);
  std::vector<int> perm(n);
  for (size_t i = 0; i < n; ++i) perm[i] = (int)i;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const MlpDev M = mlp_dev(s);
  long step = 0;
  double last = 0;
  for (int ep = 0; ep < epochs; ++ep) {
    std::shuffle(perm.begin(), perm.end(), rng);
    // the epoch's order goes up once; each minibatch reads its slice
    if (cudaMemcpyAsync(H.idx, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s->stream)) return RG_ERR_CUDA;
    double ep_loss = 0;
    int nb = 0;
    for (size_t b0 = 0; b0 + batch <= n; b0 += batch) {
      const int nblk = forward_backward(s, H.feat, H.tgt, H.idx + b0, batch);
      ++step;
      float bc1 = 1.0f - std::pow(b1, (float)step), bc2 = 1.0f - std::pow(b2, (float)step);
      RGL k_mlp_adam<<<grid_for(kGradParams, 256), 256, 0, s->stream>>>(
          H.part, nblk, H.P, H.Am, H.Av, lr, b1, b2, eps, bc1, bc2, const_cast<__nv_bfloat16*>(M.w1),
          const_cast<__nv_bfloat16*>(M.w2), const_cast<__nv_bfloat16*>(M.w3), const_cast<__nv_bfloat16*>(M.w4));
      if (ep == epochs - 1) {
        ep_loss += read_loss(s, batch, nblk);
        ++nb;
      }
    }
    if (nb) last = ep_loss / nb;
  }
  if (cudaStreamSynchronize(s->stream) || cudaGetLastError()) return RG_ERR_CUDA;
  s->mlp_ready = true;
  if (final_loss) *final_loss = (float)last;
  return RG_OK;
}

int rg_mlp_infer(rg_system* s, const float* features, float* out, size_t n) {
  if (!s || !features || !out || n == 0) return RG_ERR_ARG;
  if (!s->mlp_ready) return RG_ERR_STATE;
  float *fT = nullptr, *oT = nullptr;
  if (cudaMalloc(&fT, sizeof(float) * kMlpIn * n) || cudaMalloc(&oT, sizeof(float) * kMlpOut * n)) return RG_ERR_CUDA;
  std::vector<float> t(kMlpIn * n);
  for (size_t i = 0; i < n; ++i)
    for (int k = 0; k < kMlpIn; ++k) t[(size_t)k * n + i] = features[i * kMlpIn + k];
  cudaMemcpyAsync(fT, t.data(), sizeof(float) * kMlpIn * n, cudaMemcpyHostToDevice, s->stream);
  int warps = (int)((n + 15) / 16);
  RGL k_mlp_infer<<<(warps + 7) / 8, 256, 0, s->stream>>>(mlp_dev(s), fT, (int)n, oT);
  std::vector<float> o(kMlpOut * n);
  cudaMemcpyAsync(o.data(), oT, sizeof(float) * kMlpOut * n, cudaMemcpyDeviceToHost, s->stream);
  cudaError_t e = cudaStreamSynchronize(s->stream);
  for (size_t i = 0; i < n; ++i)
    for (int k = 0; k < kMlpOut; ++k) out[i * kMlpOut + k] = o[(size_t)k * n + i];
  cudaFree(fT);
  cudaFree(oT);
  return e == cudaSuccess ? RG_OK : RG_ERR_CUDA;
}

// Batched systems: implemented in rg_batch.cu.

}  // extern "C"
