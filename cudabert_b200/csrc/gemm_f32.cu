// fp32 CUDA-core GEMM with the same fused epilogue as the tensor-core GEMM; it is the
// projection kernel of the fp32-accuracy mode (the mode that has to stay within 1e-3 max-abs
// of the reference's fp32 model).  out[M, N] = A[M, K] x W[K, N]; W keeps the on-disk
// [in, out] layout (convert_pytorch_model_to_npys.py:62-63), so no transpose is needed.
// Replaces the same reference calls as gemm_tcgen05.cu (ops/linear.cu:91-148, 241-319).
//
// 64 x 64 tile, k-step 16, 128 threads (8 x 4 outputs each), three shared-memory stages filled with
// cp.async two k-steps ahead.  The tile is small on purpose: the shapes of this mode are a few hundred
// to a few thousand rows against N = 768..4096, and 64 x 64 tiles give every SM several CTAs to
// overlap one CTA's load latency with another's arithmetic (the reduction is never split, so a row's
// result does not depend on the batch it is in).  Rows beyond M are loaded as zero and not stored.
#include "kernels.h"
#include "ptx.cuh"

#include <atomic>

namespace cb {
namespace {

constexpr int TM = 64, TN = 64, TK = 16, F32_STAGES = 3, F32_THREADS = 128;
constexpr int A_LD = TK + 4;  // padded row of the A tile: 80 bytes, keeps 16-byte alignment

__device__ __forceinline__ float gelu_erf_f32(float x) { return x * 0.5f * (1.0f + erff(x * 0.70710678118654752f)); }

__global__ void __launch_bounds__(F32_THREADS)
gemm_f32_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int M, int N, int K,
                float* __restrict__ out, int ldo, int flags, const float* __restrict__ bias,
                const float* __restrict__ residual, const float* __restrict__ colscale,
                const int* __restrict__ m_dev) {
  griddep_wait();
  griddep_launch();
  if (m_dev) M = min(M, __ldg(m_dev));
  const int m0 = blockIdx.y * TM;
  if (m0 >= M) return;
  __shared__ __align__(16) float As[F32_STAGES][TM][A_LD];
  __shared__ __align__(16) float Bs[F32_STAGES][TK][TN];
  const int tid = threadIdx.x;
  const int n0 = blockIdx.x * TN;
  const int ty = tid >> 4, tx = tid & 15;  // 8 x 16 threads; thread owns rows ty*8 + {0..7}, columns tx*4 + {0..3}

  // every thread moves two 16-byte pieces of A and two of B per k-step
  auto load_stage = [&](int stage, int ks) {
    const int k0 = ks * TK;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = tid + F32_THREADS * j;
      const int ar = c >> 2, ak = (c & 3) * 4;
      const bool a_ok = (m0 + ar) < M;
      cp_async16(smem_u32(&As[stage][ar][ak]), A + static_cast<size_t>(a_ok ? m0 + ar : 0) * lda + k0 + ak, a_ok);
      const int br = c >> 4, bn = (c & 15) * 4;
      const bool b_ok = (n0 + bn) < N;
      cp_async16(smem_u32(&Bs[stage][br][bn]), W + static_cast<size_t>(k0 + br) * N + (b_ok ? n0 + bn : 0), b_ok);
    }
  };

  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  const int ksteps = K / TK;
  load_stage(0, 0);
  cp_async_commit();
  if (ksteps > 1) load_stage(1, 1);
  cp_async_commit();
  for (int ks = 0; ks < ksteps; ++ks) {
    cp_async_wait<1>();  // the group of k-step ks has landed (one younger group may still be in flight)
    __syncthreads();     // ... for every thread's pieces, and everyone is done with the stage refilled below
    if (ks + 2 < ksteps) load_stage((ks + 2) % F32_STAGES, ks + 2);
    cp_async_commit();
    const int st = ks % F32_STAGES;
#pragma unroll
    for (int k4 = 0; k4 < TK; k4 += 4) {
      float4 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(&As[st][ty * 8 + i][k4]);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const float4 b = *reinterpret_cast<const float4*>(&Bs[st][k4 + kk][tx * 4]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float av = kk == 0 ? a[i].x : (kk == 1 ? a[i].y : (kk == 2 ? a[i].z : a[i].w));
          acc[i][0] = fmaf(av, b.x, acc[i][0]);
          acc[i][1] = fmaf(av, b.y, acc[i][1]);
          acc[i][2] = fmaf(av, b.z, acc[i][2]);
          acc[i][3] = fmaf(av, b.w, acc[i][3]);
        }
      }
    }
  }

  const int col = n0 + tx * 4;
  if (col >= N) return;
  float4 cs = make_float4(1.f, 1.f, 1.f, 1.f), bv = make_float4(0.f, 0.f, 0.f, 0.f);
  if (flags & EPI_COLSCALE) cs = __ldg(reinterpret_cast<const float4*>(colscale + col));
  if (flags & EPI_BIAS) bv = __ldg(reinterpret_cast<const float4*>(bias + col));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = m0 + ty * 8 + i;
    if (row >= M) continue;
    float v[4] = {acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
    if (flags & EPI_COLSCALE) { v[0] *= cs.x; v[1] *= cs.y; v[2] *= cs.z; v[3] *= cs.w; }
    if (flags & EPI_BIAS) { v[0] += bv.x; v[1] += bv.y; v[2] += bv.z; v[3] += bv.w; }
    if (flags & EPI_RESIDUAL) {
      const float4 r = __ldg(reinterpret_cast<const float4*>(residual + static_cast<size_t>(row) * ldo + col));
      v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
    }
    if (flags & EPI_GELU) {
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = gelu_erf_f32(v[q]);
    }
    if (flags & EPI_TANH) {
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = tanhf(v[q]);
    }
    *reinterpret_cast<float4*>(out + static_cast<size_t>(row) * ldo + col) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// Pooler: out[b, :] = tanh(x[first row of sequence b, 0..H) . W[H, H] + bias), fp32
// (reference: copy_pooler + op_Linear + op_Tanh, ops/elementwise.cu:6-32, 57-70, utils/bert.cu:239-247).
// It is a skinny product: B rows against an H x H matrix that has to come from memory once, so what counts is
// how early and how widely that matrix is requested.  A CTA owns PN = 16 output columns; its [H][16] slab of
// weights (64 KB at H = 1024, 64 CTAs for all of them) is copied to shared memory asynchronously BEFORE
// griddep_wait, i.e. while the last LayerNorm is still running, and then serves every group of PB = 8 sequences that
// the CTA takes (gridDim.y CTAs share the groups).  256 threads are 16 columns x 16 slices of the reduction
// dimension, slice s summing k = 4 s .. 4 s + 3 of every 64; the inputs are 16-byte broadcasts and the next group's
// are on their way while this one's are used.  The 16 partial sums meet in shared memory in a fixed
// order, so a row's result does not depend on the batch.
// Measured on a B200 against 64-column CTAs that read the weights through registers after the wait (24 us at
// H = 1024 for one sequence): whole passes, BERT-base 1 x 24 417 -> 387 us, BERT-large 1 x 128 942 -> 893 us.
constexpr int PN = 16, PB = 8, PSLICES = 16;
constexpr int WPITCH = PN + 4;  // the two slices of a warp read weight rows 4 apart: 16 banks apart
constexpr int POOL_GROUPS = 2;  // 64 column slabs x 2 = 128 CTAs of 152 KB at H = 1024
constexpr int POOL_TILE_MIN_SEQS = 192;  // see pooler_f32

__global__ void __launch_bounds__(PN * PSLICES)
pooler_f32_kernel(const float* __restrict__ x, int rows_per_seq, const int* __restrict__ row_start,
                  const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out, int B, int H) {
  extern __shared__ float pool_smem[];
  float* ws = pool_smem;                 // [H][WPITCH]: the CTA's weights
  float* xs = ws + H * WPITCH;           // [2][PB][H]: this group's input rows and the next one's
  float* part = xs + 2 * H * PB;         // [PSLICES][PB][PN] partial sums
  const int tid = threadIdx.x;
  const int c = tid % PN, slice = tid / PN;
  const int n0 = blockIdx.x * PN;
  for (int i = tid; i < H * (PN / 4); i += PN * PSLICES)
    cp_async16(smem_u32(ws + (i / (PN / 4)) * WPITCH + (i % (PN / 4)) * 4),
               W + static_cast<size_t>(i / (PN / 4)) * H + n0 + (i % (PN / 4)) * 4, true);
  cp_async_commit();
  const float bv = __ldg(bias + n0 + c);
  griddep_wait();
  griddep_launch();
  // group b0's rows, zero beyond the batch, asynchronously
  auto load_x = [&](float* dst, int b0) {
    for (int i = tid; i < H / 4 * PB; i += PN * PSLICES) {
      const int r = i / (H / 4), k = (i - r * (H / 4)) * 4, bb = b0 + r;
      const float* src = x;
      if (bb < B)
        src = x + (row_start ? static_cast<size_t>(__ldg(row_start + bb)) : static_cast<size_t>(bb) * rows_per_seq) * H + k;
      cp_async16(smem_u32(dst + r * H + k), src, bb < B);
    }
  };
  const int step = gridDim.y * PB;
  int buf = 0;
  load_x(xs, blockIdx.y * PB);
  cp_async_commit();
  for (int b0 = blockIdx.y * PB; b0 < B; b0 += step, buf ^= 1) {
    if (b0 + step < B) load_x(xs + (buf ^ 1) * H * PB, b0 + step);  // last read two barriers ago
    cp_async_commit();
    cp_async_wait<1>();  // this group's rows (and the weights) are there
    __syncthreads();
    const float* xb = xs + buf * H * PB;
    float acc[PB];
#pragma unroll
    for (int r = 0; r < PB; ++r) acc[r] = 0.f;
#pragma unroll 4
    for (int k = slice * 4; k < H; k += PSLICES * 4) {
      float w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = ws[(k + j) * WPITCH + c];
#pragma unroll
      for (int r = 0; r < PB; ++r) {
        const float4 v = *reinterpret_cast<const float4*>(xb + r * H + k);
        acc[r] = fmaf(v.x, w[0], acc[r]);
        acc[r] = fmaf(v.y, w[1], acc[r]);
        acc[r] = fmaf(v.z, w[2], acc[r]);
        acc[r] = fmaf(v.w, w[3], acc[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < PB; ++r) part[(slice * PB + r) * PN + c] = acc[r];
    __syncthreads();
    if (slice < PB && b0 + slice < B) {  // row b0 + slice, column c
      float v = bv;
#pragma unroll
      for (int sl = 0; sl < PSLICES; ++sl) v += part[(sl * PB + slice) * PN + c];  // fixed order: deterministic
      out[static_cast<size_t>(b0 + slice) * H + n0 + c] = tanhf(v);
    }
  }
}

// The same for many sequences: a CTA takes 32 of them and 64 columns, a thread 4 x 4 outputs, so that two 16-byte reads of
// shared memory feed 16 multiply-adds and the product is bound by those.  The terms are added in the order of
// pooler_f32_kernel, so a row has the same bits from either: the loop runs slice after slice (k = 64 j + 4 s .. + 3 for
// s = 0 .. 15), each slice's sum is finished in registers and added to bias + the sums before.  Slices are copied
// asynchronously into two buffers, the first one's weights ahead of griddep_wait.
constexpr int PTM = 32, PTN = 64, PTHREADS = (PTM / 4) * (PTN / 4);

__global__ void __launch_bounds__(PTHREADS)
pooler_f32_tile_kernel(const float* __restrict__ x, int rows_per_seq, const int* __restrict__ row_start,
                       const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out, int B, int H) {
  extern __shared__ float pool_smem[];
  __shared__ int srow[PTM];               // row of x of the CTA's sequences, -1 beyond the batch
  const int KS = H / PSLICES, XP = KS + 4;  // a slice's terms; pitch of its inputs: a warp's two rows are 16 banks apart
  float* xs = pool_smem;                 // [2][PTM][XP]
  float* ws = xs + 2 * PTM * XP;          // [2][KS][PTN]
  const int tid = threadIdx.x;
  const int n0 = blockIdx.x * PTN, b0 = blockIdx.y * PTM;
  const int c = (tid % (PTN / 4)) * 4, r0 = (tid / (PTN / 4)) * 4;
  auto load_w = [&](int buf, int s) {
    for (int i = tid; i < KS * (PTN / 4); i += PTHREADS) {
      const int kk = i / (PTN / 4), c4 = (i % (PTN / 4)) * 4, k = (kk >> 2) * (4 * PSLICES) + 4 * s + (kk & 3);
      cp_async16(smem_u32(ws + (buf * KS + kk) * PTN + c4), W + static_cast<size_t>(k) * H + n0 + c4, true);
    }
  };
  auto load_x = [&](int buf, int s) {
    for (int i = tid; i < PTM * (KS / 4); i += PTHREADS) {
      const int r = i / (KS / 4), j = i - r * (KS / 4), row = srow[r];
      const float* src = row < 0 ? x : x + static_cast<size_t>(row) * H + j * (4 * PSLICES) + 4 * s;
      cp_async16(smem_u32(xs + (buf * PTM + r) * XP + 4 * j), src, row >= 0);
    }
  };
  load_w(0, 0);
  float v[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float bv = __ldg(bias + n0 + c + q);
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r][q] = bv;
  }
  griddep_wait();
  griddep_launch();
  if (tid < PTM) {
    const int bb = b0 + tid;
    srow[tid] = bb >= B ? -1 : row_start ? __ldg(row_start + bb) : bb * rows_per_seq;
  }
  __syncthreads();
  load_x(0, 0);
  cp_async_commit();
  for (int s = 0; s < PSLICES; ++s) {
    const int buf = s & 1;
    if (s + 1 < PSLICES) {
      load_w(buf ^ 1, s + 1);
      load_x(buf ^ 1, s + 1);
    }
    cp_async_commit();
    cp_async_wait<1>();  // all but the slice just requested
    __syncthreads();
    const float* xb = xs + (buf * PTM + r0) * XP;
    const float* wb = ws + buf * KS * PTN + c;
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[r][q] = 0.f;
#pragma unroll 4
    for (int k = 0; k < KS; k += 4) {
      float4 xv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) xv[r] = *reinterpret_cast<const float4*>(xb + r * XP + k);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(wb + (k + i) * PTN);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float a = i == 0 ? xv[r].x : i == 1 ? xv[r].y : i == 2 ? xv[r].z : xv[r].w;
          acc[r][0] = fmaf(a, w.x, acc[r][0]);
          acc[r][1] = fmaf(a, w.y, acc[r][1]);
          acc[r][2] = fmaf(a, w.z, acc[r][2]);
          acc[r][3] = fmaf(a, w.w, acc[r][3]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) v[r][q] += acc[r][q];
    __syncthreads();  // the buffer is free for the slice after next
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if (b0 + r0 + r < B)
      *reinterpret_cast<float4*>(out + static_cast<size_t>(b0 + r0 + r) * H + n0 + c) =
          make_float4(tanhf(v[r][0]), tanhf(v[r][1]), tanhf(v[r][2]), tanhf(v[r][3]));
}

}  // namespace

int pooler_f32(const float* x, int rows_per_seq, const int* row_start, const float* W, const float* bias, float* out,
               int B, int H, cudaStream_t stream) {
  if (B <= 0 || H <= 0 || (H % 64) != 0 || H > 1024) return -1;
  static std::atomic<bool> attr_set[64] = {};  // per device; a repeated set by a racing thread is harmless
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(pooler_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (1024 * (WPITCH + 2 * PB) + PSLICES * PB * PN) * static_cast<int>(sizeof(float))) != cudaSuccess ||
        cudaFuncSetAttribute(pooler_f32_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * (PTM * (1024 / PSLICES + 4) + 1024 / PSLICES * PTN) * static_cast<int>(sizeof(float))) != cudaSuccess)
      return -2;
    if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
  }
  // The slab kernel's 96 (H = 768) or 128 CTAs take their groups of eight sequences one after the other, some 2.5 us each; a tile's time does not grow until the tiles fill the SMs.  Same bits.  Slab / tiles, us (events around the
  // launch): H = 768 128 sequences 25 / 33, 192 35 / 33, 256 44 / 33, 1024 154 / 55, 4096 596 / 168; H = 1024 128 30 / 38,
  // 192 41 / 39, 256 52 / 39, 1024 187 / 82, 4096 729 / 281.
  if (B >= POOL_TILE_MIN_SEQS) {
    const dim3 grid(H / PTN, (B + PTM - 1) / PTM);
    if (grid.y > 65535) return -1;
    const size_t smem = 2 * (static_cast<size_t>(PTM) * (H / PSLICES + 4) + static_cast<size_t>(H) / PSLICES * PTN) * sizeof(float);
    return launch_pdl(pooler_f32_tile_kernel, grid, dim3(PTHREADS), smem, stream, x, rows_per_seq, row_start, W, bias, out,
                      B, H) == cudaSuccess ? 1 : -3;
  }
  // one CTA fits on an SM: beyond POOL_GROUPS groups of sequences a CTA takes several
  const int groups = (B + PB - 1) / PB;
  dim3 grid(H / PN, groups < POOL_GROUPS ? groups : POOL_GROUPS);
  const size_t smem = (static_cast<size_t>(H) * (WPITCH + 2 * PB) + PSLICES * PB * PN) * sizeof(float);
  return launch_pdl(pooler_f32_kernel, grid, dim3(PN * PSLICES), smem, stream, x, rows_per_seq, row_start, W, bias, out,
                    B, H) == cudaSuccess ? 1 : -3;
}

int gemm_f32(const float* A, int lda, const float* W, int M, int N, int K, float* out, int ldo,
             const GemmEpilogue& epi, const int* m_dev, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (N % 4) != 0 || (K % TK) != 0 || (lda % 4) != 0 || (ldo % 4) != 0) return -1;
  if ((epi.flags & EPI_BIAS) && !epi.bias) return -1;
  if ((epi.flags & EPI_RESIDUAL) && !epi.residual) return -1;
  if ((epi.flags & EPI_COLSCALE) && !epi.colscale) return -1;
  dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
  if (grid.y > 65535) return -1;
  // plain stream order: with dependent launch this kernel's forward pass took twice as long (BERT-base,
  // 8 x 128 tokens: 8.4 against 4.5 ms), its many small CTAs being scheduled ahead of their producers
  return launch_plain(gemm_f32_kernel, grid, dim3(F32_THREADS), 0, stream, A, lda, W, M, N, K, out, ldo, epi.flags,
                    epi.bias, static_cast<const float*>(epi.residual), epi.colscale, m_dev) == cudaSuccess ? 1 : -3;
}

}  // namespace cb
