// On-device GPTQ core for sm_100a: Hessian preparation, U = chol(H^-1, upper), the column-block
// quantise / error-propagation loop and the relative-MSE metric.  Replaces GPTQ._get_hessian_inverse,
// GPTQ.step and get_relative_mse_error of src/quantization/gptq.py (IST-DASLab/FP-Quant), which run
// as ~50 small torch kernels per weight column plus cuSOLVER calls.
//
// All arithmetic is fp32 (the reference disables TF32).  The reference chain
// cholesky -> cholesky_inverse -> cholesky(upper) is replaced by the mathematically equal
//   P = J H J (rows and columns reversed),  P = L L^T,  U = J L^-1 J
// because H = (J L J)(J L J)^T with J L J upper triangular, hence H^-1 = U^T U with U = (J L J)^-1.
// One factorisation and one triangular inverse instead of two factorisations and a full inverse.

#include <cstdlib>
#include <vector>
#include "common.cuh"

#include <atomic>
#include "sgemm.cuh"

namespace fpq {
// defined in hessian.cu: out = beta * out + alpha * A^T B on the tensor cores (bf16 operands, fp32 accumulation)
int gemm_atb_bf16(float* out, int64_t ldc, int64_t d1, int64_t d2, const void* A, int64_t lda, int64_t a_rows,
                  int64_t a_x0, const void* B, int64_t ldb, int64_t b_rows, int64_t b_x0, bool symmetric, bool mirror,
                  int n_seg, int64_t seg_rows, const int* a_seg_y, const int* b_seg_y, float alpha, float beta,
                  int32_t* error_flag, cudaStream_t stream, int tri = 0, int64_t chain_rows = 0);
bool gemm_atb_on_pairs(int64_t d1, int64_t d2, bool symmetric, int n_seg, int64_t seg_rows);
}  // namespace fpq

namespace fpq {
namespace {

constexpr int NB = 128;   // block size of the factorisation and of the GPTQ column blocks

// ------------------------------------------------------------------ Hessian preparation
__global__ void dead_columns_kernel(const float* __restrict__ W, int64_t rows, int64_t d, uint8_t* dead) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d) return;
  bool all_zero = true;
  for (int64_t i = 0; i < rows && all_zero; ++i) all_zero = (W[i * d + j] == 0.0f);
  dead[j] = all_zero ? 1 : 0;
}

// Rows and columns of dead input channels become rows / columns of the identity.  A block covers 16 rows x
// 256 columns and leaves at once when none of its rows and columns is dead (the usual case: nothing is).
__global__ void __launch_bounds__(256) mask_dead_kernel(float* H, int64_t d, const uint8_t* __restrict__ dead) {
  __shared__ uint8_t drow[16];
  const int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t i0 = (int64_t)blockIdx.y * 16;
  if (threadIdx.x < 16) drow[threadIdx.x] = (i0 + threadIdx.x < d) ? dead[i0 + threadIdx.x] : 0;
  const int dj = (j < d && dead[j]) ? 1 : 0;
  const int any_col = __syncthreads_or(dj);       // also publishes drow
  int any_row = 0;
#pragma unroll
  for (int r = 0; r < 16; ++r) any_row |= drow[r];
  if (!any_col && !any_row) return;
  if (j >= d) return;
  for (int r = 0; r < 16; ++r) {
    const int64_t i = i0 + r;
    if (i < d && (drow[r] || dj)) H[i * d + j] = (i == j) ? 1.0f : 0.0f;
  }
}

__global__ void damp_kernel(float* H, int64_t d, float rel_damp) {
  // one block: mean of the diagonal, then diag += rel_damp * mean
  __shared__ double part[256];
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < d; i += blockDim.x) s += (double)H[i * d + i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  const float damp = rel_damp * (float)(part[0] / (double)d);
  for (int64_t i = threadIdx.x; i < d; i += blockDim.x) H[i * d + i] += damp;
}

// ------------------------------------------------------------------ reversal / reflection
__global__ void reverse_copy_kernel(const float* __restrict__ src, float* __restrict__ dst, int64_t d) {
  const int64_t n = d * d;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (int64_t)gridDim.x * blockDim.x)
    dst[idx] = src[n - 1 - idx];   // (i, j) <- (d-1-i, d-1-j)
}

// A <- J A J.  Four elements at a time from either end (n / 8 vectors a side, the middle one by one): HBM-bound, 2 x 4 B
// read and written per element of a pair; d = 14336 in 252 us instead of 680 with single elements.
__global__ void reflect_inplace_kernel(float* A, int64_t d) {
  const int64_t n = d * d, half = n / 2;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  const int64_t vecs = (n % 4 == 0 && ((uintptr_t)A & 15) == 0) ? n / 8 : 0;
  float4* A4 = reinterpret_cast<float4*>(A);
  for (int64_t idx = t0; idx < vecs; idx += step) {
    const float4 a = A4[idx], b = A4[n / 4 - 1 - idx];
    A4[idx] = make_float4(b.w, b.z, b.y, b.x);
    A4[n / 4 - 1 - idx] = make_float4(a.w, a.z, a.y, a.x);
  }
  for (int64_t idx = 4 * vecs + t0; idx < half; idx += step) {
    const float a = A[idx], b = A[n - 1 - idx];
    A[idx] = b;
    A[n - 1 - idx] = a;
  }
}

// ------------------------------------------------------------------ diagonal block: factor + invert
// One CTA factors the nb x nb (<= 128) diagonal block A (lower Cholesky, in place) and writes
// L^-1 (lower; blocks right of the diagonal stay as the caller zeroed them) to Linv.  A non-positive or
// non-finite pivot sets *status and is replaced by 1 so that the kernel always terminates.
//
// The arithmetic is right-looking elimination column by column, with c = A[:, k] and x = X[k, :] unscaled:
//     A[i, j] = fma(-c_i, c_j / pivot, A[i, j])  (i, j > k),     X[i, :] = fma(-c_i, x / pivot, X[i, :])  (i > k),
// 1 / pivot rounded, the columns of L and the rows of X divided by sqrt(pivot) at the end.  Every element goes through
// these operations in the order of k whatever the blocking below, so the bits do not depend on it.
//
// The kernel is one chain of dependent steps, so it is laid out for a short chain: blocks of 32 columns in shared
// memory.  A block's 32 x 32 diagonal part is factored by one warp, a row per lane, in registers; a step costs one
// shuffle latency (the pivot and the whole column leave together), a reciprocal, a product and a fused multiply-add,
// no barrier.  Everything else is done by many threads at a time:
//   phase 1   warp 0 factors D_p                       | four warps: S_p = -C_(p, <p) X_(<p)
//   phase 2   four warps, one vector a thread: the rows of C below D_p and the columns of X_p (from S_p, and from the
//             unit vectors), by forward substitution
//   phase 3   all: the trailing part -= C (C / pivot)^T
// with C the unscaled columns of L and X = L^-1 by blocks of rows.  40 us in the chain of d = 4096; 48 us as one elimination
// with a barrier per column; 33 us with approximate reciprocals and sums in two halves, which changed the bits.
constexpr int CD_LD = NB + 4;         // row stride in shared memory: 16-byte rows whose starts walk through the banks
constexpr int CD_B = 32;              // block of columns
constexpr int CD_SLD = 96 + 4;
constexpr int CD_TLD = CD_B + 4;
constexpr int CD_SMEM = (2 * NB * CD_LD + CD_B * CD_SLD + (96 + 2 * CD_B) * CD_TLD + NB + CD_B) * (int)sizeof(float);

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&r);
}

// Factor the 32 x 32 block at D: its unscaled columns C in place (lower part) and transposed to DT, C / pivot transposed
// to TT, 1 / pivot to pinv, 1 / sqrt(pivot) to rinv.
__device__ __forceinline__ void factor32(float* D, float* DT, float* TT, float* pinv, float* rinv, int lane, int32_t* status) {
  float a[CD_B];
#pragma unroll
  for (int q = 0; q < CD_B / 4; ++q) {
    const float4 v = *reinterpret_cast<const float4*>(D + lane * CD_LD + 4 * q);
    a[4 * q] = v.x; a[4 * q + 1] = v.y; a[4 * q + 2] = v.z; a[4 * q + 3] = v.w;
  }
  bool bad = false;
  float my_piv = 1.0f, my_pinv = 1.0f;                     // of this row
#pragma unroll
  for (int k = 0; k < CD_B; ++k) {
    const float c = a[k];
    float piv = __shfl_sync(0xffffffffu, c, k);
    const bool ok = piv > 0.0f && isfinite(piv);
    piv = ok ? piv : 1.0f;
    bad |= !ok;
    const float r = __frcp_rn(piv);
    // rows at or above k get values that nothing reads
#pragma unroll
    for (int j = k + 1; j < CD_B; ++j) a[j] = fmaf(-c, __shfl_sync(0xffffffffu, c, j) * r, a[j]);
    if (lane == k) {
      my_piv = piv;
      my_pinv = r;
    }
  }
  // the square roots wait until here, off the chain
  float ri = rsqrtf(my_piv);
  ri = ri * fmaf(-0.5f * my_piv * ri, ri, 1.5f);           // one Newton step: full fp32 accuracy
  if (bad && lane == 0) atomicExch(status, 1);
  rinv[lane] = ri;
  pinv[lane] = my_pinv;
#pragma unroll
  for (int k = 0; k < CD_B; ++k) {
    DT[k * CD_TLD + lane] = a[k];
    TT[k * CD_TLD + lane] = a[k] * __shfl_sync(0xffffffffu, my_pinv, k);
  }
#pragma unroll
  for (int q = 0; q < CD_B / 4; ++q)
    *reinterpret_cast<float4*>(D + lane * CD_LD + 4 * q) = make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
}

// Forward substitution, every thread a vector of its own: v[j] = fma(-L[j, k], z_k, v[j]) for k < j in order, with
// z_k = v[k] (rows of A: L holds C / pivot) or v[k] / pivot (columns of X: L holds C).  L comes transposed, as broadcasts.
__device__ __forceinline__ void solve32(const float* LT, const float* pinv, bool divide, float (&v)[CD_B]) {
#pragma unroll
  for (int k = 0; k < CD_B; ++k) {
    const float z = divide ? v[k] * pinv[k] : v[k];
#pragma unroll
    for (int q = 0; q < CD_B / 4; ++q) {
      if (4 * q + 3 <= k) continue;
      const float4 l = *reinterpret_cast<const float4*>(LT + k * CD_TLD + 4 * q);
      if (4 * q > k) v[4 * q] = fmaf(-l.x, z, v[4 * q]);
      if (4 * q + 1 > k) v[4 * q + 1] = fmaf(-l.y, z, v[4 * q + 1]);
      if (4 * q + 2 > k) v[4 * q + 2] = fmaf(-l.z, z, v[4 * q + 2]);
      v[4 * q + 3] = fmaf(-l.w, z, v[4 * q + 3]);
    }
  }
}

// A[r0 + i, r0 + j] = fma(-C[i, k], T[j, k], .), k = 0 .. 31 in order, over the sixteenths on and below the diagonal.
template <int N>
__device__ __forceinline__ void trailing32(float* A, const float* Tp, int r0, int c0, int ty, int tx) {
  float acc[N][N];
#pragma unroll
  for (int r = 0; r < N; ++r)
#pragma unroll
    for (int c = 0; c <= r; ++c) acc[r][c] = A[(r0 + ty + 16 * r) * CD_LD + r0 + tx + 16 * c];
#pragma unroll
  for (int q = 0; q < CD_B / 4; ++q) {
    float4 ci[N], tj[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      ci[r] = *reinterpret_cast<const float4*>(A + (r0 + ty + 16 * r) * CD_LD + c0 + 4 * q);
      tj[r] = *reinterpret_cast<const float4*>(Tp + (tx + 16 * r) * CD_TLD + 4 * q);
    }
#pragma unroll
    for (int r = 0; r < N; ++r)
#pragma unroll
      for (int c = 0; c <= r; ++c) {
        acc[r][c] = fmaf(-ci[r].x, tj[c].x, acc[r][c]);
        acc[r][c] = fmaf(-ci[r].y, tj[c].y, acc[r][c]);
        acc[r][c] = fmaf(-ci[r].z, tj[c].z, acc[r][c]);
        acc[r][c] = fmaf(-ci[r].w, tj[c].w, acc[r][c]);
      }
  }
#pragma unroll
  for (int r = 0; r < N; ++r)
#pragma unroll
    for (int c = 0; c <= r; ++c) A[(r0 + ty + 16 * r) * CD_LD + r0 + tx + 16 * c] = acc[r][c];
}

__global__ void __launch_bounds__(256, 1) chol_diag_kernel(float* A, int64_t lda, float* Linv, int64_t ldi, int nb,
                                                        int32_t* status) {
  extern __shared__ __align__(16) float cd_smem[];
  float* As = cd_smem;                       // unscaled columns of L once they are final
  float* Y = As + NB * CD_LD;                // rows of X / pivot
  float* S = Y + NB * CD_LD;
  float* Tp = S + CD_B * CD_SLD;             // rows below the block: C / pivot
  float* DT = Tp + 96 * CD_TLD;
  float* TT = DT + CD_B * CD_TLD;
  float* rinv = TT + CD_B * CD_TLD;
  float* pinv = rinv + NB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool vec = nb == NB && lda % 4 == 0 && ((uintptr_t)A & 15) == 0;
  for (int o = tid; o < NB * NB / 4; o += 256) {
    const int i = o / (NB / 4), j = (o % (NB / 4)) * 4;
    float v[4];
    if (vec) {
      *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(A + (int64_t)i * lda + j);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = (i < nb && j + q < nb) ? A[(int64_t)i * lda + j + q] : (i == j + q ? 1.0f : 0.0f);
    }
    *reinterpret_cast<float4*>(As + i * CD_LD + j) = *reinterpret_cast<float4*>(v);
  }
  __syncthreads();
#pragma unroll 1
  for (int p = 0; p < NB / CD_B; ++p) {
    const int c0 = CD_B * p, below = NB - c0 - CD_B;
    if (warp == 0) {
      factor32(As + c0 * CD_LD + c0, DT, TT, pinv, rinv + c0, lane, status);
    } else if (p > 0 && (warp & 3) != 0 && warp < 6) {     // warps 1, 2, 3, 5: not on warp 0's scheduler
      // S = -C[c0 .. c0 + 31, 0 .. c0 - 1] Y[0 .. c0 - 1, 0 .. c0 - 1], Y lower triangular by blocks, k in order
      const int t = (warp < 4 ? warp - 1 : 3) * 32 + lane, r = t >> 2, cq = (t & 3) * 4;
      const float* Cr = As + (c0 + r) * CD_LD;
      for (int jb = 0; jb < p; ++jb) {
        const int j = jb * CD_B + cq;                      // columns j .. j + 3 and j + 16 .. j + 19
        float2 s0 = make_float2(0.0f, 0.0f), s1 = s0, s2 = s0, s3 = s0;
#pragma unroll 8
        for (int k = jb * CD_B; k < c0; ++k) {
          const float2 l = make_float2(-Cr[k], -Cr[k]);
          const float4 x0 = *reinterpret_cast<const float4*>(Y + k * CD_LD + j);
          const float4 x1 = *reinterpret_cast<const float4*>(Y + k * CD_LD + j + 16);
          s0 = fma2(l, make_float2(x0.x, x0.y), s0);
          s1 = fma2(l, make_float2(x0.z, x0.w), s1);
          s2 = fma2(l, make_float2(x1.x, x1.y), s2);
          s3 = fma2(l, make_float2(x1.z, x1.w), s3);
        }
        *reinterpret_cast<float4*>(S + r * CD_SLD + j) = make_float4(s0.x, s0.y, s1.x, s1.y);
        *reinterpret_cast<float4*>(S + r * CD_SLD + j + 16) = make_float4(s2.x, s2.y, s3.x, s3.y);
      }
    }
    __syncthreads();
    if (warp < 4) {
      // 128 vectors whatever p: `below` rows of A, then the c0 + 32 columns of X that reach this block of rows
      const bool is_x = tid >= below;
      const int col = tid - below;
      float v[CD_B];
      float* row = As + (c0 + CD_B + tid) * CD_LD + c0;    // of A
      if (!is_x) {
#pragma unroll
        for (int q = 0; q < CD_B / 4; ++q) {
          const float4 w = *reinterpret_cast<const float4*>(row + 4 * q);
          v[4 * q] = w.x; v[4 * q + 1] = w.y; v[4 * q + 2] = w.z; v[4 * q + 3] = w.w;
        }
      } else if (col < c0) {
#pragma unroll
        for (int k = 0; k < CD_B; ++k) v[k] = S[k * CD_SLD + col];
      } else {
#pragma unroll
        for (int k = 0; k < CD_B; ++k) v[k] = col - c0 == k ? 1.0f : 0.0f;
      }
      solve32(is_x ? DT : TT, pinv, is_x, v);
      if (!is_x) {
        float* trow = Tp + tid * CD_TLD;
#pragma unroll
        for (int q = 0; q < CD_B / 4; ++q) {
          *reinterpret_cast<float4*>(row + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          const float4 r = *reinterpret_cast<const float4*>(pinv + 4 * q);
          *reinterpret_cast<float4*>(trow + 4 * q) =
              make_float4(v[4 * q] * r.x, v[4 * q + 1] * r.y, v[4 * q + 2] * r.z, v[4 * q + 3] * r.w);
        }
      } else {
#pragma unroll
        for (int k = 0; k < CD_B; ++k) {
          Y[(c0 + k) * CD_LD + col] = v[k] * pinv[k];
          if (c0 + k < nb && col < nb) Linv[(int64_t)(c0 + k) * ldi + col] = v[k] * rinv[c0 + k];
        }
      }
    }
    __syncthreads();
    if (p == 0) trailing32<6>(As, Tp, c0 + CD_B, c0, tid >> 4, tid & 15);
    if (p == 1) trailing32<4>(As, Tp, c0 + CD_B, c0, tid >> 4, tid & 15);
    if (p == 2) trailing32<2>(As, Tp, c0 + CD_B, c0, tid >> 4, tid & 15);
    __syncthreads();
  }
  for (int o = tid; o < NB * NB / 4; o += 256) {
    const int i = o / (NB / 4), j = (o % (NB / 4)) * 4;
    float a[4], r[4];
    *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(As + i * CD_LD + j);
    *reinterpret_cast<float4*>(r) = *reinterpret_cast<const float4*>(rinv + j);
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = j + q > i ? 0.0f : a[q] * r[q];   // above the diagonal: what the updates left there
    if (vec) {
      *reinterpret_cast<float4*>(A + (int64_t)i * lda + j) = *reinterpret_cast<float4*>(a);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i < nb && j + q < nb) A[(int64_t)i * lda + j + q] = a[q];
    }
  }
}

// ------------------------------------------------------------------ panel below a diagonal block
// A[i, 0..127] <- sum_k A[i, k] Linv[j, k] (k <= j, in order) in place for `rows` rows: L21 = A21 L11^-T.  A CTA takes 32 rows, so
// that even a short panel spreads over the SMs, and holds Linv in shared memory; a thread has 2 x 8 outputs, the part
// of Linv above its diagonal is skipped.  Latency-bound.  Panels of a chain, average under ncu: 15 us at d = 4096 and
// 21 us at d = 14336; as a 128 x 128-tile matrix product on at most 112 CTAs 21 and 20 us.
constexpr int PANEL_ROWS = 32;
constexpr int PANEL_SMEM = (NB + PANEL_ROWS) * CD_LD * (int)sizeof(float);

__global__ void __launch_bounds__(256, 2) chol_panel_kernel(float* A, int64_t lda, int64_t rows, const float* __restrict__ Linv,
                                                            int64_t ldi) {
  extern __shared__ __align__(16) float pn_smem[];
  float* Ls = pn_smem;
  float* Ps = Ls + NB * CD_LD;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int64_t r0 = (int64_t)blockIdx.x * PANEL_ROWS;
  const bool vec = lda % 4 == 0 && ldi % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)Linv & 15) == 0;
  for (int o = tid; o < (NB + PANEL_ROWS) * NB / 4; o += 256) {
    const int i = o / (NB / 4), j = (o % (NB / 4)) * 4;
    const bool is_l = i < NB;
    const int64_t ar = r0 + i - NB;
    const float* src = is_l ? Linv + (int64_t)i * ldi + j : A + ar * lda + j;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (is_l || ar < rows) v = vec ? *reinterpret_cast<const float4*>(src) : make_float4(src[0], src[1], src[2], src[3]);
    *reinterpret_cast<float4*>((is_l ? Ls + i * CD_LD : Ps + (i - NB) * CD_LD) + j) = v;
  }
  __syncthreads();
  float acc[2][8];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[r][c] = 0.0f;
#pragma unroll
  for (int kb = 0; kb < 8; ++kb) {                         // sixteen k at a time: columns tx + 16 c with c >= kb need them
#pragma unroll 2
    for (int q = 0; q < 4; ++q) {
      const int k = 16 * kb + 4 * q;
      const float4 a0 = *reinterpret_cast<const float4*>(Ps + ty * CD_LD + k);
      const float4 a1 = *reinterpret_cast<const float4*>(Ps + (ty + 16) * CD_LD + k);
#pragma unroll
      for (int c = kb; c < 8; ++c) {
        const float4 l = *reinterpret_cast<const float4*>(Ls + (tx + 16 * c) * CD_LD + k);
        acc[0][c] = fmaf(a0.w, l.w, fmaf(a0.z, l.z, fmaf(a0.y, l.y, fmaf(a0.x, l.x, acc[0][c]))));
        acc[1][c] = fmaf(a1.w, l.w, fmaf(a1.z, l.z, fmaf(a1.y, l.y, fmaf(a1.x, l.x, acc[1][c]))));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int64_t row = r0 + ty + 16 * r;
    if (row >= rows) continue;
#pragma unroll
    for (int c = 0; c < 8; ++c) A[row * lda + tx + 16 * c] = acc[r][c];
  }
}

int grid1d(int64_t n) {
  int64_t b = (n + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 16;
  return (int)(b > cap ? cap : (b < 1 ? 1 : b));
}

// ------------------------------------------------------------------ fp32-accurate products on the tensor cores
// x in fp32 -> three bf16 terms hi + mid + lo that together carry all 24 mantissa bits.
__device__ __forceinline__ void split3(float v, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  h = __float2bfloat16_rn(v);
  const float r1 = v - __bfloat162float(h);
  m = __float2bfloat16_rn(r1);
  l = __float2bfloat16_rn(r1 - __bfloat162float(m));
}

__device__ __forceinline__ uint32_t bf16_pair(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  const __nv_bfloat162 v = __halves2bfloat162(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// in [K, N] fp32 (row stride ld_in) -> out: three planes [K, ld_out] bf16 (hi, mid, lo), plane p at row p * K.  A thread
// takes four columns (N, the strides and the addresses allowing), a block 1024 columns of rows blockIdx.y, + gridDim.y, ...
// `upper`: the elements of an upper triangular matrix left of its diagonal's vector are not written (nor read by anyone).
// HBM-bound, 4 B read and 6 B written per element; the factor of d = 14336 in 191 us instead of 816 with one element
// and a 64-bit division per thread.
__global__ void __launch_bounds__(256) split3_rows_kernel(const float* __restrict__ in, int64_t ld_in, int64_t K, int64_t N,
                                                          __nv_bfloat16* __restrict__ out, int64_t ld_out, bool upper) {
  const bool vec = N % 4 == 0 && ld_in % 4 == 0 && ld_out % 4 == 0 && ((uintptr_t)in & 15) == 0 && ((uintptr_t)out & 7) == 0;
  const int64_t n0 = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (n0 >= N) return;
  for (int64_t k = blockIdx.y; k < K; k += gridDim.y) {
    if (upper && n0 + 3 < k) return;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (vec) {
      *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(in + k * ld_in + n0);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n0 + j < N) v[j] = in[k * ld_in + n0 + j];
    }
    __nv_bfloat16 t[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) split3(v[j], t[0][j], t[1][j], t[2][j]);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      __nv_bfloat16* o = out + (p * K + k) * ld_out + n0;
      if (vec) {
        *reinterpret_cast<uint2*>(o) = make_uint2(bf16_pair(t[p][0], t[p][1]), bf16_pair(t[p][2], t[p][3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n0 + j < N) o[j] = t[p][j];
      }
    }
  }
}

int split3_rows(const float* in, int64_t ld_in, int64_t K, int64_t N, __nv_bfloat16* out, int64_t ld_out, bool upper,
                cudaStream_t st) {
  const int64_t bx = (N + 1023) / 1024;
  int64_t by = ((int64_t)sm_count() * 16 + bx - 1) / bx;
  if (by > K) by = K;
  split3_rows_kernel<<<dim3((unsigned)bx, (unsigned)by), 256, 0, st>>>(in, ld_in, K, N, out, ld_out, upper);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

// in [R, K] fp32 (row stride ld_in) -> out: three planes [K, ld_out] bf16 holding the transposed terms:
// plane p, row k, column r = term p of in[r, k]; ld_out is a multiple of 64 and out 4-byte aligned.  Tiles of 64 rows x 32
// columns through shared memory, stored as pairs of rows (128 contiguous bytes a warp).
__global__ void __launch_bounds__(256) transpose_split3_kernel(const float* __restrict__ in, int64_t ld_in, int64_t R,
                                                               int64_t K, __nv_bfloat16* __restrict__ out, int64_t ld_out) {
  __shared__ float tile[64][33];
  const int64_t r0 = (int64_t)blockIdx.x * 64, k0 = (int64_t)blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int rr = ty; rr < 64; rr += 8)
    tile[rr][tx] = (r0 + rr < R && k0 + tx < K) ? in[(r0 + rr) * ld_in + k0 + tx] : 0.0f;
  __syncthreads();
#pragma unroll
  for (int kk = ty; kk < 32; kk += 8) {
    if (k0 + kk < K) {
      __nv_bfloat16 h[2], m[2], l[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) split3(tile[2 * tx + j][kk], h[j], m[j], l[j]);
      uint32_t* o = reinterpret_cast<uint32_t*>(out + (k0 + kk) * ld_out + r0) + tx;
      o[0] = bf16_pair(h[0], h[1]);
      o[K * ld_out / 2] = bf16_pair(m[0], m[1]);
      o[K * ld_out] = bf16_pair(l[0], l[1]);
    }
  }
}

int64_t round64(int64_t x) { return (x + 63) & ~(int64_t)63; }

// C[M, N] (row stride ldc) = beta * C + alpha * A B with fp32-level accuracy on the tensor cores:
// A [M, K] row-major (lda); B [K, N] row-major (ldb), or B == nullptr for B = (the first N rows of A)^T:
// with N == M the symmetric rank-K update (only the tiles touching the lower triangle are computed), with
// N < M its first N columns.  Both factors are split
// into three bf16 terms and the six leading cross products (hi*hi, hi*mid, mid*hi, hi*lo, lo*hi, mid*mid;
// the dropped ones are below 2^-24 relative) are accumulated in fp32 in one launch whose K dimension is
// the concatenation of the six slabs.  K must be a multiple of 64.
int tc_gemm3(float* C, int64_t ldc, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B,
             int64_t ldb, float alpha, float beta, __nv_bfloat16* ws, int32_t* error_flag, cudaStream_t st, int tri = 0) {
  static const int pa[6] = {0, 0, 1, 0, 2, 1}, pb[6] = {0, 1, 0, 2, 0, 1};
  const int64_t ldat = round64(M);
  __nv_bfloat16* at3 = ws;
  dim3 tgrid((unsigned)(ldat / 64), (unsigned)((K + 31) / 32));
  transpose_split3_kernel<<<tgrid, 256, 0, st>>>(A, lda, M, K, at3, ldat);
  FPQ_CHECK_LAUNCH();
  const __nv_bfloat16* b3 = at3;
  int64_t ldbt = ldat;
  if (B) {
    ldbt = round64(N);
    __nv_bfloat16* bw = ws + 3 * K * ldat;
    if (int rc = split3_rows(B, ldb, K, N, bw, ldbt, false, st)) return rc;
    b3 = bw;
  }
  int a_y[6], b_y[6];
  for (int t = 0; t < 6; ++t) {
    a_y[t] = (int)(pa[t] * K);
    b_y[t] = (int)(pb[t] * K);
  }
  return gemm_atb_bf16(C, ldc, M, N, at3, ldat, 3 * K, 0, b3, ldbt, 3 * K, 0, B == nullptr && N == M, false, 6, K, a_y,
                       b_y, alpha, beta, error_flag, st, tri);
}

// Products at least this large go to the tensor cores; smaller ones stay on the fp32 SIMT kernel, whose
// launch is cheaper than the two conversion passes.
bool tc_worthwhile(int64_t M, int64_t N, int64_t K) {
  return K % 64 == 0 && M * N * K >= ((int64_t)1 << 25);
}

// X = L^-1 given the inverses of the diagonal blocks already in X.  The block range [lo, hi) is halved
// recursively: L^-1 = [[X11, 0], [-X22 (L21 X11), X22]], S = L21 X11 (n2 x n1) goes to `scratch`.  The
// nodes of one depth are independent, so the tree is walked level by level from the leaves: the small
// nodes of a level share two launches of the batched fp32 kernel (S for all of them, then X21 for all of
// them), the large ones go to the tensor cores one after the other.
struct TriNode { int lo, mid, hi; };

void tri_collect(std::vector<std::vector<TriNode>>& levels, int lo, int hi, int depth) {
  if (hi - lo <= 1) return;
  const int mid = (lo + hi) / 2;
  if ((int)levels.size() <= depth) levels.resize(depth + 1);
  levels[depth].push_back({lo, mid, hi});
  tri_collect(levels, lo, mid, depth + 1);
  tri_collect(levels, mid, hi, depth + 1);
}

int tri_inverse_levels(const float* L, float* X, float* scratch, __nv_bfloat16* ws, int32_t* error_flag, int64_t d,
                       int nblk, cudaStream_t st) {
  std::vector<std::vector<TriNode>> levels;
  tri_collect(levels, 0, nblk, 0);
  for (int depth = (int)levels.size() - 1; depth >= 0; --depth) {
    std::vector<TriNode> big;
    SgemmBatch s1{}, s2{};
    int64_t used = 0;
    auto flush = [&]() -> int {
      if (s1.count == 0) return FPQ_OK;
      if (int rc = sgemm_batched(s1, false, st)) return rc;
      if (int rc = sgemm_batched(s2, false, st)) return rc;
      s1.count = s2.count = 0;
      used = 0;
      return FPQ_OK;
    };
    for (const TriNode& nd : levels[depth]) {
      const int64_t r0 = (int64_t)nd.lo * NB, r1 = (int64_t)nd.mid * NB;
      const int64_t n1 = r1 - r0;
      int64_t n2 = (int64_t)nd.hi * NB - r1;
      if (r1 + n2 > d) n2 = d - r1;
      if (tc_worthwhile(n2, n1, n1) && n2 % 64 == 0) {
        big.push_back(nd);
        continue;
      }
      if (s1.count == SGEMM_MAX_BATCH)
        if (int rc = flush()) return rc;
      float* S = scratch + used;
      used += n1 * n2;
      SgemmArgs& a = s1.e[s1.count++];          // S = L21 * X11
      a = SgemmArgs{};
      a.A = L + r1 * d + r0; a.lda = d;
      a.B = X + r0 * d + r0; a.ldb = d;
      a.C = S; a.ldc = n1;
      a.M = (int)n2; a.N = (int)n1; a.K = (int)n1; a.alpha = 1.0f; a.beta = 0.0f;
      SgemmArgs& b = s2.e[s2.count++];          // X21 = -X22 * S
      b = SgemmArgs{};
      b.A = X + r1 * d + r1; b.lda = d;
      b.B = S; b.ldb = n1;
      b.C = X + r1 * d + r0; b.ldc = d;
      b.M = (int)n2; b.N = (int)n1; b.K = (int)n2; b.alpha = -1.0f; b.beta = 0.0f;
    }
    if (int rc = flush()) return rc;
    for (const TriNode& nd : big) {
      const int64_t r0 = (int64_t)nd.lo * NB, r1 = (int64_t)nd.mid * NB;
      const int64_t n1 = r1 - r0;
      int64_t n2 = (int64_t)nd.hi * NB - r1;
      if (r1 + n2 > d) n2 = d - r1;
      // S = L21 * X11 (X11 lower triangular), then X21 = -X22 * S (X22 lower triangular): the stages that
      // would only multiply the zero halves are skipped
      if (int rc = tc_gemm3(scratch, n1, n2, n1, n1, L + r1 * d + r0, d, X + r0 * d + r0, d, 1.0f, 0.0f, ws, error_flag, st, 1))
        return rc;
      if (int rc = tc_gemm3(X + r1 * d + r0, d, n2, n1, n2, X + r1 * d + r1, d, scratch, n1, -1.0f, 0.0f, ws, error_flag, st, 2))
        return rc;
    }
  }
  return FPQ_OK;
}

// ------------------------------------------------------------------ GPTQ column block
// Four threads per weight row, each holding 32 of the block's 128 columns in registers.  Columns are
// walked left to right: the owner of column i quantises it with the row's static group scale and
// turns the residual into err = (w - wq) / U[i,i]; the error is broadcast inside the quad and every
// thread subtracts err * U[i, j] from its columns j > i (src/quantization/gptq.py:166-186), in the
// same order as the reference applies them.  U's diagonal block sits in shared memory; a quad reads
// four 16-byte pieces of one row per load.  The outer loop over the four 32-column owners is a real
// loop (the unrolled body of 32 steps stays inside the instruction cache: a fully unrolled
// thread-per-row version was instruction-fetch bound at three warps per SM).  Afterwards each thread
// writes its 32 errors (as the transposed three-term bf16 operand of the trailing update), the dequantised values, rebuilt
// as grid(code) * scale exactly as they were computed, and its 16 code bytes.
constexpr int SUB = 32;   // columns per thread
// Shared-memory image of U's diagonal block: every 32-column piece of a row is shifted by another
// 16 bytes, so that the four pieces a quad reads with one 128-bit load start in different banks.
constexpr int US_LD = NB + 4 * (NB / SUB);
__device__ __forceinline__ int us_col(int col) { return col + 4 * (col / SUB); }

// Correctly rounded y / s from r = rcp(s): multiply and two fused residual corrections (valid while s, r and
// the quotient stay in the normal range; the caller checks s).
__device__ __forceinline__ float div_by(float y, float s, float r) {
  float q = y * r;
  float e = fmaf(-s, q, y);
  q = fmaf(e, r, q);
  e = fmaf(-s, q, y);
  return fmaf(e, r, q);
}
__device__ __forceinline__ bool rcp_safe(float s) {
  const float a = fabsf(s);
  return a > 7.8886e-31f /* 2^-100 */ && a < 1.2676e30f /* 2^100 */;
}
// E2M1 code of v (round to nearest, ties to even, saturating; every zero as 0x8) and its grid value.
__device__ __forceinline__ uint32_t e2m1_code_hw(float v, float& value) {
  uint32_t byte;
  asm("{ .reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; cvt.u32.u8 %0, t; }" : "=r"(byte) : "f"(0.0f), "f"(v));
  uint32_t code = byte & 0xFu;
  if ((code & 7u) == 0u) code = 8u;
  uint32_t h2;
  asm("{ .reg .b8 t; cvt.u8.u32 t, %1; cvt.rn.f16x2.e2m1x2 %0, t; }" : "=r"(h2) : "r"(code));
  value = __half2float(__ushort_as_half((unsigned short)(h2 & 0xffffu)));
  return code;
}

// G = 16 / 32: column c uses scale group c / G.  G = 1: activation order -- the columns were permuted
// beforehand and column c uses group gidx[c] of the n_groups static groups (gptq.py:146-148, 170-171);
// every thread then keeps one scale per column, so blocks are limited to 256 threads.
template <int G>
__global__ void __launch_bounds__(G == 1 ? 256 : 512) gptq_block_kernel(float* __restrict__ W, int64_t rows, int64_t C,
                                                                        int64_t c1, const float* __restrict__ scales,
                                                                        const float* __restrict__ U,
                                                                        __nv_bfloat16* __restrict__ ErrT3, int64_t lda, int64_t plane,
                                                                        uint8_t* __restrict__ codes,
                                                                        const int32_t* __restrict__ gidx, int n_groups) {
  extern __shared__ float Us[];   // NB rows of US_LD floats, then the reciprocals of the diagonal
  float* rdiag = Us + NB * US_LD;
  for (int idx = threadIdx.x; idx < NB * NB / 4; idx += blockDim.x) {
    const int i = (idx * 4) / NB, j = (idx * 4) % NB;
    *reinterpret_cast<float4*>(&Us[i * US_LD + us_col(j)]) = *reinterpret_cast<const float4*>(&U[(c1 + i) * C + c1 + j]);
  }
  bool safe = true;                                        // every division of this warp may take the reciprocal form
  for (int i = threadIdx.x; i < NB; i += blockDim.x) {
    const float dgl = U[(c1 + i) * C + c1 + i];
    rdiag[i] = rcp_safe(dgl) ? __frcp_rn(dgl) : 0.0f;      // 0 marks "divide the slow way"
    safe &= rcp_safe(dgl);
  }
  safe = __syncthreads_and(safe);
  const int lane = threadIdx.x & 31;
  const int q = lane & 3;                      // which 32 columns of the block are mine
  int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  const bool live = row < rows;
  if (!live) row = rows - 1;                   // keep the quad's shuffles uniform; nothing is stored

  constexpr int NGRP = SUB / G;
  float sc[NGRP], rsc[G == 1 ? 1 : NGRP];
#pragma unroll
  for (int g = 0; g < NGRP; ++g) {
    if (G == 1) {
      sc[g] = scales[row * n_groups + gidx[c1 + SUB * q + g]];
    } else {
      sc[g] = scales[row * (C / G) + (c1 + SUB * q) / G + g];
      rsc[g] = rcp_safe(sc[g]) ? __frcp_rn(sc[g]) : 0.0f;
      safe &= rcp_safe(sc[g]);
    }
  }
  safe = G != 1 && __all_sync(0xffffffffu, safe);
  float w[SUB], err[SUB];
  {
    const float4* wp = reinterpret_cast<const float4*>(W + row * C + c1 + SUB * q);
#pragma unroll
    for (int v = 0; v < SUB / 4; ++v) {
      const float4 t = wp[v];
      w[4 * v] = t.x; w[4 * v + 1] = t.y; w[4 * v + 2] = t.z; w[4 * v + 3] = t.w;
    }
  }
  uint32_t cw[SUB / 8];
#pragma unroll
  for (int v = 0; v < SUB / 8; ++v) cw[v] = 0;
#pragma unroll
  for (int j = 0; j < SUB; ++j) err[j] = 0.0f;

  const auto update = [&](const float* Ub, int b, int ii, float e) {
    const float e_ge = q >= b ? -e : 0.0f;   // applies to my columns right of ii when I am the owner or later
    const float e_gt = q > b ? -e : 0.0f;    // applies to all my columns only when I come after the owner
    const float4* up = reinterpret_cast<const float4*>(Ub + ii * US_LD + (SUB + 4) * q);
#pragma unroll
    for (int v = 0; v < SUB / 4; ++v) {
      const float4 u = up[v];
      w[4 * v] = fmaf(4 * v > ii ? e_ge : e_gt, u.x, w[4 * v]);
      w[4 * v + 1] = fmaf(4 * v + 1 > ii ? e_ge : e_gt, u.y, w[4 * v + 1]);
      w[4 * v + 2] = fmaf(4 * v + 2 > ii ? e_ge : e_gt, u.z, w[4 * v + 2]);
      w[4 * v + 3] = fmaf(4 * v + 3 > ii ? e_ge : e_gt, u.w, w[4 * v + 3]);
    }
  };
  // w / s and (w - wq) / U[i,i] as IEEE divisions (the reference's), computed from reciprocals where those are safe.
  // All lanes walk through the owner's arithmetic and only its results are taken: without a branch the 32 steps are
  // straight code in which the updates of one step fill the latencies of the next one's chain of dependent operations:
  // 32 us a block of 4096 rows instead of 44, 49 us of 14336 rows instead of 55 (there the shared-memory reads of U bind).
  if (safe) {
#pragma unroll 1
    for (int b = 0; b < NB / SUB; ++b) {
      const bool owner = q == b;
      const float* Ub = Us + (SUB * b) * US_LD;  // rows of U for the owner's columns
#pragma unroll
      for (int ii = 0; ii < SUB; ++ii) {
        const float s = sc[ii / G], rs = rsc[G == 1 ? 0 : ii / G];
        float gv;
        const uint32_t code = e2m1_code_hw(div_by(w[ii], s, rs), gv);
        const float diff = __fsub_rn(w[ii], __fmul_rn(gv, s));
        float e = div_by(diff, Ub[ii * US_LD + (SUB + 4) * b + ii], rdiag[SUB * b + ii]);
        cw[ii / 8] |= (owner ? code : 0u) << (4 * (ii % 8));
        err[ii] = owner ? e : err[ii];
        e = __shfl_sync(0xffffffffu, e, (lane & ~3) | b);
        update(Ub, b, ii, e);
      }
    }
  } else {
#pragma unroll 1
    for (int b = 0; b < NB / SUB; ++b) {
      const bool owner = q == b;
      const float* Ub = Us + (SUB * b) * US_LD;
#pragma unroll
      for (int ii = 0; ii < SUB; ++ii) {
        float e = 0.0f;
        if (owner) {
          const float s = sc[ii / G];
          const float rs = G == 1 ? (rcp_safe(s) ? __frcp_rn(s) : 0.0f) : rsc[G == 1 ? 0 : ii / G];
          const float qv = rs != 0.0f ? div_by(w[ii], s, rs) : __fdiv_rn(w[ii], s);
          float gv;
          const uint32_t code = e2m1_code_hw(qv, gv);
          cw[ii / 8] |= code << (4 * (ii % 8));
          const float wq = __fmul_rn(gv, s);
          const float dgl = Ub[ii * US_LD + (SUB + 4) * b + ii], rd = rdiag[SUB * b + ii];
          const float diff = __fsub_rn(w[ii], wq);
          e = rd != 0.0f ? div_by(diff, dgl, rd) : __fdiv_rn(diff, dgl);
          err[ii] = e;
        }
        e = __shfl_sync(0xffffffffu, e, (lane & ~3) | b);
        update(Ub, b, ii, e);
      }
    }
  }
  // The block's errors leave as the operand of the trailing update: three bf16 terms per value, transposed
  // (plane p of column c is row c of the block, `plane` elements apart).  They are staged in shared memory (the image
  // of U is no longer needed) so that the global stores run along the rows.
  const int rb = (int)(blockDim.x >> 2);            // rows of this block
  const int es_ld = rb + 1;
  const int r_local = (int)(threadIdx.x >> 2);
  __syncthreads();                                  // every warp has finished reading Us
  float* Es = Us;
#pragma unroll
  for (int j = 0; j < SUB; ++j) Es[(SUB * q + j) * es_ld + r_local] = err[j];
  __syncthreads();
  {
    const int64_t row0 = (int64_t)blockIdx.x * rb;
    const int pairs = rb >> 1;
    for (int idx = (int)threadIdx.x; idx < NB * pairs; idx += (int)blockDim.x) {
      const int c = idx / pairs, r0 = 2 * (idx - c * pairs);
      const int64_t g = row0 + r0;
      if (g >= lda) continue;                       // lda is even and >= rows: g + 1 < lda as well
      const float v0 = g < rows ? Es[c * es_ld + r0] : 0.0f;
      const float v1 = g + 1 < rows ? Es[c * es_ld + r0 + 1] : 0.0f;
      __nv_bfloat16 h0, m0, l0, h1, m1, l1;
      split3(v0, h0, m0, l0);
      split3(v1, h1, m1, l1);
      __nv_bfloat16* dst = ErrT3 + (int64_t)c * lda + g;
      *reinterpret_cast<__nv_bfloat162*>(dst) = __halves2bfloat162(h0, h1);
      *reinterpret_cast<__nv_bfloat162*>(dst + plane) = __halves2bfloat162(m0, m1);
      *reinterpret_cast<__nv_bfloat162*>(dst + 2 * plane) = __halves2bfloat162(l0, l1);
    }
  }
  if (!live) return;

  float4* op = reinterpret_cast<float4*>(W + row * C + c1 + SUB * q);
#pragma unroll
  for (int v = 0; v < SUB / 4; ++v) {
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = 4 * v + j;
      o[j] = __fmul_rn(e2m1_value((cw[i / 8] >> (4 * (i % 8))) & 15u), sc[i / G]);
    }
    op[v] = make_float4(o[0], o[1], o[2], o[3]);
  }
  if (codes)
    *reinterpret_cast<uint4*>(codes + row * (C / 2) + (c1 + SUB * q) / 2) = make_uint4(cw[0], cw[1], cw[2], cw[3]);
}

__global__ void diff_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = a[i] - b[i];
}

// x (or x - y) in fp32 -> two bf16 terms hi + lo (relative residual ~2^-17)
__global__ void split_bf16_kernel(const float* __restrict__ x, const float* __restrict__ y, __nv_bfloat16* __restrict__ hi,
                                  __nv_bfloat16* __restrict__ lo, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = y ? x[i] - y[i] : x[i];
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    hi[i] = h;
    lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
  }
}

// Deterministic reductions of the relative-MSE metric: every CTA writes the sum of its part to a slot of
// its own (nothing is added atomically), and one warp adds the slots in a fixed order at the end.
constexpr int MSE_DOT_BLOCKS = 1024;      // CTAs (and slots) of one frobenius_dot_kernel launch
constexpr int MSE_REGION = FPQ_RELATIVE_MSE_ACC_DOUBLES / 2;   // slots per quantity (numerator / denominator)

// partial[blockIdx.x] = weight * sum over this CTA's elements of a .* b
__global__ void __launch_bounds__(256) frobenius_dot_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                            int64_t n, double weight, double* partial) {
  __shared__ double warp_sum[8];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s += (double)a[i] * (double)b[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += warp_sum[w];
    partial[blockIdx.x] = weight * t;
  }
}

// out = mean(num) / (mean(den) + 1e-6), src/quantization/gptq.py:28-30; num / den = the sums of the first
// n_slots slots of the two regions, each lane adding its slots in index order, then a fixed shuffle tree.
__global__ void ratio_kernel(const double* acc, int n_slots, float* out, double count) {
  double v[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n_slots; i += 32) s += acc[(size_t)q * MSE_REGION + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    v[q] = s;
  }
  if (threadIdx.x == 0) out[0] = (float)((v[0] / count) / (v[1] / count + 1e-6));
}

}  // namespace
}  // namespace fpq

using namespace fpq;

extern "C" int fpq_hessian_prepare(float* H, int64_t d, const float* W, int64_t rows, float rel_damp,
                                   uint8_t* workspace, fpq_stream_t stream) {
  FPQ_CHECK_ARG(H && W && workspace, "NULL pointer");
  FPQ_CHECK_ARG(d > 0 && d <= (1 << 20) && rows > 0, "bad shape");
  cudaStream_t st = (cudaStream_t)stream;
  dead_columns_kernel<<<(unsigned)((d + 255) / 256), 256, 0, st>>>(W, rows, d, workspace);
  FPQ_CHECK_LAUNCH();
  mask_dead_kernel<<<dim3((unsigned)((d + 255) / 256), (unsigned)((d + 15) / 16)), 256, 0, st>>>(H, d, workspace);
  FPQ_CHECK_LAUNCH();
  damp_kernel<<<1, 256, 0, st>>>(H, d, rel_damp);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

// Scratch of fpq_hessian_prepare_noalloc: one "column is dead" flag per input channel.  It lives in
// the library image, so every GPU that loads the library holds these bytes until the process exits.
static __device__ __align__(256) uint8_t g_prepare_scratch[FPQ_PREPARE_NOALLOC_MAX_D];

extern "C" int fpq_hessian_prepare_noalloc(float* H, int64_t d, const float* W, int64_t rows, float rel_damp,
                                           fpq_stream_t stream) {
  FPQ_CHECK_ARG(H && W, "NULL pointer");
  FPQ_CHECK_ARG(d > 0 && rows > 0, "bad shape");
  FPQ_CHECK_ARG(d <= FPQ_PREPARE_NOALLOC_MAX_D,
                "d = %lld exceeds the built-in scratch of fpq_hessian_prepare_noalloc (%d input channels); "
                "use fpq_hessian_prepare with a caller-provided workspace",
                (long long)d, FPQ_PREPARE_NOALLOC_MAX_D);
  // The array's name is only a host-side handle; kernels need its device address, which differs per
  // GPU.  Resolve it once per device, with that device current.
  static std::atomic<uint8_t*> scratch_of_device[64];      // two threads making the first call store the same address
  int dev = 0;
  FPQ_CHECK_CUDA(cudaGetDevice(&dev));
  FPQ_CHECK_ARG(dev >= 0 && dev < 64, "device index %d out of range", dev);
  // The scratch is the current device's copy of the array, so H, W and the stream must belong to the
  // current device: a Hessian on another GPU would be masked with flags this GPU never wrote.
  cudaPointerAttributes attr{};
  FPQ_CHECK_CUDA(cudaPointerGetAttributes(&attr, H));
  FPQ_CHECK_ARG(attr.type != cudaMemoryTypeDevice || attr.device == dev,
                "H lives on device %d but the current device is %d: make the device that owns H current", attr.device, dev);
  uint8_t* scratch = scratch_of_device[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) {
    FPQ_CHECK_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&scratch), g_prepare_scratch));
    FPQ_CHECK_ARG(scratch != nullptr, "cudaGetSymbolAddress returned a null scratch address");
    scratch_of_device[dev].store(scratch, std::memory_order_release);
  }
  cudaStream_t st = (cudaStream_t)stream;
  // Every flag in [0, d) is rewritten before it is read, so nothing needs clearing between calls.
  dead_columns_kernel<<<(unsigned)((d + 255) / 256), 256, 0, st>>>(W, rows, d, scratch);
  FPQ_CHECK_LAUNCH();
  mask_dead_kernel<<<dim3((unsigned)((d + 255) / 256), (unsigned)((d + 15) / 16)), 256, 0, st>>>(H, d, scratch);
  FPQ_CHECK_LAUNCH();
  damp_kernel<<<1, 256, 0, st>>>(H, d, rel_damp);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

extern "C" int64_t fpq_cholesky_workspace_floats(int64_t d) {
  // L (d x d) | scratch of the triangular inverse (half x half) | bf16 operand splits (6 half^2 bf16 = 3 half^2 floats)
  const int64_t nblk = (d + NB - 1) / NB;
  const int64_t half = ((nblk + 1) / 2) * NB;
  return d * d + 4 * half * half + 64;
}

extern "C" int fpq_cholesky_inverse_upper(const float* H, float* U, int64_t d, float* workspace, int32_t* status,
                                          int32_t* error_flag, fpq_stream_t stream) {
  FPQ_CHECK_ARG(H && U && workspace && status && error_flag, "NULL pointer");
  FPQ_CHECK_ARG(d > 0 && d < (1ll << 30), "bad size");
  FPQ_CHECK_ARG(H != U, "U must not alias H");
  FPQ_CHECK_ARG(((uintptr_t)workspace & 15) == 0, "workspace must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const int nblk = (int)((d + NB - 1) / NB);
  const int64_t half = (int64_t)((nblk + 1) / 2) * NB;
  float* L = workspace;
  float* scratch = workspace + ((d * d + 3) & ~(int64_t)3);
  __nv_bfloat16* ws = reinterpret_cast<__nv_bfloat16*>(scratch + half * half);
  static bool configured[64] = {};
  int dev = 0;
  FPQ_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !configured[dev]) {
    FPQ_CHECK_CUDA(cudaFuncSetAttribute(chol_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CD_SMEM));
    FPQ_CHECK_CUDA(cudaFuncSetAttribute(chol_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PANEL_SMEM));
    if (dev < 64) configured[dev] = true;
  }
  FPQ_CHECK_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), st));
  reverse_copy_kernel<<<grid1d(d * d), 256, 0, st>>>(H, L, d);
  FPQ_CHECK_LAUNCH();
  FPQ_CHECK_CUDA(cudaMemsetAsync(U, 0, (size_t)d * d * sizeof(float), st));
  // Right-looking blocked Cholesky in two levels.  Inside an outer block of OB diagonal blocks the rank-128
  // updates only touch the outer block's own columns (all rows below); the rest of the trailing matrix gets
  // one rank-(OB*128) update per outer block, which reads and writes it 1/OB as often as a rank-128
  // update per diagonal block would (those updates are bound by that traffic, not by the tensor pipe).
  constexpr int OB = 4;
  const int64_t ws_elems = 6 * half * half;
  for (int ob = 0; ob < nblk; ob += OB) {
    const int64_t R = (int64_t)ob * NB;
    const int64_t Wd = (d - R) < (int64_t)OB * NB ? (d - R) : (int64_t)OB * NB;
    for (int k = ob; k < nblk && k < ob + OB; ++k) {
      const int64_t r = (int64_t)k * NB;
      const int nb = (int)((d - r) < NB ? (d - r) : NB);
      chol_diag_kernel<<<1, 256, CD_SMEM, st>>>(L + r * d + r, d, U + r * d + r, d, nb, status);
      FPQ_CHECK_LAUNCH();
      const int64_t below = d - (r + nb);
      if (below <= 0) break;
      // panel: L21 = A21 L11^-T, in place (a block with rows below it is a whole one)
      chol_panel_kernel<<<(unsigned)((below + PANEL_ROWS - 1) / PANEL_ROWS), 256, PANEL_SMEM, st>>>(
          L + (r + nb) * d + r, d, below, U + r * d + r, d);
      FPQ_CHECK_LAUNCH();
      // inner update: columns [r + nb, R + Wd) of the rows below -= L21 * (the first rows of L21)^T
      const int64_t inner = R + Wd - (r + nb);
      if (inner <= 0) continue;
      float* Cin = L + (r + nb) * d + (r + nb);
      if (nb == NB && tc_worthwhile(below, inner, nb) &&
          3 * (int64_t)nb * round64(below) <= ws_elems) {
        if (int rc = tc_gemm3(Cin, d, below, inner, nb, L + (r + nb) * d + r, d, nullptr, 0, -1.0f, 1.0f, ws, error_flag, st))
          return rc;
        continue;
      }
      SgemmArgs a{};
      a.A = L + (r + nb) * d + r; a.lda = d;
      a.B = L + (r + nb) * d + r; a.ldb = d;
      a.C = Cin; a.ldc = d;
      a.M = (int)below; a.N = (int)inner; a.K = nb; a.alpha = -1.0f; a.beta = 1.0f;
      if (int rc = sgemm(a, true, inner == below ? SGEMM_LOWER : SGEMM_PLAIN, st)) return rc;
    }
    // outer update: A22 -= P P^T (lower tiles only), P = the outer block's columns of the rows below it
    const int64_t below_o = d - (R + Wd);
    if (below_o <= 0) break;
    float* C22 = L + (R + Wd) * d + (R + Wd);
    const float* P = L + (R + Wd) * d + R;
    if (Wd % 64 == 0 && tc_worthwhile(below_o, below_o, Wd) && 3 * Wd * round64(below_o) <= ws_elems) {
      if (int rc = tc_gemm3(C22, d, below_o, below_o, Wd, P, d, nullptr, 0, -1.0f, 1.0f, ws, error_flag, st)) return rc;
      continue;
    }
    SgemmArgs a{};
    a.A = P; a.lda = d;
    a.B = P; a.ldb = d;
    a.C = C22; a.ldc = d;
    a.M = (int)below_o; a.N = (int)below_o; a.K = (int)Wd; a.alpha = -1.0f; a.beta = 1.0f;
    if (int rc = sgemm(a, true, SGEMM_LOWER, st)) return rc;
  }
  if (int rc = tri_inverse_levels(L, U, scratch, ws, error_flag, d, nblk, st)) return rc;
  reflect_inplace_kernel<<<grid1d(d * d / 2), 256, 0, st>>>(U, d);   // U <- J X J (upper triangular)
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

namespace {
int64_t align256(int64_t x) { return (x + 255) & ~(int64_t)255; }
constexpr int64_t GPTQ_OB = 4;      // column blocks whose errors are applied to the rest of the weight together
int64_t gptq_lda(int64_t rows) { return (rows + 63) & ~(int64_t)63; }
}  // namespace

extern "C" int64_t fpq_gptq_workspace_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0) return 0;
  return align256(3 * GPTQ_OB * NB * gptq_lda(rows) * 2) + align256(3 * cols * cols * 2);
}

extern "C" int fpq_gptq_quantize(float* W, int64_t rows, int64_t cols, const float* scales, int group,
                                 const float* U, uint8_t* codes, void* workspace, int32_t* error_flag,
                                 fpq_stream_t stream) {
  return fpq_gptq_quantize_ordered(W, rows, cols, scales, group, nullptr, U, codes, workspace, error_flag, stream);
}

extern "C" int fpq_gptq_quantize_ordered(float* W, int64_t rows, int64_t cols, const float* scales, int group,
                                         const int32_t* group_index, const float* U, uint8_t* codes, void* workspace,
                                         int32_t* error_flag, fpq_stream_t stream) {
  FPQ_CHECK_ARG(W && scales && U && workspace && error_flag, "NULL pointer");
  FPQ_CHECK_ARG(group == 16 || group == 32, "group must be 16 (NVFP4) or 32 (MXFP4)");
  FPQ_CHECK_ARG(rows > 0 && cols > 0 && cols % NB == 0, "cols (%lld) must be a multiple of %d", (long long)cols, NB);
  FPQ_CHECK_ARG(rows < (1ll << 30) && 3 * cols < (1ll << 31), "shape too large");
  FPQ_CHECK_ARG(((uintptr_t)W & 15) == 0 && ((uintptr_t)U & 15) == 0 && ((uintptr_t)workspace & 255) == 0 &&
                    ((uintptr_t)codes & 15) == 0, "W, U, codes must be 16-byte aligned, the workspace 256-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  static bool configured[64] = {};
  int dev = 0;
  FPQ_CHECK_CUDA(cudaGetDevice(&dev));
  const int smem = (NB * US_LD + NB) * (int)sizeof(float);
  if (dev < 64 && !configured[dev]) {
    FPQ_CHECK_CUDA(cudaFuncSetAttribute(gptq_block_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    FPQ_CHECK_CUDA(cudaFuncSetAttribute(gptq_block_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    FPQ_CHECK_CUDA(cudaFuncSetAttribute(gptq_block_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured[dev] = true;
  }
  // workspace: transposed three-term bf16 split of the errors of GPTQ_OB blocks | three-term bf16 split of U
  const int64_t lda = gptq_lda(rows), err_rows = GPTQ_OB * NB, plane = err_rows * lda;
  uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
  __nv_bfloat16* errT3 = reinterpret_cast<__nv_bfloat16*>(ws);
  __nv_bfloat16* U3 = reinterpret_cast<__nv_bfloat16*>(ws + align256(3 * plane * 2));
  if (cols > NB)      // the updates read rows of a group only right of the group: the lower triangle is left out
    if (int rc = split3_rows(U, cols, cols, cols, U3, cols, true, st)) return rc;
  // The trailing update W[:, c2:] -= Err U[c1:c2, c2:] runs on the tensor cores: both factors are split
  // into three bf16 terms and the six leading cross products (hi*hi, hi*mid, mid*hi, hi*lo, lo*hi,
  // mid*mid; the dropped ones are below 2^-24 relative) are accumulated in fp32 as one GEMM whose K
  // dimension is the concatenation of the six 128-row slabs.
  static const int pa[6] = {0, 0, 1, 0, 2, 1}, pb[6] = {0, 1, 0, 2, 0, 1};
  // Four threads per row, eight rows per warp.  The kernel is bound by the latency of its 128 dependent
  // steps, so all rows should be resident at once: warps per block are chosen so that one block per SM
  // covers everything when that is possible (14336 rows: 13 warps on 138 SMs) instead of leaving a
  // handful of blocks for a second pass.
  const int64_t units = (rows + 7) / 8;
  int wpb = (int)((units + sm_count() - 1) / sm_count());
  const int wpb_max = group_index ? 8 : 16;
  wpb = wpb < 4 ? 4 : (wpb > wpb_max ? wpb_max : wpb);
  const unsigned threads = (unsigned)wpb * 32;
  const unsigned grid = (unsigned)((units + wpb - 1) / wpb);
  // The columns right of a block are updated in two levels: after a block only those of its group of GPTQ_OB blocks,
  // after a group all others with the errors of the whole group.  The rest of W is then read and written once per
  // group (it bounds the update of a single block: 128 columns of errors are 768 of K).  Every block keeps a chain of its
  // own in the tensor core, subtracted from W by a rounded fp32 addition, in the order of the blocks: an element sees
  // the same operations whether its group is one product or (where that is too small for the pair kernel, the one that
  // splits chains) a product per block, so the codes of a row do not depend on the number of rows.
  // Updates of a 14336 x 4096 loop 1.5 ms instead of 2.3 ms, of a 4096 x 14336 one 5.5 instead of 8.3.
  const auto update = [&](int64_t e0, int64_t n_rows, int64_t u0, int64_t col, int64_t n) -> int {
    int a_y[6 * GPTQ_OB], b_y[6 * GPTQ_OB], segs = 0;
    for (int64_t r = 0; r < n_rows; r += NB)
      for (int t = 0; t < 6; ++t, ++segs) {
        a_y[segs] = (int)(pa[t] * err_rows + e0 + r);
        b_y[segs] = (int)(pb[t] * cols + u0 + r);
      }
    return gemm_atb_bf16(W + col, cols, rows, n, errT3, lda, 3 * err_rows, 0, U3, cols, 3 * cols, col, false, false, segs, NB,
                         a_y, b_y, -1.0f, 1.0f, error_flag, st, 0, 6 * NB);
  };
  const int n_groups = (int)(cols / group);
  for (int64_t g1 = 0; g1 < cols; g1 += err_rows) {
    const int64_t g2 = g1 + err_rows < cols ? g1 + err_rows : cols;
    for (int64_t c1 = g1; c1 < g2; c1 += NB) {
      __nv_bfloat16* err = errT3 + (c1 - g1) * lda;
      if (group_index)
        gptq_block_kernel<1><<<grid, threads, smem, st>>>(W, rows, cols, c1, scales, U, err, lda, plane, codes, group_index, n_groups);
      else if (group == 16)
        gptq_block_kernel<16><<<grid, threads, smem, st>>>(W, rows, cols, c1, scales, U, err, lda, plane, codes, nullptr, n_groups);
      else
        gptq_block_kernel<32><<<grid, threads, smem, st>>>(W, rows, cols, c1, scales, U, err, lda, plane, codes, nullptr, n_groups);
      FPQ_CHECK_LAUNCH();
      if (c1 + NB < g2)
        if (int rc = update(c1 - g1, NB, c1, c1 + NB, g2 - (c1 + NB))) return rc;
    }
    if (g2 >= cols) break;
    if (gemm_atb_on_pairs(rows, cols - g2, false, (int)(6 * ((g2 - g1) / NB)), NB)) {
      if (int rc = update(0, g2 - g1, g1, g2, cols - g2)) return rc;
    } else {
      for (int64_t c1 = g1; c1 < g2; c1 += NB)
        if (int rc = update(c1 - g1, NB, c1, g2, cols - g2)) return rc;
    }
  }
  return FPQ_OK;
}

extern "C" int fpq_relative_mse(const float* Wq, const float* W, const float* H, int64_t rows, int64_t d,
                                float* diff_workspace, double* acc_workspace, float* out, fpq_stream_t stream) {
  FPQ_CHECK_ARG(Wq && W && H && diff_workspace && acc_workspace && out, "NULL pointer");
  const int64_t tiles = ((rows + 127) / 128) * ((d + 127) / 128);      // CTAs of one fp32 product = partial sums
  FPQ_CHECK_ARG(tiles <= MSE_REGION, "matrix too large for the %d partial-sum slots of the workspace", MSE_REGION);
  cudaStream_t st = (cudaStream_t)stream;
  diff_kernel<<<grid1d(rows * d), 256, 0, st>>>(Wq, W, diff_workspace, rows * d);
  FPQ_CHECK_LAUNCH();
  SgemmArgs a{};
  a.lda = d; a.B = H; a.ldb = d; a.M = (int)rows; a.N = (int)d; a.K = (int)d; a.alpha = 1.0f; a.ldd = d;
  a.A = diff_workspace; a.D = diff_workspace; a.dot_out = acc_workspace;
  if (int rc = sgemm(a, false, SGEMM_DOT, st)) return rc;
  a.A = W; a.D = W; a.dot_out = acc_workspace + MSE_REGION;
  if (int rc = sgemm(a, false, SGEMM_DOT, st)) return rc;
  ratio_kernel<<<1, 32, 0, st>>>(acc_workspace, (int)tiles, out, (double)rows * (double)d);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}

extern "C" int fpq_hessian_accumulate(float* H, int64_t d, const void* xa_bf16, const void* xb_bf16, int64_t tokens,
                                      float alpha, float beta, int32_t* error_flag, fpq_stream_t stream);

// Tensor-core form of the same metric:  sum((A H) .* A) = <H, A^T A>, and A^T A is a Hessian-type product.
// A (fp32) is split into two bf16 terms hi + lo; <H, A^T A> ~= <H, hi^T hi> + 2 <H, hi^T lo> (H is symmetric),
// accurate to ~1e-5 relative -- ample for a logged error metric, and ~10x faster than the fp32 products.
extern "C" int fpq_relative_mse_tc(const float* Wq, const float* W, const float* H, int64_t rows, int64_t d,
                                   void* bf16_workspace, float* gram_workspace, double* acc_workspace, float* out,
                                   int32_t* error_flag, fpq_stream_t stream) {
  FPQ_CHECK_ARG(Wq && W && H && bf16_workspace && gram_workspace && acc_workspace && out && error_flag, "NULL pointer");
  FPQ_CHECK_ARG(rows > 0 && d > 0 && d % 8 == 0, "d must be a positive multiple of 8");
  cudaStream_t st = (cudaStream_t)stream;
  __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(bf16_workspace);
  __nv_bfloat16* lo = hi + rows * d;
  // slots [0, 1024) and [1024, 2048) of a region take the two terms of a quantity
  for (int which = 0; which < 2; ++which) {
    double* region = acc_workspace + (size_t)which * MSE_REGION;
    split_bf16_kernel<<<grid1d(rows * d), 256, 0, st>>>(which == 0 ? Wq : W, which == 0 ? W : nullptr, hi, lo, rows * d);
    FPQ_CHECK_LAUNCH();
    if (int rc = fpq_hessian_accumulate(gram_workspace, d, hi, nullptr, rows, 1.0f, 0.0f, error_flag, stream)) return rc;
    frobenius_dot_kernel<<<MSE_DOT_BLOCKS, 256, 0, st>>>(H, gram_workspace, d * d, 1.0, region);
    FPQ_CHECK_LAUNCH();
    if (int rc = fpq_hessian_accumulate(gram_workspace, d, hi, lo, rows, 1.0f, 0.0f, error_flag, stream)) return rc;
    frobenius_dot_kernel<<<MSE_DOT_BLOCKS, 256, 0, st>>>(H, gram_workspace, d * d, 2.0, region + MSE_DOT_BLOCKS);
    FPQ_CHECK_LAUNCH();
  }
  ratio_kernel<<<1, 32, 0, st>>>(acc_workspace, 2 * MSE_DOT_BLOCKS, out, (double)rows * (double)d);
  FPQ_CHECK_LAUNCH();
  return FPQ_OK;
}
