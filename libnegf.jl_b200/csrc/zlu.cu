// Batched complex FP64 LU with partial pivoting (LAPACK getrf semantics) or
// without row interchanges (lu(A, NoPivot())), and triangular inverses of the
// factors.
//
// Used by the selected inverse (the reference's be_getrf! / be_trsm! /
// be_getri!, src/backend_cpu.jl:229-265, called from
// src/selected_inverse.jl:9-206): every triangular solve with a factor is
// applied as a tensor-core GEMM with the factor's explicit inverse.
//
// LU (right-looking, panel width nb):
//   panel kernel: rows [k0, n) x columns [k0, k0+w) in shared memory, pivot
//     search per column (|re|+|im|, first maximum, as izamax), row swaps and
//     rank-1 updates inside the panel; writes ipiv (0-based, global) and the
//     inverse of the unit-lower w x w block L11 into scratch;
//   swap kernel: applies the panel's row interchanges to all other columns
//     (LAPACK's zlaswp on both sides) and copies A12 into scratch;
//   GEMMs (engine): A12 = L11^{-1} A12,  A22 -= A21 A12.
// Without row interchanges (the selected inverse of NEGF matrices) no panel of
// whole columns is needed: a kernel factors a 32 x 32 diagonal block and inverts
// its triangles, a second one substitutes A21 U^{-1} and L^{-1} A12, and the
// engine forms the Schur update as a product.  Triangular inverse: diagonal blocks
// of 32 inverted in shared memory here, then pairs of blocks joined by products to
// 64, then block columns of that width.
#include "negf_common.cuh"

namespace negf {

constexpr int LU_THREADS = 256;

__global__ void __launch_bounds__(LU_THREADS)
    zgetrf_panel_kernel(const ZLuProblem* __restrict__ probs, int k0, int nb) {
  chain_entry();
  const ZLuProblem p = probs[blockIdx.x];
  const int n = p.n;
  if (k0 >= n) return;
  const int w = min(nb, n - k0);
  const int h = n - k0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* S = reinterpret_cast<cplx*>(smem_raw);   // h x w, column-major
  double* redv = reinterpret_cast<double*>(S + (size_t)h * w);
  int* redr = reinterpret_cast<int*>(redv + LU_THREADS / 32);
  int* sp = redr + LU_THREADS / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int idx = tid; idx < h * w; idx += LU_THREADS) {
    int c = idx / h, r = idx - c * h;
    S[idx] = p.A[(k0 + r) + (size_t)(k0 + c) * p.ld];
  }
  __syncthreads();
  for (int c = 0; c < w; ++c) {
    double bv = -1.0;
    int br = -1;
    for (int r = c + tid; r < h; r += LU_THREADS) {
      double v = cabs1(S[(size_t)c * h + r]);
      if (v > bv) { bv = v; br = r; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      double v2 = __shfl_down_sync(0xffffffffu, bv, off);
      int r2 = __shfl_down_sync(0xffffffffu, br, off);
      if (v2 > bv || (v2 == bv && r2 >= 0 && (br < 0 || r2 < br))) { bv = v2; br = r2; }
    }
    if (lane == 0) { redv[warp] = bv; redr[warp] = br; }
    __syncthreads();
    if (warp == 0) {
      bv = lane < LU_THREADS / 32 ? redv[lane] : -1.0;
      br = lane < LU_THREADS / 32 ? redr[lane] : -1;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        double v2 = __shfl_down_sync(0xffffffffu, bv, off);
        int r2 = __shfl_down_sync(0xffffffffu, br, off);
        if (v2 > bv || (v2 == bv && r2 >= 0 && (br < 0 || r2 < br))) { bv = v2; br = r2; }
      }
      if (lane == 0) {
        if (br < 0) br = c;
        *sp = br;
        if (bv <= 0.0 && p.info) atomicCAS(p.info, 0, k0 + c + 1);
      }
    }
    __syncthreads();
    const int pr = *sp;
    if (tid == 0) p.ipiv[k0 + c] = k0 + pr;
    if (pr != c)
      for (int j = tid; j < w; j += LU_THREADS) {
        cplx t = S[(size_t)j * h + c];
        S[(size_t)j * h + c] = S[(size_t)j * h + pr];
        S[(size_t)j * h + pr] = t;
      }
    __syncthreads();
    cplx piv = S[(size_t)c * h + c];
    cplx inv = (piv.x == 0.0 && piv.y == 0.0) ? make_double2(0.0, 0.0) : cinv(piv);
    for (int r = c + 1 + tid; r < h; r += LU_THREADS) S[(size_t)c * h + r] = cmul(S[(size_t)c * h + r], inv);
    __syncthreads();
    const int rows = h - c - 1, cols = w - c - 1;
    for (int idx = tid; idx < rows * cols; idx += LU_THREADS) {
      int j = c + 1 + idx / rows, r = c + 1 + idx % rows;
      S[(size_t)j * h + r] = cfms(S[(size_t)j * h + r], S[(size_t)c * h + r], S[(size_t)j * h + c]);
    }
    __syncthreads();
  }
  for (int idx = tid; idx < h * w; idx += LU_THREADS) {
    int c = idx / h, r = idx - c * h;
    p.A[(k0 + r) + (size_t)(k0 + c) * p.ld] = S[idx];
  }
  // inverse of the unit lower w x w block (forward substitution per column)
  if (p.Linv && w < n) {
    for (int j = tid; j < w; j += LU_THREADS) {
      for (int i = 0; i < w; ++i) {
        cplx v;
        if (i < j) v = make_double2(0.0, 0.0);
        else if (i == j) v = make_double2(1.0, 0.0);
        else {
          v = make_double2(0.0, 0.0);
          for (int k = j; k < i; ++k) v = cfms(v, S[(size_t)k * h + i], p.Linv[k + (size_t)j * w]);
        }
        p.Linv[i + (size_t)j * w] = v;
      }
    }
  }
}

// Row interchanges of panel [k0, k0+w) on every column outside the panel,
// then T = A[k0:k0+w, k0+w:n] (w x (n-k0-w), ld w).
__global__ void zlaswp_copy_kernel(const ZLuProblem* __restrict__ probs, int k0, int nb) {
  chain_entry();
  const ZLuProblem p = probs[blockIdx.y];
  const int n = p.n;
  if (k0 >= n) return;
  const int w = min(nb, n - k0);
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < n; col += gridDim.x * blockDim.x) {
    if (col >= k0 && col < k0 + w) continue;
    cplx* a = p.A + (size_t)col * p.ld;
    for (int c = 0; c < w; ++c) {
      int r1 = k0 + c, r2 = p.ipiv[k0 + c];
      if (r1 != r2) {
        cplx t = a[r1];
        a[r1] = a[r2];
        a[r2] = t;
      }
    }
    if (col >= k0 + w)
      for (int c = 0; c < w; ++c) p.T[c + (size_t)(col - k0 - w) * w] = a[k0 + c];
  }
}

// Inverse of one nb x nb diagonal block of the packed L\U factors:
// upper -> inverse of the non-unit upper triangle, else the inverse of the
// unit lower triangle.  X is the n x n output (zero elsewhere beforehand).
__global__ void ztrtri_diag_kernel(const ZTriProblem* __restrict__ probs, int nb, int upper) {
  chain_entry();
  const ZTriProblem p = probs[blockIdx.y];
  const int j0 = blockIdx.x * nb;
  if (j0 >= p.n) return;
  const int w = min(nb, p.n - j0);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* S = reinterpret_cast<cplx*>(smem_raw);  // w x w block
  cplx* X = S + (size_t)w * w;                   // w x w inverse
  for (int idx = threadIdx.x; idx < w * w; idx += blockDim.x) {
    int c = idx / w, r = idx - c * w;
    S[idx] = p.A[(j0 + r) + (size_t)(j0 + c) * p.lda];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < w; j += blockDim.x) {
    if (upper) {
      // X[:,j]: back substitution, X[i,j] = -(sum_{k=i+1..j} U[i,k] X[k,j]) / U[i,i]
      for (int i = w - 1; i >= 0; --i) {
        cplx v;
        if (i > j) v = make_double2(0.0, 0.0);
        else {
          cplx acc = (i == j) ? make_double2(1.0, 0.0) : make_double2(0.0, 0.0);
          for (int k = i + 1; k <= j; ++k) acc = cfms(acc, S[i + (size_t)k * w], X[k + (size_t)j * w]);
          cplx d = S[i + (size_t)i * w];
          v = (d.x == 0.0 && d.y == 0.0) ? make_double2(0.0, 0.0) : cmul(acc, cinv(d));
        }
        X[i + (size_t)j * w] = v;
      }
    } else {
      for (int i = 0; i < w; ++i) {
        cplx v;
        if (i < j) v = make_double2(0.0, 0.0);
        else if (i == j) v = make_double2(1.0, 0.0);
        else {
          v = make_double2(0.0, 0.0);
          for (int k = j; k < i; ++k) v = cfms(v, S[i + (size_t)k * w], X[k + (size_t)j * w]);
        }
        X[i + (size_t)j * w] = v;
      }
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < w * w; idx += blockDim.x) {
    int c = idx / w, r = idx - c * w;
    p.X[(j0 + r) + (size_t)(j0 + c) * p.ldx] = X[idx];
  }
}

// Unpivoted LU of the diagonal block [k0, k0 + w), w <= 32, and the inverses of
// both factors, in shared memory: thread (row = lane, columns = warp + 8 q).
// Step c takes l = S[:, c] / S[c, c] off the rows below -- of the block and of
// the growing L^{-1} -- and needs one barrier, since it writes neither row nor
// column c; the columns of L are divided at the end.  U^{-1} grows the same way
// from the last column up.
constexpr int kLuDiag = 32;
__global__ void __launch_bounds__(256)
    zlu_diag_kernel(const ZLuDiagProblem* __restrict__ probs, int k0) {
  chain_entry();
  const ZLuDiagProblem p = probs[blockIdx.x];
  if (k0 >= p.n) return;
  constexpr int LD = kLuDiag + 1;
  const int w = min(kLuDiag, p.n - k0), r = threadIdx.x & 31, j0 = threadIdx.x >> 5;
  // Y: L^{-1} below the diagonal, U^{-1} (rows not yet divided) above, ones on it
  constexpr int YO = kLuDiag * LD;
  __shared__ cplx S[2 * YO], inv[kLuDiag];
  cplx* const Y = S + YO;
#pragma unroll
  for (int j = j0; j < kLuDiag; j += 8) {
    const cplx one = make_double2(r == j ? 1.0 : 0.0, 0.0);
    S[j * LD + r] = r < w && j < w ? p.A[(k0 + r) + (size_t)(k0 + j) * p.ld] : one;
    Y[j * LD + r] = one;
  }
  // reciprocal of pivot c, by the thread of that element as soon as it is final:
  // in every thread the reciprocals would load the FP64 pipe as much as the updates
  auto pivot = [&](int c) {
    const cplx piv = S[c * LD + c];
    inv[c] = cinv_pivot(piv);
    if (piv.x == 0.0 && piv.y == 0.0 && p.info) atomicCAS(p.info, 0, k0 + c + 1);
  };
  if (threadIdx.x == 0) pivot(0);
  __syncthreads();
  for (int c = 0; c < w; ++c) {
    const cplx iv = inv[c];
    if (r > c) {
      const cplx l = cmul(S[c * LD + r], iv);
#pragma unroll
      for (int j = j0; j < kLuDiag; j += 8) {
        const int m = j * LD + (j > c ? 0 : YO);
        S[m + r] = cfms_fused(S[m + r], l, S[m + c]);
      }
      if (r == c + 1 && j0 == (r & 7) && r < w) pivot(r);
    }
    __syncthreads();
  }
  for (int c = w - 1; c > 0; --c) {
    if (r < c) {
      const cplx u = cmul(S[c * LD + r], inv[c]);
#pragma unroll
      for (int j = j0; j < kLuDiag; j += 8)
        if (j >= c) Y[j * LD + r] = cfms_fused(Y[j * LD + r], u, Y[j * LD + c]);
    }
    __syncthreads();
  }
  if (r < w)
    for (int j = j0; j < w; j += 8) {
      const size_t x = (size_t)(k0 + r) + (size_t)(k0 + j) * p.n;
      p.F[(k0 + r) + (size_t)(k0 + j) * p.ldf] = r > j ? cmul(S[j * LD + r], inv[j]) : S[j * LD + r];
      const cplx y = Y[j * LD + r], zero = make_double2(0.0, 0.0);
      p.Xl[x] = r >= j ? y : zero;
      p.Xu[x] = r <= j ? cmul(y, inv[r]) : zero;
    }
}

// F21 = A21 U^{-1} and F12 = L^{-1} A12 of a panel by substitution, a thread per
// row of A21 or column of A12.  (Products with the inverses of the diagonal block
// would be faster, but without row interchanges U may have small pivots: the
// selected inverse of NEGF matrices lost a digit.)
__global__ void __launch_bounds__(64) zlu_solve_kernel(const ZLuDiagProblem* __restrict__ probs, int k0, int chunks) {
  chain_entry();
  const ZLuDiagProblem p = probs[blockIdx.y];
  const int k1 = k0 + kLuDiag;
  const bool rows = (int)blockIdx.x < chunks;
  const int i = k1 + (blockIdx.x - (rows ? 0 : chunks)) * 64 + threadIdx.x;
  if (k1 + (int)(blockIdx.x - (rows ? 0 : chunks)) * 64 >= p.n) return;
  __shared__ cplx T[kLuDiag * kLuDiag], d[kLuDiag];
  for (int e = threadIdx.x; e < kLuDiag * kLuDiag; e += 64) {
    const int r = e % kLuDiag, c = e / kLuDiag;  // T[row][column] of U, or of L transposed
    T[rows ? r * kLuDiag + c : c * kLuDiag + r] = p.F[(k0 + r) + (size_t)(k0 + c) * p.ldf];
  }
  if (threadIdx.x < kLuDiag) {
    const size_t q = k0 + threadIdx.x;
    d[threadIdx.x] = p.Xu[q + q * p.n];
  }
  __syncthreads();
  if (i >= p.n) return;
  const cplx* src = rows ? p.A + i + (size_t)k0 * p.ld : p.A + k0 + (size_t)i * p.ld;
  cplx* dst = rows ? p.F + i + (size_t)k0 * p.ldf : p.F + k0 + (size_t)i * p.ldf;
  const size_t ss = rows ? p.ld : 1, ds = rows ? p.ldf : 1;
  // right-looking substitution; the current column is always x[0] (or y[0]), so
  // that the loops are not unrolled: the straight-line form was bound by its
  // instruction fetches (22 us).  The slots past the last column hold leftovers.
  cplx x[16], y[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    x[c] = src[c * ss];
    y[c] = src[(c + 16) * ss];
  }
#pragma unroll 1
  for (int c = 0; c < 16; ++c) {
    const cplx v = rows ? cmul(x[0], d[c]) : x[0];
    const cplx* t = T + c * kLuDiag;
    dst[c * ds] = v;
#pragma unroll
    for (int j = 1; j < 16; ++j) x[j - 1] = cfms_fused(x[j], v, t[min(c + j, 15)]);
#pragma unroll
    for (int j = 0; j < 16; ++j) y[j] = cfms_fused(y[j], v, t[16 + j]);
  }
#pragma unroll 1
  for (int c = 16; c < 32; ++c) {
    const cplx v = rows ? cmul(y[0], d[c]) : y[0];
    const cplx* t = T + c * kLuDiag;
    dst[c * ds] = v;
#pragma unroll
    for (int j = 1; j < 16; ++j) y[j - 1] = cfms_fused(y[j], v, t[min(c + j, 31)]);
  }
}

// max_n: the largest matrix; the panel at k0 is complete (k0 + 32 <= n) wherever rows follow it
cudaError_t launch_zlu_solve(const void* probs, int nprob, int k0, int max_n, cudaStream_t st) {
  const int rest = max_n - k0 - kLuDiag;
  if (nprob <= 0 || rest <= 0) return cudaSuccess;
  const int chunks = (rest + 63) / 64;
  for (int base = 0; base < nprob; base += 65535) {  // grid.y is limited to 65535
    const int cnt = nprob - base < 65535 ? nprob - base : 65535;
    launch_chained(zlu_solve_kernel, dim3(2 * chunks, cnt), 64, 0, st,
                   static_cast<const ZLuDiagProblem*>(probs) + base, k0, chunks);
  }
  return cudaGetLastError();
}

cudaError_t launch_zlu_diag(const void* probs, int nprob, int k0, cudaStream_t st) {
  if (nprob <= 0) return cudaSuccess;
  launch_chained(zlu_diag_kernel, nprob, 256, 0, st, static_cast<const ZLuDiagProblem*>(probs), k0);
  return cudaGetLastError();
}

size_t zgetrf_panel_smem_bytes(int n, int nb) {
  int w = nb < n ? nb : n;
  return ((size_t)n * w * sizeof(cplx) + (LU_THREADS / 32) * (sizeof(double) + sizeof(int)) + 16 + 15) & ~size_t(15);
}

size_t ztrtri_smem_bytes(int nb) { return 2 * (size_t)nb * nb * sizeof(cplx); }

// The shared-memory attributes are process-wide: set them to the device's
// opt-in maximum so that no later plan lowers a limit another one relies on.
cudaError_t zlu_prepare(size_t panel_smem, size_t tri_smem) {
  int dev = 0, mx = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&mx, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  if (panel_smem > (size_t)mx || tri_smem > (size_t)mx) return cudaErrorInvalidValue;
  if (panel_smem) e = cudaFuncSetAttribute(zgetrf_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  if (e == cudaSuccess && tri_smem)
    e = cudaFuncSetAttribute(ztrtri_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  return e;
}

cudaError_t launch_zgetrf_panel(const void* probs, int nprob, int k0, int nb, size_t smem, cudaStream_t st) {
  if (nprob <= 0) return cudaSuccess;
  launch_chained(zgetrf_panel_kernel, nprob, LU_THREADS, smem, st, static_cast<const ZLuProblem*>(probs), k0, nb);
  return cudaGetLastError();
}

cudaError_t launch_zlaswp_copy(const void* probs, int nprob, int k0, int nb, int max_n, cudaStream_t st) {
  if (nprob <= 0) return cudaSuccess;
  dim3 grid((max_n + 127) / 128, nprob);
  launch_chained(zlaswp_copy_kernel, grid, 128, 0, st, static_cast<const ZLuProblem*>(probs), k0, nb);
  return cudaGetLastError();
}

cudaError_t launch_ztrtri_diag(const void* probs, int nprob, int nb, int upper, int max_n, size_t smem,
                               cudaStream_t st) {
  if (nprob <= 0) return cudaSuccess;
  dim3 grid((max_n + nb - 1) / nb, nprob);
  launch_chained(ztrtri_diag_kernel, grid, 64, smem, st, static_cast<const ZTriProblem*>(probs), nb, upper);
  return cudaGetLastError();
}

}  // namespace negf
