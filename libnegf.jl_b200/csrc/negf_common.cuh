// Shared device/host definitions of the B200 NEGF block kernels.
//
// Element type: complex128 stored as double2 {re, im}, blocks column-major with
// a leading dimension (the layout of a Julia Matrix{ComplexF64}, which the
// reference's CPU backend hands to LAPACK, src/backend_cpu.jl:7-20).
#pragma once

#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>

namespace negf {

using cplx = double2;

// Marks the devices on which a set-up (kernel attributes) has been done; two
// threads that meet do it twice, which is harmless.
class PerDevice {
 public:
  bool done(int dev) const { return dev >= 0 && dev < 64 && ((mask_.load() >> dev) & 1); }
  void set(int dev) {
    if (dev >= 0 && dev < 64) mask_.fetch_or(1ull << dev);
  }

 private:
  std::atomic<unsigned long long> mask_{0};
};

__host__ __device__ inline cplx cmake(double r, double i) { return make_double2(r, i); }
__host__ __device__ inline cplx cadd(cplx a, cplx b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ inline cplx csub(cplx a, cplx b) { return make_double2(a.x - b.x, a.y - b.y); }
__host__ __device__ inline cplx cmul(cplx a, cplx b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ inline cplx cconj(cplx a) { return make_double2(a.x, -a.y); }
__host__ __device__ inline cplx cneg(cplx a) { return make_double2(-a.x, -a.y); }
// a - b*c
__host__ __device__ inline cplx cfms(cplx a, cplx b, cplx c) {
  return make_double2(a.x - (b.x * c.x - b.y * c.y), a.y - (b.x * c.y + b.y * c.x));
}
// 1/a (Smith's algorithm: scaled to avoid overflow in |a|^2)
__host__ __device__ inline cplx cinv(cplx a) {
  double ar = a.x, ai = a.y;
  if (fabs(ar) >= fabs(ai)) {
    double r = ai / ar, d = ar + ai * r;
    return make_double2(1.0 / d, -r / d);
  } else {
    double r = ar / ai, d = ai + ar * r;
    return make_double2(r / d, -1.0 / d);
  }
}
#ifdef __CUDACC__
// 1/a; 0 for a = 0 and where one part is infinite and the other finite, NaN for
// any other non-finite a, as cinv gives.  a is scaled by a power of two
// (exact), so that |a|^2 = d + dl (d the rounded sum, dl what it lost) lies
// within [2^-102, 32).  1/|a|^2 starts from a single-precision reciprocal x0 and
// takes one third-order Newton-Raphson step, x0 (1 + r + r^2) with r = 1 -
// (d + dl) x0: |r| < 2^-21, so the step's error r^3 is below the FP64 rounding.
// The step is applied to re x0 and im x0 with their own rounding errors, so each
// part is rounded once: mean error 0.38 u, at most 1.0 u (of d alone and a
// rounded 1/d: 0.66 and 2.8; cinv: 0.54 and 1.6).  No branch and no compare on
// the FP64 pipe: its latency is part of every column's, and dl and the products'
// errors are ready before x0.
__device__ __forceinline__ cplx cinv_pivot(cplx a) {
  const int hx = __double2hiint(a.x) & 0x7fffffff, hy = __double2hiint(a.y) & 0x7fffffff;
  const int e = max(hx, hy) >> 20;
  const double s = __hiloint2double(max(1, 2046 - e) << 20, 0);
  const double x = a.x * s, y = a.y * s;
  const double m = hx < hy ? y : x, q = hx < hy ? x : y;
  const double mm = __dmul_rn(m, m), qq = __dmul_rn(q, q), d = __dadd_rn(mm, qq);
  const double dl = __dadd_rn(__dsub_rn(qq, __dsub_rn(d, mm)), __dadd_rn(fma(m, m, -mm), fma(q, q, -qq)));
  float xf;
  asm("rcp.approx.f32 %0, %1;" : "=f"(xf) : "f"((float)d));
  const double x0 = xf;
  const double r = fma(-dl, x0, fma(-d, x0, 1.0)), t = fma(r, r, r);
  const double cx = __dmul_rn(x, x0), cy = __dmul_rn(y, x0);
  const double rx = __dadd_rn(cx, fma(cx, t, fma(x, x0, -cx))), ry = __dadd_rn(cy, fma(cy, t, fma(y, x0, -cy)));
  const int lx = __double2loint(a.x), ly = __double2loint(a.y);
  // the parts' high words tell infinity (0x7ff00000, low word 0) from NaN; with
  // x0 = 1 / infinity = 0 every other non-finite a turns r, and so t, into NaN
  const bool inf1 = max(hx, hy) == 0x7ff00000 && (hx > hy ? lx : ly) == 0 && min(hx, hy) < 0x7ff00000;
  const bool none = (hx | hy | lx | ly) == 0 || inf1;
  return none ? make_double2(0.0, 0.0) : make_double2(rx * s, -ry * s);
}

// Chained launches.  A plan's kernels run one after the other on a stream; with
// programmatic stream serialization the CTAs of the next kernel are placed as
// soon as the current one's have started, instead of after its end and a
// launch's latency (about 2 us: RGF of 10 layers of 32 487 -> 394 us).  Each
// kernel calls chain_entry first: it lets the next one come, and waits until the
// ones before have completed, so that everything after it sees what plain stream
// order would show.  (Every kernel of a chain has to wait, also the CTAs that do
// nothing: the next one's wait covers its predecessor alone.)
__device__ __forceinline__ void chain_entry() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// CTAs of the kernel before in the calling thread's chain; negative outside one.
// A chain is a plan's direct run: captured into a graph, the launches cost its
// first pass more than they give (16 layers of 64, 64 energies: 2.7 -> 3.1 ms).
// Two kernels are chained while together they have no more CTAs than the GPU has
// SMs (148): above that the early CTAs share the SMs that are free first instead
// of spreading over all of them (Keldysh sweep of 10 layers of 300: 7.4 ms plain,
// 8.1 with every launch chained, 7.0 by this rule).
inline thread_local long long chain_ctas = -1;

template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  c.attrs = &attr;
  const long long ctas = (long long)grid.x * grid.y * grid.z;
  if (chain_ctas >= 0) {
    c.numAttrs = chain_ctas + ctas <= 148 ? 1 : 0;
    chain_ctas = ctas;
  }
  return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// a - b c with four fused operations
__device__ __forceinline__ cplx cfms_fused(cplx a, cplx b, cplx c) {
  return make_double2(fma(b.y, c.y, fma(-b.x, c.x, a.x)), fma(-b.y, c.x, fma(-b.x, c.y, a.y)));
}
#endif
// |re| + |im|: the pivot magnitude LAPACK's izamax uses (dcabs1)
__host__ __device__ inline double cabs1(cplx a) { return fabs(a.x) + fabs(a.y); }

// One problem of a batched complex GEMM:
//   C = alpha * op(A) * op(B) + beta * Cin + diag * I
// op(A) is m x k, op(B) is k x n, C and Cin are m x n (Cin may alias C).
// k == 0 turns the problem into C = beta * Cin + diag * I.
struct ZGemmProblem {
  const cplx* A;
  const cplx* B;
  const cplx* Cin;
  cplx* C;
  const cplx* diag_ptr;  // when set, diag is read from device memory (per-energy shift)
  const cplx* alpha_ptr;  // when set, multiplies alpha (read from device memory: per-energy factors)
  int m, n, k;
  int lda, ldb, ldc, ldcin;
  int pad_;
  cplx alpha, beta, diag;
};

// One matrix of a batched Gauss-Jordan inversion: W (n x n, ld) is inverted in
// place; scratch F (n x nb) and Bbuf (nb x n) hold the rank-nb update of a
// panel; used (n bytes) and piv (n ints) persist across panels; out receives
// the un-permuted inverse (n x n, ldo).
struct ZInvProblem {
  cplx* W;
  cplx* F;
  cplx* Bbuf;
  uint8_t* used;
  int* piv;
  cplx* out;
  int* info;   // set to (global column + 1) on a zero pivot, else left untouched
  int n, ld, ldo, pad_;
};

// Widest Gauss-Jordan panel: the pivot-row buffer of zgj_update_kernel.
constexpr int kGjMaxNb = 32;

// One matrix of a batched LU (zlu.cu).
struct ZLuProblem {
  cplx* A;       // n x n, ld
  int* ipiv;     // n (0-based global pivot rows)
  cplx* Linv;    // scratch nb x nb (inverse of the panel's unit-lower block)
  cplx* T;       // scratch nb x n (A12 copy)
  int* info;
  int n, ld;
};

// One matrix of a batched triangular inverse (zlu.cu).
struct ZTriProblem {
  const cplx* A;  // packed factors, n x n, lda
  cplx* X;        // output, n x n, ldx
  int n, lda, ldx, pad_;
};

// One matrix of a batched unpivoted LU with the inverses of its diagonal blocks
// (zlu.cu): F receives the packed factors of the blocks, Xu / Xl (n x n, ld n)
// the inverses of their upper and unit lower triangles.
struct ZLuDiagProblem {
  const cplx* A;
  cplx* F;
  cplx *Xu, *Xl;
  int* info;
  int n, ld, ldf, pad_;
};

// Digit split of one real-and-imaginary operand view for the Ozaki GEMM
// (zgemm_ozaki.cu): Y[r][k] = X[r*sr + k*sk] (conjugated when conj), R x K.
// The digits are stored pre-tiled for the tensor cores: for every real
// operand p (re, im, re + im), row tile t (tile_rows rows) and 32-wide K chunk
// c one contiguous block of 7 digit slices in the canonical K-major
// core-matrix order (r, k) -> (k / 16) * R * 16 + (r / 8) * 128 + (r % 8) * 16
// + k % 16; blocks ordered [p][t][c]. Left operand (tile_rows 128): each slice
// is its own R = 128 matrix. Right operand (tile_rows 64): the seven slices
// form one R = 448 matrix (row 64 i + r for slice i).
struct OzSplitProblem {
  const cplx* X;
  long long sr, sk;
  int rows, cols, rows_pad, k_pad;
  int conj, tile_rows;  // tile_rows: 128 (left operand) or 64 (right operand)
  int8_t* slices;       // 3 * 7 * rows_pad * k_pad int8 digits
  int* exps;            // [rows_pad] power-of-two row scales
};

// One complex product of the Ozaki GEMM: C = alpha A B + beta Cin + diag I
// from the digit slices of A (m x k) and of B^T (n x k).
struct OzMmaProblem {
  const int8_t* SA;
  const int* eA;
  const int8_t* SB;
  const int* eB;
  cplx* C;
  const cplx* Cin;
  const cplx* diag_ptr;
  const cplx* alpha_ptr;
  int m, n, m_pad, n_pad, k_pad, ldc, ldcin, pad_;
  cplx alpha, beta, diag;
};

// Elementwise block operations (ZBlockOp::kind).
enum ZOpKind : int {
  ZOP_COPY = 0,        // C = A
  ZOP_CTRANSPOSE = 1,  // C = A^H   (A is n x m)
  ZOP_AXPBY = 2,       // C = alpha*A + beta*C
  ZOP_FILL = 3,        // C = alpha (every entry)
  ZOP_IDENTITY = 4,    // C = alpha * I
  ZOP_HERM_PART = 5,   // C = (A + A^H)/2
  ZOP_GAMMA = 6,       // C = i (A - A^H)   (broadening of a self-energy)
  ZOP_CTRANS_AXPBY = 7,  // C = alpha*A^H + beta*C   (A is n x m)
  ZOP_ADD_DIAG = 8,    // C[r, r] += alpha
  ZOP_HERM_SUM = 9,    // C = alpha (A + A^H)
};

struct ZBlockOp {
  const cplx* A;
  cplx* C;
  const cplx* alpha_ptr;  // when set, alpha is read from device memory
  int m, n, lda, ldc;
  int kind, pad_;
  cplx alpha, beta;
};

}  // namespace negf
