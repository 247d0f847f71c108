// Batched complex FP64 GEMM on the sm_100a FP64 tensor path (DMMA).
//
// Every Schur-complement product of the RGF / RKD / selected-inverse / DDRGF
// sweeps (the reference's be_gemm!, src/backend_cpu.jl:208-219, and the
// getrs-with-explicit-inverse products that replace be_mldivide!) runs here.
//
// Design:
//  * one launch covers a whole list of independent problems of arbitrary
//    (m, n, k) -- all energies x all blocks of one sweep step; CTAs map to
//    (problem, output tile) through a prefix sum of tile counts;
//  * operands are staged through cp.async rings (each complex double is one
//    16-byte cp.async, so transposed / conjugated operands are handled on the
//    copy); FP64 has no tcgen05 kind, and on B200 mma.sync f64 and DFMA both
//    peak near 37 TFLOP/s (measured by negf_probe_fp64_peak), so DMMA is the
//    FP64 tensor path;
//  * the default form is 3M (three real products per complex one) in 32 x 32 or
//    16 x 16 tiles; a four-product kernel in 64 x 64 tiles serves gemm_form 1;
//  * epilogue: C = alpha*acc + beta*Cin + diag*I, bounds-checked.
#include "negf_common.cuh"

#include <cstdlib>

namespace negf {

// step forms of the 3M kernels (32 x 32 and 16 x 16 tiles)
constexpr int kFormTile32 = 5, kFormTile16 = 6;

namespace gemm {
constexpr int BM = 64, BN = 64, BK = 16;
constexpr int THREADS = 128;
constexpr int STAGES = 3;
constexpr int AS_LD = BM + 1;  // As[k][m]
constexpr int BS_LD = BK + 1;  // Bs[n][k]
constexpr int AS_SIZE = BK * AS_LD;
constexpr int BS_SIZE = BN * BS_LD;
constexpr int STAGE_SIZE = AS_SIZE + BS_SIZE;  // complex elements per stage
constexpr size_t SMEM_BYTES = size_t(STAGES) * STAGE_SIZE * sizeof(cplx);
}  // namespace gemm

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  int sz = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma16x8x4(double& c0, double& c1, double& c2, double& c3, double a0, double a1,
                                           double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(c0), "+d"(c1), "+d"(c2), "+d"(c3)
      : "d"(a0), "d"(a1), "d"(b0));
}

// CTA -> (problem, tile).  nprob > 0: binary search over the exclusive
// prefix sum tile_start; nprob < 0: every problem has -nprob tiles (the
// host's uniform batches), so the problem is a division away and the CTA
// skips the chain of dependent loads of the search.
__device__ __forceinline__ void zgemm_locate(int bid, const int* __restrict__ tile_start, int nprob, int& prob,
                                             int& tile) {
  if (nprob < 0) {
    const int T = -nprob;
    prob = bid / T;
    tile = bid - prob * T;
    return;
  }
  int lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_start[mid] <= bid) lo = mid; else hi = mid - 1;
  }
  prob = lo;
  tile = bid - tile_start[lo];
}

// Stage one K-slab of A (BM x BK of op(A)) and B (BK x BN of op(B)).
template <bool TA, bool TB>
__device__ __forceinline__ void load_stage(cplx* As, cplx* Bs, const ZGemmProblem& p, int m0, int n0, int k0,
                                           int tid) {
  using namespace gemm;
  // A tile: element (r, kk) of op(A)
#pragma unroll
  for (int i = 0; i < (BM * BK) / THREADS; ++i) {
    int idx = tid + i * THREADS;
    int r, kk;
    if (!TA) { r = idx % BM; kk = idx / BM; }   // contiguous in r for column-major A
    else     { kk = idx % BK; r = idx / BK; }   // contiguous in k for A^T / A^H
    int gr = m0 + r, gk = k0 + kk;
    bool ok = gr < p.m && gk < p.k;
    const cplx* src = p.A;
    if (ok) src = TA ? (p.A + gk + (size_t)gr * p.lda) : (p.A + gr + (size_t)gk * p.lda);
    cp_async16(&As[kk * AS_LD + r], src, ok);
  }
  // B tile: element (kk, c) of op(B)
#pragma unroll
  for (int i = 0; i < (BN * BK) / THREADS; ++i) {
    int idx = tid + i * THREADS;
    int c, kk;
    if (!TB) { kk = idx % BK; c = idx / BK; }   // contiguous in k for column-major B
    else     { c = idx % BN; kk = idx / BN; }   // contiguous in n for B^T / B^H
    int gc = n0 + c, gk = k0 + kk;
    bool ok = gc < p.n && gk < p.k;
    const cplx* src = p.B;
    if (ok) src = TB ? (p.B + gc + (size_t)gk * p.ldb) : (p.B + gk + (size_t)gc * p.ldb);
    cp_async16(&Bs[c * BS_LD + kk], src, ok);
  }
}

template <bool TA, bool CA, bool TB, bool CB, bool PRE>
__global__ void __launch_bounds__(gemm::THREADS, 2)
    zgemm_batched_kernel(const ZGemmProblem* __restrict__ probs, const int* __restrict__ tile_start, int nprob) {
  chain_entry();
  using namespace gemm;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* smem = reinterpret_cast<cplx*>(smem_raw);

  int lo, t;
  zgemm_locate(blockIdx.x, tile_start, nprob, lo, t);
  const ZGemmProblem p = probs[lo];
  int tiles_m = (p.m + BM - 1) / BM;
  int m0 = (t % tiles_m) * BM;
  int n0 = (t / tiles_m) * BN;

  int tid = threadIdx.x;
  int warp = tid >> 5, lane = tid & 31;
  int g = lane >> 2, tq = lane & 3;
  int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;

  // PRE (chosen per launch by the host when every problem has alpha, beta in
  // {1, -1} and a Cin): in-place updates C = +-A*B +- C, i.e. every Schur
  // update of the sweeps, start the accumulators from Cin, so the loads are
  // issued before the main loop and overlap the first operand copies instead
  // of stalling the epilogue.
  const bool preload = PRE && p.k > 0 && p.Cin != nullptr;
  const double pre_sign = p.alpha.x * p.beta.x;  // beta / alpha for alpha, beta in {1, -1}

  double acc_re[2][4][4], acc_im[2][4][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        acc_re[a][b][c] = 0.0;
        acc_im[a][b][c] = 0.0;
        if (preload) {
          int r = m0 + wm + a * 16 + g + ((c >> 1) << 3);
          int cc = n0 + wn + b * 8 + 2 * tq + (c & 1);
          if (r < p.m && cc < p.n) {
            cplx v = p.Cin[r + (size_t)cc * p.ldcin];
            acc_re[a][b][c] = pre_sign * v.x;
            acc_im[a][b][c] = pre_sign * v.y;
          }
        }
      }

  int nk = (p.k + BK - 1) / BK;
  // prologue
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load_stage<TA, TB>(smem + s * STAGE_SIZE, smem + s * STAGE_SIZE + AS_SIZE, p, m0, n0, s * BK, tid);
    cp_async_commit();
  }

  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    // prefetch the slab STAGES-1 ahead into the buffer freed last iteration
    int kn = kt + STAGES - 1;
    if (kn < nk) {
      int s = kn % STAGES;
      load_stage<TA, TB>(smem + s * STAGE_SIZE, smem + s * STAGE_SIZE + AS_SIZE, p, m0, n0, kn * BK, tid);
    }
    cp_async_commit();

    const cplx* As = smem + (kt % STAGES) * STAGE_SIZE;
    const cplx* Bs = As + AS_SIZE;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      double ar[2][2], ai[2][2], br[4], bi[4], nbi[4];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        cplx x0 = As[(kk + tq) * AS_LD + wm + mi * 16 + g];
        cplx x1 = As[(kk + tq) * AS_LD + wm + mi * 16 + g + 8];
        ar[mi][0] = x0.x; ai[mi][0] = CA ? -x0.y : x0.y;
        ar[mi][1] = x1.x; ai[mi][1] = CA ? -x1.y : x1.y;
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        cplx y = Bs[(wn + ni * 8 + g) * BS_LD + kk + tq];
        br[ni] = y.x;
        bi[ni] = CB ? -y.y : y.y;
        nbi[ni] = -bi[ni];
      }
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          double* cr = acc_re[mi][ni];
          double* ci = acc_im[mi][ni];
          dmma16x8x4(cr[0], cr[1], cr[2], cr[3], ar[mi][0], ar[mi][1], br[ni]);
          dmma16x8x4(cr[0], cr[1], cr[2], cr[3], ai[mi][0], ai[mi][1], nbi[ni]);
          dmma16x8x4(ci[0], ci[1], ci[2], ci[3], ar[mi][0], ar[mi][1], bi[ni]);
          dmma16x8x4(ci[0], ci[1], ci[2], ci[3], ai[mi][0], ai[mi][1], br[ni]);
        }
    }
  }
  cp_async_wait<0>();

  // epilogue
  const bool has_ab = p.k > 0;
  const bool has_cin = (p.beta.x != 0.0 || p.beta.y != 0.0) && p.Cin != nullptr && !preload;
  const cplx dg = p.diag_ptr ? *p.diag_ptr : p.diag;
  const cplx al = p.alpha_ptr ? cmul(p.alpha, *p.alpha_ptr) : p.alpha;
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int r = m0 + wm + mi * 16 + g + ((e >> 1) << 3);
        int c = n0 + wn + ni * 8 + 2 * tq + (e & 1);
        if (r < p.m && c < p.n) {
          cplx v = make_double2(0.0, 0.0);
          if (has_ab) {
            double xr = acc_re[mi][ni][e], xi = acc_im[mi][ni][e];
            v.x = al.x * xr - al.y * xi;
            v.y = al.x * xi + al.y * xr;
          }
          if (has_cin) {
            cplx ci = p.Cin[r + (size_t)c * p.ldcin];
            v.x += p.beta.x * ci.x - p.beta.y * ci.y;
            v.y += p.beta.x * ci.y + p.beta.y * ci.x;
          }
          if (r == c) { v.x += dg.x; v.y += dg.y; }
          p.C[r + (size_t)c * p.ldc] = v;
        }
      }
}

// ---------------------------------------------------------------------------
// 3M kernels (Gauss's complex product): three real DMMA products per complex
// product instead of four,
//   P1 = Ar Br,  P2 = Ai Bi,  P3 = (Ar + Ai)(Br + Bi),
//   Re C = P1 - P2,  Im C = P3 - P1 - P2,
// the scheme of zgemm3m (normwise stable; the imaginary part carries an
// absolute error of a few ulps of |A||B| instead of |Im C|).
//
// 16 WM x 16 WN tiles by WM WN WK warps of 16 x 16, the WK warps of a part
// sharing its K slabs (their sums meet in shared memory); four CTAs of 128
// threads per SM, so that the fixed latency of a tile -- descriptor, operands,
// Cin (read before the K loop), stores -- hides behind other tiles' products.
// Bound: FP64 tensor time.  64 products of 256 x 256 x 256 take 236 us, 36.4
// TFLOP/s of 8 m n k (64 x 64 tiles with one CTA of 256 threads per SM: 264 us);
// one 256 product 10.9 us in 16 x 16 tiles, 17.0 in 32 x 32 (64 x 64: 38, 16 CTAs
// on 148 SMs); 205 of 32 x 32 x 32 7.3 us (18 in 64 x 64, three quarters padding).
namespace gemm_st {
constexpr int THREADS = 128, BK = 16, STAGES = 2;
constexpr int BLD = BK + 4;  // Bs[n][k]; 4 mod 8 and (A) 2 mod 8: no bank conflicts between a fragment's rows
template <int WM, int WN>
constexpr size_t smem_bytes() {
  return (size_t)STAGES * (BK * (16 * WM + 2) + 16 * WN * BLD) * sizeof(cplx);
}
}  // namespace gemm_st

template <bool TA, bool CA, bool TB, bool CB, int WM, int WN, int WK>
__global__ void __launch_bounds__(gemm_st::THREADS, 4)
    zgemm3m_tile_kernel(const ZGemmProblem* __restrict__ probs, const int* __restrict__ tile_start, int nprob) {
  chain_entry();
  using namespace gemm_st;
  static_assert(WM * WN * WK * 32 == THREADS, "warp layout");
  static_assert(WK == 1 || (size_t)WM * WN * (WK - 1) * 24 * 32 * sizeof(double) <= smem_bytes<WM, WN>(), "partial sums");
  static_assert(smem_bytes<WM, WN>() <= 48 * 1024, "no opt-in shared memory");
  constexpr int BM = 16 * WM, BN = 16 * WN, ALD = BM + 2;
  constexpr int AS = BK * ALD, STAGE = AS + BN * BLD;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* smem = reinterpret_cast<cplx*>(smem_raw);
  int lo, t;
  zgemm_locate(blockIdx.x, tile_start, nprob, lo, t);
  const ZGemmProblem& p = probs[lo];
  const int pm = p.m, pn = p.n, pk = p.k, lda = p.lda, ldb = p.ldb;
  const cplx* const pA = p.A;
  const cplx* const pB = p.B;
  const int tiles_m = (pm + BM - 1) / BM;
  const int m0 = (t % tiles_m) * BM, n0 = (t / tiles_m) * BN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  const int wk = warp / (WM * WN), wm = (warp % WM) * 16, wn = (warp / WM % WN) * 16;
  auto load = [&](int kt) {
    cplx* As = smem + (kt % STAGES) * STAGE;
    cplx* Bs = As + AS;
    const int k0 = kt * BK;
#pragma unroll
    for (int i = tid; i < BM * BK; i += THREADS) {
      const int r = TA ? i / BK : i % BM, kk = TA ? i % BK : i / BM, gr = m0 + r, gk = k0 + kk;
      const bool ok = gr < pm && gk < pk;
      cp_async16(&As[kk * ALD + r], ok ? (TA ? pA + gk + (size_t)gr * lda : pA + gr + (size_t)gk * lda) : pA, ok);
    }
#pragma unroll
    for (int i = tid; i < BN * BK; i += THREADS) {
      const int c = TB ? i % BN : i / BK, kk = TB ? i / BN : i % BK, gc = n0 + c, gk = k0 + kk;
      const bool ok = gc < pn && gk < pk;
      cp_async16(&Bs[c * BLD + kk], ok ? (TB ? pB + gc + (size_t)gk * ldb : pB + gk + (size_t)gc * ldb) : pB, ok);
    }
  };
  const int nk = (pk + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load(s);
    cp_async_commit();
  }
  const cplx beta = p.beta;
  const cplx* const Cin = p.Cin;
  const bool has_cin = wk == 0 && (beta.x != 0.0 || beta.y != 0.0) && Cin != nullptr;
  cplx old[2][4];
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = m0 + wm + g + ((e >> 1) << 3), c = n0 + wn + x * 8 + 2 * tq + (e & 1);
      old[x][e] = has_cin && r < pm && c < pn ? Cin[r + (size_t)c * p.ldcin] : make_double2(0.0, 0.0);
    }
  double P1[2][4] = {}, P2[2][4] = {}, P3[2][4] = {};
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (kt + STAGES - 1 < nk) load(kt + STAGES - 1);
    cp_async_commit();
    const cplx* As = smem + (kt % STAGES) * STAGE + wm + g;
    const cplx* Bs = smem + (kt % STAGES) * STAGE + AS + (wn + g) * BLD + tq;
#pragma unroll
    for (int kk = 4 * wk; kk < BK; kk += 4 * WK) {
      const cplx x0 = As[(kk + tq) * ALD], x1 = As[(kk + tq) * ALD + 8];
      const double i0 = CA ? -x0.y : x0.y, i1 = CA ? -x1.y : x1.y;
      const double s0 = x0.x + i0, s1 = x1.x + i1;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const cplx y = Bs[x * 8 * BLD + kk];
        const double yi = CB ? -y.y : y.y;
        dmma16x8x4(P1[x][0], P1[x][1], P1[x][2], P1[x][3], x0.x, x1.x, y.x);
        dmma16x8x4(P2[x][0], P2[x][1], P2[x][2], P2[x][3], i0, i1, yi);
        dmma16x8x4(P3[x][0], P3[x][1], P3[x][2], P3[x][3], s0, s1, y.x + yi);
      }
    }
  }
  cp_async_wait<0>();
  if (WK > 1) {
    // [part][WK - 1][24][32]: the sums of the warps with wk > 0
    double* red = reinterpret_cast<double*>(smem_raw) + (size_t)(warp % (WM * WN)) * (WK - 1) * 24 * 32 + lane;
    __syncthreads();
    if (wk > 0)
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          double* q = red + (wk - 1) * 24 * 32 + (x * 4 + e) * 96;
          q[0] = P1[x][e];
          q[32] = P2[x][e];
          q[64] = P3[x][e];
        }
    __syncthreads();
    if (wk > 0) return;
    for (int w = 0; w < WK - 1; ++w)
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const double* q = red + w * 24 * 32 + (x * 4 + e) * 96;
          P1[x][e] += q[0];
          P2[x][e] += q[32];
          P3[x][e] += q[64];
        }
  }
  const cplx dg = p.diag_ptr ? *p.diag_ptr : p.diag;
  const cplx al = p.alpha_ptr ? cmul(p.alpha, *p.alpha_ptr) : p.alpha;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = m0 + wm + g + ((e >> 1) << 3), c = n0 + wn + x * 8 + 2 * tq + (e & 1);
      if (r >= pm || c >= pn) continue;
      cplx v = make_double2(0.0, 0.0);
      if (pk > 0) {
        const double xr = P1[x][e] - P2[x][e], xi = P3[x][e] - P1[x][e] - P2[x][e];
        v.x = al.x * xr - al.y * xi;
        v.y = al.x * xi + al.y * xr;
      }
      if (has_cin) {
        v.x += beta.x * old[x][e].x - beta.y * old[x][e].y;
        v.y += beta.x * old[x][e].y + beta.y * old[x][e].x;
      }
      if (r == c) {
        v.x += dg.x;
        v.y += dg.y;
      }
      p.C[r + (size_t)c * p.ldc] = v;
    }
}

using ZGemmKernel = void (*)(const ZGemmProblem*, const int*, int);

template <bool PRE>
static ZGemmKernel pick_kernel_t(int ia, int ib) {
#define NEGF_K(TA, CA, TB, CB) zgemm_batched_kernel<TA, CA, TB, CB, PRE>
  switch (ia * 3 + ib) {
    case 0: return NEGF_K(false, false, false, false);
    case 1: return NEGF_K(false, false, true, false);
    case 2: return NEGF_K(false, false, true, true);
    case 3: return NEGF_K(true, false, false, false);
    case 4: return NEGF_K(true, false, true, false);
    case 5: return NEGF_K(true, false, true, true);
    case 6: return NEGF_K(true, true, false, false);
    case 7: return NEGF_K(true, true, true, false);
    default: return NEGF_K(true, true, true, true);
  }
#undef NEGF_K
}

// The 3M form is the default; NEGF_ZGEMM=4m selects the four-product kernel.
static bool use_3m() {
  static const bool v = [] {
    const char* e = std::getenv("NEGF_ZGEMM");
    return !(e && (e[0] == '4'));
  }();
  return v;
}

template <int WM, int WN, int WK>
static ZGemmKernel pick_tile_t(int ia, int ib) {
#define NEGF_K(TA, CA, TB, CB) zgemm3m_tile_kernel<TA, CA, TB, CB, WM, WN, WK>
  switch (ia * 3 + ib) {
    case 0: return NEGF_K(false, false, false, false);
    case 1: return NEGF_K(false, false, true, false);
    case 2: return NEGF_K(false, false, true, true);
    case 3: return NEGF_K(true, false, false, false);
    case 4: return NEGF_K(true, false, true, false);
    case 5: return NEGF_K(true, false, true, true);
    case 6: return NEGF_K(true, true, false, false);
    case 7: return NEGF_K(true, true, true, false);
    default: return NEGF_K(true, true, true, true);
  }
#undef NEGF_K
}

static int op_index(char op) { return op == 'N' ? 0 : (op == 'T' ? 1 : 2); }

static ZGemmKernel pick_kernel(char opA, char opB, bool pre) {
  const int ia = op_index(opA), ib = op_index(opB);
  return pre ? pick_kernel_t<true>(ia, ib) : pick_kernel_t<false>(ia, ib);
}

size_t zgemm_smem_bytes() { return gemm::SMEM_BYTES; }

// Raise the dynamic shared-memory limit of one op variant of the four-product
// kernel (both accumulator initialisations) on the current device; done when a
// plan is finalised, outside any stream capture.
cudaError_t zgemm_prepare(char opA, char opB) {
  for (int v = 0; v < 2; ++v) {
    cudaError_t e = cudaFuncSetAttribute(pick_kernel(opA, opB, v & 1), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)gemm::SMEM_BYTES);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Output tiles of a problem under a step form.
int zgemm_tiles_form(int form, int m, int n) {
  if (m <= 0 || n <= 0) return 0;
  const int b = form == kFormTile32 ? 32 : form == kFormTile16 ? 16 : gemm::BM;
  return ((m + b - 1) / b) * ((n + b - 1) / b);
}

// The kernel of a step: the four-product one for form 1 (or by NEGF_ZGEMM=4m),
// else 3M in 32 x 32 tiles, in 16 x 16 tiles when there are fewer than 96 of the
// former: a CTA's time is then the step's (one 256 product, 64 tiles: 17.0 against
// 10.9 us; two, 128 tiles: 17.7 against 18.7 us).  The 16 x 16 form adds its K
// slabs in another order, so fixed_order (results that do not depend on what else
// is in the batch) keeps to 32 x 32.
int zgemm_choose_form(int form, const ZGemmProblem* probs, int nprob, bool fixed_order) {
  if (form == 1 || (form == 0 && !use_3m())) return 1;
  if (fixed_order) return kFormTile32;
  long long tiles = 0;
  for (int i = 0; i < nprob; ++i) tiles += zgemm_tiles_form(kFormTile32, probs[i].m, probs[i].n);
  return tiles < 96 ? kFormTile16 : kFormTile32;
}

// True when the problem qualifies for the accumulator preload variant.
bool zgemm_preload_ok(const ZGemmProblem& p) {
  return p.k > 0 && p.Cin != nullptr && p.alpha_ptr == nullptr && p.alpha.y == 0.0 && p.beta.y == 0.0 &&
         (p.alpha.x == 1.0 || p.alpha.x == -1.0) && (p.beta.x == 1.0 || p.beta.x == -1.0);
}

// Host launchers.  probs_dev / tile_start_dev are device arrays prepared by
// the caller (tile_start has nprob entries, exclusive prefix sum of tile
// counts).  preload may only be set when zgemm_preload_ok holds for every
// problem of the launch.
cudaError_t launch_zgemm_batched_ex(char opA, char opB, bool preload, const ZGemmProblem* probs_dev,
                                    const int* tile_start_dev, int nprob, int total_tiles, cudaStream_t stream,
                                    int form, int uniform_tiles) {
  if (nprob <= 0 || total_tiles <= 0) return cudaSuccess;
  static const bool uniform_on = [] {
    const char* e = std::getenv("NEGF_ZGEMM_UNIFORM");
    return !(e && e[0] == '0');
  }();
  // every problem has uniform_tiles tiles: the kernels locate their problem by
  // division (signalled by a negative count)
  if (uniform_on && uniform_tiles > 0 && (long long)uniform_tiles * nprob == total_tiles) nprob = -uniform_tiles;
  if (form == kFormTile32 || form == kFormTile16) {
    const int ia = op_index(opA), ib = op_index(opB);
    if (form == kFormTile32)
      launch_chained(pick_tile_t<2, 2, 1>(ia, ib), total_tiles, gemm_st::THREADS, gemm_st::smem_bytes<2, 2>(), stream,
                     probs_dev, tile_start_dev, nprob);
    else
      launch_chained(pick_tile_t<1, 1, 4>(ia, ib), total_tiles, gemm_st::THREADS, gemm_st::smem_bytes<1, 1>(), stream,
                     probs_dev, tile_start_dev, nprob);
    return cudaGetLastError();
  }
  launch_chained(pick_kernel(opA, opB, preload), total_tiles, gemm::THREADS, gemm::SMEM_BYTES, stream, probs_dev,
                 tile_start_dev, nprob);
  return cudaGetLastError();
}

// The four-product kernel without accumulator preload.
cudaError_t launch_zgemm_batched(char opA, char opB, const ZGemmProblem* probs_dev, const int* tile_start_dev,
                                 int nprob, int total_tiles, cudaStream_t stream) {
  if (nprob <= 0 || total_tiles <= 0) return cudaSuccess;
  launch_chained(pick_kernel(opA, opB, false), total_tiles, gemm::THREADS, gemm::SMEM_BYTES, stream, probs_dev,
                 tile_start_dev, nprob);
  return cudaGetLastError();
}

int zgemm_tiles(int m, int n) { return zgemm_tiles_form(1, m, n); }

}  // namespace negf
