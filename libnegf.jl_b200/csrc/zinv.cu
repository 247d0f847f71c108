// Batched complex FP64 block inversion by blocked Gauss-Jordan with partial
// pivoting.
//
// The reference factors every diagonal Schur complement with zgetrf and then
// applies X^{-1} through zgetrs (be_lu! / be_mldivide!, src/backend_cpu.jl:
// 147-206); the downward pass needs X^{-1} explicitly anyway
// (src/matinvertndiag_rgf.jl:169,180).  Here X^{-1} is formed once, so every
// later use is a tensor-core GEMM.
//
// Algorithm (per matrix, n x n, panel width nb):
//   for each panel K = [k0, k0+nb):
//     * the panel kernel (one CTA per matrix) runs the in-place Gauss-Jordan
//       steps of the n x nb slab W[:,K] in shared memory.  No rows are swapped;
//       the pivot row of column c is recorded in piv[c];
//     * the update kernel applies W += slab W[P, :] to the other columns (and
//       sets the pivot rows P to slab W[P, :]).
//   Finally inv(X)[r, piv[c]] = W[piv[r], c]; a gather kernel writes the
//   un-permuted inverse to its destination.
// When n * n fits in shared memory the whole matrix is one panel and no update
// is needed.
#include "negf_common.cuh"

namespace negf {

namespace gj {
constexpr int SW = 8;  // columns of a sub-panel, factored in registers
}

struct GjPanelArgs {
  int k0;      // first column of this panel
  int nb;      // panel width (columns)
  int blocked; // 1: zgj_update_kernel follows; 2: write F and Bbuf for a GEMM update
};

__device__ __forceinline__ void gj_cp16(cplx* smem, const cplx* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
// with in = false: zeros (any valid address)
__device__ __forceinline__ void gj_cp16z(cplx* smem, const cplx* gmem, bool in, const cplx* any) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(in ? gmem : any), "r"(in ? 16 : 0));
}
__device__ __forceinline__ void gj_cp_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

__device__ __forceinline__ void gj_dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// Pivot candidates compare as 32-bit keys: the leading 21 bits of |re| + |im|
// (exponent and 10 mantissa bits) in the upper 22, over 1023 - row, so that one
// REDUX gives value and row.  The upper part is 0 without a candidate, 1 for an
// exact zero and larger for every other value.  The pivot is within 0.1 % of the
// largest |re| + |im| of its column, the lowest row among those that share the
// leading bits; the growth bound of partial pivoting changes by that factor only.
// (Values below 2^-1032 all share them; the reciprocal of each overflows.)
__device__ __forceinline__ unsigned gj_key(double v, int row) {
  const unsigned hi = __double2hiint(v);
  return (((hi >> 10) + ((hi | (unsigned)__double2loint(v)) != 0u ? 2u : 1u)) << 10) | (unsigned)(1023 - row);
}

// Gauss-Jordan on an n x w slab held in shared memory (column-major, odd
// leading dimension ldw), one CTA per matrix, in sub-panels of SW = 8 columns:
//  * the sub-panel is factored in registers, one row per thread (RT rows for n
//    > T).  Per column: every thread inverts its own entry while one warp
//    reduction (REDUX) of the keys finds the warp's pivot candidate, whose lane
//    publishes its row divided by the pivot; one barrier; every thread merges
//    the T/32 keys, reads the winner's row and updates its own;
//  * W[pivot rows, other columns] is copied aside (Bb) and the other columns of
//    the slab take the rank-8 update on the FP64 tensor path (16 x 8 tiles, k =
//    8, four real products): W += S Bb, and W = S Bb at the pivot rows (the
//    form W += (S - E_P) Bb would lose digits where |S| is far below 1).
// What bounds it: the latency of a column (690 cycles with one warp of rows, 800
// with four, 980 with eight: two reduction rounds, a barrier of the warps with
// rows, one reciprocal, and some 250 instructions per warp) and the FP64 pipe of
// one SM in the rank-8 updates.  Eight columns keep a row in 32 registers; wider
// sub-panels do more of the n w^2 work in the latency-bound form, narrower ones
// add update passes over shared memory.  A 256 x 32 panel takes 35 us (104 us
// with the whole slab in registers and one rank-1 step per column).
template <int T, int RT>
__global__ void __launch_bounds__(T, 1)
    zgj_panel_kernel(const ZInvProblem* __restrict__ probs, GjPanelArgs args) {
  chain_entry();
  using gj::SW;
  const ZInvProblem p = probs[blockIdx.x];
  const int n = p.n;
  const int k0 = args.k0;
  if (n <= 0 || k0 >= n) return;
  const int w = min(args.nb, n - k0);
  constexpr int NW = T / 32;
  const int ldw = n | 1;
  const int wt = (w + SW - 1) / SW;  // column tiles of the slab
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* S = reinterpret_cast<cplx*>(smem_raw);       // ldw x 8 wt
  cplx* Bb = S + (size_t)ldw * SW * wt;               // 8 wt columns of 8 pivot-row values
  cplx* slot = Bb + (size_t)SW * SW * wt;             // [2][NW][SW] candidate rows
  uint4* part = reinterpret_cast<uint4*>(slot + 2 * NW * SW);  // [2][NW] candidate keys
  int* sh_piv = reinterpret_cast<int*>(part + 2 * NW / 4);     // w
  int* sh_dead = sh_piv + w;
  uint8_t* at = reinterpret_cast<uint8_t*>(sh_dead + 1);        // n: the sub-panel whose pivot row a row is

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int j = warp; j < w; j += NW)
    for (int r = lane; r < n; r += 32) gj_cp16(S + (size_t)j * ldw + r, p.W + r + (size_t)(k0 + j) * p.ld);
  bool used[RT];
#pragma unroll
  for (int k = 0; k < RT; ++k) {
    const int r = tid + k * T;
    used[k] = r >= n || (k0 > 0 && p.used[r]);
  }
  for (int c = tid; c < w; c += T) sh_piv[c] = 0;  // valid row indices even if the column loop stops early
  for (int r = tid; r < n; r += T) at[r] = 255;
  if (tid < 2 * NW) reinterpret_cast<unsigned*>(part)[tid] = 0u;
  gj_cp_wait();
  __syncthreads();

  // warps without rows only take part in the rank-8 updates
  const int pw = min(NW, (n + 31) / 32);
  const bool active = warp < pw;
  if (tid == 0) *sh_dead = 0;  // a column without a candidate row: the host reports the info code
  bool dead = false;
  for (int s0 = 0; s0 < w && !dead; s0 += SW) {
    const int sw = min(SW, w - s0);
    cplx a[RT][SW];
#pragma unroll
    for (int k = 0; k < RT; ++k)
#pragma unroll
      for (int j = 0; j < SW; ++j) {
        const int r = tid + k * T;
        a[k][j] = (r < n && j < sw) ? S[(size_t)(s0 + j) * ldw + r] : make_double2(0.0, 0.0);
      }
    // candidate of the current column: this thread's key (NaN rows never qualify; an
    // arithmetic NaN may carry a sign, so the comparison is unsigned) and entry
    unsigned key = 0, wkey = 0;
    cplx cand = make_double2(0.0, 0.0);
    auto search = [&] {
      key = 0;
#pragma unroll
      for (int k = 0; k < RT; ++k) {
        const double v = cabs1(a[k][0]);
        const unsigned q = !used[k] && (unsigned)__double2hiint(v) <= 0x7ff00000u ? gj_key(v, tid + k * T) : 0u;
        if (q > key) {
          key = q;
          cand = a[k][0];
        }
      }
      wkey = __reduce_max_sync(0xffffffffu, key);
    };
    if (active) search();
    // The current column is always register column 0: a step writes column q to
    // register column q - 1 and the finished column to the last one, so the loop
    // is not unrolled.
#pragma unroll 1
    for (int j = 0; active && j < sw; ++j) {
      const int buf = (j & 1) * NW;
      if (lane == 0) reinterpret_cast<unsigned*>(part)[buf + warp] = wkey;
      if (key == wkey && key != 0u) {
        cplx* ws = slot + (buf + warp) * SW;
#pragma unroll
        for (int k = 0; k < RT; ++k)
          if (RT == 1 || tid + k * T == 1023 - (int)(key & 1023u))
#pragma unroll
            for (int q = 1; q < SW; ++q) ws[q] = a[k][q];
        ws[0] = cinv_pivot(cand);
      }
      unsigned best = wkey;
      if (pw == 1) {
        __syncwarp();
      } else {
        asm volatile("bar.sync 1, %0;" ::"r"(pw * 32) : "memory");  // the warps with rows
#pragma unroll
        for (int q = 0; q < NW / 4; ++q) {
          const uint4 x = part[buf / 4 + q];  // zero for the warps without rows
          best = max(max(best, max(x.x, x.y)), max(x.z, x.w));
        }
      }
      const int pr = 1023 - (int)(best & 1023u);
      if (best < 2048u) {  // no candidate row, or zeros only (uniform)
        if (tid == 0 && p.info) atomicCAS(p.info, 0, k0 + s0 + j + 1);
        if (best == 0u) {
          if (tid == 0) {
            *sh_dead = 1;
            sh_piv[s0 + j] = -1;
          }
          break;
        }
      }
      const cplx* row = slot + (buf + ((pr % T) >> 5)) * SW;
      if (tid == pw * 32 - 1) {
        sh_piv[s0 + j] = pr;
        at[pr] = (uint8_t)(s0 / SW);
      }
      // row r -= f row(pivot) with f = a[r][j] / pivot; the pivot row itself is
      // 0 - (-1/pivot) row(pivot)
      const cplx pv = row[0];
      cplx f[RT];
      bool prow[RT];
#pragma unroll
      for (int k = 0; k < RT; ++k) {
        f[k] = cmul(a[k][0], pv);
        prow[k] = tid + k * T == pr;
        used[k] = used[k] || prow[k];
        if (prow[k]) f[k] = cneg(pv);
      }
      // the next column goes first, so that its search overlaps the others' arithmetic
#pragma unroll
      for (int q = 1; q < SW; ++q) {
        const cplx x = row[q];
#pragma unroll
        for (int k = 0; k < RT; ++k)
          a[k][q - 1] = cfms_fused(prow[k] ? make_double2(0.0, 0.0) : a[k][q], f[k], x);
        if (q == 1) search();
      }
#pragma unroll
      for (int k = 0; k < RT; ++k) a[k][SW - 1] = cneg(f[k]);
    }
    // column j of the sub-panel is register column SW - sw + j
#pragma unroll
    for (int k = 0; k < RT; ++k)
#pragma unroll
      for (int q = 0; q < SW; ++q) {
        const int r = tid + k * T, j = q - (SW - sw);
        if (r < n && j >= 0) S[(size_t)(s0 + j) * ldw + r] = a[k][q];
      }
    __syncthreads();
    dead = *sh_dead != 0;
    if (dead || wt == 1) continue;
    // the pivot rows in the other columns (unused k of a last, narrower tile: zero)
    for (int i = tid; i < SW * SW * wt; i += T) {
      const int q = i / SW, j = i % SW;
      Bb[q * SW + (j ^ ((q & 1) << 2))] =
          q < w && j < sw ? S[(size_t)q * ldw + sh_piv[s0 + j]] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    // rank-8 update of the other column tiles: warps take row tiles of 16 and,
    // with fewer row tiles than warps, share the column tiles of one
    const int mt = (n + 15) / 16, ng = mt >= NW ? 1 : NW / mt;
    const int g = lane >> 2, tq = lane & 3, ks = s0 / SW;
    const int m_step = mt >= NW ? NW : mt;
    if (warp < m_step * ng)
      for (int m = warp % m_step; m < mt; m += m_step) {
        const int r0 = m * 16 + g, r1 = r0 + 8;
        const bool i0 = r0 < n, i1 = r1 < n;
        double ar[2][2], ai[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kk = tq + 4 * h;
          cplx x0 = make_double2(0.0, 0.0), x1 = x0;
          if (kk < sw && i0) x0 = S[(size_t)(s0 + kk) * ldw + r0];
          if (kk < sw && i1) x1 = S[(size_t)(s0 + kk) * ldw + r1];
          ar[h][0] = x0.x; ai[h][0] = x0.y;
          ar[h][1] = x1.x; ai[h][1] = x1.y;
        }
        // the next tile's values (zero at the sub-panel's pivot rows) are read
        // while this tile's products run
        const bool o0 = i0 && at[r0] != ks, o1 = i1 && at[r1] != ks;
        cplx c[4], b[2], cn[4], bn[2];
        auto load = [&](int u, cplx (&cc)[4], cplx (&bb)[2]) {
          const int ct = u + (u >= ks ? 1 : 0);
          const cplx* C0 = S + (size_t)(ct * SW + 2 * tq) * ldw + r0;
          const cplx z = make_double2(0.0, 0.0);
          cc[0] = o0 ? C0[0] : z;
          cc[1] = o0 ? C0[ldw] : z;
          cc[2] = o1 ? C0[8] : z;
          cc[3] = o1 ? C0[ldw + 8] : z;
          const cplx* B = Bb + (size_t)(ct * SW + g) * SW;
          bb[0] = B[tq ^ ((g & 1) << 2)];
          bb[1] = B[(tq + 4) ^ ((g & 1) << 2)];
        };
        const int u0 = warp / m_step;
        if (u0 < wt - 1) load(u0, c, b);
        for (int u = u0; u < wt - 1; u += ng) {
          if (u + ng < wt - 1) load(u + ng, cn, bn);
          double re[4], im[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            re[e] = c[e].x;
            im[e] = c[e].y;
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            gj_dmma(re, ar[h][0], ar[h][1], b[h].x);
            gj_dmma(im, ar[h][0], ar[h][1], b[h].y);
            gj_dmma(re, ai[h][0], ai[h][1], -b[h].y);
            gj_dmma(im, ai[h][0], ai[h][1], b[h].x);
          }
          cplx* C0 = S + (size_t)((u + (u >= ks ? 1 : 0)) * SW + 2 * tq) * ldw + r0;
          if (i0) {
            C0[0] = make_double2(re[0], im[0]);
            C0[ldw] = make_double2(re[1], im[1]);
          }
          if (i1) {
            C0[8] = make_double2(re[2], im[2]);
            C0[ldw + 8] = make_double2(re[3], im[3]);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) c[e] = cn[e];
          b[0] = bn[0];
          b[1] = bn[1];
        }
      }
    __syncthreads();
  }
  __syncthreads();

  // write back slab, pivots and used flags
  for (int j = warp; j < w; j += NW)
    for (int r = lane; r < n; r += 32) p.W[r + (size_t)(k0 + j) * p.ld] = S[(size_t)j * ldw + r];
  for (int c = tid; c < w; c += T) p.piv[k0 + c] = sh_piv[c];
#pragma unroll
  for (int k = 0; k < RT; ++k)
    if (tid + k * T < n) p.used[tid + k * T] = used[k] ? 1 : 0;
  if (args.blocked == 1) return;
  // F = slab - E_P  (n x w, ld n)
  for (int j = warp; j < w; j += NW) {
    const int pj = sh_piv[j];
    for (int r = lane; r < n; r += 32) {
      cplx v = S[(size_t)j * ldw + r];
      if (r == pj) v.x -= 1.0;
      p.F[r + (size_t)j * n] = v;
    }
  }
  // Bbuf = W[P, :] with panel columns zeroed  (w x n, ld w): element e = c +
  // j w is W[piv_c, j].  The pivot rows are scattered 16-byte elements, so they
  // are gathered with asynchronous copies (all in flight at once) over the slab,
  // which is written back by now, and stored from there in order.
  __syncthreads();
  for (int e = tid; e < w * n; e += T) {
    const int c = e % w, j = e / w;
    gj_cp16(S + e, p.W + max(sh_piv[c], 0) + (size_t)j * p.ld);
  }
  gj_cp_wait();
  for (int e = tid; e < w * n; e += T) {
    const int j = e / w;
    p.Bbuf[e] = j < k0 || j >= k0 + w ? S[e] : make_double2(0.0, 0.0);
  }
}

// The whole inversion of a matrix that fits shared memory (n <= 112): the same
// sub-panels, with the next one factored beside the rank-8 updates by the
// current one, once all warps have updated its 8 columns.  1, 2 or 4 warps factor
// (n <= 32, 64, 112; one row per thread).  One or two are alone on their
// scheduler partitions (warp mod 4): FP64 tensor instructions of a warp beside
// them would delay every step of the column loop.  Odd CTAs take the opposite
// partitions, so that CTAs that share an SM spread over all of them.
// Bound: the latency of the column loop (690 to 950 cycles a column) up to n =
// 64, the FP64 pipes of one SM above.  Against one sub-panel and one update after
// the other: one matrix of 50: 30 us (42), of 64: 36 (52), 592 of them 112 (124);
// 512 of 32: 24 (41); one of 100: 106 (111), 296 of them 217 (224).  Two
// factoring warps with two rows per thread take 7 % longer at 100.
template <int T>
__global__ void __launch_bounds__(T, 512 / T) zgj_whole_kernel(const ZInvProblem* __restrict__ probs) {
  chain_entry();
  using gj::SW;
  const ZInvProblem p = probs[blockIdx.x];
  const int n = p.n;
  if (n <= 0) return;
  constexpr int NW = T / 32;
  const int ldw = n | 1, wt = (n + SW - 1) / SW, mt = (n + 15) / 16;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* S = reinterpret_cast<cplx*>(smem_raw);       // ldw x 8 wt
  cplx* Bb = S + (size_t)ldw * SW * wt;               // 8 wt columns of 8 pivot-row values
  cplx* slot = Bb + (size_t)SW * SW * wt;             // [2][4][SW] candidate rows
  unsigned* part = reinterpret_cast<unsigned*>(slot + 8 * SW);  // [2][4] candidate keys
  int* sh_piv = reinterpret_cast<int*>(part + 8);     // n
  int* sh_dead = sh_piv + n;
  uint8_t* at = reinterpret_cast<uint8_t*>(sh_dead + 1);  // n: the sub-panel whose pivot row a row is

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
  const int pw = n > 64 ? 4 : n > 32 ? 2 : 1, PT = 32 * pw;  // warps that factor
  const int pbase = pw == 4 ? 0 : pw == 2 ? 2 * (blockIdx.x & 1) : blockIdx.x & 3;
  const int pidx = warp - pbase;  // 0 .. pw - 1: factors
  const bool factors = pidx >= 0 && pidx < pw;
  // the updating warps: those of the other partitions, or the second four
  const int part4 = warp & 3, upart = 4 - pw;
  const bool updates = pw == 4 ? warp >= 4 : part4 < pbase || part4 >= pbase + pw;
  const int nu = pw == 4 ? NW - 4 : upart * (NW / 4);
  const int uidx = pw == 4 ? warp - 4 : (part4 < pbase ? part4 : part4 - pw) + upart * (warp >> 2);
  const int ptid = pidx * 32 + lane;

  for (int j = warp; j < n; j += NW)
    for (int r = lane; r < n; r += 32) gj_cp16(S + (size_t)j * ldw + r, p.W + r + (size_t)j * p.ld);
  for (int r = tid; r < n; r += T) at[r] = 255;
  if (tid == 0) *sh_dead = 0;
  gj_cp_wait();
  __syncthreads();

  bool used = ptid >= n;

  // Gauss-Jordan steps of columns [s0, s0 + 8), in registers (warps that factor)
  auto factor = [&](int s0) {
    const int sw = min(SW, n - s0);
    cplx a[SW];
#pragma unroll
    for (int j = 0; j < SW; ++j)
      a[j] = (ptid < n && j < sw) ? S[(size_t)(s0 + j) * ldw + ptid] : make_double2(0.0, 0.0);
    unsigned key = 0, wkey = 0;
    auto search = [&] {
      const double v = cabs1(a[0]);
      key = !used && (unsigned)__double2hiint(v) <= 0x7ff00000u ? gj_key(v, ptid) : 0u;
      wkey = __reduce_max_sync(0xffffffffu, key);
    };
    search();
#pragma unroll 1
    for (int j = 0; j < sw; ++j) {
      const int buf = (j & 1) * 4;
      if (key == wkey && key != 0u) {
        cplx* ws = slot + (buf + pidx) * SW;
#pragma unroll
        for (int q = 1; q < SW; ++q) ws[q] = a[q];
        ws[0] = cinv_pivot(a[0]);
      }
      unsigned best = wkey;
      if (pw == 1) {
        __syncwarp();
      } else {
        if (lane == 0) part[buf + pidx] = wkey;
        asm volatile("bar.sync 1, %0;" ::"r"(PT) : "memory");
        best = max(part[buf], part[buf + 1]);
        if (pw == 4) best = max(best, max(part[buf + 2], part[buf + 3]));
      }
      const int pr = 1023 - (int)(best & 1023u);
      const cplx* row = slot + (buf + (pr % PT >> 5)) * SW;
      if (best < 2048u) {  // no candidate row, or zeros only (uniform)
        if (ptid == 0 && p.info) atomicCAS(p.info, 0, s0 + j + 1);
        if (best == 0u) {
          if (ptid == 0) *sh_dead = 1;
          break;
        }
      }
      if (ptid == PT - 1) {
        sh_piv[s0 + j] = pr;
        at[pr] = (uint8_t)(s0 / SW);
      }
      const cplx pv = row[0];
      const bool prow = ptid == pr;
      const cplx f = prow ? cneg(pv) : cmul(a[0], pv);
      used = used || prow;
#pragma unroll
      for (int q = 1; q < SW; ++q) {
        // the product apart, as in the updates: 3 % less error, no time
        const cplx x = row[q], c = prow ? make_double2(0.0, 0.0) : a[q];
        a[q - 1] = make_double2(c.x + fma(f.y, x.y, -f.x * x.x), c.y - fma(f.y, x.x, f.x * x.y));
        if (q == 1) search();
      }
      a[SW - 1] = cneg(f);
    }
#pragma unroll
    for (int q = 0; q < SW; ++q) {
      const int j = q - (SW - sw);
      if (ptid < n && j >= 0) S[(size_t)(s0 + j) * ldw + ptid] = a[q];
    }
  };
  // rank-8 update by sub-panel s of the column tiles [t0, t1) except s and skip, as
  // worker w of nw: row tiles of 16, or with more workers than row tiles a share
  // of the column tiles.  The products are summed apart and added to S last: in
  // one chain on S the error of an inverse is 15 to 20 % larger (above n = 112 the
  // rank-32 update sets the error, and the panels keep the one chain).
  auto update = [&](int s, int t0, int t1, int skip, int w, int nw) {
    const int sw = min(SW, n - s * SW), ms = min(mt, nw), ng = nw / ms;
    if (w >= ms * ng) return;
    const cplx z = make_double2(0.0, 0.0);
    for (int m = w % ms; m < mt; m += ms) {
      const int r0 = m * 16 + g, r1 = r0 + 8;
      const bool i0 = r0 < n, i1 = r1 < n;
      const bool o0 = i0 && at[r0] != s, o1 = i1 && at[r1] != s;  // pivot rows take the product alone
      cplx x0[2], x1[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int kk = tq + 4 * h;
        x0[h] = kk < sw && i0 ? S[(size_t)(s * SW + kk) * ldw + r0] : z;
        x1[h] = kk < sw && i1 ? S[(size_t)(s * SW + kk) * ldw + r1] : z;
      }
      for (int ct = t0 + w / ms; ct < t1; ct += ng) {
        if (ct == s || ct == skip) continue;
        cplx* C0 = S + (size_t)(ct * SW + 2 * tq) * ldw + r0;
        const cplx c00 = o0 ? C0[0] : z, c01 = o0 ? C0[ldw] : z, c10 = o1 ? C0[8] : z, c11 = o1 ? C0[ldw + 8] : z;
        double rr[4] = {}, ri[4] = {}, ii[4] = {}, ir[4] = {};
        const cplx* B = Bb + (size_t)(ct * SW + g) * SW;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const cplx y = B[(tq + 4 * h) ^ ((g & 1) << 2)];
          gj_dmma(rr, x0[h].x, x1[h].x, y.x);
          gj_dmma(ri, x0[h].x, x1[h].x, y.y);
          gj_dmma(ii, x0[h].y, x1[h].y, y.y);
          gj_dmma(ir, x0[h].y, x1[h].y, y.x);
        }
        if (i0) {
          C0[0] = make_double2(c00.x + (rr[0] - ii[0]), c00.y + (ri[0] + ir[0]));
          C0[ldw] = make_double2(c01.x + (rr[1] - ii[1]), c01.y + (ri[1] + ir[1]));
        }
        if (i1) {
          C0[8] = make_double2(c10.x + (rr[2] - ii[2]), c10.y + (ri[2] + ir[2]));
          C0[ldw + 8] = make_double2(c11.x + (rr[3] - ii[3]), c11.y + (ri[3] + ir[3]));
        }
      }
    }
  };

  if (factors) factor(0);
  __syncthreads();
  for (int s = 0; s < wt; ++s) {
    if (*sh_dead) return;  // singular: info is set, out is left untouched
    if (wt == 1) break;
    // the pivot rows in the other columns (unused k of a last, narrower tile: zero)
    const int sw = min(SW, n - s * SW);
    for (int i = tid; i < SW * SW * wt; i += T) {
      const int q = i / SW, j = i % SW;
      Bb[q * SW + (j ^ ((q & 1) << 2))] =
          q < n && j < sw ? S[(size_t)q * ldw + sh_piv[s * SW + j]] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (s + 1 == wt) {
      update(s, 0, wt, -1, warp, NW);
    } else {
      update(s, s + 1, s + 2, -1, warp, NW);  // the next 8 columns first, by all warps
      __syncthreads();
      if (factors) factor((s + 1) * SW);
      else if (updates) update(s, 0, wt, s + 1, uidx, nu);
    }
    __syncthreads();
  }
  // un-permuted: out[r, piv[c]] = S[piv[r], c]
  for (int c = warp; c < n; c += NW) {
    cplx* o = p.out + (size_t)sh_piv[c] * p.ldo;
    const cplx* Sc = S + (size_t)c * ldw;
    for (int r = lane; r < n; r += 32) o[r] = Sc[sh_piv[r]];
  }
}

// The rank-w update after a panel, in place: W[:, j] += S W[P, j] for the columns
// j outside the panel, without the old value at the pivot rows P; S is the
// panel's slab W[:, k0 .. k0 + w).  A CTA owns BN columns of one matrix and all
// of its rows: it gathers its part of the pivot rows first (nobody else writes
// those columns), then takes row tiles of 64, with the next tile's S rows in
// flight while it multiplies (3M products on the FP64 tensor path, as in the
// batched GEMM).
// Bounds: FP64 tensor time (8 n^2 w flops per matrix at 3/4) against 32 n^2
// bytes of W from L2 or HBM.  64 matrices of 256, w = 32: 53 us, 20 TFLOP/s of
// 8 n^2 w (69 us with the pivot rows staged through memory by the panel and
// the batched GEMM, whose gather also cost the panel 16 us).  BN = 32 for
// batches that fill the GPU; 16 columns when there are fewer CTAs than two per
// SM, since a CTA's row tiles run one after the other (one matrix: 15 us).
template <int BN>
__global__ void __launch_bounds__(256, 2)
    zgj_update_kernel(const ZInvProblem* __restrict__ probs, int k0, int nb, int stripes) {
  chain_entry();
  constexpr int BM = 64, ALD = BM + 2, BLD = kGjMaxNb + 4, NI = BN / 16;
  const int prob = blockIdx.x / stripes, c0 = (blockIdx.x - prob * stripes) * BN;
  const ZInvProblem& pp = probs[prob];
  const int n = pp.n, ld = pp.ld;
  if (c0 >= n || k0 >= n) return;
  const int w = min(nb, n - k0);
  if (c0 >= k0 && min(c0 + BN, n) <= k0 + w) return;  // the panel's own columns
  cplx* const W = pp.W;
  const int* const piv = pp.piv + k0;
  const int kp = (w + 3) & ~3;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* As = reinterpret_cast<cplx*>(smem_raw);  // [2][nb][ALD]: S rows of a tile, As[k][m]
  cplx* Bs = As + 2 * (size_t)((nb + 3) & ~3) * ALD;  // [BN][BLD]: pivot rows, Bs[n][k]
  uint8_t* isp = reinterpret_cast<uint8_t*>(Bs + BN * BLD);  // n: pivot rows of this panel
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  auto load_a = [&](int rt, int buf) {
    cplx* A = As + (size_t)buf * ((nb + 3) & ~3) * ALD;
    for (int i = tid; i < kp * BM; i += 256) {
      const int r = i % BM, kk = i / BM, gr = rt * BM + r;
      gj_cp16z(A + kk * ALD + r, W + gr + (size_t)(k0 + kk) * ld, gr < n && kk < w, W);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  load_a(0, 0);
  for (int i = tid; i < BN * kp; i += 256) {
    const int kk = i % kp, c = i / kp;
    const bool in = kk < w && c0 + c < n;
    const int pr = in ? max(piv[kk], 0) : 0;
    gj_cp16z(Bs + c * BLD + kk, W + pr + (size_t)(c0 + c) * ld, in, W);
  }
  asm volatile("cp.async.commit_group;\n" ::);
  for (int r = tid; r < n; r += 256) isp[r] = 0;
  __syncthreads();
  if (tid < w && piv[tid] >= 0) isp[piv[tid]] = 1;
  const int wm = (warp & 3) * 16, wn = (warp >> 2) * (BN / 2);
  const int nrt = (n + BM - 1) / BM;
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  for (int rt = 0; rt < nrt; ++rt) {
    if (rt + 1 < nrt) load_a(rt + 1, (rt + 1) & 1);
    // the old values of this warp's 16 x BN/2 part (zero at pivot rows)
    cplx old[NI][4];
#pragma unroll
    for (int x = 0; x < NI; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = rt * BM + wm + g + ((e >> 1) << 3), c = c0 + wn + x * 8 + 2 * tq + (e & 1);
        old[x][e] = r < n && c < n && !isp[r] ? W[r + (size_t)c * ld] : make_double2(0.0, 0.0);
      }
    double P1[NI][4] = {}, P2[NI][4] = {}, P3[NI][4] = {};
    const cplx* A = As + (size_t)(rt & 1) * ((nb + 3) & ~3) * ALD + wm + g;
    const cplx* B = Bs + (wn + g) * BLD + tq;
#pragma unroll 2
    for (int kk = 0; kk < kp; kk += 4) {
      const cplx x0 = A[(kk + tq) * ALD], x1 = A[(kk + tq) * ALD + 8];
      const double s0 = x0.x + x0.y, s1 = x1.x + x1.y;
#pragma unroll
      for (int x = 0; x < NI; ++x) {
        const cplx y = B[x * 8 * BLD + kk];
        gj_dmma(P1[x], x0.x, x1.x, y.x);
        gj_dmma(P2[x], x0.y, x1.y, y.y);
        gj_dmma(P3[x], s0, s1, y.x + y.y);
      }
    }
#pragma unroll
    for (int x = 0; x < NI; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = rt * BM + wm + g + ((e >> 1) << 3), c = c0 + wn + x * 8 + 2 * tq + (e & 1);
        if (r < n && c < n && (c < k0 || c >= k0 + w))
          W[r + (size_t)c * ld] = make_double2(old[x][e].x + (P1[x][e] - P2[x][e]),
                                               old[x][e].y + (P3[x][e] - P1[x][e] - P2[x][e]));
      }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
  }
}

// out[r, j] = W[piv[r], q[j]] with q the inverse permutation of piv:
// out[r, piv[c]] = W[piv[r], c].
__global__ void zgj_unpermute_kernel(const ZInvProblem* __restrict__ probs) {
  chain_entry();
  const ZInvProblem p = probs[blockIdx.y];
  const int n = p.n;
  // one thread per (r, c) element of W's column c -> output column piv[c]
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n * n; idx += gridDim.x * blockDim.x) {
    int c = idx / n, r = idx - c * n;
    int pc = p.piv[c], pr = p.piv[r];
    if (pc < 0 || pr < 0) continue;
    p.out[r + (size_t)pc * p.ldo] = p.W[pr + (size_t)c * p.ld];
  }
}

size_t zgj_panel_smem_bytes(int n, int nb) {
  const size_t w = nb < n ? nb : n, w8 = (w + gj::SW - 1) / gj::SW * gj::SW;
  size_t b = (size_t)(n | 1) * w8 * sizeof(cplx) + w8 * gj::SW * sizeof(cplx);
  b += 2 * 8 * (gj::SW * sizeof(cplx) + sizeof(unsigned)) + (w + 1) * sizeof(int) + n;
  return (b + 15) & ~size_t(15);
}

// Panels: one thread per row up to 256 rows (four warps up to 128, whose barriers
// are cheaper), then two and four rows per thread.  Whole matrices: four warps up
// to 32 rows, then eight.
cudaError_t launch_zgj_panel(const ZInvProblem* probs_dev, int nprob, int k0, int nb, int blocked, size_t smem,
                             cudaStream_t stream, int max_n) {
  if (nprob <= 0) return cudaSuccess;
  GjPanelArgs a{k0, nb, blocked};
  if (!blocked) {
    if (max_n <= 32) launch_chained(zgj_whole_kernel<128>, nprob, 128, smem, stream, probs_dev);
    else launch_chained(zgj_whole_kernel<256>, nprob, 256, smem, stream, probs_dev);
  } else if (max_n <= 128) launch_chained(zgj_panel_kernel<128, 1>, nprob, 128, smem, stream, probs_dev, a);
  else if (max_n <= 256) launch_chained(zgj_panel_kernel<256, 1>, nprob, 256, smem, stream, probs_dev, a);
  else if (max_n <= 512) launch_chained(zgj_panel_kernel<256, 2>, nprob, 256, smem, stream, probs_dev, a);
  else launch_chained(zgj_panel_kernel<256, 4>, nprob, 256, smem, stream, probs_dev, a);
  return cudaGetLastError();
}

static size_t zgj_update_smem_bytes(int max_n, int nb, int bn) {
  return (2 * (size_t)((nb + 3) & ~3) * 66 + (size_t)bn * (kGjMaxNb + 4)) * sizeof(cplx) + ((max_n + 15) & ~15);
}

cudaError_t launch_zgj_update(const ZInvProblem* probs_dev, int nprob, int k0, int nb, int max_n, cudaStream_t stream) {
  if (nprob <= 0) return cudaSuccess;
  if (nb > kGjMaxNb) return cudaErrorInvalidValue;
  const int s32 = (max_n + 31) / 32;
  if ((long long)nprob * s32 >= 2 * 148) {
    launch_chained(zgj_update_kernel<32>, nprob * s32, 256, zgj_update_smem_bytes(max_n, nb, 32), stream, probs_dev,
                   k0, nb, s32);
  } else {
    const int s16 = (max_n + 15) / 16;
    launch_chained(zgj_update_kernel<16>, nprob * s16, 256, zgj_update_smem_bytes(max_n, nb, 16), stream, probs_dev,
                   k0, nb, s16);
  }
  return cudaGetLastError();
}

// Raise the dynamic shared-memory limit of the panel kernels (outside capture).
// The attribute is process-wide, so it is always set to the device's opt-in
// maximum: a later, smaller request never lowers the limit another live plan
// relies on.
cudaError_t zgj_prepare(size_t smem) {
  int dev = 0, mx = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&mx, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  if (smem > (size_t)mx) return cudaErrorInvalidValue;
  static PerDevice set;
  if (set.done(dev)) return cudaSuccess;
  for (const void* f : {(const void*)zgj_panel_kernel<128, 1>, (const void*)zgj_panel_kernel<256, 1>,
                        (const void*)zgj_panel_kernel<256, 2>, (const void*)zgj_panel_kernel<256, 4>,
                        (const void*)zgj_whole_kernel<128>, (const void*)zgj_whole_kernel<256>,
                        (const void*)zgj_update_kernel<16>, (const void*)zgj_update_kernel<32>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
  if (e == cudaSuccess) set.set(dev);
  return e;
}

cudaError_t launch_zgj_unpermute(const ZInvProblem* probs_dev, int nprob, int max_n, cudaStream_t stream) {
  if (nprob <= 0) return cudaSuccess;
  int per = max_n * max_n;
  int bx = (per + 255) / 256;
  if (bx > 64) bx = 64;
  dim3 grid(bx, nprob);
  launch_chained(zgj_unpermute_kernel, grid, 256, 0, stream, probs_dev);
  return cudaGetLastError();
}

}  // namespace negf
