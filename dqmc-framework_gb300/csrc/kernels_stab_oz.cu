// kernels_stab_oz.cu — stabilization of HBM walkers (32 < N <= 768): the UDT
// push and the Green's assembly as Householder factorizations whose blocked
// matrix products run on the BF16 tensor cores at FP64 accuracy (mixed walkers
// with N >= 128, WalkerDev::ozstab 1) or in FP64 (FP64 walkers, and mixed ones
// below 128 sites, where a product does not fill the tensor core's tiles; 2).
//
// Reference: SvdStack::push (src/svd_stack.cpp:34-87) factors the B-chain with
// MKL dgesvd and compute_equaltime_greens (include/utils/numerical_stable.hpp:
// 186-239) assembles G through an LU inverse.  The plain path restates them
// with column-pivoted QR (kernels_general.cu), a latency-bound FP64 loop.  Here
//   push:   with tensor-core products the columns of the chain are ordered
//           once by norm (pre-pivoting, Bai, Lee, Li and Xu, Linear Algebra
//           Appl. 435 (2011) 659) and factored by blocked Householder QR with
//           32-column panels.  Each panel is factored in FP64 in shared memory
//           (LAPACK dgeqr2 and dlarft order); the trailing update A -= V T^T
//           (V^T A) is two products.  With FP64 products the QR pivots on every
//           column (zqrp_kernel).  The formation of Q and F = D^-1 R P^T F_prev
//           are products in both.
//   greens: M = Dlmax^-1 U_L^T U_R Drmax^-1 + Dlmin F_L F_R^T Drmin and
//           Y = Dlmax^-1 U_L^T; M = QR by the same blocked Householder; X =
//           R^-1 Q^T Y by blocked reflector application and blocked back
//           substitution (FP64 diagonal blocks); G = U_R Drmax^-1 X.  Boundary
//           steps (one stack empty) form M = Y + Dmin F and G = X or X^T.
//   dynamic half-sweep (compute_dynamic_greens, include/utils/numerical_stable.hpp:
//           246-325): the same factorization of M also solves the second
//           right-hand side Y2 = Dlmin F_L, X2 = M^-1 Y2; then G(t,0) = U_R
//           Drmax^-1 X2 and G(0,t) = -F_R^T Drmin X (at t = beta, right stack
//           empty: G(beta,0) = X2, G(0,beta) = -X).
// Every product slices its two FP64 operands once (zslice_kernel, tensor-core
// images) into 8 integer slices of 7 bits (56 significant bits, K <= 256) or 9
// of 6 (54 bits, K <= 1024) and multiplies them on the BF16 tensor cores with
// FP32 accumulation (exact for the leading weight groups; zgemm_tc_kernel
// streams the slices through oztc::mainloop): an FP64-class GEMM.  The panel
// folds its T factor into the reflectors (Vt = V T, or V T^T when forming Q),
// so applying a block reflector is two products.  Panels, diagonal solves,
// reflectors and reductions are native FP64.  G equals the pivoted-QR path's
// mathematically; the UDT factors differ only in the column order of the QR.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <utility>

#include "dqmc_device.cuh"
#include "ozaki.cuh"
#include "oz_tc.cuh"
#include "tcgen05.cuh"

namespace dqmc {

namespace {

constexpr int TB = 32;           // Householder panel width
constexpr int QW = 8;            // warps of a CTA of the column-pivoted QR

__device__ __forceinline__ double zwarp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void zstack_tops(const WalkerDev& w, int mode, int j, int& nl, int& nr) {
  if (mode == MODE_FWD) { nl = j + 1; nr = w.nstack - 1 - j; }
  else if (mode == MODE_BWD) { nl = w.nstack - 1 - j; nr = j + 1; }
  else { nl = 0; nr = w.nstack; }
}

// per-spin scratch: scr = X (matrix being factored) | Y (right-hand sides);
// zwk = Wb [TB N] | W2 [TB N] | T factors [ceil(N/TB) TB TB] | invd | four
// diagonal scale vectors | perm | line exponents of the operands of the
// current product, A and up to three parts of B (stab_scratch_elems)
struct ZScr {
  double *X, *Y, *Wb, *W2, *Tb, *invd, *dlmaxi, *drmaxi, *dlmin, *drmin;
  int *perm, *expA, *expB;
};
__device__ __forceinline__ ZScr zscr(const WalkerDev& w, int sp) {
  const long long NN = (long long)w.N * w.N;
  const long long TN = (long long)TB * w.N;
  const long long TT = (long long)TB * TB * ((w.N + TB - 1) / TB);
  ZScr z;
  z.X = w.scr + sp * 2 * NN;
  z.Y = z.X + NN;
  double* wk = w.zwk + sp * w.zwk_stride;
  z.Wb = wk;
  z.W2 = wk + TN;
  z.Tb = wk + 2 * TN;
  z.invd = wk + 2 * TN + TT;
  z.dlmaxi = z.invd + w.N;
  z.drmaxi = z.dlmaxi + w.N;
  z.dlmin = z.drmaxi + w.N;
  z.drmin = z.dlmin + w.N;
  z.perm = reinterpret_cast<int*>(z.drmin + w.N);
  z.expA = z.perm + w.N;
  z.expB = z.expA + w.N;
  return z;
}

// Wb of a product's part: the further parts occur in the Green's assembly only, where the chain's two
// buffers are free (the push has factored it, the next step writes it anew)
__device__ __forceinline__ double* zwb(const WalkerDev& w, const ZScr& z, int sp, int part) {
  return part == 0 ? z.Wb : w.chain + ((long long)(part - 1) * w.S + sp) * w.N * w.N;
}

// An operand of C = op(A) op(B).  Element (row, col) of the stored block sits at
// p[col * ld + row'] with row' = rowmap ? rowmap[row] : row.  For A the logical
// element (i, k) is stored (i, k), or (k, i) when tr; for B the logical (k, i)
// is stored (k, i), or (i, k) when tr (i: output row of A / column of B).
struct ZOpnd {
  const double* p;
  long long ld;
  int tr;
  int kind;            // 0 full, 1 unit lower (Householder vectors), 2 upper with diagonal
  const int* rowmap;
  const double* ks;    // multiplier along k, or null
};
struct ZJob {
  ZOpnd a, b;
  double* c;
  long long ldc;
  int M, N, K;
  int beta;            // 1: C += (-1)^neg AB
  int neg;             // 1: the product enters negated (an operand modifier, no FP64 multiply)
  const double* rs;    // row multiplier of the product, or null
  const double* cs;    // column multiplier, or null
  int out;             // 1: Green's function output (wrap error, trace, spin copy);
                       // 2: time-displaced output (wrap error against the propagated value)
};

// the ping-pong slot of G(t,0) or G(0,t) at slice t ([parity][S][N*N])
__device__ __forceinline__ double* zdyn_slot(double* base, const WalkerDev& w, int sp, int t) {
  return base + ((long long)(t & 1) * w.S + sp) * w.N * w.N;
}

__device__ __forceinline__ double zel(const ZOpnd& o, int i, int k, bool isB) {
  const int row = (o.tr != (int)isB) ? k : i;
  const int col = (o.tr != (int)isB) ? i : k;
  double v;
  if (o.kind == 1 && row <= col) v = (row == col) ? 1.0 : 0.0;
  else if (o.kind == 2 && row > col) v = 0.0;
  else v = o.p[(long long)col * o.ld + (o.rowmap ? o.rowmap[row] : row)];
  if (o.ks) v *= o.ks[k];
  return v;
}

// The block reflector of panel p is I - V_p T_p V_p^T.  Its T factor is folded
// into the reflectors once per panel in FP64, Vt = V_p T_p (applying Q_p^T:
// T_p^T V_p^T A = Vt^T A) or Vt = V_p T_p^T (applying Q_p), so that every
// application is two products: Wb = Vt^T A, A -= V_p Wb.
enum ZOp {
  // Q_p^T applied to the trailing matrix X(j0:, j0+pb:) (part 0) and, in the Green's assembly, to
  // the right-hand sides Y(j0:, :) (part 1) and Y2(j0:, :) (part 2, the dynamic half-sweep): the
  // parts are further columns of one product
  Z_QR_W = 0,    // Wb[part] = (V_p T_p)^T part
  Z_QR_UPD,      // part -= V_p Wb[part]
  Z_Q_W,         // Wb = (V_p T_p^T)^T U(j0:, j0:)   (forming Q, backward)
  Z_Q_UPD,       // U(j0:, j0:) -= V_p Wb
  Z_F,           // F = D^-1 R P^T F_prev
  Z_GA,          // M = Dlmax^-1 U_L^T U_R Drmax^-1
  Z_GB,          // M += Dlmin F_L F_R^T Drmin
  Z_TR_UPD,      // Y(j0:j0+pb, :) -= R(j0:j0+pb, j0+pb:) Y(j0+pb:, :) (part 0), Y2 likewise (part 1)
  Z_GG,          // G = U_R Drmax^-1 X
  Z_GRAM,        // Zg = V_p^T V_p (pb x pb, into Wb): the Gram matrix of the panel's reflectors
  Z_VT,          // Vt = V_p T_p (m x pb, into W2), T_p from ztfac_kernel
  // the dynamic half-sweep's outputs (second right-hand side Y2: dynx)
  Z_DT0_OUT,     // G(t,0) = U_R Drmax^-1 X2
  Z_D0T_OUT,     // G(0,t) = -F_R^T Drmin X
};

// A launch's column tiles: `first` of part p0, then `rest` of each further part
struct ZTiles {
  int first, rest, p0;
  __device__ __forceinline__ int part(int x) const { return p0 + (x < first ? 0 : 1 + (x - first) / rest); }
  __device__ __forceinline__ int col(int x) const { return x < first ? x : (x - first) % rest; }
};

// the job of op's part (columns of the product; parts share the operand A)
__device__ bool zjob(const WalkerDev& w, int op, int mode, int j, int p, int sp, int part, ZJob& jb) {
  if (j >= w.nstack) return false;
  const int N = w.N;
  const long long NN = (long long)N * N;
  const ZScr z = zscr(w, sp);
  const int j0 = p * TB;
  const int m = N - j0, pb = min(TB, m);
  jb = ZJob{};
  const bool panel_op = op != Z_F && op != Z_GA && op != Z_GB && op != Z_GG;
  if (panel_op && j0 >= N) return false;
  const ZOpnd Vp{z.X + (long long)j0 * N + j0, N, 0, 1, nullptr, nullptr};
  const ZOpnd VtT{z.W2, N, 1, 0, nullptr, nullptr};  // Vt^T (Vt: m x pb, ld N, in W2)
  const ZOpnd Wbo{z.Wb, TB, 0, 0, nullptr, nullptr};
  int nl = 0, nr = 0;
  zstack_tops(w, mode, j, nl, nr);
  const int side = (mode == MODE_FWD) ? 0 : 1;
  switch (op) {
    case Z_QR_W:
    case Z_QR_UPD: {
      if (part == 2 && !w.dynx) return false;
      const int nt = (part == 0) ? m - pb : N;
      if (nt <= 0) return false;
      double* C = (part == 0) ? z.X + (long long)(j0 + pb) * N + j0 : (part == 1 ? z.Y : w.dynx + sp * NN) + j0;
      double* Wp = zwb(w, z, sp, part);
      if (op == Z_QR_W) {
        jb.a = VtT;
        jb.b = ZOpnd{C, N, 0, 0, nullptr, nullptr};
        jb.c = Wp; jb.ldc = TB; jb.M = pb; jb.N = nt; jb.K = m;
      } else {
        jb.a = Vp;
        jb.b = ZOpnd{Wp, TB, 0, 0, nullptr, nullptr};
        jb.c = C; jb.ldc = N; jb.M = m; jb.N = nt; jb.K = pb;
        jb.beta = 1; jb.neg = 1;
      }
      return true;
    }
    case Z_Q_W:
    case Z_Q_UPD: {
      double* Uo = stack_level(w, side, sp, j);
      if (op == Z_Q_W) {
        jb.a = VtT;
        jb.b = ZOpnd{Uo + (long long)j0 * N + j0, N, 0, 0, nullptr, nullptr};
        jb.c = z.Wb; jb.ldc = TB; jb.M = pb; jb.N = m; jb.K = m;
      } else {
        jb.a = Vp;
        jb.b = Wbo;
        jb.c = Uo + (long long)j0 * N + j0; jb.ldc = N; jb.M = m; jb.N = m; jb.K = pb;
        jb.beta = 1; jb.neg = 1;
      }
      return true;
    }
    case Z_F: {
      if (j == 0) return false;
      double* lv = stack_level(w, side, sp, j);
      const double* fp = stack_level(w, side, sp, j - 1) + NN;
      jb.a = ZOpnd{z.X, N, 0, 2, nullptr, nullptr};
      jb.b = ZOpnd{fp, N, 0, 0, z.perm, nullptr};
      jb.rs = z.invd;
      jb.c = lv + NN; jb.ldc = N; jb.M = N; jb.N = N; jb.K = N;
      return true;
    }
    case Z_GA:
    case Z_GB:
    case Z_GG: {
      if (!(nl > 0 && nr > 0)) return false;
      const double* UL = stack_level(w, 0, sp, nl - 1);
      const double* UR = stack_level(w, 1, sp, nr - 1);
      if (op == Z_GA) {
        jb.a = ZOpnd{UL, N, 1, 0, nullptr, nullptr};
        jb.b = ZOpnd{UR, N, 0, 0, nullptr, nullptr};
        jb.rs = z.dlmaxi; jb.cs = z.drmaxi;
        jb.c = z.X; jb.ldc = N; jb.M = N; jb.N = N; jb.K = N;
      } else if (op == Z_GB) {
        jb.a = ZOpnd{UL + NN, N, 0, 0, nullptr, nullptr};
        jb.b = ZOpnd{UR + NN, N, 1, 0, nullptr, nullptr};
        jb.rs = z.dlmin; jb.cs = z.drmin;
        jb.c = z.X; jb.ldc = N; jb.M = N; jb.N = N; jb.K = N; jb.beta = 1;
      } else {
        jb.a = ZOpnd{UR, N, 0, 0, nullptr, z.drmaxi};
        jb.b = ZOpnd{z.Y, N, 0, 0, nullptr, nullptr};
        jb.c = w.G + sp * NN; jb.ldc = N; jb.M = N; jb.N = N; jb.K = N; jb.out = 1;
      }
      return true;
    }
    case Z_TR_UPD: {
      if (j0 + pb >= N) return false;
      if (part == 1 && !w.dynx) return false;
      double* Yr = (part == 0) ? z.Y : w.dynx + sp * NN;
      jb.a = ZOpnd{z.X + (long long)(j0 + pb) * N + j0, N, 0, 0, nullptr, nullptr};
      jb.b = ZOpnd{Yr + j0 + pb, N, 0, 0, nullptr, nullptr};
      jb.c = Yr + j0; jb.ldc = N; jb.M = pb; jb.N = N; jb.K = N - j0 - pb;
      jb.beta = 1; jb.neg = 1;
      return true;
    }
    case Z_GRAM:
      jb.a = ZOpnd{z.X + (long long)j0 * N + j0, N, 1, 1, nullptr, nullptr};  // V_p^T
      jb.b = Vp;
      jb.c = z.Wb; jb.ldc = TB; jb.M = pb; jb.N = pb; jb.K = m;
      return true;
    case Z_VT:
      jb.a = Vp;
      jb.b = ZOpnd{z.Tb + (long long)p * TB * TB, TB, 0, 2, nullptr, nullptr};  // T_p, upper with diagonal
      jb.c = z.W2; jb.ldc = N; jb.M = m; jb.N = pb; jb.K = pb;
      return true;
    case Z_DT0_OUT:
    case Z_D0T_OUT: {
      // forward step j of the dynamic half-sweep, both stacks present
      if (!w.gt0 || !w.dynx || mode != MODE_FWD || !(nl > 0 && nr > 0)) return false;
      const int t_end = min((j + 1) * w.pace, w.Lt);
      const double* UR = stack_level(w, 1, sp, nr - 1);
      if (op == Z_DT0_OUT) {
        jb.a = ZOpnd{UR, N, 0, 0, nullptr, z.drmaxi};
        jb.b = ZOpnd{w.dynx + sp * NN, N, 0, 0, nullptr, nullptr};
        jb.c = zdyn_slot(w.gt0, w, sp, t_end);
      } else {
        jb.a = ZOpnd{UR + NN, N, 1, 0, nullptr, z.drmin};  // F_R^T, times Drmin along k
        jb.b = ZOpnd{z.Y, N, 0, 0, nullptr, nullptr};
        jb.c = zdyn_slot(w.g0t, w, sp, t_end);
        jb.neg = 1;
      }
      jb.ldc = N; jb.M = N; jb.N = N; jb.K = N; jb.out = 2;
      return true;
    }
  }
  return false;
}

// Where a product's slices lie in zsl: one image of the lines of A, then those of B's parts, each
// rounded up to 32, and K rounded up to 32, so that a spin needs the room of two N x N operands
// whatever the product (2 N lines of K = N; a panel's 32 lines beside its trailing columns and N
// right-hand sides are no more).  A third part of K = m would need more: it takes the second one's
// lines after that has been used (Z_QR_W of the dynamic half-sweep).  A tile reads 128 lines of A,
// also past the image's last one: only where the image is far below the room, and what it reads
// there ends in rows that are not stored.
struct ZImage {
  int line_b, nlb;  // the part's first line, 8-line blocks of the image
  long long sst;    // elements of a slice
};
__device__ __forceinline__ ZImage zimage(const WalkerDev& w, int op, int p, const ZJob& jb, int part) {
  const auto up = [](int x) { return (x + 31) / 32 * 32; };
  const int nr = up(w.N), M = up(jb.M), Kp = up(jb.K);
  ZImage im;
  int lines;
  if (op == Z_QR_W || op == Z_QR_UPD) {
    const int rest = up(max(w.N - (p + 1) * TB, 0));  // part 0: the trailing columns
    const int slot = (op == Z_QR_W) ? min(part, 1) : part;
    im.line_b = M + (slot == 0 ? 0 : rest + (slot - 1) * nr);
    lines = M + rest + (op == Z_QR_W ? 1 : 2) * nr;
  } else {
    im.line_b = M + part * up(jb.N);
    lines = M + (op == Z_TR_UPD ? 2 : 1) * up(jb.N);
  }
  im.nlb = lines / 8;
  im.sst = (long long)lines * Kp;
  return im;
}
// the start of spin sp's slices (room for 9 slices of two N x N operands a spin)
__device__ __forceinline__ unsigned short* zslices(const WalkerDev& w, int sp) {
  return w.zsl + (long long)sp * 2 * 9 * ozaki::tc_lines(w.N) * w.zld;
}

// fixed-point magnitude |x| / 2^e with Q fraction bits (e >= exp_bound(x), Q <= 62)
__device__ __forceinline__ unsigned long long zfixed(double x, int e, int Q, bool& neg) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  neg = (b >> 63) != 0;
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex == 0) return 0ULL;
  const unsigned long long mant = (b & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL;
  const int s = ex - 1075 - e + Q;  // |x| 2^{Q-e} = mant 2^s
  if (s >= 0) return mant << s;     // s <= Q - 53 here
  if (s <= -64) return 0ULL;
  return mant >> (-s);
}

}  // namespace

// --------------------------------------------------------------------------
// Slicing of both operands of a product, once per product: blockIdx.y + y0 = 0 the
// rows of op(A), 1 + part the columns of op(B); 32 lines per CTA.  Pass 1: the line
// exponents (8 k groups per line); pass 2: 32 x 32 tiles staged through
// shared memory so that loads run along the stored matrix.  Output: S
// slices in the tensor core's shared-memory image (ozaki::tc_index, zimage), zero
// past K up to a multiple of 32.
// --------------------------------------------------------------------------
template <int S, int B>
__global__ void __launch_bounds__(256) zslice_kernel(const WalkerDev* __restrict__ W, int op, int mode, int j, int p,
                                                     int y0) {
  const int wi = blockIdx.z >> 1, sp = blockIdx.z & 1;
  const WalkerDev& w = W[wi];
  if (w.ozstab != 1 || sp >= w.S) return;
  ZJob jb;
  const int y = blockIdx.y + y0;
  const bool isB = y != 0;
  // A by the part that every step has
  const int part = isB ? y - 1 : (gridDim.y > 2 && (op == Z_QR_W || op == Z_QR_UPD)) ? 1 : 0;
  if (!zjob(w, op, mode, j, p, sp, part, jb)) return;
  if ((jb.K <= 256) != (B == 7)) return;
  const ZOpnd& o = isB ? jb.b : jb.a;
  const int nlines = isB ? jb.N : jb.M;
  const int l0 = blockIdx.x * 32;
  if (l0 >= nlines) return;
  constexpr int Q = S * B;
  const int N = w.N, Kp = (jb.K + 31) / 32 * 32;
  const ZScr z = zscr(w, sp);
  const ZImage im = zimage(w, op, p, jb, part);
  unsigned short* out = zslices(w, sp) + (isB ? im.line_b / 8 * 128 : 0);
  // lines contiguous in memory when the stored row index runs along the line
  const bool line_fast = (o.tr == (int)isB);
  __shared__ int s_e[8][32];
  __shared__ double s_t[32][33];
  {
    const int ll = line_fast ? (threadIdx.x & 31) : (threadIdx.x >> 3);
    const int kg = line_fast ? (threadIdx.x >> 5) : (threadIdx.x & 7);
    const int line = l0 + ll;
    int e = -1100;
    if (line < nlines)
      for (int k0 = kg; k0 < jb.K; k0 += 64) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int k = k0 + 8 * u;
          x[u] = (k < jb.K) ? zel(o, line, k, isB) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) e = max(e, ozaki::exp_bound(x[u]));
      }
    s_e[kg][ll] = e;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int m = s_e[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < 8; ++q) m = max(m, s_e[q][threadIdx.x]);
    s_e[0][threadIdx.x] = m;
    if (l0 + threadIdx.x < nlines) (isB ? z.expB + (long long)part * N : z.expA)[l0 + threadIdx.x] = m;
  }
  __syncthreads();
  for (int k0 = 0; k0 < Kp; k0 += 32) {
    for (int e = threadIdx.x; e < 32 * 32; e += 256) {
      const int ll = line_fast ? (e & 31) : (e >> 5), kk = line_fast ? (e >> 5) : (e & 31);
      const int line = l0 + ll, k = k0 + kk;
      s_t[ll][kk] = (line < nlines && k < jb.K) ? zel(o, line, k, isB) : 0.0;
    }
    __syncthreads();
    {  // one line and 4 consecutive k per thread: one 8-byte store per slice
      const int kq = threadIdx.x & 7, ll = threadIdx.x >> 3, line = l0 + ll;
      if (line < nlines) {
        unsigned long long q[4];
        bool ng[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = zfixed(s_t[ll][kq * 4 + u], s_e[0][ll], Q, ng[u]);
        unsigned short* o = out + ozaki::tc_index(line, k0 + kq * 4, im.nlb);
#pragma unroll
        for (int s2 = 0; s2 < S; ++s2) {
          ushort4 v;
          v.x = ozaki::slice_bf16q(q[0], s2, B, Q, ng[0]);
          v.y = ozaki::slice_bf16q(q[1], s2, B, Q, ng[1]);
          v.z = ozaki::slice_bf16q(q[2], s2, B, Q, ng[2]);
          v.w = ozaki::slice_bf16q(q[3], s2, B, Q, ng[3]);
          *reinterpret_cast<ushort4*>(o + s2 * im.sst) = v;
        }
      }
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------------
// The product on the 5th-generation tensor cores (tcgen05): a 128 x NT output
// tile per CTA, the S weight groups accumulated in TMEM (S NT columns), the
// pre-sliced operands streamed by oztc::mainloop (bulk copies through a ring
// of NS stages of 16-deep k chunks).  The 56-bit configuration runs 128 x 32
// tiles with 2 stages so that two CTAs share an SM (256 TMEM columns, 80 KB of
// shared memory and at most 128 registers each): one CTA's epilogue overlaps
// the other's copies and MMAs.
// --------------------------------------------------------------------------
template <int S, int B, int NT, int NS, int MINB>
__global__ void __launch_bounds__(256, MINB) zgemm_tc_kernel(const WalkerDev* __restrict__ W, int op, int mode, int j,
                                                             int p, int trace_slot, ZTiles tl) {
  constexpr int MT = 128;
  constexpr int CW = (MINB > 1) ? 8 : 16;  // TMEM columns per load in the epilogue
  constexpr unsigned TCOLS = (S * NT <= 256) ? 256u : 512u;
  static_assert(MINB == 1 || S * NT <= 256, "two CTAs per SM need at most 256 TMEM columns each");
  const int wi = blockIdx.z >> 1, sp = blockIdx.z & 1;
  const WalkerDev& w = W[wi];
  if (w.ozstab != 1 || sp >= w.S) return;
  ZJob jb;
  const int part = tl.part(blockIdx.x);
  if (!zjob(w, op, mode, j, p, sp, part, jb)) return;
  if ((jb.K <= 256) != (B == 7)) return;
  const int r0 = blockIdx.y * MT, c0 = tl.col(blockIdx.x) * NT;
  if (r0 >= jb.M || c0 >= jb.N) return;
  extern __shared__ __align__(1024) unsigned char tsm[];
  __shared__ int eA[MT], eB[NT];
  __shared__ __align__(8) unsigned long long full[NS], done[NS];
  __shared__ unsigned tbase;
  __shared__ int s_fail, s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const ZScr z = zscr(w, sp);
  const int N = w.N;
  if (tid < MT) eA[tid] = (r0 + tid < jb.M) ? z.expA[r0 + tid] : -1100;
  if (tid < NT) eB[tid] = (c0 + tid < jb.N) ? z.expB[(long long)part * N + c0 + tid] : -1100;
  if (tid == 0) {
    s_fail = 0;
    s_last = -1;
    for (int i = 0; i < NS; ++i) {
      tc::mbar_init(&full[i]);
      tc::mbar_init(&done[i]);
    }
    tc::mbar_fence_init();
  }
  if (warp == 0) tc::alloc(&tbase, TCOLS);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const unsigned taddr = tbase;
  if (tid == 0) {
    const ZImage im = zimage(w, op, p, jb, part);
    const unsigned short* zA = zslices(w, sp);
    bool ok;
    s_last = oztc::mainloop<S, MT, NT, NS>(tsm, full, done, taddr, zA + (long long)(r0 / 8) * 128,
                                            zA + (long long)((im.line_b + c0) / 8) * 128, im.sst, im.nlb * 128LL,
                                            (jb.K + 15) / 16, ok);
    s_fail = ok ? 0 : 1;
  }
  __syncthreads();
  {
    const int last = s_last;
    const bool mma_done = last >= 0 && tc::mbar_wait(&done[last % NS], (last / NS) & 1);
    if (__syncthreads_or(!mma_done || s_fail) && tid == 0) s_fail = 1;
  }
  tc::fence_after();
  __syncthreads();

  // epilogue: warp w reads TMEM lanes 32 (w & 3) .. + 31 (rows), column half (w >> 2)
  const long long NN = (long long)w.N * w.N;
  double err = 0.0;
  bool finite = true;
  double* tr = (jb.out && w.trace && trace_slot >= 0 && trace_slot < w.trace_cap)
                   ? w.trace + ((long long)trace_slot * 2 + sp) * NN : nullptr;
  const bool check = (jb.out == 2) || (jb.out && !(mode == MODE_INIT || (mode == MODE_BWD && j == w.nstack - 1)));
  const int q4 = warp & 3, half = warp >> 2;
  const int rl = q4 * 32 + lane, r = r0 + rl;
  // K <= 32: every group sum is below 2^22 and converts with an FP32 add (the conversion
  // unit does ~15 per clock per SM); warps whose 32 rows are all past M skip the epilogue
  const bool small_k = jb.K <= 32;
  if (!s_fail && r0 + q4 * 32 < jb.M) {
    for (int cc = half * (NT / 2); cc < (half + 1) * (NT / 2); cc += CW) {
      uint32_t v[S][CW];
#pragma unroll
      for (int m = 0; m < S; ++m) tc::ldw<CW>(v[m], taddr + ((unsigned)(q4 * 32) << 16) + (unsigned)(m * NT + cc));
      tc::wait_ld();
#pragma unroll
      for (int u = 0; u < CW; ++u) {
        const int cl = cc + u, col = c0 + cl;
        if (r >= jb.M || col >= jb.N) continue;
        long long hi = 0, lo = 0;
        if (small_k) {
#pragma unroll
          for (int m = 0; m < 4; ++m) hi = (hi << B) + (long long)ozaki::f2i_small(__uint_as_float(v[m][u]));
#pragma unroll
          for (int m = 4; m < S; ++m) lo = (lo << B) + (long long)ozaki::f2i_small(__uint_as_float(v[m][u]));
        } else {
#pragma unroll
          for (int m = 0; m < 4; ++m) hi = (hi << B) + (long long)__float2int_rn(__uint_as_float(v[m][u]));
#pragma unroll
          for (int m = 4; m < S; ++m) lo = (lo << B) + (long long)__float2int_rn(__uint_as_float(v[m][u]));
        }
        const int e = eA[rl] + eB[cl];
        double val = ozaki::combine_hilo<S, B>(hi, lo, e);
        if (jb.rs) val *= jb.rs[r];
        if (jb.cs) val *= jb.cs[col];
        const long long o = (long long)col * jb.ldc + r;
        if (!jb.out) {
          if (jb.neg) val = -val;
          jb.c[o] = jb.beta ? jb.c[o] + val : val;
        } else if (jb.out == 2) {
          if (jb.neg) val = -val;
          err = fmax(err, fabs(val - jb.c[o]));
          if (!isfinite(val)) finite = false;
          jb.c[o] = val;
        } else {
          if (check) err = fmax(err, fabs(val - jb.c[o]));
          if (!isfinite(val)) finite = false;
          jb.c[o] = val;
          if (tr) tr[o] = val;
          if (w.S == 1) {
            jb.c[NN + o] = val;
            if (tr) tr[NN + o] = val;
          }
        }
      }
    }
  }
  if (s_fail && tid == 0) atomicOr(w.status, ST_TIMEOUT);
  if (jb.out) {
    if (!finite) atomicOr(w.status, ST_NONFINITE_G);
    if (check) {
      for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
      if (lane == 0) atomicMax(w.wrap_bits, (unsigned long long)__double_as_longlong(err));
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::dealloc(taddr, TCOLS);
}

// --------------------------------------------------------------------------
// The same product in FP64 (ozstab 2): a 16 x 16 output tile per CTA, an element per thread, K in
// steps of 32 through shared memory, operands read through zel.  FP64 issue bounds it (one warp
// operation per 19 cycles and SM), so the tile is small: a product of 32 rows and K = 256 still
// reaches 32 SMs per matrix.
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(256) zgemm_f64_kernel(const WalkerDev* __restrict__ W, int op, int mode, int j, int p,
                                                        int trace_slot, ZTiles tl) {
  const int wi = blockIdx.z >> 1, sp = blockIdx.z & 1;
  const WalkerDev& w = W[wi];
  if (w.ozstab != 2 || sp >= w.S) return;
  ZJob jb;
  if (!zjob(w, op, mode, j, p, sp, tl.part(blockIdx.x), jb)) return;
  const int r0 = blockIdx.y * 16, c0 = tl.col(blockIdx.x) * 16;
  if (r0 >= jb.M || c0 >= jb.N) return;
  __shared__ double As[32][17], Bs[32][17];
  const int tid = threadIdx.x, lane = tid & 31;
  const int rl = tid & 15, cl = tid >> 4, r = r0 + rl, col = c0 + cl;
  const bool a_fast = jb.a.tr == 0, b_fast = jb.b.tr == 1;  // lines contiguous in memory
  double acc4[4] = {0.0, 0.0, 0.0, 0.0};  // k mod 4: independent FMA chains, and shorter sums
  // the upper (kind 2, not transposed) operand A is zero left of the diagonal
  const int k_first = (jb.a.kind == 2 && !jb.a.tr) ? r0 / 32 * 32 : 0;
  for (int k0 = k_first; k0 < jb.K; k0 += 32) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = tid + 256 * u;
      const int la = a_fast ? e & 15 : e >> 5, ka = a_fast ? e >> 4 : e & 31;
      As[ka][la] = (r0 + la < jb.M && k0 + ka < jb.K) ? zel(jb.a, r0 + la, k0 + ka, false) : 0.0;
      const int lb = b_fast ? e & 15 : e >> 5, kb = b_fast ? e >> 4 : e & 31;
      Bs[kb][lb] = (c0 + lb < jb.N && k0 + kb < jb.K) ? zel(jb.b, c0 + lb, k0 + kb, true) : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 32; ++k) acc4[k & 3] = fma(As[k][rl], Bs[k][cl], acc4[k & 3]);
    __syncthreads();
  }
  const double acc = (acc4[0] + acc4[1]) + (acc4[2] + acc4[3]);
  const long long NN = (long long)w.N * w.N;
  const bool check = (jb.out == 2) || (jb.out && !(mode == MODE_INIT || (mode == MODE_BWD && j == w.nstack - 1)));
  double err = 0.0;
  if (r < jb.M && col < jb.N) {
    double val = acc;
    if (jb.rs) val *= jb.rs[r];
    if (jb.cs) val *= jb.cs[col];
    if (jb.neg) val = -val;
    const long long o = (long long)col * jb.ldc + r;
    if (!jb.out) {
      jb.c[o] = jb.beta ? jb.c[o] + val : val;
    } else {
      if (check) err = fabs(val - jb.c[o]);
      if (!isfinite(val)) atomicOr(w.status, ST_NONFINITE_G);
      jb.c[o] = val;
      if (jb.out == 1) {
        double* tr = (w.trace && trace_slot >= 0 && trace_slot < w.trace_cap)
                         ? w.trace + ((long long)trace_slot * 2 + sp) * NN : nullptr;
        if (tr) tr[o] = val;
        if (w.S == 1) {
          jb.c[NN + o] = val;
          if (tr) tr[NN + o] = val;
        }
      }
    }
  }
  if (check) {
    for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
    if (lane == 0) atomicMax(w.wrap_bits, (unsigned long long)__double_as_longlong(err));
  }
}

// the B-chain of spin sp that the push of step j factors
__device__ __forceinline__ const double* zchain(const WalkerDev& w, int mode, int j, int sp) {
  const int k = (mode == MODE_FWD) ? j : (w.nstack - 1 - j);
  const int nsl = min((k + 1) * w.pace, w.Lt) - k * w.pace;
  return w.chain + (long long)((w.cb ? 0 : (nsl & 1)) * w.S + sp) * w.N * w.N;
}

// --------------------------------------------------------------------------
// Push preparation with tensor-core products: column norms of the chain, order by decreasing norm
// (ties by index), X = chain(:, perm).  One CTA per (walker, spin).
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(256) zpush_prep_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (w.ozstab != 1 || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const double* Cin = zchain(w, mode, j, sp);
  const ZScr z = zscr(w, sp);
  extern __shared__ long long zkey[];  // [N] norm bit patterns
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c = wid; c < N; c += 8) {
    double s = 0.0;
    for (int r = lane; r < N; r += 32) {
      const double a = Cin[(long long)c * N + r];
      s = fma(a, a, s);
    }
    s = zwarp_sum(s);
    if (lane == 0) zkey[c] = __double_as_longlong(sqrt(s));  // >= 0 (or NaN): bit order = value order
  }
  for (int k = threadIdx.x; k < N; k += 256) z.perm[k] = k;
  __syncthreads();
  for (int c = threadIdx.x; c < N; c += 256) {
    const long long kc = zkey[c];
    int rank = 0;
    for (int c2 = 0; c2 < N; ++c2) {
      const long long k2 = zkey[c2];
      rank += (k2 > kc || (k2 == kc && c2 < c)) ? 1 : 0;
    }
    z.perm[rank] = c;
  }
  __syncthreads();
  for (int k = wid; k < N; k += 8) {
    const int c = z.perm[k];
    for (int r = lane; r < N; r += 32) z.X[(long long)k * N + r] = Cin[(long long)c * N + r];
  }
}

// --------------------------------------------------------------------------
// Householder panel p of X (rows j0:N, columns j0:j0+pb) in shared memory:
// reflectors into X below the diagonal, R on and above, tau on the diagonal of the panel's T
// slot; for the push also D = |diag R| into the stack level and 1/D.
//
// Column c takes one barrier.  Warps 1-7 apply its reflector to columns c + 2 ..., at most five
// each: the dot products of a warp's columns share their loads and their shuffle steps (zsum4,
// zsum8).  Meanwhile warp 0 applies it to column c + 1 and forms that column's reflector (norm, a
// square root, the two quotients on two lanes, the scaling).  Every sum keeps the order of one
// column at a time (a norm over 256 threads, dot products over a warp): the 49-bit products of a
// stabilization interval amplify a change of rounding here to 1e-6 of the s-wave sum at beta = 10.
// What bounds it: the FP64 rate of one SM (2 m pb^2 operations) for long panels, warp 0's chain
// for short ones.
// A pass of 6 walkers of 16 x 16 (with ztfac_kernel): 59.8 ms with four barriers a column and
// serial quotients, 55.6 with two barriers and reordered sums, the same with this form;
// 128 walkers 794, 771, and 3 ms (of 683) more than the reordered sums.
// --------------------------------------------------------------------------
// Sums of 4 (8) values over the warp, value k left in lanes 8 k .. 8 k + 7 (4 k .. 4 k + 3)
__device__ __forceinline__ double zsum4(double a0, double a1, double a2, double a3, int lane) {
  const bool h = lane & 16, q = lane & 8;
  double x = (h ? a2 : a0) + __shfl_xor_sync(0xffffffffu, h ? a0 : a2, 16);
  double y = (h ? a3 : a1) + __shfl_xor_sync(0xffffffffu, h ? a1 : a3, 16);
  double v = (q ? y : x) + __shfl_xor_sync(0xffffffffu, q ? x : y, 8);
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double zsum8(const double (&a)[8], int lane) {
  const bool h = lane & 16, q = lane & 8, e = lane & 4;
  double x[4], y[2];
#pragma unroll
  for (int k = 0; k < 4; ++k) x[k] = (h ? a[k + 4] : a[k]) + __shfl_xor_sync(0xffffffffu, h ? a[k] : a[k + 4], 16);
#pragma unroll
  for (int k = 0; k < 2; ++k) y[k] = (q ? x[k + 2] : x[k]) + __shfl_xor_sync(0xffffffffu, q ? x[k] : x[k + 2], 8);
  double v = (e ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, e ? y[0] : y[1], 4);
  for (int o = 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// kinds: the kinds of walkers (WalkerDev::ozstab, a bit each) that take part
__global__ void __launch_bounds__(256) zqr_panel_kernel(const WalkerDev* __restrict__ W, int mode, int j, int p,
                                                        int push, int kinds) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (!(w.ozstab & kinds) || sp >= w.S || j >= w.nstack) return;
  const int N = w.N, j0 = p * TB;
  if (j0 >= N) return;
  const int m = N - j0, pb = min(TB, m);
  const ZScr z = zscr(w, sp);
  extern __shared__ double P[];  // [TB][m], P[c * m + r]
  __shared__ double s_tau[TB];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int c = wid; c < pb; c += 8)
    for (int r = lane; r < m; r += 32) P[c * m + r] = z.X[(long long)(j0 + c) * N + j0 + r];
  __syncthreads();
  // warp 0: the reflector of column c (norm in 8 strided parts, added in their order)
  auto reflector = [&](int c) {
    double* x = P + c * m;
    double s[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = 0.0;
    for (int r0 = c + 1; r0 < m; r0 += 256) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int r = r0 + 32 * q + lane;
        if (r < m) s[q] = fma(x[r], x[r], s[q]);
      }
    }
    __syncwarp();
    const double v = zsum8(s, lane);
    const int nq = min(8, (m - c - 1 + 31) / 32);
    double n2 = __shfl_sync(0xffffffffu, v, 0);
    for (int q = 1; q < nq; ++q) n2 += __shfl_sync(0xffffffffu, v, 4 * q);
    const double alpha = x[c];
    const double nrm = sqrt(alpha * alpha + n2);
    const bool any = n2 != 0.0;
    const double beta = alpha >= 0 ? -nrm : nrm;
    // lane 0: tau = (beta - alpha) / beta, lane 1: scale = 1 / (alpha - beta)
    const double d = beta - alpha, quo = __ddiv_rn(lane == 1 ? 1.0 : d, lane == 1 ? -d : beta);
    const double tau = __shfl_sync(0xffffffffu, quo, 0), scal = __shfl_sync(0xffffffffu, quo, 1);
    if (lane == 0) {
      s_tau[c] = any ? tau : 0.0;
      x[c] = any ? beta : alpha;
    }
    if (any)
      for (int r = c + 1 + lane; r < m; r += 32) x[r] *= scal;
    __syncwarp();
  };
  if (wid == 0) reflector(0);
  __syncthreads();
  for (int c = 0; c + 1 < pb; ++c) {
    const double* x = P + c * m;
    const double tau = s_tau[c];
    if (wid == 0) {
      double* a = P + (c + 1) * m;
      if (tau != 0.0) {
        double d = 0.0;
        for (int r = c + 1 + lane; r < m; r += 32) d = fma(x[r], a[r], d);
        d = zwarp_sum(d) + a[c];
        const double wv = tau * d;
        __syncwarp();
        if (lane == 0) a[c] -= wv;
        for (int r = c + 1 + lane; r < m; r += 32) a[r] = fma(-wv, x[r], a[r]);
        __syncwarp();
      }
      reflector(c + 1);
    } else if (tau != 0.0) {
      // columns c + 2 + (wid - 1) + 7 k, at most 5; lane k forms column k's factor
      const int c0 = c + 1 + wid, nc = (c0 < pb) ? (pb - c0 + 6) / 7 : 0;
      if (nc > 0) {
        double acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.0;
        for (int r = c + 1 + lane; r < m; r += 32) {
          const double xr = x[r];
#pragma unroll
          for (int k = 0; k < 5; ++k)
            if (k < nc) acc[k] = fma(xr, P[(c0 + 7 * k) * m + r], acc[k]);
        }
        __syncwarp();
        const bool four = nc <= 4;
        const double v = four ? zsum4(acc[0], acc[1], acc[2], acc[3], lane) : zsum8(acc, lane);
        double d = __shfl_sync(0xffffffffu, v, (four ? 8 : 4) * lane & 31), wv = 0.0;
        if (lane < nc) {
          double* a = P + (c0 + 7 * lane) * m;
          d += a[c];
          wv = tau * d;
          a[c] -= wv;
        }
        double f[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) f[k] = -__shfl_sync(0xffffffffu, wv, k);
        for (int r = c + 1 + lane; r < m; r += 32) {
          const double xr = x[r];
          double y[5];
#pragma unroll
          for (int k = 0; k < 5; ++k) y[k] = (k < nc) ? P[(c0 + 7 * k) * m + r] : 0.0;
#pragma unroll
          for (int k = 0; k < 5; ++k)
            if (k < nc) P[(c0 + 7 * k) * m + r] = fma(f[k], xr, y[k]);
        }
      }
    }
    __syncthreads();
  }
  for (int c = wid; c < pb; c += 8)
    for (int r = lane; r < m; r += 32) z.X[(long long)(j0 + c) * N + j0 + r] = P[c * m + r];
  // the Gram matrix V^T V, the T factor and Vt = V T follow as products (Z_GRAM,
  // ztfac_kernel, Z_VT); the panel leaves tau on the diagonal of its T slot
  double* Tg = z.Tb + (long long)p * TB * TB;
  for (int e = tid; e < TB * TB; e += 256) {
    const int r = e % TB, c = e / TB;
    Tg[e] = (r == c && c < pb) ? s_tau[c] : 0.0;
  }
  if (push && tid < pb) {
    const int side = (mode == MODE_FWD) ? 0 : 1;
    double* Do = stack_level(w, side, sp, j) + 2 * (long long)N * N;
    const double d = fabs(P[tid * m + tid]);
    Do[j0 + tid] = d;
    z.invd[j0 + tid] = (d != 0.0) ? 1.0 / d : 0.0;
    if (d == 0.0 || !isfinite(d)) atomicOr(w.status, ST_SINGULAR);
  }
}

// --------------------------------------------------------------------------
// The push's factorization with FP64 products (ozstab 2): column-pivoted Householder QR of the
// chain (LAPACK dlaqp2: partial norms downdated, and summed again once half of their digits are
// gone).  An order fixed beforehand costs a graded chain its accuracy: at U = 6, beta = 6, pace 10
// the assembled G of a 12 x 12 walker was 4e-10 off its long-double value with columns ordered once
// by norm (10 x 10: 1.5e-11), 1.9e-12 (1.3e-12) with a pivot per column.
//
// A cluster of P CTAs per (walker, spin), a warp per column (column c: CTA c mod P, warp c / P mod
// QW, its partial norm in lane c / (P QW)).  Columns stay where they are, in shared memory (SM) or
// in Y, and column k of the result goes to X once it is chosen.  A step has two cluster barriers:
// the warp of the chosen column writes the reflector to every CTA's shared memory; then each warp
// takes the dot products of its columns, four at a time, and with row k their partial norms, sends
// its largest one to all CTAs and updates rows k + 1 .. while that travels.  A column's sums are
// one warp's whatever P is, so results do not depend on it.
// What bounds it: the chain of a step (norm, square root, division, two barriers, two reductions:
// 10 us at N = 256), then FP64 issue.  A push of 16 walkers of 16 x 16 2.4 ms (panels and products
// without pivoting: 1.9); a pass of them 30.1 ms (29.2; 91 with a thread per column), of 32 walkers
// of 9 x 9 22.2 (21.9; 26).  Columns in L2 instead of shared memory 32.6 and 22.9, 16 warps a CTA
// 30.0 and 22.3 (9 x 9 at P = 4: 23.2).
// --------------------------------------------------------------------------
template <int P, bool SM>
__global__ void __launch_bounds__(32 * QW) __cluster_dims__(P, 1, 1)
    zqrp_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  namespace cg = cooperative_groups;
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1, rank = blockIdx.x;
  const WalkerDev& w = W[wi];
  // the whole cluster leaves or stays
  if (w.ozstab != 2 || sp >= w.S || j >= w.nstack) return;
  cg::cluster_group cl = cg::this_cluster();
  auto barrier = [&]() {
    if (P > 1) cl.sync();
    else __syncthreads();
  };
  const int N = w.N, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double* Cin = zchain(w, mode, j, sp);
  const ZScr z = zscr(w, sp);
  double* Do = stack_level(w, (mode == MODE_FWD) ? 0 : 1, sp, j) + 2 * (long long)N * N;
  extern __shared__ double vsh[];  // [2][N] the reflectors of steps k even and odd, then the CTA's columns
  auto column = [&](int q) {       // of this warp
    return SM ? vsh + (long long)(2 + wid + QW * q) * N : z.Y + (long long)(rank + P * (wid + QW * q)) * N;
  };
  __shared__ long long s_key[QW * P];
  __shared__ int s_col[QW * P];
  __shared__ double s_tau;
  // lane q: column rank + P (wid + 8 q), its squared partial norm and the last one summed in full
  const int mycol = rank + P * (wid + QW * lane);
  bool active = mycol < N;
  double n1 = 0.0, n2 = 0.0;
  for (int q = 0, c = rank + P * wid; c < N; ++q, c += QW * P) {
    double s = 0.0, *a = column(q);
    for (int r = lane; r < N; r += 32) {
      const double x = Cin[(long long)c * N + r];
      a[r] = x;
      s = fma(x, x, s);
    }
    s = zwarp_sum(s);
    if (lane == q) n1 = n2 = s;
  }
  __syncwarp();
  // (key, col) of the largest key in the warp, ties to the lowest column; key < 0: none
  auto warp_best = [&](long long& key, int& col) {
    const int hi = (int)(key >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = (hi == mh) ? (unsigned)key : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
    col = __reduce_min_sync(0xffffffffu, (hi == mh && (unsigned)key == ml) ? col : 0x7fffffff);
    key = ((long long)mh << 32) | ml;
  };
  auto send = [&](long long key, int col) {  // the warp's candidate, to every CTA
    warp_best(key, col);
    if (lane < P) {
      *((P > 1) ? cl.map_shared_rank(&s_key[rank * QW + wid], lane) : &s_key[wid]) = key;
      *((P > 1) ? cl.map_shared_rank(&s_col[rank * QW + wid], lane) : &s_col[wid]) = col;
    }
  };
  auto norm_key = [&]() { return active ? (__double_as_longlong(n1) & 0x7fffffffffffffffLL) : -1LL; };
  if (P > 1) cl.sync();  // every CTA runs before its shared memory is written
  send(norm_key(), mycol);
  barrier();
  for (int k = 0; k < N; ++k) {
    double* v = vsh + (k & 1) * N;  // rows k + 1 ..; a slow warp may still read the previous one
    long long key = -1;
    int pc = 0x7fffffff;
#pragma unroll
    for (int q = 0; q < (QW * P + 31) / 32; ++q) {
      const int e = lane + 32 * q;
      if (e < QW * P && (s_key[e] > key || (s_key[e] == key && s_col[e] < pc))) { key = s_key[e]; pc = s_col[e]; }
    }
    warp_best(key, pc);
    const bool owner = pc % P == rank && pc / P % QW == wid;
    double beta = 0.0, quo = 0.0;
    if (owner) {
      // its reflector: rows k + 1 .. scaled, to every CTA
      const double* a = column(pc / P / QW);
      double s0 = 0.0, s1 = 0.0;
      int r = k + 1 + lane;
      for (; r + 32 < N; r += 64) {
        s0 = fma(a[r], a[r], s0);
        s1 = fma(a[r + 32], a[r + 32], s1);
      }
      if (r < N) s0 = fma(a[r], a[r], s0);
      const double xn2 = zwarp_sum(s0 + s1), alpha = a[k];
      const bool any = xn2 != 0.0;
      const double nrm = sqrt(alpha * alpha + xn2);
      beta = any ? (alpha >= 0 ? -nrm : nrm) : alpha;
      // lane 0: tau = (beta - alpha) / beta, lane 1: scale = 1 / (alpha - beta), lane 2: 1 / |beta|
      const double d = beta - alpha;
      quo = __ddiv_rn(lane == 0 ? d : 1.0, lane == 0 ? beta : lane == 1 ? -d : fabs(beta));
      const double tau = any ? __shfl_sync(0xffffffffu, quo, 0) : 0.0;
      const double scal = any ? __shfl_sync(0xffffffffu, quo, 1) : 1.0;
      for (r = k + 1 + lane; r < N; r += 32) {
        const double y = a[r] * scal;
#pragma unroll
        for (int p = 0; p < P; ++p) *((P > 1) ? cl.map_shared_rank(&v[r], p) : &v[r]) = y;
      }
      if (lane < P) *((P > 1) ? cl.map_shared_rank(&s_tau, lane) : &s_tau) = tau;
      if (mycol == pc) active = false;
    }
    barrier();
    const double tau = s_tau;
    // column k of R and V to X, with what else the step settles (its stores are not waited for at a barrier)
    auto settle = [&]() {
      const double* a = column(pc / P / QW);
      double* x = z.X + (long long)k * N;
      for (int r = lane; r < k; r += 32) x[r] = a[r];
      for (int r = k + 1 + lane; r < N; r += 32) x[r] = v[r];
      const double inv = __shfl_sync(0xffffffffu, quo, 2), ab = fabs(beta);
      if (lane == 0) {
        x[k] = beta;
        z.perm[k] = pc;
        z.Tb[(long long)(k / TB) * TB * TB + (k % TB) * (TB + 1)] = tau;  // the diagonal of its T factor
        Do[k] = ab;
        z.invd[k] = (ab != 0.0) ? inv : 0.0;
        if (ab == 0.0 || !isfinite(ab)) atomicOr(w.status, ST_SINGULAR);
      }
    };
    if (k + 1 == N) {
      if (owner) settle();
      break;
    }
    // A(k:, c) -= tau v (v^T A(k:, c)), v = [1; v]: row k and with it the partial norms first, so that
    // the next candidates travel while rows k + 1 .. are updated
    const unsigned mine = __ballot_sync(0xffffffffu, active);
    double fc = 0.0;  // lane q: -tau (v^T A(k:, c)) of its column
    bool again = false;
    for (unsigned todo = mine; todo;) {
      int q[4], n = 0;
      double* a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        q[u] = todo ? __ffs(todo) - 1 : q[0];
        if (todo) ++n;
        todo &= todo - 1;
        a[u] = column(q[u]);
      }
      double d[4] = {0.0, 0.0, 0.0, 0.0};
      for (int r = k + 1 + lane; r < N; r += 32) {
        const double vr = v[r];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < n) d[u] = fma(vr, a[u][r], d[u]);
      }
      // lanes 8 u .. 8 u + 7: column u
      const double dot = zsum4(d[0], d[1], d[2], d[3], lane);
      const int g = lane >> 3;
      double* ag = (g & 2) ? ((g & 1) ? a[3] : a[2]) : ((g & 1) ? a[1] : a[0]);
      const double top = ag[k], f = tau * (dot + top), rk = top - f;
      __syncwarp();
      if ((lane & 7) == 0 && g < n) ag[k] = rk;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double fu = -__shfl_sync(0xffffffffu, f, 8 * u), ru = __shfl_sync(0xffffffffu, rk, 8 * u);
        if (u < n && lane == q[u]) {
          fc = fu;
          n1 = fma(-ru, ru, n1);
          again = n1 <= 1.4901161193847656e-08 * n2;
        }
      }
    }
    auto update = [&]() {
      for (unsigned todo = mine; todo;) {
        int n = 0;
        double* a[4];
        double f[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int q = todo ? __ffs(todo) - 1 : 0;
          if (todo) ++n;
          todo &= todo - 1;
          a[u] = column(q);
          f[u] = __shfl_sync(0xffffffffu, fc, q);
        }
        int r = k + 1 + lane;
        for (; r + 32 < N; r += 64) {  // two rows' loads before their stores
          const double v0 = v[r], v1 = v[r + 32];
          double y[4], x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (u < n) { y[u] = a[u][r]; x[u] = a[u][r + 32]; }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (u < n) { a[u][r] = fma(f[u], v0, y[u]); a[u][r + 32] = fma(f[u], v1, x[u]); }
        }
        if (r < N) {
          const double v0 = v[r];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (u < n) a[u][r] = fma(f[u], v0, a[u][r]);
        }
      }
      __syncwarp();
    };
    const unsigned full = __ballot_sync(0xffffffffu, again);
    if (full) update();
    for (unsigned m = full; m; m &= m - 1) {
      const int q = __ffs(m) - 1;
      const double* a = column(q);
      double s = 0.0;
      for (int r = k + 1 + lane; r < N; r += 32) s = fma(a[r], a[r], s);
      s = zwarp_sum(s);
      if (lane == q) n1 = n2 = s;
    }
    send(norm_key(), mycol);
    if (P > 1) {
      cg::cluster_group::arrival_token t = cl.barrier_arrive();
      if (!full) update();
      if (owner) settle();
      cl.barrier_wait(std::move(t));
    } else {
      if (!full) update();
      if (owner) settle();
      __syncthreads();
    }
  }
}

// The T factor of a panel (LAPACK dlarft, forward, columnwise) from Zg = V^T V (Zg[k][c], k < c) and tau:
// T(c, c) = tau_c, T(i, c) = -tau_c sum_{i <= k < c} T(i, k) Zg(k, c).
// Row i needs no other row: a warp takes rows i = warp mod 8, lane c holds the sum of column c, and
// step k broadcasts T(i, k).  No barriers, four rows a warp in flight; the sums run in dlarft's order.
__device__ __forceinline__ void zt_rows(const double (&Zg)[TB][TB + 1], const double* s_tau, int pb, double* Tg) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double tau = s_tau[lane];
  double acc[4] = {0.0, 0.0, 0.0, 0.0};  // rows wid + 8 u
  for (int k = wid; k + 1 < pb; ++k) {
    const double zk = Zg[k][lane];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = wid + 8 * u;
      if (i > k) continue;  // uniform in the warp
      const double t = __shfl_sync(0xffffffffu, (i == k) ? tau : -tau * acc[u], k);
      if (lane > k) acc[u] = fma(t, zk, acc[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = wid + 8 * u;
    Tg[lane * TB + i] = (i < pb && lane < pb && lane >= i) ? (lane == i ? tau : -tau * acc[u]) : 0.0;
  }
}

// The T factor of panel p, its Gram matrix from the Z_GRAM product (in Wb), tau on the diagonal of its slot
__global__ void __launch_bounds__(256) ztfac_kernel(const WalkerDev* __restrict__ W, int mode, int j, int p, int kinds) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (!(w.ozstab & kinds) || sp >= w.S || j >= w.nstack) return;
  const int N = w.N, j0 = p * TB;
  if (j0 >= N) return;
  const int pb = min(TB, N - j0), tid = threadIdx.x;
  const ZScr z = zscr(w, sp);
  __shared__ double Zg[TB][TB + 1];
  __shared__ double s_tau[TB];
  double* Tg = z.Tb + (long long)p * TB * TB;
  for (int e = tid; e < TB * TB; e += 256) {
    const int k = e % TB, c = e / TB;
    Zg[k][c] = (k < c && c < pb) ? z.Wb[(long long)c * TB + k] : 0.0;
    if (k == c) s_tau[c] = (c < pb) ? Tg[e] : 0.0;
  }
  __syncthreads();
  zt_rows(Zg, s_tau, pb, Tg);
}

// The T factors of zqrp_kernel's panels, all in one launch (a CTA per walker, spin and panel): with the
// factorization behind them the panels do not wait for one another.  The Gram matrix of the
// reflectors is summed here, 32 rows at a time, four sums of a column c a thread (k = warp + 8 u).
__global__ void __launch_bounds__(256) zqrp_tfac_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1, p = blockIdx.x;
  const WalkerDev& w = W[wi];
  if (w.ozstab != 2 || sp >= w.S || j >= w.nstack) return;
  const int N = w.N, j0 = p * TB;
  if (j0 >= N) return;
  const int m = N - j0, pb = min(TB, m), tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const ZScr z = zscr(w, sp);
  __shared__ double Zg[TB][TB + 1], V[TB][TB + 1];  // V[c][r]
  __shared__ double s_tau[TB];
  double* Tg = z.Tb + (long long)p * TB * TB;
  if (tid < TB) s_tau[tid] = (tid < pb) ? Tg[tid * (TB + 1)] : 0.0;
  double g[4] = {0.0, 0.0, 0.0, 0.0};
  for (int r0 = 0; r0 < m; r0 += TB) {
    __syncthreads();
    for (int c = wid; c < TB; c += 8) {
      const int r = r0 + lane;
      V[c][lane] = (c >= pb || r >= m || r < c) ? 0.0 : (r == c) ? 1.0 : z.X[(long long)(j0 + c) * N + j0 + r];
    }
    __syncthreads();
#pragma unroll 8
    for (int r = 0; r < TB; ++r) {
      const double vc = V[lane][r];
#pragma unroll
      for (int u = 0; u < 4; ++u) g[u] = fma(V[wid + 8 * u][r], vc, g[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) Zg[wid + 8 * u][lane] = (wid + 8 * u < lane) ? g[u] : 0.0;
  __syncthreads();
  zt_rows(Zg, s_tau, pb, Tg);
}

// Vt = V_p T_p^T (m x pb, ld N) for forming Q: Vt(r, c) = sum_{c <= q <= r} V(r, q) T(c, q).
// 32 rows per CTA, V and T staged in shared memory.
__global__ void __launch_bounds__(256) zvt_kernel(const WalkerDev* __restrict__ W, int mode, int j, int p) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.ozstab || sp >= w.S || j >= w.nstack) return;
  const int N = w.N, j0 = p * TB;
  if (j0 >= N) return;
  const int m = N - j0, pb = min(TB, m), r0 = blockIdx.x * 32;
  if (r0 >= m) return;
  const ZScr z = zscr(w, sp);
  __shared__ double sV[TB][33], sT[TB][33];  // sV[q][rl] = V(r0 + rl, q), sT[q][c] = T(c, q)
  const double* Tg = z.Tb + (long long)p * TB * TB;
  for (int e = threadIdx.x; e < TB * TB; e += 256) {
    const int rl = e & 31, q = e >> 5, r = r0 + rl;
    double v = 0.0;
    if (q < pb && r < m) v = (r > q) ? z.X[(long long)(j0 + q) * N + j0 + r] : (r == q ? 1.0 : 0.0);
    sV[q][rl] = v;
    sT[q][rl] = (q < pb && rl < pb) ? Tg[q * TB + rl] : 0.0;  // T(rl, q), zero below the diagonal
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * pb; e += 256) {
    const int rl = e & 31, c = e >> 5, r = r0 + rl;
    if (r >= m) continue;
    double s = 0.0;
    for (int q = c; q < pb; ++q) s = fma(sV[q][rl], sT[q][c], s);
    z.W2[(long long)c * N + r] = s;
  }
}

// U = I before forming Q; at the first level F = D^-1 R P^T directly
__global__ void __launch_bounds__(256) zpush_fin_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.ozstab || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  const int side = (mode == MODE_FWD) ? 0 : 1;
  double* Uo = stack_level(w, side, sp, j);
  double* Fo = Uo + NN;
  const ZScr z = zscr(w, sp);
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < NN; e += (long long)gridDim.x * 256) {
    const int r = (int)(e % N), c = (int)(e / N);
    Uo[e] = (r == c) ? 1.0 : 0.0;
    if (j == 0) Fo[(long long)z.perm[c] * N + r] = (r <= c) ? z.X[e] * z.invd[r] : 0.0;
  }
}

// --------------------------------------------------------------------------
// Green's preparation: scale vectors; Y = Dmax^-1 U^T (col-major); boundary
// steps also M = Y + Dmin F.  Grid over the N^2 elements.
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(256) zgreens_prep_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.ozstab || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  int nl, nr;
  zstack_tops(w, mode, j, nl, nr);
  const ZScr z = zscr(w, sp);
  const bool both = nl > 0 && nr > 0;
  const double* lv = (nl > 0) ? stack_level(w, 0, sp, nl - 1) : stack_level(w, 1, sp, nr - 1);
  const double* U = lv;
  const double* F = lv + NN;
  const double* D = lv + 2 * NN;
  if (blockIdx.x == 0 && both) {
    const double* DR = stack_level(w, 1, sp, nr - 1) + 2 * NN;
    for (int k = threadIdx.x; k < N; k += 256) {
      z.dlmaxi[k] = 1.0 / fmax(D[k], 1.0);
      z.dlmin[k] = fmin(D[k], 1.0);
      z.drmaxi[k] = 1.0 / fmax(DR[k], 1.0);
      z.drmin[k] = fmin(DR[k], 1.0);
    }
  }
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < NN; e += (long long)gridDim.x * 256) {
    const int r = (int)(e % N), c = (int)(e / N);
    const double dr = D[r];
    const double y = U[(long long)r * N + c] / fmax(dr, 1.0);  // (Dmax^-1 U^T)(r, c)
    z.Y[e] = y;
    if (!both) z.X[e] = y + fmin(dr, 1.0) * F[e];
  }
}

// back substitution of the diagonal block p: R_pp X(j0:j0+pb, c) = Y(j0:j0+pb, c), thread per
// column; rhs (blockIdx.z) 0: Y, 1: the dynamic half-sweep's second right-hand side (dynx)
__global__ void __launch_bounds__(128) ztrsm_diag_kernel(const WalkerDev* __restrict__ W, int mode, int j, int p) {
  const int rhs = blockIdx.z;
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.ozstab || sp >= w.S || j >= w.nstack) return;
  if (rhs && !w.dynx) return;
  const int N = w.N, j0 = p * TB;
  if (j0 >= N) return;
  const int pb = min(TB, N - j0);
  const ZScr z = zscr(w, sp);
  __shared__ double R[TB][TB + 1];
  __shared__ double rinv[TB];
  for (int e = threadIdx.x; e < TB * TB; e += 128) {
    const int i = e % TB, k = e / TB;
    R[i][k] = (i < pb && k < pb && i <= k) ? z.X[(long long)(j0 + k) * N + j0 + i] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < TB) {  // rows past a partial panel: 0 (their x stays 0)
    const double d = R[threadIdx.x][threadIdx.x];
    rinv[threadIdx.x] = (d != 0.0) ? 1.0 / d : 0.0;
    if (d == 0.0 && threadIdx.x < pb && blockIdx.x == 0) atomicOr(w.status, ST_SINGULAR);
  }
  __syncthreads();
  const int c = blockIdx.x * 128 + threadIdx.x;
  if (c >= N) return;
  double* y = (rhs ? w.dynx + (long long)sp * N * N : z.Y) + (long long)c * N + j0;
  double x[TB];
#pragma unroll
  for (int i = 0; i < TB; ++i) x[i] = (i < pb) ? y[i] : 0.0;
#pragma unroll
  for (int i = TB - 1; i >= 0; --i) {
    double s = x[i];
#pragma unroll
    for (int k = i + 1; k < TB; ++k) s = fma(-R[i][k], x[k], s);
    x[i] = s * rinv[i];
  }
#pragma unroll
  for (int i = 0; i < TB; ++i)
    if (i < pb) y[i] = x[i];
}

// boundary steps: G = X (left stack present) or X^T (right only), wrap error, trace
__global__ void __launch_bounds__(256) zgreens_out_kernel(const WalkerDev* __restrict__ W, int mode, int j,
                                                          int trace_slot) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.ozstab || sp >= w.S || j >= w.nstack) return;
  int nl, nr;
  zstack_tops(w, mode, j, nl, nr);
  if (nl > 0 && nr > 0) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  const ZScr z = zscr(w, sp);
  double* G = w.G + sp * NN;
  double* tr = (w.trace && trace_slot >= 0 && trace_slot < w.trace_cap) ? w.trace + ((long long)trace_slot * 2 + sp) * NN
                                                                       : nullptr;
  const bool transpose_out = (nl == 0);
  const bool check = !(mode == MODE_INIT || (mode == MODE_BWD && j == w.nstack - 1));
  double err = 0.0;
  bool finite = true;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < NN; e += (long long)gridDim.x * 256) {
    const int r = (int)(e % N), c = (int)(e / N);
    const double v = transpose_out ? z.Y[(long long)r * N + c] : z.Y[e];
    if (check) err = fmax(err, fabs(v - G[e]));
    if (!isfinite(v)) finite = false;
    G[e] = v;
    if (tr) tr[e] = v;
    if (w.S == 1) {
      G[NN + e] = v;
      if (tr) tr[NN + e] = v;
    }
  }
  if (!finite) atomicOr(w.status, ST_NONFINITE_G);
  if (check) {
    for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
    if ((threadIdx.x & 31) == 0) atomicMax(w.wrap_bits, (unsigned long long)__double_as_longlong(err));
  }
}

// dynamic half-sweep, forward step j: the second right-hand side Y2 = min(D_L, 1) F_L of the
// left stack's top level, column-major into dynx
__global__ void __launch_bounds__(256) zdyn_prep_kernel(const WalkerDev* __restrict__ W, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.ozstab || !w.dynx || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  const double* lv = stack_level(w, 0, sp, j);  // forward step j: left stack of j + 1 levels
  const double* F = lv + NN;
  const double* D = lv + 2 * NN;
  double* Y2 = w.dynx + sp * NN;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < NN; e += (long long)gridDim.x * 256) {
    const int r = (int)(e % N);
    Y2[e] = fmin(D[r], 1.0) * F[e];
  }
}

// dynamic half-sweep at t = beta (right stack empty): G(beta,0) = X2, G(0,beta) = -X, with
// their wrap errors against the propagated values
__global__ void __launch_bounds__(256) zdyn_boundary_kernel(const WalkerDev* __restrict__ W, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.ozstab || !w.gt0 || !w.dynx || sp >= w.S || j != w.nstack - 1) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  const ZScr z = zscr(w, sp);
  double* t0 = zdyn_slot(w.gt0, w, sp, w.Lt);
  double* ot = zdyn_slot(w.g0t, w, sp, w.Lt);
  const double* X2 = w.dynx + sp * NN;
  double err = 0.0;
  bool finite = true;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < NN; e += (long long)gridDim.x * 256) {
    const double a = X2[e], b = -z.Y[e];
    err = fmax(err, fmax(fabs(a - t0[e]), fabs(b - ot[e])));
    if (!isfinite(a) || !isfinite(b)) finite = false;
    t0[e] = a;
    ot[e] = b;
  }
  if (!finite) atomicOr(w.status, ST_NONFINITE_G);
  for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
  if ((threadIdx.x & 31) == 0) atomicMax(w.wrap_bits, (unsigned long long)__double_as_longlong(err));
}

// --------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------
// the two product configurations: 56 bits (K <= 256) and 54 bits (K <= 1024)
#define ZGEMM56 zgemm_tc_kernel<8, 7, 32, 2, 2>
#define ZGEMM54 zgemm_tc_kernel<9, 6, 32, 4, 1>
static size_t ztc_smem(int S, int NT, int NS) { return (size_t)NS * oztc::stage_bytes(S, 128, NT); }
static size_t zpanel_smem(int maxN) { return sizeof(double) * (size_t)TB * maxN; }

// dynamic shared memory: two reflectors, and the columns of a CTA where they fit
static size_t zqrp_smem(int N, int P, bool sm) {
  return sizeof(double) * (size_t)N * (2 + (sm ? ((N + P - 1) / P + QW - 1) / QW * QW : 0));
}
constexpr size_t kQrpSmem = 224 * 1024;

cudaError_t configure_stab_oz_kernels(int maxN) {
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(ZGEMM56, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ztc_smem(8, 32, 2))))
    return e;
  if ((e = cudaFuncSetAttribute(ZGEMM54, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ztc_smem(9, 32, 4))))
    return e;
  if ((e = cudaFuncSetAttribute(zqr_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)zpanel_smem(maxN > 0 ? maxN : 1))))
    return e;
  const void* qrp[4] = {(const void*)zqrp_kernel<1, true>, (const void*)zqrp_kernel<2, true>,
                        (const void*)zqrp_kernel<4, true>, (const void*)zqrp_kernel<8, true>};
  for (const void* f : qrp)
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQrpSmem))) return e;
  return cudaSuccess;
}

// doubles of scratch a spin's stabilization takes in zwk
size_t stab_scratch_elems(int N) {
  return 2ull * TB * N + (size_t)TB * TB * ((N + TB - 1) / TB) + 5ull * N + (5ull * N + 1) / 2;
}

// The largest output of an operation over walkers of up to n sites: rows, and columns of part 0
// and of each further part (zjob).  The trailing matrix shrinks with the panels: in grids for the
// whole matrix more than half of the factorization's CTAs had no work (N = 256), and each waited
// for 80 KB of shared memory to start.  Grids of the extent: 128 walkers of 16 x 16 690 -> 680 ms
// a sweep pair, 32 walkers of 9 x 9 in FP64 22.2 -> 21.8, set-up of 48 of 12 x 12 17.9 -> 17.5.
struct ZExtent {
  int rows, cols0, cols;
};
static ZExtent zextent(int op, int p, int n) {
  const int m = std::max(n - p * TB, 0), pb = std::min(TB, m);
  switch (op) {
    case Z_QR_W: return {pb, m - pb, n};
    case Z_QR_UPD: return {m, m - pb, n};
    case Z_Q_W: return {pb, m, m};
    case Z_Q_UPD: return {m, m, m};
    case Z_TR_UPD: return {m > TB ? pb : 0, n, n};
    case Z_GRAM: return {pb, pb, pb};
    case Z_VT: return {m, pb, pb};
    default: return {n, n, n};
  }
}

// The parts p0 .. p0 + parts - 1 of a product; slice_a: A too (else its slices are still there)
static void zgemm_tc(const WalkerDev* W, int nw, StabSizes zs, int op, int mode, int j, int p, int trace_slot, int p0,
                     int parts, bool slice_a, cudaStream_t st) {
  // the walkers' contraction lengths, minN to maxN: a panel's width, what is left from panel p
  // on, or N; each configuration is launched only where some walker's length takes it (at
  // N = 576 half of the launches had no work)
  const bool width = op == Z_QR_UPD || op == Z_Q_UPD || op == Z_VT;
  const bool rest = op == Z_QR_W || op == Z_Q_W || op == Z_GRAM || op == Z_TR_UPD;
  const int off = rest ? p * TB + (op == Z_TR_UPD ? TB : 0) : 0;
  const int minN = width ? TB : zs.tc_min - off, maxN = width ? TB : zs.tc - off;
  const ZExtent x = zextent(op, p, zs.tc);
  const int cols = p0 ? x.cols : x.cols0;  // of part p0
  const ZTiles tl{(cols + 31) / 32, (x.cols + 31) / 32, p0};
  const dim3 g(tl.first + (parts - 1) * tl.rest, (x.rows + 127) / 128, 2 * nw);
  const dim3 gs((std::max(x.rows, parts > 1 ? x.cols : cols) + 31) / 32, parts + (slice_a ? 1 : 0), 2 * nw);
  const int y0 = slice_a ? 0 : 1 + p0;
  if (!g.x || !g.y) return;
  if (minN <= 256) zslice_kernel<8, 7><<<gs, 256, 0, st>>>(W, op, mode, j, p, y0);
  if (maxN > 256) zslice_kernel<9, 6><<<gs, 256, 0, st>>>(W, op, mode, j, p, y0);
  if (minN <= 256) ZGEMM56<<<g, 256, ztc_smem(8, 32, 2), st>>>(W, op, mode, j, p, trace_slot, tl);
  if (maxN > 256) ZGEMM54<<<g, 256, ztc_smem(9, 32, 4), st>>>(W, op, mode, j, p, trace_slot, tl);
}

static void zgemm(const WalkerDev* W, int nw, StabSizes zs, int op, int mode, int j, int p, int trace_slot,
                  cudaStream_t st, int parts = 1) {
  if (zs.f64) {
    const ZExtent x = zextent(op, p, zs.f64);
    const ZTiles tl{(x.cols0 + 15) / 16, (x.cols + 15) / 16, 0};
    const dim3 g(tl.first + (parts - 1) * tl.rest, (x.rows + 15) / 16, 2 * nw);
    if (g.x && g.y) zgemm_f64_kernel<<<g, 256, 0, st>>>(W, op, mode, j, p, trace_slot, tl);
  }
  if (!zs.tc) return;
  const bool apart = op == Z_QR_W && parts == 3;  // part 2 after part 1, in its lines (zimage)
  zgemm_tc(W, nw, zs, op, mode, j, p, trace_slot, 0, apart ? 2 : parts, true, st);
  if (apart) zgemm_tc(W, nw, zs, op, mode, j, p, trace_slot, 2, 1, false, st);
}

static int zkinds(StabSizes zs) { return (zs.tc ? 1 : 0) | (zs.f64 ? 2 : 0); }

// Householder panel p: the FP64 column factorization, then its Gram matrix, T factor and
// Vt = V T (the block reflector in the form the trailing products apply)
static void zpanel(const WalkerDev* W, int nw, StabSizes zs, int mode, int j, int p, int push, cudaStream_t st) {
  zqr_panel_kernel<<<2 * nw, 256, zpanel_smem(zs.max()), st>>>(W, mode, j, p, push, zkinds(zs));
  zgemm(W, nw, zs, Z_GRAM, mode, j, p, -1, st);
  ztfac_kernel<<<2 * nw, 256, 0, st>>>(W, mode, j, p, zkinds(zs));
  zgemm(W, nw, zs, Z_VT, mode, j, p, -1, st);
}

template <int P>
static void launch_qrp_p(const WalkerDev* W, int nw, int N, int mode, int j, cudaStream_t st) {
  const dim3 g(P, 2 * nw);
  const size_t sm = zqrp_smem(N, P, true);
  if (sm <= kQrpSmem) zqrp_kernel<P, true><<<g, 32 * QW, sm, st>>>(W, mode, j);
  else zqrp_kernel<P, false><<<g, 32 * QW, zqrp_smem(N, P, false), st>>>(W, mode, j);
}

// CTAs per matrix: as many as shared memory needs for the columns (a lane per column and warp asks
// for N <= 256 P), then twice as many while every CTA of the batch's matrices still has an SM of its own.
// Measured at P = 1, 2, 4, 8: a pass of 16 walkers of 16 x 16 (one spin; 1 and 2 do not fit) 41.7,
// 36.2, 30.1, 30.3 ms; of 32 of 9 x 9 (two spins) 22.4, 22.1, 22.3, 23.0; of a mixed batch of 64
// walkers, 48 of them of 36 to 100 sites, 299, 300, 303, 310, its set-up 56, 54, 53, 56.
static void launch_qrp(const WalkerDev* W, int nw, StabSizes zs, int mode, int j, cudaStream_t st) {
  const int N = zs.f64;
  int P = 1, dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  while (P < 8 && (N > 32 * QW * P || zqrp_smem(N, P, true) > kQrpSmem || 2 * P * zs.f64_mats <= sms)) P *= 2;
  if (P == 8) launch_qrp_p<8>(W, nw, N, mode, j, st);
  else if (P == 4) launch_qrp_p<4>(W, nw, N, mode, j, st);
  else if (P == 2) launch_qrp_p<2>(W, nw, N, mode, j, st);
  else launch_qrp_p<1>(W, nw, N, mode, j, st);
}

// Walkers of both kinds in one launch range: the pivoted QR (few CTAs, a chain of N steps) runs on the
// side stream, beside the panels of the others.  One after the other, a pass of 44 walkers of sides 6,
// 8, 10 and 12, whose groups mix sides, took 294 ms instead of 278, and the set-up of 64 walkers, all in
// one range, 56 instead of 45.
void oz_push(int mode, const WalkerDev* W, int nw, int j, StabSizes zs, SideStream side, cudaStream_t st) {
  const int maxN = zs.max(), np = (maxN + TB - 1) / TB;
  const StabSizes tc{zs.tc, 0, zs.tc_min, 0};
  const bool beside = zs.tc && zs.f64 && side.st;
  if (zs.f64) {
    const cudaStream_t qs = beside ? side.st : st;
    if (beside) {
      cudaEventRecord(side.fork, st);
      cudaStreamWaitEvent(qs, side.fork, 0);
    }
    launch_qrp(W, nw, zs, mode, j, qs);
    zqrp_tfac_kernel<<<dim3((zs.f64 + TB - 1) / TB, 2 * nw), 256, 0, qs>>>(W, mode, j);
    if (beside) cudaEventRecord(side.join, qs);
  }
  if (zs.tc) zpush_prep_kernel<<<2 * nw, 256, sizeof(long long) * zs.tc, st>>>(W, mode, j);
  for (int p = 0; p * TB < zs.tc; ++p) {
    zpanel(W, nw, tc, mode, j, p, 1, st);
    zgemm(W, nw, tc, Z_QR_W, mode, j, p, -1, st);
    zgemm(W, nw, tc, Z_QR_UPD, mode, j, p, -1, st);
  }
  if (beside) cudaStreamWaitEvent(st, side.join, 0);
  zpush_fin_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, mode, j);
  zgemm(W, nw, zs, Z_F, mode, j, 0, -1, st);
  for (int p = np - 1; p >= 0; --p) {
    zvt_kernel<<<dim3((maxN + 31) / 32, 2 * nw), 256, 0, st>>>(W, mode, j, p);
    zgemm(W, nw, zs, Z_Q_W, mode, j, p, -1, st);
    zgemm(W, nw, zs, Z_Q_UPD, mode, j, p, -1, st);
  }
}

// The Green's assembly; with dyn (forward steps of the dynamic half-sweep) the same
// factorization of M also solves the second right-hand side and G(t,0), G(0,t) follow.
void oz_greens(int mode, const WalkerDev* W, int nw, int j, int trace_slot, StabSizes zs, cudaStream_t st, bool dyn) {
  const int maxN = zs.max(), np = (maxN + TB - 1) / TB;
  zgreens_prep_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, mode, j);
  if (dyn) zdyn_prep_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, j);
  zgemm(W, nw, zs, Z_GA, mode, j, 0, -1, st);
  zgemm(W, nw, zs, Z_GB, mode, j, 0, -1, st);
  // Q^T goes to the trailing columns and the right-hand sides in the same launches (8 walkers of
  // 24 x 24 with the dynamic half-sweep: 216 -> 206 ms a pass, 128 walkers of 16 x 16 767 -> 751)
  for (int p = 0; p < np; ++p) {
    zpanel(W, nw, zs, mode, j, p, 0, st);
    zgemm(W, nw, zs, Z_QR_W, mode, j, p, -1, st, dyn ? 3 : 2);
    zgemm(W, nw, zs, Z_QR_UPD, mode, j, p, -1, st, dyn ? 3 : 2);
  }
  for (int p = np - 1; p >= 0; --p) {
    zgemm(W, nw, zs, Z_TR_UPD, mode, j, p, -1, st, dyn ? 2 : 1);
    ztrsm_diag_kernel<<<dim3((maxN + 127) / 128, 2 * nw, dyn ? 2 : 1), 128, 0, st>>>(W, mode, j, p);
  }
  zgemm(W, nw, zs, Z_GG, mode, j, 0, trace_slot, st);
  zgreens_out_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, mode, j, trace_slot);
  if (dyn) {
    zgemm(W, nw, zs, Z_DT0_OUT, mode, j, 0, -1, st);
    zgemm(W, nw, zs, Z_D0T_OUT, mode, j, 0, -1, st);
    zdyn_boundary_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, j);
  }
}

}  // namespace dqmc
