// kernels_general.cu — FP64 plain-method kernels for walkers whose G does not
// fit in shared memory (N > 64, up to 1024).
//
// G, the B-chain and the stacks stay in HBM/L2; a half-sweep runs slice by
// slice as a short sequence of batched launches:
//   wrap (two products in the factors of exp(-dtau K), the diagonal
//   exp(+/-alpha s) fused) -> Metropolis (submatrix updates, kernels_submatrix.cu)
//   -> measurement -> B-chain step (one product).
// Stabilization: of walkers of 33 to 768 sites in kernels_stab_oz.cu; of the
// others, and of shared-memory walkers in the dynamic half-sweep, here:
// column-pivoted QR with one thread per column (row-major copy, coalesced across
// threads), Green's assembly by batched GEMMs and an LU solve with one thread
// per column of [M | Y].
//
// Reference behaviour is the same as kernels_fp64.cu (src/dqmc_walker.cpp,
// src/model/*.cpp, src/svd_stack.cpp, include/utils/numerical_stable.hpp,
// src/measure/measure_methods.cpp); only the data placement differs.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "dqmc_device.cuh"

namespace dqmc {

namespace {

__device__ __forceinline__ double warp_sum_g(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ bool is_general(const WalkerDev& w) { return w.path != 0; }

// Slice t handled at step j, in-segment index q (false when q is past the segment).
__device__ __forceinline__ bool slice_of(const WalkerDev& w, int mode, int j, int q, int& t, int& nsl, int& t_hi) {
  if (j >= w.nstack) return false;
  const int k = (mode == MODE_FWD) ? j : (w.nstack - 1 - j);
  const int t_lo = k * w.pace + 1;
  t_hi = min((k + 1) * w.pace, w.Lt);
  nsl = t_hi - t_lo + 1;
  if (q >= nsl) return false;
  t = (mode == MODE_FWD) ? t_lo + q : t_hi - q;
  return true;
}

__device__ __forceinline__ double* chain_buf(const WalkerDev& w, int spin, int which) {
  return w.chain + ((long long)which * w.S + spin) * w.N * w.N;
}

}  // namespace

// --------------------------------------------------------------------------
// Batched FP64 GEMM, 64x64 output tile per CTA, 16-deep K steps staged in
// SMEM, 4x4 register tile per thread.  The operation (operands, transposes,
// fused diagonal scalings, epilogue) is selected by OP; each CTA finds its
// walker, spin and slice from the descriptors.
// --------------------------------------------------------------------------
enum GemmOp {
  OP_GA = 6,       // M  = Dlmax^-1 (U_L^T U_R) Drmax^-1
  OP_GB = 7,       // M += Dlmin (F_L F_R^T) Drmin
  OP_GG = 8,       // G  = (U_R Drmax^-1) X, wrap error, trace
  // dynamic half-sweep (sweep_for_dynamic_greens, src/dqmc_walker.cpp:424-524)
  OP_DT0_OUT = 11, // G(t,0) = (U_R Drmax^-1) X1, X1 = M^-1 Dlmin F_L; wrap error
  OP_D0T_OUT = 12, // G(0,t) = -(F_R^T Drmin) X, X = M^-1 Dlmax^-1 U_L^T; wrap error
};

constexpr int kTile = 64, kTk = 16;

template <int OP>
__global__ void __launch_bounds__(256) gemm_op_kernel(const WalkerDev* __restrict__ W, int mode, int j, int q,
                                                      int trace_slot) {
  const int wi = blockIdx.z >> 1, sp = blockIdx.z & 1;
  const WalkerDev& w = W[wi];
  if (!is_general(w) || sp >= w.S) return;
  const int N = w.N;
  const int r0 = blockIdx.y * kTile, c0 = blockIdx.x * kTile;
  if (r0 >= N || c0 >= N) return;
  constexpr bool dyn_out = OP == OP_DT0_OUT || OP == OP_D0T_OUT;
  if (dyn_out && !w.gt0) return;
  if (j >= w.nstack || w.ozstab) return;  // ozstab: stabilized by kernels_stab_oz.cu

  const long long NN = (long long)N * N;
  double* G = w.G + sp * NN;
  const double* A = nullptr;
  const double* B = nullptr;
  double* C = nullptr;
  // stack tops for the Green's assembly (lengths after this step's push)
  int nl = 0, nr = 0;
  if (mode == MODE_FWD) { nl = j + 1; nr = w.nstack - 1 - j; }
  else if (mode == MODE_BWD) { nl = w.nstack - 1 - j; nr = j + 1; }
  else { nl = 0; nr = w.nstack; }
  if (!(nl > 0 && nr > 0)) return;  // boundary steps: prep/out kernels
  const double* UL = nl ? stack_level(w, 0, sp, nl - 1) : nullptr;
  const double* UR = nr ? stack_level(w, 1, sp, nr - 1) : nullptr;
  const double* DL = UL ? UL + 2 * NN : nullptr;
  const double* DR = UR ? UR + 2 * NN : nullptr;
  double* scr = w.scr + sp * 2 * NN;  // M (col-major), Y/X (row-major)
  // dynamic buffers: [2][S][N*N], slot = parity of the slice
  const int t_end = min((j + 1) * w.pace, w.Lt);  // forward step j ends at this slice
  auto dbuf = [&](double* base, int par) { return base + ((long long)(par & 1) * w.S + sp) * NN; };
  switch (OP) {
    case OP_GA: A = UL; B = UR; C = scr; break;
    case OP_GB: A = UL + NN; B = UR + NN; C = scr; break;      // F_L, F_R
    case OP_GG: A = UR; B = scr + NN; C = G; break;           // U_R, X (row-major)
    case OP_DT0_OUT: A = UR; B = w.dynx + sp * NN; C = dbuf(w.gt0, t_end); break;   // X1 row-major
    case OP_D0T_OUT: A = UR + NN; B = scr + NN; C = dbuf(w.g0t, t_end); break;      // F_R, X row-major
  }

  __shared__ double As[kTk][kTile + 1];
  __shared__ double Bs[kTk][kTile + 1];
  __shared__ double s_red[8];
  __shared__ double s_inv[(OP == OP_GG || dyn_out) ? kMaxN : 1];  // 1 / max(D_R, 1) or min(D_R, 1) along k
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  if (OP == OP_GG || OP == OP_DT0_OUT) {
    for (int k = tid; k < N; k += 256) s_inv[k] = 1.0 / fmax(DR[k], 1.0);
    __syncthreads();
  } else if (OP == OP_D0T_OUT) {
    for (int k = tid; k < N; k += 256) s_inv[k] = fmin(DR[k], 1.0);
    __syncthreads();
  }
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;

  for (int k0 = 0; k0 < N; k0 += kTk) {
    // A tile: rows r0..r0+63, k k0..k0+15 -> As[kk][rr]
#pragma unroll
    for (int e = tid; e < kTile * kTk; e += 256) {
      const int rr = e % kTile, kk = e / kTile;
      const int r = r0 + rr, k = k0 + kk;
      double v = 0.0;
      if (r < N && k < N) {
        switch (OP) {
          case OP_GA: v = A[(long long)r * N + k]; break;  // U_L^T (r,k) = U_L(k,r)
          case OP_GB: v = A[(long long)k * N + r]; break;
          case OP_GG: v = A[(long long)k * N + r] * s_inv[k]; break;  // U_R(r,k) / drmax_k
          case OP_DT0_OUT: v = A[(long long)k * N + r] * s_inv[k]; break;
          case OP_D0T_OUT: v = A[(long long)r * N + k] * s_inv[k]; break;  // F_R^T(r,k) drmin_k
        }
      }
      As[kk][rr] = v;
    }
    // B tile: k k0..k0+15, cols c0..c0+63 -> Bs[kk][cc]
#pragma unroll
    for (int e = tid; e < kTile * kTk; e += 256) {
      const int kk = e % kTk, cc = e / kTk;
      const int k = k0 + kk, c = c0 + cc;
      double v = 0.0;
      if (k < N && c < N) {
        switch (OP) {
          case OP_GA: v = B[(long long)c * N + k]; break;
          case OP_GB: v = B[(long long)k * N + c]; break;  // F_R^T(k,c) = F_R(c,k)
          case OP_GG: v = B[(long long)k * N + c]; break;                     // X row-major
          case OP_DT0_OUT: v = B[(long long)k * N + c]; break;  // X1 row-major
          case OP_D0T_OUT: v = B[(long long)k * N + c]; break;  // X row-major
        }
      }
      Bs[kk][cc] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kTk; ++kk) {
      double av[4], bv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) av[a] = As[kk][ty + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) bv[b] = Bs[kk][tx + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fma(av[a], bv[b], acc[a][b]);
    }
    __syncthreads();
  }

  // epilogue
  double err = 0.0;
  bool finite = true;
  double* tr = (OP == OP_GG && w.trace && trace_slot >= 0 && trace_slot < w.trace_cap)
                   ? w.trace + ((long long)trace_slot * 2 + sp) * NN : nullptr;
  const bool check = (OP == OP_GG) && !(mode == MODE_INIT || (mode == MODE_BWD && j == w.nstack - 1));
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int r = r0 + ty + 16 * a, c = c0 + tx + 16 * b;
      if (r >= N || c >= N) continue;
      double v = acc[a][b];
      const long long o = (long long)c * N + r;
      switch (OP) {
        case OP_D0T_OUT: v = -v; break;
        case OP_GA: v /= fmax(DL[r], 1.0) * fmax(DR[c], 1.0); break;
        case OP_GB: v *= fmin(DL[r], 1.0) * fmin(DR[c], 1.0); break;
        default: break;
      }
      if (OP == OP_GB) {
        C[o] += v;
      } else if (dyn_out) {
        err = fmax(err, fabs(v - C[o]));
        if (!isfinite(v)) finite = false;
        C[o] = v;
      } else if (OP == OP_GG) {
        if (check) err = fmax(err, fabs(v - C[o]));
        if (!isfinite(v)) finite = false;
        C[o] = v;
        if (tr) tr[o] = v;
        if (w.S == 1) {
          C[NN + o] = v;
          if (tr) tr[NN + o] = v;
        }
      } else {
        C[o] = v;
      }
    }
  if (OP == OP_GG || dyn_out) {
    if (!finite) atomicOr(w.status, ST_NONFINITE_G);
    if (check || dyn_out) {
      for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
      if ((tid & 31) == 0) s_red[tid >> 5] = err;
      __syncthreads();
      if (tid == 0) {
        double m = 0;
        for (int k = 0; k < 8; ++k) m = fmax(m, s_red[k]);
        atomicMax(w.wrap_bits, (unsigned long long)__double_as_longlong(m));
      }
    }
  }
}

// --------------------------------------------------------------------------
// One slice's products with B on global matrices, in the factors of exp(-+dtau K): the two
// plaquette layers of a checkerboard walker (any path), else one ring exponential per lattice
// direction (FP64 walkers; the mixed path's dense walkers take the tensor-core products).
//   KIN_WL_FWD  G <- diag(e+) K G         KIN_WR_FWD  G <- G K^-1 diag(e-)
//   KIN_WR_BWD  G <- G diag(e+) K         KIN_WL_BWD  G <- K^-1 diag(e-) G
//   KIN_CH_FWD  chain' = diag(e+) K chain KIN_CH_BWD  chain' = K^T diag(e+) chain
//   KIN_DT0     G(t,0) = diag(e+) K G(t-1,0)   KIN_D0T  G(0,t) = G(0,t-1) K^-1 diag(e-)
// (mult_B_from_left and its relatives, src/model/repulsive_hubbard.cpp:158-243, with the
// checkerboard's layer order, src/checkerboard/square.cpp:130-226.)  A left product mixes a
// column's sites, a right product a row's, so a CTA takes about 2048 elements of whole columns or
// rows into shared memory, does every pass there and writes them back once: 2 L (3 L) FMAs an
// element instead of N, and one read and one write of the matrix.  As a batched 64 x 64-tile GEMM a
// product of 16 walkers of 16 x 16 took 0.80 ms; a pass of them (48 products) went from 163 to 135
// ms, of 32 walkers of 9 x 9 from 52 to 38 ms.
// --------------------------------------------------------------------------
enum KinOp { KIN_WL_FWD, KIN_WR_FWD, KIN_WR_BWD, KIN_WL_BWD, KIN_CH_FWD, KIN_CH_BWD, KIN_DT0, KIN_D0T };
constexpr int kKinElems = 2048, kKinPer = kKinElems / 256;
// columns (rows) a CTA takes
__host__ __device__ inline int kin_lines(int N) { return kKinElems / N; }

__global__ void __launch_bounds__(256) kin_op_kernel(const WalkerDev* __restrict__ W, int op, int mode, int j, int q) {
  const WalkerDev& w = W[blockIdx.z];
  const int sp = blockIdx.y;
  if (!is_general(w) || sp >= w.S || (w.path == 2 && !w.cb)) return;
  const int N = w.N, L = w.L, V = kin_lines(N), v0 = blockIdx.x * V, nv = min(V, N - v0);
  if (nv <= 0) return;
  int t, nsl, t_hi;
  if (!slice_of(w, mode, j, q, t, nsl, t_hi)) return;
  if ((op == KIN_DT0 || op == KIN_D0T) && !w.gt0) return;
  const long long NN = (long long)N * N;
  const bool right = op == KIN_WR_FWD || op == KIN_WR_BWD || op == KIN_D0T;
  const bool inv = op == KIN_WR_FWD || op == KIN_WL_BWD || op == KIN_D0T;
  const bool pre = op == KIN_WR_BWD || op == KIN_WL_BWD || op == KIN_CH_BWD;  // else the diagonal comes last
  const double* src = w.G + sp * NN;
  double* dst = w.G + sp * NN;
  if (op == KIN_CH_FWD || op == KIN_CH_BWD) {  // ping-pong, checkerboard walkers in place
    src = chain_buf(w, sp, w.cb ? 0 : q & 1);
    dst = chain_buf(w, sp, w.cb ? 0 : (q + 1) & 1);
  } else if (op == KIN_DT0 || op == KIN_D0T) {
    double* base = op == KIN_DT0 ? w.gt0 : w.g0t;
    src = base + ((long long)((t - 1) & 1) * w.S + sp) * NN;
    dst = base + ((long long)(t & 1) * w.S + sp) * NN;
  }
  __shared__ double m[kKinElems], sc[kMaxN], e[32];
  const int tid = threadIdx.x;
  const bool plain = mode == MODE_INIT && w.cb;  // the set-up keeps the plain plaquette product (plaq_product)
  for (int i = tid; i < N; i += 256) {
    const int sf = (w.model == 0 && sp == 1) ? -1 : 1, s = w.fields[(long long)(t - 1) * N + i];
    const int up = ((inv ? -1 : 1) * sf * s > 0) ? 0 : 1;
    sc[i] = plain ? (up ? w.e_ma : w.e_pa) : w.kin_e[inv][up];
  }
  if (!w.cb && tid < L) e[tid] = w.kin[(inv ? L : 0) + tid];
  // element k of the tile: site and line, left k = line N + site (contiguous in the matrix),
  // right k = site nv + line
  const int nel = N * nv, ss = right ? nv : 1;
  int site[kKinPer];
#pragma unroll
  for (int u = 0; u < kKinPer; ++u) {
    const int k = tid + 256 * u;
    site[u] = right ? k / nv : k % N;
  }
  auto gofs = [&](int k, int s) { return right ? (long long)s * N + v0 + (k - s * nv) : (long long)v0 * N + k; };
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kKinPer; ++u) {
    const int k = tid + 256 * u;
    if (k < nel) {
      const double x = src[gofs(k, site[u])];
      m[k] = pre ? x * sc[site[u]] : x;
    }
  }
  __syncthreads();
  if (w.cb) {
    const int nq = (L >> 1) * (L >> 1), first = pre ? 0 : 1;  // layer A (parity 0) or B first
    const double h = inv ? -w.cb_h : w.cb_h;
    const int sv = right ? 1 : N;
    for (int p = 0; p < 2; ++p) {
      for (int it = tid; it < nq * nv; it += 256) {
        const int pq = right ? it / nv : it % nq, v = right ? it % nv : it / nq;
        int idx[4];
        plaq_sites(L, pq, first ^ p, idx);
        double x[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = m[idx[a] * ss + v * sv];
        if (plain) plaq_product(x, w.cbP);
        else plaq_apply(x, h);
#pragma unroll
        for (int a = 0; a < 4; ++a) m[idx[a] * ss + v * sv] = x[a];
      }
      __syncthreads();
    }
  } else {
    for (int d = 0, st = 1; d < w.dim; ++d, st *= L) {
      double acc[kKinPer];
      int x[kKinPer], base[kKinPer];
      const int step = st * ss;
#pragma unroll
      for (int u = 0; u < kKinPer; ++u) {
        const int k = tid + 256 * u;
        x[u] = (k < nel) ? (site[u] / st) % L : 0;
        base[u] = (k < nel) ? k - x[u] * step : 0;
        acc[u] = 0.0;
      }
      for (int y = 0; y < L; ++y)
#pragma unroll
        for (int u = 0; u < kKinPer; ++u)
          if ((tid & ~31) + 256 * u < nel)  // uniform in the warp
            acc[u] = fma(e[abs(x[u] - y)], m[base[u] + y * step], acc[u]);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kKinPer; ++u)
        if (tid + 256 * u < nel) m[tid + 256 * u] = acc[u];
      __syncthreads();
    }
  }
#pragma unroll
  for (int u = 0; u < kKinPer; ++u) {
    const int k = tid + 256 * u;
    if (k < nel) dst[gofs(k, site[u])] = pre ? m[k] : m[k] * sc[site[u]];
  }
}

// --------------------------------------------------------------------------
// Chain start of step j: chain <- U_top diag(D_top) or I (general walkers).
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(256) chain_init_general_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!is_general(w) || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const int side = (mode == MODE_FWD) ? 0 : 1;
  const double* lv = j ? stack_level(w, side, sp, j - 1) : nullptr;
  double* C = chain_buf(w, sp, 0);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)N * N;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e % N), c = (int)(e / N);
    C[e] = lv ? lv[e] * lv[2LL * N * N + c] : ((r == c) ? 1.0 : 0.0);
  }
}

// --------------------------------------------------------------------------
// Equal-time measurement on global G (general N); mode/j/q select the slot as
// in the SMEM kernels.  after_stab = 1 measures the slot closing the step
// with the fresh G (forward) or slot Lt-1 with the final G(0) (backward).
//
// A cluster of P CTAs per walker shares the pairs of 32-site tiles (I <= J); rank 0 adds the
// parts, read from the other CTAs' shared memory, in rank order.  Unordered site pairs {i, j} are
// visited once, 13 FP64 operations (9 with one spin matrix), with X = G_ij G_ji summed over spins
// and the sites' sums n and differences m of 1 - G_ii:
//   n(k)          ff_ij G_ji + ff_ji G_ij, spins summed (ff is not even on odd sides)
//   SDW, CDW      (ff_ij + ff_ji) (m_i m_j - X), (n_i n_j - X)
//   s-wave        Gu_ij Gd_ij + Gu_ji Gd_ji
// The tile above the diagonal is read along its columns, the one below through shared memory.
// FP64 throughput of one SM and the strided reads of G(j, i) bounded the one-CTA form: 264 us a
// slice for 6 walkers of two spins at N = 256, 222 us for 128 walkers of one.
// --------------------------------------------------------------------------
// CTAs that share a walker's tile pairs: by its own size, so that its sums are added in the same order
// whatever else is in the launch (the cluster is the largest walker's)
__host__ __device__ inline int measure_ctas(int N) {
  const int nt = (N + 31) / 32, pairs = nt * (nt + 1) / 2;
  return pairs >= 8 ? 8 : pairs >= 4 ? 4 : pairs >= 2 ? 2 : 1;
}

template <int P>
__global__ void __launch_bounds__(256) __cluster_dims__(P, 1, 1)
    measure_general_kernel(const WalkerDev* __restrict__ W, int mode, int j, int q, int after_stab) {
  namespace cg = cooperative_groups;
  const WalkerDev& w = W[blockIdx.y];
  const int rank = blockIdx.x;
  // the whole cluster leaves or stays
  if (!is_general(w)) return;
  double sg;
  if (after_stab) {
    if (j >= w.nstack) return;
    if (mode == MODE_BWD && j != w.nstack - 1) return;
    sg = (mode == MODE_BWD) ? *w.sign_Lt : *w.sign;
  } else {
    int t, nsl, t_hi;
    if (!slice_of(w, mode, j, q, t, nsl, t_hi)) return;
    const bool here = (mode == MODE_FWD) ? (t != t_hi) : (t != w.Lt);
    if (!here) return;
    sg = *w.sign;
  }
  const int N = w.N, L = w.L, LL = L * L;
  const long long NN = (long long)N * N;
  const bool one = (w.S == 1);
  const double* gu = w.G;
  const double* gd = one ? w.G : w.G + NN;
  extern __shared__ double sh[];
  double* sn = sh;           // n_i = (1 - gu_ii) + (1 - gd_ii)
  double* sm = sh + N;       // m_i = (1 - gu_ii) - (1 - gd_ii)
  double* ff = sh + 2 * N;
  int* sxyz = reinterpret_cast<int*>(ff + N);  // x | y << 10 | z << 20
  __shared__ double s_t[2][32][33];            // the tiles below the diagonal, [spin][i][j]
  __shared__ double red[8 * 8], part[8];
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = threadIdx.x; i < N; i += 256) {
    const double a = gu[(long long)i * N + i], b = gd[(long long)i * N + i];
    const double du = 1.0 - a, dd = 1.0 - b, n = du + dd, mm = du - dd;
    sn[i] = n;
    sm[i] = mm;
    ff[i] = w.ff[i];
    sxyz[i] = (i % L) | ((i / L) % L) << 10 | (i / LL) << 20;  // z = 0 on the square lattice
    if (rank == 0) {
      const double ab = a + b, x = fma(du, a, dd * b);
      v[0] += ab;
      v[1] = fma(du, dd, v[1]);
      v[2] += fma(-2.0 * a, b, ab);
      // bonds to the +x, +y (, +z) neighbours (measure_methods.cpp:87-95)
      for (int d = 0; d < w.dim; ++d) {
        const long long c = (long long)site_nn(L, i, d) * N + i;
        v[3] += gu[c] + gd[c];
      }
      // the pair i = j (Fourier factor 1)
      v[4] += ab;
      v[5] += fma(mm, mm, x);
      v[6] += fma(n, n, x);
      v[7] = fma(du, dd, v[7]);
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nt = (N + 31) / 32, share = measure_ctas(N);
  double p4 = 0.0, p5 = 0.0, p6 = 0.0, p7 = 0.0;
  int k = 0;  // tile pairs, dealt to the CTAs in turn
  for (int tj = 0; tj < nt; ++tj)
    for (int ti = 0; ti <= tj; ++ti, ++k) {
      if (k % share != rank) continue;
      const int i0 = ti * 32, j0 = tj * 32, i = i0 + lane;
      __syncthreads();  // the previous tile's readers are done
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // column i of the tile below: G(j, i), lanes along j
        const int c = wid + 8 * u;
        const bool in = j0 + lane < N && i0 + c < N;
        s_t[0][c][lane] = in ? gu[(long long)(i0 + c) * N + j0 + lane] : 0.0;
        if (!one) s_t[1][c][lane] = in ? gd[(long long)(i0 + c) * N + j0 + lane] : 0.0;
      }
      double gij[2][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int jj = j0 + wid + 8 * u;
        const bool in = i < N && jj < N;
        gij[0][u] = in ? gu[(long long)jj * N + i] : 0.0;
        gij[1][u] = (in && !one) ? gd[(long long)jj * N + i] : 0.0;
      }
      __syncthreads();
      const int ci = (i < N) ? sxyz[i] : 0, xi = ci & 1023, yi = (ci >> 10) & 1023, zi = ci >> 20;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int cj = wid + 8 * u, jj = j0 + cj;
        if (jj >= N) continue;  // uniform in the warp
        if (i >= N || i >= jj) continue;
        const int c = sxyz[jj], dx = (c & 1023) - xi, dy = ((c >> 10) & 1023) - yi, dz = (c >> 20) - zi;
        const double f_ij = ff[(dx + (dx < 0 ? L : 0)) + (dy + (dy < 0 ? L : 0)) * L + (dz + (dz < 0 ? L : 0)) * LL];
        const double f_ji = ff[(-dx + (dx > 0 ? L : 0)) + (-dy + (dy > 0 ? L : 0)) * L + (-dz + (dz > 0 ? L : 0)) * LL];
        const double f = f_ij + f_ji, a = gij[0][u], at = s_t[0][lane][cj];
        if (one) {  // m = 0; the spins' factor 2 of n(k) and X follows the loop
          const double x = a * at;
          p4 = fma(f_ij, at, p4);
          p4 = fma(f_ji, a, p4);
          p5 = fma(f, x, p5);
          p6 = fma(f, fma(0.5 * sn[i], sn[jj], -x), p6);
          p7 = fma(a, a, p7);
          p7 = fma(at, at, p7);
        } else {
          const double b = gij[1][u], bt = s_t[1][lane][cj];
          const double x = fma(b, bt, a * at);
          p4 = fma(f_ij, at + bt, p4);
          p4 = fma(f_ji, a + b, p4);
          p5 = fma(f, fma(sm[i], sm[jj], -x), p5);
          p6 = fma(f, fma(sn[i], sn[jj], -x), p6);
          p7 = fma(a, b, p7);
          p7 = fma(at, bt, p7);
        }
      }
    }
  v[4] += one ? 2.0 * p4 : p4;
  v[5] += one ? -2.0 * p5 : p5;
  v[6] += one ? 2.0 * p6 : p6;
  v[7] += p7;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const double s = warp_sum_g(v[e]);
    if (lane == 0) red[e * 8 + wid] = s;
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    double s = 0.0;
    for (int e = 0; e < 8; ++e) s += red[threadIdx.x * 8 + e];
    part[threadIdx.x] = s;
  }
  cg::cluster_group cl = cg::this_cluster();
  if (P > 1) cl.sync();
  else __syncthreads();
  if (rank == 0 && threadIdx.x < kNumObs) {
    // thread k adds observable k
    const int o = threadIdx.x;
    const int src[kNumObs] = {0, 1, 3, 4, 2, 5, 6, 7, 0};
    double tot = 0.0;
    for (int p = 0; p < P; ++p) {
      const double* rp = (P > 1) ? cl.map_shared_rank(part, p) : part;
      tot += rp[src[o]];
    }
    const double n = (double)N;
    double add = sg * tot / n;
    if (o == 0) add = sg * (2.0 - tot / n);
    if (o == 2) add = sg * (2.0 * w.hop_t) * tot / n;
    if (o == 3) add = sg * (1.0 - 0.5 * tot / n);
    if (o == 5 || o == 6) add = sg * tot / (n * n);
    if (o == 8) add = sg;
    w.obs[o] += add;
    w.obs_cnt[o] += 1;
  }
  if (P > 1) cl.sync();  // the parts stay until rank 0 has read them
}

// CTAs per walker: the largest walker's, at most a portable cluster of 8
static void launch_measure_general(const WalkerDev* W, int nw, int maxN, int mode, int j, int q, int after_stab,
                                   cudaStream_t st) {
  const int P = measure_ctas(maxN);
  const size_t sm = (size_t)maxN * (3 * sizeof(double) + sizeof(int));
  if (P == 8) measure_general_kernel<8><<<dim3(8, nw), 256, sm, st>>>(W, mode, j, q, after_stab);
  else if (P == 4) measure_general_kernel<4><<<dim3(4, nw), 256, sm, st>>>(W, mode, j, q, after_stab);
  else if (P == 2) measure_general_kernel<2><<<dim3(2, nw), 256, sm, st>>>(W, mode, j, q, after_stab);
  else measure_general_kernel<1><<<dim3(1, nw), 256, sm, st>>>(W, mode, j, q, after_stab);
}

// --------------------------------------------------------------------------
// Column-pivoted QR push, general N: one CTA per (walker, spin), thread per
// column, matrix in a row-major HBM/L2 scratch (coalesced across threads).
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) push_general_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (!is_general(w) || w.ozstab || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  const int side = (mode == MODE_FWD) ? 0 : 1;
  int nsl = 0;
  {
    const int k = (mode == MODE_FWD) ? j : (w.nstack - 1 - j);
    nsl = min((k + 1) * w.pace, w.Lt) - k * w.pace;
  }
  const double* Cin = w.cb ? chain_buf(w, sp, 0) : chain_buf(w, sp, nsl & 1);
  double* X = w.scr + sp * 2 * NN;  // row-major: X[r*N + c]
  extern __shared__ double sh[];
  double* v = sh;          // reflector / scratch column [N]
  double* vn1 = sh + N;
  double* vn2 = sh + 2 * N;
  double* tau = sh + 3 * N;
  double* invd = sh + 4 * N;
  int* perm = (int*)(sh + 5 * N);
  __shared__ int s_piv;
  __shared__ double s_tau, s_scal;
  __shared__ long long s_key[32];
  __shared__ int s_idx[32];
  const int tj = threadIdx.x;
  const bool own = tj < N;
  auto Xat = [&](int r, int c) -> double& { return X[(long long)r * N + c]; };

  if (own) {
    double s0 = 0, s1 = 0;
    for (int r = 0; r < N; ++r) {
      const double a = Cin[(long long)tj * N + r];
      Xat(r, tj) = a;
      if (r & 1) s1 = fma(a, a, s1); else s0 = fma(a, a, s0);
    }
    vn1[tj] = vn2[tj] = sqrt(s0 + s1);
    perm[tj] = tj;
  }
  __syncthreads();
  const double tol3z = 1.4901161193847656e-08;
  const int nwarps = (blockDim.x + 31) >> 5;
  for (int k = 0; k < N; ++k) {
    // pivot
    long long key = (own && tj >= k) ? __double_as_longlong(vn1[tj]) : -1LL;
    int bi = tj;
    for (int o = 16; o > 0; o >>= 1) {
      const long long ok = __shfl_xor_sync(0xffffffffu, key, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ok > key || (ok == key && oi < bi)) { key = ok; bi = oi; }
    }
    if ((tj & 31) == 0) { s_key[tj >> 5] = key; s_idx[tj >> 5] = bi; }
    __syncthreads();
    if (tj == 0) {
      long long bk = s_key[0];
      int b = s_idx[0];
      for (int q = 1; q < nwarps; ++q)
        if (s_key[q] > bk || (s_key[q] == bk && s_idx[q] < b)) { bk = s_key[q]; b = s_idx[q]; }
      s_piv = b;
    }
    __syncthreads();
    const int pv = s_piv;
    if (pv != k) {
      if (own) {  // thread tj swaps row tj of columns k and pv
        const double a = Xat(tj, k);
        Xat(tj, k) = Xat(tj, pv);
        Xat(tj, pv) = a;
      }
      if (tj == 0) {
        const int tp = perm[k]; perm[k] = perm[pv]; perm[pv] = tp;
        double tv = vn1[k]; vn1[k] = vn1[pv]; vn1[pv] = tv;
        tv = vn2[k]; vn2[k] = vn2[pv]; vn2[pv] = tv;
      }
      __syncthreads();
    }
    // reflector: column k rows > k into v (SMEM), norm by block reduction
    double xr = 0.0;
    if (own && tj > k) { xr = Xat(tj, k); v[tj] = xr; }
    double s = warp_sum_g(xr * xr);
    if ((tj & 31) == 0) s_key[tj >> 5] = __double_as_longlong(s);
    __syncthreads();
    if (tj == 0) {
      double xn2 = 0;
      for (int q = 0; q < nwarps; ++q) xn2 += __longlong_as_double(s_key[q]);
      const double alpha = Xat(k, k);
      double t2 = 0.0, beta = alpha, scal = 1.0;
      if (xn2 != 0.0) {
        const double nrm = sqrt(alpha * alpha + xn2);
        beta = alpha >= 0 ? -nrm : nrm;
        t2 = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
      s_tau = t2; s_scal = scal;
      tau[k] = t2;
      Xat(k, k) = beta;
    }
    __syncthreads();
    if (own && tj > k) {
      const double vv = v[tj] * s_scal;
      v[tj] = vv;
      Xat(tj, k) = vv;
    }
    __syncthreads();
    const double tk = s_tau;
    if (own && tj > k) {
      if (tk != 0.0) {
        double a0 = Xat(k, tj), a1 = 0.0;
        int r = k + 1;
        for (; r + 1 < N; r += 2) {
          a0 = fma(v[r], Xat(r, tj), a0);
          a1 = fma(v[r + 1], Xat(r + 1, tj), a1);
        }
        if (r < N) a0 = fma(v[r], Xat(r, tj), a0);
        const double wv = (a0 + a1) * tk;
        Xat(k, tj) -= wv;
        for (r = k + 1; r < N; ++r) Xat(r, tj) = fma(-wv, v[r], Xat(r, tj));
      }
      const double v1 = vn1[tj];
      if (v1 != 0.0) {
        double tmp = fabs(Xat(k, tj)) / v1;
        tmp = fmax(0.0, 1.0 - tmp * tmp);
        const double r2 = v1 / vn2[tj];
        if (tmp * r2 * r2 <= tol3z) {
          double q0 = 0, q1 = 0;
          int r = k + 1;
          for (; r + 1 < N; r += 2) {
            q0 = fma(Xat(r, tj), Xat(r, tj), q0);
            q1 = fma(Xat(r + 1, tj), Xat(r + 1, tj), q1);
          }
          if (r < N) q0 = fma(Xat(r, tj), Xat(r, tj), q0);
          vn1[tj] = vn2[tj] = sqrt(q0 + q1);
        } else {
          vn1[tj] = v1 * sqrt(tmp);
        }
      }
    }
    __syncthreads();
  }
  // D and F = (D^-1 R P^T) F_prev
  double* lv = stack_level(w, side, sp, j);
  double* Uo = lv;
  double* Fo = lv + NN;
  double* Do = lv + 2 * NN;
  if (own) {
    const double d = fabs(Xat(tj, tj));
    Do[tj] = d;
    invd[tj] = (d != 0.0) ? 1.0 / d : 0.0;
    if (d == 0.0 || !isfinite(d)) atomicOr(w.status, ST_SINGULAR);
  }
  __syncthreads();
  if (own) {
    const int c = tj;
    if (j == 0) {
      double* fc = Fo + (long long)perm[c] * N;
      for (int i = 0; i < N; ++i) fc[i] = (i <= c) ? Xat(i, c) * invd[i] : 0.0;
    } else {
      const double* fp = stack_level(w, side, sp, j - 1) + NN + (long long)c * N;
      double* fo = Fo + (long long)c * N;
      for (int i = 0; i < N; ++i) {
        double a0 = 0.0, a1 = 0.0;
        int k = i;
        for (; k + 1 < N; k += 2) {
          a0 = fma(Xat(i, k), fp[perm[k]], a0);
          a1 = fma(Xat(i, k + 1), fp[perm[k + 1]], a1);
        }
        if (k < N) a0 = fma(Xat(i, k), fp[perm[k]], a0);
        fo[i] = (a0 + a1) * invd[i];
      }
    }
  }
  __syncthreads();
  // Q in place (dorg2r order); reflector i staged into v
  for (int i = N - 1; i >= 0; --i) {
    const double ti = tau[i];
    if (own && tj > i) v[tj] = Xat(tj, i);
    __syncthreads();
    if (i < N - 1 && own && tj > i && ti != 0.0) {
      double a0 = Xat(i, tj), a1 = 0.0;
      int r = i + 1;
      for (; r + 1 < N; r += 2) {
        a0 = fma(v[r], Xat(r, tj), a0);
        a1 = fma(v[r + 1], Xat(r + 1, tj), a1);
      }
      if (r < N) a0 = fma(v[r], Xat(r, tj), a0);
      const double wv = (a0 + a1) * ti;
      Xat(i, tj) -= wv;
      for (r = i + 1; r < N; ++r) Xat(r, tj) = fma(-wv, v[r], Xat(r, tj));
    }
    __syncthreads();
    if (own) {
      const int r = tj;
      if (r > i) Xat(r, i) = v[r] * -ti;
      else if (r == i) Xat(r, i) = 1.0 - ti;
      else Xat(r, i) = 0.0;
    }
    __syncthreads();
  }
  if (own)
    for (int r = 0; r < N; ++r) Uo[(long long)tj * N + r] = Xat(r, tj);
}

// --------------------------------------------------------------------------
// Green's assembly support (general N).
//   prep: boundary cases build M and Y; general case builds Y = Dlmax^-1 U_L^T
//         (M comes from OP_GA/OP_GB).  M col-major in scr, Y row-major in scr+NN.
//   lu:   solve M X = Y (partial pivoting), thread per column of [M | Y], X in Y.
//   out:  boundary cases write G = X (or X^T) with wrap error and trace.
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(256) greens_prep_general_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!is_general(w) || w.ozstab || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  int nl, nr;
  if (mode == MODE_FWD) { nl = j + 1; nr = w.nstack - 1 - j; }
  else if (mode == MODE_BWD) { nl = w.nstack - 1 - j; nr = j + 1; }
  else { nl = 0; nr = w.nstack; }
  double* M = w.scr + sp * 2 * NN;
  double* Y = M + NN;
  const bool both = nl > 0 && nr > 0;
  const double* lv = (nl > 0) ? stack_level(w, 0, sp, nl - 1) : stack_level(w, 1, sp, nr - 1);
  const double* U = lv;
  const double* F = lv + NN;
  const double* D = lv + 2 * NN;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < NN; e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e / N), c = (int)(e % N);   // Y row-major: Y[r*N + c]
    const double y = U[(long long)r * N + c] / fmax(D[r], 1.0);  // (Dmax^-1 U^T)(r,c)
    Y[e] = y;
    if (!both) M[(long long)c * N + r] = y + fmin(D[r], 1.0) * F[(long long)c * N + r];
  }
}

__global__ void __launch_bounds__(1024) lu_solve_general_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (!is_general(w) || w.ozstab || sp >= w.S || j >= w.nstack) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  double* M = w.scr + sp * 2 * NN;  // col-major
  double* Y = M + NN;               // row-major
  extern __shared__ double sh[];
  double* l = sh;  // multipliers of the current step
  __shared__ int s_p;
  __shared__ int s_bad;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) s_bad = 0;
  for (int k = 0; k < N; ++k) {
    if (tid < 32) {  // pivot: warp argmax of |M(r,k)|, r >= k, on the integer bit patterns
      long long key = -1;
      int bi = k;
      for (int r = k + tid; r < N; r += 32) {
        const long long a = __double_as_longlong(M[(long long)k * N + r]) & 0x7fffffffffffffffLL;
        if (a > key) { key = a; bi = r; }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const long long ok = __shfl_xor_sync(0xffffffffu, key, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ok > key || (ok == key && oi < bi)) { key = ok; bi = oi; }
      }
      if (tid == 0) { s_p = bi; if (key == 0) s_bad = 1; }
    }
    __syncthreads();
    const int p = s_p;
    if (w.dpiv && tid == 0) w.dpiv[sp * N + k] = p;  // kept for a second right-hand side
    if (p != k) {  // swap rows k and p of M (all columns) and Y
      for (int c = tid; c < N; c += nt) {
        double* mc = M + (long long)c * N;
        const double a = mc[k]; mc[k] = mc[p]; mc[p] = a;
        const double b = Y[(long long)k * N + c]; Y[(long long)k * N + c] = Y[(long long)p * N + c];
        Y[(long long)p * N + c] = b;
      }
      __syncthreads();
    }
    const double piv = M[(long long)k * N + k];
    const double inv = (piv != 0.0) ? 1.0 / piv : 0.0;
    for (int r = k + 1 + tid; r < N; r += nt) {
      const double lr = M[(long long)k * N + r] * inv;
      M[(long long)k * N + r] = lr;
      l[r] = lr;
    }
    __syncthreads();
    // columns of M right of k, then all columns of Y (row-major: thread per column c)
    for (int c = k + 1 + tid; c < N; c += nt) {
      double* mc = M + (long long)c * N;
      const double mk = mc[k];
      if (mk != 0.0)
        for (int r = k + 1; r < N; ++r) mc[r] = fma(-l[r], mk, mc[r]);
    }
    for (int c = tid; c < N; c += nt) {
      const double yk = Y[(long long)k * N + c];
      if (yk != 0.0)
        for (int r = k + 1; r < N; ++r) Y[(long long)r * N + c] = fma(-l[r], yk, Y[(long long)r * N + c]);
    }
    __syncthreads();
  }
  // back substitution, thread per column of Y (reciprocal diagonal staged in l)
  for (int k = tid; k < N; k += nt) l[k] = 1.0 / M[(long long)k * N + k];
  __syncthreads();
  for (int c = tid; c < N; c += nt) {
    for (int k = N - 1; k >= 0; --k) {
      const double yk = Y[(long long)k * N + c] * l[k];
      Y[(long long)k * N + c] = yk;
      for (int r = 0; r < k; ++r) Y[(long long)r * N + c] = fma(-M[(long long)k * N + r], yk, Y[(long long)r * N + c]);
    }
  }
  if (tid == 0 && s_bad) atomicOr(w.status, ST_SINGULAR);
}

__global__ void __launch_bounds__(256) greens_out_general_kernel(const WalkerDev* __restrict__ W, int mode, int j,
                                                                 int trace_slot) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!is_general(w) || w.ozstab || sp >= w.S || j >= w.nstack) return;
  int nl, nr;
  if (mode == MODE_FWD) { nl = j + 1; nr = w.nstack - 1 - j; }
  else if (mode == MODE_BWD) { nl = w.nstack - 1 - j; nr = j + 1; }
  else { nl = 0; nr = w.nstack; }
  if (nl > 0 && nr > 0) return;  // general case finished by OP_GG
  const int N = w.N;
  const long long NN = (long long)N * N;
  const double* X = w.scr + sp * 2 * NN + NN;  // row-major
  double* G = w.G + sp * NN;
  double* tr = (w.trace && trace_slot >= 0 && trace_slot < w.trace_cap) ? w.trace + ((long long)trace_slot * 2 + sp) * NN
                                                                       : nullptr;
  const bool transpose_out = (nl == 0);
  const bool check = !(mode == MODE_INIT || (mode == MODE_BWD && j == w.nstack - 1));
  double err = 0.0;
  bool finite = true;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < NN; e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e % N), c = (int)(e / N);  // G col-major (r, c)
    const double v = transpose_out ? X[(long long)c * N + r] : X[(long long)r * N + c];
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

// sign(det G_up det G_dn) for general walkers: LU with partial pivoting of a copy in scr (col-major),
// a CTA per spin in a cluster of two.  Per column one barrier: warp 0 updates the next column in
// shared memory and finds its pivot and multipliers while the other warps update the rest, lanes
// along the rows; the row exchange happens in the update.  The order of the FMAs on an element is
// that of the plain right-looking LU.  48 walkers of 12 x 12: 6.1 ms with both spins in one CTA, a
// serial pivot search and a thread per column; a warm start of them went from 23.9 to 18.1 ms.
__global__ void __launch_bounds__(512) __cluster_dims__(2, 1, 1) sign_general_kernel(const WalkerDev* __restrict__ W) {
  namespace cg = cooperative_groups;
  const WalkerDev& w = W[blockIdx.y];
  const int sp = blockIdx.x;  // the cluster's rank
  if (!is_general(w)) return;
  if (w.S == 1) {  // equal spins: the determinants' signs multiply to +1
    if (sp == 0 && threadIdx.x == 0) *w.sign = 1.0;
    return;
  }
  const int N = w.N, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const long long NN = (long long)N * N;
  extern __shared__ double sh[];
  double* l = sh;             // [2][N] multipliers of columns k, k + 1
  double* col = sh + 2 * N;   // [N] the pivot column
  __shared__ int s_p[2], s_neg;
  double* M = w.scr + sp * 2 * NN;
  const double* Gg = w.G + sp * NN;
  for (long long e = threadIdx.x; e < NN; e += blockDim.x) M[e] = Gg[e];
  int neg = 0;
  // warp 0: pivot of column k (the first largest |a| of rows k.., kept in col) and its multipliers
  auto factor = [&](int k, int buf) {
    long long key = -1;
    int p = k;
    for (int r = k + lane; r < N; r += 32) {
      long long a = __double_as_longlong(col[r]) & 0x7fffffffffffffffLL;
      if (a > 0x7ff0000000000000LL) a = (r == k) ? a : -1;  // a NaN is the largest only on the diagonal
      if (a > key) { key = a; p = r; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const long long ok = __shfl_xor_sync(0xffffffffu, key, o);
      const int op = __shfl_xor_sync(0xffffffffu, p, o);
      if (ok > key || (ok == key && op < p)) { key = ok; p = op; }
    }
    const double piv = col[p], below = col[k], inv = 1.0 / piv;
    neg += (p != k ? 1 : 0) + (piv < 0 ? 1 : 0);
    for (int r = k + 1 + lane; r < N; r += 32) l[buf * N + r] = ((r == p) ? below : col[r]) * inv;
    if (lane == 0) s_p[buf] = p;
    __syncwarp();
  };
  __syncthreads();
  if (wid == 0) {
    for (int r = lane; r < N; r += 32) col[r] = M[r];
    __syncwarp();
    factor(0, 0);
  }
  __syncthreads();
  for (int k = 0; k + 1 < N; ++k) {
    const int buf = k & 1, p = s_p[buf];
    const double* lk = l + buf * N;
    if (wid == 0) {  // column k + 1 first: the next pivot is found while the others update
      const double* mc = M + (long long)(k + 1) * N;
      const double mk = mc[p], old = mc[k];
      for (int r = k + 1 + lane; r < N; r += 32) col[r] = fma(-lk[r], mk, (r == p) ? old : mc[r]);
      __syncwarp();
      factor(k + 1, buf ^ 1);
    } else {
      for (int c = k + 1 + wid; c < N; c += nwarp - 1) {
        double* mc = M + (long long)c * N;
        const double mk = mc[p], old = mc[k];
        __syncwarp();  // row p is read before its lane writes it
        for (int r = k + 1 + lane; r < N; r += 32) mc[r] = fma(-lk[r], mk, (r == p) ? old : mc[r]);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) s_neg = neg;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  if (sp == 0 && threadIdx.x == 0) *w.sign = ((s_neg + *cl.map_shared_rank(&s_neg, 1)) % 2 == 0) ? 1.0 : -1.0;
  cl.sync();
}

// --------------------------------------------------------------------------
// Dynamic half-sweep (sweep_for_dynamic_greens, src/dqmc_walker.cpp:424-524):
// the forward half-sweep with the fields fixed, carrying G(t,0) and G(0,t)
// besides G(t,t).  At each stabilization, with M and X = M^-1 Dlmax^-1 U_L^T of
// the equal-time assembly (LU pivots kept):
//   G(t,0) = U_R Drmax^-1 M^-1 (Dlmin F_L)     (compute_dynamic_greens, :246-325)
//   G(0,t) = -F_R^T Drmin X                     (push-through form of the second
//            formula, exact for any right factor F; the reference's form needs an
//            orthogonal V)
// and at t = beta (right stack empty, H = Dmax^-1 U^T + Dmin F):
//   G(beta,0) = H^-1 Dmin F,  G(0,beta) = -H^-1 Dmax^-1 U^T = -G(beta,beta).
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(256) dyn_init_kernel(const WalkerDev* __restrict__ W) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.gt0 || sp >= w.S) return;
  const long long NN = (long long)w.N * w.N;
  const double* G = w.G + sp * NN;
  double* t0 = w.gt0 + sp * NN;  // parity slot 0 (t = 0)
  double* ot = w.g0t + sp * NN;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < NN; e += (long long)gridDim.x * 256) {
    const int r = (int)(e % w.N), c = (int)(e / w.N);
    t0[e] = G[e];
    ot[e] = G[e] - ((r == c) ? 1.0 : 0.0);
  }
}

// X1 = M^-1 (Dlmin F_L) with the LU factors and pivots left by lu_solve_general_kernel;
// thread per column of the right-hand side (row-major, coalesced across threads)
__global__ void __launch_bounds__(1024) dyn_resolve_kernel(const WalkerDev* __restrict__ W, int j) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (!w.gt0 || w.ozstab || sp >= w.S || j >= w.nstack) return;  // tensor-core walkers: oz_greens
  const int N = w.N;
  const long long NN = (long long)N * N;
  const int nl = j + 1;  // forward step j: left stack holds j + 1 levels
  const double* lv = stack_level(w, 0, sp, nl - 1);
  const double* F = lv + NN;
  const double* D = lv + 2 * NN;
  const double* M = w.scr + sp * 2 * NN;  // LU factors, col-major
  const int* piv = w.dpiv + sp * N;
  double* X = w.dynx + sp * NN;  // row-major
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    for (int r = 0; r < N; ++r) X[(long long)r * N + c] = fmin(D[r], 1.0) * F[(long long)c * N + r];
    // the factorization swapped whole rows (multipliers included): all swaps first, then L and U
    for (int k = 0; k < N; ++k) {
      const int p = piv[k];
      if (p != k) {
        const double a = X[(long long)k * N + c];
        X[(long long)k * N + c] = X[(long long)p * N + c];
        X[(long long)p * N + c] = a;
      }
    }
    for (int k = 0; k < N; ++k) {
      const double yk = X[(long long)k * N + c];
      if (yk != 0.0)
        for (int r = k + 1; r < N; ++r) X[(long long)r * N + c] = fma(-M[(long long)k * N + r], yk, X[(long long)r * N + c]);
    }
    for (int k = N - 1; k >= 0; --k) {
      const double yk = X[(long long)k * N + c] / M[(long long)k * N + k];
      X[(long long)k * N + c] = yk;
      for (int r = 0; r < k; ++r) X[(long long)r * N + c] = fma(-M[(long long)k * N + r], yk, X[(long long)r * N + c]);
    }
  }
}

// t = beta (forward step nstack - 1): G(beta,0) = X1, G(0,beta) = -X, with their wrap errors
__global__ void __launch_bounds__(256) dyn_boundary_kernel(const WalkerDev* __restrict__ W, int j) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (!w.gt0 || w.ozstab || sp >= w.S || j != w.nstack - 1) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  const int par = w.Lt & 1;
  double* t0 = w.gt0 + ((long long)par * w.S + sp) * NN;
  double* ot = w.g0t + ((long long)par * w.S + sp) * NN;
  const double* X1 = w.dynx + sp * NN;        // row-major
  const double* X = w.scr + sp * 2 * NN + NN;  // row-major
  double err = 0.0;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < NN; e += (long long)gridDim.x * 256) {
    const int r = (int)(e % N), c = (int)(e / N);
    const double a = X1[(long long)r * N + c], b = -X[(long long)r * N + c];
    err = fmax(err, fmax(fabs(a - t0[e]), fabs(b - ot[e])));
    t0[e] = a;
    ot[e] = b;
  }
  for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
  if ((threadIdx.x & 31) == 0) atomicMax(w.wrap_bits, (unsigned long long)__double_as_longlong(err));
}

// G(k,tau) += sign / N sum_ij FF(r_j - r_i) (G_up(t,0)(j,i) + G_dn(t,0)(j,i)) / 2 at the listed tau
// (measure_greens_functions, src/measure/measure_methods.cpp:278-308).  phase 0: slices inside
// the interval (after propagation); 1: the interval's last slice (after stabilization);
// 2: tau = 0 from G(beta,beta) after the sweep.  A cluster of kDynCtas CTAs per walker shares the
// columns, displacements and sites; rank 0 adds the parts in rank order.  One CTA per walker took
// 1.0 ms a listed tau for 8 walkers of 24 x 24.
constexpr int kDynCtas = 8;
__global__ void __launch_bounds__(256) __cluster_dims__(kDynCtas, 1, 1)
    dyn_measure_kernel(const WalkerDev* __restrict__ W, int j, int q, int phase) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const WalkerDev& w = W[blockIdx.y];
  const int rank = blockIdx.x;
  if (!w.gt0 || j >= w.nstack) return;
  int t;
  if (phase == 2) {
    t = 0;
  } else {
    const int t_lo = j * w.pace + 1, t_hi = min((j + 1) * w.pace, w.Lt);
    if (phase == 0) {
      if (q >= t_hi - t_lo) return;  // the last slice of the interval is measured after stabilization
      t = t_lo + q;
    } else {
      t = t_hi;
    }
    if (t >= w.Lt) return;  // tau = beta is not measured
  }
  int slot = -1;
  for (int k = 0; k < w.dyn_ntau; ++k)
    if (w.dyn_taus[k] == t) slot = k;
  const int N = w.N, L = w.L, S = w.S;
  const long long NN = (long long)N * N;
  const double sg = *w.sign;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  extern __shared__ double dsh[];  // [L] cos(-r kx1), phase 2 also [N] e_i and [N] B_i
  __shared__ double red[8][4], part[4];
  // FourierFactor(r, 1) of the reference's k-star 1 = (2 pi / L, 0) on the site (r, 0)
  const double kx1 = (double)((L + 1) / 2 + 1) / L * 2 * M_PI - M_PI;
  for (int r = threadIdx.x; r < L; r += blockDim.x) dsh[r] = cos(-r * kx1);
  __syncthreads();
  if (slot >= 0) {
    // G(t,t), G(t,0), G(0,t); at tau = 0 the reference's index Lt-1: G(beta,beta), G(beta,0), G(0,beta)
    const int tb = (phase == 2) ? (w.Lt & 1) : (t & 1);
    const double* gtt[2] = {w.G, w.G + (S == 2 ? NN : 0)};
    const double* gt0[2] = {w.gt0 + (long long)tb * S * NN, w.gt0 + ((long long)tb * S + (S == 2)) * NN};
    const double* g0t[2] = {w.g0t + (long long)tb * S * NN, w.g0t + ((long long)tb * S + (S == 2)) * NN};
    // G(k,tau) and the density of states read G(beta,beta) at tau = 0 (Greentt(Lt-1))
    const double* gk[2] = {phase == 2 ? gtt[0] : gt0[0], phase == 2 ? gtt[1] : gt0[1]};
    double v = 0.0, tr = 0.0, cpart = 0.0, rcor = 0.0;
    // cubic lattice: G(k,tau) only; the stiffness is a square-lattice observable
    // (dqmc_initializer.cpp:233-237, measure_methods.cpp:350)
    if (w.dim == 3)
      for (int jj = rank * 8 + wid; jj < N; jj += 8 * kDynCtas)
        for (int i = lane; i < N; i += 32)
          v += w.ff[site_disp(L, 3, i, jj)] * (gk[0][(long long)i * N + jj] + gk[1][(long long)i * N + jj]);
    for (int jj = rank * 8 + wid; jj < N && w.dim == 2; jj += 8 * kDynCtas) {
      const int xj = jj % L, yj = jj / L;
      const int jpx = (xj + 1) % L + L * yj;
      for (int i = lane; i < N; i += 32) {
        const int xi = i % L, yi = i / L;
        int dx = xj - xi, dy = yj - yi;
        dx += (dx < 0) ? L : 0;
        dy += (dy < 0) ? L : 0;
        v += w.ff[dx + dy * L] * (gk[0][(long long)i * N + jj] + gk[1][(long long)i * N + jj]);  // G(jj, i)
        // correlated current-current term of the stiffness (i, jj): measure_methods.cpp:400-407
        const int ipx = (xi + 1) % L + L * yi;
        const double fq = dsh[dx] - dsh[dy];
        double c = 0.0;
        for (int sp = 0; sp < S; ++sp) {
          const double* a = g0t[sp];
          const double* b = gt0[sp];
          c += -a[(long long)jpx * N + ipx] * b[(long long)i * N + jj] + a[(long long)jpx * N + i] * b[(long long)ipx * N + jj] +
               a[(long long)jj * N + ipx] * b[(long long)i * N + jpx] - a[(long long)jj * N + i] * b[(long long)ipx * N + jpx];
        }
        rcor += fq * ((S == 1) ? 2.0 * c : c);
      }
    }
    // per-displacement sums S(r) = sum_i G(i + r, i) (both spins): G(k,tau) = sum_r cos(k r) S(r)
    for (int r = rank * 8 + wid; r < N; r += 8 * kDynCtas) {
      const int rx = r % L, ry = r / L;
      double sr = 0.0;
      for (int i = lane; i < N; i += 32) {
        const int jj = (w.dim == 2) ? (i % L + rx) % L + L * ((i / L + ry) % L) : site_shift(L, 3, i, r);
        sr += gk[0][(long long)i * N + jj] + gk[1][(long long)i * N + jj];
      }
      sr = warp_sum_g(sr);
      if (lane == 0) w.dyn_r[(long long)slot * N + r] += sg * 0.5 * sr / N;
    }
    for (int i = rank * 256 + threadIdx.x; i < N; i += 256 * kDynCtas) {
      const long long d = (long long)i * N + i;
      const int ipx = site_nn(L, i, 0);
      tr += gk[0][d] + gk[1][d];
      cpart += g0t[0][d] * gt0[0][d] + g0t[1][d] * gt0[1][d];
      // parts that wait for G(beta,beta): d_i of the spin susceptibility, A_i of the stiffness
      double* dv = w.dyn_vec + (long long)slot * 2 * N;
      dv[i] = (1.0 - gtt[0][d]) - (1.0 - gtt[1][d]);
      dv[N + i] = (gtt[0][(long long)ipx * N + i] - gtt[0][(long long)i * N + ipx]) +
                  (gtt[1][(long long)ipx * N + i] - gtt[1][(long long)i * N + ipx]);
    }
    v = warp_sum_g(v);
    tr = warp_sum_g(tr);
    cpart = warp_sum_g(cpart);
    rcor = warp_sum_g(rcor);
    if (lane == 0) {
      red[wid][0] = v;
      red[wid][1] = tr;
      red[wid][2] = cpart;
      red[wid][3] = rcor;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
      double s = 0.0;
      for (int k = 0; k < 8; ++k) s += red[k][threadIdx.x];
      part[threadIdx.x] = s;
    }
    cl.sync();  // the parts, and dyn_vec
    if (rank == 0 && threadIdx.x == 0) {
      double tot[4] = {0.0, 0.0, 0.0, 0.0};
      for (int k = 0; k < kDynCtas; ++k)
        for (int m = 0; m < 4; ++m) tot[m] += cl.map_shared_rank(part, k)[m];
      w.dyn_sum[slot] += sg * 0.5 * tot[0] / N;
      w.dyn_cnt[slot] += 1;
      w.dyn_obs[slot * 3 + 0] += sg * 0.5 * tot[1] / N;
      w.dyn_part[slot * 2 + 0] = tot[2];
      w.dyn_part[slot * 2 + 1] = tot[3];
    }
    cl.sync();  // the parts stay until rank 0 has read them
  }
  if (phase != 2) return;
  // end of the half-sweep: g00 = G(beta,beta) completes the spin susceptibility and the
  // uncorrelated stiffness term of every listed tau (measure_methods.cpp:345-461)
  __syncthreads();
  double* e = dsh + L;
  double* B = e + N;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const long long d = (long long)i * N + i;
    const int ipx = site_nn(L, i, 0);
    const double* g0 = w.G;
    const double* g1 = w.G + (S == 2 ? NN : 0);
    e[i] = (1.0 - g0[d]) - (1.0 - g1[d]);
    B[i] = (g0[(long long)ipx * N + i] - g0[(long long)i * N + ipx]) + (g1[(long long)ipx * N + i] - g1[(long long)i * N + ipx]);
  }
  __syncthreads();
  for (int k = rank; k < w.dyn_ntau; k += kDynCtas) {
    const double* dv = w.dyn_vec + (long long)k * 2 * N;
    double ch = 0.0, un = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) ch += dv[i] * e[i];
    for (int jj = wid; jj < N && w.dim == 2; jj += 8) {
      const int xj = jj % L, yj = jj / L;
      for (int i = lane; i < N; i += 32) {
        int dx = xj - i % L, dy = yj - i / L;
        dx += (dx < 0) ? L : 0;
        dy += (dy < 0) ? L : 0;
        un += (dsh[dx] - dsh[dy]) * dv[N + jj] * B[i];
      }
    }
    ch = warp_sum_g(ch);
    un = warp_sum_g(un);
    if (lane == 0) {
      red[wid][0] = ch;
      red[wid][1] = un;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double c2 = 0.0, u2 = 0.0;
      for (int q2 = 0; q2 < 8; ++q2) {
        c2 += red[q2][0];
        u2 += red[q2][1];
      }
      const double n = (double)N;
      w.dyn_obs[k * 3 + 1] += 0.25 * sg / n * (c2 - w.dyn_part[k * 2 + 0]);
      if (w.dim == 2) w.dyn_obs[k * 3 + 2] += 0.25 * w.hop_t * w.hop_t * sg * (w.dyn_part[k * 2 + 1] - u2) / (n * n);
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------------
// host-side launchers for general walkers
// --------------------------------------------------------------------------
static dim3 gemm_grid(int maxN, int nw) {
  const int t = (maxN + kTile - 1) / kTile;
  return dim3(t, t, 2 * nw);
}

void mixed_wrap_fwd(const WalkerDev* W, int nw, int maxN, int j, int q, cudaStream_t st);
void mixed_wrap_bwd(const WalkerDev* W, int nw, int maxN, int j, int q, cudaStream_t st);
void mixed_chain(const WalkerDev* W, int nw, int maxN, int mode, int j, int q, cudaStream_t st);
void mixed_dynamic_prop(const WalkerDev* W, int nw, int maxN, int j, int q, cudaStream_t st);

void launch_metropolis_delayed(const WalkerDev* W, int nw, int mode, int j, int q, int maxN, int S_max, int KD,
                               int tc_flush, cudaStream_t st);
void launch_metropolis_sub64(const WalkerDev* W, int nw, int mode, int j, int q, int maxN, int S_max, cudaStream_t st);
void launch_metropolis_sub(const WalkerDev* W, int nw, int mode, int j, int q, int maxN, int S_max, cudaStream_t st);
void launch_metropolis_sub_split(const WalkerDev* W, int nw, int mode, int j, int q, int maxN, int S_max,
                                 cudaStream_t st);

// One slice of general walkers in three launch groups (timed separately by the
// host): the dense products before the updates (forward wrap), the Metropolis
// updates with the fused measurement, and the products after them (B-chain
// step and backward wrap).
static void launch_kin(const WalkerDev* W, int nw, int maxN, int op, int mode, int j, int q, cudaStream_t st) {
  const int V = kin_lines(maxN);
  kin_op_kernel<<<dim3((maxN + V - 1) / V, 2, nw), 256, 0, st>>>(W, op, mode, j, q);
}

void general_slice_pre(int mode, const WalkerDev* W, int nw, int j, int q, int maxN, bool any_dense, bool any_cb,
                       bool mixed, cudaStream_t st) {
  if (mode != MODE_FWD) return;
  // in a mixed batch the dense products go through the tensor cores (kernels_ozaki.cu)
  if (any_cb || (any_dense && !mixed)) {
    launch_kin(W, nw, maxN, KIN_WL_FWD, mode, j, q, st);
    launch_kin(W, nw, maxN, KIN_WR_FWD, mode, j, q, st);
  }
  if (any_dense && mixed) mixed_wrap_fwd(W, nw, maxN, j, q, st);
}

void general_slice_metro(int mode, const WalkerDev* W, int nw, int j, int q, int maxN, int measure, bool mixed,
                         int kd, int smax, int tc_flush, cudaStream_t st) {
  if (mode == MODE_INIT) return;
  if (!mixed) launch_metropolis_sub64(W, nw, mode, j, q, maxN, smax, st);
  else if (tc_flush == 2) launch_metropolis_sub(W, nw, mode, j, q, maxN, smax, st);
  else if (tc_flush == 3) launch_metropolis_sub_split(W, nw, mode, j, q, maxN, smax, st);
  else launch_metropolis_delayed(W, nw, mode, j, q, maxN, smax, kd, tc_flush, st);
  if (measure) launch_measure_general(W, nw, maxN, mode, j, q, 0, st);
}

void general_slice_post(int mode, const WalkerDev* W, int nw, int j, int q, int maxN, bool any_dense, bool any_cb,
                        bool mixed, cudaStream_t st) {
  const bool kin = any_cb || (any_dense && !mixed), mixed_dense = any_dense && mixed;
  if (kin) launch_kin(W, nw, maxN, mode == MODE_FWD ? KIN_CH_FWD : KIN_CH_BWD, mode, j, q, st);
  if (mixed_dense) mixed_chain(W, nw, maxN, mode, j, q, st);
  if (mode == MODE_BWD) {
    if (kin) {
      launch_kin(W, nw, maxN, KIN_WR_BWD, mode, j, q, st);
      launch_kin(W, nw, maxN, KIN_WL_BWD, mode, j, q, st);
    }
    if (mixed_dense) mixed_wrap_bwd(W, nw, maxN, j, q, st);
  }
}

// One slice of the dynamic half-sweep in three launch groups (timed apart by the host):
// the wrap; the G(t,0) and G(0,t) steps with the G(k,tau) measurement; the B-chain step.
// Dense walkers through the products (on the tensor cores for mixed walkers),
// checkerboard walkers through the plaquette passes.
void general_dynamic_wrap(const WalkerDev* W, int nw, int j, int q, int maxN, bool mixed, bool any_dense,
                          bool any_cb, cudaStream_t st) {
  general_slice_pre(MODE_FWD, W, nw, j, q, maxN, any_dense, any_cb, mixed, st);
}

void general_dynamic_prop(const WalkerDev* W, int nw, int j, int q, int maxN, bool mixed, bool any_dense,
                          bool any_cb, cudaStream_t st) {
  if (any_cb || (any_dense && !mixed)) {
    launch_kin(W, nw, maxN, KIN_DT0, MODE_FWD, j, q, st);
    launch_kin(W, nw, maxN, KIN_D0T, MODE_FWD, j, q, st);
  }
  if (any_dense && mixed) mixed_dynamic_prop(W, nw, maxN, j, q, st);
  dyn_measure_kernel<<<dim3(kDynCtas, nw), 256, sizeof(double) * 32, st>>>(W, j, q, 0);
}

void general_dynamic_chain(const WalkerDev* W, int nw, int j, int q, int maxN, bool mixed, bool any_dense,
                           bool any_cb, cudaStream_t st) {
  general_slice_post(MODE_FWD, W, nw, j, q, maxN, any_dense, any_cb, mixed, st);
}

// stabilization of the dynamic pieces after general_greens of forward step j (walkers
// stabilized by the tensor-core blocked QR get theirs from oz_greens)
void general_dynamic_stab(const WalkerDev* W, int nw, int j, int maxN, cudaStream_t st) {
  const dim3 g = gemm_grid(maxN, nw);
  const int threads = std::min(1024, ((maxN + 31) / 32) * 32);
  dyn_resolve_kernel<<<2 * nw, threads, 0, st>>>(W, j);
  gemm_op_kernel<OP_DT0_OUT><<<g, 256, 0, st>>>(W, MODE_FWD, j, 0, -1);
  gemm_op_kernel<OP_D0T_OUT><<<g, 256, 0, st>>>(W, MODE_FWD, j, 0, -1);
  dyn_boundary_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, j);
}
// G(k,tau) measurement at the stabilization slice of forward step j (after both paths)
void general_dynamic_stab_measure(const WalkerDev* W, int nw, int j, cudaStream_t st) {
  dyn_measure_kernel<<<dim3(kDynCtas, nw), 256, sizeof(double) * 32, st>>>(W, j, 0, 1);
}

void general_dynamic_begin(const WalkerDev* W, int nw, cudaStream_t st) {
  dyn_init_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W);
}
void general_dynamic_end(const WalkerDev* W, int nw, int maxN, cudaStream_t st) {
  dyn_measure_kernel<<<dim3(kDynCtas, nw), 256, sizeof(double) * (32 + 2 * maxN), st>>>(W, 0, 0, 2);
}

void general_chain_init(int mode, const WalkerDev* W, int nw, int j, cudaStream_t st) {
  chain_init_general_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, mode, j);
}

void general_push(int mode, const WalkerDev* W, int nw, int j, int maxN, cudaStream_t st) {
  const int threads = ((maxN + 31) / 32) * 32;
  push_general_kernel<<<2 * nw, threads, sizeof(double) * 5 * maxN + sizeof(int) * maxN, st>>>(W, mode, j);
}

void general_greens(int mode, const WalkerDev* W, int nw, int j, int trace_slot, int maxN, cudaStream_t st) {
  const dim3 g = gemm_grid(maxN, nw);
  // general case needs M from the two GEMMs; boundary cases skip them (kernels exit)
  if (mode != MODE_INIT) {
    gemm_op_kernel<OP_GA><<<g, 256, 0, st>>>(W, mode, j, 0, -1);
    gemm_op_kernel<OP_GB><<<g, 256, 0, st>>>(W, mode, j, 0, -1);
  }
  greens_prep_general_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, mode, j);
  const int threads = std::min(1024, ((maxN + 31) / 32) * 32);
  lu_solve_general_kernel<<<2 * nw, threads, sizeof(double) * maxN, st>>>(W, mode, j);
  if (mode != MODE_INIT) gemm_op_kernel<OP_GG><<<g, 256, 0, st>>>(W, mode, j, 0, trace_slot);
  greens_out_general_kernel<<<dim3(64, 2 * nw), 256, 0, st>>>(W, mode, j, trace_slot);
}

void general_measure_after(int mode, const WalkerDev* W, int nw, int j, int maxN, cudaStream_t st) {
  launch_measure_general(W, nw, maxN, mode, j, 0, 1, st);
}

void general_sign(const WalkerDev* W, int nw, int maxN, cudaStream_t st) {
  sign_general_kernel<<<dim3(2, nw), 512, 3 * sizeof(double) * maxN, st>>>(W);
}

}  // namespace dqmc
