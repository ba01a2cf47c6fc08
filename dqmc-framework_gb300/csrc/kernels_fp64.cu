// kernels_fp64.cu — FP64 plain-method kernels, SMEM-resident (N <= 64).
//
// One CTA owns one walker (segment, measurement, sign) or one (walker, spin)
// (stabilization).  GB300 executes FP64 at a small fraction of its FP32 rate,
// so these kernels are FP64-pipe bound: they keep G in shared memory for a
// whole stabilization segment, avoid redundant FP64 work (the reference's
// per-call MatrixV() re-product, the separate chain x U GEMM of the push) and
// use column-pivoted Householder QR instead of an SVD for the UDV stack.
//
// Reference behaviour restated here:
//   segment_kernel  src/dqmc_walker.cpp:246-325 / 334-412 (wrap, Metropolis,
//                   B-chain), src/dqmc_walker.cpp:173-197 (Metropolis),
//                   src/model/repulsive_hubbard.cpp:112-243 and
//                   src/model/attractive_hubbard.cpp:112-245 (ratio, update, B),
//                   src/checkerboard/square.cpp:66-226 (break-up order),
//                   src/measure/measure_methods.cpp:22-255 (fused measurement).
//   push_kernel     src/svd_stack.cpp:34-61 (stack push; QRP replaces dgesvd).
//   greens_kernel   include/utils/numerical_stable.hpp:34-239 (stable G, wrap error).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "dqmc_device.cuh"

namespace dqmc {

// --------------------------------------------------------------------------
// small helpers
// --------------------------------------------------------------------------
__device__ __forceinline__ double& at(double* m, int ld, int r, int c) { return m[(long long)c * ld + r]; }
__device__ __forceinline__ double at(const double* m, int ld, int r, int c) { return m[(long long)c * ld + r]; }

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block reduction of NV values (all threads call); result valid in thread 0.
template <int NV>
__device__ void block_sum(double (&v)[NV], double* red /* >= NV*8 */) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double s = warp_sum(v[k]);
    if (lane == 0) red[k * 8 + wid] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double s = 0;
      for (int q = 0; q < kThreads / 32; ++q) s += red[k * 8 + q];
      v[k] = s;
    }
  }
  __syncthreads();
}

__device__ double block_max(double v, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_max(v);
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double m = 0;
  for (int q = 0; q < kThreads / 32; ++q) m = fmax(m, red[q]);
  __syncthreads();
  return m;
}

// k / d as (k mul) >> 20 with mul = small_div_mul(d): exact for k d < 2^20 (N <= 64: k < 2 N^2, d <= N)
__device__ __forceinline__ unsigned small_div_mul(int d) { return ((1u << 20) + d - 1) / d; }
__device__ __forceinline__ int small_div(int k, unsigned mul) { return (int)(((unsigned)k * mul) >> 20); }

// spin factor of the B matrices: repulsive couples spin down with -1, attractive +1
__device__ __forceinline__ int spin_sign(const WalkerDev& w, int spin) {
  return (w.model == 0 && spin == 1) ? -1 : 1;
}
// exp(+/- alpha) for the product sgn * s, with the checkerboard products' constant factor folded
// in when fold (inv: of the products with exp(+dtau K))
__device__ __forceinline__ double bdiag(const WalkerDev& w, int sgn_times_s, int inv, bool fold) {
  if (fold) return w.kin_e[inv][sgn_times_s > 0 ? 0 : 1];
  return sgn_times_s > 0 ? w.e_pa : w.e_ma;
}

// --------------------------------------------------------------------------
// Checkerboard passes (src/checkerboard/square.cpp).  A layer of parity p
// mixes the 4 sites {(x,y),(x+1,y),(x,y+1),(x+1,y+1)} of every plaquette with
// corner (x,y), x = p, p+2, ..., y likewise.  Plaquettes of one layer are
// disjoint, so one pass updates the matrix in place.
//   left pass : rows r_a  <- sum_b P[a][b] rows r_b     (optionally pre/post-scaled)
//   right pass: cols c_b  <- sum_a cols c_a P[a][b]
// --------------------------------------------------------------------------
// One layer's pass: rows (left) or, RIGHT, columns of every plaquette; PRE scales the inputs by d
// at their site, POST the outputs
template <bool RIGHT, bool PRE, bool POST, bool PLAIN>
__device__ __forceinline__ void cb_pass(double* M, int ld, int N, int L, int parity, double h, const double* d,
                                        const double* P) {
  const int nq = (L >> 1) * (L >> 1);
  for (int it = threadIdx.x; it < nq * N; it += kThreads) {
    const int q = RIGHT ? it / N : it % nq, x = RIGHT ? it % N : it / nq;
    int idx[4];
    plaq_sites(L, q, parity, idx);
    double v[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      v[a] = RIGHT ? at(M, ld, x, idx[a]) : at(M, ld, idx[a], x);
      if (PRE) v[a] *= d[idx[a]];
    }
    if (PLAIN) plaq_product(v, P);
    else plaq_apply(v, h);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      if (POST) v[a] *= d[idx[a]];
      (RIGHT ? at(M, ld, x, idx[a]) : at(M, ld, idx[a], x)) = v[a];
    }
  }
}

// --------------------------------------------------------------------------
// Block GEMM for N <= 64: out(r,c) = sum_{k >= kbeg} A(r,k) B(k,c).  Output e = r + N c belongs
// to thread e % 256, so a warp holds consecutive rows of one or two columns: A is read along
// rows, B as a broadcast.  An FP64 warp instruction costs 64 cycles, an operand load a few, so
// the mapping spends no FMA on padding (N = 36: 41 warp FMAs per k, 72 with a 48 x 48 register
// tiling) and shares no operands across registers.  The caller-supplied loaders/stores make it
// serve in-place products (SMEM or global: everyone reads before anyone writes).
// --------------------------------------------------------------------------
template <int T, class FA, class FB, class FS>
__device__ __forceinline__ void flat_gemm(int N, int kbeg, FA A, FB B, FS store) {
  const int NN = N * N, w0 = threadIdx.x & ~31;
  double acc[T];
  int r[T], c[T];
#pragma unroll
  for (int u = 0; u < T; ++u) {
    const int e = min((int)threadIdx.x + u * kThreads, NN - 1);
    acc[u] = 0.0;
    r[u] = e % N;
    c[u] = e / N;
  }
#pragma unroll(T == 1 ? 8 : T == 3 ? 4 : 2)
  for (int k = kbeg; k < N; ++k) {
#pragma unroll
    for (int u = 0; u < T; ++u)
      if (w0 + u * kThreads < NN)  // uniform in the warp
        acc[u] = fma(A(r[u], k), B(k, c[u]), acc[u]);
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < T; ++u)
    if ((int)threadIdx.x + u * kThreads < NN) store(r[u], c[u], acc[u]);
  __syncthreads();
}

// The same for 50 < N <= 64: row tid % 64, columns tid / 64 + 4 u, so a thread keeps one row.
template <class FA, class FB, class FS>
__device__ __forceinline__ void row_gemm(int N, int kbeg, FA A, FB B, FS store) {
  constexpr int T = 16;
  const int r = threadIdx.x & 63, c0 = threadIdx.x >> 6;
  double acc[T];
#pragma unroll
  for (int u = 0; u < T; ++u) acc[u] = 0.0;
  if (r < N)
    for (int k = kbeg; k < N; ++k) {
      const double a = A(r, k);
#pragma unroll
      for (int u = 0; u < T; ++u)
        if (c0 + 4 * u < N) acc[u] = fma(a, B(k, c0 + 4 * u), acc[u]);
    }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < T; ++u)
    if (r < N && c0 + 4 * u < N) store(r, c0 + 4 * u, acc[u]);
  __syncthreads();
}

// outputs per thread: 1 up to N = 16, 3 up to 27, 6 up to 39, 10 up to 50, 16 up to 64
template <class FA, class FB, class FS>
__device__ __forceinline__ void block_gemm(int N, FA A, FB B, FS store, int kbeg = 0) {
  if (N <= 16) flat_gemm<1>(N, kbeg, A, B, store);
  else if (N <= 27) flat_gemm<3>(N, kbeg, A, B, store);
  else if (N <= 39) flat_gemm<6>(N, kbeg, A, B, store);
  else if (N <= 50) flat_gemm<10>(N, kbeg, A, B, store);
  else row_gemm(N, kbeg, A, B, store);
}

// --------------------------------------------------------------------------
// B-matrix products for one slice on the nm matrices M, M + ms, ... (leading dimension ld; the
// spins of a walker), in place.  exp(-+dtau K) is applied in its factors: the two plaquette layers
// of a checkerboard walker, else one ring exponential per lattice direction (2 L or 3 L FMAs an
// element instead of N, two or three passes over the matrix).  Each pass writes every element
// from the L elements of its line, M -> tmp and back (tmp: nm matrices, leading dimension ldt).
//   RIGHT 0: M <- post A pre M (rows),  1: M <- M pre A post (columns),  A = exp(-dtau K) or, INV,
//   its inverse; sc: the diagonal, applied first (PRE) or last, of matrix m at sc + m * scs.
//   PLAIN: the plain plaquette product (plaq_product), sc without the constant factor.
// --------------------------------------------------------------------------
template <bool RIGHT, bool INV, bool PRE, bool PLAIN = false>
__device__ __noinline__ void kin_product(const WalkerDev& w, double* M, int ms, int ld, int nm,
                                         double* tmp, int tms, int ldt, const double* sc, int scs,
                                         const double* ring) {
  const int N = w.N, L = w.L, NN = N * N;
  if (w.cb) {
    // B M and M B^-1: layer B (parity 1) then A; B^T M, M B and B^-1 M: A then B
    for (int m = 0; m < nm; ++m) {
      double* X = M + (long long)m * ms;
      const double* d = sc + m * scs;
      const double h = INV ? -w.cb_h : w.cb_h;
      const int p0 = PRE ? 0 : 1;
      cb_pass<RIGHT, PRE, false, PLAIN>(X, ld, N, L, p0, h, d, w.cbP);
      __syncthreads();
      cb_pass<RIGHT, false, !PRE, PLAIN>(X, ld, N, L, p0 ^ 1, h, d, w.cbP);
      __syncthreads();
    }
    return;
  }
  const double* e = ring + (INV ? L : 0);
  const unsigned dN = small_div_mul(N), dL = small_div_mul(L);
  // element k: matrix m, row r, column c
  auto split = [&](int k, int& m, int& r, int& c) {
    m = (k >= NN) ? 1 : 0;
    c = small_div(k - m * NN, dN);
    r = k - m * NN - c * N;
  };
  if (PRE) {
    for (int k = threadIdx.x; k < nm * NN; k += kThreads) {
      int m, r, c;
      split(k, m, r, c);
      M[(long long)m * ms + c * ld + r] *= sc[m * scs + (RIGHT ? c : r)];
    }
    __syncthreads();
  }
  const double* in = M;
  double* out = tmp;
  int ims = ms, ild = ld, oms = tms, old = ldt;
  for (int d = 0, st = 1; d < w.dim; ++d, st *= L) {
    const bool last = d == w.dim - 1;
    const int step = RIGHT ? st * ild : st;
    for (int k = threadIdx.x; k < nm * NN; k += kThreads) {
      int m, r, c;
      split(k, m, r, c);
      const int site = RIGHT ? c : r;
      int x = site;
      for (int a = 0; a < d; ++a) x = small_div(x, dL);
      x -= L * small_div(x, dL);
      const double* p = in + (long long)m * ims + c * ild + r - x * step;
      double acc = 0.0;
      for (int y = 0; y < L; ++y) acc = fma(e[abs(x - y)], p[y * step], acc);
      if (last && !PRE) acc *= sc[m * scs + site];
      out[(long long)m * oms + c * old + r] = acc;
    }
    __syncthreads();
    in = out;
    out = (in == tmp) ? M : tmp;
    ims = (in == tmp) ? tms : ms;
    ild = (in == tmp) ? ldt : ld;
    oms = (in == tmp) ? ms : tms;
    old = (in == tmp) ? ld : ldt;
  }
  if (in == tmp) {  // three directions: back to M
    for (int k = threadIdx.x; k < nm * NN; k += kThreads) {
      int m, r, c;
      split(k, m, r, c);
      M[(long long)m * ms + c * ld + r] = tmp[(long long)m * tms + c * ldt + r];
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------------
// Fused equal-time measurement (measure_methods.cpp:22-255), split in two: measure_slice adds
// one slice's sums into each thread's accumulators, measure_close reduces them over the CTA and
// adds them to the walker's observables, once per launch.  The reduction of 8 FP64 values
// costs a warp 40 adds of 64 cycles and thread 0 its divisions, more than a slice's sums at
// small N.  Unordered pairs {i, j} are visited once (lanes over i, j = i + d mod N), with
// X = G_ij G_ji summed over spins and the site's sums and differences of 1 - G_ii: 14 FP64
// operations per pair against 13 per ordered pair for the sums written out.
// gu/gd in shared memory (ld), sg the recorded sign of the slice.
// --------------------------------------------------------------------------
struct MeasureAcc {
  // sign * sums: 0 trace, 1 double occupancy, 2 local spin, 3 kinetic, 4 n(k), 5 spin and
  // 6 charge structure factor, 7 s-wave pairing; all times sg
  double v[8];
  double sg;      // the common factor, +1 or -1
  double sign_sum;
  int slices;
};

__device__ __forceinline__ void measure_open(MeasureAcc& m) {
#pragma unroll
  for (int k = 0; k < 8; ++k) m.v[k] = 0.0;
  m.sg = 1.0;
  m.sign_sum = 0.0;
  m.slices = 0;
}

// scratch: 3N doubles
__device__ void measure_slice(const WalkerDev& w, const double* gu, const double* gd, int ld, double sg,
                              double* scratch, MeasureAcc& m) {
  const int N = w.N, L = w.L, LL = L * L;
  double* ssum = scratch;       // (1 - gu_ii) + (1 - gd_ii)
  double* sdif = scratch + N;   // (1 - gu_ii) - (1 - gd_ii)
  double* ff = scratch + 2 * N;
  __shared__ signed char s_x[kMaxSmemN], s_y[kMaxSmemN], s_z[kMaxSmemN];
  if (sg != m.sg) {
#pragma unroll
    for (int k = 0; k < 8; ++k) m.v[k] = -m.v[k];
    m.sg = sg;
  }
  m.sign_sum += sg;
  ++m.slices;
  // one warp per 32 sites for the site sums
  for (int i = threadIdx.x; i < N; i += kThreads) {
    const double a = at(gu, ld, i, i), b = at(gd, ld, i, i);
    const double du = 1.0 - a, dd = 1.0 - b, ab = a + b, n = du + dd, q = du - dd;
    ssum[i] = n;
    sdif[i] = q;
    ff[i] = w.ff[i];
    s_x[i] = (signed char)(i % L);
    s_y[i] = (signed char)((i / L) % L);
    s_z[i] = (signed char)(i / LL);  // 0 on the square lattice
    m.v[0] += ab;
    m.v[1] = fma(du, dd, m.v[1]);
    m.v[2] += fma(-2.0 * a, b, ab);
    // bonds to the +x, +y (, +z) neighbours (measure_methods.cpp:87-95)
    const int jx = site_nn(L, i, 0), jy = site_nn(L, i, 1);
    double kin = at(gu, ld, i, jx) + at(gd, ld, i, jx) + at(gu, ld, i, jy) + at(gd, ld, i, jy);
    if (w.dim == 3) {
      const int jz = site_nn(L, i, 2);
      kin += at(gu, ld, i, jz) + at(gd, ld, i, jz);
    }
    m.v[3] += kin;
    // the pair i = j (Fourier factor 1)
    const double x = fma(du, a, dd * b);
    m.v[4] += ab;
    m.v[5] += fma(q, q, x);
    m.v[6] += fma(n, n, x);
    m.v[7] = fma(du, dd, m.v[7]);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double p4 = 0.0, p5 = 0.0, p6 = 0.0;
  for (int d = 1 + wid; 2 * d <= N; d += kThreads / 32)
    for (int i = lane; i < ((2 * d == N) ? d : N); i += 32) {
      const int j = (i + d < N) ? i + d : i + d - N;
      // both displacements: on odd sides the momentum pi is not the lattice's and the table not even
      const int dx = s_x[j] - s_x[i], dy = s_y[j] - s_y[i], dz = s_z[j] - s_z[i];
      const double f_ij = ff[(dx + (dx < 0 ? L : 0)) + (dy + (dy < 0 ? L : 0)) * L + (dz + (dz < 0 ? L : 0)) * LL];
      const double f_ji = ff[(-dx + (dx > 0 ? L : 0)) + (-dy + (dy > 0 ? L : 0)) * L + (-dz + (dz > 0 ? L : 0)) * LL];
      const double f = f_ij + f_ji;
      const double gu_ij = at(gu, ld, i, j), gu_ji = at(gu, ld, j, i);
      const double gd_ij = at(gd, ld, i, j), gd_ji = at(gd, ld, j, i);
      const double x = fma(gd_ij, gd_ji, gu_ij * gu_ji);
      p4 = fma(f_ij, gu_ji + gd_ji, p4);
      p4 = fma(f_ji, gu_ij + gd_ij, p4);
      p5 = fma(f, fma(sdif[i], sdif[j], -x), p5);
      p6 = fma(f, fma(ssum[i], ssum[j], -x), p6);
      m.v[7] = fma(gu_ij, gd_ij, m.v[7]);
      m.v[7] = fma(gu_ji, gd_ji, m.v[7]);
    }
  m.v[4] += p4;
  m.v[5] += p5;
  m.v[6] += p6;
  __syncthreads();
}

__device__ void measure_close(const WalkerDev& w, MeasureAcc& m, double* red) {
  block_sum<8>(m.v, red);
  if (threadIdx.x == 0 && m.slices) {
    const double n = (double)w.N, sn = m.sg / n, snn = sn / n;
    double* o = w.obs;
    o[0] += 2.0 * m.sign_sum - m.v[0] * sn;
    o[1] += m.v[1] * sn;
    o[2] += (2.0 * w.hop_t) * (m.v[3] * sn);
    o[3] += m.sign_sum - 0.5 * (m.v[4] * sn);
    o[4] += m.v[2] * sn;
    o[5] += m.v[5] * snn;
    o[6] += m.v[6] * snn;
    o[7] += m.v[7] * sn;
    o[8] += m.sign_sum;
    for (int k = 0; k < kNumObs; ++k) w.obs_cnt[k] += m.slices;
  }
  __syncthreads();
}

// --------------------------------------------------------------------------
// shared memory of the segment kernel with the chain beside G: two CTAs still share an SM up to N = 50
__host__ __device__ inline bool segment_chain_smem(int maxN) { return maxN <= 50; }
// and the products take both spins' matrices in one pass up to N = 36 (64 KB of shared memory)
__host__ __device__ inline bool segment_joint_spins(int maxN) { return maxN <= 36; }

// --------------------------------------------------------------------------
// Segment kernel: the slices of one stabilization interval for one walker.
//   MODE_FWD: for t up:   wrap into t, Metropolis(t), measure, chain <- B(t) chain
//   MODE_BWD: for t down: Metropolis(t), measure, chain <- B(t)^T chain, wrap out of t
//   MODE_INIT: chain <- B(t)^T chain only (initial_svd_stacks)
// The chain starts from U_top diag(D_top) of the stack being pushed (or I), so
// the push needs no separate (chain x U) product: B_p..B_1 (U D) = ((B_p..B_1) U) D
// column by column, the scale-separated order svd_stack.cpp:51 asks for.
// --------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kThreads, 2) segment_kernel(const WalkerDev* __restrict__ W, int j, int measure,
                                                           int maxN) {
  const WalkerDev& w = W[blockIdx.x];
  if (j >= w.nstack || w.path != 0) return;
  extern __shared__ double smem[];
  const int N = w.N, ld = N + 1, S = w.S, Lt = w.Lt, p = w.pace;
  double* Gs[2];
  Gs[0] = smem;
  Gs[1] = (S == 2) ? smem + (long long)N * ld : smem;
  double* vec = smem + (long long)S * N * ld;  // ucol[2][N], wrow[2][N]
  double* dtab = vec + 4 * N;                   // [2 spins][2 (pos,neg)][N]
  double* red = dtab + 4 * N;                   // 64
  double* scratch = red + 64;                   // 3N
  // the running chain lives beside G in shared memory where that leaves room for two CTAs an SM
  const bool chain_smem = segment_chain_smem(maxN);
  double* Cs = scratch + 3 * N;
  const int ldc = chain_smem ? ld : N;
  // the products' second buffer, for both spins at once where small walkers need the parallelism
  double* tmp = Cs + (chain_smem ? (long long)S * N * ld : 0);
  const int nm = (segment_joint_spins(maxN)) ? S : 1;
  __shared__ double ring[2 * 8];
  __shared__ int s_next;
  __shared__ double s_f[2], s_sign;
  __shared__ int8_t s_field[kMaxSmemN];
  __shared__ double s_uni[kMaxSmemN];

  const int k = (MODE == MODE_FWD) ? j : (w.nstack - 1 - j);
  const int t_lo = k * p + 1, t_hi = min((k + 1) * p, Lt);
  const int side = (MODE == MODE_FWD) ? 0 : 1;

  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int nwarp = kThreads / 32;
  if (!w.cb && threadIdx.x < 2 * w.L) ring[threadIdx.x] = w.kin[threadIdx.x];
  // chain <- U_top diag(D_top)  or  I
  for (int sp = 0; sp < S; ++sp) {
    double* C = chain_smem ? Cs + (long long)sp * N * ld : w.chain + (long long)sp * N * N;
    const double* lv = (j == 0) ? nullptr : stack_level(w, side, sp, j - 1);
    for (int c = wid; c < N; c += nwarp) {
      const double dc = lv ? lv[2LL * N * N + c] : 1.0;
      for (int r = lane; r < N; r += 32)
        C[(long long)c * ldc + r] = lv ? lv[(long long)c * N + r] * dc : ((r == c) ? 1.0 : 0.0);
    }
  }
  if (MODE != MODE_INIT) {
    for (int sp = 0; sp < S; ++sp) {
      const double* Gg = w.G + (long long)sp * N * N;
      for (int c = wid; c < N; c += nwarp)
        for (int r = lane; r < N; r += 32) at(Gs[sp], ld, r, c) = Gg[(long long)c * N + r];
    }
  }
  __syncthreads();

  double sign = *w.sign;  // warp 0 keeps it current
  long long acc_count = 0;
  const unsigned long long sweep = (w.rng == 1) ? *w.sweep_ctr : 0ULL;
  const int nsl = t_hi - t_lo + 1;
  MeasureAcc meas;
  measure_open(meas);
  const SiteScan scan(w, lane);
  for (int q = 0; q < nsl; ++q) {
    const int t = (MODE == MODE_FWD) ? t_lo + q : t_hi - q;
    const int eff = t - 1;  // 1 <= t <= Lt
    const int8_t* frow = w.fields + (long long)eff * N;
    for (int i = threadIdx.x; i < N; i += kThreads) {
      s_field[i] = frow[i];
      if (MODE != MODE_INIT)
        s_uni[i] = (w.rng == 0) ? w.uni[(MODE == MODE_FWD) ? (eff * N + i) : ((Lt - t) * N + i)]
                                : philox_uniform(w.seed, (unsigned)w.widx, sweep, (unsigned)(eff * N + i));
    }
    __syncthreads();
    // scale tables for this slice: dtab[sp][0][i] = e^{+sa s_i}, dtab[sp][1][i] = e^{-sa s_i}
    for (int e = threadIdx.x; e < S * N; e += kThreads) {
      const int sp = e / N, i = e % N;
      const int ss = spin_sign(w, sp) * (int)s_field[i];
      dtab[(sp * 2 + 0) * N + i] = bdiag(w, ss, 0, MODE != MODE_INIT || !w.cb);
      dtab[(sp * 2 + 1) * N + i] = bdiag(w, -ss, 1, MODE != MODE_INIT || !w.cb);
    }
    __syncthreads();

    if (MODE == MODE_FWD) {  // wrap_from_0_to_beta(t-1): G <- B(t) G B(t)^-1
      for (int sp = 0; sp < S; sp += nm) {
        kin_product<false, false, false>(w, Gs[sp], N * ld, ld, nm, tmp, N * ld, ld, dtab + sp * 2 * N, 2 * N, ring);
        kin_product<true, true, false>(w, Gs[sp], N * ld, ld, nm, tmp, N * ld, ld, dtab + (sp * 2 + 1) * N, 2 * N,
                    ring);
      }
    }

    if (MODE != MODE_INIT) {
      // Metropolis over sites i = 0..N-1 (dqmc_walker.cpp:173-197), two barriers per accept.
      // After the first, warps 1 .. 2S form the update's vectors u = f G(:, i) and
      // w = e_i - G(i, :)^T and warp 0 reads the diagonal as it stands; after the second,
      // warp 0 scans the sites past i for the next accept while warps 1 .. 7 apply the rank-1
      // update.  The scan uses the diagonal that the pending update will produce, computed with
      // the same fma the update uses (bit-identical).
      double dg[4];  // windows of 16 sites that cover N <= 64
      const double* su = vec + scan.sp * N;
      const double* sw = vec + (2 + scan.sp) * N;
      if (wid == 0) {
        const int nx = scan.next<4>(w, [&](int, int l) { return at(Gs[scan.sp], ld, l, l); }, 0, N, s_uni, s_field, s_f,
                                    sign, acc_count);
        if (lane == 0) s_next = nx;
      }
      __syncthreads();
      while (true) {
        const int i = s_next;
        if (i >= N) break;
        if (wid == 0) {
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int l = i + 1 + b * scan.width + scan.dl;
            dg[b] = (l < N) ? at(Gs[scan.sp], ld, l, l) : 0.0;
          }
        } else if (wid <= 2 * S) {
          const int sp = (wid - 1) % S, role = (wid - 1) / S;
          const double* g = Gs[sp];
          double* o = vec + (2 * role + sp) * N;
          const double f = s_f[sp];
          for (int r = lane; r < N; r += 32)
            o[r] = role ? ((r == i) ? 1.0 : 0.0) - at(g, ld, i, r)  // e_i - G(i,:)
                        : f * at(g, ld, r, i);                      // f u
        }
        __syncthreads();
        if (wid == 0) {
          const int nx = scan.next<4>(w, [&](int b, int l) { return fma(-sw[l], su[l], dg[b]); }, i + 1, N, s_uni,
                                      s_field, s_f, sign, acc_count);
          if (lane == 0) s_next = nx;
        } else {
          // warps 1..7: the S N columns in turn, rows lane and lane + 32 (N <= 16: two columns
          // at a time, 16 lanes each)
          const int per = (N <= 16) ? 2 : 1;
          const int sub = (per == 2) ? lane >> 4 : 0, r0 = (per == 2) ? lane & 15 : lane, r1 = lane + 32;
          for (int qc = (wid - 1) * per + sub; qc < S * N; qc += per * (nwarp - 1)) {
            const int sp = (qc >= N) ? 1 : 0, c = qc - sp * N;
            double* g = Gs[sp];
            const double* u = vec + sp * N;
            const double wc = -vec[(2 + sp) * N + c];
            if (r0 < N) at(g, ld, r0, c) = fma(wc, u[r0], at(g, ld, r0, c));
            if (per == 1 && r1 < N) at(g, ld, r1, c) = fma(wc, u[r1], at(g, ld, r1, c));
          }
        }
        __syncthreads();
      }
      if (threadIdx.x == 0) s_sign = sign;
      // write back the flipped fields of this slice
      int8_t* frw = w.fields + (long long)eff * N;
      for (int i = threadIdx.x; i < N; i += kThreads) frw[i] = s_field[i];
      // the slice's B matrices below use the updated fields
      for (int e = threadIdx.x; e < S * N; e += kThreads) {
        const int sp = e / N, i = e % N;
        const int ss = spin_sign(w, sp) * (int)s_field[i];
        dtab[(sp * 2 + 0) * N + i] = bdiag(w, ss, 0, MODE != MODE_INIT || !w.cb);
        dtab[(sp * 2 + 1) * N + i] = bdiag(w, -ss, 1, MODE != MODE_INIT || !w.cb);
      }
      __syncthreads();

      // equal-time measurement of slot t-1 (the slot closing a forward
      // segment and slot Lt-1 of the backward sweep are measured after
      // their stabilization, dqmc_walker.cpp:307-310 and :408-411)
      if (measure) {
        const bool here = (MODE == MODE_FWD) ? (t != t_hi) : (t != Lt);
        if (here) measure_slice(w, Gs[0], Gs[1], ld, s_sign, scratch, meas);
      }
      if (MODE == MODE_BWD && t == Lt && threadIdx.x == 0) *w.sign_Lt = sign;
    }

    // B-chain of the stabilization interval
    for (int sp = 0; sp < S; sp += nm) {
      double* C = chain_smem ? Cs + (long long)sp * N * ld : w.chain + (long long)sp * N * N;
      if (MODE == MODE_FWD) {
        kin_product<false, false, false>(w, C, N * ldc, ldc, nm, tmp, N * ld, ld, dtab + sp * 2 * N, 2 * N, ring);
      } else {
        // B^T: the plaquette layers in the order of the inverse's left product
        kin_product<false, false, true, MODE == MODE_INIT>(w, C, N * ldc, ldc, nm, tmp, N * ld, ld, dtab + sp * 2 * N, 2 * N, ring);
      }
    }

    if (MODE == MODE_BWD) {  // wrap_from_beta_to_0(t): G <- B(t)^-1 G B(t)
      for (int sp = 0; sp < S; sp += nm) {
        kin_product<true, false, true>(w, Gs[sp], N * ld, ld, nm, tmp, N * ld, ld, dtab + sp * 2 * N, 2 * N, ring);
        kin_product<false, true, true>(w, Gs[sp], N * ld, ld, nm, tmp, N * ld, ld, dtab + (sp * 2 + 1) * N, 2 * N,
                    ring);
      }
    }
    __syncthreads();
  }

  if (chain_smem)
    for (int sp = 0; sp < S; ++sp) {
      double* C = w.chain + (long long)sp * N * N;
      for (int c = wid; c < N; c += nwarp)
        for (int r = lane; r < N; r += 32) C[(long long)c * N + r] = at(Cs + (long long)sp * N * ld, ld, r, c);
    }
  if (MODE != MODE_INIT) {
    for (int sp = 0; sp < S; ++sp) {
      double* Gg = w.G + (long long)sp * N * N;
      for (int c = wid; c < N; c += nwarp)
        for (int r = lane; r < N; r += 32) Gg[(long long)c * N + r] = at(Gs[sp], ld, r, c);
    }
    if (measure) measure_close(w, meas, red);
    if (threadIdx.x == 0) {
      *w.sign = sign;
      *w.accepts += acc_count;
    }
  }
}

// --------------------------------------------------------------------------
// Stack push (svd_stack.cpp:34-61 with QRP for the SVD):
//   X = chain (= B_p..B_1 U_top D_top), X P = Q R,
//   U = Q, D = |diag R|, F_new = (D^-1 R P^T) F_prev.
// One CTA of kPushThreads per (walker, spin); thread j owns column j.  GB300
// issues an FP64 warp instruction every ~64 cycles per SM sub-partition, so
// the kernel avoids FP64 shuffle reductions in the O(N^3) parts: every dot
// product runs down one thread's own column.  Q is formed in place from the
// reflectors (LAPACK dorg2r order), so one N x N tile of SMEM suffices.
// --------------------------------------------------------------------------
constexpr int kPushThreads = 64;

// argmax of non-negative key over threads (ties -> lowest index); all threads get it
__device__ __forceinline__ int block64_argmax(double v, int idx, bool valid, int* s_i, long long* s_k) {
  long long key = valid ? __double_as_longlong(v) : -1LL;  // non-negative doubles order as integers
  int bi = idx;
  for (int o = 16; o > 0; o >>= 1) {
    const long long ok = __shfl_xor_sync(0xffffffffu, key, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ok > key || (ok == key && oi < bi)) { key = ok; bi = oi; }
  }
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { s_k[wid] = key; s_i[wid] = bi; }
  __syncthreads();
  int best = s_i[0];
  long long bk = s_k[0];
  for (int q = 1; q < kPushThreads / 32; ++q)
    if (s_k[q] > bk || (s_k[q] == bk && s_i[q] < best)) { bk = s_k[q]; best = s_i[q]; }
  __syncthreads();
  return best;
}

__device__ __forceinline__ double block64_sum(double v, double* s_d) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) s_d[wid] = v;
  __syncthreads();
  double t = 0;
  for (int q = 0; q < kPushThreads / 32; ++q) t += s_d[q];
  __syncthreads();
  return t;
}

// x . y over r0 <= r < n in two alternating chains from a0, and y += f x, four rows' loads ahead of
// their FMAs: a thread walks its own column, so a load that waits for the previous store is latency
__device__ __forceinline__ double push_dot(const double* x, const double* y, int r, int n, double a0) {
  double a1 = 0.0;
  for (; r + 3 < n; r += 4) {
    const double x0 = x[r], x1 = x[r + 1], x2 = x[r + 2], x3 = x[r + 3];
    const double y0 = y[r], y1 = y[r + 1], y2 = y[r + 2], y3 = y[r + 3];
    a0 = fma(x0, y0, a0);
    a1 = fma(x1, y1, a1);
    a0 = fma(x2, y2, a0);
    a1 = fma(x3, y3, a1);
  }
  for (; r + 1 < n; r += 2) {
    a0 = fma(x[r], y[r], a0);
    a1 = fma(x[r + 1], y[r + 1], a1);
  }
  if (r < n) a0 = fma(x[r], y[r], a0);
  return a0 + a1;
}
__device__ __forceinline__ void push_axpy(const double* x, double* y, int r, int n, double f) {
  for (; r + 3 < n; r += 4) {
    const double x0 = x[r], x1 = x[r + 1], x2 = x[r + 2], x3 = x[r + 3];
    const double y0 = y[r], y1 = y[r + 1], y2 = y[r + 2], y3 = y[r + 3];
    y[r] = fma(f, x0, y0);
    y[r + 1] = fma(f, x1, y1);
    y[r + 2] = fma(f, x2, y2);
    y[r + 3] = fma(f, x3, y3);
  }
  for (; r < n; ++r) y[r] = fma(f, x[r], y[r]);
}

template <int MODE>
__global__ void __launch_bounds__(kPushThreads) push_kernel(const WalkerDev* __restrict__ W, int j) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (j >= w.nstack || sp >= w.S || w.path != 0) return;
  extern __shared__ double smem[];
  const int N = w.N, ld = N + 1;
  const int side = (MODE == MODE_FWD) ? 0 : 1;
  double* X = smem;
  double* vn1 = X + (long long)N * ld;
  double* vn2 = vn1 + N;
  double* tau = vn2 + N;
  double* invd = tau + N;
  int* perm = (int*)(invd + N);
  __shared__ int s_i[kPushThreads / 32];
  __shared__ long long s_k[kPushThreads / 32];
  __shared__ double s_d[kPushThreads / 32];
  __shared__ double s_tau, s_scal, s_beta;
  const int tj = threadIdx.x;  // column / row owned by this thread
  const bool own = tj < N;

  const double* C = w.chain + (long long)sp * N * N;
  for (int c = 0; c < N; ++c)
    if (own) at(X, ld, tj, c) = C[(long long)c * N + tj];
  __syncthreads();
  if (own) {
    double s0 = 0, s1 = 0;
    int r = 0;
    for (; r + 1 < N; r += 2) {
      const double a = at(X, ld, r, tj), b = at(X, ld, r + 1, tj);
      s0 = fma(a, a, s0);
      s1 = fma(b, b, s1);
    }
    if (r < N) s0 = fma(at(X, ld, r, tj), at(X, ld, r, tj), s0);
    vn1[tj] = vn2[tj] = sqrt(s0 + s1);
    perm[tj] = tj;
  }
  __syncthreads();

  const double tol3z = 1.4901161193847656e-08;  // sqrt(eps), LAPACK dlaqp2
  for (int k = 0; k < N; ++k) {
    // ---- pivot: largest remaining column norm
    const int pv = block64_argmax(own ? vn1[tj] : 0.0, tj, own && tj >= k, s_i, s_k);
    if (pv != k) {
      if (own) {
        const double a = at(X, ld, tj, k);
        at(X, ld, tj, k) = at(X, ld, tj, pv);
        at(X, ld, tj, pv) = a;
      }
      if (tj == 0) {
        const int tp = perm[k]; perm[k] = perm[pv]; perm[pv] = tp;
        double tv = vn1[k]; vn1[k] = vn1[pv]; vn1[pv] = tv;
        tv = vn2[k]; vn2[k] = vn2[pv]; vn2[pv] = tv;
      }
      __syncthreads();
    }
    // ---- Householder reflector of X[k:,k]: row r > k held by thread r
    const double xr = (own && tj > k) ? at(X, ld, tj, k) : 0.0;
    const double xnorm2 = block64_sum(xr * xr, s_d);
    if (tj < 2) {  // lane 0: tau = (beta - alpha) / beta, lane 1: scale = 1 / (alpha - beta)
      const double alpha = at(X, ld, k, k);
      double q = (tj == 0) ? 0.0 : 1.0, beta = alpha;
      if (xnorm2 != 0.0) {
        const double nrm = sqrt(alpha * alpha + xnorm2);
        beta = alpha >= 0 ? -nrm : nrm;
        q = (tj == 0 ? beta - alpha : 1.0) / (tj == 0 ? beta : alpha - beta);
      }
      if (tj == 0) { s_tau = q; s_beta = beta; tau[k] = q; }
      else s_scal = q;
    }
    __syncthreads();
    if (own && tj > k) at(X, ld, tj, k) *= s_scal;
    if (tj == 0) at(X, ld, k, k) = s_beta;
    __syncthreads();
    // ---- trailing update of column tj > k, then its norm downdate
    const double tk = s_tau;
    if (own && tj > k && tk != 0.0) {
      const double* xk = X + k * ld;
      double* xj = X + tj * ld;
      const double wv = push_dot(xk, xj, k + 1, N, xj[k]) * tk;
      xj[k] -= wv;
      push_axpy(xk, xj, k + 1, N, -wv);
    }
    if (own && tj > k) {
      const double v1 = vn1[tj];
      if (v1 != 0.0) {
        double tmp = fabs(at(X, ld, k, tj)) / v1;
        tmp = fmax(0.0, 1.0 - tmp * tmp);
        const double r2 = v1 / vn2[tj];
        if (tmp * r2 * r2 <= tol3z) {
          double q0 = 0, q1 = 0;
          int r = k + 1;
          for (; r + 1 < N; r += 2) {
            q0 = fma(at(X, ld, r, tj), at(X, ld, r, tj), q0);
            q1 = fma(at(X, ld, r + 1, tj), at(X, ld, r + 1, tj), q1);
          }
          if (r < N) q0 = fma(at(X, ld, r, tj), at(X, ld, r, tj), q0);
          vn1[tj] = vn2[tj] = sqrt(q0 + q1);
        } else {
          vn1[tj] = v1 * sqrt(tmp);
        }
      }
    }
    __syncthreads();
  }

  // ---- D = |diag R| and the right factor F = (D^-1 R P^T) F_prev
  double* lv = stack_level(w, side, sp, j);
  double* Uo = lv;
  double* Fo = lv + (long long)N * N;
  double* Do = lv + 2LL * N * N;
  if (own) {
    const double d = fabs(at(X, ld, tj, tj));
    Do[tj] = d;
    invd[tj] = (d != 0.0) ? 1.0 / d : 0.0;
    if (d == 0.0 || !isfinite(d)) atomicOr(w.status, ST_SINGULAR);
  }
  __syncthreads();
  if (j == 0) {
    // F = T: column perm[c] of T holds R(:,c)/D for rows i <= c
    if (own) {
      const int c = tj;
      double* fc = Fo + (long long)perm[c] * N;
      for (int i = 0; i < N; ++i) fc[i] = (i <= c) ? at(X, ld, i, c) * invd[i] : 0.0;
    }
  } else if (own) {
    // thread c: F_new(i,c) = sum_{k>=i} (R(i,k)/D(i)) F_prev(perm[k], c)
    const int c = tj;
    const double* fp = stack_level(w, side, sp, j - 1) + (long long)N * N + (long long)c * N;
    double* fo = Fo + (long long)c * N;
    for (int i = 0; i < N; ++i) {
      double a0 = 0.0, a1 = 0.0;
      int k = i;
      for (; k + 3 < N; k += 4) {  // four terms' loads ahead of their FMAs
        const double f0 = __ldg(fp + perm[k]), f1 = __ldg(fp + perm[k + 1]);
        const double f2 = __ldg(fp + perm[k + 2]), f3 = __ldg(fp + perm[k + 3]);
        const double x0 = at(X, ld, i, k), x1 = at(X, ld, i, k + 1);
        const double x2 = at(X, ld, i, k + 2), x3 = at(X, ld, i, k + 3);
        a0 = fma(x0, f0, a0);
        a1 = fma(x1, f1, a1);
        a0 = fma(x2, f2, a0);
        a1 = fma(x3, f3, a1);
      }
      for (; k + 1 < N; k += 2) {
        a0 = fma(at(X, ld, i, k), __ldg(fp + perm[k]), a0);
        a1 = fma(at(X, ld, i, k + 1), __ldg(fp + perm[k + 1]), a1);
      }
      if (k < N) a0 = fma(at(X, ld, i, k), __ldg(fp + perm[k]), a0);
      fo[i] = (a0 + a1) * invd[i];
    }
  }
  __syncthreads();

  // ---- Q = H_0 H_1 ... H_{N-1}, formed in place (dorg2r order)
  for (int i = N - 1; i >= 0; --i) {
    const double ti = tau[i];
    if (i < N - 1 && own && tj > i) {
      // apply H_i to column tj (rows i..N-1), v = [1; X(i+1:,i)]
      const double* xi = X + i * ld;
      double* xj = X + tj * ld;
      const double wv = push_dot(xi, xj, i + 1, N, xj[i]) * ti;
      xj[i] -= wv;
      push_axpy(xi, xj, i + 1, N, -wv);
    }
    __syncthreads();
    if (own) {  // column i of Q: thread tj handles row tj
      const int r = tj;
      if (r > i) at(X, ld, r, i) *= -ti;
      else if (r == i) at(X, ld, r, i) = 1.0 - ti;
      else at(X, ld, r, i) = 0.0;
    }
    __syncthreads();
  }
  for (int c = 0; c < N; ++c)
    if (own) Uo[(long long)c * N + tj] = at(X, ld, tj, c);
}

// --------------------------------------------------------------------------
// In-SMEM LU with partial pivoting of M, applied on the fly to the right-hand
// sides Y (forward substitution fused), then back substitution: Y <- M^-1 Y.
// Returns false if a zero pivot was met.  Warp 0 finds a pivot by the bits of
// its magnitude and forms its reciprocal once, for the multipliers and for the
// back substitution: a division in every warp was a fifth of the kernel's FP64
// operations at N = 64.
// --------------------------------------------------------------------------
__device__ bool lu_solve_smem(double* M, double* Y, int N, int ld) {
  __shared__ int s_p;
  __shared__ int s_bad;
  __shared__ double s_inv[kMaxSmemN];  // 1 / pivot
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_bad = 0;
  for (int k = 0; k < N; ++k) {
    if (wid == 0) {
      long long best = -1;
      int bi = k;
      for (int r = k + lane; r < N; r += 32) {
        const long long a = __double_as_longlong(at(M, ld, r, k)) & 0x7fffffffffffffffLL;
        if (a > best && a <= 0x7ff0000000000000LL) { best = a; bi = r; }  // a NaN is never the largest
      }
      for (int o = 16; o > 0; o >>= 1) {
        const long long ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      const double inv = 1.0 / at(M, ld, bi, k);
      if (lane == 0) { s_p = bi; s_inv[k] = inv; if (best == 0) s_bad = 1; }
    }
    __syncthreads();
    const int pr = s_p;
    if (wid == 1) {  // column k: the exchange and the multipliers
      const double piv = at(M, ld, pr, k), top = at(M, ld, k, k), inv = (piv != 0.0) ? s_inv[k] : 0.0;
      __syncwarp();
      if (lane == 0) at(M, ld, k, k) = piv;
      for (int r = k + 1 + lane; r < N; r += 32) at(M, ld, r, k) = ((r == pr) ? top : at(M, ld, r, k)) * inv;
    } else if (pr != k) {
      for (int c = (wid == 0) ? lane : threadIdx.x - 32; c < 2 * N; c += kThreads - 32) {
        if (c == k) continue;
        double* m = (c < N) ? M : Y;
        const int cc = (c < N) ? c : c - N;
        const double tmp = at(m, ld, k, cc);
        at(m, ld, k, cc) = at(m, ld, pr, cc);
        at(m, ld, pr, cc) = tmp;
      }
    }
    __syncthreads();
    const int nr = N - k - 1;
    const unsigned dn = small_div_mul(max(nr, 1));
    // trailing update of M (cols k+1..N-1) and of Y (all cols)
    for (int e = threadIdx.x; e < nr * (nr + N); e += kThreads) {
      const int cc = small_div(e, dn), r = k + 1 + e - cc * nr;
      const double l = at(M, ld, r, k);
      double* m = (cc < nr) ? M : Y;
      const int c = (cc < nr) ? k + 1 + cc : cc - nr;
      at(m, ld, r, c) = fma(-l, at(m, ld, k, c), at(m, ld, r, c));
    }
    __syncthreads();
  }
  for (int k = N - 1; k >= 0; --k) {
    const double inv = s_inv[k];
    for (int c = threadIdx.x; c < N; c += kThreads) at(Y, ld, k, c) *= inv;
    __syncthreads();
    const unsigned dk = small_div_mul(max(k, 1));
    for (int e = threadIdx.x; e < k * N; e += kThreads) {
      const int c = small_div(e, dk), r = e - c * k;
      at(Y, ld, r, c) = fma(-at(M, ld, r, k), at(Y, ld, k, c), at(Y, ld, r, c));
    }
    __syncthreads();
  }
  return s_bad == 0;
}

// --------------------------------------------------------------------------
// Fresh equal-time G from the two stacks (numerical_stable.hpp:186-239):
//   general:  G = (U_R Drmax^-1) [ Dlmax^-1 U_L^T U_R Drmax^-1 + Dlmin F_L F_R^T Drmin ]^-1 (Dlmax^-1 U_L^T)
//   right empty (t = Lt): G = (Dmax^-1 U^T + Dmin F)^-1 Dmax^-1 U^T  of the left stack
//   left  empty (t = 0):  G = [same of the right stack]^T
// Also the wrap error max|G_fresh - G| (matrix_compare_error, :34-47) and the trace.
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 2) greens_kernel(const WalkerDev* __restrict__ W, int mode, int j,
                                                          int check_error, int trace_slot) {
  const int wi = blockIdx.x >> 1, sp = blockIdx.x & 1;
  const WalkerDev& w = W[wi];
  if (j >= w.nstack || sp >= w.S || w.path != 0) return;
  extern __shared__ double smem[];
  const int N = w.N, ld = N + 1, ns = w.nstack;
  double* Ms = smem;
  double* Ys = Ms + (long long)N * ld;
  double* dl_max = Ys + (long long)N * ld;
  double* dl_min = dl_max + N;
  double* dr_max = dl_min + N;
  double* dr_min = dr_max + N;
  double* red = dr_min + N;  // 64

  // the final stabilization of the backward sweep (t = 0) and the initial G
  // are not compared with a wrapped G (dqmc_walker.cpp:399-405, :137-147)
  if (mode == MODE_INIT || (mode == MODE_BWD && j == ns - 1)) check_error = 0;
  int nl, nr;  // stack lengths after this step's push/pop
  if (mode == MODE_FWD) { nl = j + 1; nr = ns - 1 - j; }
  else if (mode == MODE_BWD) { nl = ns - 1 - j; nr = j + 1; }
  else { nl = 0; nr = ns; }

  const double* UL = nullptr; const double* FL = nullptr; const double* DL = nullptr;
  const double* UR = nullptr; const double* FR = nullptr; const double* DR = nullptr;
  if (nl > 0) {
    const double* lv = stack_level(w, 0, sp, nl - 1);
    UL = lv; FL = lv + (long long)N * N; DL = lv + 2LL * N * N;
  }
  if (nr > 0) {
    const double* lv = stack_level(w, 1, sp, nr - 1);
    UR = lv; FR = lv + (long long)N * N; DR = lv + 2LL * N * N;
  }
  auto split = [&](const double* D, double* mx, double* mn) {
    for (int i = threadIdx.x; i < N; i += kThreads) {
      const double d = D[i];
      if (d >= 1.0) { mx[i] = d; mn[i] = 1.0; } else { mx[i] = 1.0; mn[i] = d; }
    }
  };
  bool transpose_out = false;
  if (nl > 0 && nr > 0) {
    split(DL, dl_max, dl_min);
    split(DR, dr_max, dr_min);
    __syncthreads();
    // M = Dlmax^-1 (U_L^T U_R) Drmax^-1 + Dlmin (F_L F_R^T) Drmin
    block_gemm(N, [&](int r, int k) { return __ldg(UL + (long long)r * N + k); },
               [&](int k, int c) { return __ldg(UR + (long long)c * N + k); },
               [&](int r, int c, double v) { at(Ms, ld, r, c) = v / (dl_max[r] * dr_max[c]); });
    block_gemm(N, [&](int r, int k) { return __ldg(FL + (long long)k * N + r); },
               [&](int k, int c) { return __ldg(FR + (long long)k * N + c); },
               [&](int r, int c, double v) { at(Ms, ld, r, c) += v * dl_min[r] * dr_min[c]; });
    for (int e = threadIdx.x; e < N * N; e += kThreads) {
      const int r = e % N, c = e / N;  // Y = Dlmax^-1 U_L^T
      at(Ys, ld, r, c) = UL[(long long)r * N + c] / dl_max[r];
    }
  } else {
    const double* U = (nl > 0) ? UL : UR;
    const double* F = (nl > 0) ? FL : FR;
    const double* D = (nl > 0) ? DL : DR;
    transpose_out = (nl == 0);
    split(D, dl_max, dl_min);
    __syncthreads();
    for (int e = threadIdx.x; e < N * N; e += kThreads) {
      const int r = e % N, c = e / N;
      const double y = U[(long long)r * N + c] / dl_max[r];
      at(Ys, ld, r, c) = y;
      at(Ms, ld, r, c) = y + dl_min[r] * F[(long long)c * N + r];
    }
  }
  __syncthreads();
  const bool ok = lu_solve_smem(Ms, Ys, N, ld);
  if (!ok && threadIdx.x == 0) atomicOr(w.status, ST_SINGULAR);

  double* G = w.G + (long long)sp * N * N;
  double* tr = (w.trace && trace_slot >= 0 && trace_slot < w.trace_cap)
                   ? w.trace + ((long long)trace_slot * 2 + sp) * N * N : nullptr;
  double err = 0.0;
  bool finite = true;
  if (nl > 0 && nr > 0) {
    for (int i = threadIdx.x; i < N; i += kThreads) dr_min[i] = 1.0 / dr_max[i];
    __syncthreads();
    // G = (U_R Drmax^-1) Y; the product is formed in registers, compared, stored
    block_gemm(N, [&](int r, int k) { return __ldg(UR + (long long)k * N + r) * dr_min[k]; },
               [&](int k, int c) { return at(Ys, ld, k, c); },
               [&](int r, int c, double v) {
                 const long long o = (long long)c * N + r;
                 if (check_error) err = fmax(err, fabs(v - G[o]));
                 if (!isfinite(v)) finite = false;
                 G[o] = v;
                 if (tr) tr[o] = v;
               });
  } else {
    for (int e = threadIdx.x; e < N * N; e += kThreads) {
      const int r = e % N, c = e / N;
      const double v = transpose_out ? at(Ys, ld, c, r) : at(Ys, ld, r, c);
      if (check_error) err = fmax(err, fabs(v - G[e]));
      if (!isfinite(v)) finite = false;
      G[e] = v;
      if (tr) tr[e] = v;
    }
  }
  if (!finite) atomicOr(w.status, ST_NONFINITE_G);
  if (check_error) {
    const double m = block_max(err, red);
    if (threadIdx.x == 0) atomicMax(w.wrap_bits, (unsigned long long)__double_as_longlong(m));
  }
  // attractive: spin down mirrors spin up
  if (w.S == 1) {
    __syncthreads();
    double* Gd = w.G + (long long)N * N;
    for (int e = threadIdx.x; e < N * N; e += kThreads) Gd[e] = G[e];
    if (tr) {
      double* trd = tr + (long long)N * N;
      for (int e = threadIdx.x; e < N * N; e += kThreads) trd[e] = G[e];
    }
  }
}

// Measurement of a slot whose recorded G is the fresh one (after greens_kernel).
__global__ void __launch_bounds__(kThreads) measure_kernel(const WalkerDev* __restrict__ W, int mode, int j) {
  const WalkerDev& w = W[blockIdx.x];
  if (j >= w.nstack || w.path != 0) return;
  if (mode == MODE_BWD && j != w.nstack - 1) return;
  extern __shared__ double smem[];
  const int N = w.N, ld = N + 1;
  double* gu = smem;
  double* gd = (w.S == 2) ? smem + (long long)N * ld : smem;
  double* red = smem + 2LL * N * ld;
  double* scratch = red + 64;
  for (int sp = 0; sp < w.S; ++sp) {
    const double* Gg = w.G + (long long)sp * N * N;
    double* d = sp ? gd : gu;
    for (int e = threadIdx.x; e < N * N; e += kThreads) at(d, ld, e % N, e / N) = Gg[e];
  }
  __syncthreads();
  const double sg = (mode == MODE_BWD) ? *w.sign_Lt : *w.sign;
  MeasureAcc meas;
  measure_open(meas);
  measure_slice(w, gu, gd, ld, sg, scratch, meas);
  measure_close(w, meas, red);
}

// sign(det G_up det G_dn) (dqmc_walker.cpp:150-163) via in-SMEM LU.
__global__ void __launch_bounds__(kThreads) sign_kernel(const WalkerDev* __restrict__ W) {
  const WalkerDev& w = W[blockIdx.x];
  if (w.path != 0) return;
  extern __shared__ double smem[];
  const int N = w.N, ld = N + 1;
  double* M = smem;
  __shared__ int s_neg;
  if (threadIdx.x == 0) s_neg = 0;
  int total_neg = 0;
  for (int sp = 0; sp < 2; ++sp) {
    const double* Gg = w.G + (long long)sp * N * N;
    for (int e = threadIdx.x; e < N * N; e += kThreads) at(M, ld, e % N, e / N) = Gg[e];
    __syncthreads();
    // LU with partial pivoting, counting swaps and negative pivots
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __shared__ int s_p;
    for (int k = 0; k < N; ++k) {
      if (wid == 0) {
        double best = -1.0;
        int bi = k;
        for (int r = k + lane; r < N; r += 32) {
          const double a = fabs(at(M, ld, r, k));
          if (a > best) { best = a; bi = r; }
        }
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0) s_p = bi;
      }
      __syncthreads();
      const int pr = s_p;
      if (pr != k) {
        for (int c = threadIdx.x; c < N; c += kThreads) {
          const double tmp = at(M, ld, k, c);
          at(M, ld, k, c) = at(M, ld, pr, c);
          at(M, ld, pr, c) = tmp;
        }
        if (threadIdx.x == 0) ++s_neg;
      }
      __syncthreads();
      const double piv = at(M, ld, k, k);
      if (threadIdx.x == 0 && piv < 0) ++s_neg;
      const double inv = (piv != 0.0) ? 1.0 / piv : 0.0;
      for (int r = k + 1 + threadIdx.x; r < N; r += kThreads) at(M, ld, r, k) *= inv;
      __syncthreads();
      const int nr = N - k - 1;
      for (int e = threadIdx.x; e < nr * nr; e += kThreads) {
        const int r = k + 1 + e % nr, c = k + 1 + e / nr;
        at(M, ld, r, c) = fma(-at(M, ld, r, k), at(M, ld, k, c), at(M, ld, r, c));
      }
      __syncthreads();
    }
    total_neg = s_neg;
  }
  if (threadIdx.x == 0) *w.sign = (total_neg % 2 == 0) ? 1.0 : -1.0;
}

// half-sweep counter of the Philox stream (a kernel, so a captured graph advances it)
__global__ void bump_counter_kernel(unsigned long long* ctr) { *ctr += 1ULL; }
void launch_bump(unsigned long long* ctr, cudaStream_t st) { bump_counter_kernel<<<1, 1, 0, st>>>(ctr); }

// MeasureHandler::normalize_stats + write_stats_to_bins + clear_temporary
// (src/measure/measure_handler.cpp:170-277) for every walker on the device:
// bin = sum / (count <sign>), the sign bin |<sign>|, accumulators cleared.
// bins: [walker][nbins][kNumObs].
__global__ void bin_close_kernel(const WalkerDev* __restrict__ W, int nw, double* bins, int nbins, int bin) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  const WalkerDev& h = W[w];
  const double sign = h.obs[kNumObs - 1] / (double)h.obs_cnt[kNumObs - 1];
  double* out = bins + ((long long)w * nbins + bin) * kNumObs;
  for (int k = 0; k < kNumObs - 1; ++k) out[k] = h.obs[k] / ((double)h.obs_cnt[k] * sign);
  out[kNumObs - 1] = fabs(sign);
  for (int k = 0; k < kNumObs; ++k) {
    h.obs[k] = 0.0;
    h.obs_cnt[k] = 0;
  }
}
void launch_bin_close(const WalkerDev* W, int nw, double* bins, int nbins, int bin, cudaStream_t st) {
  bin_close_kernel<<<(nw + 127) / 128, 128, 0, st>>>(W, nw, bins, nbins, bin);
}

// --------------------------------------------------------------------------
// FP64 FMA throughput probe: 8 independent register FMA chains per thread.
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) fp64_fma_probe(double* out, int iters, double a, double b) {
  double x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = threadIdx.x * 1e-3 + k;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = fma(x[k], a, b);
  }
  double s = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += x[k];
  if (s == 12345.678) out[blockIdx.x] = s;  // keeps the chains live
}

double run_fp64_probe(cudaError_t* err) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  double* d = nullptr;
  *err = cudaMalloc(&d, sizeof(double) * sms * 8);
  if (*err) return 0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int iters = 4096, blocks = sms * 8;
  fp64_fma_probe<<<blocks, kThreads>>>(d, iters, 0.999999, 1e-7);  // warm-up
  cudaEventRecord(e0);
  fp64_fma_probe<<<blocks, kThreads>>>(d, iters, 0.999999, 1e-7);
  cudaEventRecord(e1);
  *err = cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(d);
  if (*err == cudaSuccess) *err = cudaGetLastError();
  return 2.0 * 8.0 * iters * (double)blocks * kThreads / (ms * 1e-3) / 1e9;
}

// --------------------------------------------------------------------------
// host-side launch helpers
// --------------------------------------------------------------------------
size_t segment_smem_bytes(int N, int S) {
  const size_t mats = S * (segment_chain_smem(N) ? 2 : 1) + (segment_joint_spins(N) ? S : 1);
  return sizeof(double) * (mats * N * (N + 1) + 8 * N + 64 + 3 * N);
}
size_t push_smem_bytes(int N) { return sizeof(double) * ((size_t)N * (N + 1) + 4 * N) + sizeof(int) * N; }
size_t greens_smem_bytes(int N) { return sizeof(double) * (2 * (size_t)N * (N + 1) + 4 * N + 64); }
size_t measure_smem_bytes(int N) { return sizeof(double) * (2 * (size_t)N * (N + 1) + 64 + 3 * N); }

cudaError_t configure_fp64_kernels(int maxN) {
  // the largest of both placements of the chain
  const size_t s1 = std::max(segment_smem_bytes(maxN, 2), segment_smem_bytes(50, 2)), s2 = push_smem_bytes(maxN), s3 = greens_smem_bytes(maxN),
               s4 = measure_smem_bytes(maxN);
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(segment_kernel<MODE_INIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1))) return e;
  if ((e = cudaFuncSetAttribute(segment_kernel<MODE_FWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1))) return e;
  if ((e = cudaFuncSetAttribute(segment_kernel<MODE_BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1))) return e;
  if ((e = cudaFuncSetAttribute(push_kernel<MODE_INIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2))) return e;
  if ((e = cudaFuncSetAttribute(push_kernel<MODE_FWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2))) return e;
  if ((e = cudaFuncSetAttribute(push_kernel<MODE_BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2))) return e;
  if ((e = cudaFuncSetAttribute(greens_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3))) return e;
  if ((e = cudaFuncSetAttribute(measure_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s4))) return e;
  if ((e = cudaFuncSetAttribute(sign_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3))) return e;
  return cudaSuccess;
}

void launch_segment(int mode, const WalkerDev* W, int nw, int j, int measure, int maxN, cudaStream_t st) {
  const size_t sm = segment_smem_bytes(maxN, 2);
  if (mode == MODE_INIT) segment_kernel<MODE_INIT><<<nw, kThreads, sm, st>>>(W, j, 0, maxN);
  else if (mode == MODE_FWD) segment_kernel<MODE_FWD><<<nw, kThreads, sm, st>>>(W, j, measure, maxN);
  else segment_kernel<MODE_BWD><<<nw, kThreads, sm, st>>>(W, j, measure, maxN);
}
void launch_push(int mode, const WalkerDev* W, int nw, int j, int maxN, cudaStream_t st) {
  const size_t sm = push_smem_bytes(maxN);
  if (mode == MODE_INIT) push_kernel<MODE_INIT><<<2 * nw, kPushThreads, sm, st>>>(W, j);
  else if (mode == MODE_FWD) push_kernel<MODE_FWD><<<2 * nw, kPushThreads, sm, st>>>(W, j);
  else push_kernel<MODE_BWD><<<2 * nw, kPushThreads, sm, st>>>(W, j);
}
void launch_greens(int mode, const WalkerDev* W, int nw, int j, int check, int trace_slot, int maxN, cudaStream_t st) {
  greens_kernel<<<2 * nw, kThreads, greens_smem_bytes(maxN), st>>>(W, mode, j, check, trace_slot);
}
void launch_measure(int mode, const WalkerDev* W, int nw, int j, int maxN, cudaStream_t st) {
  measure_kernel<<<nw, kThreads, measure_smem_bytes(maxN), st>>>(W, mode, j);
}
void launch_sign(const WalkerDev* W, int nw, int maxN, cudaStream_t st) {
  sign_kernel<<<nw, kThreads, greens_smem_bytes(maxN), st>>>(W);
}

}  // namespace dqmc
