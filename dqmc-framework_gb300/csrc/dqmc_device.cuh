// dqmc_device.cuh — device data model of a walker batch (FP64 plain method).
//
// One WalkerDev per walker, in device memory.  Everything a CTA needs to run
// one walker's segment or stabilization is reachable from it: the Green's
// functions, the B-chain buffer, the UDT stacks, the Ising fields, the dense
// exp(+/-dtau K) (shared by walkers with equal lattice parameters), the
// Fourier table of the measured momentum and the per-walker accumulators.
//
// Layouts (all column-major, leading dimension N, 256-byte aligned bases):
//   G      [2][N*N]      spin 0 = up, spin 1 = down (attractive: spin 1 aliases 0)
//   chain  [S][N*N]      running B-chain product of the current segment
//   stack  [side][S][level] { U (N*N) | F (N*N) | D (N) }, side 0 left, 1 right
//   fields [Lt][N] int8  +/-1, slice-major (reference: Lt x N Eigen matrix of doubles)
#pragma once
#include <cstdint>

namespace dqmc {

constexpr int kThreads = 256;
constexpr int kMaxSmemN = 64;    // N handled by the SMEM-resident kernels
constexpr int kMaxN = 1024;      // largest N of the general (HBM-resident) kernels
constexpr int kNumObs = 9;

enum SweepMode { MODE_INIT = 0, MODE_FWD = 1, MODE_BWD = 2 };

// status bits (per walker)
enum : int {
  ST_NONFINITE_G = 1,
  ST_SINGULAR = 2,
  ST_NONFINITE_RATIO = 4,
  ST_TIMEOUT = 8,  // a bounded device-side wait gave up (the kernel skipped its output)
};

struct WalkerDev {
  int N, L, Lt, pace, nstack, S, model, cb;  // model: 0 repulsive, 1 attractive
  int dim;                                    // 2 square (N = L^2), 3 cubic (N = L^3)
  int rng;                                    // 0 host uniforms, 1 Philox
  int path;                                   // 0 SMEM FP64, 1 HBM FP64, 2 HBM mixed (tensor-core products)
  double hop_t;
  // B-matrix diagonal factors exp(+alpha), exp(-alpha)
  double e_pa, e_ma;
  // ratio constants indexed by [s>0 ? 0 : 1]: exp(-2 alpha s) - 1, exp(+2 alpha s) - 1, exp(2 alpha s)
  double cm[2], cp[2], ex2[2];
  double cbP[16], cbI[16];   // checkerboard plaquettes exp(+dtau t h) e^{0.5 dtau mu}, inverse
  // Factored exp(-+dtau K), index [0] and its inverse [1].  Checkerboard: the plaquette is
  // f c^2 [[1, h], [h, 1]] (x) [[1, h], [h, 1]] (its inverse has -h).  Otherwise the Kronecker
  // product of one ring exponential per direction: kin [2][L], by the distance |x - x'| on the ring
  // of L sites.  kin_e: exp(+alpha), exp(-alpha), for checkerboard walkers times the (f c^2)^2 of a
  // product's two passes.
  double cb_h, kin_e[2][2];
  const double* kin;
  double* G;                 // [2][N*N]
  double* chain;             // [S][N*N] (general walkers: [2][S][N*N], ping-pong)
  double* work;              // mixed walkers: product temporary [S][N*N]
  double* scr;               // general walkers: stabilization scratch [S][2][N*N]
  // mixed walkers, submatrix Metropolis: per spin T [N][32] FP64, then the BF16
  // slices of T and of G0(:, accepted sites) [2][6][N][40] and their exponents [2][N]
  unsigned char* msub;
  // time-displaced Green's functions (dynamic half-sweep), allocated on first use:
  // G(t,0) and G(0,t) ping-pong [2][S][N*N], second right-hand side [S][N*N],
  // LU pivots [S][N], G(k,tau) accumulators [dyn_ntau]
  double* gt0;
  double* g0t;
  double* dynx;
  int* dpiv;
  double* dyn_sum;
  long long* dyn_cnt;
  const int* dyn_taus;
  int dyn_ntau;
  // dynamic observables: sums [tau][3] (density of states, spin susceptibility, stiffness),
  // per-half-sweep parts awaiting G(beta,beta): vectors [tau][2][N] and scalars [tau][2]
  double* dyn_obs;
  double* dyn_vec;
  double* dyn_part;
  double* dyn_r;  // [tau][N] sign * 0.5 sum_i (G_up + G_dn)(i + r, i) / N: G(k,tau) of any k
  int zld;                   // line stride of zsl (N rounded up to 32)
  // tensor-core stabilization: BF16 slices of the operands of the current product, A and up to
  // three parts of B, in the room of two N x N operands: [S][2][9 slices][N][zld]
  unsigned short* zsl;
  // mixed walkers: BF16 slices of the operand being multiplied, [S][slices][N][ldk]
  unsigned short* sl;
  int* sle;                  // slice exponents [S][N]
  int ldk;                   // padded slice row length (multiple of 16)
  int slice_bits, slices;
  // constant slices of exp(-dtau K) and exp(+dtau K) as left (A) and right (B) operands
  const unsigned short* kA; const unsigned short* kB; const unsigned short* iA; const unsigned short* iB;
  const int* kAe; const int* kBe; const int* iAe; const int* iBe;
  double* stack;             // see header
  long long lvl_stride;      // doubles per stack level (2 N^2 + N, padded)
  long long side_stride;     // doubles per side (S * nstack * lvl_stride)
  int8_t* fields;            // [Lt][N]
  const double* ff;          // Fourier factor per displacement index, measured k
  double* obs;               // [kNumObs] sums of sign * O
  long long* obs_cnt;        // [kNumObs]
  double* sign;              // current configuration sign
  double* sign_Lt;           // sign recorded at t = Lt of the backward half-sweep
  unsigned long long* wrap_bits;  // running max |G_fresh - G_wrapped| (bit pattern)
  long long* accepts;
  int* status;
  const double* uni;         // parity uniforms of the current half-sweep [Lt*N]
  unsigned long long seed;   // Philox key
  const unsigned long long* sweep_ctr;  // Philox counter word: the batch's half-sweep index (device)
  double* trace;             // [trace_cap][2][N*N] or null
  int trace_cap;
  int ozstab;                // stabilization by the blocked QR (kernels_stab_oz.cu): 1 with tensor-core
                             // products, 2 with FP64 products, 0 not
  double* zwk;               // its scratch per spin, zwk_stride doubles apart
  long long zwk_stride;
  int widx;                  // index of the walker in its batch (Philox counter word)
  // iteration limit of the wraps' and B-chain products' waits for their operands to land
  // (oz_prod_tc_kernel); kDefaultWaitLimit unless a test lowers it (dqmc_set_wait_limit)
  int wait_limit;
};

// The largest N of a batch's walkers stabilized with tensor-core and with FP64 products (0: none),
// the smallest of the former, and the matrices (walkers times spins) of the latter in the whole batch
struct StabSizes {
  int tc, f64, tc_min, f64_mats;
  __host__ __device__ int max() const { return tc > f64 ? tc : f64; }
};

// A stream beside the launch's own, with the events that fork it off and join it; null: none
struct SideStream {
  cudaStream_t st;
  cudaEvent_t fork, join;
};

constexpr int kDefaultWaitLimit = 1 << 24;

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11): uniform double in [0,1)
// keyed by the walker's seed, counter (site attempt, half-sweep, walker).
__device__ __forceinline__ double philox_uniform(unsigned long long seed, unsigned walker, unsigned long long sweep,
                                                 unsigned attempt) {
  unsigned c0 = attempt, c1 = (unsigned)sweep, c2 = (unsigned)(sweep >> 32), c3 = walker;
  unsigned k0 = (unsigned)seed, k1 = (unsigned)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const unsigned hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const unsigned n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  const unsigned long long m = ((unsigned long long)(c0 >> 5) << 26) | (unsigned long long)(c1 >> 6);
  return (double)m * (1.0 / 9007199254740992.0);
}

// Metropolis ratio of flipping the field s of a site whose equal-time diagonals are
// gu = G_up(i,i), gd = G_dn(i,i) (si = 0 for s = +1, 1 for s = -1):
//   repulsive   r = (1 + (1 - gu)(e^{-2as} - 1)) (1 + (1 - gd)(e^{+2as} - 1))
//   attractive  r = e^{2as} (1 + (1 - gu)(e^{-2as} - 1)) (1 + (1 - gd)(e^{-2as} - 1))
// (get_update_ratio, src/model/repulsive_hubbard.cpp:112-124 and
// src/model/attractive_hubbard.cpp:112-125), each operation rounded on its own in the
// reference's order, never contracted into an FMA, so equal diagonals give bit-equal
// ratios and decisions on every path.  Every Metropolis kernel evaluates it here.
struct FlipRatio {
  double r;       // the ratio
  double ru, rd;  // its spin factors 1 + (1 - G_ii) Delta
  double cu, cd;  // Delta_up, Delta_dn (e^{-+2as} - 1)
};

__device__ __forceinline__ FlipRatio flip_ratio(const WalkerDev& w, int si, double gu, double gd) {
  FlipRatio q;
  q.cu = w.cm[si];
  q.cd = (w.model == 0) ? w.cp[si] : w.cm[si];
  q.ru = __dadd_rn(1.0, __dmul_rn(__dsub_rn(1.0, gu), q.cu));
  q.rd = __dadd_rn(1.0, __dmul_rn(__dsub_rn(1.0, gd), q.cd));
  q.r = (w.model == 0) ? __dmul_rn(q.ru, q.rd) : __dmul_rn(__dmul_rn(w.ex2[si], q.ru), q.rd);
  return q;
}

// The factors f_sigma = Delta_sigma / (1 + (1 - G_ii) Delta_sigma) of the accepted flip's
// rank-1 update (update_greens_function, src/model/repulsive_hubbard.cpp:127-155; the
// attractive model's factor_dn equals factor_up, src/model/attractive_hubbard.cpp:149).
__device__ __forceinline__ void flip_factors(const WalkerDev& w, const FlipRatio& q, double* f) {
  f[0] = __ddiv_rn(q.cu, q.ru);
  f[1] = (w.model == 0) ? __ddiv_rn(q.cd, q.rd) : f[0];
}

// Metropolis decisions of one warp.  The lanes evaluate the ratios of a window of sites at once
// (both spins of 16 sites when the spins differ, 32 sites otherwise); the lowest accepted site is
// the next accept of the sequential visit, since every site before it saw the same diagonal.  An
// FP64 instruction holds the warp 64 cycles for one lane or for 32, so a window costs what one
// site costs, and each spin's factor 1 + (1 - G_ii) Delta and its division Delta / factor share
// an instruction.  The uniform is compared through its bit pattern: u < min(1, |r|) is u < |r|
// for u in [0, 1), and doubles of one sign order as integers (a NaN ratio accepts, as fmin does).
// What bounds an accept at N = 16 (2700 cycles) is this chain: 5 dependent FP64 operations and the
// division (9 more) at 64 cycles each, 2100 cycles with its shared-memory and shuffle latencies
// beside the update's FMAs.  One thread visiting the sites in turn, with the Philox rounds and
// the descriptor's loads in the chain, made a pass of 4 x 4, beta = 4 take 11.0 ms, this 8.1 ms
// (with measure_slice, flat_gemm and the shared-memory chain); 256 walkers of 8 x 8 240 -> 208 ms.
struct SiteScan {
  int S, width, sp, dl;           // spins, sites per window, this lane's spin and site in the window
  double c[2], e2[2];             // Delta of this lane's spin and exp(2 alpha s), by field s = +1, -1

  __device__ __forceinline__ SiteScan(const WalkerDev& w, int lane) {
    S = w.S;
    width = (S == 2) ? 16 : 32;
    sp = (S == 2) ? lane >> 4 : 0;
    dl = lane & (width - 1);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      c[k] = (w.model == 0 && sp == 1) ? w.cp[k] : w.cm[k];
      e2[k] = w.ex2[k];
    }
  }
  // The next accepted site from `from` on (N: none; NW windows reach N); diag(b, l) is the current
  // diagonal element of this lane's spin at site l < N of window b.  Flips the field and leaves
  // the update's factors in f[2].  The whole warp calls; sign and accepts are uniform in it.
  template <int NW, class Diag>
  __device__ __forceinline__ int next(const WalkerDev& w, Diag diag, int from, int N, const double* uni,
                                      int8_t* field, double* f, double& sign, long long& accepts) const {
#pragma unroll
    for (int b = 0; b < NW; ++b) {
      const int base = from + b * width;
      if (base >= N) break;
      const int l = base + dl;
      const bool in = l < N;
      const double g = in ? diag(b, l) : 0.0;
      const int s = in ? field[l] : 1;
      const double ck = s > 0 ? c[0] : c[1];
      const double qs = __dadd_rn(1.0, __dmul_rn(__dsub_rn(1.0, g), ck));
      const double fq = __ddiv_rn(ck, qs);  // beside the acceptance, not after it
      // reference operation order (flip_ratio)
      const double r = (S == 2) ? __dmul_rn(qs, __shfl_xor_sync(0xffffffffu, qs, 16))
                                : __dmul_rn(__dmul_rn(s > 0 ? e2[0] : e2[1], qs), qs);
      const long long rb = __double_as_longlong(r), ab = rb & 0x7fffffffffffffffLL;
      const bool acc = in && __double_as_longlong(in ? uni[l] : 0.0) < ab;
      const unsigned mask = __ballot_sync(0xffffffffu, acc) & (S == 2 ? 0xffffu : 0xffffffffu);
      const int first = mask ? __ffs(mask) - 1 : 32;
      if (in && dl <= first && ab >= 0x7ff0000000000000LL) atomicOr(w.status, ST_NONFINITE_RATIO);
      if (mask) {
        if (dl == first) {
          f[sp] = fq;
          if (S == 1) f[1] = fq;
          if (sp == 0) field[l] = (int8_t)(-s);
        }
        const long long rf = __shfl_sync(0xffffffffu, rb, first);
        // r >= 0 (false for a NaN)
        if (!((rf >= 0 && rf <= 0x7ff0000000000000LL) || rf == (long long)0x8000000000000000ULL)) sign = -sign;
        ++accepts;
        return base + first;
      }
    }
    return N;
  }
};

// The sites of plaquette q of a checkerboard layer (corner (x, y), x and y of the layer's parity)
__device__ __forceinline__ void plaq_sites(int L, int q, int parity, int (&idx)[4]) {
  const int half = L >> 1;
  const int x = 2 * (q % half) + parity, y = 2 * (q / half) + parity;
  const int x1 = (x + 1) % L, y1 = (y + 1) % L;
  idx[0] = x + L * y;
  idx[1] = x1 + L * y;
  idx[2] = x + L * y1;
  idx[3] = x1 + L * y1;
}

// The plaquette matrix is f c^2 [[1, h], [h, 1]] (x) [[1, h], [h, 1]] with c = cosh, h = tanh of
// +-dtau t: applied as two butterflies of 8 FMAs on the plaquette's 4 values instead of a 4 x 4
// product of 4 multiplies and 12 FMAs (an FP64 warp instruction holds its pipe for 64 cycles,
// and the passes are half of a checkerboard slice's FP64 work).  The factors f c^2 of a product's
// two passes are folded into the diagonal scale of the product (bdiag).
__device__ __forceinline__ void plaq_apply(double (&v)[4], double h) {
  const double a0 = fma(h, v[1], v[0]), a1 = fma(h, v[0], v[1]);
  const double a2 = fma(h, v[3], v[2]), a3 = fma(h, v[2], v[3]);
  v[0] = fma(h, a2, a0);
  v[1] = fma(h, a3, a1);
  v[2] = fma(h, a0, a2);
  v[3] = fma(h, a1, a3);
}

// The plain 4 x 4 product: the set-up keeps it, because the sign it takes from an LU of the
// initial G is rounding noise once G has eigenvalues below its rounding (8 x 8 at beta = 8), and
// a given seed has to keep its sign.
__device__ __forceinline__ void plaq_product(double (&v)[4], const double* P) {
  double o[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    o[a] = P[a * 4 + 0] * v[0];
    o[a] = fma(P[a * 4 + 1], v[1], o[a]);
    o[a] = fma(P[a * 4 + 2], v[2], o[a]);
    o[a] = fma(P[a * 4 + 3], v[3], o[a]);
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) v[a] = o[a];
}

// Site i of a walker's lattice is x + L y (+ L^2 z).  The displacement from site i to site j
// as the site index of its vector, each component mod L (src/lattice/square.cpp:88-105,
// src/lattice/cubic.cpp:112-132), and the neighbour of site i in direction +x, +y or +z.
__device__ __forceinline__ int site_disp(int L, int dim, int i, int j) {
  if (dim == 2) {
    int dx = j % L - i % L, dy = j / L - i / L;
    dx += (dx < 0) ? L : 0;
    dy += (dy < 0) ? L : 0;
    return dx + dy * L;
  }
  const int LL = L * L;
  int dx = j % L - i % L, dy = (j / L) % L - (i / L) % L, dz = j / LL - i / LL;
  dx += (dx < 0) ? L : 0;
  dy += (dy < 0) ? L : 0;
  dz += (dz < 0) ? L : 0;
  return dx + dy * L + dz * LL;
}
__device__ __forceinline__ int site_nn(int L, int i, int a) {
  const int w = (a == 0) ? 1 : (a == 1) ? L : L * L;
  const int c = (i / w) % L;
  return i + ((c + 1) % L - c) * w;
}
// the site at displacement r from site i
__device__ __forceinline__ int site_shift(int L, int dim, int i, int r) {
  int j = 0;
  for (int a = 0, w = 1; a < dim; ++a, w *= L) j += (((i / w) % L + (r / w) % L) % L) * w;
  return j;
}

__host__ __device__ inline double* stack_level(const WalkerDev& w, int side, int spin, int level) {
  return w.stack + side * w.side_stride + ((long long)spin * w.nstack + level) * w.lvl_stride;
}

}  // namespace dqmc
