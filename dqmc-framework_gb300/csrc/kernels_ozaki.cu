// kernels_ozaki.cu — the mixed-precision products of the sweep: FP64-accurate
// (49-bit) matrix products on the BF16 tensor cores (see ozaki.cuh).
//
// Slicing is integer work on the FP64 bit patterns; the product runs the
// S(S+1)/2 slice pairs on the BF16 tensor cores (tcgen05, TMEM accumulators)
// with FP32 accumulation, exact by construction, one accumulator per weight group, and
// recombines the groups in the epilogue.  Used for the wraps and the B-chain (the reference's
// mult_B_from_left/right, mult_invB_*, mult_transB_from_left,
// src/model/repulsive_hubbard.cpp:158-243, src/model/model_base.cpp:7-35).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "dqmc_device.cuh"
#include "ozaki.cuh"
#include "oz_tc.cuh"
#include "tcgen05.cuh"

namespace dqmc {

using ozaki::kMaxSlices;

// --------------------------------------------------------------------------
// Slicing.  role 0 (left operand, A): lines are rows r, k runs over columns.
// role 1 (right operand, B): lines are columns c, k runs over rows.  X is
// column-major N x N (ld N).  pre (may be null) scales element k of every line
// before slicing.  out: the tensor-core image (ozaki::tc_index, slice stride
// ozaki::tc_slice_elems).  One CTA of 256 threads per 32 lines.
// --------------------------------------------------------------------------
struct SliceJob {
  const double* X;
  unsigned short* out;  // BF16 bits, S slices
  int* exps;            // [N]
  const double* pre;    // along k, or null
};

__device__ __forceinline__ double xelem(const double* X, int N, int role, int line, int k) {
  return role == 0 ? X[(long long)k * N + line] : X[(long long)line * N + k];
}

__device__ void slice_lines(const SliceJob& job, int N, int ldk, int role, int bits, int slices, int line0) {
  __shared__ int s_e[8][32];
  __shared__ double s_t[32][33];
  const int tid = threadIdx.x;
  // pass 1: exponent per line (integer max of exponent bounds)
  {
    const int ll = (role == 0) ? (tid & 31) : (tid >> 3);   // line in block
    const int kg = (role == 0) ? (tid >> 5) : (tid & 7);    // k group of 8
    int e = -1100;
    const int line = line0 + ll;
    if (line < N)
      for (int k = kg; k < N; k += 8) {
        double x = xelem(job.X, N, role, line, k);
        if (job.pre) x *= job.pre[k];
        e = max(e, ozaki::exp_bound(x));
      }
    s_e[kg][ll] = e;
  }
  __syncthreads();
  if (tid < 32) {
    int e = s_e[0][tid];
    for (int g = 1; g < 8; ++g) e = max(e, s_e[g][tid]);
    s_e[0][tid] = e;
    if (line0 + tid < N) job.exps[line0 + tid] = e;
  }
  __syncthreads();
  // pass 2: 32 x 32 tiles, staged so the BF16 writes run along k
  for (int k0 = 0; k0 < ldk; k0 += 32) {
    for (int e2 = tid; e2 < 32 * 32; e2 += blockDim.x) {
      int ll, kk;
      if (role == 0) { ll = e2 & 31; kk = e2 >> 5; } else { kk = e2 & 31; ll = e2 >> 5; }
      const int line = line0 + ll, k = k0 + kk;
      double x = 0.0;
      if (line < N && k < N) {
        x = xelem(job.X, N, role, line, k);
        if (job.pre) x *= job.pre[k];
      }
      s_t[ll][kk] = x;
    }
    __syncthreads();
    const int Q = bits * slices;
    {
      // one line and 4 consecutive k per thread: one 8-byte store per slice
      const int kq = tid & 7, ll = tid >> 3;
      const int line = line0 + ll, k = k0 + kq * 4;
      if (line < N && k < ldk) {
        unsigned long long q[4];
        bool ng[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = ozaki::fixedq(s_t[ll][kq * 4 + u], s_e[0][ll], Q, ng[u]);
        const long long sstride = (long long)ozaki::tc_slice_elems(N, ldk);
        unsigned short* o = job.out + ozaki::tc_index(line, k, ozaki::tc_lines(N) / 8);
        for (int s = 0; s < slices; ++s) {
          ushort4 v;
          v.x = ozaki::slice_bf16q(q[0], s, bits, Q, ng[0]);
          v.y = ozaki::slice_bf16q(q[1], s, bits, Q, ng[1]);
          v.z = ozaki::slice_bf16q(q[2], s, bits, Q, ng[2]);
          v.w = ozaki::slice_bf16q(q[3], s, bits, Q, ng[3]);
          *reinterpret_cast<ushort4*>(o + s * sstride) = v;
        }
      }
    }
    __syncthreads();
  }
}

struct ProdJob {
  const unsigned short* A;  // S slices, tensor-core images
  const unsigned short* B;
  const int* ea;
  const int* eb;
};

namespace {
__device__ __forceinline__ bool oz_slice_of(const WalkerDev& w, int mode, int j, int q, int& t) {
  if (j >= w.nstack) return false;
  const int k = (mode == MODE_FWD) ? j : (w.nstack - 1 - j);
  const int t_lo = k * w.pace + 1, t_hi = min((k + 1) * w.pace, w.Lt);
  if (q >= t_hi - t_lo + 1) return false;
  t = (mode == MODE_FWD) ? t_lo + q : t_hi - q;
  return true;
}
__device__ __forceinline__ double oz_bscale(const WalkerDev& w, int t, int spin, int sgn, int i) {
  const int sf = (w.model == 0 && spin == 1) ? -1 : 1;
  const int s = w.fields[(long long)(t - 1) * w.N + i];
  return (sgn * sf * s > 0) ? w.e_pa : w.e_ma;
}
__device__ __forceinline__ double* oz_chain(const WalkerDev& w, int spin, int which) {
  return w.chain + ((long long)which * w.S + spin) * w.N * w.N;
}
}  // namespace

// Operations of one slice (same meaning as gemm_op_kernel's):
//   OZ_WL_FWD  work   = diag(e+) expK G          (A: expK const, B: G)
//   OZ_WR_FWD  G      = work expK^-1 diag(e-)    (A: work,       B: invK const)
//   OZ_CH_FWD  chain' = diag(e+) expK chain      (A: expK const, B: chain)
//   OZ_CH_BWD  chain' = expK^T diag(e+) chain    (A: expK^T = expK as B-slices, B: diag(e+) chain)
//   OZ_WR_BWD  work   = G diag(e+) expK          (A: G diag(e+), B: expK const)
//   OZ_WL_BWD  G      = expK^-1 diag(e-) work    (A: invK const, B: diag(e-) work)
// and the time-displaced steps of the dynamic half-sweep (the reference's
// mult_B_from_left and mult_invB_from_right, src/dqmc_walker.cpp:455-466), on the
// ping-pong slots [parity][S][N*N] of G(t,0) and G(0,t):
//   OZ_DT0     G(t,0) = diag(e+) expK G(t-1,0)   (A: expK const, B: G(t-1,0))
//   OZ_D0T     G(0,t) = G(0,t-1) expK^-1 diag(e-) (A: G(0,t-1),   B: invK const)
enum OzOp { OZ_WL_FWD = 0, OZ_WR_FWD = 1, OZ_CH_FWD = 2, OZ_CH_BWD = 3, OZ_WR_BWD = 4, OZ_WL_BWD = 5,
            OZ_DT0 = 6, OZ_D0T = 7 };

__device__ __forceinline__ double* oz_dyn(double* base, const WalkerDev& w, int spin, int t) {
  return base + ((long long)(t & 1) * w.S + spin) * w.N * w.N;
}

// slice the per-walker operand of op OP: grid (ceil(N/32), 2*nw), 256 threads
template <int OP>
__global__ void __launch_bounds__(256) oz_slice_kernel(const WalkerDev* __restrict__ W, int mode, int j, int q) {
  const int wi = blockIdx.y >> 1, sp = blockIdx.y & 1;
  const WalkerDev& w = W[wi];
  if (w.path != 2 || w.cb || sp >= w.S) return;
  int t;
  if (!oz_slice_of(w, mode, j, q, t)) return;
  const int N = w.N;
  const long long NN = (long long)N * N;
  __shared__ double s_pre[1024];
  int role = 1, sgn = 0;
  const double* X = nullptr;
  switch (OP) {
    case OZ_WL_FWD: X = w.G + sp * NN; role = 1; break;
    case OZ_WR_FWD: X = w.work + sp * NN; role = 0; break;
    case OZ_CH_FWD: X = oz_chain(w, sp, q & 1); role = 1; break;
    case OZ_CH_BWD: X = oz_chain(w, sp, q & 1); role = 1; sgn = +1; break;
    case OZ_WR_BWD: X = w.G + sp * NN; role = 0; sgn = +1; break;
    case OZ_WL_BWD: X = w.work + sp * NN; role = 1; sgn = -1; break;
    case OZ_DT0: X = w.gt0 ? oz_dyn(w.gt0, w, sp, t - 1) : nullptr; role = 1; break;
    case OZ_D0T: X = w.g0t ? oz_dyn(w.g0t, w, sp, t - 1) : nullptr; role = 0; break;
  }
  if (!X) return;
  if (sgn)
    for (int k = threadIdx.x; k < N; k += blockDim.x) s_pre[k] = oz_bscale(w, t, sp, sgn, k);
  __syncthreads();
  SliceJob job{X, w.sl + (long long)sp * w.slices * ozaki::tc_slice_elems(N, w.ldk), w.sle + (long long)sp * N,
               sgn ? s_pre : nullptr};
  slice_lines(job, N, w.ldk, role, w.slice_bits, w.slices, blockIdx.x * 32);
}

// Product of op OP on the 5th-generation tensor cores: a 128 x NT output
// tile per CTA with the S weight groups accumulated in TMEM (S x NT columns),
// the operands streamed by oztc::mainloop (bulk copies through a ring of NS
// stages of 16-deep k chunks).  Two tile shapes per slice configuration, picked
// per batch by the autotuner (dqmc_init_greens): 128 x 32 tiles, two CTAs per SM
// (at most 256 TMEM columns, 105 KB (7 slices, 3 stages) or 80 KB (8 slices, 2
// stages) of shared memory and 128 registers each), or 128 x 64 tiles, one CTA
// per SM (512 TMEM columns, 3 or 4 stages).  Shape SH = 0 is 128 x 32 for the
// 49-bit configuration (7 slices, K <= 256) and 128 x 64 for the 48-bit one (8
// slices); SH = 1 swaps them.
__host__ __device__ constexpr int oz_tc_nt(int S, int SH) { return ((S <= 7) == (SH == 0)) ? 32 : 64; }
__host__ __device__ constexpr int oz_tc_stages(int S, int SH) {
  return oz_tc_nt(S, SH) == 32 ? (S <= 7 ? 3 : 2) : (S <= 7 ? 3 : 4);
}
__host__ __device__ constexpr int oz_tc_minb(int S, int SH) { return oz_tc_nt(S, SH) == 32 ? 2 : 1; }
__host__ __device__ constexpr int oz_tc_stage_bytes(int S, int SH) {
  return oztc::stage_bytes(S, 128, oz_tc_nt(S, SH));
}

// One 128 x NT tile (rows r0.., columns c0..) of a product of N x N operands: epi(rl, r, cl, col,
// value) per element inside the matrix.  Returns whether a wait ran out (epi was then not called);
// all 256 threads call.
template <int S, int NT, int NS, int MINB, class Epi>
__device__ __forceinline__ bool oz_tc_tile(const ProdJob& job, int N, int ldk, int r0, int c0, int wait_limit,
                                           unsigned char* tsm, Epi epi) {
  constexpr int MT = 128;
  constexpr int CW = (MINB > 1) ? 8 : 16;  // TMEM columns per load in the epilogue
  constexpr unsigned TCOLS = (S * NT <= 256) ? 256u : 512u;
  __shared__ int eA[MT], eB[NT];
  __shared__ __align__(8) unsigned long long full[NS], done[NS];
  __shared__ unsigned tbase;
  __shared__ int s_fail, s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < MT) eA[tid] = (r0 + tid < N) ? job.ea[r0 + tid] : -1100;
  if (tid < NT) eB[tid] = (c0 + tid < N) ? job.eb[c0 + tid] : -1100;
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
    // chunk c of the tile: (c * nlb + line0 / 8) 8-line blocks of 128 elements into each slice
    const long long sstride = (long long)ozaki::tc_slice_elems(N, ldk);
    const long long cstep = (long long)(ozaki::tc_lines(N) / 8) * 128;
    bool ok;
    s_last = oztc::mainloop<S, MT, NT, NS>(tsm, full, done, taddr, job.A + (long long)(r0 / 8) * 128,
                                            job.B + (long long)(c0 / 8) * 128, sstride, cstep, ldk / 16, ok,
                                            wait_limit);
    s_fail = ok ? 0 : 1;
  }
  __syncthreads();
  const int last = s_last;
  const bool mma_done = last >= 0 && tc::mbar_wait(&done[last % NS], (last / NS) & 1);
  const int failed = __syncthreads_or(!mma_done || s_fail);
  tc::fence_after();
  constexpr int SB = (S <= 7) ? 7 : 6;  // bits per slice of the configuration (ozaki::cfg_for_k)
  const int q4 = warp & 3, half = warp >> 2;
  const int rl = q4 * 32 + lane, r = r0 + rl;
  if (!failed) {
    for (int cc = half * (NT / 2); cc < (half + 1) * (NT / 2); cc += CW) {
      uint32_t v[S][CW];
#pragma unroll
      for (int m = 0; m < S; ++m) tc::ldw<CW>(v[m], taddr + ((unsigned)(q4 * 32) << 16) + (unsigned)(m * NT + cc));
      tc::wait_ld();
      if (r < N) {
#pragma unroll
        for (int u = 0; u < CW; ++u) {
          const int cl = cc + u, col = c0 + cl;
          if (col >= N) continue;
          long long hi = 0, lo = 0;
#pragma unroll
          for (int m = 0; m < 4; ++m) hi = (hi << SB) + (long long)__float2int_rn(__uint_as_float(v[m][u]));
#pragma unroll
          for (int m = 4; m < S; ++m) lo = (lo << SB) + (long long)__float2int_rn(__uint_as_float(v[m][u]));
          epi(rl, r, cl, col, ozaki::combine_hilo<S, (S <= 7 ? 7 : 6)>(hi, lo, eA[rl] + eB[cl]));
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::dealloc(taddr, TCOLS);
  return failed != 0;
}

template <int OP, int S, int SH>
__global__ void __launch_bounds__(256, oz_tc_minb(S, SH)) oz_prod_tc_kernel(const WalkerDev* __restrict__ W, int mode,
                                                                            int j, int q) {
  constexpr int MT = 128, NT = oz_tc_nt(S, SH), NS = oz_tc_stages(S, SH);
  const int wi = blockIdx.z >> 1, sp = blockIdx.z & 1;
  const WalkerDev& w = W[wi];
  if (w.path != 2 || w.cb || sp >= w.S || w.slices != S) return;
  int t;
  if (!oz_slice_of(w, mode, j, q, t)) return;
  const int N = w.N, ldk = w.ldk;
  const int r0 = blockIdx.y * MT, c0 = blockIdx.x * NT;
  if (r0 >= N || c0 >= N) return;
  const long long NN = (long long)N * N;
  const long long sstride = (long long)ozaki::tc_slice_elems(N, ldk);
  const unsigned short* ws = w.sl + (long long)sp * w.slices * sstride;
  const int* we = w.sle + (long long)sp * N;
  ProdJob job{};
  double* out = nullptr;
  switch (OP) {
    case OZ_WL_FWD: job = ProdJob{w.kA, ws, w.kAe, we}; out = w.work + sp * NN; break;
    case OZ_WR_FWD: job = ProdJob{ws, w.iB, we, w.iBe}; out = w.G + sp * NN; break;
    case OZ_CH_FWD: job = ProdJob{w.kA, ws, w.kAe, we}; out = oz_chain(w, sp, (q + 1) & 1); break;
    case OZ_CH_BWD: job = ProdJob{w.kB, ws, w.kBe, we}; out = oz_chain(w, sp, (q + 1) & 1); break;
    case OZ_WR_BWD: job = ProdJob{ws, w.kB, we, w.kBe}; out = w.work + sp * NN; break;
    case OZ_WL_BWD: job = ProdJob{w.iA, ws, w.iAe, we}; out = w.G + sp * NN; break;
    case OZ_DT0: job = ProdJob{w.kA, ws, w.kAe, we}; out = w.gt0 ? oz_dyn(w.gt0, w, sp, t) : nullptr; break;
    case OZ_D0T: job = ProdJob{ws, w.iB, we, w.iBe}; out = w.g0t ? oz_dyn(w.g0t, w, sp, t) : nullptr; break;
  }
  if (!out) return;
  extern __shared__ __align__(1024) unsigned char tsm[];
  __shared__ double s_scale[MT];  // exp(+-alpha s) of the output rows (or columns); read after the tile's barriers
  const int tid = threadIdx.x;
  constexpr bool row_scale = OP == OZ_WL_FWD || OP == OZ_CH_FWD || OP == OZ_DT0;
  constexpr bool col_scale = OP == OZ_WR_FWD || OP == OZ_D0T;
  if (row_scale) {
    if (tid < MT) s_scale[tid] = (r0 + tid < N) ? oz_bscale(w, t, sp, +1, r0 + tid) : 0.0;
  } else if (col_scale) {
    if (tid < NT) s_scale[tid] = (c0 + tid < N) ? oz_bscale(w, t, sp, -1, c0 + tid) : 0.0;
  }
  const bool failed = oz_tc_tile<S, NT, NS, oz_tc_minb(S, SH)>(
      job, N, ldk, r0, c0, w.wait_limit, tsm, [&](int rl, int r, int cl, int col, double val) {
        if (row_scale) val *= s_scale[rl];
        if (col_scale) val *= s_scale[cl];
        out[(long long)col * N + r] = val;
      });
  if (failed && tid == 0) atomicOr(w.status, ST_TIMEOUT);
}

// constant operands (exp(-dtau K), exp(+dtau K)), sliced once per batch
__global__ void __launch_bounds__(256) oz_const_slice_kernel(const double* X, unsigned short* out, int* exps, int N,
                                                             int ldk, int role, int bits, int slices) {
  SliceJob job{X, out, exps, nullptr};
  slice_lines(job, N, ldk, role, bits, slices, blockIdx.x * 32);
}

// ---- stand-alone product C = A B: A, B column-major N x N on the device -----------
// One product is a matter of latency: both operands are sliced by one launch (8 lines a CTA, 8
// consecutive k a thread, so that every element is read once from its own sector and each slice is
// a 16-byte store), and the tiles run the sweep's tensor-core loop.  N = 256: 27 us a product, bound
// by the two launches and the 16 chunks of a tile one after the other; 74 us as two slicing launches
// of 32 lines a CTA and a 64 x 64-tile mma.sync product.
__global__ void __launch_bounds__(256) oz_slice_pair_kernel(const double* A, const double* B, unsigned short* sa,
                                                            int* ea, unsigned short* sb, int* eb, int N, int ldk,
                                                            int bits, int slices) {
  const bool isB = blockIdx.y == 1;
  const double* X = isB ? B : A;
  unsigned short* out = isB ? sb : sa;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // A's lines are rows (8 consecutive elements of a column), B's are columns
  const int ll = isB ? warp : lane & 7, kg = isB ? lane : warp * 4 + (lane >> 3), line = blockIdx.x * 8 + ll;
  __shared__ int s_e[8];
  if (tid < 8) s_e[tid] = -1100;
  __syncthreads();
  double x[8];
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + kg * 8 + u;
      x[u] = (line < N && k < N) ? (isB ? X[(long long)line * N + k] : X[(long long)k * N + line]) : 0.0;
    }
  };
  int e = -1100;
  for (int k0 = 0; k0 < ldk; k0 += 256) {
    load(k0);
#pragma unroll
    for (int u = 0; u < 8; ++u) e = max(e, ozaki::exp_bound(x[u]));
  }
  atomicMax(&s_e[ll], e);
  __syncthreads();
  e = s_e[ll];
  if (tid < 8 && blockIdx.x * 8 + tid < N) (isB ? eb : ea)[blockIdx.x * 8 + tid] = s_e[tid];
  if (line >= N) return;
  const int Q = bits * slices;
  const long long sstride = (long long)ozaki::tc_slice_elems(N, ldk);
  for (int k0 = 0; k0 < ldk; k0 += 256) {
    const int k = k0 + kg * 8;
    if (k >= ldk) break;
    if (ldk > 256) load(k0);
    unsigned long long q[8];
    bool ng[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) q[u] = ozaki::fixedq(x[u], e, Q, ng[u]);
    unsigned short* o = out + ozaki::tc_index(line, k, ozaki::tc_lines(N) / 8);
    for (int s2 = 0; s2 < slices; ++s2) {
      unsigned v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        v[u] = (unsigned)ozaki::slice_bf16q(q[2 * u], s2, bits, Q, ng[2 * u]) |
               ((unsigned)ozaki::slice_bf16q(q[2 * u + 1], s2, bits, Q, ng[2 * u + 1]) << 16);
      *reinterpret_cast<uint4*>(o + s2 * sstride) = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
}

// 128 x 32 tiles, the deepest ring that fits (one CTA per SM: a product has few tiles)
__host__ __device__ constexpr int oz_one_stages(int S) { return S <= 7 ? 6 : 5; }
template <int S>
__global__ void __launch_bounds__(256, 1) oz_one_prod_kernel(ProdJob job, double* C, int N, int ldk) {
  extern __shared__ __align__(1024) unsigned char tsm[];
  // a wait that runs out leaves the tile unwritten: no status word here, the caller's C shows NaN
  const int r0 = blockIdx.y * 128, c0 = blockIdx.x * 32;
  const bool failed = oz_tc_tile<S, 32, oz_one_stages(S), 1>(
      job, N, ldk, r0, c0, kDefaultWaitLimit, tsm,
      [&](int, int r, int, int col, double val) { C[(long long)col * N + r] = val; });
  if (failed)
    for (int e = threadIdx.x; e < 128 * 32; e += 256) {
      const int r = r0 + (e & 127), col = c0 + (e >> 7);
      if (r < N && col < N) C[(long long)col * N + r] = __longlong_as_double(0x7ff8000000000000LL);
    }
}

static size_t oz_tc_smem(int S, int SH) { return (size_t)oz_tc_stages(S, SH) * oz_tc_stage_bytes(S, SH); }
static size_t oz_one_smem(int S) { return (size_t)oz_one_stages(S) * oztc::stage_bytes(S, 128, 32); }

cudaError_t configure_ozaki_kernels() {
  cudaError_t e;
#define OZCFG(OP)                                                                                         \
  if ((e = cudaFuncSetAttribute(oz_prod_tc_kernel<OP, 7, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                (int)oz_tc_smem(7, 0))) ||                                                 \
      (e = cudaFuncSetAttribute(oz_prod_tc_kernel<OP, 8, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                (int)oz_tc_smem(8, 0))) ||                                                 \
      (e = cudaFuncSetAttribute(oz_prod_tc_kernel<OP, 7, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                (int)oz_tc_smem(7, 1))) ||                                                 \
      (e = cudaFuncSetAttribute(oz_prod_tc_kernel<OP, 8, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                (int)oz_tc_smem(8, 1))))                                                   \
  return e
  OZCFG(OZ_WL_FWD); OZCFG(OZ_WR_FWD); OZCFG(OZ_CH_FWD); OZCFG(OZ_CH_BWD);
  OZCFG(OZ_WR_BWD); OZCFG(OZ_WL_BWD); OZCFG(OZ_DT0); OZCFG(OZ_D0T);
#undef OZCFG
  if ((e = cudaFuncSetAttribute(oz_one_prod_kernel<7>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)oz_one_smem(7))) ||
      (e = cudaFuncSetAttribute(oz_one_prod_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)oz_one_smem(8))))
    return e;
  return cudaSuccess;
}

// tile shape of the products issued by this host thread (the issuing batch's tuned shape)
static thread_local int g_oz_shape = 0;
void oz_set_shape(int shape) { g_oz_shape = shape ? 1 : 0; }

template <int OP, int SH>
static void oz_op_shape(const WalkerDev* W, int nw, int maxN, int mode, int j, int q, cudaStream_t st) {
  const dim3 g7((maxN + oz_tc_nt(7, SH) - 1) / oz_tc_nt(7, SH), (maxN + 127) / 128, 2 * nw);
  oz_prod_tc_kernel<OP, 7, SH><<<g7, 256, oz_tc_smem(7, SH), st>>>(W, mode, j, q);
  if (maxN > 256) {
    const dim3 g8((maxN + oz_tc_nt(8, SH) - 1) / oz_tc_nt(8, SH), (maxN + 127) / 128, 2 * nw);
    oz_prod_tc_kernel<OP, 8, SH><<<g8, 256, oz_tc_smem(8, SH), st>>>(W, mode, j, q);
  }
}

template <int OP>
static void oz_op(const WalkerDev* W, int nw, int maxN, int mode, int j, int q, cudaStream_t st) {
  oz_slice_kernel<OP><<<dim3((maxN + 31) / 32, 2 * nw), 256, 0, st>>>(W, mode, j, q);
  if (g_oz_shape) oz_op_shape<OP, 1>(W, nw, maxN, mode, j, q, st);
  else oz_op_shape<OP, 0>(W, nw, maxN, mode, j, q, st);
}

// the slice work of mixed walkers (wraps and chain through the tensor cores)
void mixed_wrap_fwd(const WalkerDev* W, int nw, int maxN, int j, int q, cudaStream_t st) {
  oz_op<OZ_WL_FWD>(W, nw, maxN, MODE_FWD, j, q, st);
  oz_op<OZ_WR_FWD>(W, nw, maxN, MODE_FWD, j, q, st);
}
void mixed_chain(const WalkerDev* W, int nw, int maxN, int mode, int j, int q, cudaStream_t st) {
  if (mode == MODE_FWD) oz_op<OZ_CH_FWD>(W, nw, maxN, mode, j, q, st);
  else oz_op<OZ_CH_BWD>(W, nw, maxN, mode, j, q, st);
}
// the time-displaced steps of the dynamic half-sweep for mixed walkers
void mixed_dynamic_prop(const WalkerDev* W, int nw, int maxN, int j, int q, cudaStream_t st) {
  oz_op<OZ_DT0>(W, nw, maxN, MODE_FWD, j, q, st);
  oz_op<OZ_D0T>(W, nw, maxN, MODE_FWD, j, q, st);
}
void mixed_wrap_bwd(const WalkerDev* W, int nw, int maxN, int j, int q, cudaStream_t st) {
  oz_op<OZ_WR_BWD>(W, nw, maxN, MODE_BWD, j, q, st);
  oz_op<OZ_WL_BWD>(W, nw, maxN, MODE_BWD, j, q, st);
}

void oz_slice_const(const double* X, unsigned short* out, int* exps, int N, int ldk, int role, int bits, int slices,
                    cudaStream_t st) {
  oz_const_slice_kernel<<<(N + 31) / 32, 256, 0, st>>>(X, out, exps, N, ldk, role, bits, slices);
}

void oz_selftest(const double* A, const double* B, double* C, unsigned short* sa, int* ea, unsigned short* sb, int* eb,
                 int N, cudaStream_t st) {
  const ozaki::SliceCfg cfg = ozaki::cfg_for_k(N);
  const int ldk = (N + 15) / 16 * 16;
  oz_slice_pair_kernel<<<dim3((N + 7) / 8, 2), 256, 0, st>>>(A, B, sa, ea, sb, eb, N, ldk, cfg.bits, cfg.slices);
  const dim3 g((N + 31) / 32, (N + 127) / 128);
  const ProdJob job{sa, sb, ea, eb};
  if (cfg.slices == 7) oz_one_prod_kernel<7><<<g, 256, oz_one_smem(7), st>>>(job, C, N, ldk);
  else oz_one_prod_kernel<8><<<g, 256, oz_one_smem(8), st>>>(job, C, N, ldk);
}

}  // namespace dqmc
