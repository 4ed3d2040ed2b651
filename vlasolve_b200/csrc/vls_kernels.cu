// vls_kernels.cu -- sm_100a kernels of the split semi-Lagrangian step.
//
// Per step (linked mode, vlasovSolver21_spline.hxx:680-801):
//   scan      radial moment partials -> bins -> enclosed mass -> kick shift
//   ucol      per (J slice, strip of r columns): natural-BC spline solve along
//             u, kick gather at U+shift(r), second solve along u of the kicked
//             values -> G (u-direction coefficients of the kicked f)
//   prer      per (J slice, rows of G): solve along r -> C (2D coefficients)
//   edge      per delayed-kernel chain: spline value at the chain tail; for the
//             persistent strip drift also the chain fronts' and the far cells'
//             values, into f
//   drift     per cell: 4x4 gather of C at the host-tabulated footpoint, or the
//             delayed-kernel ring-buffer front (persistent strips: what edge
//             left in f), or 0; radial moment partials of the result (the next
//             step's moment) in the epilogue
//
// The 2D prefilter of the reference (r-solves, then u-solves on every column,
// localSpline.hxx:1238-1258) is applied here as u-solves then r-solves; the
// tensor-product operator is the same.  The Thomas recursion of one line
// (localSpline.hxx:953-1182) is split into segments that run in parallel:
// each segment first replays K rows of the recursion before its start (the
// forward and backward recursions contract by 2-sqrt(3) = 0.268 per row, so
// K = 32 rows reach FP64 rounding and K = 20 rows reach 1e-11).  The per-row
// coefficients are the reference's own (tabulated on the host in its
// operation order).  Recursions run in FP64 in both precisions.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>

#include "vls_async.cuh"
#include "vls_dd.cuh"
#include "vls_internal.h"

namespace vls {

// warm-up rows of a segment: FP64 storage needs the recursion to contract to
// FP64 rounding (0.268^32 = 5e-19), FP32 storage to well below FP32 rounding
// (0.268^16 = 7e-10)
template <typename T>
struct Prec;
template <>
struct Prec<double> {
  static constexpr int K = 32;
};
template <>
struct Prec<float> {
  static constexpr int K = 16;
};

template <typename T>
__device__ __forceinline__ T bv2(T x) {
  return x * x * x;
}
template <typename T>
__device__ __forceinline__ T bv1(T x) {
  return T(1) + T(3) * x + T(3) * x * x - T(3) * x * x * x;
}

// s / 36 without the bias of a rounded 1/36 factor: in FP32 the constant is
// split in two floats (hi + lo = 1/36 to 1e-17), so the product carries only
// the final rounding.  A biased factor would scale every drifted value the
// same way in every step and show up as a steady mass drift.
template <typename T>
__device__ __forceinline__ T over36(T s) {
  return s * (T(1) / T(36));
}
template <>
__device__ __forceinline__ float over36<float>(float s) {
  return __fmaf_rn(s, 0.02777777798473835f, s * -2.0696057367874943e-10f);
}

// ----------------------------------------------------------- async copies
// cp.async (LDGSTS): element-wise global -> shared copies that stay in flight
// together; the tiles' global rows are only 4-byte aligned (r-pitch N_r).
template <typename T>
__device__ __forceinline__ void cp_async(T *smem, const T *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem),
               "n"((int)sizeof(T))
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// ----------------------------------------------------------- segment solve
// One line of the padded natural-BC system lives at b[k*ks], k = 0..M-1.  On
// entry rows 1..M-2 hold the data; on exit rows 0..M-1 hold the coefficients.
// A thread owns interior rows [k0, k1).  The four stages are separated by
// __syncthreads() (see solve_lines).  R is the arithmetic of the recursion.
// The per-row coefficients rp_k, q_k are read from shared memory for rows
// below kc and replaced by their limits from row kc on (they are equal there
// in the recursion's precision), which removes two shared loads per element.
template <typename R>
struct Coef {
  const R *rp, *q;
  R rpi, qi, sixth;
  int kc;
  __device__ __forceinline__ R rpk(int k) const { return k < kc ? rp[k] : rpi; }
  __device__ __forceinline__ R qk(int k) const { return k < kc ? q[k] : qi; }
};

template <int K, typename R>
struct Seg {
  template <typename S>
  __device__ __forceinline__ static R fwd_warm(const S *b, int ks, int k0, const Coef<R> &cf) {
    R d = R(0);
    int ks0 = k0 - K;
    if (ks0 < 1) ks0 = 1;
#pragma unroll 4
    for (int k = ks0; k < k0; ++k) d = ((R)b[k * ks] - d * cf.sixth) * cf.rpk(k);
    return d;
  }
  template <typename S>
  __device__ __forceinline__ static void fwd_main(S *b, int ks, int k0, int k1, R d,
                                  const DirTables &t, const Coef<R> &cf) {
    R dprev = d;
    int k = k0;
    const int kt = min(k1, max(k0, cf.kc));
#pragma unroll 4
    for (; k < kt; ++k) {
      dprev = d;
      d = ((R)b[k * ks] - d * cf.sixth) * cf.rp[k];
      b[k * ks] = (S)d;
    }
#pragma unroll 4
    for (; k < k1; ++k) {
      dprev = d;
      d = ((R)b[k * ks] - d * cf.sixth) * cf.rpi;
      b[k * ks] = (S)d;
    }
    if (k1 == t.M - 1 && k1 > k0) {
      // last row (localSpline.hxx:1145-1152): d = d_{M-2}, dprev = d_{M-3}
      const R num = (R(0) - (R)t.hi2 * dprev) - (R)t.L1 * d;
      b[(t.M - 1) * ks] = (S)(num / (R)t.L2);
    }
  }
  template <typename S>
  __device__ __forceinline__ static R bwd_warm(const S *b, int ks, int k1, const DirTables &t,
                               const Coef<R> &cf) {
    int kst = k1 + K - 1;
    R c;
    if (kst >= t.M - 2) {
      kst = t.M - 2;
      c = (R)b[(t.M - 1) * ks];
    } else {
      c = R(0);
    }
#pragma unroll 4
    for (int k = kst; k >= k1; --k) c = (R)b[k * ks] - cf.qk(k) * c;
    return c;
  }
  template <typename S>
  __device__ __forceinline__ static void bwd_main(S *b, int ks, int k0, int k1, R c,
                                  const DirTables &t, const Coef<R> &cf) {
    R cnext = c;
    int k = k1 - 1;
    const int kt = max(k0, cf.kc);
#pragma unroll 4
    for (; k >= kt; --k) {
      cnext = c;
      c = (R)b[k * ks] - cf.qi * c;
      b[k * ks] = (S)c;
    }
#pragma unroll 4
    for (; k >= k0; --k) {
      cnext = c;
      c = (R)b[k * ks] - cf.q[k] * c;
      b[k * ks] = (S)c;
    }
    if (k0 == 1 && k1 > k0) {
      // first row (localSpline.hxx:1171): c_0 = (0 - a01 c_1) - a02 c_2
      b[0] = (S)((R(0) - (R)t.a01 * c) - (R)t.a02 * cnext);
    }
  }
};

// segment bounds: interior rows [1, M-1) split into nseg pieces of odd length
__device__ __forceinline__ void seg_bounds(int M, int nseg, int s, int &k0,
                                           int &k1) {
  int n = M - 2;
  int L = (n + nseg - 1) / nseg;
  L |= 1;
  k0 = 1 + s * L;
  k1 = k0 + L;
  if (k0 > M - 1) k0 = M - 1;
  if (k1 > M - 1) k1 = M - 1;
}

// rp, q: the direction's tables in the recursion type (shared memory)
template <int K, typename R, typename S>
__device__ __forceinline__ void solve_lines(S *base, int ks, int k0, int k1,
                            const DirTables &t, const R *rp, const R *q) {
  Coef<R> cf;
  cf.rp = rp;
  cf.q = q;
  cf.rpi = (R)t.rp_inf;
  cf.qi = (R)t.q_inf;
  cf.sixth = R(1) / R(6);
  cf.kc = sizeof(R) == 4 ? t.kc32 : t.kc64;
  R d = Seg<K, R>::fwd_warm(base, ks, k0, cf);
  __syncthreads();
  Seg<K, R>::fwd_main(base, ks, k0, k1, d, t, cf);
  __syncthreads();
  R c = Seg<K, R>::bwd_warm(base, ks, k1, t, cf);
  __syncthreads();
  Seg<K, R>::bwd_main(base, ks, k0, k1, c, t, cf);
  __syncthreads();
}

// copies the direction's Thomas tables into shared memory as type R
template <typename R>
__device__ __forceinline__ void load_tables(R *rp, R *q, const DirTables &t) {
  for (int k = threadIdx.x; k < t.M; k += blockDim.x) {
    rp[k] = (R)__ldg(t.rp + k);
    q[k] = (R)__ldg(t.q + k);
  }
}

__host__ __device__ constexpr size_t align16(size_t b) { return (b + 15) / 16 * 16; }

// ------------------------------------------------------------------ ucol
// Block: TW columns (r) x NSEG segments (u), lane = column, so a shared row
// access by a warp is one (FP32) or two (FP64) wavefronts.  Shared memory:
// the Thomas tables and two buffers of (N_u+3) rows x TW in the recursion
// type R (row N_u+2 is an always-zero guard row); global f and G are type T,
// so T -> R and R -> T conversions happen once per element, at the tile load
// and at the tile store.
constexpr int UC_THREADS = 256;
template <typename R>
struct UcolCfg {
  static constexpr int TW = sizeof(R) == 4 ? 16 : 8;
  static constexpr int NSEG = UC_THREADS / TW;
};

// loads rows 1..nu of a TW-column tile of f (r0.., slice base fs) into buf
template <typename T, typename R, int TW>
__device__ __forceinline__ void load_col_tile(R *buf, const T *__restrict__ fs,
                                              int nu, int nr, int r0) {
  if constexpr (sizeof(T) == sizeof(R)) {
    for (int e = threadIdx.x; e < nu * TW; e += blockDim.x) {
      const int k = e / TW + 1, c = e % TW;
      const int rr = r0 + c;
      if (rr < nr)
        cp_async(reinterpret_cast<T *>(&buf[k * TW + c]), fs + (size_t)(k - 1) * nr + rr);
      else
        buf[k * TW + c] = R(0);
    }
    cp_async_wait_all();
  } else {
    // four loads in flight per thread, then convert
    const int n = nu * TW;
    for (int e0 = threadIdx.x; e0 < n; e0 += 4 * blockDim.x) {
      T v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = e0 + q * blockDim.x;
        const int k = e / TW + 1, c = e % TW, rr = r0 + c;
        v[q] = (e < n && rr < nr) ? __ldg(fs + (size_t)(k - 1) * nr + rr) : T(0);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = e0 + q * blockDim.x;
        if (e < n) buf[(e / TW + 1) * TW + e % TW] = (R)v[q];
      }
    }
  }
}

// exact per-cell kick index computation (vlasovSolver21_spline.hxx:760-762,
// localSpline.hxx:426-429), used where the column's fractional shift lies
// within 1e-9 of a node
template <typename R, int TW>
__device__ __forceinline__ R kick_exact(const R *cb, const Geometry &g, int u,
                                        double s) {
  const double newU = __ldg(g.U + u) + s;
  if (!(newU > g.u0 && newU < g.umax)) return R(0);  // outside (or NaN) -> 0
  const double y = (newU - g.su) * g.hu;
  const double fl = floor(y);
  const R fr = (R)(y - fl);
  const int Ny = 1 + (int)fl;
  return (bv2<R>(R(1) - fr) * cb[(Ny - 1) * TW] + bv1<R>(R(1) - fr) * cb[Ny * TW] +
          bv1<R>(fr) * cb[(Ny + 1) * TW] + bv2<R>(fr) * cb[(Ny + 2) * TW]) /
         R(6);
}

// TW columns per block (UcolCfg<R>::TW, or half of it where two buffers of
// that many long columns exceed a block's shared memory)
template <typename T, typename R, bool KICK, int TW>
__global__ void __launch_bounds__(UC_THREADS)
    ucol_kernel(const T *__restrict__ f, T *__restrict__ G,
                const double *__restrict__ shift, Geometry g, DirTables tu) {
  constexpr int NSEG = UC_THREADS / TW;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int M = g.nu + 2;
  const int rows = M + 1;
  R *rp = reinterpret_cast<R *>(smem_raw);
  R *qq = rp + M;
  R *bufA = reinterpret_cast<R *>(smem_raw + align16(2 * M * sizeof(R)));
  R *bufB = bufA + (size_t)rows * TW;
  const int tid = threadIdx.x;
  const int col = tid % TW;
  const int seg = tid / TW;
  const int r0 = blockIdx.x * TW;
  const int jl = blockIdx.y;        // slice within the batch (scratch index)
  const int j = g.j0 + jl;          // global slice
  const int r = r0 + col;

  load_tables<R>(rp, qq, tu);
  if (tid < TW) {
    bufA[0 * TW + tid] = R(0);
    bufA[(M - 1) * TW + tid] = R(0);
    bufA[M * TW + tid] = R(0);
    bufB[0 * TW + tid] = R(0);
    bufB[(M - 1) * TW + tid] = R(0);
    bufB[M * TW + tid] = R(0);
  }
  load_col_tile<T, R, TW>(bufA, f + (size_t)j * g.nu * g.nr, g.nu, g.nr, r0);
  __syncthreads();
  int k0, k1;
  seg_bounds(M, NSEG, seg, k0, k1);
  solve_lines<Prec<T>::K, R>(bufA + col, TW, k0, k1, tu, rp, qq);

  R *out = bufA;
  if (KICK) {
    // kick (vlasovSolver21_spline.hxx:758-763, localSpline.hxx:423-441 with
    // the r-direction (1,4,1)/6 weights folded into the u-only coefficients).
    // The shift is constant along the column and the u grid is uniform, so
    // y_u = u + s*hu: one fraction and one integer offset serve every row,
    // unless that fraction is within 1e-9 of a node (then every row takes
    // the exact per-cell path).
    const double s = (r < g.nr) ? __ldg(shift + r) : 0.0;
    const double qf = s * g.hu;
    const double fl = floor(qf);
    const double frd = qf - fl;
    const bool fast = frd > 1e-9 && frd < 1.0 - 1e-9 && fabs(qf) < 1e6;
    const int o = fast ? (int)fl : 0;
    const R fr = (R)frd;
    const R w0 = bv2<R>(R(1) - fr) / R(6), w1 = bv1<R>(R(1) - fr) / R(6);
    const R w2 = bv1<R>(fr) / R(6), w3 = bv2<R>(fr) / R(6);
    // rows with 0 < u + qf < nu - 1 are inside (strictly, as :761)
    const int ulo = fast ? (int)floor(-qf) + 1 : 0;
    const int uhi = fast ? (int)ceil((double)(g.nu - 1) - qf) - 1 : -1;
    const R *cb = bufA + col;
    if (fast) {
#pragma unroll 4
      for (int k = k0; k < k1; ++k) {
        const int u = k - 1;
        R v = R(0);
        if (u >= ulo && u <= uhi) {
          const R *p = cb + (k + o - 1) * TW;
          v = w0 * p[0] + w1 * p[TW] + w2 * p[2 * TW] + w3 * p[3 * TW];
        }
        bufB[k * TW + col] = v;
      }
    } else {
      for (int k = k0; k < k1; ++k) bufB[k * TW + col] = kick_exact<R, TW>(cb, g, k - 1, s);
    }
    __syncthreads();
    solve_lines<Prec<T>::K, R>(bufB + col, TW, k0, k1, tu, rp, qq);
    out = bufB;
  }
  T *Gs = G + (size_t)jl * M * g.gp;
  for (int e = tid; e < M * TW; e += UC_THREADS) {
    const int k = e / TW, c = e % TW;
    const int rr = r0 + c;
    if (rr < g.nr) Gs[(size_t)k * g.gp + rr] = (T)out[k * TW + c];
  }
}

template <typename T, typename R>
cudaError_t launch_ucol(bool kick, const T *f, T *G, const double *shift,
                        const Geometry &g, const DirTables &tu, cudaStream_t st) {
  constexpr int TW = UcolCfg<R>::TW;
  auto smem_for = [&](int tw) {
    return align16(2 * (size_t)(g.nu + 2) * sizeof(R)) + 2 * (size_t)(g.nu + 3) * tw * sizeof(R);
  };
  auto go = [&](auto kern, int tw) {
    const size_t smem = smem_for(tw);
    dim3 grid((g.nr + tw - 1) / tw, g.nb);
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, UC_THREADS, smem, st>>>(f, G, shift, g, tu);
    return cudaGetLastError();
  };
  // 227 KB per block: FP64 columns of more than ~1600 rows take half the columns
  if (smem_for(TW) > 232448)
    return kick ? go(ucol_kernel<T, R, true, TW / 2>, TW / 2)
                : go(ucol_kernel<T, R, false, TW / 2>, TW / 2);
  return kick ? go(ucol_kernel<T, R, true, TW>, TW) : go(ucol_kernel<T, R, false, TW>, TW);
}

// ------------------------------------------------------------------ prer
// Block: ROWS rows of G (lane = row) x NSEG long segments along r.  The
// shared row pitch is 1 mod 32 (FP32) or odd (FP64) so that the lanes, which
// walk different rows at the same column, hit distinct banks.  Shared rows
// are in the recursion type R.
template <typename R>
struct PrerCfg {
  static constexpr int ROWS = sizeof(R) == 4 ? 32 : 16;
  static constexpr int NSEG = 8;
  static constexpr int THREADS = ROWS * NSEG;
};

__host__ __device__ inline int prer_pitch(int M, int elem) {
  int P = M + 1;
  if (elem == 4)
    P = (P + 31) / 32 * 32 + 1;
  else
    P |= 1;
  return P;
}

// ROWS rows of G per block (PrerCfg<R>::ROWS, or half of it where a tile of
// that many long rows exceeds a block's shared memory)
template <typename T, typename R, int ROWS>
__global__ void __launch_bounds__(ROWS * PrerCfg<R>::NSEG)
    prer_kernel(const T *__restrict__ G, T *__restrict__ C, Geometry g,
                DirTables tr) {
  constexpr int NSEG = PrerCfg<R>::NSEG, NT = ROWS * NSEG;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int M = g.nr + 2;
  const int LS = prer_pitch(M, sizeof(R));
  R *rp = reinterpret_cast<R *>(smem_raw);
  R *qq = rp + M;
  R *buf = reinterpret_cast<R *>(smem_raw + align16(2 * M * sizeof(R)));
  const int tid = threadIdx.x;
  const int rho = tid % ROWS;
  const int seg = tid / ROWS;
  const int j = blockIdx.y;  // slice within the batch (G and C are batch scratch)
  const int kr0 = blockIdx.x * ROWS;
  const int nrows = g.nu + 2;
  const T *Gs = G + (size_t)j * nrows * g.gp;
  load_tables<R>(rp, qq, tr);
  // rows of the tile, each copied by the whole block (no index division)
  for (int p = 0; p < ROWS; ++p) {
    const int kr = kr0 + p;
    R *dst = buf + p * LS + 1;
    if (kr < nrows) {
      const T *src = Gs + (size_t)kr * g.gp;
      if constexpr (sizeof(T) == sizeof(R)) {
        for (int k = tid; k < g.nr; k += NT) cp_async(reinterpret_cast<T *>(dst + k), src + k);
      } else {
        for (int k = tid; k < g.nr; k += NT) dst[k] = (R)__ldg(src + k);
      }
    } else {
      for (int k = tid; k < g.nr; k += NT) dst[k] = R(0);
    }
  }
  if constexpr (sizeof(T) == sizeof(R)) cp_async_wait_all();
  __syncthreads();
  int k0, k1;
  seg_bounds(M, NSEG, seg, k0, k1);
  solve_lines<Prec<T>::K, R>(buf + rho * LS, 1, k0, k1, tr, rp, qq);
  T *Cs = C + (size_t)j * (g.nu + 3) * g.pc;
  for (int p = 0; p < ROWS; ++p) {
    const int kr = kr0 + p;
    if (kr >= nrows) break;
    T *dst = Cs + (size_t)kr * g.pc;
    const R *src = buf + p * LS;
    for (int k = tid; k < M; k += NT) dst[k] = (T)src[k];
  }
}

template <typename T, typename R>
cudaError_t launch_prer(const T *G, T *C, const Geometry &g, const DirTables &tr,
                        cudaStream_t st) {
  constexpr int ROWS = PrerCfg<R>::ROWS, NSEG = PrerCfg<R>::NSEG;
  const int M = g.nr + 2;
  auto smem_for = [&](int rows) {
    return align16(2 * (size_t)M * sizeof(R)) +
           (size_t)rows * prer_pitch(M, sizeof(R)) * sizeof(R);
  };
  // 227 KB per block: FP64 rows of more than ~1600 columns take half the rows
  if (smem_for(ROWS) > 232448) {
    constexpr int H = ROWS / 2;
    const size_t smem = smem_for(H);
    dim3 grid((g.nu + 2 + H - 1) / H, g.nb);
    cudaError_t e = cudaFuncSetAttribute(
        prer_kernel<T, R, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    prer_kernel<T, R, H><<<grid, H * NSEG, smem, st>>>(G, C, g, tr);
    return cudaGetLastError();
  }
  const size_t smem = smem_for(ROWS);
  dim3 grid((g.nu + 2 + ROWS - 1) / ROWS, g.nb);
  cudaError_t e = cudaFuncSetAttribute(
      prer_kernel<T, R, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  prer_kernel<T, R, ROWS><<<grid, ROWS * NSEG, smem, st>>>(G, C, g, tr);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ gather
// localSpline::evaluateC(int,double,int,double), localSpline.hxx:381-398:
// taps at padded columns rI..rI+3 and rows uI..uI+3 (FP64 form).
template <typename T>
__device__ __forceinline__ T eval2d(const T *Cj, int pc, int rI, T x, int uI, T y) {
  const T b2xI = bv2<T>(T(1) - x), b1xI = bv1<T>(T(1) - x);
  const T b1x = bv1<T>(x), b2x = bv2<T>(x);
  const T *p = Cj + (size_t)uI * pc + rI;
  const T s0 = p[0] * b2xI + p[1] * b1xI + p[2] * b1x + p[3] * b2x;
  p += pc;
  const T s1 = p[0] * b2xI + p[1] * b1xI + p[2] * b1x + p[3] * b2x;
  p += pc;
  const T s2 = p[0] * b2xI + p[1] * b1xI + p[2] * b1x + p[3] * b2x;
  p += pc;
  const T s3 = p[0] * b2xI + p[1] * b1xI + p[2] * b1x + p[3] * b2x;
  return over36<T>(bv2<T>(T(1) - y) * s0 + bv1<T>(T(1) - y) * s1 +
                           bv1<T>(y) * s2 + bv2<T>(y) * s3);
}

// FP32 form with packed f32x2 arithmetic: the x and y weights are computed
// pairwise, and rows (0,1) and (2,3) are accumulated pairwise.
//
// Difference form: with c the tap at (row 1, column 1), the value is
// c + (1/36) sum w_x w_y (C - c), which equals (1/36) sum w_x w_y C because
// the cubic B-spline weights of each direction sum to 6.  In FP32 the
// rounded weights do not sum to 6 exactly and the rounding of the 16 products
// is proportional to C; both errors are the same in every step of a nearly
// stationary state (the footpoints, hence the weights, never change), so
// they add up coherently over thousands of steps.  Taken on the differences
// C - c, which are small where f is smooth, they shrink by the same factor:
// over 2000 Plummer steps on 257 x 257 x 64 the energy drift of the FP32 path
// stays 9e-7 off the FP64 path's (rms over 40 scale radii), with 1.7e-6 for
// undivided taps at the one radius where the difference form gave 1.5e-7.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// tap (a, b) = row a, column b of the 4 x 4 block, from ld(a, b)
template <class Ld>
__device__ __forceinline__ float gather_f32x2(const Ld &ld, float x, float y) {
  const float2 t = f2(x, y);
  const float2 one = f2(1.f, 1.f), three = f2(3.f, 3.f), m3 = f2(-3.f, -3.f);
  const float2 sv = __fadd2_rn(one, f2(-t.x, -t.y));  // 1 - t
  const float2 t2 = __fmul2_rn(t, t), t3 = __fmul2_rn(t2, t);
  const float2 s2 = __fmul2_rn(sv, sv), s3 = __fmul2_rn(s2, sv);
  // BV1(v) = 1 + 3v + 3v^2 - 3v^3
  const float2 a1 = __ffma2_rn(m3, s3, __ffma2_rn(three, s2, __ffma2_rn(three, sv, one)));
  const float2 b1 = __ffma2_rn(m3, t3, __ffma2_rn(three, t2, __ffma2_rn(three, t, one)));
  // x weights: (s3.x, a1.x, b1.x, t3.x); y weights: (s3.y, a1.y, b1.y, t3.y)
  const float2 wx0 = f2(s3.x, s3.x), wx1 = f2(a1.x, a1.x), wx2 = f2(b1.x, b1.x),
               wx3 = f2(t3.x, t3.x);
  const float c = ld(1, 1);
  const float2 mc = f2(-c, -c);
  float2 r01 = __fmul2_rn(__fadd2_rn(f2(ld(0, 0), ld(1, 0)), mc), wx0);
  r01 = __ffma2_rn(__fadd2_rn(f2(ld(0, 1), c), mc), wx1, r01);
  r01 = __ffma2_rn(__fadd2_rn(f2(ld(0, 2), ld(1, 2)), mc), wx2, r01);
  r01 = __ffma2_rn(__fadd2_rn(f2(ld(0, 3), ld(1, 3)), mc), wx3, r01);
  float2 r23 = __fmul2_rn(__fadd2_rn(f2(ld(2, 0), ld(3, 0)), mc), wx0);
  r23 = __ffma2_rn(__fadd2_rn(f2(ld(2, 1), ld(3, 1)), mc), wx1, r23);
  r23 = __ffma2_rn(__fadd2_rn(f2(ld(2, 2), ld(3, 2)), mc), wx2, r23);
  r23 = __ffma2_rn(__fadd2_rn(f2(ld(2, 3), ld(3, 3)), mc), wx3, r23);
  // y weights (rows 0..3) applied pairwise, times 1/36
  const float2 acc = __ffma2_rn(r23, f2(b1.y, t3.y), __fmul2_rn(r01, f2(s3.y, a1.y)));
  return c + over36<float>(acc.x + acc.y);
}

// from C in global memory (row pitch pc), taps from Cj + off
__device__ __forceinline__ float eval2d_f32x2(const float *Cj, int pc, int off, float x,
                                              float y) {
  const float *p = Cj + off;
  return gather_f32x2([&](int a, int b) { return p[a * pc + b]; }, x, y);
}

// FP32 storage: every gather in the difference form
template <>
__device__ __forceinline__ float eval2d<float>(const float *Cj, int pc, int rI, float x, int uI,
                                               float y) {
  return eval2d_f32x2(Cj, pc, uI * pc + rI, x, y);
}

constexpr int DR_W = 8;  // warps per drift block

// FP32 tables, 8 bytes per cell: word = index << FP_FBITS | round(frac * 2^FP_FBITS)
// per direction; FP_OUT / FP_CHAIN in the first word mark the two special kinds
// (the second word then holds the chain id).  The 21 fraction bits are the low
// mantissa bits of a float in [4, 5), whose spacing is 2^-21: one logic
// operation and a subtraction of 4, no shift and no int->float convert.
constexpr int FP_FBITS = 21;
constexpr uint32_t FP_FMASK = (1u << FP_FBITS) - 1u;
constexpr uint32_t FP_OUT = 0xFFFFFFFFu, FP_CHAIN = 0xFFFFFFFEu;

__device__ __forceinline__ float frac21(uint32_t w) {
  return __uint_as_float(0x40800000u | (w & FP_FMASK)) - 4.0f;
}
// both directions' fractions of one cell
__device__ __forceinline__ float2 frac21x2(uint2 w) {
  return __fadd2_rn(make_float2(__uint_as_float(0x40800000u | (w.x & FP_FMASK)),
                                __uint_as_float(0x40800000u | (w.y & FP_FMASK))),
                    make_float2(-4.f, -4.f));
}

// ------------------------------------------------------- TMA-staged drift
// Most drift footpoints lie within a few cells of their own node, so each
// block (a strip of 32 r columns of one J slice) walks down the rows in
// chunks of DW_CH and has the tensor-memory accelerator bring the matching
// DW_ROWS x DW_COLS window of the coefficient slice into shared memory,
// double buffered and signalled through an mbarrier.  Taps inside the window
// are read from shared memory; footpoints outside it (far displacements) read
// the coefficients from global memory.  Every mbarrier wait is bounded: on
// timeout the block records an error flag and falls back to global reads.
//
// Footpoints are fixed for the run, so each window's first row is chosen once
// per chunk (window_rows_kernel): the one that holds most of the chunk's tap
// blocks, which drift together by up to hundreds of rows at small radii (4.7 %
// of the in-box cells of the 513 x 513 Hernquist grid lie outside it, 10.8 %
// outside windows that start 12 rows above their chunk).  Chunks with every
// cell outside the box (20 % of them) store zeros, stage nothing and read no
// footpoints.  FP64 drift 0.379 -> 0.305 ms on 513 x 513 x 128 Hernquist,
// 0.106 -> 0.095 on 201 x 201 x 200 UDF, the narrower windows included.
constexpr int DW_CH = 16, DW_XOFF = (DW_COLS - 32) / 2;
constexpr int DT_THREADS = 256;  // 8 warps x 32 columns; 2 rows per warp per chunk
template <typename T>
struct Cell {
  int rI, uI, kind;
  uint32_t ch;
  T x, y;
};

// Footpoint words as loaded (decoded only where the cell is computed, so that
// prefetched loads stay in flight)
template <typename T>
struct RawCell;
template <>
struct RawCell<float> {
  uint2 w;
};
template <>
struct RawCell<double> {
  int code;
  double x, y;
};
__device__ __forceinline__ RawCell<float> load_raw(const int32_t *, const float *,
                                                   const float *,
                                                   const uint2 *__restrict__ fp2, size_t i) {
  RawCell<float> c;
  c.w = __ldg(fp2 + i);
  return c;
}
__device__ __forceinline__ RawCell<double> load_raw(const int32_t *__restrict__ idx,
                                                    const double *__restrict__ fx,
                                                    const double *__restrict__ fy,
                                                    const uint2 *, size_t i) {
  RawCell<double> c;
  c.code = __ldg(idx + i);
  c.x = __ldg(fx + i);
  c.y = __ldg(fy + i);
  return c;
}
// kinds: 0 gather, 1 outside (0), 2 delayed-kernel chain front
__device__ __forceinline__ Cell<float> decode(const RawCell<float> &r) {
  Cell<float> c;
  const uint2 w = r.w;
  const bool ok = w.x < FP_CHAIN;
  c.kind = ok ? 0 : (w.x == FP_OUT ? 1 : 2);
  c.ch = w.y;
  c.rI = ok ? (int)(w.x >> FP_FBITS) : 0;
  c.uI = ok ? (int)(w.y >> FP_FBITS) : 0;
  c.x = frac21(w.x);
  c.y = frac21(w.y);
  return c;
}
__device__ __forceinline__ Cell<double> decode(const RawCell<double> &r) {
  Cell<double> c;
  const int code = r.code;
  c.kind = code >= 0 ? 0 : (code == -1 ? 1 : 2);
  c.ch = (uint32_t)(-2 - code);
  c.rI = code >= 0 ? (code & 0xffff) : 0;
  c.uI = code >= 0 ? (code >> 16) : 0;
  c.x = code >= 0 ? r.x : 0.0;
  c.y = code >= 0 ? r.y : 0.0;
  return c;
}

// 4x4 gather from a shared window of row pitch PITCH (immediate offsets)
template <int PITCH, typename T>
__device__ __forceinline__ T eval_pitch(const T *p, T x, T y) {
  const T b2xI = bv2<T>(T(1) - x), b1xI = bv1<T>(T(1) - x);
  const T b1x = bv1<T>(x), b2x = bv2<T>(x);
  const T s0 = p[0] * b2xI + p[1] * b1xI + p[2] * b1x + p[3] * b2x;
  const T s1 = p[PITCH] * b2xI + p[PITCH + 1] * b1xI + p[PITCH + 2] * b1x + p[PITCH + 3] * b2x;
  const T s2 = p[2 * PITCH] * b2xI + p[2 * PITCH + 1] * b1xI + p[2 * PITCH + 2] * b1x +
               p[2 * PITCH + 3] * b2x;
  const T s3 = p[3 * PITCH] * b2xI + p[3 * PITCH + 1] * b1xI + p[3 * PITCH + 2] * b1x +
               p[3 * PITCH + 3] * b2x;
  return over36<T>(bv2<T>(T(1) - y) * s0 + bv1<T>(T(1) - y) * s1 +
                           bv1<T>(y) * s2 + bv2<T>(y) * s3);
}
template <int PITCH>
__device__ __forceinline__ float eval_pitch(const float *p, float x, float y) {
  return gather_f32x2([&](int a, int b) { return p[a * PITCH + b]; }, x, y);
}

constexpr int DW_MAX_CH = 2048 / DW_CH;   // chunks of the tallest slice
constexpr int16_t DW_EMPTY = INT16_MIN;  // a chunk with nothing to gather or read

// first window row of each (slice, strip, chunk): one warp each
template <typename T>
__global__ void __launch_bounds__(128)
    window_rows_kernel(const int32_t *__restrict__ idx, const uint2 *__restrict__ fp2,
                       int16_t *__restrict__ rows, int nr, int nu, int nj) {
  __shared__ uint16_t hist[4][2048];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ns = (nr + 31) / 32, nch = (nu + DW_CH - 1) / DW_CH;
  const size_t k = (size_t)blockIdx.x * 4 + w;
  if (k >= (size_t)nj * ns * nch) return;
  const int c = (int)(k % nch), s = (int)(k / nch % ns);
  const size_t j = k / ((size_t)nch * ns);
  uint16_t *h = hist[w];
  for (int y = lane; y < 2048; y += 32) h[y] = 0;
  __syncwarp();
  const int r = 32 * s + lane, x0 = 32 * s - DW_XOFF;
  bool some = false;
  for (int u = c * DW_CH; u < min((c + 1) * DW_CH, nu); ++u) {
    int y = -1;
    if (r < nr) {
      const size_t cell = (j * nu + u) * nr + r;
      int rI;
      if constexpr (sizeof(T) == 4) {
        const uint2 q = __ldg(fp2 + cell);
        some = some || q.x != FP_OUT;
        rI = (int)(q.x >> FP_FBITS);
        y = q.x < FP_CHAIN ? (int)(q.y >> FP_FBITS) : -1;
      } else {
        const int code = __ldg(idx + cell);
        some = some || code != -1;
        rI = code & 0xffff;
        y = code >= 0 ? code >> 16 : -1;
      }
      if (rI - x0 < 0 || rI - x0 > DW_COLS - 4) y = -1;
    }
    // lanes with the same row add once
    const unsigned same = __match_any_sync(0xffffffffu, y);
    if (y >= 0 && lane == __ffs(same) - 1) h[y] += (uint16_t)__popc(same);
    __syncwarp();
  }
  // the start whose DW_ROWS - 3 tap rows hold most cells, the first of equals
  int best = -1, by = 0;
  for (int y = lane; y < nu; y += 32) {
    int n = 0;
    for (int q = y; q < min(y + DW_ROWS - 3, nu); ++q) n += h[q];
    if (n > best) {
      best = n;
      by = y;
    }
  }
  for (int d = 16; d > 0; d >>= 1) {
    const int n = __shfl_xor_sync(0xffffffffu, best, d), y = __shfl_xor_sync(0xffffffffu, by, d);
    if (n > best || (n == best && y < by)) {
      best = n;
      by = y;
    }
  }
  some = __any_sync(0xffffffffu, some);
  if (lane == 0) rows[k] = some ? (int16_t)by : DW_EMPTY;
}

size_t window_rows_count(int nr, int nu, int nj) {
  return (size_t)nj * ((nr + 31) / 32) * ((nu + DW_CH - 1) / DW_CH);
}
template <typename T>
cudaError_t launch_window_rows(const int32_t *idx, const uint2 *fp2, int16_t *rows, int nr, int nu,
                               int nj, cudaStream_t st) {
  window_rows_kernel<T><<<(unsigned)((window_rows_count(nr, nu, nj) + 3) / 4), 128, 0, st>>>(
      idx, fp2, rows, nr, nu, nj);
  return cudaGetLastError();
}

template <typename T>
__global__ void __launch_bounds__(DT_THREADS)
    drift_tma_kernel(const __grid_constant__ CUtensorMap tmC, const T *C,
                     T *__restrict__ f,
                     const int32_t *__restrict__ idx, const T *__restrict__ fx,
                     const T *__restrict__ fy, const uint2 *__restrict__ fp2,
                     const int16_t *__restrict__ win_rows,
                     const int64_t *__restrict__ ch_start, const int32_t *__restrict__ ch_len,
                     const T *ch_val, int64_t ndrift, MomentTables mt,
                     double *__restrict__ partial, unsigned int *err, uint32_t spins,
                     Geometry g) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T *win = reinterpret_cast<T *>(smem_raw);  // two windows
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw + 2 * DW_COLS * DW_ROWS * sizeof(T));
  __shared__ double red[DT_THREADS / 32][32];
  constexpr uint32_t BYTES = DW_COLS * DW_ROWS * sizeof(T);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int r0 = blockIdx.x * 32, r = r0 + lane;
  const int jl = blockIdx.y, j = g.j0 + jl;  // batch-local / global slice
  const int nch = (g.nu + DW_CH - 1) / DW_CH;
  const int x0 = r0 - DW_XOFF;
  // the chunks' window rows, and the list of those that are not empty
  __shared__ int16_t wy[DW_MAX_CH];
  __shared__ uint8_t list[DW_MAX_CH];
  __shared__ int nlist;
  const size_t row0 = (size_t)j * g.nu * g.nr + r;
  const bool col_ok = r < g.nr;
  RawCell<T> nxt[2];
  auto words_of = [&](int c) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = c * DW_CH + w + 8 * q;
      nxt[q] = load_raw(idx, fx, fy, fp2, row0 + (size_t)(u < g.nu && col_ok ? u : 0) * g.nr);
    }
  };
  chain_begin();
  words_of(0);  // the first chunk's, unless it turns out to be empty
  if (w == 0) {
    const int16_t *src = win_rows + ((size_t)j * gridDim.x + blockIdx.x) * nch;
    int n = 0;
    for (int c0 = 0; c0 < nch; c0 += 32) {
      const int c = c0 + lane;
      const int16_t y = c < nch ? __ldg(src + c) : DW_EMPTY;
      const unsigned m = __ballot_sync(0xffffffffu, y != DW_EMPTY);
      if (c < nch) wy[c] = y;
      if (y != DW_EMPTY) list[n + __popc(m & ((1u << lane) - 1u))] = (uint8_t)c;
      n += __popc(m);
    }
    __syncwarp();
    if (lane == 0) {
      nlist = n;
      mbar_init(&bar[0], 1);
      mbar_init(&bar[1], 1);
      mbar_fence_init();
      for (int k = 0; k < 2 && k < n; ++k) {
        mbar_expect_tx(&bar[k], BYTES);
        tma_load_3d(win + k * DW_COLS * DW_ROWS, &tmC, x0, wy[list[k]], jl, &bar[k]);
      }
    }
  }
  __syncthreads();
  const int nl = nlist;
  const T *Cj = C + (size_t)jl * (g.nu + 3) * g.pc;
  if (nl > 0 && list[0] != 0) words_of(list[0]);
  double acc = 0.0;
  // copy bookkeeping (meaningful in thread 0, which issues every copy): the
  // list entry last sent to each buffer and whether its completion was observed
  int last0 = 0, last1 = 1;
  unsigned pending = (nl > 0 ? 1u : 0u) | (nl > 1 ? 2u : 0u);  // bit b: buffer b's copy not yet seen
  bool issuing = true;
  for (int k = 0; k < nl; ++k) {
    const int c = list[k];
    const RawCell<T> cur[2] = {nxt[0], nxt[1]};
    if (k + 1 < nl) words_of(list[k + 1]);
    const int b = k & 1;
    // after one failed wait this thread waits no more (it reads C globally)
    const bool have = issuing && mbar_wait_bounded(&bar[b], (uint32_t)((k >> 1) & 1), spins);
    if (have) pending &= ~(1u << b);
    if (!have && issuing) {
      issuing = false;  // never stack a second copy onto an unfinished one
      atomicOr(err, 1u);
    }
    const T *wb = win + b * DW_COLS * DW_ROWS;
    const int y0 = wy[c];
    T part = T(0);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = c * DW_CH + w + 8 * q;
      if (u < g.nu && col_ok) {
        const Cell<T> cl = decode(cur[q]);
        T v = T(0);
        if (cl.kind == 0) {
          const int wr = cl.uI - y0, wc = cl.rI - x0;
          if (have && wr >= 0 && wr <= DW_ROWS - 4 && wc >= 0 && wc <= DW_COLS - 4)
            v = eval_pitch<DW_COLS>(wb + wr * DW_COLS + wc, cl.x, cl.y);
          else
            v = eval2d<T>(Cj, g.pc, cl.rI, cl.x, cl.uI, cl.y);
        } else if (cl.kind == 2) {
          const int L = __ldg(ch_len + cl.ch);
          v = ch_val[__ldg(ch_start + cl.ch) + ndrift % L];
        }
        f[row0 + (size_t)u * g.nr] = v;
        part += (T)__ldg(mt.bu + u) * v;
      }
    }
    acc += (double)part;
    __syncthreads();  // every warp is done with window b
    if (tid == 0 && issuing && k + 2 < nl) {
      fence_proxy_async();
      mbar_expect_tx(&bar[b], BYTES);
      tma_load_3d(win + b * DW_COLS * DW_ROWS, &tmC, x0, wy[list[k + 2]], jl, &bar[b]);
      if (b) last1 = k + 2; else last0 = k + 2;
      pending |= 1u << b;
    }
  }
  // the empty chunks
  for (int c = 0; c < nch; ++c) {
    if (wy[c] != DW_EMPTY) continue;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = c * DW_CH + w + 8 * q;
      if (u < g.nu && col_ok) f[row0 + (size_t)u * g.nr] = T(0);
    }
  }
  // a copy whose wait timed out may still be in flight: wait for it (bounded)
  // before the block's shared memory is released
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      const int lb = b ? last1 : last0;
      if (((pending >> b) & 1u) && lb < nl &&
          !mbar_wait_bounded(&bar[b], (uint32_t)((lb >> 1) & 1)))
        atomicOr(err, 2u);
    }
  }
  red[w][lane] = acc;
  __syncthreads();
  if (w == 0 && col_ok) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < DT_THREADS / 32; ++k) s += red[k][lane];
    partial[(size_t)j * g.nr + r] = __ldg(mt.wj + j) * s;
  }
}

template <typename T>
cudaError_t launch_drift_tma(const CUtensorMap *tmC, const T *C, T *f, const int32_t *idx,
                             const T *fx, const T *fy, const uint2 *fp2, const int16_t *win_rows,
                             const int64_t *ch_start, const int32_t *ch_len,
                             const T *ch_val, int64_t ndrift, const MomentTables &mt,
                             double *partial, unsigned int *err, uint32_t spins,
                             const Geometry &g, cudaStream_t st) {
  const size_t smem = 2 * DW_COLS * DW_ROWS * sizeof(T) + 2 * sizeof(uint64_t);
  cudaError_t e = cudaFuncSetAttribute(drift_tma_kernel<T>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((g.nr + 31) / 32, g.nb);
  return chain_launch(drift_tma_kernel<T>, grid, dim3(DT_THREADS), smem, st, *tmC, C, f, idx, fx,
                      fy, fp2, win_rows, ch_start, ch_len, ch_val, ndrift, mt, partial, err, spins, g);
}

// ------------------------------------------------------------ strip drift
// FP32 storage: the coefficient strip of 32 output columns (DS_WC columns
// starting DS_XL to the left, all N_u + 3 rows) is staged in shared memory, so
// that a cell can read any row of it: the footpoints' u displacements
// reach hundreds of rows while their r displacements stay within a few
// columns.  Cells whose taps leave the strip's columns gather from global
// memory.
// The kinds of a trip, DS_TRIP rows of one strip (32 columns) of a slice:
// nothing to compute (every cell outside the box: 0), regular (every cell
// gathers inside the strip, and from row to row each column's 4 x 4 taps move
// by exactly one coefficient row), anything else.  Footpoints vary so slowly
// along u that 57 % of the trips are regular and 18 % empty on the
// 513 x 513 x 256 Hernquist grid (48 % and 17 % on 257 x 257 x 128 Plummer).
// They are fixed for the run, so the kinds are found once per table.
constexpr int DS_TRIP = 8;
enum { TRIP_ANY = 0, TRIP_REGULAR = 1, TRIP_EMPTY = 2 };
__host__ __device__ inline int strip_blocks(int nr) {
  // N_r = 32 k + 1 (every grid of the form 2^n + 1): k strips, the last one's
  // block also takes the last column; 2.4 % faster than a block of one column
  // on the 513 x 513 x 256 case
  return (nr % 32 == 1 && nr > 32) ? nr / 32 : (nr + 31) / 32;
}
__host__ __device__ inline int strip_trips(int nu) { return (nu + DS_TRIP - 1) / DS_TRIP; }
constexpr int DS_WC = 48, DS_XL = (DS_WC - 32) / 2;  // columns staged, and left of the strip
// consumer warps of a block (one producer warp besides) and footpoint rows in
// flight per warp.  Drift of 513 x 513 x 256 Hernquist / 257 x 257 x 128
// Plummer / 395 x 307 x 77 UDF / 1025 x 1025 x 64 PLDF in us, four rows: 17
// warps 261 / 51.4 / 55.7 / 313, 19 (96 registers) 249 / 48.4 / 53.9 / 300, 21
// 260 / 51.5 / 53.8 / 318, 23 (80) 252 / 51.7 / 53.6 / 298.  In an earlier form
// (plain order of the tasks) 31 warps and two rows took 295 / 61, 13 and four
// 309 / 52, 19 and eight 282 / 51.
constexpr int STRIP_WARPS = 19;
constexpr int DS_AHEAD = 4;

// one warp per trip (lanes past N_r take the last column, as the drift does)
__global__ void __launch_bounds__(256)
    trip_kind_kernel(const uint2 *__restrict__ fp2, uint8_t *__restrict__ kinds, int nr, int nu,
                     int nj) {
  const int ns = strip_blocks(nr), nt = strip_trips(nu);
  const size_t k = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (k >= (size_t)nj * ns * nt) return;
  const int t = (int)(k % nt), s = (int)(k / nt % ns);
  const size_t j = k / ((size_t)nt * ns);
  const int r = min(32 * s + (int)(threadIdx.x & 31), nr - 1), x0 = 32 * s - DS_XL;
  bool regular = DS_TRIP * (t + 1) <= nu, empty = true;
  uint32_t px = 0, py = 0;
  for (int q = 0; q < DS_TRIP && DS_TRIP * t + q < nu; ++q) {
    const uint2 w = __ldg(fp2 + (j * nu + DS_TRIP * t + q) * nr + r);
    const uint32_t ix = w.x >> FP_FBITS, iy = w.y >> FP_FBITS;
    empty = empty && w.x == FP_OUT;
    regular = regular && w.x < FP_CHAIN && ix - (uint32_t)x0 < (uint32_t)(DS_WC - 3) &&
              (q == 0 || (ix == px && iy == py + 1u));
    px = ix;
    py = iy;
  }
  const bool all_regular = __all_sync(0xffffffffu, regular);
  const bool all_empty = __all_sync(0xffffffffu, empty);
  if ((threadIdx.x & 31) == 0)
    kinds[k] = all_regular ? TRIP_REGULAR : all_empty ? TRIP_EMPTY : TRIP_ANY;
}

size_t trip_kinds_bytes(int nr, int nu, int nj) {
  return (size_t)nj * strip_blocks(nr) * strip_trips(nu);
}

// Edge cells: those whose value the drift kernels do not gather themselves.
// Chain fronts, and, with a strip layout, cells whose taps leave the strip's
// columns (0.4 % of the cells of the 513 x 513 x 256 Hernquist grid, all in
// its first columns).  edge_kernel writes their values into f before the
// drift, which reads them there for its moment sums.  Word of such a cell:
// neither outside nor gathering in the strip.
__device__ __forceinline__ bool in_strip(uint2 w, int x0) {
  return w.x < FP_CHAIN && (w.x >> FP_FBITS) - (uint32_t)x0 < (uint32_t)(DS_WC - 3);
}
// the far-tap cells of each slice (cell index within the slice): one block
// per slice; counts them, or fills the slice's part of the list
__global__ void __launch_bounds__(1024)
    far_cells_kernel(const uint2 *__restrict__ fp2, const uint32_t *__restrict__ base,
                     uint32_t *__restrict__ count, uint32_t *__restrict__ list, int nr, int nu) {
  __shared__ uint32_t n;
  const int ns = strip_blocks(nr);
  const uint32_t cells = (uint32_t)nr * (uint32_t)nu;
  if (threadIdx.x == 0) n = 0u;
  __syncthreads();
  const uint2 *ws = fp2 + (size_t)blockIdx.x * cells;
  for (uint32_t i = threadIdx.x; i < cells; i += blockDim.x) {
    const uint2 w = __ldg(ws + i);
    const int x0 = 32 * min((int)(i % (uint32_t)nr) / 32, ns - 1) - DS_XL;
    if (w.x < FP_CHAIN && !in_strip(w, x0)) {
      const uint32_t at = atomicAdd(&n, 1u);
      if (list) list[base[blockIdx.x] + at] = i;
    }
  }
  __syncthreads();
  if (!list && threadIdx.x == 0) count[blockIdx.x] = n;
}

cudaError_t launch_trip_kinds(const uint2 *fp2, uint8_t *kinds, int nr, int nu, int nj,
                              cudaStream_t st) {
  const size_t n = trip_kinds_bytes(nr, nu, nj);
  trip_kind_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(fp2, kinds, nr, nu, nj);
  return cudaGetLastError();
}
cudaError_t launch_far_cells(const uint2 *fp2, const uint32_t *base, uint32_t *count,
                             uint32_t *list, int nr, int nu, int nj, cudaStream_t st) {
  far_cells_kernel<<<nj, 1024, 0, st>>>(fp2, base, count, list, nr, nu);
  return cudaGetLastError();
}

// The 4 x 4 taps of one cell of a regular trip, in four row slots: at row K
// of the trip tap row a sits in slot (K + a) & 3, so that the next row drops
// the first tap row and loads one new one, into slot (K + 3) & 3.  A slot
// holds the row's second tap and the other three taps' differences from it,
// formed once when the row is loaded.
struct TapWin {
  float b[4], d0[4], d2[4], d3[4];
  template <int S>
  __device__ __forceinline__ void row(const float *p) {
    const float c = p[1];
    b[S & 3] = c;
    d0[S & 3] = p[0] - c;
    d2[S & 3] = p[2] - c;
    d3[S & 3] = p[3] - c;
  }
  // Difference form (see gather_f32x2) about c, the second tap of the second
  // row: c + (1/36) sum_a wy_a (6 (b_a - c) + sum_{m != 1} wx_m d_am); the x
  // weight of column 1 is not needed because each direction's weights sum to
  // 6, and every rounding but the last acts on differences.  Weights of both
  // directions pairwise, not divided by 6: the rounded 1/6 would lean every
  // weight the same way in every step (energy drift of the 2000-step Plummer
  // 257 x 257 x 128 case 1.4e-6 off the FP64 path's with weights times a
  // rounded 1/6).  No less exact than the general gather: one evaluation has
  // the same rms error against 64 bits (2.43e-8 of the value, 2.55e-8 where
  // neighbouring taps differ by a tenth), 200 steps of 513 x 513 x 256
  // Hernquist 1.73e-6 against 1.74e-6 (mean of 14 runs, relative L2 of f), the
  // energy drift after 2000 Plummer steps 7.9e-7 against 9.0e-7 and after 1000
  // UDF steps 3.8e-7 against 4.7e-7 (rms over 40 radii); single runs scatter
  // by as much as these values, with either form.
  template <int K>
  __device__ __forceinline__ float eval(float2 t) const {
    constexpr int S0 = K & 3, S1 = (K + 1) & 3, S2 = (K + 2) & 3, S3 = (K + 3) & 3;
    const float2 one = f2(1.f, 1.f), three = f2(3.f, 3.f);
    const float2 s = __fadd2_rn(one, f2(-t.x, -t.y));
    const float2 t2 = __fmul2_rn(t, t), w3 = __fmul2_rn(t2, t);
    const float2 w0 = __fmul2_rn(__fmul2_rn(s, s), s);
    const float2 w2 = __ffma2_rn(f2(-3.f, -3.f), w3,
                                 __ffma2_rn(three, t2, __ffma2_rn(three, t, one)));
    const float wy1 = __fmaf_rn(
        s.y, __fmaf_rn(s.y, __fmaf_rn(s.y, -3.f, 3.f), 3.f), 1.f);
    const float c = b[S1];
    const float z1 = __fmaf_rn(w3.x, d3[S1], __fmaf_rn(w2.x, d2[S1], w0.x * d0[S1]));
    const float z0 = __fmaf_rn(
        w3.x, d3[S0], __fmaf_rn(w2.x, d2[S0], __fmaf_rn(w0.x, d0[S0], 6.f * (b[S0] - c))));
    const float z2 = __fmaf_rn(
        w3.x, d3[S2], __fmaf_rn(w2.x, d2[S2], __fmaf_rn(w0.x, d0[S2], 6.f * (b[S2] - c))));
    const float z3 = __fmaf_rn(
        w3.x, d3[S3], __fmaf_rn(w2.x, d2[S3], __fmaf_rn(w0.x, d0[S3], 6.f * (b[S3] - c))));
    return c + over36<float>(__fmaf_rn(
                   w3.y, z3, __fmaf_rn(w2.y, z2, __fmaf_rn(wy1, z1, w0.y * z0))));
  }
};

// Rows [8 t, 8 t + 8) of one strip column per lane.  In a regular trip the
// taps of row K + 1 are those of row K one coefficient row further down, so a
// cell loads 4 new taps instead of 16 and needs no index, test or vote; the
// others test every cell and gather its 16 taps, or read the value of an edge
// cell.  q: the footpoint words of the trip's first DS_AHEAD rows on entry, of
// the rows at `pn` on return (in flight that many rows ahead); rows past the
// slice read the next slice or the tables' padding (FOOT_PAD_ROWS rows).  Returns
// the trip's moment sum.
__device__ __forceinline__ double strip_trip(bool regular, const float *win, const float *bu,
                                             int x0, int rows_left, uint2 (&q)[DS_AHEAD],
                                             const uint2 *p, const uint2 *pn, float *o,
                                             uint32_t nr) {
  static_assert(DS_TRIP <= FOOT_PAD_ROWS, "a trip's loads reach past the padding rows");
  constexpr int WC = DS_WC;
  double acc = 0.0;
  if (regular) {
    // moment weights of the trip's rows (the table is padded to whole trips)
    const float4 bl = *reinterpret_cast<const float4 *>(bu);
    const float4 bh = *(reinterpret_cast<const float4 *>(bu) + 1);
    const float bk[DS_TRIP] = {bl.x, bl.y, bl.z, bl.w, bh.x, bh.y, bh.z, bh.w};
    const float *q0 = win + (int)(q[0].y >> FP_FBITS) * WC + ((int)(q[0].x >> FP_FBITS) - x0);
    TapWin tw;
    tw.row<0>(q0);
    tw.row<1>(q0 + WC);
    tw.row<2>(q0 + 2 * WC);
    float part = 0.f;
    p = DS_AHEAD < DS_TRIP ? p + DS_AHEAD * nr : pn;
#define VLS_REGULAR_ROW(K)                          \
  {                                                 \
    const float2 xy = frac21x2(q[(K) % DS_AHEAD]);  \
    q[(K) % DS_AHEAD] = __ldg(p);                   \
    p = (K) == DS_TRIP - DS_AHEAD - 1 ? pn : p + nr; \
    tw.row<(K) + 3>(q0 + ((K) + 3) * WC);           \
    const float v = tw.eval<K>(xy);                 \
    *o = v;                                         \
    o += nr;                                        \
    if ((K) & 1)                                    \
      acc += (double)(part + bk[K] * v);            \
    else                                            \
      part = bk[K] * v;                             \
  }
    VLS_REGULAR_ROW(0)
    VLS_REGULAR_ROW(1)
    VLS_REGULAR_ROW(2)
    VLS_REGULAR_ROW(3)
    VLS_REGULAR_ROW(4)
    VLS_REGULAR_ROW(5)
    VLS_REGULAR_ROW(6)
    VLS_REGULAR_ROW(7)
#undef VLS_REGULAR_ROW
    return acc;
  }
#pragma unroll 1
  for (int k = 0; k < DS_TRIP; k += 2) {
    const uint2 c[2] = {q[0], q[1]};
#pragma unroll
    for (int h = 0; h + 2 < DS_AHEAD; ++h) q[h] = q[h + 2];
    const int ka = k + DS_AHEAD;  // the rows two words of which are loaded now
    const uint2 *pp = ka < DS_TRIP ? p + ka * nr : pn + (ka - DS_TRIP) * nr;
    q[DS_AHEAD - 2] = __ldg(pp);
    q[DS_AHEAD - 1] = __ldg(pp + nr);
    float v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t wc = (c[h].x >> FP_FBITS) - (uint32_t)x0;
      const bool in = c[h].x < FP_CHAIN && wc < (uint32_t)(WC - 3), row = k + h < rows_left;
      float edge = 0.f;
      if (!in && c[h].x != FP_OUT && row) edge = o[h * nr];
      const float2 xy = frac21x2(c[h]);
      v[h] = eval_pitch<WC>(win + (in ? (c[h].y >> FP_FBITS) * WC + wc : 0u), xy.x, xy.y);
      v[h] = in ? v[h] : edge;
      if (row)
        o[h * nr] = v[h];
      else
        v[h] = 0.f;
    }
    acc += (double)(bu[k] * v[0] + bu[k + 1] * v[1]);
    o += 2 * nr;
  }
  return acc;
}

// Shared memory of the strip drift: NB strip buffers (nch boxes of `rows`
// rows), then per buffer the column sums of every warp and the trips' kinds,
// then the moment weights where they fit (else they are read in global
// memory: strips of 568 .. 573 rows with two buffers, 1148 and 1149 with one).
// The boxes hold N_u + 3 rows with as little excess as even heights of at most
// 256 rows give (16-byte-multiple boxes on 128-byte boundaries).
struct StripSmem {
  size_t strip, red, kinds, total;  // bytes: one buffer's parts, everything
  int nch, rows, nt;
};
__host__ __device__ inline StripSmem strip_smem(int nu, int nw, int nb, bool weights) {
  StripSmem s;
  s.nch = (nu + 3 + 255) / 256;
  s.rows = (nu + 3 + 2 * s.nch - 1) / (2 * s.nch) * 2;
  s.nt = strip_trips(nu);
  s.strip = (size_t)s.nch * s.rows * DS_WC * sizeof(float);
  s.red = ((size_t)nw * 33 * sizeof(double) + 15) / 16 * 16;
  s.kinds = (size_t)(s.nt + 15) / 16 * 16;
  s.total = nb * (s.strip + s.red + s.kinds) +
            (weights ? (size_t)s.nt * DS_TRIP * sizeof(float) : 0);
  return s;
}


// Block: NW consumer warps and a producer warp; persistent, a task being one
// strip (32 output columns) of one J slice.  The producer keeps NB strips
// staged or in flight: it issues a strip's TMA boxes and fetches its trips'
// kinds (full barrier); when every consumer is done with a strip (done
// barrier) it sums their column sums in warp order and refills the buffer
// with the strip NB tasks later.  The consumers take the strips' trips in
// turn without a block barrier: a warp that has no more trips in a strip goes
// on to the next one, so neither the staging of a strip nor the uneven cost
// of its trips (only the rows near v_r = 0 of the inner columns gather at
// all) leaves the SM idle.  Which warp takes which trip depends on (strip,
// slice) alone, and every sum is taken in a fixed order, so the moments do
// not depend on the grid or the batching.
//
// What bounds it: about 60 instructions per cell in regular trips and 110 in
// the others at some 60 % of the issue slots, and a quarter of the time waits
// for a strip.  drift_strip_block_kernel (a block per strip, every cell with
// its 16 taps and the rare cells gathered in place; 116 instructions per cell)
// took 0.311 ms on the 513 x 513 x 256 Hernquist case, 0.373 on 1025 x 1025 x
// 64 PLDF and 0.057 on 257 x 257 x 128 Plummer; this form 0.249, 0.300 and
// 0.048, and edge_kernel 0.012, 0.018 and 0.001 more than the tails alone.
//
// Waits are bounded.  A consumer whose wait for a strip ran out (`spins`
// polls) gathers that strip's cells from global memory; the producer waits
// (full limit) for a strip's own boxes before it refills its buffer and
// before the block ends, whatever the consumers did.
template <int NW, int NB, int MINB, bool WEIGHTS>
__global__ void __launch_bounds__(32 * (NW + 1), MINB)
    drift_strip_kernel(const __grid_constant__ CUtensorMap tmS, const float *C,
                       float *f, const uint2 *__restrict__ fp2,
                       const uint8_t *__restrict__ trip_kinds, MomentTables mt,
                       double *__restrict__ partial, unsigned int *err, uint32_t spins,
                       uint32_t rot, Geometry g) {
  constexpr int WC = DS_WC;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[NB], done[NB];
  const StripSmem L = strip_smem(g.nu, NW, NB, WEIGHTS);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int ns = strip_blocks(g.nr), ntask = ns * g.nb, nt = L.nt;
  const bool extra = ns * 32 < g.nr;  // the last strip also takes the last column
  unsigned char *kinds0 = smem_raw + NB * (L.strip + L.red);
  float *wsm = reinterpret_cast<float *>(kinds0 + NB * L.kinds);
  const float *bus = WEIGHTS ? wsm : mt.bu32;
  auto buf_win = [&](int b) { return reinterpret_cast<float *>(smem_raw + b * L.strip); };
  auto buf_red = [&](int b) {
    return reinterpret_cast<double *>(smem_raw + NB * L.strip + b * L.red);
  };
  if (tid == 0) {
    for (int b = 0; b < NB; ++b) {
      mbar_init(&full[b], 2);  // the boxes, and the kinds
      mbar_init(&done[b], NW);
    }
    mbar_fence_init();
  }
  chain_begin();
  if constexpr (WEIGHTS)
    for (int u = tid; u < nt * DS_TRIP; u += 32 * (NW + 1)) wsm[u] = __ldg(mt.bu32 + u);
  __syncthreads();
  // this block's i-th task: one of the i-th gridDim.x tasks in turn
  auto task_of = [&](int i) {
    return i * (int)gridDim.x + (int)((blockIdx.x + (uint32_t)i * rot) % gridDim.x);
  };
  const int whole = ntask / (int)gridDim.x;
  const int nmine = whole + (task_of(whole) < ntask ? 1 : 0);

  if (w == NW) {  // ------------------------------------------------ producer
    // a strip's boxes; then its trips' kinds (into registers, then into the
    // buffer), and its share of its slice's footpoint words into L2, where
    // the trips find them a strip or two later, in flight DS_AHEAD rows ahead
    auto issue = [&](int i) {
      const int task = task_of(i), b = i % NB;
      const int jl = task / ns, sx = task - jl * ns;
      if (lane == 0) {
        mbar_expect_tx(&full[b], (uint32_t)L.strip);
        for (int c = 0; c < L.nch; ++c)
          tma_load_3d(buf_win(b) + (size_t)c * L.rows * WC, &tmS, sx * 32 - DS_XL, c * L.rows, jl,
                      &full[b]);
      }
      __syncwarp();
    };
    // into L2 only for strips of up to 352 rows, a line found by measuring.
    // Drift in us with / without: 257 x 257 x 128 48.5 / 51.6, 395 x 307 x 77
    // 54.0 / 55.2, 257 x 352 x 128 60.2 / 62.9, 257 x 384 x 128 65.6 / 67.2;
    // 513 x 441 x 128 119.5 / 118.4, 513 x 513 x 256 260 / 249, 1025 x 1025 x
    // 64 317 / 300.  Few strips in flight do not move it: 513 x 513 x 32 56.2 /
    // 55.3, 1025 x 1025 x 8 59.5 / 58.2.
    const bool l2_words = g.nu <= 352;
    constexpr int KPL = 5;  // kinds per lane: strips of up to 1280 rows
    uint8_t kd[KPL];
    auto fetch = [&](int i) {
      const int task = task_of(i);
      const int jl = task / ns, sx = task - jl * ns;
      const uint8_t *src = trip_kinds + ((size_t)(g.j0 + jl) * ns + sx) * nt;
#pragma unroll
      for (int k = 0; k < KPL; ++k) kd[k] = lane + 32 * k < nt ? __ldg(src + lane + 32 * k) : 0;
    };
    auto words_to_l2 = [&](int i) {
      const int task = task_of(i);
      const int jl = task / ns, sx = task - jl * ns;
      const uint64_t lo = (uint64_t)(g.j0 + jl) * g.nu * g.nr * 8u;
      const uint64_t n = (uint64_t)g.nu * g.nr * 8u, part = (n / (ns * 32u) + 31u) & ~15ull;
      const uint64_t at = (uint64_t)(sx * 32 + lane) * part;
      if (at < n)
        bulk_prefetch_l2(reinterpret_cast<const char *>(fp2) + ((lo + at) & ~15ull),
                         (uint32_t)part);
    };
    auto kinds_in = [&](int b) {
#pragma unroll
      for (int k = 0; k < KPL; ++k)
        if (lane + 32 * k < nt) kinds0[b * L.kinds + lane + 32 * k] = kd[k];
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[b]);
    };
    int issued = 0;
    for (; issued < NB && issued < nmine; ++issued) {
      issue(issued);
      fetch(issued);
      kinds_in(issued % NB);
      if (l2_words && issued) words_to_l2(issued);
    }
    for (int i = 0; i < nmine; ++i) {
      const int b = i % NB;
      const uint32_t par = (uint32_t)(i / NB) & 1u;
      const bool refill = issued < nmine;
      if (refill) fetch(issued);
      const bool landed = mbar_wait_idle(&full[b], par);
      const bool finished = mbar_wait_idle(&done[b], par);
      if (!__all_sync(0xffffffffu, landed && finished)) {
        // nothing more is staged; the loads in flight are awaited
        if (lane == 0) atomicOr(err, 2u);
        for (int k = i + 1; k < issued; ++k) mbar_wait_idle(&full[k % NB], (uint32_t)(k / NB) & 1u);
        break;
      }
      if (refill) {
        fence_proxy_async();
        issue(issued);
      }
      const int task = task_of(i);
      const int jl = task / ns, sx = task - jl * ns, j = g.j0 + jl;
      const double *red = buf_red(b);
      double sum = 0.0, sumx = 0.0;
#pragma unroll 8
      for (int k = 0; k < NW; ++k) sum += red[k * 32 + lane];
      if (extra && sx == ns - 1 && lane == 0)
        for (int k = 0; k < NW; ++k) sumx += red[NW * 32 + k];
      __syncwarp();
      // the buffer's sums are read: its next strip may complete
      if (refill) {
        kinds_in(b);
        if (l2_words) words_to_l2(issued);
        ++issued;
      }
      const double wj = __ldg(mt.wj + j);
      if (sx * 32 + lane < g.nr) partial[(size_t)j * g.nr + sx * 32 + lane] = wj * sum;
      if (extra && sx == ns - 1 && lane == 0)
        partial[(size_t)j * g.nr + sx * 32 + 32] = wj * sumx;
    }
    return;
  }

  // ----------------------------------------------------------------- consumer
  const uint32_t nr = (uint32_t)g.nr;
  uint2 q[DS_AHEAD];
  auto load_q = [&](const uint2 *p) {
#pragma unroll
    for (int k = 0; k < DS_AHEAD; ++k) q[k] = __ldg(p + k * nr);
  };
  // this warp's first trip of task i
  auto first_trip = [&](int task) {
    const int jl = task / ns;
    const uint32_t o = (uint32_t)(((uint64_t)(g.j0 + jl) * ns + (task - jl * ns)) * nt % NW);
    return (int)((w + NW - o) % NW);
  };
  auto words = [&](int task, int t) {
    const int jl = task / ns, sx = task - jl * ns;
    return fp2 + ((size_t)(g.j0 + jl) * g.nu + DS_TRIP * t) * nr +
           min(sx * 32 + lane, g.nr - 1);
  };
  int task = task_of(0);
  if (nmine > 0) {
    load_q(words(task, min(first_trip(task), nt - 1)));
  }
  for (int i = 0; i < nmine; ++i) {
    const int b = i % NB;
    const int jl = task / ns, sx = task - jl * ns, j = g.j0 + jl;
    const int x0 = sx * 32 - DS_XL;
    const int tnext = task_of(i + 1);
    const float *win = buf_win(b);
    const unsigned char *kinds = kinds0 + b * L.kinds;
    const bool ok = __all_sync(
        0xffffffffu, mbar_wait_idle(&full[b], (uint32_t)(i / NB) & 1u, spins));
    if (!ok && lane == 0) atomicOr(err, 1u);
    const uint2 *ws = words(task, 0);
    float *os = f + (size_t)j * g.nu * nr + min(sx * 32 + lane, g.nr - 1);
    double acc = 0.0;
    int t = first_trip(task);
    if (!ok) {
      // not staged in time (nor are its kinds): from global memory
      const float *Cj = C + (size_t)jl * (g.nu + 3) * g.pc;
      for (; t < nt; t += NW)
        for (int u = DS_TRIP * t; u < min(DS_TRIP * (t + 1), g.nu); ++u) {
          RawCell<float> c;
          c.w = __ldg(ws + (size_t)u * nr);
          const Cell<float> cl = decode(c);
          float v = 0.f;
          if (cl.kind == 0)
            v = eval2d<float>(Cj, g.pc, cl.rI, cl.x, cl.uI, cl.y);
          else if (cl.kind == 2)
            v = os[(size_t)u * nr];
          os[(size_t)u * nr] = v;
          acc += (double)(__ldg(mt.bu32 + u) * v);
        }
    }
    bool loaded = true;  // q holds trip t's words (if there is one)
    bool ahead = false;  // q holds the next strip's first words
    while (t < nt) {
      const unsigned char kd = kinds[t];
      float *o = os + (size_t)(DS_TRIP * t) * nr;
      const int left = g.nu - DS_TRIP * t;
      if (kd == TRIP_EMPTY) {
        const int n = min(DS_TRIP, left);
        for (int k = 0; k < n; ++k) {
          *o = 0.f;
          o += nr;
        }
        t += NW;
        loaded = false;
        continue;
      }
      const uint2 *p = ws + (size_t)(DS_TRIP * t) * nr;
      if (!loaded) load_q(p);
      // the words after this trip's: the next trip's, or the next strip's
      const int t2 = t + NW;
      const bool more = t2 < nt && kinds[t2] != TRIP_EMPTY;
      const uint2 *pn = more ? p + (size_t)(DS_TRIP * NW) * nr
                        : i + 1 < nmine && t2 >= nt
                            ? words(tnext, min(first_trip(tnext), nt - 1))
                            : p;
      acc += strip_trip(kd == TRIP_REGULAR, win, bus + DS_TRIP * t, x0, left, q, p, pn, o, nr);
      loaded = more;
      ahead = t2 >= nt;
      t = t2;
    }
    double acc2 = 0.0;
    if (extra && sx == ns - 1) {
      // the last column (the strip's columns r0 - 8 .. r0 + 39 cover it), one
      // row per thread
      const int rx = sx * 32 + 32;
      for (int u = w * 32 + lane; u < g.nu; u += 32 * NW) {
        const size_t cell = ((size_t)j * g.nu + u) * nr + rx;
        const uint2 c = __ldg(fp2 + cell);
        float v = 0.f;
        if (ok && in_strip(c, x0))
          v = eval_pitch<WC>(
              win + (c.y >> FP_FBITS) * WC + ((c.x >> FP_FBITS) - (uint32_t)x0), frac21(c.x),
              frac21(c.y));
        else if (c.x < FP_CHAIN)
          v = eval2d<float>(C + (size_t)jl * (g.nu + 3) * g.pc, g.pc, (int)(c.x >> FP_FBITS),
                            frac21(c.x), (int)(c.y >> FP_FBITS), frac21(c.y));
        else if (c.x == FP_CHAIN)
          v = f[cell];
        f[cell] = v;
        acc2 += (double)(__ldg(mt.bu32 + u) * v);
      }
      for (int d = 16; d > 0; d >>= 1) acc2 += __shfl_down_sync(0xffffffffu, acc2, d);
    }
    // a strip not awaited above: the producer is done with this buffer's sums
    // of NB tasks ago only once this task's boxes are in
    if (!ok && !__all_sync(0xffffffffu, mbar_wait_idle(&full[b], (uint32_t)(i / NB) & 1u)))
      return;
    double *red = buf_red(b);
    red[w * 32 + lane] = acc;
    if (lane == 0) red[NW * 32 + w] = acc2;
    __syncwarp();
    if (lane == 0) mbar_arrive(&done[b]);
    if (!ahead && i + 1 < nmine) {
      load_q(words(tnext, min(first_trip(tnext), nt - 1)));
    }
    task = tnext;
  }
}

// Strips in blocks: 32 output columns x every row of one J slice per block,
// the whole strip staged in boxes of DSB_ROWS rows; lanes walk the rows of
// a column in turn, footpoints two rows ahead; a warp vote per two rows sends
// the rare cells (taps outside the strip, chain fronts and, after a wait that
// ran out, every cell) to global memory.
//
// For FP64 handles that ask for strips (the windowed drift is the faster one
// and FP64's default: 513 x 513 x 128 Hernquist STRIP1 0.366 ms against 0.300,
// 257 x 253 x 128 STRIP2 0.100 against 0.094), and for FP32 grids of short
// strips (drift_strip_in_blocks).  What bounds it: 116 instructions per cell
// in FP32, footpoint loads in FP64.
constexpr int DSB_ROWS = 64, DSB_AHEAD = 2;
template <typename T, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB)
    drift_strip_block_kernel(const __grid_constant__ CUtensorMap tmS, const T *C,
                             T *__restrict__ f, const int32_t *__restrict__ idx,
                             const T *__restrict__ fx, const T *__restrict__ fy,
                             const uint2 *__restrict__ fp2,
                             const int64_t *__restrict__ ch_start,
                             const int32_t *__restrict__ ch_len, const T *ch_val,
                             int64_t ndrift, MomentTables mt, double *__restrict__ partial,
                             unsigned int *err, uint32_t spins, Geometry g) {
  constexpr int WC = DS_WC, PF = DSB_AHEAD;
  static_assert(NW * PF + 1 <= FOOT_PAD_ROWS, "the loads ahead reach past the padding rows");
  constexpr uint32_t BYTES = DSB_ROWS * WC * sizeof(T);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ double red[NW][32];
  const int rows = g.nu + 3, nch = (rows + DSB_ROWS - 1) / DSB_ROWS;
  T *win = reinterpret_cast<T *>(smem_raw);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw + (size_t)nch * BYTES);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int r0 = blockIdx.x * 32, r = r0 + lane, x0 = r0 - DS_XL;
  const int jl = blockIdx.y, j = g.j0 + jl;
  const bool col_ok = r < g.nr;
  chain_begin();
  if (tid == 0) {
    for (int c = 0; c < nch; ++c) mbar_init(&bar[c], 1);
    mbar_fence_init();
    for (int c = 0; c < nch; ++c) {
      mbar_expect_tx(&bar[c], BYTES);
      tma_load_3d(win + (size_t)c * DSB_ROWS * WC, &tmS, x0, c * DSB_ROWS, jl, &bar[c]);
    }
  }
  __syncthreads();
  const T *Cj = C + (size_t)jl * rows * g.pc;
  auto weight = [&](int u) -> T {
    if constexpr (sizeof(T) == 4)
      return __ldg(mt.bu32 + u);
    else
      return __ldg(mt.bu + u);
  };
  // rows w, w + NW, ...; loads ahead run past the slice into the next one or
  // the tables' padding, and lanes past N_r read the next row's words
  const size_t sb = (size_t)j * g.nu * g.nr;
  const uint32_t step = (uint32_t)NW * (uint32_t)g.nr;
  uint32_t off = (uint32_t)w * (uint32_t)g.nr + (uint32_t)r;
  RawCell<T> q[PF];
#pragma unroll
  for (int k = 0; k < PF; ++k) q[k] = load_raw(idx, fx, fy, fp2, sb + off + k * step);
  bool staged = true;
  for (int c = 0; c < nch && staged; ++c) staged = mbar_wait_bounded(&bar[c], 0u, spins);
  if (!staged) atomicOr(err, 1u);
  const uint32_t wcap = staged ? (uint32_t)(WC - 3) : 0u;
  // the in-strip gather, run for every lane with the tap offset zeroed where
  // it does not apply (rare: the value comes from slow instead)
  auto fast = [&](const RawCell<T> &c, bool ok, bool &rare) {
    const Cell<T> cl = decode(c);
    const uint32_t wc = (uint32_t)(cl.rI - x0);
    const bool in = ok && cl.kind == 0 && wc < wcap;
    rare = ok && !in;
    return eval_pitch<WC>(win + (in ? cl.uI * WC + (int)wc : 0), cl.x, cl.y);
  };
  auto slow = [&](const RawCell<T> &c) {
    const Cell<T> cl = decode(c);
    if (cl.kind == 0) return eval2d<T>(Cj, g.pc, cl.rI, cl.x, cl.uI, cl.y);
    if (cl.kind == 2) return ch_val[__ldg(ch_start + cl.ch) + ndrift % __ldg(ch_len + cl.ch)];
    return T(0);
  };
  double acc = 0.0;
  for (int u = w; u < g.nu; u += NW * PF) {
    T v[PF];
    RawCell<T> c[PF];
    bool rare[PF], any = false;
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      c[k] = q[k];
      if (u + NW * k < g.nu) q[k] = load_raw(idx, fx, fy, fp2, sb + off + (PF + k) * step);
      v[k] = fast(c[k], col_ok && u + NW * k < g.nu, rare[k]);
      any |= rare[k];
    }
    if (__any_sync(0xffffffffu, any)) {
#pragma unroll
      for (int k = 0; k < PF; ++k)
        if (rare[k]) v[k] = slow(c[k]);
    }
    T part = T(0);
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      if (u + NW * k < g.nu && col_ok) {
        f[sb + off] = v[k];
        part += weight(u + NW * k) * v[k];
      }
      off += step;
    }
    acc += (double)part;
  }
  // N_r = 32 k + 1: the last block also takes the last column, one row per
  // thread (its strip covers columns r0 - 8 .. r0 + 39)
  const bool extra = (int)gridDim.x * 32 < g.nr && blockIdx.x == gridDim.x - 1;
  double acc2 = 0.0;
  if (extra)
    for (int u = tid; u < g.nu; u += 32 * NW) {
      const size_t cell = sb + (size_t)u * g.nr + r0 + 32;
      const RawCell<T> c = load_raw(idx, fx, fy, fp2, cell);
      bool rare;
      T v = fast(c, true, rare);
      if (rare) v = slow(c);
      f[cell] = v;
      acc2 += (double)(weight(u) * v);
    }
  // every box must have landed before the block's shared memory is released
  if (tid == 0)
    for (int c = 0; c < nch; ++c)
      if (!mbar_wait_bounded(&bar[c], 0u)) atomicOr(err, 2u);
  red[w][lane] = acc;
  __syncthreads();
  if (w == 0 && col_ok) {
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < NW; ++k) sum += red[k][lane];
    partial[(size_t)j * g.nr + r] = __ldg(mt.wj + j) * sum;
  }
  if (extra) {
    __syncthreads();
    red[w][lane] = acc2;
    __syncthreads();
    if (tid == 0) {
      double sum = 0.0;
      for (int k = 0; k < NW; ++k)
        for (int l = 0; l < 32; ++l) sum += red[k][l];
      partial[(size_t)j * g.nr + r0 + 32] = __ldg(mt.wj + j) * sum;
    }
  }
}

// Strip layouts (the DRIFT_* kinds).  FP32: DRIFT_STRIP2, two strip buffers
// per persistent block; DRIFT_STRIP1, one (strips too tall for two).  Strips
// in blocks: DRIFT_STRIP2, two blocks per SM; DRIFT_STRIP1, one.  DRIFT_WINDOW: none, the
// windowed kernel, which FP64 takes unless a strip is asked for.  `want` !=
// DRIFT_AUTO asks for one kind, returned only if it fits (else DRIFT_WINDOW).
template <typename T>
static size_t strip_block_smem(int nu) {
  const int nch = (nu + 3 + DSB_ROWS - 1) / DSB_ROWS;
  return (size_t)nch * (DSB_ROWS * DS_WC * sizeof(T) + sizeof(uint64_t));
}
static bool strip_fits(int nu, int nb, bool weights) {
  // 227 KB of shared memory per block with the barriers; strips of 576 and
  // 1152 rows at most (taller ones, which would fit without the weights, have
  // been measured with windows only)
  return nu + 3 <= 1152 / nb && strip_smem(nu, STRIP_WARPS, nb, weights).total + 256 <= 232448;
}
template <typename T>
int drift_strip_width(int nu, int want) {
  if (want == DRIFT_WINDOW || (sizeof(T) == 8 && want == DRIFT_AUTO)) return DRIFT_WINDOW;
  bool fit2, fit1;
  if (sizeof(T) == 8) {
    // 228 KB per SM, 1 KB of it reserved per block; the blocks' sums are static
    const size_t n = strip_block_smem<T>(nu);
    fit2 = 2 * (n + 16 * 32 * sizeof(double) + 1024) <= 233472;
    fit1 = n + 32 * 32 * sizeof(double) <= 232448;
  } else {
    fit2 = strip_fits(nu, 2, false);
    fit1 = strip_fits(nu, 1, false);
  }
  if (want == DRIFT_STRIP2) return fit2 ? DRIFT_STRIP2 : DRIFT_WINDOW;
  if (want == DRIFT_STRIP1) return fit1 ? DRIFT_STRIP1 : DRIFT_WINDOW;
  return fit2 ? DRIFT_STRIP2 : fit1 ? DRIFT_STRIP1 : DRIFT_WINDOW;
}
// Strips of fewer than 15 trips (N_u <= 112) leave most of the persistent
// block's consumer warps without one, and each task costs its producer some
// 3 us whatever its length (four or eight strip buffers instead of two change
// nothing).  Drift in us, FP32 Hernquist, 128 slices, blocks / persistent:
// 720 x 33 34.5 / 58.2, 395 x 33 22.9 / 37.4, 720 x 65 49.8 / 63.8, 257 x 97
// 28.9 / 29.1, 720 x 105 65.1 / 70.0; 257 x 113 32.1 / 30.2, 129 x 129 24.3 /
// 23.4, 257 x 257 56.4 / 45.4.  Blocks need no pass for the far cells either
// (step of 257 x 97 x 128 59.5 us against 61.4).  Slices of one strip stay
// with the persistent blocks (33 x 97 x 128 15.4 / 12.6).  The rule takes the
// whole grid's sizes, not a batch's: results do not depend on the batching.
template <typename T>
bool drift_strip_in_blocks(int nr, int nu) {
  return sizeof(T) == 8 || (strip_trips(nu) < 15 && strip_blocks(nr) > 1);
}
int drift_strip_box_rows(int nu, bool blocks) {
  return blocks ? DSB_ROWS : strip_smem(nu, 1, 1, false).rows;
}

// A block's tasks are task b of the first `grid` ones, task (b + rot) % grid of
// the next, and so on: its strip moves by (grid + rot) % ns each time.  148
// blocks and 32 strips without rotation give every block 8 of the 32 strips,
// whose cost differs by a factor of six, so blocks drift apart in a long run:
// the drift of 1025 x 1025 x 512 PLDF took 5.28 us a slice (4.70 with 128
// slices), of 513 x 513 x 2048 1.24 (256: 1.06).  With steps coprime to ns and
// between 0.2 and 0.45 of it from either side 4.55 and 0.89, 513 x 513 x 256
// Hernquist 0.263 -> 0.248 ms; a step of one strip is worse than none (1025 x
// 1025 x 64 0.377 against 0.303), and so is one of half of them (0.326).
// Rotations from 3 on are the better ones in shorter runs (513 x 513 x 256
// 0.248 with 3, 0.253 with 1; 1025 x 1025 x 64 0.300 and 0.313), from 1 on where
// a larger one would go round the blocks more than once (1025 x 1025 x 512 4.92
// and 4.55).  Runs of fewer than 12 tasks a block keep the plain order: there
// the last tasks decide (257 x 352 x 128 0.060, rotated 0.064; 257 x 257 x 128
// 0.049, 0.047).
static int strip_rotation(int ntask, int grid, int ns) {
  if (ntask < 12 * grid) return 0;
  auto far = [&](int rot) {
    const int step = (grid + rot) % ns, near = std::min(step, ns - step);
    return std::gcd(step, ns) == 1 && 5 * near >= ns && 20 * near <= 9 * ns;
  };
  const int first = ntask < 60 * grid ? 3 : 1;
  for (int rot = 0; rot < first + ns; rot += rot ? 1 : first)
    if (far(rot)) return rot;
  for (int rot = 0; rot < ns; ++rot)  // 2 and 6 strips
    if (std::gcd(grid + rot, ns) == 1) return rot;
  return 0;
}

template <int NW, int NB, int MINB, bool WEIGHTS>
static cudaError_t drift_strip_go(const CUtensorMap *tmS, const float *C, float *f,
                                  const uint2 *fp2, const uint8_t *trip_kinds,
                                  const MomentTables &mt, double *partial, unsigned int *err,
                                  uint32_t spins, const Geometry &g, cudaStream_t st) {
  const size_t smem = strip_smem(g.nu, NW, NB, WEIGHTS).total;
  auto kern = drift_strip_kernel<NW, NB, MINB, WEIGHTS>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return e;
  const int ns = strip_blocks(g.nr), ntask = ns * g.nb, grid = std::min(ntask, nsm * MINB);
  const int rot = strip_rotation(ntask, grid, ns);
  return chain_launch(kern, dim3(grid), dim3(32 * (NW + 1)), smem, st, *tmS, C, f, fp2, trip_kinds,
                      mt, partial, err, spins, (uint32_t)rot, g);
}

cudaError_t launch_drift_strip(const CUtensorMap *tmS, int kind, const float *C, float *f,
                               const uint2 *fp2, const uint8_t *trip_kinds,
                               const MomentTables &mt, double *partial, unsigned int *err,
                               uint32_t spins, const Geometry &g, cudaStream_t st) {
  auto go = [&](auto with, auto without, int nb) {
    return (strip_fits(g.nu, nb, true) ? with : without)(tmS, C, f, fp2, trip_kinds, mt, partial,
                                                         err, spins, g, st);
  };
  switch (kind) {
    case DRIFT_STRIP2:
      return go(drift_strip_go<STRIP_WARPS, 2, 1, true>, drift_strip_go<STRIP_WARPS, 2, 1, false>,
                2);
    case DRIFT_STRIP1:
      return go(drift_strip_go<STRIP_WARPS, 1, 1, true>, drift_strip_go<STRIP_WARPS, 1, 1, false>,
                1);
    default:
      return cudaErrorInvalidValue;
  }
}

template <typename T>
cudaError_t launch_drift_strip_blocks(const CUtensorMap *tmS, int kind, const T *C, T *f,
                                      const int32_t *idx, const T *fx, const T *fy,
                                      const uint2 *fp2, const int64_t *ch_start,
                                      const int32_t *ch_len, const T *ch_val, int64_t ndrift,
                                      const MomentTables &mt, double *partial, unsigned int *err,
                                      uint32_t spins, const Geometry &g, cudaStream_t st) {
  const size_t smem = strip_block_smem<T>(g.nu);
  auto go = [&](auto kern, int nw) {
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return chain_launch(kern, dim3(strip_blocks(g.nr), g.nb), dim3(32 * nw), smem, st, *tmS, C, f,
                        idx, fx, fy, fp2, ch_start, ch_len, ch_val, ndrift, mt, partial, err,
                        spins, g);
  };
  switch (kind) {
    case DRIFT_STRIP2:
      return go(drift_strip_block_kernel<T, 16, 2>, 16);
    case DRIFT_STRIP1:
      return go(drift_strip_block_kernel<T, 32, 1>, 32);
    default:
      return cudaErrorInvalidValue;
  }
}

// ------------------------------------------------------------- edge cells
// One thread per chain (slice jl: chains [chain_lo[j], chain_lo[j + 1])) and,
// for the strip drift (EDGE), per far-tap cell of the slice.
//
// Chain: the spline value at its tail goes into the ring slot that becomes
// the tail, and, for the strip drift, the front of the ring, this drift's
// value of the chain's cell, into f; a chain of one element has its tail as
// front.  The front is loaded before the tail's gather, so that the two
// latencies overlap.  (The windowed drift reads the fronts itself: 0.010 ms
// less here, nothing there, on 513 x 513 x 128 in FP64.)
template <typename T, bool EDGE>
__global__ void __launch_bounds__(256)
    edge_kernel(const T *C, T *__restrict__ f, T *__restrict__ ch_val,
                const int64_t *__restrict__ ch_start, const int32_t *__restrict__ ch_len,
                const uint32_t *__restrict__ ch_at, const int32_t *__restrict__ t_idx,
                const double *__restrict__ t_x, const double *__restrict__ t_y,
                const int32_t *__restrict__ chain_lo, int64_t ndrift,
                const uint32_t *__restrict__ far_base, const uint32_t *__restrict__ far,
                const uint2 *__restrict__ fp2, Geometry g) {
  chain_begin();
  const int jl = blockIdx.y, j = g.j0 + jl;
  const T *Cj = C + (size_t)jl * (g.nu + 3) * g.pc;
  const size_t sb = (size_t)j * g.nu * g.nr;
  int e = blockIdx.x * 256 + threadIdx.x;
  const int c = __ldg(chain_lo + j) + e, hi = __ldg(chain_lo + j + 1);
  if (c < hi) {
    const int32_t L = __ldg(ch_len + c), code = __ldg(t_idx + c);
    T *ring = ch_val + __ldg(ch_start + c);
    // 32-bit remainder of the drift count
    const uint32_t at = ndrift <= 0xffffffffll ? (uint32_t)ndrift % (uint32_t)L
                                               : (uint32_t)(ndrift % L);
    const T front = EDGE ? ring[at] : T(0);
    T v = T(0);
    if (code >= 0)
      v = eval2d<T>(Cj, g.pc, code & 0xffff, (T)__ldg(t_x + c), code >> 16, (T)__ldg(t_y + c));
    ring[at == 0 ? L - 1 : at - 1] = v;
    if (EDGE) f[sb + __ldg(ch_at + c)] = L == 1 ? v : front;
    return;
  }
  if constexpr (EDGE) {
    e -= hi - __ldg(chain_lo + j);
    const uint32_t k = __ldg(far_base + j) + (uint32_t)e;
    if (k >= __ldg(far_base + j + 1)) return;
    const size_t cell = sb + __ldg(far + k);
    RawCell<float> w;
    w.w = __ldg(fp2 + cell);
    const Cell<float> cl = decode(w);
    f[cell] = eval2d<float>(Cj, g.pc, cl.rI, cl.x, cl.uI, cl.y);
  }
}

// most: the largest number of edge cells in a slice of this launch
template <typename T>
cudaError_t launch_edge(const T *C, T *f, T *ch_val, const EdgeTables &t, int64_t ndrift,
                        const uint2 *fp2, int most, const Geometry &g, cudaStream_t st) {
  if (most <= 0) return cudaSuccess;
  auto go = [&](auto kern) {
    return chain_launch(kern, dim3((most + 255) / 256, g.nb), dim3(256), 0, st, C, f, ch_val,
                        t.ch_start, t.ch_len, t.ch_at, t.t_idx, t.t_x, t.t_y, t.chain_lo, ndrift,
                        t.far_base, t.far, fp2, g);
  };
  if constexpr (sizeof(T) == 4)
    if (t.far_base) return go(edge_kernel<T, true>);
  return go(edge_kernel<T, false>);
}

// ------------------------------------------------------------------ moment
template <typename T>
__global__ void __launch_bounds__(32 * DR_W)
    moment_kernel(const T *f, MomentTables mt,
                  double *__restrict__ partial, Geometry g) {
  chain_begin();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  const int j = blockIdx.y;
  double acc = 0.0;
  if (r < g.nr)
    for (int u = w; u < g.nu; u += DR_W)
      acc += __ldg(mt.bu + u) * (double)f[((size_t)j * g.nu + u) * g.nr + r];
  __shared__ double red[DR_W][32];
  red[w][lane] = acc;
  __syncthreads();
  if (w == 0 && r < g.nr) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < DR_W; ++k) s += red[k][lane];
    partial[(size_t)j * g.nr + r] = __ldg(mt.wj + j) * s;
  }
}

template <typename T>
cudaError_t launch_moment(const T *f, const MomentTables &mt, double *partial,
                          const Geometry &g, cudaStream_t st) {
  dim3 grid((g.nr + 31) / 32, g.nj);
  return chain_launch(moment_kernel<T>, grid, dim3(32 * DR_W), 0, st, f, mt, partial, g);
}

// -------------------------------------------------------------- scan
constexpr int SC_THREADS = 1024;
constexpr int SC_RB = 32;  // r columns per reduction block

// grid: ceil(N_r / SC_RB) blocks; each reduces partial[:, r-strip] over J
// (compensated) into T2.  The last block to finish (threadfence reduction
// pattern, no spin-wait) computes bins, the exclusive scan, mtot and shift.
// `count` is a per-handle device counter that the last block resets to 0.

__global__ void __launch_bounds__(SC_THREADS)
    scan_kernel(const double *partial, MomentTables mt,
                double *__restrict__ T2, double *__restrict__ bins,
                double *__restrict__ Mr, double *__restrict__ shift,
                double *__restrict__ mtot, unsigned int *count, unsigned int *status,
                Geometry g) {
  __shared__ dd sh[SC_THREADS];
  __shared__ bool last;
  const int tid = threadIdx.x;
  chain_begin();
  {
    const int lr = tid % SC_RB, jg = tid / SC_RB;  // 32 groups of J
    const int ngroups = SC_THREADS / SC_RB;
    const int r = blockIdx.x * SC_RB + lr;
    dd acc{0.0, 0.0};
    if (r < g.nr)
      for (int j = jg; j < g.nj; j += ngroups)
        acc = dd_add(acc, dd{partial[(size_t)j * g.nr + r], 0.0});
    sh[tid] = acc;
    __syncthreads();
    for (int s = ngroups / 2; s > 0; s >>= 1) {
      if (jg < s) sh[tid] = dd_add(sh[tid], sh[tid + s * SC_RB]);
      __syncthreads();
    }
    if (jg == 0 && r < g.nr) T2[r] = sh[tid].hi + sh[tid].lo;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const unsigned int done = atomicAdd(count, 1u);
    last = (done == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // bins (each thread up to 2 consecutive r), then a block-wide exclusive scan
  const int per = (g.nr + SC_THREADS - 1) / SC_THREADS;  // 1 or 2
  double b[2] = {0.0, 0.0};
  dd loc{0.0, 0.0};
  for (int q = 0; q < per; ++q) {
    const int r = tid * per + q;
    if (r < g.nr) {
      const double t2 = *((volatile double *)T2 + r);
      const double t3 = (r + 1 < g.nr) ? *((volatile double *)T2 + r + 1) : 0.0;
      b[q] = (r < g.nr - 1) ? __ldg(mt.dR4 + r) * (t2 + t3) : 0.0;
      bins[r] = b[q];
      loc = dd_add(loc, dd{b[q], 0.0});
    }
  }
  // inclusive warp scan of loc
  const int lane = tid & 31, wid = tid >> 5;
  dd inc = loc;
  for (int d = 1; d < 32; d <<= 1) {
    dd o = dd_shfl_up(inc, d);
    if (lane >= d) inc = dd_add(inc, o);
  }
  __shared__ dd wsum[SC_THREADS / 32];
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    dd x = wsum[lane];
    dd xi = x;
    for (int d = 1; d < 32; d <<= 1) {
      dd o = dd_shfl_up(xi, d);
      if (lane >= d) xi = dd_add(xi, o);
    }
    wsum[lane] = dd_add(xi, dd{-x.hi, -x.lo});  // exclusive
    if (lane == 31) {
      const double total = xi.hi + xi.lo;
      *mtot = total;
      // every cell enters the mass with a positive weight, so a NaN or an
      // infinity anywhere in f makes the total non-finite
      if (!isfinite(total)) atomicOr(status, 2u);
    }
  }
  __syncthreads();
  dd ex = dd_add(wsum[wid], dd_add(inc, dd{-loc.hi, -loc.lo}));
  for (int q = 0; q < per; ++q) {
    const int r = tid * per + q;
    if (r < g.nr) {
      const double m = ex.hi + ex.lo;
      Mr[r] = m;
      shift[r] = m * __ldg(mt.Rcoef + r);
      ex = dd_add(ex, dd{b[q], 0.0});
    }
  }
  if (tid == 0) *count = 0u;
}

cudaError_t launch_scan(const double *partial, const MomentTables &mt,
                        double *T2, double *bins, double *Mr, double *shift,
                        double *mtot, unsigned int *count, unsigned int *status,
                        const Geometry &g, cudaStream_t st) {
  if (g.nr > 2 * SC_THREADS) return cudaErrorInvalidValue;
  const unsigned blocks = (g.nr + SC_RB - 1) / SC_RB;
  return chain_launch(scan_kernel, dim3(blocks), dim3(SC_THREADS), 0, st, partial, mt, T2, bins, Mr,
                      shift, mtot, count, status, g);
}

// ------------------------------------------------------------------ stats
// integrate() of Ek, S, L1, L2 (quadrature21.hxx:56-85, integrand21.hxx:82-145)
// Block: one J slice, stats_rows rows of u cells; a thread takes one r cell and
// walks down the rows, so that the radius' terms (J^2 / rm^2, a division) are
// formed once and each f row pair is loaded once.  Every term enters its sum
// compensated; block partials in double-double, 4 quantities x (hi, lo).
// Bound by the FP64 pipe (the logarithm of every non-zero cell and four
// compensated sums): 513 x 513 x 256 FP32 0.555 -> 0.359 ms (the whole call,
// its final sums and copies included, 1.11 -> 0.39 ms) against 8-row blocks
// with the division, five loads and renormalised sums per cell.
//
// 16 rows a block, fewer where those blocks leave SMs idle (two per SM wanted:
// the whole call on 2048 x 33 x 8 FP32 61 us, 110 with 16 rows always).
constexpr int ST_THREADS = 256;
static int stats_rows(int nu, int nj) {
  int rows = 16;
  while (rows > 2 && (int64_t)((nu - 1 + rows - 1) / rows) * nj < 2 * 148) rows /= 2;
  return rows;
}

template <typename T>
__global__ void __launch_bounds__(ST_THREADS)
    stats_kernel(const T *f, const double *__restrict__ R,
                 const double *__restrict__ U, const double *__restrict__ J,
                 const double *__restrict__ dR, const double *__restrict__ dU,
                 const double *__restrict__ Ct1, double *__restrict__ part, int rows,
                 Geometry g) {
  chain_begin();
  const int j = blockIdx.y;
  const int u0 = blockIdx.x * rows, u1 = min(u0 + rows, g.nu - 1);
  dd acc[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
  const double Jj = __ldg(J + j), ct = __ldg(Ct1 + j);
  for (int r = threadIdx.x; r < g.nr - 1 && u0 < u1; r += ST_THREADS) {
    const double dr = __ldg(dR + r);
    if (dr <= 0) continue;
    const double rm = __ldg(R + r) + 0.5 * dr;
    const double v2 = Jj * Jj / (rm * rm);
    const T *p = f + ((size_t)j * g.nu + u0) * g.nr + r;
    double lo = (double)p[0] + (double)p[1];
#pragma unroll 4
    for (int u = u0; u < u1; ++u) {
      p += g.nr;
      const double hi = (double)p[0] + (double)p[1];
      const double avg = (lo + hi) * 0.25;
      lo = hi;
      const double du = __ldg(dU + u);
      // a zero cell adds nothing (a NaN is not skipped)
      if (du <= 0 || avg == 0.0) continue;
      const double um = __ldg(U + u) + 0.5 * du;
      const double w = ct * du * dr;
      dd_acc(acc[0], w * (0.5 * avg * (um * um + v2)));
      dd_acc(acc[1], w * ((avg <= 0) ? 0.0 : -avg * log(avg)));
      dd_acc(acc[2], w * fabs(avg));
      dd_acc(acc[3], w * (avg * avg));
    }
  }
  for (int q = 0; q < 4; ++q)
    for (int d = 16; d > 0; d >>= 1) acc[q] = dd_add(acc[q], dd_shfl_down(acc[q], d));
  __shared__ dd ws[ST_THREADS / 32][4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0)
    for (int q = 0; q < 4; ++q) ws[wid][q] = acc[q];
  __syncthreads();
  if (threadIdx.x < 4) {
    const int q = threadIdx.x;
    const size_t b = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
    dd s{0, 0};
    for (int k = 0; k < ST_THREADS / 32; ++k) s = dd_add(s, ws[k][q]);
    part[b * 8 + 2 * q] = s.hi;
    part[b * 8 + 2 * q + 1] = s.lo;
  }
}

// block q: quantity q of all block partials, in a fixed order
__global__ void __launch_bounds__(ST_THREADS)
    stats_sum_kernel(const double *part, int nblk, double *__restrict__ out4) {
  chain_begin();
  const int q = blockIdx.x;
  dd s{0, 0};
  for (int b = threadIdx.x; b < nblk; b += ST_THREADS) {
    const double2 p = reinterpret_cast<const double2 *>(part + (size_t)b * 8)[q];
    s = dd_add(s, dd{p.x, p.y});
  }
  for (int d = 16; d > 0; d >>= 1) s = dd_add(s, dd_shfl_down(s, d));
  __shared__ dd ws[ST_THREADS / 32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < ST_THREADS / 32; ++k) s = dd_add(s, ws[k]);
    out4[q] = s.hi + s.lo;
  }
}

size_t stats_blocks(int nu, int nj) {
  const int rows = stats_rows(nu, nj);
  return (size_t)((nu - 1 + rows - 1) / rows) * nj;
}

template <typename T>
cudaError_t launch_stats(const T *f, const double *R, const double *U,
                         const double *J, const double *dR, const double *dU,
                         const double *Ct1, double *part, double *out4,
                         const Geometry &g, cudaStream_t st) {
  const int rows = stats_rows(g.nu, g.nj);
  dim3 grid((g.nu - 1 + rows - 1) / rows, g.nj);
  const cudaError_t e = chain_launch(stats_kernel<T>, grid, dim3(ST_THREADS), 0, st, f, R, U, J,
                                     dR, dU, Ct1, part, rows, g);
  if (e != cudaSuccess) return e;
  return chain_launch(stats_sum_kernel, dim3(4), dim3(ST_THREADS), 0, st, part,
                      (int)stats_blocks(g.nu, g.nj), out4);
}

// ------------------------------------------------------------ conversions
template <typename T>
__global__ void convert_in_kernel(const double *__restrict__ s, T *__restrict__ d,
                                  size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    d[i] = (T)s[i];
}
template <typename T>
__global__ void convert_out_kernel(const T *__restrict__ s, double *__restrict__ d,
                                   size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    d[i] = (double)s[i];
}
template <typename T>
__global__ void nonfinite_kernel(const T *__restrict__ s, size_t n,
                                 unsigned int *flag) {
  unsigned int bad = 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    bad |= !isfinite((double)s[i]);
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1u);
}

static unsigned grid_for(size_t n) {
  size_t b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  if (b == 0) b = 1;
  return (unsigned)b;
}

template <typename T>
cudaError_t launch_convert_in(const double *src, T *dst, size_t n,
                              cudaStream_t st) {
  convert_in_kernel<T><<<grid_for(n), 256, 0, st>>>(src, dst, n);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_convert_out(const T *src, double *dst, size_t n,
                               cudaStream_t st) {
  convert_out_kernel<T><<<grid_for(n), 256, 0, st>>>(src, dst, n);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_nonfinite(const T *f, size_t n, unsigned int *flag,
                             cudaStream_t st) {
  nonfinite_kernel<T><<<grid_for(n), 256, 0, st>>>(f, n, flag);
  return cudaGetLastError();
}

#define VLS_INST(T)                                                            \
  template int drift_strip_width<T>(int, int);                                  \
  template bool drift_strip_in_blocks<T>(int, int);                             \
  template cudaError_t launch_drift_strip_blocks<T>(                            \
      const CUtensorMap *, int, const T *, T *, const int32_t *, const T *, const T *, \
      const uint2 *, const int64_t *, const int32_t *, const T *, int64_t,       \
      const MomentTables &, double *, unsigned int *, uint32_t, const Geometry &, \
      cudaStream_t);                                                            \
  template cudaError_t launch_drift_tma<T>(                                     \
      const CUtensorMap *, const T *, T *, const int32_t *, const T *, const T *, \
      const uint2 *, const int16_t *, const int64_t *, const int32_t *, const T *, \
      int64_t, const MomentTables &, double *, unsigned int *, uint32_t,         \
      const Geometry &, cudaStream_t);                                          \
  template cudaError_t launch_window_rows<T>(const int32_t *, const uint2 *, int16_t *, int, \
                                             int, int, cudaStream_t);           \
  template cudaError_t launch_edge<T>(const T *, T *, T *, const EdgeTables &, int64_t, \
                                      const uint2 *, int, const Geometry &, cudaStream_t); \
  template cudaError_t launch_moment<T>(const T *, const MomentTables &,        \
                                        double *, const Geometry &,             \
                                        cudaStream_t);                          \
  template cudaError_t launch_stats<T>(                                         \
      const T *, const double *, const double *, const double *,                \
      const double *, const double *, const double *, double *, double *,       \
      const Geometry &, cudaStream_t);                                          \
  template cudaError_t launch_convert_in<T>(const double *, T *, size_t,        \
                                            cudaStream_t);                      \
  template cudaError_t launch_convert_out<T>(const T *, double *, size_t,       \
                                             cudaStream_t);                     \
  template cudaError_t launch_nonfinite<T>(const T *, size_t, unsigned int *,   \
                                           cudaStream_t);

VLS_INST(float)
VLS_INST(double)

#define VLS_INST_TR(T, R)                                                       \
  template cudaError_t launch_ucol<T, R>(bool, const T *, T *, const double *,  \
                                         const Geometry &, const DirTables &,   \
                                         cudaStream_t);                         \
  template cudaError_t launch_prer<T, R>(const T *, T *, const Geometry &,      \
                                         const DirTables &, cudaStream_t);

VLS_INST_TR(double, double)
VLS_INST_TR(float, double)
VLS_INST_TR(float, float)

}  // namespace vls
