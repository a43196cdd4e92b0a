// GROG self-calibration and gridding (src/GROG.jl).
//
// grog_calib (src/GROG.jl:14-51), per spoke of Nr samples and Nc coils:
//   G = (D1 \ D2)^T with D1 = rows 1..Nr-1, D2 = rows 2..Nr,   v = log(G),
// then lnG[:, i, j] = nm \ v[:, i, j] over all spokes, nm = Nr * (k_2 - k_1).
// The least squares run in float64 through the normal equations (Gram
// matrices accumulated in float64, Gauss-Jordan with partial pivoting); the
// principal matrix logarithm runs in float32, the precision the reference
// computes log(G) in, by inverse scaling and squaring: Denman-Beavers square
// roots until ||Y - I||_F <= 0.8, then log(Y) = 2 atanh((Y - I)(Y + I)^{-1}) by
// its power series, times 2^s (Higham, Functions of Matrices, SIAM 2008, ch. 11).
// (A quadrature that needed ||Y - I||_F <= 1/4 took one or two more square roots,
// whose roundings 2^s multiplies, and twelve more inversions.)
//
// grog_gridding! (src/GROG.jl:73-102): per sample and dimension the grid index
// follows the reference's float32/float64 promotion bit for bit, and
// data <- exp(shift lnG_d) data is applied as exp(s_j lnG_d) exp((shift - s_j) lnG_d)
// on the Nc x Nrep block: the first factor from a per-call table over a grid of
// s_j, the second as a Horner-evaluated Taylor series of its action (the
// reference forms the Higham-2005 Pade exponential of each float32 matrix and
// multiplies).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "common.cuh"

namespace mrsr {

constexpr int kGrogMaxCoils = 32;
// log(Y) = 2 atanh(Z), Z = (Y - I)(Y + I)^{-1}: 21 terms of the series, in blocks of three.  With
// ||Y - I|| <= 0.8, |z| <= 2/3 and what is left out is below 1e-9 of the result.
constexpr float kLogMax2 = 0.64f;  // 0.8^2
constexpr int kLogBlocks = 7;

// ------------------------------------------------------- spoke Grams ---
// A = D1^H D1, B = D1^H D2 for spoke `blockIdx.x`; one thread per (i, j).  The sums run on
// the float32 cores in float-float form: each product is split exactly into p + e (one
// FMA) and added to a (hi, lo) pair by Knuth's TwoSum, the compensated dot product of
// Ogita, Rump and Oishi (SIAM J. Sci. Comput. 26, 2005): the result is as accurate as a
// float64 sum up to a relative n^2 u^2 of sum |d_i d_j| (u = 2^-24), which float64
// itself only meets to n u_64.  The rounded intrinsics keep the compiler from fusing the
// product into the following addition, which would lose the exact split.
struct FF {
  float hi = 0.f, lo = 0.f;
};
__device__ __forceinline__ void ff_madd(FF& s, float a, float b) {
  const float p = __fmul_rn(a, b);
  const float e = fmaf(a, b, -p);  // a b = p + e exactly
  const float t = __fadd_rn(s.hi, p);
  const float z = __fsub_rn(t, s.hi);
  const float err = __fadd_rn(__fsub_rn(s.hi, __fsub_rn(t, z)), __fsub_rn(p, z));  // s.hi + p = t + err
  s.hi = t;
  s.lo = __fadd_rn(s.lo, __fadd_rn(err, e));
}
__device__ __forceinline__ double ff_value(const FF& s) { return (double)s.hi + (double)s.lo; }

constexpr int kGramRows = 128;  // samples of a spoke staged in shared memory at a time

struct GramArgs {
  const float2* data;   // (ns_pf, nt, nc, nrep)
  int64_t ns_pf, nt;
  int nc, nrep, nr, spf;  // spokes per frame
  double2* AB;          // [spoke][2][nc][nc] (column-major i + nc j)
};

__global__ void __launch_bounds__(1024, 2) k_grog_gram(GramArgs a) {
  extern __shared__ float2 sd[];  // [row][coil], row stride nc + 1 (conflict-free staging)
  const int n = a.nc, ld = n + 1;
  const int64_t ip = blockIdx.x;
  const int64_t rep = ip / ((int64_t)a.spf * a.nt);
  const int64_t rem = ip - rep * a.spf * a.nt;
  const int64_t t = rem / a.spf;
  const int64_t sif = rem - t * a.spf;
  const int64_t ns_tot = a.ns_pf * a.nt;
  const float2* src = a.data + sif * a.nr + a.ns_pf * t + ns_tot * a.nc * rep;  // coil stride ns_tot
  const int i = threadIdx.x % kGrogMaxCoils, j = threadIdx.x / kGrogMaxCoils;
  const bool act = i < n && j < n;
  FF are, aim, bre, bim;
  for (int r0 = 0; r0 + 1 < a.nr; r0 += kGramRows) {
    const int rows = min(kGramRows + 1, a.nr - r0);  // one extra row: B reads sample r + 1
    __syncthreads();
    for (int e = threadIdx.x; e < rows * n; e += blockDim.x) {
      const int r = e % rows, c = e / rows;
      sd[r * ld + c] = src[r0 + r + ns_tot * c];
    }
    __syncthreads();
    if (act) {
      const int last = min(kGramRows, a.nr - 1 - r0);
      for (int r = 0; r < last; ++r) {
        const float2 di = sd[r * ld + i], dj = sd[r * ld + j], dk = sd[(r + 1) * ld + j];
        // conj(di) dj and conj(di) dk
        ff_madd(are, di.x, dj.x);
        ff_madd(are, di.y, dj.y);
        ff_madd(aim, di.x, dj.y);
        ff_madd(aim, -di.y, dj.x);
        ff_madd(bre, di.x, dk.x);
        ff_madd(bre, di.y, dk.y);
        ff_madd(bim, di.x, dk.y);
        ff_madd(bim, -di.y, dk.x);
      }
    }
  }
  if (act) {
    double2* out = a.AB + ip * 2 * a.nc * a.nc;
    out[i + a.nc * j] = make_double2(ff_value(are), ff_value(aim));
    out[a.nc * a.nc + i + a.nc * j] = make_double2(ff_value(bre), ff_value(bim));
  }
}

// ------------------------------------------ small dense linear algebra ---
// One CTA of four warps per spoke, n <= 32.  Matrices sit in registers, a warp on every fourth
// column and lane r on row r, so an elimination step is two shuffles and four multiply-adds per
// column and one barrier; only the pivot column goes through shared memory.  Pivoting is
// implicit: rows stay where they are, the pivot of step k is the largest entry of column k in a
// row not used before, and the permutation is undone when the result is written.
constexpr int kGjWarps = 4;
constexpr int kGjThreads = 32 * kGjWarps;
constexpr int kGjCols = kGrogMaxCoils / kGjWarps;  // columns of an n x n matrix per warp

template <class C> struct Cx;
template <> struct Cx<double2> {
  using R = double;
  static constexpr double kTiny = 1e-280;  // |pivot|^2 below this: the column is singular
  static __device__ __forceinline__ double2 mk(double x, double y) { return make_double2(x, y); }
};
template <> struct Cx<float2> {
  using R = float;
  static constexpr float kTiny = 1e-36f;
  static __device__ __forceinline__ float2 mk(float x, float y) { return make_float2(x, y); }
};
template <class C> __device__ __forceinline__ C cx_zero() { return Cx<C>::mk(0, 0); }
template <class C> __device__ __forceinline__ C cx_mul(C a, C b) {
  return Cx<C>::mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <class C> __device__ __forceinline__ C cx_sub(C a, C b) { return Cx<C>::mk(a.x - b.x, a.y - b.y); }
// a - b c
template <class C> __device__ __forceinline__ C cx_msub(C a, C b, C c) {
  return Cx<C>::mk(a.x - b.x * c.x + b.y * c.y, a.y - b.x * c.y - b.y * c.x);
}
template <class C> __device__ __forceinline__ typename Cx<C>::R cx_abs2(C a) { return a.x * a.x + a.y * a.y; }
template <class C> __device__ __forceinline__ C cx_shfl(C v, int src) {
  return Cx<C>::mk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// Lane of the largest v >= 0 among the lanes of `in` (at least one); the first of equals.
__device__ __forceinline__ int lane_of_max(float v, bool in) {
  const unsigned key = in ? __float_as_uint(v) + 1u : 0u;  // non-negative floats order like their bits
  return __ffs(__ballot_sync(0xffffffffu, key == __reduce_max_sync(0xffffffffu, key))) - 1;
}
__device__ __forceinline__ int lane_of_max(double v, bool in) {
  const unsigned hi = in ? (unsigned)__double2hiint(v) + 1u : 0u;
  const bool top = hi == __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = top ? (unsigned)__double2loint(v) : 0u;
  const unsigned best = __reduce_max_sync(0xffffffffu, lo);
  return __ffs(__ballot_sync(0xffffffffu, top && lo == best)) - 1;
}

// Pivot record of one elimination step, double-buffered by step parity.
template <class C> struct GjStep {
  C f[2][kGrogMaxCoils];  // column k
  C rinv[2];              // 1 / pivot, 0 if |pivot|^2 < kTiny
  int p[2];               // pivot row
};

// Pivot of a column (lane r holding row r) among the rows outside `used`, first of the largest;
// writes record b.
template <class C>
__device__ __forceinline__ void gj_pivot(C v, unsigned used, int n, GjStep<C>& st, int b) {
  const int lane = threadIdx.x & 31;
  const int p = lane_of_max(cx_abs2(v), lane < n && !((used >> lane) & 1u));
  const C vp = cx_shfl(v, p);
  st.f[b][lane] = v;
  if (lane == 0) {
    const typename Cx<C>::R d = cx_abs2(vp);
    const bool s = !(d >= Cx<C>::kTiny);
    st.p[b] = p;
    st.rinv[b] = s ? cx_zero<C>() : Cx<C>::mk(vp.x / d, -vp.y / d);
  }
}

// One step's shared part: the lane's multiplier (0 in the pivot row, and all 0 for a singular
// column, whose unknown comes out as 0), the rows used so far, and what the pivot row's lane keeps.
template <class C>
struct GjLane {
  unsigned used = 0;
  int step = 0;            // the step that took this lane's row
  C rinv = cx_zero<C>();   // 1 / its pivot
  __device__ __forceinline__ C take(const GjStep<C>& st, int k, int& p) {
    const int lane = threadIdx.x & 31, b = k & 1;
    p = st.p[b];
    const C ri = st.rinv[b];
    const C g = cx_mul(st.f[b][lane], ri);
    used |= 1u << p;
    if (lane == p) {
      step = k;
      rinv = ri;
      return cx_zero<C>();
    }
    return g;
  }
};

// X = A^{-1} B for column-major n x n A, B in global memory; out(i, j, X_ij).  The pivot row goes
// through shared memory (rows[warp]), where one lane per column scales it: float64 runs at 1/60
// of the float32 rate, and every lane scaling the entry it gets by a shuffle doubles its work.
template <class C, class Out>
__device__ __forceinline__ void gj_solve(const C* A, const C* B, int n, GjStep<C>& st, C (*rows)[2 * kGjCols], Out&& out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  C v[2 * kGjCols];  // columns of A, then of B
#pragma unroll
  for (int q = 0; q < kGjCols; ++q) {
    const int c = warp + kGjWarps * q;
    const bool in = lane < n && c < n;
    v[q] = in ? A[lane + n * c] : cx_zero<C>();
    v[kGjCols + q] = in ? B[lane + n * c] : cx_zero<C>();
  }
  unsigned used = 0;
  int mine = 0;  // the step that took this lane's row
  if (warp == 0) gj_pivot(v[0], used, n, st, 0);
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const int b = k & 1, p = st.p[b];
    const C ri = st.rinv[b], f = st.f[b][lane];
    const bool sing = ri.x == 0 && ri.y == 0;
    used |= 1u << p;
    if (lane == p) {
      mine = k;
#pragma unroll
      for (int q = 0; q < 2 * kGjCols; ++q) rows[warp][q] = v[q];
    }
    __syncwarp();
    if (lane < 2 * kGjCols) rows[warp][lane] = cx_mul(rows[warp][lane], ri);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2 * kGjCols; ++q) {
      const int c = warp + kGjWarps * q;  // columns of A up to k are not read again
      const bool of_b = q >= kGjCols;
      if (of_b || (c > k && c < n)) {
        const C rk = rows[warp][q];
        if (lane != p) {
          if (!sing) v[q] = cx_sub(v[q], cx_mul(f, rk));
        } else if (!sing || of_b) {  // a singular column: its unknown is 0
          v[q] = rk;
        }
        if (!of_b && c == k + 1) gj_pivot(v[q], used, n, st, b ^ 1);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < kGjCols; ++q) {
    const int c = warp + kGjWarps * q;
    if (lane < n && c < n) out(mine, c, v[kGjCols + q]);
  }
}

// dst = A^{-1} (shared memory, column-major n x n) for the matrix whose entry (i, j) is a(i, j),
// in place in registers: a processed column turns into a column of the inverse.  AtStep: pivot
// rows are scaled by 1 / pivot at their step (twice the instructions).
template <bool AtStep, class C, class In>
__device__ __forceinline__ void gj_invert(C* dst, int n, GjStep<C>& st, In&& a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  C v[kGjCols];
  int pc[kGjCols];
#pragma unroll
  for (int q = 0; q < kGjCols; ++q) {
    const int c = warp + kGjWarps * q;
    v[q] = lane < n && c < n ? a(lane, c) : cx_zero<C>();
    pc[q] = 0;
  }
  GjLane<C> own;
  if (warp == 0) gj_pivot(v[0], own.used, n, st, 0);
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    int p;
    const C g = own.take(st, k, p);
    if constexpr (AtStep) {
      const C ri = st.rinv[k & 1], f = st.f[k & 1][lane];
      const bool sing = ri.x == 0 && ri.y == 0;
#pragma unroll
      for (int q = 0; q < kGjCols; ++q) {
        const C rk = cx_mul(cx_shfl(v[q], p), ri);
        if (lane != p) {
          if (!sing) v[q] = cx_sub(v[q], cx_mul(f, rk));
        } else if (!sing || warp + kGjWarps * q < k) {
          v[q] = rk;
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < kGjCols; ++q) v[q] = cx_msub(v[q], g, cx_shfl(v[q], p));
    }
    if (warp == k % kGjWarps) {  // column k: what is left of the unit column of row p
#pragma unroll
      for (int q = 0; q < kGjCols; ++q)
        if (q == k / kGjWarps) {
          v[q] = lane != p ? Cx<C>::mk(-g.x, -g.y) : AtStep ? own.rinv : Cx<C>::mk(1, 0);
          pc[q] = p;
        }
    }
    if (k + 1 < n && warp == (k + 1) % kGjWarps) {
#pragma unroll
      for (int q = 0; q < kGjCols; ++q)
        if (q == (k + 1) / kGjWarps) gj_pivot(v[q], own.used, n, st, (k & 1) ^ 1);
    }
    __syncthreads();
  }
  // row p_i, column k holds entry (i, p_k) of the inverse (times pivot i)
#pragma unroll
  for (int q = 0; q < kGjCols; ++q) {
    const int c = warp + kGjWarps * q;
    if (lane < n && c < n) dst[own.step + n * pc[q]] = AtStep ? v[q] : cx_mul(v[q], own.rinv);
  }
  __syncthreads();
}

// acc[q] += (A B)(lane, warp + 4 q) for column-major n x n matrices in shared memory
__device__ __forceinline__ void mat_mul_acc(float2* acc, const float2* A, const float2* B, int n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = lane < n ? lane : 0;
  auto step = [&](float2 u, int q, float2 v) {
    acc[q].x = fmaf(u.x, v.x, fmaf(-u.y, v.y, acc[q].x));
    acc[q].y = fmaf(u.x, v.y, fmaf(u.y, v.x, acc[q].y));
  };
  int l = 0;
  if ((n & 1) == 0) {  // two entries of B per 16-byte load
    for (; l < n; l += 2) {
      const float2 u0 = A[row + n * l], u1 = A[row + n * (l + 1)];
#pragma unroll
      for (int q = 0; q < kGjCols; ++q) {
        const int c = warp + kGjWarps * q;
        if (c < n) {
          const float4 v = *reinterpret_cast<const float4*>(B + l + n * c);
          step(u0, q, make_float2(v.x, v.y));
          step(u1, q, make_float2(v.z, v.w));
        }
      }
    }
  }
  for (; l < n; ++l) {
    const float2 u = A[row + n * l];
#pragma unroll
    for (int q = 0; q < kGjCols; ++q) {
      const int c = warp + kGjWarps * q;
      if (c < n) step(u, q, B[l + n * c]);
    }
  }
}

// Block sum of a per-thread value (all threads receive it).
__device__ __forceinline__ float block_sum(float acc, float* red) {
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  float s = 0.f;
  for (int w = 0; w < kGjWarps; ++w) s += red[w];
  __syncthreads();
  return s;
}

// Per spoke: G = X^T in float32, X = A^{-1} B in float64 (A is a Gram matrix: its condition
// number is the square of the data's).
__global__ void __launch_bounds__(kGjThreads) k_grog_solve(const double2* AB, int n, float2* G) {
  __shared__ GjStep<double2> st;
  __shared__ double2 rows[kGjWarps][2 * kGjCols];
  const int64_t nn = n * n;
  const double2* A = AB + (int64_t)blockIdx.x * 2 * nn;
  float2* g = G + (int64_t)blockIdx.x * nn;
  gj_solve(A, A + nn, n, st, rows, [&](int i, int j, double2 x) { g[j + n * i] = make_float2((float)x.x, (float)x.y); });
}

struct LogArgs {
  const float2* G;      // [spoke][nc][nc]
  int nc;
  double2* vth;         // [spoke][nc][nc] = log(G)
  int* err;
};

// One spoke: v = log(G) in float32 (the reference works in the data's float32 throughout).
// For 32 coils about 30 inversions and 40 products, bound by instruction issue: 1000 spokes take
// 1.6 ms, and k_grog_solve 0.73 ms (float64 rate), against 5.9 ms for the two with the matrices
// in shared memory, right-hand sides carried along and 12 inversions in the quadrature.
__global__ void __launch_bounds__(kGjThreads, 7) k_grog_log(LogArgs a) {
  extern __shared__ __align__(16) float2 lsm[];
  const int n = a.nc, nn = n * n;
  __shared__ GjStep<float2> st;
  __shared__ float red[kGjWarps];
  float2* Y = lsm;            // root iterate
  float2* Z = lsm + nn;       // M of the iteration, then X
  float2* T = lsm + 2 * nn;   // inverses
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // each thread owns the entries (lane, warp + 4 q) of every matrix
  auto entries = [&](auto&& f) {
#pragma unroll
    for (int q = 0; q < kGjCols; ++q) {
      const int c = warp + kGjWarps * q;
      if (lane < n && c < n) f(q, lane + n * c, lane == c);
    }
  };
  const float2* G = a.G + (int64_t)blockIdx.x * nn;
  entries([&](int, int e, bool) { Y[e] = G[e]; });
  // inverse scaling: square roots until ||Y - I||_F <= 0.8, each by the product form of
  // the Denman-Beavers iteration (Cheng, Higham, Kenney and Laub, SIAM J. Matrix Anal.
  // Appl. 22, 2001): M0 = Y0 = A, Y <- Y (I + M^{-1}) / 2, M <- I/2 + (M + M^{-1}) / 4;
  // Y -> A^{1/2} and M -> I quadratically.  With Y = A^{1/2} (I + E), M = (I + E)^2 and the
  // step maps E to E^2 / 2: once ||M - I||_F^2 <= 1e-8 n, one more step brings E to the
  // float32 rounding level.  Spokes have eigenvalues e^{i (pi - d)} with d down to 1e-4: the
  // first root's M then comes within d^2 / 4 of singular, and what it gives depends on each
  // rounding, so the inversions of the first two roots (and k_grog_solve) scale a pivot row at
  // its step, the order the results of this code have always had; the following roots stay
  // clear of the negative axis and their inversions scale the rows at the end.
  int s = 0;
  for (; s < 40; ++s) {
    float d2 = 0.f;
    entries([&](int, int e, bool diag) {
      float2 v = Y[e];
      Z[e] = v;
      if (diag) v.x -= 1.f;
      d2 += v.x * v.x + v.y * v.y;
    });
    if (!(block_sum(d2, red) > kLogMax2)) break;
    bool last = false;
    for (int it = 0; it < 40; ++it) {
      auto m = [&](int i, int j) { return Z[i + n * j]; };
      if (s < 2)
        gj_invert<true>(T, n, st, m);
      else
        gj_invert<false>(T, n, st, m);
      float2 acc[kGjCols];
      entries([&](int q, int e, bool) { acc[q] = Y[e]; });
      mat_mul_acc(acc, Y, T, n);  // Y (I + M^{-1})
      __syncthreads();
      float dacc = 0.f;
      entries([&](int q, int e, bool diag) {
        Y[e] = make_float2(0.5f * acc[q].x, 0.5f * acc[q].y);
        float2 m = make_float2(0.25f * (Z[e].x + T[e].x) + (diag ? 0.5f : 0.f), 0.25f * (Z[e].y + T[e].y));
        Z[e] = m;
        if (diag) m.x -= 1.f;
        dacc += m.x * m.x + m.y * m.y;
      });
      const float tot = block_sum(dacc, red);
      if (last) break;
      last = tot <= 1e-8f * n;
    }
  }
  if (s >= 40 && threadIdx.x == 0) atomicExch(a.err, 2);
  // 2 atanh(Z) = 2 Z sum_k W^k / (2 k + 1), W = Z^2, the sum by Horner's rule in W^3
  gj_invert<false>(T, n, st, [&](int i, int j) {
    const float2 v = Y[i + n * j];
    return make_float2(v.x + (i == j ? 1.f : 0.f), v.y);
  });
  entries([&](int, int e, bool diag) {
    if (diag) Y[e].x -= 1.f;
  });
  __syncthreads();
  float2 acc[kGjCols], w1[kGjCols], w2[kGjCols];
  // acc = A B (+ what acc holds), stored to dst
  auto product = [&](const float2* A, const float2* B, float2* dst, bool add) {
    if (!add) {
#pragma unroll
      for (int q = 0; q < kGjCols; ++q) acc[q] = make_float2(0.f, 0.f);
    }
    mat_mul_acc(acc, A, B, n);
    __syncthreads();
    entries([&](int q, int e, bool) { dst[e] = acc[q]; });
    __syncthreads();
  };
  product(Y, T, Z, false);  // Z
  product(Z, Z, Y, false);  // W
#pragma unroll
  for (int q = 0; q < kGjCols; ++q) w1[q] = acc[q];
  product(Y, Y, T, false);  // W^2
#pragma unroll
  for (int q = 0; q < kGjCols; ++q) w2[q] = acc[q];
  product(Y, T, T, false);  // W^3
  for (int b = kLogBlocks - 1; b >= 0; --b) {
    const float c0 = 1.f / (float)(6 * b + 1), c1 = 1.f / (float)(6 * b + 3), c2 = 1.f / (float)(6 * b + 5);
    entries([&](int q, int, bool diag) {
      acc[q] = make_float2(fmaf(c2, w2[q].x, fmaf(c1, w1[q].x, diag ? c0 : 0.f)), fmaf(c2, w2[q].y, c1 * w1[q].y));
    });
    if (b == kLogBlocks - 1) {
      entries([&](int q, int e, bool) { Y[e] = acc[q]; });
      __syncthreads();
    } else {
      product(T, Y, Y, true);
    }
  }
#pragma unroll
  for (int q = 0; q < kGjCols; ++q) acc[q] = make_float2(0.f, 0.f);
  mat_mul_acc(acc, Z, Y, n);
  const double sc = ldexp(2.0, s);
  double2* out = a.vth + (int64_t)blockIdx.x * nn;
  entries([&](int q, int e, bool) { out[e] = make_double2(sc * acc[q].x, sc * acc[q].y); });
}

// nm (nspk x d) and the d x d pseudo-inverse factor P = (nm^T nm)^{-1}; single CTA.
struct NmArgs {
  const float* trj;   // (d, ns_pf, nt)
  int d, nr, spf;
  int64_t ns_pf, nt, nspk0;  // spokes of one repetition
  double* nm;         // [nspk0][d]
  double* Pinv;       // [d][d]
  int nrep;
};

__global__ void k_grog_nm(NmArgs a) {
  __shared__ double red[9][32];
  double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int64_t ip = threadIdx.x; ip < a.nspk0; ip += blockDim.x) {
    const int64_t t = ip / a.spf, sif = ip - t * a.spf;
    const int64_t s0 = sif * a.nr;
    double v[3];
    for (int dd = 0; dd < a.d; ++dd) {
      const float k0 = a.trj[dd + (int64_t)a.d * (s0 + a.ns_pf * t)];
      const float k1 = a.trj[dd + (int64_t)a.d * (s0 + 1 + a.ns_pf * t)];
      const float df = __fsub_rn(k1, k0);
      v[dd] = (double)__fmul_rn(df, (float)a.nr);  // Float32 diff times Int Nr -> Float32
      a.nm[ip * a.d + dd] = v[dd];
    }
    for (int p = 0; p < a.d; ++p)
      for (int q = 0; q < a.d; ++q) acc[p * 3 + q] += v[p] * v[q];
  }
  for (int e = 0; e < 9; ++e) {
    double x = acc[e];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[e][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double m[9];
    for (int e = 0; e < 9; ++e) {
      double s = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[e][w];
      m[e] = s * a.nrep;  // the nm rows repeat once per repetition
    }
    if (a.d == 2) {
      const double det = m[0] * m[4] - m[1] * m[3];
      a.Pinv[0] = m[4] / det;
      a.Pinv[1] = -m[1] / det;
      a.Pinv[2] = -m[3] / det;
      a.Pinv[3] = m[0] / det;
    } else {
      const double A = m[0], B = m[1], C = m[2], D = m[3], E = m[4], F = m[5], G = m[6], H = m[7], I = m[8];
      const double c00 = E * I - F * H, c01 = -(D * I - F * G), c02 = D * H - E * G;
      const double det = A * c00 + B * c01 + C * c02;
      double inv[9] = {c00, -(B * I - C * H), B * F - C * E, c01, A * I - C * G, -(A * F - C * D), c02,
                       -(A * H - B * G), A * E - B * D};
      for (int e = 0; e < 9; ++e) {
        const int r = e / 3, c = e % 3;
        a.Pinv[r * 3 + c] = inv[r * 3 + c] / det;
      }
    }
  }
}

// lnG[d, i, j] = sum_p (P nm^T)[d, p] v[p, i, j] over all spokes (all repetitions).  A block
// takes 32 entries, its 32 warps every 32nd spoke, in float64, joined in a fixed order: 76 us
// for 1000 spokes of 32 coils against 810 us for a thread per entry over all spokes.
__global__ void __launch_bounds__(1024) k_grog_lng(const double* nm, const double* Pinv, const double2* vth, int d, int nc,
                                                   int64_t nspk0, int nrep, float2* lnG) {
  __shared__ double2 part[32][33];
  const int nn = nc * nc, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;
  double2 acc[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
  for (int64_t p = warp; p < nspk0 * nrep; p += 32) {
    const int64_t ip = p % nspk0;
    const double2 v = e < nn ? vth[p * nn + e] : make_double2(0, 0);
    for (int dd = 0; dd < d; ++dd) {
      double c = 0.0;
      for (int q = 0; q < d; ++q) c += Pinv[dd * d + q] * nm[ip * d + q];
      acc[dd].x += c * v.x;
      acc[dd].y += c * v.y;
    }
  }
  for (int dd = 0; dd < d; ++dd) {
    part[warp][lane] = acc[dd];
    __syncthreads();
    if (warp == 0 && e < nn) {
      double2 t = make_double2(0, 0);
      for (int w = 0; w < 32; ++w) {
        t.x += part[w][lane].x;
        t.y += part[w][lane].y;
      }
      lnG[dd + (int64_t)d * e] = make_float2((float)t.x, (float)t.y);
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------- gridding ---
// exp(shift L_d) v for every sample, factored as exp(s_j L_d) exp((shift - s_j) L_d) v with
// s_j = j h the table point nearest the shift: the table exp(s_j L_d), j = -J..J, is built
// once per call, and the remaining factor, ||(shift - s_j) L_d||_1 <= h ||L_d||_1 / 2 <= 1/2,
// needs a Taylor polynomial of degree <= 8 instead of a scaled degree-24 series.
constexpr int kGridTabMax = 8;       // J <= 8: 17 tables of n x n in shared memory
constexpr int kExpTaylor = 12;       // table entries: ||.||_1 <= 1 after scaling, 1/13! < 2^-32
constexpr float kGridTol = 7.4505806e-9f;  // 2^-27: Taylor truncation bound of the remainder

// Table of exp(s_j L) for s_j = (blockIdx.x - J) h, one CTA per entry: scaling to
// ||s_j L / 2^q||_1 <= 1, degree-12 Taylor polynomial by Horner, q squarings (float32,
// the precision the reference forms its exponentials in).
struct TabArgs {
  const float2* lnG;  // (d, nc, nc)
  int d, dd, n, J;
  float h, lnorm;     // table spacing, ||L_dd||_1
  float2* tab;        // [2J + 1][nc][nc]
};

__global__ void __launch_bounds__(1024) k_grog_exp_table(TabArgs a) {
  __shared__ float2 Y[kGrogMaxCoils * kGrogMaxCoils], E[kGrogMaxCoils * kGrogMaxCoils],
      T[kGrogMaxCoils * kGrogMaxCoils];
  const int n = a.n, nn = n * n;
  const float s = (float)((int)blockIdx.x - a.J) * a.h;
  const float nrm = fabsf(s) * a.lnorm;
  int q = 0;
  while (nrm > ldexpf(1.f, q) && q < 60) ++q;
  const float sc = ldexpf(s, -q);
  for (int e = threadIdx.x; e < nn; e += blockDim.x) {
    const float2 l = a.lnG[a.dd + (int64_t)a.d * e];
    Y[e] = make_float2(sc * l.x, sc * l.y);
    E[e] = make_float2((e % n) == (e / n) ? 1.f : 0.f, 0.f);
  }
  __syncthreads();
  auto matmul = [&](const float2* A, const float2* B) {  // T = A B
    for (int e = threadIdx.x; e < nn; e += blockDim.x) {
      const int i = e % n, c = e / n;
      float2 acc = make_float2(0.f, 0.f);
      for (int l = 0; l < n; ++l) acc = cadd(acc, cmul(A[i + n * l], B[l + n * c]));
      T[e] = acc;
    }
    __syncthreads();
  };
  for (int k = kExpTaylor; k >= 1; --k) {  // E <- I + (Y / k) E
    matmul(Y, E);
    const float rk = 1.f / (float)k;
    for (int e = threadIdx.x; e < nn; e += blockDim.x)
      E[e] = make_float2(((e % n) == (e / n) ? 1.f : 0.f) + rk * T[e].x, rk * T[e].y);
    __syncthreads();
  }
  for (int r = 0; r < q; ++r) {
    matmul(E, E);
    for (int e = threadIdx.x; e < nn; e += blockDim.x) E[e] = T[e];
    __syncthreads();
  }
  float2* out = a.tab + (int64_t)blockIdx.x * nn;
  for (int e = threadIdx.x; e < nn; e += blockDim.x) out[e] = E[e];
}

struct GridArgs {
  float2* data;           // (ns_pf, nt, nc, nrep), in place
  const float* trj;       // (d, ns_pf, nt)
  const float2* lnG;      // (d, nc, nc)
  const float2* tab;      // [2J + 1][nc][nc] for dimension dd
  int32_t* trj_cart;      // (d, ns_pf, nt)
  int d, dd, nc, nrep, J;
  int64_t ns_pf, nt, Nd, nr;
  float h, lnorm;         // table spacing, ||lnG_dd||_1 (max column sum)
};

// One pass per dimension, in the reference's order.  A warp takes 32 samples: lane i first works
// out sample i's grid index, shift and polynomial degree (float64 as in the reference, once per
// sample and not once per lane: float64 is 1/60 of the float32 rate), then lane i owns coil i and
// the samples go through in fours.  Row i of L stays in lane i's registers; a product reads the
// four vectors from shared memory, two entries per 16-byte broadcast load.  NC: coils rounded up
// to a multiple of 8.  Table j sits at j n^2 in shared memory, column-major.
// 512k samples, 32 coils: 0.96 ms a dimension against 2.17 ms with a shuffle pair per vector
// entry and every lane repeating the float64 index arithmetic; bound by the shared-memory pipe
// (80%) and by instruction issue (69%).
constexpr int kGridWarps = 16, kGridFly = 4;

template <int NC>
__global__ void __launch_bounds__(32 * kGridWarps, 1) k_grog_grid(GridArgs a) {
  extern __shared__ __align__(16) float2 gsm[];
  __shared__ __align__(16) float2 wbuf[kGridWarps][kGridFly][NC];
  const int n = a.nc, nn = n * n, ntab = 2 * a.J + 1;
  for (int e = threadIdx.x; e < ntab * nn; e += blockDim.x) gsm[e] = a.tab[e];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool row = lane < n;
  float2 Lr[NC];  // row `lane` of L
#pragma unroll
  for (int j = 0; j < NC; ++j) Lr[j] = row && j < n ? a.lnG[a.dd + (int64_t)a.d * (lane + n * j)] : make_float2(0.f, 0.f);
  __syncthreads();
  const int64_t total = a.ns_pf * a.nt;
  const int64_t nwarps = (int64_t)gridDim.x * kGridWarps;
  auto madd = [](float2& acc, float2 m, float x, float y) {
    acc.x = fmaf(m.x, x, fmaf(-m.y, y, acc.x));
    acc.y = fmaf(m.x, y, fmaf(m.y, x, acc.y));
  };
  for (int64_t l0 = ((int64_t)blockIdx.x * kGridWarps + w) * 32; l0 < total; l0 += nwarps * 32) {
    // lane i: sample l0 + i
    float del = 0.f;
    int jt = 0, q = 0, m = 0;
    if (l0 + lane < total) {
      const int64_t li = l0 + lane;
      const float p = __fmul_rn(a.trj[a.dd + (int64_t)a.d * li], (float)a.Nd);  // Float32 * Int -> Float32
      const double t = __dadd_rn((double)p, 0.5);                                // + 1/2 -> Float64
      const double k = rint(t);                                                  // round: ties to even
      const double shift = __ddiv_rn(__dmul_rn(__dsub_rn(k, t), (double)a.nr), (double)a.Nd);
      a.trj_cart[a.dd + (int64_t)a.d * li] = (int32_t)((int64_t)k + a.Nd / 2);
      const float s = (float)shift;
      jt = max(-a.J, min(a.J, (int)rintf(s / a.h)));
      del = s - (float)jt * a.h;
      const float nrm = fabsf(del) * a.lnorm;
      while (nrm > ldexpf(1.f, q) && q < 20) ++q;  // normally 0: the remainder is within half a table step
      const float x = ldexpf(nrm, -q);
      del = ldexpf(del, -q);
      for (float tm = x; tm > kGridTol && m < 30;) {  // smallest degree with x^(m+1) / (m+1)! <= 2^-27
        ++m;
        tm *= x / (float)(m + 1);
      }
    }
    const int cnt = total - l0 < 32 ? (int)(total - l0) : 32;
    for (int s0 = 0; s0 < cnt; s0 += kGridFly) {
      float sq[kGridFly];
      int js[kGridFly], reps[kGridFly], most = 1, deg = 0;
#pragma unroll
      for (int u = 0; u < kGridFly; ++u) {
        sq[u] = __shfl_sync(0xffffffffu, del, s0 + u);
        js[u] = __shfl_sync(0xffffffffu, jt, s0 + u) + a.J;
        reps[u] = 1 << __shfl_sync(0xffffffffu, q, s0 + u);
        most = max(most, reps[u]);
        deg = max(deg, __shfl_sync(0xffffffffu, m, s0 + u));
      }
      for (int rep = 0; rep < a.nrep; ++rep) {
        float2* base = a.data + l0 + s0 + total * ((int64_t)a.nc * rep + lane);
        float2 v[kGridFly], z[kGridFly];
#pragma unroll
        for (int u = 0; u < kGridFly; ++u) v[u] = row && s0 + u < cnt ? base[u] : make_float2(0.f, 0.f);
        for (int rr = 0; rr < most; ++rr) {
#pragma unroll
          for (int u = 0; u < kGridFly; ++u) z[u] = v[u];
          for (int mm = deg; mm >= 1; --mm) {  // Horner: z = v + (sq/m) L (v + (sq/(m-1)) L (... ))
            if (lane < NC) {
#pragma unroll
              for (int u = 0; u < kGridFly; ++u) wbuf[w][u][lane] = z[u];
            }
            __syncwarp();
            float2 acc[kGridFly];
#pragma unroll
            for (int u = 0; u < kGridFly; ++u) acc[u] = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < NC; j += 2) {
#pragma unroll
              for (int u = 0; u < kGridFly; ++u) {
                const float4 x = *reinterpret_cast<const float4*>(&wbuf[w][u][j]);
                madd(acc[u], Lr[j], x.x, x.y);
                madd(acc[u], Lr[j + 1], x.z, x.w);
              }
            }
            __syncwarp();
            const float rm = 1.f / (float)mm;
#pragma unroll
            for (int u = 0; u < kGridFly; ++u) {
              const float c = sq[u] * rm;
              z[u] = make_float2(fmaf(c, acc[u].x, v[u].x), fmaf(c, acc[u].y, v[u].y));
            }
          }
#pragma unroll
          for (int u = 0; u < kGridFly; ++u)
            if (rr < reps[u]) v[u] = z[u];
        }
        // exp(s_j L) from the table
        if (lane < NC) {
#pragma unroll
          for (int u = 0; u < kGridFly; ++u) wbuf[w][u][lane] = v[u];
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kGridFly; ++u) {
          const float2* E = gsm + js[u] * nn + (row ? lane : 0);
          float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
          for (int j = 0; j < n; ++j) {
            const float2 x = wbuf[w][u][j];
            madd(acc, E[n * j], x.x, x.y);
          }
          if (row && s0 + u < cnt) base[u] = acc;
        }
        __syncwarp();
      }
    }
  }
}

template <int NC>
static int launch_grog_grid(const GridArgs& g, int64_t total, int sms, cudaStream_t st) {
  const size_t smem = sizeof(float2) * (size_t)(2 * g.J + 1) * g.nc * g.nc;
  MRSR_CHECK_CUDA(cudaFuncSetAttribute(k_grog_grid<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(total, 32 * kGridWarps), sms));
  k_grog_grid<NC><<<blocks, 32 * kGridWarps, smem, st>>>(g);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

static int grog_sms() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 1;
  }();
  return n;
}

}  // namespace mrsr

using namespace mrsr;

extern "C" int mrsr_grog_calib(int ndims, int64_t nr, int64_t ns_per_frame, int64_t nt, int ncoils, int nrep,
                               const float* data, const float* trj, float* lnG_out, mrsr_stream_t stream) {
  MRSR_CALL_SCOPE(reinterpret_cast<cudaStream_t>(stream));
  MRSR_REQUIRE(ndims == 2 || ndims == 3, MRSR_ERR_ARG, "ndims must be 2 or 3");
  MRSR_REQUIRE(data && trj && lnG_out, MRSR_ERR_ARG, "NULL argument to mrsr_grog_calib");
  MRSR_REQUIRE(nr >= 2 && ns_per_frame % nr == 0, MRSR_ERR_ARG, "samples per frame must be a multiple of Nr >= 2");
  MRSR_REQUIRE(ncoils >= 1 && ncoils <= kGrogMaxCoils, MRSR_ERR_UNSUPPORTED, "GROG supports 1..%d coils",
               kGrogMaxCoils);
  MRSR_REQUIRE(nrep >= 1, MRSR_ERR_ARG, "nrep must be >= 1");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int spf = (int)(ns_per_frame / nr);
  const int64_t nspk0 = (int64_t)spf * nt, nspk = nspk0 * nrep;
  const int nn = ncoils * ncoils;
  DevBuf AB, G, vth, nm, Pinv, err;
  MRSR_TRY(AB.alloc(sizeof(double2) * 2 * nn * nspk));
  MRSR_TRY(G.alloc(sizeof(float2) * nn * nspk));
  MRSR_TRY(vth.alloc(sizeof(double2) * nn * nspk));
  MRSR_TRY(nm.alloc(sizeof(double) * ndims * nspk0));
  MRSR_TRY(Pinv.alloc(sizeof(double) * 9));
  MRSR_TRY(err.alloc(sizeof(int)));
  MRSR_CHECK_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), st));
  const size_t smem_g = sizeof(float2) * (kGramRows + 1) * (ncoils + 1);
  GramArgs ga{reinterpret_cast<const float2*>(data), ns_per_frame, nt, ncoils, nrep, (int)nr, spf, AB.as<double2>()};
  k_grog_gram<<<(unsigned)nspk, 1024, smem_g, st>>>(ga);
  MRSR_LAUNCH_CHECK();
  k_grog_solve<<<(unsigned)nspk, kGjThreads, 0, st>>>(AB.as<double2>(), ncoils, G.as<float2>());
  MRSR_LAUNCH_CHECK();
  const LogArgs la{G.as<float2>(), ncoils, vth.as<double2>(), err.as<int>()};
  k_grog_log<<<(unsigned)nspk, kGjThreads, sizeof(float2) * 3 * nn, st>>>(la);
  MRSR_LAUNCH_CHECK();
  NmArgs na{trj, ndims, (int)nr, spf, ns_per_frame, nt, nspk0, nm.as<double>(), Pinv.as<double>(), nrep};
  k_grog_nm<<<1, 1024, 0, st>>>(na);
  MRSR_LAUNCH_CHECK();
  k_grog_lng<<<(unsigned)cdiv(nn, 32), 1024, 0, st>>>(nm.as<double>(), Pinv.as<double>(), vth.as<double2>(), ndims,
                                                     ncoils, nspk0, nrep, reinterpret_cast<float2*>(lnG_out));
  MRSR_LAUNCH_CHECK();
  int herr = 0;
  MRSR_CHECK_CUDA(cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  MRSR_CHECK_CUDA(cudaStreamSynchronize(st));
  MRSR_REQUIRE(herr == 0, MRSR_ERR_ARG, "matrix logarithm did not converge (a spoke operator has eigenvalues near 0)");
  return MRSR_OK;
}

extern "C" int mrsr_grog_gridding(int ndims, const int64_t* img_shape, int64_t nr, int64_t ns_per_frame, int64_t nt,
                                  int ncoils, int nrep, float* data, const float* trj, const float* lnG,
                                  int32_t* trj_cart_out, mrsr_stream_t stream) {
  MRSR_CALL_SCOPE(reinterpret_cast<cudaStream_t>(stream));
  MRSR_REQUIRE(ndims == 2 || ndims == 3, MRSR_ERR_ARG, "ndims must be 2 or 3");
  MRSR_REQUIRE(img_shape && data && trj && lnG && trj_cart_out, MRSR_ERR_ARG, "NULL argument to mrsr_grog_gridding");
  MRSR_REQUIRE(ncoils >= 1 && ncoils <= kGrogMaxCoils, MRSR_ERR_UNSUPPORTED, "GROG supports 1..%d coils",
               kGrogMaxCoils);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // ||lnG_d||_1 on the host (tiny)
  std::vector<float2> h((size_t)ndims * ncoils * ncoils);
  MRSR_CHECK_CUDA(cudaMemcpyAsync(h.data(), lnG, sizeof(float2) * h.size(), cudaMemcpyDeviceToHost, st));
  MRSR_CHECK_CUDA(cudaStreamSynchronize(st));
  const int nn = ncoils * ncoils;
  DevBuf tab;
  MRSR_TRY(tab.alloc(sizeof(float2) * (2 * kGridTabMax + 1) * nn * ndims));
  const int64_t total = ns_per_frame * nt;
  for (int dd = 0; dd < ndims; ++dd) {
    float lnorm = 0.f;
    for (int j = 0; j < ncoils; ++j) {
      float s = 0.f;
      for (int i = 0; i < ncoils; ++i) {
        const float2 v = h[dd + (size_t)ndims * (i + (size_t)ncoils * j)];
        s += std::sqrt(v.x * v.x + v.y * v.y);
      }
      lnorm = std::max(lnorm, s);
    }
    // |shift| <= Nr / (2 N_d); spacing h with h ||L||_1 <= 1 unless that needs more than 2 kGridTabMax + 1 tables
    const double smax = 0.5 * (double)nr / (double)img_shape[dd];
    int J = 0;
    float hs = 1.f;
    if (lnorm > 0.f) {
      J = (int)std::min<double>(kGridTabMax, std::ceil(smax * lnorm));
      hs = J > 0 ? (float)std::max(1.0 / lnorm, smax / J) : 1.f;
    }
    float2* tabd = tab.as<float2>() + (size_t)dd * (2 * kGridTabMax + 1) * nn;
    TabArgs ta{reinterpret_cast<const float2*>(lnG), ndims, dd, ncoils, J, hs, lnorm, tabd};
    k_grog_exp_table<<<(unsigned)(2 * J + 1), 1024, 0, st>>>(ta);
    MRSR_LAUNCH_CHECK();
    GridArgs g{};
    g.data = reinterpret_cast<float2*>(data);
    g.trj = trj;
    g.lnG = reinterpret_cast<const float2*>(lnG);
    g.tab = tabd;
    g.trj_cart = trj_cart_out;
    g.d = ndims;
    g.dd = dd;
    g.nc = ncoils;
    g.nrep = nrep;
    g.J = J;
    g.ns_pf = ns_per_frame;
    g.nt = nt;
    g.Nd = img_shape[dd];
    g.nr = nr;
    g.h = hs;
    g.lnorm = lnorm;
    switch ((ncoils + 7) / 8) {
      case 1: MRSR_TRY(launch_grog_grid<8>(g, total, grog_sms(), st)); break;
      case 2: MRSR_TRY(launch_grog_grid<16>(g, total, grog_sms(), st)); break;
      case 3: MRSR_TRY(launch_grog_grid<24>(g, total, grog_sms(), st)); break;
      default: MRSR_TRY(launch_grog_grid<32>(g, total, grog_sms(), st)); break;
    }
  }
  MRSR_CHECK_CUDA(cudaStreamSynchronize(st));
  return MRSR_OK;
}
