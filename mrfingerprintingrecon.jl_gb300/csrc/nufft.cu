// NUFFT kernels and the paths built on them:
//  * calculate_kmask_indcs / calculate_kernel_noncartesian -> NFFTNormalOp(img_shape, trj, U)
//    (src/NFFTNormalOp.jl:106-225, ext/MRISubspaceReconCUDAExt/NFFTNormalOp.jl:75-191)
//  * calculate_backprojection (src/BackProjection.jl:23-102, ext/.../BackProjection.jl:1-71)
//  * the forward model of the reference tests (test/reconstruct_radial.jl:62-74)
#include <algorithm>
#include <array>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "normalop.cuh"
#include "nufft.cuh"

namespace mrsr {

// ------------------------------------------------------------ samples ---

__device__ __forceinline__ int64_t sample_lin(const SampleSet& S, int64_t i) { return S.list ? S.list[i] - 1 : i; }

// frame of linear sample index li (32-bit division when the operands allow)
__device__ __forceinline__ int64_t frame_of(int64_t li, int64_t ns_pf) {
  return (li | ns_pf) < (1ll << 31) ? (int64_t)((unsigned)li / (unsigned)ns_pf) : li / ns_pf;
}

__global__ void k_mask_to_flags(const uint8_t* mask, int64_t n, uint8_t* flags) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    flags[i] = mask[i] ? 1 : 0;
}

int SampleList::init(int d, const float* trj, int64_t ns_pf, int64_t nt, const uint8_t* mask, cudaStream_t st) {
  set.trj = trj;
  set.d = d;
  set.ns_pf = ns_pf;
  set.nt = nt;
  const int64_t n = ns_pf * nt;
  if (!mask) {
    set.list = nullptr;
    set.n = n;
    return MRSR_OK;
  }
  DevBuf flags;
  MRSR_TRY(flags.alloc(std::max<int64_t>(n, 1)));
  k_mask_to_flags<<<(unsigned)std::min<int64_t>(cdiv(n, 256), 65535), 256, 0, st>>>(mask, n, flags.as<uint8_t>());
  MRSR_LAUNCH_CHECK();
  int64_t cnt = 0;
  MRSR_TRY(compact_nonzero(flags.as<uint8_t>(), n, list, &cnt, st));
  set.list = list.as<int64_t>();
  set.n = cnt;
  return MRSR_OK;
}

// ------------------------------------------------------- ES kernel ---

static double es_phi_host(double z) {
  if (std::fabs(z) >= 1.0) return 0.0;
  return std::exp((double)kEsBeta * (std::sqrt(1.0 - z * z) - 1.0));
}

// Gauss-Legendre nodes/weights on [-1, 1] (Newton iteration on P_n from the Chebyshev guess).
static void gauss_legendre(int n, std::vector<double>& x, std::vector<double>& w) {
  x.assign(n, 0.0);
  w.assign(n, 0.0);
  for (int i = 0; i < (n + 1) / 2; ++i) {
    double z = std::cos(M_PI * (i + 0.75) / (n + 0.5));
    double pp = 0.0;
    for (int it = 0; it < 100; ++it) {
      double p1 = 1.0, p2 = 0.0;
      for (int j = 1; j <= n; ++j) {
        const double p3 = p2;
        p2 = p1;
        p1 = ((2.0 * j - 1.0) * z * p2 - (j - 1.0) * p3) / j;
      }
      pp = n * (z * p1 - p2) / (z * z - 1.0);
      const double dz = p1 / pp;
      z -= dz;
      if (std::fabs(dz) < 1e-15) break;
    }
    x[i] = -z;
    x[n - 1 - i] = z;
    w[i] = w[n - 1 - i] = 2.0 / ((1.0 - z * z) * pp * pp);
  }
}

// psi_hat(j) = (w/2) int_{-1}^{1} phi(z) cos(pi j w z / M) dz.  The tables are cached per
// (device, M, jmin, count) for the life of the process (a few KB each, never freed): one
// costs count x 200 host cosines, and every kernel build, backprojection and forward model
// needs d of them.
int es_inv_psi_table(int64_t M, int64_t jmin, int64_t count, const float** out) {
  static std::mutex mu;
  static std::map<std::array<int64_t, 4>, float*> cache;
  static std::vector<double> gx, gw, gphi;
  int dev = 0;
  MRSR_CHECK_CUDA(cudaGetDevice(&dev));
  const std::array<int64_t, 4> key{dev, M, jmin, count};
  std::lock_guard<std::mutex> lock(mu);
  const auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return MRSR_OK;
  }
  if (gx.empty()) {
    gauss_legendre(200, gx, gw);
    gphi.resize(gx.size());
    for (size_t q = 0; q < gx.size(); ++q) gphi[q] = gw[q] * es_phi_host(gx[q]);
  }
  std::vector<float> h(count);
  const double hw = 0.5 * kEsWidth;
  for (int64_t i = 0; i < count; ++i) {
    const double j = (double)(jmin + i);
    double s = 0.0;
    for (size_t q = 0; q < gx.size(); ++q) s += gphi[q] * std::cos(M_PI * j * kEsWidth * gx[q] / (double)M);
    h[i] = (float)(1.0 / (hw * s));
  }
  float* d = nullptr;
  MRSR_CHECK_CUDA(cudaMalloc(&d, sizeof(float) * std::max<int64_t>(count, 1)));
  const cudaError_t e = cudaMemcpy(d, h.data(), sizeof(float) * count, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    MRSR_CHECK_CUDA(e);
  }
  cache[key] = d;
  *out = d;
  return MRSR_OK;
}

// --------------------------------------------------------- spreading ---

// one fixed-point term: a = value * 2^(e - 21), added as round(a * 2^21)
__device__ __forceinline__ void fx_add(long long* q, float a) {
  atomicAdd(reinterpret_cast<unsigned long long*>(q), (unsigned long long)fx_term(a));
}

__device__ __forceinline__ int wrap32(int l, int M) {
  l %= M;
  return l < 0 ? l + M : l;
}

// l mod M for -M < l < M (no division)
__device__ __forceinline__ int64_t wrap_near(int64_t l, int64_t M) { return l < 0 ? l + M : l; }

// Element e of an array of `planes` planes of (N0, N1, N2) cells -> plane and per-axis
// position.  Below 2^31 elements by magic-number divisions (FastDiv); this GPU divides 64-bit
// integers in software, tens of instructions each.
struct Decomp {
  int d = 0;
  bool fast = false;
  int64_t cells = 1, N[3] = {1, 1, 1};
  FastDiv fcells, fN[2];
  void init(int dims, const int64_t* n, int64_t planes) {
    d = dims;
    cells = 1;
    for (int i = 0; i < 3; ++i) {
      N[i] = i < dims ? n[i] : 1;
      cells *= N[i];
    }
    fast = cells * planes < (1ll << 31);
    if (fast) {
      fcells = FastDiv((uint32_t)cells);
      fN[0] = FastDiv((uint32_t)N[0]);
      fN[1] = FastDiv((uint32_t)N[1]);
    }
  }
  __device__ __forceinline__ int split(int64_t e, int64_t* pos) const {
    if (fast) {
      const uint32_t ue = (uint32_t)e, pl = fcells.div(ue);
      uint32_t r = ue - pl * fcells.d;
      const uint32_t q0 = fN[0].div(r);
      pos[0] = r - q0 * fN[0].d;
      r = q0;
      const uint32_t q1 = fN[1].div(r);
      pos[1] = r - q1 * fN[1].d;
      pos[2] = q1;
      return (int)pl;
    }
    const int pl = (int)(e / cells);
    int64_t r = e - (int64_t)pl * cells;
    pos[0] = r % N[0];
    r /= N[0];
    pos[1] = r % N[1];
    pos[2] = r / N[1];
    return pl;
  }
};

// Taps of one sample owned by a lane of its warp: lane = t1 + 8 * t2a (t1 < 8, t2a < 4), and
// its J = w^d / 32 taps are t2 = t2a + 4 (j & 1), t3 = j >> 1.  Weights (times `sc`) and
// grid cells (< 2^32, checked by the launchers) are formed once per sample, with 32-bit wraps.
template <int J>
__device__ __forceinline__ void lane_taps(const SampleSet& S, const int64_t* M, int64_t li, int lane, float sc,
                                          float* w, unsigned* cell) {
  constexpr int d = J == 2 ? 2 : 3;
  float kd[3] = {0.f, 0.f, 0.f};
  for (int dd = 0; dd < d; ++dd) kd[dd] = S.trj[dd + (int64_t)d * li];
  float wt;
  int64_t l0[3] = {0, 0, 0};
  es_lane_weight(kd, M, d, lane, &wt, l0);
  const int t1 = lane & 7, t2a = lane >> 3;
  const float wx = __shfl_sync(0xffffffffu, wt, t1) * sc;
  const unsigned x = wrap32((int)l0[0] + t1, (int)M[0]);
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int t2 = t2a + 4 * (j & 1), t3 = j >> 1;
    float wj = wx * __shfl_sync(0xffffffffu, wt, kEsWidth + t2);
    unsigned c = x + (unsigned)M[0] * (unsigned)wrap32((int)l0[1] + t2, (int)M[1]);
    if (d == 3) {
      wj *= __shfl_sync(0xffffffffu, wt, 2 * kEsWidth + t3);
      c += (unsigned)(M[0] * M[1]) * (unsigned)wrap32((int)l0[2] + t3, (int)M[2]);
    }
    w[j] = wj;
    cell[j] = c;
  }
}

// One warp per kept sample, for sets of 2^31 samples or more (the tile-sorted kernels below take the
// others).  A channel's value is formed once per sample; its terms go to the grid as 64-bit atomics.
template <int J>
__global__ void __launch_bounds__(256, 2) k_spread_lambda(SpreadLambdaArgs a, const int* order) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const float sc = a.fs->scale;
  const int64_t chs = (int64_t)a.nq * a.cells;
  for (int64_t i = warp; i < a.S.n; i += nwarps) {
    const int64_t n = order ? (int64_t)order[i] : i;
    const int64_t li = sample_lin(a.S, n);
    const int64_t t = frame_of(li, a.S.ns_pf);
    float w[J];
    unsigned cell[J];
    lane_taps<J>(a.S, a.M, li, lane, sc, w, cell);
    for (int ch = 0; ch < a.np; ++ch) {
      const int p = a.p0 + ch;
      int k2 = 0;
      while ((k2 + 1) * (k2 + 2) / 2 <= p) ++k2;
      const int k1 = p - k2 * (k2 + 1) / 2;
      float2 v;  // conj(U[t,k1]) * U[t,k2]
      if (a.u_complex) {
        const float2* u = reinterpret_cast<const float2*>(a.U);
        v = cmulc(u[t + a.S.nt * k2], u[t + a.S.nt * k1]);
      } else {
        const float* u = reinterpret_cast<const float*>(a.U);
        v = make_float2(u[t + a.S.nt * k2] * u[t + a.S.nt * k1], 0.f);
      }
      long long* q = a.q + (int64_t)ch * chs;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        fx_add(q + cell[j], v.x * w[j]);
        if (a.nq == 2) fx_add(q + a.cells + cell[j], v.y * w[j]);
      }
    }
  }
}

// The same for data channels: also without a basis (each sample then has one channel).
template <int J>
__global__ void __launch_bounds__(256, 2) k_spread_data(SpreadDataArgs a, const int* order) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int d = J == 2 ? 2 : 3;
  const float sc = a.fs->scale;
  const int64_t ns_tot = a.S.ns_pf * a.S.nt;
  for (int64_t i = warp; i < a.S.n; i += nwarps) {
    const int64_t n = order ? (int64_t)order[i] : i;
    const int64_t li = sample_lin(a.S, n);
    const int64_t t = frame_of(li, a.S.ns_pf);
    float dcf = 1.f;
    if (a.dcf_kind == MRSR_DCF_RADIAL_3D || a.dcf_kind == MRSR_DCF_RADIAL_2D) {
      float s2 = 0.f;
      for (int dd = 0; dd < d; ++dd) {
        const float k = a.S.trj[dd + (int64_t)d * li];
        s2 = __fadd_rn(s2, __fmul_rn(k, k));
      }
      dcf = a.dcf_kind == MRSR_DCF_RADIAL_3D ? s2 : sqrtf(s2);
    } else if (a.dcf_kind == MRSR_DCF_ARRAY) {
      dcf = a.dcf[n];
    }
    float w[J];
    unsigned cell[J];
    lane_taps<J>(a.S, a.M, li, lane, sc * dcf, w, cell);
    const int kb = a.U ? 0 : (int)t;  // U = I(nt): only coefficient t
    const int ke = a.U ? a.K : (int)t + 1;
    for (int c = 0; c < a.nc; ++c) {
      const float2 y = a.data[li + ns_tot * (a.c0 + c)];
      for (int k = kb; k < ke; ++k) {
        float2 v;
        if (!a.U) {
          v = y;
        } else if (a.u_complex) {
          v = cmulc(y, reinterpret_cast<const float2*>(a.U)[t + a.S.nt * k]);  // y * conj(U)
        } else {
          const float uu = reinterpret_cast<const float*>(a.U)[t + a.S.nt * k];
          v = make_float2(y.x * uu, y.y * uu);
        }
        long long* q = a.q + ((int64_t)c * a.K + k) * 2 * a.cells;
#pragma unroll
        for (int j = 0; j < J; ++j) {
          fx_add(q + cell[j], v.x * w[j]);
          fx_add(q + a.cells + cell[j], v.y * w[j]);
        }
      }
    }
  }
}

// 3D data spreading with a basis, sets of 2^31 samples or more, into a [cell][part] accumulator (the NP <= 32 parts of a
// coil batch consecutive: re and im of each coil and coefficient).  One warp per sample,
// lanes over the parts: a lane forms its part's value once, then adds its 512 terms, and
// the 32 atomics of one warp instruction land on one cell's consecutive parts (a few
// 32-byte sectors instead of one sector per lane).  Samples in 8^3-tile order.
__global__ void __launch_bounds__(256, 2) k_spread_data_cp(SpreadDataArgs a, const int* order, int NP) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const float sc = a.fs->scale;
  const int64_t ns_tot = a.S.ns_pf * a.S.nt;
  const bool live = lane < NP;
  const int ch = live ? lane >> 1 : 0, qpart = lane & 1;
  const int c = ch / a.K, k = ch - c * a.K;
  const int M0 = (int)a.M[0], M1 = (int)a.M[1], M2 = (int)a.M[2];
  for (int64_t i = warp; i < a.S.n; i += nwarps) {
    const int64_t n = order ? (int64_t)order[i] : i;
    const int64_t li = sample_lin(a.S, n);
    const int64_t t = frame_of(li, a.S.ns_pf);
    const float kd[3] = {a.S.trj[3 * li], a.S.trj[1 + 3 * li], a.S.trj[2 + 3 * li]};
    float dcf = 1.f;
    if (a.dcf_kind == MRSR_DCF_RADIAL_3D || a.dcf_kind == MRSR_DCF_RADIAL_2D) {
      float s2 = 0.f;
      for (int dd = 0; dd < 3; ++dd) s2 = __fadd_rn(s2, __fmul_rn(kd[dd], kd[dd]));
      dcf = a.dcf_kind == MRSR_DCF_RADIAL_3D ? s2 : sqrtf(s2);
    } else if (a.dcf_kind == MRSR_DCF_ARRAY) {
      dcf = a.dcf[n];
    }
    float wt;
    int64_t l0[3] = {0, 0, 0};
    es_lane_weight(kd, a.M, 3, lane, &wt, l0);
    float wx[kEsWidth], wy[kEsWidth], wz[kEsWidth];
#pragma unroll
    for (int j = 0; j < kEsWidth; ++j) {
      wx[j] = __shfl_sync(0xffffffffu, wt, j);
      wy[j] = __shfl_sync(0xffffffffu, wt, kEsWidth + j);
      wz[j] = __shfl_sync(0xffffffffu, wt, 2 * kEsWidth + j);
    }
    if (!live) continue;
    const float2 y = a.data[li + ns_tot * (a.c0 + c)];
    float2 vv;
    if (a.u_complex) {
      vv = cmulc(y, reinterpret_cast<const float2*>(a.U)[t + a.S.nt * k]);  // y * conj(U)
    } else {
      const float uu = reinterpret_cast<const float*>(a.U)[t + a.S.nt * k];
      vv = make_float2(y.x * uu, y.y * uu);
    }
    const float v = (qpart ? vv.y : vv.x) * sc * dcf;
    unsigned ix[kEsWidth];
    const int x0 = wrap32((int)l0[0], M0), y0 = wrap32((int)l0[1], M1), z0 = wrap32((int)l0[2], M2);
#pragma unroll
    for (int j = 0; j < kEsWidth; ++j) ix[j] = (unsigned)((x0 + j) % M0);
#pragma unroll 1
    for (int t3 = 0; t3 < kEsWidth; ++t3) {
      const unsigned zoff = (unsigned)((z0 + t3) % M2) * (unsigned)M1;
      const float v3 = v * wz[t3];
#pragma unroll
      for (int t2 = 0; t2 < kEsWidth; ++t2) {
        const unsigned rowc = (zoff + (unsigned)((y0 + t2) % M1)) * (unsigned)M0;
        const float w23 = v3 * wy[t2];
#pragma unroll
        for (int t1 = 0; t1 < kEsWidth; ++t1) {
          const unsigned cell = rowc + ix[t1];
          atomicAdd(reinterpret_cast<unsigned long long*>(a.q + (int64_t)cell * NP + lane),
                    (unsigned long long)fx_term(w23 * wx[t1]));
        }
      }
    }
  }
}

// [cell][NP] fixed-point accumulator -> [NP / 2][cell] float2 planes: 32 cells per block
// through a shared tile (coalesced on both sides)
__global__ void k_fixed_to_grid_cp(const long long* q, int NP, int64_t cells, const FixedScale* fs, float2* out) {
  __shared__ float tile[32][33];
  const float inv = fs->inv;
  const int64_t cell0 = (int64_t)blockIdx.x * 32;
  const int nc = cells - cell0 < 32 ? (int)(cells - cell0) : 32;
  for (int e = threadIdx.x; e < nc * NP; e += blockDim.x) {
    const int c = e / NP, p = e - c * NP;
    tile[c][p] = fx_to_float(q[(cell0 + c) * NP + p]) * inv;
  }
  __syncthreads();
  const int nch = NP / 2;
  for (int e = threadIdx.x; e < nch * 32; e += blockDim.x) {
    const int chn = e >> 5, c = e & 31;
    if (c < nc) out[(int64_t)chn * cells + cell0 + c] = make_float2(tile[c][2 * chn], tile[c][2 * chn + 1]);
  }
}

// taps of one sample that can land on the same cell (the w taps wrap around a grid shorter than w)
static double taps_per_cell(int d, const int64_t* M) {
  double t = 1.0;
  for (int i = 0; i < d; ++i) t *= (double)cdiv(kEsWidth, M[i]);
  return t;
}

static unsigned spread_blocks(int64_t n) { return (unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(n * 32, 256), 1), 152 * 64); }

// The w tap weights and wrapped tap indices of one sample along one dimension, in the
// arithmetic of es_lane_weight (every tap of one thread).
__device__ __forceinline__ void es_axis(float k, int M, float* w, int* idx) {
  const int hw = kEsWidth / 2;
  const float m = (float)M;
  const float uh = __fmul_rn(k, m);
  const float ul = fmaf(k, m, -uh);
  const float f = floorf(uh);
  const float r = __fadd_rn(__fsub_rn(uh, f), ul);
  const int c = r > 0.f ? 1 : 0;
  int l = ((int)f - hw + c) % M;
  if (l < 0) l += M;
#pragma unroll
  for (int t = 0; t < kEsWidth; ++t) {
    const float z = ((float)(c - hw + t) - r) * (1.f / hw);
    w[t] = (fabsf(z) < 1.f) ? expf(kEsBeta * (sqrtf(1.f - z * z) - 1.f)) : 0.f;
    idx[t] = l;
    l = l + 1 == M ? 0 : l + 1;
  }
}

// ------------------------------------------------------ tile sorts ---
//
// Samples counting-sorted by the tile (kTile3 or kSpTile cells a side) that holds
// their first tap; a work item is a chunk of samples of one tile.  The samples are counted in
// at most kSegs segments of consecutive ones, and a chunk takes whole segments of its tile, as
// many as fit; a segment of a tile with more samples than a chunk takes is put in order first
// (k_tile_order) and cut.  So which samples a chunk holds does not depend on the order in which
// the atomics land; their order inside it does.  (The interpolation, where a sample's result
// does not depend on its chunk, takes one segment and no order.)
constexpr int kSegs = 64;
// samples per segment, at least: with 8192, a small scan's crowded tiles are ordered by few blocks
// (32^2, 12800 samples, a backprojection 0.19 ms; 0.145 with 2048, 0.15 with 1024)
constexpr int kSegMin = 2048;
constexpr int kChunk = 1024;                // samples per work item of the interpolation kernels
constexpr int kTiledThreads = 512;

// Counts the samples of a warp per tile: one atomic per run of equal tiles (neighbours along a
// trajectory share a tile).  Returns the sample's place among its tile's, given the counter's
// value before.
__device__ __forceinline__ int tile_count(int* counter, int t, bool act) {
  const int lane = threadIdx.x & 31;
  const unsigned grp = __match_any_sync(0xffffffffu, act ? t : -1);
  const int lead = __ffs(grp) - 1;
  int base = 0;
  if (act && lane == lead) base = atomicAdd(&counter[t], __popc(grp));
  base = __shfl_sync(0xffffffffu, base, lead);
  return base + __popc(grp & ((1u << lane) - 1u));
}

// home tile of every kept sample: the tile holding its first tap (l0 of es_lane_weight)
__global__ void k_tile_home(SampleSet S, int M0, int M1, int M2, int tile, int64_t seg, int ntiles, int* tile_of,
                            int* counts) {
  const int hw = kEsWidth / 2;
  const int M[3] = {M0, M1, M2};
  const int ntx = (M0 + tile - 1) / tile, nty = (M1 + tile - 1) / tile;
  for (int64_t n0 = blockIdx.x * (int64_t)blockDim.x; n0 < S.n; n0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = n0 + threadIdx.x;
    const bool act = n < S.n;
    const int64_t li = act ? sample_lin(S, n) : 0;
    int l0[3] = {0, 0, 0};
    for (int dd = 0; dd < S.d; ++dd) {
      const float m = (float)M[dd];
      const float kd = act ? S.trj[dd + (int64_t)S.d * li] : 0.f;
      const float uh = __fmul_rn(kd, m);  // the arithmetic of es_lane_weight, operation for operation
      const float ul = fmaf(kd, m, -uh);
      const float f = floorf(uh);
      const float r = __fadd_rn(__fsub_rn(uh, f), ul);
      int l = ((int)f - hw + (r > 0.f ? 1 : 0)) % M[dd];
      l0[dd] = l < 0 ? l + M[dd] : l;
    }
    const int t = l0[0] / tile + ntx * (l0[1] / tile + nty * (l0[2] / tile));
    if (act) tile_of[n] = t;
    tile_count(counts + (n0 / seg) * ntiles, t, act);  // seg is a multiple of the block
  }
}

// Walks tile t's segments (counts[segment][tile]): each(segment, samples), and chunk(first,
// count) per work item, positions counted from `first`.
template <class Each, class Chunk>
__device__ __forceinline__ void tile_chunks(const int* counts, int nseg, int ntiles, int t, int first, int most, Each each,
                                            Chunk chunk) {
  int cur = 0;
  for (int g = 0; g < nseg; ++g) {
    const int c = counts[(int64_t)g * ntiles + t];
    each(g, c);
    if (c == 0) continue;
    if (cur != 0 && cur + c > most) {
      chunk(first, cur);
      first += cur;
      cur = 0;
    }
    cur += c;
    while (cur > most) {
      chunk(first, most);
      first += most;
      cur -= most;
    }
  }
  if (cur != 0) chunk(first, cur);
}

// per tile: samples and chunks over its segments
__global__ void k_tile_chunks(const int* counts, int nseg, int ntiles, int most, int* total, int* nch) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x) {
    int sum = 0, n = 0;
    tile_chunks(counts, nseg, ntiles, t, 0, most, [&](int, int c) { sum += c; }, [&](int, int) { ++n; });
    total[t] = sum;
    nch[t] = n;
  }
}

// one block: offsets of the tiles' sample lists and of their chunks, and the chunk count
__global__ void __launch_bounds__(1024) k_tile_scan(const int* total, const int* nch, int ntiles, int* offset, int* choff,
                                                    int* nitems) {
  __shared__ int s_n[32], s_c[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int bn = 0, bc = 0;  // totals of the tiles before this round's
  for (int t0 = 0; t0 < ntiles; t0 += 1024) {
    const int t = t0 + threadIdx.x;
    const int vn = t < ntiles ? total[t] : 0, vc = t < ntiles ? nch[t] : 0;
    int xn = vn, xc = vc;
    for (int o = 1; o < 32; o <<= 1) {
      const int yn = __shfl_up_sync(0xffffffffu, xn, o), yc = __shfl_up_sync(0xffffffffu, xc, o);
      if (lane >= o) {
        xn += yn;
        xc += yc;
      }
    }
    if (lane == 31) {
      s_n[warp] = xn;
      s_c[warp] = xc;
    }
    __syncthreads();
    int wn = 0, wc = 0, an = 0, ac = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) {
        wn += s_n[w];
        wc += s_c[w];
      }
      an += s_n[w];
      ac += s_c[w];
    }
    if (t < ntiles) {
      offset[t] = bn + wn + xn - vn;
      choff[t] = bc + wc + xc - vc;
    }
    bn += an;
    bc += ac;
    __syncthreads();
  }
  if (threadIdx.x == 0) *nitems = bc;
}

// per tile: its segments' places in the sorted order (written over counts), its work items
// (tile, first sorted position, count, -) and the segments with more samples than a chunk takes
__global__ void k_tile_items(int* counts, int nseg, int ntiles, int most, const int* offset, const int* choff, int4* items,
                             int2* big, int* nbig) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x) {
    int pos = offset[t], ch = choff[t];
    tile_chunks(counts, nseg, ntiles, t, pos, most,
                [&](int g, int c) {
                  counts[(int64_t)g * ntiles + t] = pos;
                  if (c > most) big[atomicAdd(nbig, 1)] = make_int2(pos, c);
                  pos += c;
                },
                [&](int first, int c) { items[ch++] = make_int4(t, first, c, 0); });
  }
}

// Puts the samples of the `big` segments in order, a block each; tmp: room for all samples.  A
// segment's samples are distinct numbers of [g seg, (g + 1) seg): a bitmap of a window of that range
// is set from the list and read back in order, one window after the other.  A list that is short
// beside the range (length^2 <= seg / 2) is ranked by comparing all pairs, which is cheaper there.
// Comparing pairs for every list took n^2 / 64 steps on scans that crowd into few tiles:
// backprojections of 5M samples in the middle tenth of a 64^2 k-space 144 -> 2.7 ms, of 20M
// samples on 64^2 82 -> 10.3.
constexpr int kOrderThreads = 1024;
constexpr int kOrderWords = 8192;  // 32-bit words of the bitmap
__global__ void __launch_bounds__(kOrderThreads) k_tile_order(const int2* big, const int* nbig, int64_t n, int64_t seg,
                                                              int* order, int* tmp) {
  __shared__ unsigned bits[kOrderWords];
  __shared__ int wsum[kOrderThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b = blockIdx.x; b < *nbig; b += gridDim.x) {
    const int2 s = big[b];
    for (int i = threadIdx.x; i < s.y; i += kOrderThreads) tmp[s.x + i] = order[s.x + i];
    __syncthreads();
    if ((int64_t)s.y * s.y <= seg / 2) {
      for (int i = threadIdx.x; i < s.y; i += kOrderThreads) {
        const int v = tmp[s.x + i];
        int r = 0;
        for (int j = 0; j < s.y; ++j) r += tmp[s.x + j] < v;
        order[s.x + r] = v;
      }
      continue;
    }
    const int64_t first = tmp[s.x] / seg * seg, end = min(first + seg, n);
    int* out = order + s.x;
    for (int64_t w0 = first; w0 < end; w0 += 32 * kOrderWords) {
      const int words = (int)min((int64_t)kOrderWords, (end - w0 + 31) / 32);
      for (int i = threadIdx.x; i < words; i += kOrderThreads) bits[i] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < s.y; i += kOrderThreads) {
        const int64_t d = tmp[s.x + i] - w0;
        if (d >= 0 && d < 32 * kOrderWords) atomicOr(&bits[d >> 5], 1u << (d & 31));
      }
      __syncthreads();
      for (int i0 = 0; i0 < words; i0 += kOrderThreads) {
        const int i = i0 + threadIdx.x;
        unsigned m = i < words ? bits[i] : 0u;
        const int c = __popc(m);
        int x = c;  // inclusive scan of the counts over the block
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        int all = 0, before = 0;
        for (int w = 0; w < kOrderThreads / 32; ++w) {
          if (w < warp) before += wsum[w];
          all += wsum[w];
        }
        int* o = out + before + x - c;
        for (; m; m &= m - 1) *o++ = (int)(w0 + 32 * i + __ffs(m) - 1);
        out += all;
        __syncthreads();
      }
    }
  }
}

__global__ void k_tile_scatter(int64_t n, int64_t seg, int ntiles, const int* tile_of, int* cursor, int* order) {
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = i0 + threadIdx.x;
    const bool act = i < n;
    const int place = tile_count(cursor + (i0 / seg) * ntiles, act ? tile_of[i] : 0, act);
    if (act) order[place] = (int)i;
  }
}

// Density compensation of kept sample n at linear index li (src/BackProjection.jl:169-181).
__device__ __forceinline__ float sample_dcf(const SampleSet& S, int64_t n, int64_t li, int kind, const float* dcf) {
  if (kind == MRSR_DCF_ARRAY) return dcf[n];
  if (kind != MRSR_DCF_RADIAL_3D && kind != MRSR_DCF_RADIAL_2D) return 1.f;
  float s2 = 0.f;
  for (int dd = 0; dd < S.d; ++dd) {
    const float k = S.trj[dd + (int64_t)S.d * li];
    s2 = __fadd_rn(s2, __fmul_rn(k, k));
  }
  return kind == MRSR_DCF_RADIAL_3D ? s2 : sqrtf(s2);
}

// Per-sample tap record of the tile-sorted kernels, in sorted order: the separable weights
// (the density compensation folded into wy), the wrapped first tap, the linear sample index
// and its frame.  Formed once per sample set, read by every part group (a broadcast load
// per sample instead of the weights, shuffles and index arithmetic per group).
struct __align__(16) TapRec {
  float wx[kEsWidth], wy[kEsWidth];
  int li, t, lx0, ly0;
};

__global__ void k_tile_prep(SampleSet S, int M0, int M1, const int* order, int dcf_kind, const float* dcf,
                            TapRec* rec) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < S.n; s += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = order[s];
    const int64_t li = sample_lin(S, n);
    const float k0 = S.trj[2 * li], k1 = S.trj[2 * li + 1];
    TapRec r;
    int ix[kEsWidth], iy[kEsWidth];
    es_axis(k0, M0, r.wx, ix);
    es_axis(k1, M1, r.wy, iy);
    const float w = sample_dcf(S, n, li, dcf_kind, dcf);
#pragma unroll
    for (int j = 0; j < kEsWidth; ++j) r.wy[j] *= w;
    r.li = (int)li;
    r.t = (int)frame_of(li, S.ns_pf);
    r.lx0 = ix[0];
    r.ly0 = iy[0];
    rec[s] = r;
  }
}

int TileSort::prep(const SampleSet& S, int dcf_kind, const float* dcf, cudaStream_t st) {
  if (S.d == 3) return prep3(S, dcf_kind, dcf, st);
  MRSR_REQUIRE(S.ns_pf * S.nt < (1ll << 31), MRSR_ERR_UNSUPPORTED, "tile records: < 2^31 samples per set");
  MRSR_TRY(rec.alloc(sizeof(TapRec) * std::max<int64_t>(S.n, 1)));
  const unsigned gb = (unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(S.n, 256), 1), 152 * 16);
  k_tile_prep<<<gb, 256, 0, st>>>(S, m0, m1, order.as<int>(), dcf_kind, dcf, rec.as<TapRec>());
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

int TileSort::build(const SampleSet& S, const int64_t* M, int tile_, int most, bool stable, cudaStream_t st) {
  MRSR_REQUIRE(S.n < (1ll << 31), MRSR_ERR_UNSUPPORTED, "tile sort: < 2^31 samples");
  const int64_t nt = cdiv(M[0], tile_) * cdiv(M[1], tile_) * (S.d == 3 ? cdiv(M[2], tile_) : 1);
  MRSR_REQUIRE(nt < (1ll << 31) && M[0] < (1ll << 24) && M[1] < (1ll << 24) && (S.d == 2 || M[2] < (1ll << 24)),
               MRSR_ERR_UNSUPPORTED, "tile sort: too many tiles");
  tile = tile_;
  ntiles = (int)nt;
  ntx = (int)cdiv(M[0], tile);
  nty = (int)cdiv(M[1], tile);
  m0 = (int)M[0];
  m1 = (int)M[1];
  m2 = S.d == 3 ? (int)M[2] : 1;
  const int64_t seg = cdiv(stable ? std::max<int64_t>(kSegMin, cdiv(S.n, kSegs)) : std::max<int64_t>(S.n, 1), 256) * 256;
  const int nseg = (int)std::max<int64_t>(1, cdiv(S.n, seg));
  // two neighbouring chunks of a tile hold more than `most` samples
  const int64_t maxitems = ntiles + 2 * cdiv(S.n, most);
  DevBuf big, nbig, tmp;
  MRSR_TRY(big.alloc(sizeof(int2) * (size_t)(S.n / most + 1)));
  MRSR_TRY(nbig.alloc(sizeof(int)));
  if (stable) MRSR_TRY(tmp.alloc(sizeof(int) * std::max<int64_t>(S.n, 1)));
  MRSR_CHECK_CUDA(cudaMemsetAsync(nbig.p, 0, sizeof(int), st));
  const size_t cbytes = sizeof(int) * (size_t)ntiles * nseg;
  MRSR_TRY(counts.alloc(cbytes));
  MRSR_TRY(total.alloc(sizeof(int) * ntiles));
  MRSR_TRY(nch.alloc(sizeof(int) * ntiles));
  MRSR_TRY(offset.alloc(sizeof(int) * ntiles));
  MRSR_TRY(choff.alloc(sizeof(int) * ntiles));
  MRSR_TRY(tile_of.alloc(sizeof(int) * std::max<int64_t>(S.n, 1)));
  MRSR_TRY(order.alloc(sizeof(int) * std::max<int64_t>(S.n, 1)));
  MRSR_TRY(items.alloc(sizeof(int4) * maxitems));
  MRSR_TRY(nitems.alloc(sizeof(int)));
  MRSR_TRY(next.alloc(sizeof(unsigned long long)));
  MRSR_CHECK_CUDA(cudaMemsetAsync(counts.p, 0, cbytes, st));
  const unsigned gb = (unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(S.n, 256), 1), 152 * 16);
  const unsigned gt = (unsigned)std::max<int64_t>(cdiv(ntiles, 64), 1);
  k_tile_home<<<gb, 256, 0, st>>>(S, m0, m1, m2, tile, seg, ntiles, tile_of.as<int>(), counts.as<int>());
  MRSR_LAUNCH_CHECK();
  k_tile_chunks<<<gt, 64, 0, st>>>(counts.as<int>(), nseg, ntiles, most, total.as<int>(), nch.as<int>());
  MRSR_LAUNCH_CHECK();
  k_tile_scan<<<1, 1024, 0, st>>>(total.as<int>(), nch.as<int>(), ntiles, offset.as<int>(), choff.as<int>(),
                                  nitems.as<int>());
  MRSR_LAUNCH_CHECK();
  k_tile_items<<<gt, 64, 0, st>>>(counts.as<int>(), nseg, ntiles, most, offset.as<int>(), choff.as<int>(), items.as<int4>(),
                                  big.as<int2>(), nbig.as<int>());
  MRSR_LAUNCH_CHECK();
  k_tile_scatter<<<gb, 256, 0, st>>>(S.n, seg, ntiles, tile_of.as<int>(), counts.as<int>(), order.as<int>());
  MRSR_LAUNCH_CHECK();
  if (stable) {
    k_tile_order<<<152, kOrderThreads, 0, st>>>(big.as<int2>(), nbig.as<int>(), S.n, seg, order.as<int>(), tmp.as<int>());
    MRSR_LAUNCH_CHECK();
  }
  return MRSR_OK;
}

constexpr int kTile3 = 8;                      // 3D interpolation windows
constexpr int kWin3 = kTile3 + kEsWidth - 1;   // 15
constexpr int kWin3Cells = kWin3 * kWin3 * kWin3;

// 3D tap record: weights along x, y, z (the density compensation folded into wz), the
// wrapped first tap, the linear sample index and its frame, in sorted order.
struct __align__(16) TapRec3 {
  float wx[kEsWidth], wy[kEsWidth], wz[kEsWidth];
  int li, t, lx0, ly0, lz0, pad0, pad1, pad2;
};
static_assert(sizeof(TapRec3) == 128, "TapRec3 is eight 16-byte loads");

__global__ void k_tile_prep3(SampleSet S, int M0, int M1, int M2, const int* order, int dcf_kind, const float* dcf,
                             TapRec3* rec) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < S.n; s += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = order[s];
    const int64_t li = sample_lin(S, n);
    const float k0 = S.trj[3 * li], k1 = S.trj[3 * li + 1], k2 = S.trj[3 * li + 2];
    TapRec3 r;
    int ix[kEsWidth], iy[kEsWidth], iz[kEsWidth];
    es_axis(k0, M0, r.wx, ix);
    es_axis(k1, M1, r.wy, iy);
    es_axis(k2, M2, r.wz, iz);
    const float w = sample_dcf(S, n, li, dcf_kind, dcf);
#pragma unroll
    for (int j = 0; j < kEsWidth; ++j) r.wz[j] *= w;
    r.li = (int)li;
    r.t = (int)frame_of(li, S.ns_pf);
    r.lx0 = ix[0];
    r.ly0 = iy[0];
    r.lz0 = iz[0];
    r.pad0 = r.pad1 = r.pad2 = 0;
    rec[s] = r;
  }
}

int TileSort::prep3(const SampleSet& S, int dcf_kind, const float* dcf, cudaStream_t st) {
  MRSR_REQUIRE(S.ns_pf * S.nt < (1ll << 31), MRSR_ERR_UNSUPPORTED, "tile records: < 2^31 samples per set");
  MRSR_TRY(rec.alloc(sizeof(TapRec3) * std::max<int64_t>(S.n, 1)));
  const unsigned gb = (unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(S.n, 256), 1), 152 * 16);
  k_tile_prep3<<<gb, 256, 0, st>>>(S, m0, m1, m2, order.as<int>(), dcf_kind, dcf, rec.as<TapRec3>());
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

}  // namespace mrsr

#include "spread_rows.cuh"
#include "spread_windows.cuh"

namespace mrsr {

int spread_lambda(const SpreadLambdaArgs& a, const TileSort* ts, cudaStream_t st) {
  if (a.S.n == 0) return MRSR_OK;
  if (ts && ts->rec.p) {
    const LamParts parts{a.U, a.umax, a.u_complex, a.nq, a.p0, a.S.nt};
    if (ts->tile != kSpTile) return spread_windows(a.M, a.cells, a.np * a.nq, a.q, a.fs, *ts, parts, st);
    return spread_rows(a.S.d, a.M, a.cells, a.np * a.nq, a.q, a.fs, a.bad, *ts, parts, st);
  }
  MRSR_REQUIRE(a.cells < (1ll << 32), MRSR_ERR_UNSUPPORTED, "spreading grid of 2^32 cells or more");
  const int* order = ts ? ts->order.as<int>() : nullptr;
  if (a.S.d == 2)
    k_spread_lambda<2><<<spread_blocks(a.S.n), 256, 0, st>>>(a, order);
  else
    k_spread_lambda<16><<<spread_blocks(a.S.n), 256, 0, st>>>(a, order);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

int spread_data(const SpreadDataArgs& a, const TileSort* ts, cudaStream_t st) {
  if (a.S.n == 0) return MRSR_OK;
  if (ts && a.U && ts->rec.p && ts->tile != kSpTile) {
    const DataParts parts{a.data, a.U, nullptr, nullptr, a.u_complex, a.K, a.c0, a.nc, a.S.nt, a.S.ns_pf * a.S.nt};
    return spread_windows(a.M, a.cells, 2 * a.nc * a.K, a.q, a.fs, *ts, parts, st);
  }
  if (ts && a.U && ts->rec.p) {
    const unsigned gb = (unsigned)std::min<int64_t>(cdiv(a.S.n, 256), 152 * 16);
    MRSR_CHECK_CUDA(cudaMemsetAsync(a.tmax, 0, sizeof(float) * (size_t)ts->ntiles * a.nc, st));
    k_tile_absmax<<<gb, 256, 0, st>>>(a.S, ts->tile_of.as<int>(), a.data, a.c0, a.nc, a.dcf_kind, a.dcf,
                                      reinterpret_cast<unsigned*>(a.tmax));
    MRSR_LAUNCH_CHECK();
    const DataParts parts{a.data, a.U, a.umax, a.tmax, a.u_complex, a.K, a.c0, a.nc, a.S.nt, a.S.ns_pf * a.S.nt};
    return spread_rows(a.S.d, a.M, a.cells, 2 * a.nc * a.K, a.q, a.fs, a.bad, *ts, parts, st);
  }
  MRSR_REQUIRE(a.cells < (1ll << 32), MRSR_ERR_UNSUPPORTED, "spreading grid of 2^32 cells or more");
  const int* order = ts && a.S.d == 3 ? ts->order.as<int>() : nullptr;
  if (a.S.d == 3 && a.U && 2 * a.nc * a.K <= 32) {  // [cell][part] accumulator (the 3D backprojection)
    k_spread_data_cp<<<spread_blocks(a.S.n), 256, 0, st>>>(a, order, 2 * a.nc * a.K);
    MRSR_LAUNCH_CHECK();
    return MRSR_OK;
  }
  if (a.S.d == 2)
    k_spread_data<2><<<spread_blocks(a.S.n), 256, 0, st>>>(a, order);
  else
    k_spread_data<16><<<spread_blocks(a.S.n), 256, 0, st>>>(a, order);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

// ------------------------------------------------------- fixed point ---

// amax[slot] = max |f[i]| as float bits (non-negative floats order like their bit patterns), over the
// finite entries with `finite`
__global__ void k_absmax(const float* f, int64_t n, bool finite, unsigned* amax) {
  float m = 0.f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = fabsf(f[i]);
    if (!finite || finite_value(v)) m = fmaxf(m, v);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(amax, __float_as_uint(m));
}

// e = min(62 - ceil(log2(nterms * bound)), 40 - ceil(log2(bound))), bound = mult * prod
// amax; e clamped so that 2^(e - 21) and 2^-e are normal floats
__global__ void k_fixed_scale(const unsigned* amax, int nf, double mult, double nterms, FixedScale* out) {
  double bound = mult;
  for (int i = 0; i < nf; ++i) bound *= (double)__uint_as_float(amax[i]);
  int e = 0;
  if (bound > 0.0) e = min(62 - (int)ceil(log2(nterms * bound)), kFxTermBits - (int)ceil(log2(bound)));
  e = max(-100, min(120, e));
  out->scale = ldexpf(1.f, e - kFxLoBits);
  out->inv = ldexpf(1.f, -e);
}

int fixed_scale(const float* const* f, const int64_t* n, int nf, double mult, double nterms, bool finite, FixedScale* out,
                cudaStream_t st) {
  MRSR_REQUIRE(nf >= 0 && nf <= 3, MRSR_ERR_ARG, "fixed_scale: at most 3 factors");
  DevBuf am;
  MRSR_TRY(am.alloc(4 * sizeof(unsigned)));
  MRSR_CHECK_CUDA(cudaMemsetAsync(am.p, 0, 4 * sizeof(unsigned), st));
  for (int i = 0; i < nf; ++i) {
    const unsigned g = (unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(n[i], 1024), 1), 152 * 8);
    k_absmax<<<g, 256, 0, st>>>(f[i], n[i], finite, am.as<unsigned>() + i);
    MRSR_LAUNCH_CHECK();
  }
  k_fixed_scale<<<1, 1, 0, st>>>(am.as<unsigned>(), nf, mult, nterms, out);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

// fixed-point planes -> float2 grids
__global__ void k_fixed_to_grid(const long long* q, int nq, int64_t cells, int64_t total, const FixedScale* fs,
                                float2* out) {
  const float inv = fs->inv;
  auto cvt = [inv](long long v) { return fx_to_float(v) * inv; };
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ch = e / cells, cell = e - ch * cells;
    const long long* qc = q + ch * nq * cells + cell;
    out[e] = make_float2(cvt(qc[0]), nq == 2 ? cvt(qc[cells]) : 0.f);
  }
}

int fixed_to_grid(const long long* q, int nq, int64_t cells, int64_t nch, const FixedScale* fs, float2* out,
                  cudaStream_t st) {
  const int64_t total = cells * nch;
  const unsigned g = (unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(total, 256), 1), 152 * 32);
  k_fixed_to_grid<<<g, 256, 0, st>>>(q, nq, cells, total, fs, out);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

// ----------------------------------------------------------- kmask ---

// Gaussian-footprint mask: cells i0-3 .. i0+4 (mod G) per dimension around
// i0 = floor(fl32(-k * G)) for every kept sample (src/NFFTNormalOp.jl:106-118).  The union
// of the boxes is the seed set {i0} dilated by the box: cell j is marked iff some seed lies
// in j-4 .. j+3 along every dimension.  One byte store per sample marks the seeds, then one
// pass per dimension ORs each cell's 8 neighbours along it (separable, exact for boolean
// masks), instead of 8^d scattered byte stores per sample.
__global__ void k_kmask_seed(SampleSet S, int64_t G0, int64_t G1, int64_t G2, uint8_t* seeds) {
  const int d = S.d;
  const int G[3] = {(int)G0, (int)G1, (int)G2};
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < S.n; n += (int64_t)gridDim.x * blockDim.x) {
    const int64_t li = sample_lin(S, n);
    int64_t cell = 0, stride = 1;
    for (int dd = 0; dd < d; ++dd) {
      const float p = __fmul_rn(-S.trj[dd + (int64_t)d * li], (float)G[dd]);
      int l = (int)floorf(p) % G[dd];
      if (l < 0) l += G[dd];
      cell += (int64_t)l * stride;
      stride *= G[dd];
    }
    seeds[cell] = 1;
  }
}

// out[j] = OR of in[j + s], s = -4 .. 3 (mod G) along dimension `axis`
__global__ void k_kmask_dilate(const uint8_t* in, int64_t G0, int64_t G1, int64_t G2, int axis, uint8_t* out) {
  const int64_t total = G0 * G1 * G2;
  const int64_t stride = axis == 0 ? 1 : (axis == 1 ? G0 : G0 * G1);
  const int64_t Ga = axis == 0 ? G0 : (axis == 1 ? G1 : G2);
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < total; c += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = (c / stride) % Ga;
    const int64_t base = c - j * stride;
    uint8_t v = 0;
#pragma unroll
    for (int s = -4; s <= 3; ++s) {
      int64_t k = (j + s) % Ga;
      if (k < 0) k += Ga;
      v |= in[base + k * stride];
    }
    out[c] = v ? 1 : 0;
  }
}

// ----------------------------------------------------- Λ precompute ---

struct FoldArgs {
  int d;
  int64_t G[3], M[3];
  int64_t gcells, mcells;
  int P;
  int real_u;
  Decomp dc;              // element -> (p, cell position) over (G0, G1, G2) x P
  const float2* g;        // [P][mcells] after the inverse DFT
  const float* ipsi[3];   // 1/psi_hat(j) for j = -G/2 .. G/2
  float2* c;              // [P][gcells]
};

// c~[p] for the Toeplitz kernel: complex basis uses j in [-G/2, G/2) (FFT
// order, src/NFFTNormalOp.jl:142-158); a real basis follows the real-input
// transform + brfft of :197-214: along dim 1 only j1 in [0, G1/2] is used,
// interior terms doubled, and Λ = Re(FFT(c~)).
__global__ void k_lambda_fold(FoldArgs a) {
  const int64_t total = a.gcells * a.P;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t pd[3] = {0, 0, 0};
    const int p = a.dc.split(e, pd);
    float scale = 1.f;
    int64_t l = 0, mul = 1;
    bool zero = false;
    for (int dd = 0; dd < a.d; ++dd) {
      const int64_t Gd = a.G[dd], half = Gd / 2;
      int64_t j;
      if (a.real_u && dd == 0) {
        if (pd[0] > half) {
          zero = true;
          j = 0;
        } else {
          j = pd[0];
          if (j != 0 && j != half) scale *= 2.f;
        }
      } else {
        j = pd[dd] < half ? pd[dd] : pd[dd] - Gd;
      }
      scale *= a.ipsi[dd][j + half];
      l += wrap_near(j, a.M[dd]) * mul;
      mul *= a.M[dd];
    }
    float2 v = zero ? make_float2(0.f, 0.f) : a.g[(int64_t)p * a.mcells + l];
    a.c[e] = make_float2(v.x * scale, v.y * scale);
  }
}

__global__ void k_lambda_gather(const float2* lam, int64_t gcells, int P, const int64_t* kmask, int64_t nk, int real_u,
                                void* packed) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nk; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t cell = kmask[i] - 1;
    for (int p = 0; p < P; ++p) {
      const float2 v = lam[(int64_t)p * gcells + cell];
      if (real_u)
        reinterpret_cast<float*>(packed)[p + (int64_t)P * i] = v.x;
      else
        reinterpret_cast<float2*>(packed)[p + (int64_t)P * i] = v;
    }
  }
}

static unsigned grid1d(int64_t n) { return (unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(n, 256), 1), 65535); }

// kmask + packed Λ (P, nk) for a trajectory and basis
static int compute_lambda(int d, const int64_t* G, const SampleSet& S, const void* U, int u_complex, int K, DevBuf& kmask,
                          int64_t* nk_out, DevBuf& packed, cudaStream_t st) {
  const int64_t gcells = G[0] * G[1] * (d == 3 ? G[2] : 1);
  MRSR_REQUIRE(S.n > 0, MRSR_ERR_ARG, "AssertionError: Mask removes all samples, cannot compute kernel.");
  // kmask
  {
    DevBuf flags, tmp;
    MRSR_TRY(flags.alloc(gcells));
    MRSR_TRY(tmp.alloc(gcells));
    MRSR_CHECK_CUDA(cudaMemsetAsync(flags.p, 0, gcells, st));
    const int64_t G2 = d == 3 ? G[2] : 1;
    k_kmask_seed<<<(unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(S.n, 256), 1), 152 * 64), 256, 0, st>>>(
        S, G[0], G[1], G2, flags.as<uint8_t>());
    MRSR_LAUNCH_CHECK();
    uint8_t* src = flags.as<uint8_t>();
    uint8_t* dst = tmp.as<uint8_t>();
    for (int ax = 0; ax < d; ++ax) {
      k_kmask_dilate<<<grid1d(gcells), 256, 0, st>>>(src, G[0], G[1], G2, ax, dst);
      MRSR_LAUNCH_CHECK();
      std::swap(src, dst);
    }
    MRSR_TRY(compact_nonzero(src, gcells, kmask, nk_out, st));
  }
  const int P = K * (K + 1) / 2;
  int64_t M[3] = {1, 1, 1};
  for (int i = 0; i < d; ++i) M[i] = 2 * G[i];
  const int64_t mcells = M[0] * M[1] * M[2];
  FftNd fM, fG;
  MRSR_TRY(fM.init(d, M));
  MRSR_TRY(fG.init(d, G));
  const float* ipsi[3] = {nullptr, nullptr, nullptr};
  for (int i = 0; i < d; ++i) MRSR_TRY(es_inv_psi_table(M[i], -G[i] / 2, G[i] + 1, &ipsi[i]));
  // channel batches of ~2 GB of upsampled float2 grid; in 3D a batch fills the four parts of a
  // window group
  const int nq = u_complex ? 2 : 1;  // a real basis spreads real values
  const int64_t max_bytes = 2ll << 30;
  int pb = (int)std::max<int64_t>(1, std::min<int64_t>(P, max_bytes / (mcells * (int64_t)sizeof(float2))));
  const bool tiled = S.n < (1ll << 31) && S.ns_pf * S.nt < (1ll << 31);
  const bool rows = tiled && (d == 2 || rows_pay(nq * pb, nq * P, S.n, mcells));
  if (d == 3 && !rows) pb = std::max(pb, std::min(P, kP3 / nq));
  DevBuf grid, qgrid, cgrid, fsb, umax;
  const size_t qbytes = rows ? spread_rows_bytes(nq * pb, mcells) : sizeof(long long) * nq * mcells * pb;
  MRSR_TRY(grid.alloc(sizeof(float2) * mcells * pb));
  MRSR_TRY(qgrid.alloc(qbytes));
  MRSR_TRY(cgrid.alloc(sizeof(float2) * gcells * P));
  // The call synchronises after these are freed.  Where they are more than the pool keeps, freed on
  // the call's stream they went back to the driver there, and the next call mapped them anew (192^3,
  // K = 3, calls in a row 129 ms against 88; 128^3, K = 5, 72 against 67).
  grid.side = qgrid.side = cgrid.side = grid.bytes + qgrid.bytes + cgrid.bytes > kPoolKeep;
  // fixed-point scale: |term| <= (2 if complex) max|U|^2 (the kernel taps are <= 1), and a cell
  // of the upsampled grid gets at most ceil(w / M) taps per sample and dimension
  MRSR_TRY(fsb.alloc(sizeof(FixedScale)));
  {
    const float* uf = reinterpret_cast<const float*>(U);
    const int64_t nu = S.nt * (int64_t)K * (u_complex ? 2 : 1);
    const float* f[2] = {uf, uf};
    const int64_t n[2] = {nu, nu};
    MRSR_TRY(fixed_scale(f, n, 2, u_complex ? 2.0 : 1.0, (double)S.n * taps_per_cell(d, M), rows, fsb.as<FixedScale>(), st));
  }
  TileSort ts;
  const bool ordered = S.n < (1ll << 31) && d == 3;
  if (tiled || ordered) MRSR_TRY(ts.build(S, M, rows ? kSpTile : kTile3, rows ? spread_chunk(d, S.n) : kChunk, rows, st));
  if (tiled) MRSR_TRY(ts.prep(S, MRSR_DCF_NONE, nullptr, st));
  if (rows) {
    MRSR_TRY(basis_max(S, U, u_complex, K, nq * P, umax, st));
  }
  const TileSort* tsp = tiled || ordered ? &ts : nullptr;
  MRSR_TRY(packed.alloc((u_complex ? 8 : 4) * (size_t)P * std::max<int64_t>(*nk_out, 1)));
  // channels in batches of pb: spread, inverse DFT on the upsampled grid, deconvolve and fold onto the 2x grid
  for (int p0 = 0; p0 < P; p0 += pb) {
    const int np = std::min(pb, P - p0);
    int* bad = rows ? umax.as<int>() + K + nq * p0 : nullptr;
    MRSR_CHECK_CUDA(cudaMemsetAsync(qgrid.p, 0, rows ? spread_rows_bytes(nq * np, mcells) : sizeof(long long) * nq * mcells * np, st));
    SpreadLambdaArgs sa{S, {M[0], M[1], M[2]}, mcells, U, u_complex, K, P, p0, np, nq, qgrid.as<long long>(),
                        fsb.as<FixedScale>(), umax.as<float>(), bad};
    MRSR_TRY(spread_lambda(sa, tsp, st));
    if (rows)
      MRSR_TRY(parts_to_grid(qgrid.as<long long>(), nq, mcells, nq * np, fsb.as<FixedScale>(), bad, grid.as<float2>(),
                             st));
    else
      MRSR_TRY(fixed_to_grid(qgrid.as<long long>(), nq, mcells, np, fsb.as<FixedScale>(), grid.as<float2>(), st));
    MRSR_TRY(fM.run(grid.as<float2>(), np, +1, 1.0f, st));
    FoldArgs fa;
    fa.d = d;
    for (int i = 0; i < 3; ++i) {
      fa.G[i] = i < d ? G[i] : 1;
      fa.M[i] = M[i];
      fa.ipsi[i] = ipsi[i];
    }
    fa.gcells = gcells;
    fa.mcells = mcells;
    fa.P = np;
    fa.dc.init(d, G, np);
    fa.real_u = u_complex ? 0 : 1;
    fa.g = grid.as<float2>();
    fa.c = cgrid.as<float2>() + (int64_t)p0 * gcells;
    k_lambda_fold<<<grid1d(gcells * np), 256, 0, st>>>(fa);
    MRSR_LAUNCH_CHECK();
  }
  MRSR_TRY(fG.run(cgrid.as<float2>(), P, -1, 1.0f, st));
  k_lambda_gather<<<grid1d(*nk_out), 256, 0, st>>>(cgrid.as<float2>(), gcells, P, kmask.as<int64_t>(), *nk_out,
                                                   u_complex ? 0 : 1, packed.p);
  MRSR_LAUNCH_CHECK();
  MRSR_CHECK_CUDA(cudaStreamSynchronize(st));
  return MRSR_OK;
}


// ------------------------------------------------ backprojection fold ---

struct BpFoldArgs {
  int d;
  int64_t N[3], M[3], nimg, mcells;
  int K, c0, nc, ncoils;
  Decomp dc;              // element -> (k, image position) over img x K
  const float2* g;        // [(c - c0) K + k][mcells]
  const float* ipsi[3];   // 1/psi_hat(j), j = -N/2 ...
  const float2* cmaps;    // (img..., ncoils) or null -> per-coil output
  float2* out;
};

// out[r, k] += sum_c conj(S_c(r)) x_ck(r)  (src/BackProjection.jl:96), or
// out[r, k, c] = x_ck(r) without coil maps (:54); x_ck(r) = g[(r - N/2) mod M] / psi_hat.
__global__ void k_bp_fold(BpFoldArgs a) {
  const int64_t total = a.nimg * a.K;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t pos[3];
    const int k = a.dc.split(e, pos);
    const int64_t r = e - (int64_t)k * a.nimg;
    int64_t l = 0, mul = 1;
    float sc = 1.f;
    for (int dd = 0; dd < a.d; ++dd) {
      const int64_t rd = pos[dd];
      const int64_t j = rd - a.N[dd] / 2;
      sc *= a.ipsi[dd][rd];
      l += wrap_near(j, a.M[dd]) * mul;
      mul *= a.M[dd];
    }
    if (a.cmaps) {
      float2 acc = make_float2(0.f, 0.f);
      for (int c = 0; c < a.nc; ++c) {
        const float2 v = a.g[((int64_t)c * a.K + k) * a.mcells + l];
        acc = cadd(acc, cmulc(v, a.cmaps[r + a.nimg * (a.c0 + c)]));
      }
      a.out[e] = cadd(a.out[e], cscale(acc, sc));
    } else {
      for (int c = 0; c < a.nc; ++c) {
        const float2 v = a.g[((int64_t)c * a.K + k) * a.mcells + l];
        a.out[r + a.nimg * (k + (int64_t)a.K * (a.c0 + c))] = cscale(v, sc);
      }
    }
  }
}

// ------------------------------------------------------ forward model ---

struct FwdPlaceArgs {
  int d;
  int64_t N[3], M[3], nimg, mcells;
  int K, c;              // coil c + blockIdx.y
  Decomp dc;             // element -> (k, image position) over img x K
  const float2* x;       // (img..., K)
  const float2* cmaps;   // (img..., ncoils) or null
  const float* ipsi[3];
  float2* g;             // [coil][K][mcells], zeroed
};

__global__ void k_fwd_place(FwdPlaceArgs a) {
  const int64_t total = a.nimg * a.K;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t pos[3];
    const int k = a.dc.split(e, pos);
    const int64_t r = e - (int64_t)k * a.nimg;
    int64_t l = 0, mul = 1;
    float sc = 1.f;
    for (int dd = 0; dd < a.d; ++dd) {
      const int64_t rd = pos[dd];
      sc *= a.ipsi[dd][rd];
      l += wrap_near(rd - a.N[dd] / 2, a.M[dd]) * mul;
      mul *= a.M[dd];
    }
    float2 v = a.x[e];
    if (a.cmaps) v = cmul(a.cmaps[r + a.nimg * (a.c + (int)blockIdx.y)], v);
    a.g[((int64_t)blockIdx.y * a.K + k) * a.mcells + l] = cscale(v, sc);
  }
}

struct InterpArgs {
  SampleSet S;
  int64_t M[3], mcells;
  int K, c, u_complex;
  const void* U;
  const float2* g;       // [mcells][K] after the forward DFT: a cell's K planes side by side
  float2* data;          // (ns_pf, nt, ncoils)
};

// [K][mcells] -> [mcells][K]: after the forward DFT the interpolation reads all K planes at
// each tap, so the K values of a cell are put next to each other (one or two 32-byte sectors
// per tap instead of K).
__global__ void k_interleave(const float2* __restrict__ g, float2* __restrict__ gi, int K, int64_t mcells) {
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < mcells; l += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < K) gi[l * K + k] = g[(int64_t)k * mcells + l];
  }
}

// 2D: one thread per kept sample, the w^2 taps of the K gridded planes summed in the thread
// (no cross-lane reduction); the 32 samples of a warp are consecutive along the trajectory,
// so their taps share cache lines.
__global__ void __launch_bounds__(256) k_interp(InterpArgs a) {
  const int d = a.S.d;
  const int64_t ns_tot = a.S.ns_pf * a.S.nt;
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < a.S.n; n += (int64_t)gridDim.x * blockDim.x) {
    const int64_t li = sample_lin(a.S, n);
    const int64_t t = frame_of(li, a.S.ns_pf);
    float wx[kEsWidth], wy[kEsWidth], wz[kEsWidth];
    int ix[kEsWidth], iy[kEsWidth], iz[kEsWidth];
    es_axis(a.S.trj[(int64_t)d * li], (int)a.M[0], wx, ix);
    es_axis(a.S.trj[1 + (int64_t)d * li], (int)a.M[1], wy, iy);
    if (d == 3) {
      es_axis(a.S.trj[2 + (int64_t)d * li], (int)a.M[2], wz, iz);
    } else {
#pragma unroll
      for (int j = 0; j < kEsWidth; ++j) {
        wz[j] = j == 0 ? 1.f : 0.f;
        iz[j] = 0;
      }
    }
    float2 z[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) z[k] = make_float2(0.f, 0.f);
    const int nz = d == 3 ? kEsWidth : 1;
#pragma unroll 1
    for (int t3 = 0; t3 < nz; ++t3) {
      const int64_t base3 = (int64_t)iz[t3] * a.M[0] * a.M[1];
      const float w3 = wz[t3];
#pragma unroll
      for (int t2 = 0; t2 < kEsWidth; ++t2) {
        const float w23 = wy[t2] * w3;
        const int64_t row = base3 + (int64_t)iy[t2] * a.M[0];
#pragma unroll
        for (int t1 = 0; t1 < kEsWidth; ++t1) {
          const float w = w23 * wx[t1];
          const float2* cell = a.g + (row + ix[t1]) * a.K;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < a.K) {
              const float2 gv = __ldg(cell + k);
              z[k].x = fmaf(w, gv.x, z[k].x);
              z[k].y = fmaf(w, gv.y, z[k].y);
            }
        }
      }
    }
    float2 y = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < a.K) {
        if (a.u_complex)
          y = cadd(y, cmul(reinterpret_cast<const float2*>(a.U)[t + a.S.nt * k], z[k]));
        else
          y = cadd(y, cscale(z[k], reinterpret_cast<const float*>(a.U)[t + a.S.nt * k]));
      }
    }
    a.data[li + ns_tot * a.c] = y;
  }
}

// acc += (w, w) * g on both components at once
__device__ __forceinline__ float2 fma2(float2 w, float2 g, float2 acc) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(*reinterpret_cast<const unsigned long long*>(&w)), "l"(*reinterpret_cast<const unsigned long long*>(&g)),
        "l"(*reinterpret_cast<const unsigned long long*>(&acc)));
  return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(*reinterpret_cast<const unsigned long long*>(&a)), "l"(*reinterpret_cast<const unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}

// 2D on the tile sort (tiles of 16 x 16 cells): a work unit, up to 1024 samples of one tile and
// a group of at most 16 planes (whole coils, K planes each), loads the group's 23 x 23-cell
// window into shared memory ([cell][17], so that neither the loads along the cells nor the reads
// along the planes meet a bank twice), and each half of a warp takes a sample, a lane per plane:
// 64 taps of one 8-byte load and one packed multiply-add.  The lane of a coil's first plane then
// sums the coil's planes times the basis.  All coils run in one launch.  Same weights and
// summation order as k_interp (w = (wy * 1) * wx, taps y-major).
// 256^2, 512k samples, 20 coils, K = 5: the whole forward model 1.50 against 4.14 ms, of which
// this kernel took 3.3 ms with a thread per sample and one coil's K planes in the window (reads
// at random cells meet banks twice and more); bound by the shared-memory reads (26 GB, 0.7 ms
// at 128 bytes a cycle and SM).
constexpr int kWinPitch = 17;
struct InterpTiledArgs {
  int M0, M1, K, cpg, nc, c0, u_complex, ntx;
  int64_t nt, ns_tot, cells;
  const void* U;
  const float2* g;         // [nc * K][cells]
  float2* data;            // (ns_pf, nt, ncoils)
  const TapRec* rec;       // tap records in sorted order
  const int4* items;       // (tile, first sorted position, count, -)
  const int* nitems;
  unsigned long long* next;  // work counter, zeroed before the launch
};

__global__ void __launch_bounds__(kTiledThreads, 3) k_interp_tiled(InterpTiledArgs a) {
  extern __shared__ float2 wk[];  // [kWinCells][kWinPitch]
  __shared__ unsigned long long s_unit;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = kTiledThreads / 32;
  const int half = lane >> 4, ch = lane & 15;
  const int K = a.K, cl = ch / K, k0 = cl * K;  // the lane's coil in the group and its first plane
  const int nitems = *a.nitems;
  const int ngroups = (a.nc + a.cpg - 1) / a.cpg;
  const unsigned long long total = (unsigned long long)nitems * ngroups;
  for (;;) {
    if (threadIdx.x == 0) s_unit = atomicAdd(a.next, 1ull);
    __syncthreads();
    const unsigned long long u = s_unit;
    if (u >= total) break;
    const int grp = (int)(u / nitems);
    const int4 item = a.items[u - (unsigned long long)grp * nitems];
    const int ox = (item.x % a.ntx) * kSpTile, oy = (item.x / a.ntx) * kSpTile;
    const int coils = min(a.cpg, a.nc - grp * a.cpg), np = coils * K;  // planes of the group
    const float2* g = a.g + (int64_t)grp * a.cpg * K * a.cells;
    for (int e = threadIdx.x; e < np * kWinCells; e += kTiledThreads) {
      const int p = e / kWinCells, c = e - p * kWinCells;
      const int row = c / kSpWin, col = c - row * kSpWin;
      wk[c * kWinPitch + p] = g[p * a.cells + wrap32(ox + col, a.M0) + (int64_t)a.M0 * wrap32(oy + row, a.M1)];
    }
    __syncthreads();
    for (int s0 = warp * 2; s0 < item.z; s0 += nwarps * 2) {
      const bool act = s0 + half < item.z;
      const float4* r4 = reinterpret_cast<const float4*>(a.rec + item.y + (act ? s0 + half : s0));
      float2 wx[kEsWidth];
      float wy[kEsWidth];
      {
        const float4 q0 = r4[0], q1 = r4[1], q2 = r4[2], q3 = r4[3];
        wx[0] = make_float2(q0.x, q0.x); wx[1] = make_float2(q0.y, q0.y);
        wx[2] = make_float2(q0.z, q0.z); wx[3] = make_float2(q0.w, q0.w);
        wx[4] = make_float2(q1.x, q1.x); wx[5] = make_float2(q1.y, q1.y);
        wx[6] = make_float2(q1.z, q1.z); wx[7] = make_float2(q1.w, q1.w);
        wy[0] = q2.x; wy[1] = q2.y; wy[2] = q2.z; wy[3] = q2.w;
        wy[4] = q3.x; wy[5] = q3.y; wy[6] = q3.z; wy[7] = q3.w;
      }
      const int4 ri = reinterpret_cast<const int4*>(r4)[4];  // li, t, lx0, ly0
      // the sort put the first tap in this tile (the same float arithmetic); the clamp keeps any
      // other position inside the window
      const int lx = min(max(ri.z - ox, 0), kSpTile - 1), ly = min(max(ri.w - oy, 0), kSpTile - 1);
      const float2* w = wk + (ly * kSpWin + lx) * kWinPitch + (ch < np ? ch : 0);
      float2 z = make_float2(0.f, 0.f);
#pragma unroll
      for (int t2 = 0; t2 < kEsWidth; ++t2) {
        const float2 w23 = make_float2(wy[t2], wy[t2]);
#pragma unroll
        for (int t1 = 0; t1 < kEsWidth; ++t1) z = fma2(mul2(w23, wx[t1]), w[(t2 * kSpWin + t1) * kWinPitch], z);
      }
      float2 y = make_float2(0.f, 0.f);
      for (int k = 0; k < K; ++k) {
        const int src = (half << 4) | ((k0 + k) & 15);
        const float2 zk = make_float2(__shfl_sync(0xffffffffu, z.x, src), __shfl_sync(0xffffffffu, z.y, src));
        if (a.u_complex)
          y = cadd(y, cmul(reinterpret_cast<const float2*>(a.U)[ri.y + a.nt * k], zk));
        else
          y = cadd(y, cscale(zk, reinterpret_cast<const float*>(a.U)[ri.y + a.nt * k]));
      }
      if (act && ch == k0 && cl < coils) a.data[ri.x + a.ns_tot * (a.c0 + grp * a.cpg + cl)] = y;
    }
    __syncthreads();
  }
}

// 3D: one warp per sample, lanes over its 512 taps (16 each, lane_taps), one shuffle
// reduction per plane; for 512 taps per sample this beats a thread per sample (which
// serialises 512 x K gathers in one thread).
__global__ void __launch_bounds__(256) k_interp3(InterpArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t ns_tot = a.S.ns_pf * a.S.nt;
  for (int64_t n = warp; n < a.S.n; n += nwarps) {
    const int64_t li = sample_lin(a.S, n);
    const int64_t t = frame_of(li, a.S.ns_pf);
    float w[16];
    unsigned cell[16];
    lane_taps<16>(a.S, a.M, li, lane, 1.f, w, cell);
    float2 z[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) z[k] = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < a.K) {
          const float2 gv = __ldg(a.g + (int64_t)cell[j] * a.K + k);
          z[k].x = fmaf(w[j], gv.x, z[k].x);
          z[k].y = fmaf(w[j], gv.y, z[k].y);
        }
    }
    float2 y = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < a.K) {
        float2 v = z[k];
        for (int o = 16; o > 0; o >>= 1) {
          v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
          v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (a.u_complex)
          y = cadd(y, cmul(reinterpret_cast<const float2*>(a.U)[t + a.S.nt * k], v));
        else
          y = cadd(y, cscale(v, reinterpret_cast<const float*>(a.U)[t + a.S.nt * k]));
      }
    }
    if (lane == 0) a.data[li + ns_tot * a.c] = y;
  }
}

// 3D on the tile sort (the backprojection's 8^3 tiles and tap records): a work item, up to
// 1024 samples whose first tap lies in one tile, loads the tile's 15^3-cell window of the K
// interleaved planes into shared memory once (216 KB for K = 8); a warp per sample, lanes over
// its 512 taps as in k_interp3 (lane = x tap + 8 y tap, 16 taps each), one shuffle reduction
// per plane.
struct InterpTiled3Args {
  int M0, M1, M2, K, c, u_complex, ntx, nty;
  int64_t nt, ns_tot;
  const void* U;
  const float2* g;         // [mcells][K]
  float2* data;            // (ns_pf, nt, ncoils)
  const TapRec3* rec;      // tap records in sorted order
  const int4* items;       // (tile, first sorted position, count, -)
  const int* nitems;
  int* next;               // work counter, zeroed before the launch
};

__global__ void __launch_bounds__(kTiledThreads, 1) k_interp_tiled3(InterpTiled3Args a) {
  extern __shared__ float2 wk[];  // [kWin3Cells][K]
  __shared__ int s_item;
  const int K = a.K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int t1 = lane & 7, t2a = lane >> 3;
  const int nitems = *a.nitems;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(a.next, 1);
    __syncthreads();
    const int it = s_item;
    if (it >= nitems) break;
    const int4 item = a.items[it];
    const int tx = item.x % a.ntx, ty = (item.x / a.ntx) % a.nty, tz = item.x / (a.ntx * a.nty);
    const int ox = tx * kTile3, oy = ty * kTile3, oz = tz * kTile3;
    for (int cw = threadIdx.x; cw < kWin3Cells; cw += blockDim.x) {
      const int wz = cw / (kWin3 * kWin3), r2 = cw - wz * kWin3 * kWin3, wy = r2 / kWin3, wx = r2 - wy * kWin3;
      const float2* src = a.g + (wrap32(ox + wx, a.M0) +
                                 (int64_t)a.M0 * (wrap32(oy + wy, a.M1) + (int64_t)a.M1 * wrap32(oz + wz, a.M2))) * K;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < K) wk[cw * K + k] = src[k];
    }
    __syncthreads();
    for (int sidx = warp; sidx < item.z; sidx += nwarps) {
      const TapRec3& r = a.rec[item.y + sidx];
      const int li = r.li, t = r.t, lx0 = r.lx0, ly0 = r.ly0, lz0 = r.lz0;
      const int lx = lx0 - ox, ly = ly0 - oy, lz = lz0 - oz;
      const bool in_win = (unsigned)lx < (unsigned)kTile3 && (unsigned)ly < (unsigned)kTile3 && (unsigned)lz < (unsigned)kTile3;
      const float wxl = r.wx[t1];
      float2 z[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) z[k] = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int t2 = t2a + 4 * (j & 1), t3 = j >> 1;
        const float w = (wxl * r.wy[t2]) * r.wz[t3];
        // the sort put the first tap in this tile (the same float arithmetic); a sample
        // outside it would read the grid itself
        const float2* cell =
            in_win ? wk + (((lz + t3) * kWin3 + ly + t2) * kWin3 + lx + t1) * K
                   : a.g + (wrap32(lx0 + t1, a.M0) +
                            (int64_t)a.M0 * (wrap32(ly0 + t2, a.M1) + (int64_t)a.M1 * wrap32(lz0 + t3, a.M2))) * K;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < K) {
            const float2 gv = cell[k];
            z[k].x = fmaf(w, gv.x, z[k].x);
            z[k].y = fmaf(w, gv.y, z[k].y);
          }
      }
      float2 y = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k < K) {
          float2 v = z[k];
          for (int o = 16; o > 0; o >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
          }
          if (a.u_complex)
            y = cadd(y, cmul(reinterpret_cast<const float2*>(a.U)[t + a.nt * k], v));
          else
            y = cadd(y, cscale(v, reinterpret_cast<const float*>(a.U)[t + a.nt * k]));
        }
      }
      if (lane == 0) a.data[li + a.ns_tot * a.c] = y;
    }
    __syncthreads();
  }
}

static int check_smooth(int d, const int64_t* G) {
  for (int i = 0; i < d; ++i) {
    int rad[kMaxStages], ns;
    MRSR_REQUIRE(build_radices((int)G[i], rad, &ns), MRSR_ERR_ARG,
                 "AssertionError: img_shape_os has to be composed of the prime factors 2, 3, and 5 (cf. NonuniformFFTs.jl "
                 "documentation).");
  }
  return MRSR_OK;
}

}  // namespace mrsr

using namespace mrsr;

static cudaStream_t nstream(mrsr_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

extern "C" int mrsr_nfft_normalop_create(int ndims, const int64_t* img_shape, int64_t ns_per_frame, int64_t nt,
                                         const float* trj, const uint8_t* sample_mask, const void* U, int u_is_complex,
                                         int K, const float* cmaps, int ncoils, int precision, mrsr_stream_t stream,
                                         mrsr_normalop** out) {
  MRSR_CALL_SCOPE(reinterpret_cast<cudaStream_t>(stream));
  MRSR_REQUIRE(out, MRSR_ERR_ARG, "out is NULL");
  *out = nullptr;
  MRSR_REQUIRE(trj && U, MRSR_ERR_ARG, "trj and U must be device pointers");
  MRSR_REQUIRE(ns_per_frame >= 1 && nt >= 1, MRSR_ERR_ARG, "empty trajectory");
  cudaStream_t st = nstream(stream);
  mrsr_normalop* op = new mrsr_normalop();
  int s = op_init_geometry(op, MRSR_KIND_NFFT, ndims, img_shape, K, cmaps != nullptr, ncoils, precision);
  if (s == MRSR_OK) s = op_set_cmaps(op, cmaps, st);
  SampleList sl;
  DevBuf kmask, packed;
  int64_t nk = 0;
  if (s == MRSR_OK) s = check_smooth(ndims, op->geo.g);
  if (s == MRSR_OK) s = sl.init(ndims, trj, ns_per_frame, nt, sample_mask, st);
  if (s == MRSR_OK) s = compute_lambda(ndims, op->geo.g, sl.set, U, u_is_complex, K, kmask, &nk, packed, st);
  if (s == MRSR_OK) s = op_set_lambda_packed(op, packed.p, u_is_complex, kmask.as<int64_t>(), nk, st);
  if (s == MRSR_OK) s = op_finalize(op, st);
  if (s != MRSR_OK) {
    delete op;
    return s;
  }
  *out = op;
  return MRSR_OK;
}

extern "C" int mrsr_backprojection(int ndims, const int64_t* img_shape, int64_t ns_per_frame, int64_t nt, int ncoils,
                                   const float* data, const float* trj, const uint8_t* sample_mask, const void* U,
                                   int u_is_complex, int K, const float* cmaps, int dcf_kind, const float* dcf_array,
                                   float* out, mrsr_stream_t stream) {
  MRSR_CALL_SCOPE(reinterpret_cast<cudaStream_t>(stream));
  MRSR_REQUIRE(ndims == 2 || ndims == 3, MRSR_ERR_ARG, "ndims must be 2 or 3");
  MRSR_REQUIRE(img_shape && data && trj && out, MRSR_ERR_ARG, "NULL argument to mrsr_backprojection");
  MRSR_REQUIRE(ncoils >= 1 && ns_per_frame >= 1 && nt >= 1, MRSR_ERR_ARG, "empty data");
  if (!U) K = (int)nt;
  MRSR_REQUIRE(K >= 1, MRSR_ERR_ARG, "K must be >= 1");
  MRSR_REQUIRE(U != nullptr || K <= 1 << 20, MRSR_ERR_ARG, "too many frames for an identity basis");
  MRSR_REQUIRE(dcf_kind >= MRSR_DCF_NONE && dcf_kind <= MRSR_DCF_ARRAY, MRSR_ERR_ARG,
               "`density_compensation` can only be `:radial_3D`, `:radial_2D`, `:none`, or of type `AbstractArray`");
  MRSR_REQUIRE(dcf_kind != MRSR_DCF_ARRAY || dcf_array, MRSR_ERR_ARG, "density compensation array is NULL");
  cudaStream_t st = nstream(stream);
  int64_t N[3] = {1, 1, 1}, M[3] = {1, 1, 1};
  for (int i = 0; i < ndims; ++i) {
    N[i] = img_shape[i];
    M[i] = 2 * N[i];
  }
  MRSR_TRY(check_smooth(ndims, M));
  const int64_t nimg = N[0] * N[1] * N[2], mcells = M[0] * M[1] * M[2];
  SampleList sl;
  MRSR_TRY(sl.init(ndims, trj, ns_per_frame, nt, sample_mask, st));
  MRSR_REQUIRE(sl.set.n > 0, MRSR_ERR_ARG, "AssertionError: Sample mask removes all samples, cannot compute backprojection.");
  FftNd fM;
  MRSR_TRY(fM.init(ndims, M));
  const float* ipsi[3] = {nullptr, nullptr, nullptr};
  for (int i = 0; i < ndims; ++i) MRSR_TRY(es_inv_psi_table(M[i], -(N[i] / 2), N[i], &ipsi[i]));
  // coil batches of ~2 GB of float2 grid
  const int64_t max_bytes = 2ll << 30;
  const int64_t per_coil = (int64_t)K * mcells * (int64_t)sizeof(float2);
  int cc = (int)std::max<int64_t>(1, std::min<int64_t>(ncoils, max_bytes / std::max<int64_t>(per_coil, 1)));
  // 3D with a basis: the batch's parts (2 per coil and coefficient) interleaved per cell, at
  // most 32 (one per lane of k_spread_data_cp)
  const bool tiled = U != nullptr && sl.set.n < (1ll << 31) && ns_per_frame * nt < (1ll << 31);
  const bool parts_layout = ndims == 3 && U != nullptr && !tiled && 2 * K <= 32;
  if (parts_layout) cc = std::min(cc, 16 / K);
  const bool rows = tiled && (ndims == 2 || rows_pay(2 * K * cc, 2 * K * ncoils, sl.set.n, mcells));
  DevBuf grid, qgrid, fsb;
  MRSR_TRY(grid.alloc((size_t)per_coil * cc));
  // fixed-point re and im, 8 bytes each
  MRSR_TRY(qgrid.alloc(rows ? spread_rows_bytes(2 * K * cc, mcells) : (size_t)per_coil * 2 * cc));
  // fixed-point scale: |term component| <= max|data| max|U| (x2 for complex U) x dcf bound,
  // at most ceil(w / M) taps per sample, cell and dimension
  MRSR_TRY(fsb.alloc(sizeof(FixedScale)));
  // an identity basis gives every sample one channel: the global kernel
  {
    const float* f[3];
    int64_t n[3];
    int nf = 0;
    double mult = 1.0;
    f[nf] = data;
    n[nf++] = 2 * ns_per_frame * nt * (int64_t)ncoils;
    if (U) {
      f[nf] = reinterpret_cast<const float*>(U);
      n[nf++] = nt * (int64_t)K * (u_is_complex ? 2 : 1);
      if (u_is_complex) mult *= 2.0;
    }
    if (dcf_kind == MRSR_DCF_RADIAL_2D) mult *= 0.5 * std::sqrt((double)ndims);  // |k| <= sqrt(d) / 2
    if (dcf_kind == MRSR_DCF_RADIAL_3D) mult *= 0.25 * ndims;                   // |k|^2 <= d / 4
    if (dcf_kind == MRSR_DCF_ARRAY) {
      f[nf] = dcf_array;
      n[nf++] = sl.set.n;
    }
    MRSR_TRY(fixed_scale(f, n, nf, mult, (double)sl.set.n * taps_per_cell(ndims, M), rows, fsb.as<FixedScale>(), st));
  }
  TileSort ts;
  DevBuf umax, tmax;
  const bool ordered = ndims == 3 && sl.set.n < (1ll << 31);
  if (tiled || ordered) MRSR_TRY(ts.build(sl.set, M, rows ? kSpTile : kTile3, rows ? spread_chunk(ndims, sl.set.n) : kChunk, rows, st));
  if (tiled) MRSR_TRY(ts.prep(sl.set, dcf_kind, dcf_array, st));
  if (rows) {
    MRSR_TRY(tmax.alloc(sizeof(float) * (size_t)ts.ntiles * cc));
    MRSR_TRY(basis_max(sl.set, U, u_is_complex, K, 2 * K * ncoils, umax, st));
  }
  const int64_t out_elems = nimg * K * (cmaps ? 1 : ncoils);
  if (cmaps) MRSR_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(float2) * out_elems, st));
  for (int c0 = 0; c0 < ncoils; c0 += cc) {
    const int nc = std::min(cc, ncoils - c0);
    int* bad = rows ? umax.as<int>() + K + 2 * K * c0 : nullptr;
    MRSR_CHECK_CUDA(cudaMemsetAsync(qgrid.p, 0, rows ? spread_rows_bytes(2 * K * nc, mcells) : (size_t)per_coil * 2 * nc, st));
    SpreadDataArgs sa{sl.set, {M[0], M[1], M[2]}, mcells, reinterpret_cast<const float2*>(data), c0, nc, U,
                      u_is_complex, K, dcf_kind, dcf_array, qgrid.as<long long>(), fsb.as<FixedScale>(), umax.as<float>(),
                      tmax.as<float>(), bad};
    MRSR_TRY(spread_data(sa, tiled || ordered ? &ts : nullptr, st));
    if (rows) {
      MRSR_TRY(parts_to_grid(qgrid.as<long long>(), 2, mcells, 2 * K * nc, fsb.as<FixedScale>(), bad,
                             grid.as<float2>(), st));
    } else if (parts_layout) {
      k_fixed_to_grid_cp<<<(unsigned)cdiv(mcells, 32), 256, 0, st>>>(qgrid.as<long long>(), 2 * nc * K, mcells,
                                                                    fsb.as<FixedScale>(), grid.as<float2>());
      MRSR_LAUNCH_CHECK();
    } else {
      MRSR_TRY(fixed_to_grid(qgrid.as<long long>(), 2, mcells, (int64_t)nc * K, fsb.as<FixedScale>(),
                             grid.as<float2>(), st));
    }
    MRSR_TRY(fM.run(grid.as<float2>(), (int64_t)nc * K, +1, 1.0f, st));
    BpFoldArgs fa;
    fa.d = ndims;
    for (int i = 0; i < 3; ++i) {
      fa.N[i] = N[i];
      fa.M[i] = M[i];
      fa.ipsi[i] = ipsi[i];
    }
    fa.nimg = nimg;
    fa.mcells = mcells;
    fa.K = K;
    fa.dc.init(ndims, N, K);
    fa.c0 = c0;
    fa.nc = nc;
    fa.ncoils = ncoils;
    fa.g = grid.as<float2>();
    fa.cmaps = reinterpret_cast<const float2*>(cmaps);
    fa.out = reinterpret_cast<float2*>(out);
    k_bp_fold<<<grid1d(nimg * K), 256, 0, st>>>(fa);
    MRSR_LAUNCH_CHECK();
  }
  return MRSR_OK;  // asynchronous on `st`; the temporaries are freed in stream order
}

extern "C" int mrsr_forward_model(int ndims, const int64_t* img_shape, int64_t ns_per_frame, int64_t nt, int ncoils,
                                  const float* x, const float* trj, const void* U, int u_is_complex, int K,
                                  const float* cmaps, float* data_out, mrsr_stream_t stream) {
  MRSR_CALL_SCOPE(reinterpret_cast<cudaStream_t>(stream));
  MRSR_REQUIRE(ndims == 2 || ndims == 3, MRSR_ERR_ARG, "ndims must be 2 or 3");
  MRSR_REQUIRE(img_shape && x && trj && U && data_out, MRSR_ERR_ARG, "NULL argument to mrsr_forward_model");
  MRSR_REQUIRE(K >= 1 && K <= 8, MRSR_ERR_UNSUPPORTED, "forward model supports 1 <= K <= 8");
  MRSR_REQUIRE(ncoils >= 1, MRSR_ERR_ARG, "ncoils must be >= 1");
  MRSR_REQUIRE(cmaps || ncoils == 1, MRSR_ERR_ARG, "cmaps == NULL requires ncoils == 1");
  cudaStream_t st = nstream(stream);
  int64_t N[3] = {1, 1, 1}, M[3] = {1, 1, 1};
  for (int i = 0; i < ndims; ++i) {
    N[i] = img_shape[i];
    M[i] = 2 * N[i];
  }
  MRSR_TRY(check_smooth(ndims, M));
  const int64_t nimg = N[0] * N[1] * N[2], mcells = M[0] * M[1] * M[2];
  SampleList sl;
  MRSR_TRY(sl.init(ndims, trj, ns_per_frame, nt, nullptr, st));
  FftNd fM;
  MRSR_TRY(fM.init(ndims, M));
  const float* ipsi[3] = {nullptr, nullptr, nullptr};
  for (int i = 0; i < ndims; ++i) MRSR_TRY(es_inv_psi_table(M[i], -(N[i] / 2), N[i], &ipsi[i]));
  // the interpolation runs on the tile sort of the samples (built once for all coils)
  TileSort ts;
  const bool small = sl.set.n < (1ll << 31) && ns_per_frame * nt < (1ll << 31);
  const bool tiled = ndims == 2 && small && M[0] < (1ll << 24) && M[1] < (1ll << 24);
  const int64_t ntiles3 = cdiv(M[0], kTile3) * cdiv(M[1], kTile3) * cdiv(M[2], kTile3);
  const bool tiled3 = ndims == 3 && small && ntiles3 < (1ll << 31) && mcells < (1ll << 32);
  if (tiled) {
    MRSR_TRY(ts.build(sl.set, M, kSpTile, kChunk, false, st));
    MRSR_TRY(ts.prep(sl.set, MRSR_DCF_NONE, nullptr, st));
  } else if (tiled3) {
    MRSR_TRY(ts.build(sl.set, M, kTile3, kChunk, false, st));
    MRSR_TRY(ts.prep(sl.set, MRSR_DCF_NONE, nullptr, st));
  }
  // coils per pass: all of a 2 GB batch in the 2D tile-sorted kernel, one elsewhere
  const int cc = tiled ? (int)std::max<int64_t>(1, std::min<int64_t>(ncoils, (2ll << 30) / ((int64_t)sizeof(float2) * K * mcells))) : 1;
  DevBuf grid, gridi;
  MRSR_TRY(grid.alloc(sizeof(float2) * K * mcells * cc));
  if (!tiled) MRSR_TRY(gridi.alloc(sizeof(float2) * K * mcells));
  const size_t win_bytes = sizeof(float2) * kWinCells * kWinPitch;
  const size_t win3_bytes = sizeof(float2) * kWin3Cells * (size_t)K;
  if (tiled) MRSR_CHECK_CUDA(cudaFuncSetAttribute(k_interp_tiled, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)win_bytes));
  if (tiled3)
    MRSR_CHECK_CUDA(cudaFuncSetAttribute(k_interp_tiled3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)win3_bytes));
  for (int c = 0; c < ncoils; c += cc) {
    const int nc = std::min(cc, ncoils - c);
    MRSR_CHECK_CUDA(cudaMemsetAsync(grid.p, 0, sizeof(float2) * K * mcells * nc, st));
    FwdPlaceArgs pa;
    pa.d = ndims;
    for (int i = 0; i < 3; ++i) {
      pa.N[i] = N[i];
      pa.M[i] = M[i];
      pa.ipsi[i] = ipsi[i];
    }
    pa.nimg = nimg;
    pa.mcells = mcells;
    pa.K = K;
    pa.dc.init(ndims, N, K);
    pa.c = c;
    pa.x = reinterpret_cast<const float2*>(x);
    pa.cmaps = reinterpret_cast<const float2*>(cmaps);
    pa.g = grid.as<float2>();
    k_fwd_place<<<dim3(grid1d(nimg * K), nc), 256, 0, st>>>(pa);
    MRSR_LAUNCH_CHECK();
    MRSR_TRY(fM.run(grid.as<float2>(), (int64_t)nc * K, -1, 1.0f, st));
    if (!tiled) {
      k_interleave<<<grid1d(mcells), 256, 0, st>>>(grid.as<float2>(), gridi.as<float2>(), K, mcells);
      MRSR_LAUNCH_CHECK();
    }
    InterpArgs ia{sl.set, {M[0], M[1], M[2]}, mcells, K, c, u_is_complex, U, gridi.as<float2>(),
                  reinterpret_cast<float2*>(data_out)};
    if (tiled3) {
      InterpTiled3Args ta;
      ta.M0 = (int)M[0];
      ta.M1 = (int)M[1];
      ta.M2 = (int)M[2];
      ta.K = K;
      ta.c = c;
      ta.u_complex = u_is_complex;
      ta.ntx = ts.ntx;
      ta.nty = ts.nty;
      ta.nt = nt;
      ta.ns_tot = ns_per_frame * nt;
      ta.U = U;
      ta.g = gridi.as<float2>();
      ta.data = reinterpret_cast<float2*>(data_out);
      ta.rec = ts.rec.as<TapRec3>();
      ta.items = ts.items.as<int4>();
      ta.nitems = ts.nitems.as<int>();
      ta.next = ts.next.as<int>();
      MRSR_CHECK_CUDA(cudaMemsetAsync(ts.next.p, 0, sizeof(int), st));
      k_interp_tiled3<<<152, kTiledThreads, win3_bytes, st>>>(ta);
    } else if (ndims == 3) {
      MRSR_REQUIRE(mcells < (1ll << 32), MRSR_ERR_UNSUPPORTED, "forward model grid of 2^32 cells or more");
      k_interp3<<<spread_blocks(sl.set.n), 256, 0, st>>>(ia);
    } else if (tiled) {
      InterpTiledArgs ta;
      ta.M0 = (int)M[0];
      ta.M1 = (int)M[1];
      ta.K = K;
      ta.cpg = 16 / K;
      ta.nc = nc;
      ta.c0 = c;
      ta.u_complex = u_is_complex;
      ta.ntx = ts.ntx;
      ta.nt = nt;
      ta.ns_tot = ns_per_frame * nt;
      ta.cells = mcells;
      ta.U = U;
      ta.g = grid.as<float2>();
      ta.data = reinterpret_cast<float2*>(data_out);
      ta.rec = ts.rec.as<TapRec>();
      ta.items = ts.items.as<int4>();
      ta.nitems = ts.nitems.as<int>();
      ta.next = ts.next.as<unsigned long long>();
      MRSR_CHECK_CUDA(cudaMemsetAsync(ts.next.p, 0, sizeof(unsigned long long), st));
      k_interp_tiled<<<152 * 3, kTiledThreads, win_bytes, st>>>(ta);
    } else {
      k_interp<<<(unsigned)std::min<int64_t>(std::max<int64_t>(cdiv(sl.set.n, 256), 1), 152 * 64), 256, 0, st>>>(ia);
    }
    MRSR_LAUNCH_CHECK();
  }
  return MRSR_OK;  // asynchronous on `st`
}
