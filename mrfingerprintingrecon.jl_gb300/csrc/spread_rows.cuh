// Tile-sorted spreading with register accumulators (2D, and 3D where rows_pay in
// spread_windows.cuh says so; nufft.cu).
//
// Samples are counting-sorted by the tile (16 cells a side) that holds their first tap; the
// footprints of a tile's samples lie in a window of 23 cells a side.  A work unit is a chunk of at
// most 384 samples of one tile and, in 3D, one z-plane of the window; it takes the window's rows
// twelve at a time and the accumulator parts (the real and imaginary planes of the channels) in
// groups of P.  A lane owns one part of one window row and keeps the row's 23 sums in
// registers, so a term costs one multiply-add and no shared-memory atomic.  The chunk's samples
// are ordered by their x position in shared memory, and the loop over them is unrolled over the
// 16 positions, so which 8 of the 23 sums a sample adds to is known at compile time.
//
// Sums are integers, so a cell does not depend on the order in which samples, chunks or units
// land: with 2^a the largest power of two that keeps |value| 2^a within 2^29 for every sample
// of the tile (a bound per tile and part, formed from maxima, which do not depend on an order
// either), a term is rint(value wy [wz] 2^a) * rint(wx 2^25), and the at most 384 terms of a
// chunk stay below 2^63.  (The sums run on unsigned products of value + 2^31, modulo 2^64; what
// the offset adds is the sum of the row's x taps times 2^31, kept per column beside.)  The row
// is then rounded once to the grid's units 2^-e and added with one 64-bit atomic per cell, the
// lanes of a warp on the consecutive parts of a [cell][P] grid.  The results are as far from
// 64-bit sums as those of terms rounded to 2^-40 of the largest one (1.6e-7 on 256^2, 512k
// samples, 20 coils; with 27 bits for the values instead of 29, 1.7e-7).
//
// An integer cannot hold an infinity or a NaN, so the maxima (which run over the samples and
// frames that are used) are infinite where one of their entries is not finite.  Such a bound marks
// its part in `bad`, and the conversion to float makes every cell of a marked part NaN, as a float
// sum's transform would be.  (A check of every value instead took 4% of the backprojection of
// 256^2, 20 coils.)
//
// 256^2, 512k samples, 20 coils, K = 5 (200 parts): 1.51 ms against 2.93 ms for windows of 32-bit
// limbs in shared memory, two shared atomics and about eight instructions per term; the 15
// parts of the kernel precompute on 512^2: 0.23 against 0.46 ms; 64^3, 307k samples, 8 coils,
// K = 4: 2.93 against 6.28 ms.  An inner step takes 20 instructions for the 8 terms of a sample
// and row, at 24 warps per SM; it waits on shared-memory loads, and the stages around it
// (ordering, values, barriers) take the rest of the time.  32 x 32 + 64-bit multiply-adds alone
// run at 18 T/s, 32-bit shared atomics at 9.5 T/s, and a float form (two limbs, four FMAs per
// term) at 7 T/s.
// Tiles of 16: the flush is 2.07 (2D) or 2.97 (3D) atomics per grid cell and part, against
// 2.5 and 6.6 with tiles of 12 (2D) and 8 (3D), and 64-bit atomics run at 0.73 T/s.
#pragma once

namespace mrsr {

constexpr int kSpTile = 16;
constexpr int kSpWin = kSpTile + kEsWidth - 1;  // 23
constexpr int kWinCells = kSpWin * kSpWin;
constexpr int kSpWarps = 12;
constexpr int kSpThreads = kSpWarps * 32;
constexpr int kSpChunk = kSpThreads;          // samples of a chunk, at most: one per thread
constexpr int kSpValBits = 29, kSpTapBits = 25;
static_assert((unsigned long long)kSpChunk << (kSpValBits + kSpTapBits) < 7ull << 60, "a chunk's sums must fit in 63 bits");

struct SpreadRowsArgs {
  int M0, M1, M2;
  int64_t cells;
  int nparts;              // parts to spread
  long long* q;            // [ceil(nparts / P)][cells][P]
  const FixedScale* fs;
  int* bad;                // [nparts], cleared by k_basis_max: set for parts that hold a value that is not finite
  int ntx, nty;
  const void* rec;         // TapRec (2D) or TapRec3 (3D) in sorted order
  const int4* items;       // (tile, first sorted position, count, -)
  const int* nitems;
  unsigned long long* next;  // work counter, zeroed before the launch
};

// bound of a product of two values from their bounds: NaN if one of them is not finite
__device__ __forceinline__ float part_bound(float a, float b) {
  return finite_value(a) && finite_value(b) ? fminf(a * b, kFltMax) : __int_as_float(0x7fc00000);
}

// Part p of the Λ precompute: pair p0 + p / nq (k1 <= k2, packed k2 (k2 + 1) / 2 + k1), plane
// p % nq; value conj(U[t,k1]) U[t,k2] (k_spread_lambda's value).  umax[k]: k_basis_max of U.
struct LamParts {
  const void* U;
  const float* umax;
  int u_complex, nq, p0;
  int64_t nt;
  struct Lane {
    int64_t o1, o2;  // columns k1, k2 of U
    float bd;
    int q;
  };
  __device__ Lane bind(int part, int) const {
    const int ch = part / nq, q = part - ch * nq, p = p0 + ch;
    int k2 = 0;
    while ((k2 + 1) * (k2 + 2) / 2 <= p) ++k2;
    const int k1 = p - k2 * (k2 + 1) / 2;
    return Lane{nt * k1, nt * k2, umax ? part_bound(umax[k1], umax[k2]) : 0.f, q};
  }
  __device__ __forceinline__ float value(const Lane& L, int, int t) const {
    if (u_complex) {
      const float2* u = reinterpret_cast<const float2*>(U) + t;
      const float2 v = cmulc(u[L.o2], u[L.o1]);  // conj(U[t,k1]) * U[t,k2]
      return L.q ? v.y : v.x;
    }
    const float* u = reinterpret_cast<const float*>(U) + t;
    return u[L.o2] * u[L.o1];
  }
};

// Part p of the backprojection: channel p / 2 = (coil c0 + c) K + k, plane p % 2; value
// y_c conj(U[t,k]) (k_spread_data's value; the tap weights carry the density compensation).
// tmax[tile][c]: largest component of the tile's samples times their density compensation
// (k_tile_absmax).
struct DataParts {
  const float2* data;
  const void* U;
  const float *umax, *tmax;
  int u_complex, K, c0, nc;
  int64_t nt, ns_tot;
  struct Lane {
    const float2* y;  // samples of coil c
    int64_t ok;       // column k of U
    float bd;
    int q;
  };
  __device__ Lane bind(int part, int tile) const {
    const int ch = part >> 1, c = ch / K, k = ch - c * K;
    return Lane{data + ns_tot * (c0 + c), nt * k, tmax ? part_bound(tmax[(int64_t)tile * nc + c], umax[k]) : 0.f, part & 1};
  }
  __device__ __forceinline__ float value(const Lane& L, int li, int t) const {
    if (u_complex) {
      const float2 v = cmulc(L.y[li], (reinterpret_cast<const float2*>(U) + t)[L.ok]);  // y * conj(U)
      return L.q ? v.y : v.x;
    }
    const float uu = (reinterpret_cast<const float*>(U) + t)[L.ok];
    return reinterpret_cast<const float*>(L.y + li)[L.q] * uu;
  }
};

// used[t] = 1 for the frames (zeroed before) that have a kept sample
__global__ void k_frames_used(SampleSet S, uint8_t* used) {
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < S.n; n += (int64_t)gridDim.x * blockDim.x)
    used[frame_of(sample_lin(S, n), S.ns_pf)] = 1;
}

// umax[k] = max over the used frames t (all without `used`) of |U[t,k]| (real) or |re| + |im|
// (complex), infinite if one of them is not finite; one block per column.  Clears the nbad marks.
__global__ void k_basis_max(const void* U, int64_t nt, int cplx, const uint8_t* used, float* umax, int* bad, int nbad) {
  __shared__ float red[32];
  const int k = blockIdx.x;
  for (int i = k * blockDim.x + threadIdx.x; i < nbad; i += gridDim.x * blockDim.x) bad[i] = 0;
  float m = 0.f;
  for (int64_t t = threadIdx.x; t < nt; t += blockDim.x) {
    if (used && !used[t]) continue;
    float v;
    if (cplx) {
      const float2 u = reinterpret_cast<const float2*>(U)[t + nt * k];
      v = fabsf(u.x) + fabsf(u.y);
    } else {
      v = fabsf(reinterpret_cast<const float*>(U)[t + nt * k]);
    }
    m = finite_value(v) ? fmaxf(m, v) : __int_as_float(0x7f800000);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, red[w]);
    umax[k] = m;
  }
}

// umax: K maxima followed by nparts marks
static int basis_max(const SampleSet& S, const void* U, int cplx, int K, int nparts, DevBuf& umax, cudaStream_t st) {
  DevBuf used;
  MRSR_TRY(umax.alloc(sizeof(float) * K + sizeof(int) * nparts));
  if (S.n < S.ns_pf * S.nt) {  // a mask may have taken all samples of a frame
    MRSR_TRY(used.alloc(S.nt));
    MRSR_CHECK_CUDA(cudaMemsetAsync(used.p, 0, S.nt, st));
    k_frames_used<<<(unsigned)std::min<int64_t>(cdiv(S.n, 256), 152 * 16), 256, 0, st>>>(S, used.as<uint8_t>());
    MRSR_LAUNCH_CHECK();
  }
  k_basis_max<<<K, 256, 0, st>>>(U, S.nt, cplx, used.as<uint8_t>(), umax.as<float>(), umax.as<int>() + K, nparts);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

// tmax[tile][c] (zeroed before) = largest max(|re|, |im|) * |density compensation| over the
// tile's samples of coil c0 + c, infinite if one of them is not finite.  Neighbouring samples share
// a tile: one atomic per run of equal tiles in a warp and coil.
__global__ void k_tile_absmax(SampleSet S, const int* tile_of, const float2* data, int c0, int nc, int dcf_kind,
                              const float* dcf, unsigned* tmax) {
  const int64_t ns_tot = S.ns_pf * S.nt;
  const int lane = threadIdx.x & 31;
  for (int64_t n0 = blockIdx.x * (int64_t)blockDim.x; n0 < S.n; n0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = n0 + threadIdx.x;
    const bool act = n < S.n;
    const int64_t li = act ? sample_lin(S, n) : 0;
    const int tile = act ? tile_of[n] : -1;
    const float w = act ? fabsf(sample_dcf(S, n, li, dcf_kind, dcf)) : 0.f;
    const unsigned grp = __match_any_sync(0xffffffffu, tile);
    const bool lead = act && (int)(__ffs(grp) - 1) == lane;
    for (int c = 0; c < nc; ++c) {
      unsigned b = 0;
      if (act) {
        const float2 y = data[li + ns_tot * (c0 + c)];
        const float v = fmaxf(fabsf(y.x), fabsf(y.y)) * w;
        b = finite_value(y.x) && finite_value(y.y) && finite_value(v) ? __float_as_uint(v) : 0x7f800000u;
      }
      b = __reduce_max_sync(grp, b);
      if (lead && b) atomicMax(&tmax[(int64_t)tile * nc + c], b);
    }
  }
}

// acc += v * w, 32 x 32 + 64 bits, unsigned (one instruction; the signed form takes 1.5)
__device__ __forceinline__ void sp_mad(unsigned long long& acc, unsigned v, unsigned w) {
  acc += (unsigned long long)v * w;
}

// A warp keeps the rows of 32 / P lane groups.
template <int P, int D, class Parts>
__global__ void __launch_bounds__(kSpThreads, 2) k_spread_rows(SpreadRowsArgs a, Parts parts) {
  using Rec = typename std::conditional<D == 3, TapRec3, TapRec>::type;
  constexpr int RW = 32 / P;                      // rows of a warp at a time
  constexpr int RU = kSpWarps * RW;               // rows of the block at a time
  constexpr int NZ = D == 3 ? kSpWin : 1;         // window planes
  constexpr int NB = kSpChunk;
  constexpr int NK = kSpTile * kSpTile;           // (lx, ly) bins
  // a staged sample: P values times 2^a (and wz), the x taps times 2^25 (int), the y taps of the
  // rows 0 .. 23 (0 outside its footprint)
  constexpr int TX = P, TY = P + kEsWidth, TW = P + 32;
  extern __shared__ __align__(16) float slots[];  // [NB][TW]
  float4* list = reinterpret_cast<float4*>(slots + NB * TW);  // [NB] staged samples: index, frame, place, wz
  int* start = reinterpret_cast<int*>(list + NB);  // [NK + 1] first staged sample of every bin
  int* bins = start + NK + 4;                      // [NK]
  unsigned long long* csum = reinterpret_cast<unsigned long long*>(bins + NK);  // [ly][24] sums of x taps
  __shared__ int wsum[NK / 64];
  __shared__ unsigned long long s_unit;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int part = lane % P, rsub = lane / P;
  const int nitems = *a.nitems;
  const int ngroups = (a.nparts + P - 1) / P;
  const unsigned long long total = (unsigned long long)nitems * NZ;
  const int e_grid = (int)((__float_as_uint(a.fs->scale) >> 23) & 255u) - 127 + kFxLoBits;
  const Rec* recs = reinterpret_cast<const Rec*>(a.rec);
  for (int b = tid; b < NK; b += kSpThreads) bins[b] = 0;
  for (;;) {
    if (tid == 0) s_unit = atomicAdd(a.next, 1ull);
    __syncthreads();
    const unsigned long long u = s_unit;
    if (u >= total) break;
    const int z = (int)(u % NZ);
    const int4 item = a.items[u / NZ];
    const int tx = item.x % a.ntx, tyz = item.x / a.ntx;
    const int ox = tx * kSpTile, oy = (D == 3 ? tyz % a.nty : tyz) * kSpTile, oz = (D == 3 ? tyz / a.nty : 0) * kSpTile;
    // the samples (in 3D, those whose footprint meets the plane), counted by (lx, ly)
    int key = -1, rank = 0;
    float4 ent = make_float4(0.f, 0.f, 0.f, 1.f);
    if (tid < item.z) {
      const Rec& r = recs[item.y + tid];
      const int4 ri = *reinterpret_cast<const int4*>(&r.li);  // li, t, lx0, ly0
      const int lx = ri.z - ox, ly = ri.w - oy;
      // the sort put the first tap in this tile (the same float arithmetic)
      bool use = (unsigned)lx < (unsigned)kSpTile && (unsigned)ly < (unsigned)kSpTile;
      if constexpr (D == 3) {
        const int lz = r.lz0 - oz;
        use = use && (unsigned)lz < (unsigned)kSpTile && (unsigned)(z - lz) < (unsigned)kEsWidth;
        if (use) ent.w = r.wz[z - lz];
      }
      if (use) {
        key = lx * kSpTile + ly;
        rank = atomicAdd(&bins[key], 1);
        ent.x = __int_as_float(ri.x);
        ent.y = __int_as_float(ri.y);
        ent.z = __int_as_float(key | (tid << 8));
      }
    }
    for (int t = tid; t < kSpTile * (kSpWin + 1); t += kSpThreads) csum[t] = 0;
    __syncthreads();
    // exclusive scan of the bins; thread t < NK / 2 takes bins 2 t and 2 t + 1
    int2 cc = make_int2(0, 0);
    int x = 0;
    if (tid < NK / 2) {
      cc = reinterpret_cast<int2*>(bins)[tid];
      reinterpret_cast<int2*>(bins)[tid] = make_int2(0, 0);
      x = cc.x + cc.y;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) wsum[warp] = x;
    }
    __syncthreads();
    int ns = 0;
    for (int w = 0; w < NK / 64; ++w) {
      if (w < warp) x += wsum[w];
      ns += wsum[w];
    }
    if (tid < NK / 2) reinterpret_cast<int2*>(start)[tid] = make_int2(x - cc.x - cc.y, x - cc.y);
    if (tid == 0) start[NK] = ns;
    __syncthreads();
    if (ns == 0) continue;
    if (key >= 0) list[start[key] + rank] = ent;
    __syncthreads();
    // taps of the staged samples, a warp each
#pragma unroll 1
    for (int i = warp; i < ns; i += kSpWarps) {
      const int pl = __float_as_int(list[i].z);         // ly | lx << 4 | place in the item << 8
      const int dy = lane - kEsWidth - (pl & 15);       // lanes 8 .. 31: rows 0 .. 23
      const Rec& r = recs[item.y + (pl >> 8)];
      const float* src = lane < kEsWidth ? r.wx + lane : r.wy + dy;  // one load for all lanes
      const float tap = lane < kEsWidth || (unsigned)dy < (unsigned)kEsWidth ? *src : 0.f;
      if (lane < kEsWidth) {
        const int w = __float2int_rn(tap * (float)(1 << kSpTapBits));
        reinterpret_cast<int*>(slots)[i * TW + TX + lane] = w;
        atomicAdd(&csum[(pl & 15) * (kSpWin + 1) + ((pl >> 4) & 15) + lane], (unsigned long long)w);
      } else {
        slots[i * TW + TX + lane] = tap;
      }
    }
    for (int grp = 0; grp < ngroups; ++grp) {
      const int gpart = grp * P + part;
      const bool live = gpart < a.nparts;
      const typename Parts::Lane L = parts.bind(live ? gpart : 0, item.x);
      // 2^a: bound < 2^ex
      float bd = live ? L.bd : 0.f;
      if (!(bd >= 0.f)) {
        a.bad[gpart] = 1;
        bd = 0.f;
      }
      const int ex = max((int)(__float_as_uint(bd) >> 23), 1) - 126;
      const int ea = min(kSpValBits - ex, 126);
      const float scale = bd > 0.f ? __int_as_float((ea + 127) << 23) : 0.f;
      // values of the staged samples, two at a time
      for (int i0 = warp * RW + rsub; i0 < ns; i0 += RU * 2) {
        float val[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int i = i0 + j * RU;
          if (i >= ns) break;
          const float4 en = list[i];
          val[j] = live ? parts.value(L, __float_as_int(en.x), __float_as_int(en.y)) : 0.f;
          if constexpr (D == 3) val[j] *= en.w;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int i = i0 + j * RU;
          if (i >= ns) break;
          slots[i * TW + part] = val[j] * scale;
        }
      }
      __syncthreads();
      // The warp's rows, RU apart (a warp near the window's edge, whose rows few samples meet, has
      // another one inside it), meet the samples of ly in [ylo, yhi), one x position at a time:
      // which sums a sample meets is fixed in each of the unrolled loops.
#pragma unroll 1
      for (int wrow = warp * RW; wrow < kSpWin; wrow += RU) {
        const int row = wrow + rsub;
        const int ylo = max(wrow - (kEsWidth - 1), 0), yhi = min(wrow + RW, kSpTile);
        // acc 2^-(ea + 25) in units of 2^-e_grid: sh > 0, as the grid resolves 2^-40 of the
        // largest term and the products 2^-54 of the tile's
        const int sh = min(max(ea + kSpTapBits - e_grid, 1), 62);
        unsigned long long s1 = 0;  // column `lane`: the x taps the warp will add 2^31 times
        if (lane < kSpWin)
          for (int y = ylo; y < yhi; ++y) s1 += csum[y * (kSpWin + 1) + lane];
        s1 <<= 31;
        unsigned long long acc[kSpWin];
#pragma unroll
        for (int c = 0; c < kSpWin; ++c) acc[c] = (1ull << (sh - 1)) - __shfl_sync(0xffffffffu, s1, c);
        const float* pv = slots + part;
        const float* py = slots + TY + min(row, kSpWin);
        const int *plo = start + ylo, *phi = start + yhi;
#pragma unroll
        for (int lx = 0; lx < kSpTile; ++lx) {
          int o = plo[lx * kSpTile] * TW;
          const int e = phi[lx * kSpTile] * TW;
#pragma unroll 2
          for (; o < e; o += TW) {
            const uint4 ta = *reinterpret_cast<const uint4*>(slots + TX + o);
            const uint4 tb = *reinterpret_cast<const uint4*>(slots + TX + 4 + o);
            const unsigned vy = (unsigned)__float2int_rn(pv[o] * py[o]) ^ 0x80000000u;  // + 2^31
            sp_mad(acc[lx + 0], vy, ta.x);
            sp_mad(acc[lx + 1], vy, ta.y);
            sp_mad(acc[lx + 2], vy, ta.z);
            sp_mad(acc[lx + 3], vy, ta.w);
            sp_mad(acc[lx + 4], vy, tb.x);
            sp_mad(acc[lx + 5], vy, tb.y);
            sp_mad(acc[lx + 6], vy, tb.z);
            sp_mad(acc[lx + 7], vy, tb.w);
          }
        }
        if (live && row < kSpWin && bd > 0.f) {
          const int64_t rowc = (int64_t)a.M0 * (wrap32(oy + row, a.M1) + (int64_t)a.M1 * (D == 3 ? wrap32(oz + z, a.M2) : 0));
          unsigned long long* g = reinterpret_cast<unsigned long long*>(a.q) + ((int64_t)grp * a.cells + rowc) * P + part;
          if (ox + kSpWin <= a.M0) {
            g += (int64_t)ox * P;
#pragma unroll
            for (int c = 0; c < kSpWin; ++c) {
              const long long qv = (long long)acc[c] >> sh;
              if (qv != 0) atomicAdd(g + c * P, (unsigned long long)qv);
            }
          } else {
            int gx = wrap32(ox, a.M0);
#pragma unroll
            for (int c = 0; c < kSpWin; ++c) {
              const long long qv = (long long)acc[c] >> sh;
              if (qv != 0) atomicAdd(g + (int64_t)gx * P, (unsigned long long)qv);
              gx = gx + 1 == a.M0 ? 0 : gx + 1;
            }
          }
        }
      }
      __syncthreads();  // the values are consumed
    }
  }
}

// Lanes a group of parts is spread with: 8 for at most 8 parts, else the wider of 16 and 32
// whose groups keep the lanes busier.  A warp with two rows (P = 16) also meets the samples
// that touch only one of them, so its lanes are worth 8 / 9 of those of P = 32.
// (The padding costs memory too: on the largest grid that the transforms take, 9685 x 3228 cells,
// 1.7 GB for one part and 3.7 GB, the most, for 17.  Cells of the live parts alone made the atomics'
// strides run-time values: 256^2, 20 coils, a backprojection 2.16 -> 2.18 ms.)
inline int spread_lanes(int nparts) {
  if (nparts <= 8) return 8;
  int best = 32;
  double cost = 1e300;
  for (int P = 32; P >= 16; P >>= 1) {
    const double c = (double)((nparts + P - 1) / P * P) * (8 + 32 / P - 1);
    if (c < cost - 1e-9) {
      cost = c;
      best = P;
    }
  }
  return best;
}

template <int P, int D, class Parts>
static int launch_spread_rows(const SpreadRowsArgs& a, const Parts& parts, cudaStream_t st) {
  constexpr int smem = kSpChunk * (P + 32 + 4) * (int)sizeof(float) + (2 * kSpTile * kSpTile + 4) * (int)sizeof(int) +
                       kSpTile * (kSpWin + 1) * (int)sizeof(long long);
  MRSR_CHECK_CUDA(cudaFuncSetAttribute(k_spread_rows<P, D, Parts>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  MRSR_CHECK_CUDA(cudaMemsetAsync(a.next, 0, sizeof(unsigned long long), st));
  k_spread_rows<P, D, Parts><<<152 * 2, kSpThreads, smem, st>>>(a, parts);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

// q: [ceil(nparts / P)][cells][P] with P = spread_lanes(nparts), zeroed
template <class Parts>
static int spread_rows(int d, const int64_t* M, int64_t cells, int nparts, long long* q, const FixedScale* fs, int* bad,
                       const TileSort& ts, const Parts& parts, cudaStream_t st) {
  MRSR_REQUIRE(ts.tile == kSpTile && ts.m0 == (int)M[0] && ts.m1 == (int)M[1] && (d == 2 || ts.m2 == (int)M[2]),
               MRSR_ERR_STATE, "tile sort built for another grid");
  MRSR_REQUIRE(ts.rec.p != nullptr, MRSR_ERR_STATE, "tile sort without tap records");
  const SpreadRowsArgs a{ts.m0, ts.m1, d == 3 ? ts.m2 : 1, cells, nparts, q, fs, bad, ts.ntx, ts.nty, ts.rec.p,
                         ts.items.as<int4>(), ts.nitems.as<int>(), ts.next.as<unsigned long long>()};
  switch (spread_lanes(nparts)) {
    case 8: return d == 3 ? launch_spread_rows<8, 3>(a, parts, st) : launch_spread_rows<8, 2>(a, parts, st);
    case 16: return d == 3 ? launch_spread_rows<16, 3>(a, parts, st) : launch_spread_rows<16, 2>(a, parts, st);
    default: return d == 3 ? launch_spread_rows<32, 3>(a, parts, st) : launch_spread_rows<32, 2>(a, parts, st);
  }
}

// [group][cell][P] accumulators -> out[channel][cell], channel = nq parts (re, and im or 0):
// 64 cells of one group per block through a shared tile, coalesced on both sides; NaN in the parts
// that are marked in `bad`.
template <int P>
__global__ void __launch_bounds__(256) k_parts_to_grid(const long long* q, int nq, int64_t cells, int nparts,
                                                       const FixedScale* fs, const int* bad, float2* out) {
  constexpr int NC = 64;
  __shared__ float tile[P][NC + 1];
  static_assert(256 % P == 0, "a thread converts one part");
  const int64_t cell0 = (int64_t)blockIdx.x * NC;
  const int grp = blockIdx.y;
  const int nc = cells - cell0 < NC ? (int)(cells - cell0) : NC;
  const long long* qg = q + ((int64_t)grp * cells + cell0) * P;
  const int part = grp * P + threadIdx.x % P;
  const float inv = part < nparts && bad[part] ? __int_as_float(0x7fc00000) : fs->inv;
  for (int e = threadIdx.x; e < nc * P; e += 256) tile[e % P][e / P] = fx_to_float(qg[e]) * inv;
  __syncthreads();
  const int ncu = min(P, nparts - grp * P) / nq;  // channels of the group
  for (int e = threadIdx.x; e < ncu * NC; e += 256) {
    const int ch = e / NC, c = e % NC;
    if (c < nc)
      out[((int64_t)grp * (P / nq) + ch) * cells + cell0 + c] = make_float2(tile[ch * nq][c], nq == 2 ? tile[ch * nq + 1][c] : 0.f);
  }
}

static int parts_to_grid(const long long* q, int nq, int64_t cells, int nparts, const FixedScale* fs, const int* bad,
                         float2* out, cudaStream_t st) {
  const int P = spread_lanes(nparts);
  const dim3 g((unsigned)cdiv(cells, 64), (unsigned)cdiv(nparts, P));
  if (P == 8)
    k_parts_to_grid<8><<<g, 256, 0, st>>>(q, nq, cells, nparts, fs, bad, out);
  else if (P == 16)
    k_parts_to_grid<16><<<g, 256, 0, st>>>(q, nq, cells, nparts, fs, bad, out);
  else
    k_parts_to_grid<32><<<g, 256, 0, st>>>(q, nq, cells, nparts, fs, bad, out);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

// Samples of a chunk: 384, fewer where 2D samples would not give every block a unit (a rule on the
// number of samples alone, as chunks decide the rounding): 32^2, 12800 samples, 160 parts, a
// backprojection 0.43 -> 0.27 ms, 8 parts 0.21 -> 0.19.
inline int spread_chunk(int d, int64_t n) {
  if (d == 3) return kSpChunk;
  return (int)std::min<int64_t>(kSpChunk, std::max<int64_t>(64, cdiv(n, 304 * 32) * 32));
}

// bytes of the accumulators of `nparts` parts
inline size_t spread_rows_bytes(int nparts, int64_t cells) {
  const int P = spread_lanes(nparts);
  return sizeof(long long) * (size_t)cells * (size_t)cdiv(nparts, P) * P;
}

}  // namespace mrsr
