// Tile-sorted 3D spreading with shared-memory windows (nufft.cu), for the part counts and grids
// where spread_rows.cuh does not pay (rows_pay).
//
// Samples in 8^3 tiles (home tile of the first tap), work items of at most kChunk samples of one
// tile x a group of kP3 = 4 parts, a window of (8 + w - 1)^3 = 15^3 cells x 4 parts of 32-bit
// limbs in shared memory (106 KB: two CTAs per SM), and one global 64-bit atomic per nonzero
// window cell at the flush, a warp on consecutive cells.  A warp takes one sample at a time:
// lane = 8 part + t1 (part < 4, x tap t1 < 8), so a warp instruction adds 8 consecutive cells of
// 4 parts, and the part stride (3384 = 24 mod 32 words) puts the four 8-cell runs in disjoint
// bank ranges: no bank conflicts.  A term enters as its two fx_split limbs, round(a) and the
// 21-bit remainder: 32-bit shared atomics run at about five times the rate of 64-bit ones, and
// the limb sums of kChunk terms cannot overflow.  Every grid cell is the exact integer sum of
// its rounded terms, whatever order the samples and items land in.
#pragma once

namespace mrsr {

static_assert(kChunk * (1ll << (kFxLoBits - 1)) < (1ll << 31), "low limb sums must fit in 31 bits");
static_assert(kChunk * (1ll << (kFxTermBits - kFxLoBits)) < (1ll << 31), "high limb sums must fit in 31 bits");
constexpr int kWin3Stride = 3384;                      // part stride, = 24 (mod 32)
constexpr int kP3 = 4;
constexpr int kWindowsSmem = 2 * kP3 * kWin3Stride * (int)sizeof(int);
static_assert(kWin3Stride >= kWin3Cells && kWin3Stride % 32 == 24 && kWin3Stride % 4 == 0, "3D window stride");

struct SpreadWindowsArgs {
  int M0, M1, M2;
  int64_t cells;
  int nparts;
  long long* q;            // [nparts][cells]
  const FixedScale* fs;
  int ntx, nty;
  const TapRec3* rec;
  const int4* items;
  const int* nitems;
  int* next;
};

template <class Parts>
__global__ void __launch_bounds__(kTiledThreads, 2) k_spread_windows(SpreadWindowsArgs a, Parts parts) {
  extern __shared__ __align__(16) int win3[];  // [2][kP3][kWin3Stride]
  int* wlo = win3;
  int* whi = win3 + kP3 * kWin3Stride;
  __shared__ int s_item;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int part = lane >> 3, t1 = lane & 7;
  const int nitems = *a.nitems;
  const int ngroups = (a.nparts + kP3 - 1) / kP3;
  const int total = nitems * ngroups;
  const float sc = a.fs->scale;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(a.next, 1);
    __syncthreads();
    const int it = s_item;
    if (it >= total) break;
    const int grp = it / nitems;
    const int4 item = a.items[it - grp * nitems];
    const int gpart = grp * kP3 + part;
    const bool live_part = gpart < a.nparts;
    const typename Parts::Lane L = parts.bind(live_part ? gpart : 0, 0);
    const int tx = item.x % a.ntx, tyz = item.x / a.ntx;
    const int ox = tx * kTile3, oy = (tyz % a.nty) * kTile3, oz = (tyz / a.nty) * kTile3;
    int4* w4 = reinterpret_cast<int4*>(win3);
    for (int i = threadIdx.x; i < 2 * kP3 * kWin3Stride / 4; i += blockDim.x) w4[i] = make_int4(0, 0, 0, 0);
    __syncthreads();
    if (live_part) {
      for (int smp = warp; smp < item.z; smp += nwarps) {
        const float4* r4 = reinterpret_cast<const float4*>(a.rec + item.y + smp);
        float wy[kEsWidth], wz[kEsWidth];
        {
          const float4 q2 = r4[2], q3 = r4[3], q4 = r4[4], q5 = r4[5];
          wy[0] = q2.x; wy[1] = q2.y; wy[2] = q2.z; wy[3] = q2.w;
          wy[4] = q3.x; wy[5] = q3.y; wy[6] = q3.z; wy[7] = q3.w;
          wz[0] = q4.x; wz[1] = q4.y; wz[2] = q4.z; wz[3] = q4.w;
          wz[4] = q5.x; wz[5] = q5.y; wz[6] = q5.z; wz[7] = q5.w;
        }
        const float wx1 = reinterpret_cast<const float*>(r4)[t1];
        const int4 ri = reinterpret_cast<const int4*>(r4)[6];  // li, t, lx0, ly0
        const int lz0 = reinterpret_cast<const int*>(r4)[28];
        const float v = parts.value(L, ri.x, ri.y) * sc * wx1;
        const int lx = ri.z - ox, ly = ri.w - oy, lz = lz0 - oz;
        if ((unsigned)lx < (unsigned)kTile3 && (unsigned)ly < (unsigned)kTile3 && (unsigned)lz < (unsigned)kTile3) {
          const int base = part * kWin3Stride + (lz * kWin3 + ly) * kWin3 + lx + t1;
          int* pl = wlo + base;
          int* ph = whi + base;
#pragma unroll
          for (int t3 = 0; t3 < kEsWidth; ++t3) {
            const float v3 = v * wz[t3];
#pragma unroll
            for (int t2 = 0; t2 < kEsWidth; ++t2) {
              int hi, lo;
              fx_split_prod(v3, wy[t2], hi, lo);
              atomicAdd(pl + (t3 * kWin3 + t2) * kWin3, lo);
              atomicAdd(ph + (t3 * kWin3 + t2) * kWin3, hi);
            }
          }
        } else {
          // the sort put the first tap in this tile (the same float arithmetic); a sample
          // outside it goes straight to the grid rather than out of the window
          long long* g = a.q + (int64_t)gpart * a.cells;
          const int64_t x = wrap32(ri.z + t1, a.M0);
          for (int t3 = 0; t3 < kEsWidth; ++t3)
            for (int t2 = 0; t2 < kEsWidth; ++t2) {
              const int64_t row = (int64_t)a.M0 * (wrap32(ri.w + t2, a.M1) + (int64_t)a.M1 * wrap32(lz0 + t3, a.M2));
              atomicAdd(reinterpret_cast<unsigned long long*>(g + row + x),
                        (unsigned long long)fx_term(v * wz[t3] * wy[t2]));
            }
        }
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kP3 * kWin3Cells; e += blockDim.x) {
      const int p = e / kWin3Cells, c = e - p * kWin3Cells;
      const int gp = grp * kP3 + p;
      if (gp >= a.nparts) continue;
      const int w = p * kWin3Stride + c;
      const long long v = (long long)whi[w] * (1ll << kFxLoBits) + (long long)wlo[w];
      if (v == 0) continue;
      const int cx = c % kWin3, cyz = c / kWin3;
      const int cy = cyz % kWin3, cz = cyz / kWin3;
      const int64_t cell = wrap32(ox + cx, a.M0) +
                           (int64_t)a.M0 * (wrap32(oy + cy, a.M1) + (int64_t)a.M1 * wrap32(oz + cz, a.M2));
      atomicAdd(reinterpret_cast<unsigned long long*>(a.q + (int64_t)gp * a.cells + cell), (unsigned long long)v);
    }
    __syncthreads();
  }
}

template <class Parts>
static int spread_windows(const int64_t* M, int64_t cells, int nparts, long long* q, const FixedScale* fs,
                          const TileSort& ts, const Parts& parts, cudaStream_t st) {
  MRSR_REQUIRE(ts.tile == kTile3 && ts.rec.p && ts.m0 == (int)M[0] && ts.m1 == (int)M[1] && ts.m2 == (int)M[2],
               MRSR_ERR_STATE, "3D tile sort built for another grid or without tap records");
  const SpreadWindowsArgs a{ts.m0, ts.m1, ts.m2, cells, nparts, q, fs, ts.ntx, ts.nty,
                            ts.rec.as<TapRec3>(), ts.items.as<int4>(), ts.nitems.as<int>(), ts.next.as<int>()};
  MRSR_CHECK_CUDA(cudaFuncSetAttribute(k_spread_windows<Parts>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWindowsSmem));
  MRSR_CHECK_CUDA(cudaMemsetAsync(a.next, 0, sizeof(int), st));
  k_spread_windows<Parts><<<152 * 2, kTiledThreads, kWindowsSmem, st>>>(a, parts);
  MRSR_LAUNCH_CHECK();
  return MRSR_OK;
}

// Whether `total` parts in batches of `parts` (a pass over the samples each) of n samples on
// `cells` cells go to spread_rows.cuh.  That kernel pays a fixed price per chunk and window plane,
// whatever the parts, and for the lanes it pads them with; this one pays per four parts.
// Measured on whole calls (here / rows, ms): kernel precompute of 64^3, 154k samples, 3 parts 2.3 / 2.8, 10
// parts 5.8 / 4.5, 15 parts 8.2 / 5.5; backprojection on 256^3 cells, 1.6M samples, 8 parts 5.5 /
// 7.3, 16 parts 10.2 / 9.0, 32 parts 19.8 / 13.4; 4.9M samples, 24 parts 27.8 / 31.9, 32 parts
// 36.7 / 32.2, 40 parts (48 lanes) 48.9 / 52.0; on 64^3 cells, 13k samples, 20 parts 0.42 / 0.48,
// 32 parts 0.51 / 0.49.  Its padded grids cost memory: over 8 GiB a batch it is not taken (kernel
// precompute of 128^3, K = 5: 89 / 114 ms).
inline bool rows_pay(int parts, int total, int64_t n, int64_t cells) {
  auto padded = [](int p) { const int P = spread_lanes(p); return p ? cdiv(p, P) * P : 0; };
  const int64_t lanes = total / parts * padded(parts) + padded(total % parts);
  if (spread_rows_bytes(parts, cells) + sizeof(long long) * (size_t)parts * cells > (8ull << 30)) return false;
  if (cells >= 1 << 19 && 10 * n <= cells) return parts >= 8.5 + 70.0 * (double)n / (double)cells;
  return parts >= 28 && 10 * lanes <= 11 * (int64_t)total;
}

}  // namespace mrsr
