// Projector kernels for sm_103a: Ax (ray-driven, one warp per ray) and Atx
// (voxel-driven, one thread per voxel), standalone and fused with the SART
// per-view update.  Compiled with -fmad=false (see projector.cuh).
//
// Atx stages the view's ray slopes in shared memory: each block first finds
// the detector window its 32x8 voxel tile projects to, computes the slopes
// of those rays once (two divisions per detector column, four per 3D ray),
// then every (voxel, bin) pair reads them instead of dividing again.
#include <algorithm>
#include <type_traits>
#include "kernels.h"
#include "projector.cuh"

namespace asd {

namespace {

constexpr int kAxWarps = 4;             // warps per Ax block
constexpr int kAtxThreads = kTileThreads;
constexpr int kTabA = 512;              // detector columns staged per block
constexpr int kTabC = 1536;             // 3D rays staged per block

__device__ __forceinline__ bool tile_voxel(const Dims &D, int &ix, int &iy,
                                           int &iz) {
  return asd::tile_voxel(D.nx, D.ny, D.nz, ix, iy, iz);
}

// Extents of an instance's volume (nx*ny*nz) and view (na*nb), for ASD_IN.
__device__ __forceinline__ long long nvox(const Dims &D) {
  return (long long)D.nx * D.ny * D.nz;
}
__device__ __forceinline__ long long nray(const Dims &D) { return (long long)D.na * D.nb; }

int atx_blocks(const Dims &d) {
  const dim3 g = tile_grid(d.nx, d.ny, d.nz, 1);
  return (int)(g.x * g.y);
}

// ------------------------------------------------------------------- Ax
// One warp per ray: lane l takes columns l, l + 32, ..., and the lanes'
// partial sums are added by the xor butterfly.  Every forward kernel sums a
// ray this way, so a ray's total does not depend on the kernel that computed
// it.  (Two warps per ray: 14 % slower for a batch of 64 and 27 % for 256^3.)
constexpr int kAxBlock = kAxWarps * 32;  // threads per block

// Ray (ia, ib) of a view.
__device__ __forceinline__ RayMarch ax_ray(const ViewGeo &G, const Dims &D, int ia, int ib,
                                           bool &planar) {
  const float zd = G.z_det[ib];
  planar = D.nz == 1 && zd == 0.0f;
  return ray_setup(G, D, G.y_det[ia], zd);
}
// This lane's partial sums of ray R over its columns (no cross-lane sum).
template <class Loader>
__device__ __forceinline__ void ax_lane_partial(const RayMarch &R, bool planar, Loader ld,
                                                float &ys, float &ss) {
  const int lane = threadIdx.x & 31;
  ys = 0.f;
  ss = 0.f;
  // fan beams: two columns of loads per round (four or eight: 5.4 and 5.7 us
  // against 4.4 a 512^2 view); single slices with detector rows: one (its
  // three pieces per column already keep loads in flight)
  if (planar)
    ray_columns_planar_fast<2>(R, lane, 32, ld, ys, ss);
  else
    ray_columns_fast<1>(R, lane, 32, ld, ys, ss);
}

// Cone beams of many rays: a warp takes kAxRows neighbouring rows of a detector
// column, whose rays share their in-plane march.  One 256^3 view of a reconstruction,
// 512^2 detector: 283 us with one row a warp, 243 with two, 227 with four,
// 243 with eight; four rows at 7 blocks per SM (72 registers instead of the
// 95 it would take; issue 77 %) 206 us, 6 blocks 208, 8 blocks 213.
constexpr int kAxRows = 4, kAxRowBlocks = 7;
// Warps of a view: (rows of kAxRows) x columns, the rows of a column first.
__host__ __device__ __forceinline__ long long ax_warps3(const Dims &d) {
  return (long long)((d.nb + kAxRows - 1) / kAxRows) * d.na;
}
// Detector column and first row of warp w (w < ax_warps3, rays < 2^31).
__device__ __forceinline__ void ax_rows(const Dims &D, long long w, int &ia, int &ib0) {
  const unsigned n = (unsigned)((D.nb + kAxRows - 1) / kAxRows);
  ia = (int)((unsigned)w / n);
  ib0 = (int)((unsigned)w % n) * kAxRows;
}
// Totals of rays (ia, ib0 + k); rows past the detector repeat its last one.
template <class Loader>
__device__ __forceinline__ void ax_rows_sum(const ViewGeo &G, const Dims &D, int ia, int ib0,
                                            Loader ld, float (&ys)[kAxRows],
                                            float (&ss)[kAxRows]) {
  const float yd = G.y_det[ia];
  RayMarch R = ray_setup(G, D, yd, G.z_det[ib0]);
  float slope2[kAxRows], lfac[kAxRows];
#pragma unroll
  for (int k = 0; k < kAxRows; k++) {
    const RayMarch Rk = ray_setup(G, D, yd, G.z_det[min(ib0 + k, D.nb - 1)]);
    slope2[k] = Rk.slope2;
    lfac[k] = Rk.lfac;
    ys[k] = ss[k] = 0.f;
  }
  ray_columns_rows<kAxRows>(R, slope2, lfac, threadIdx.x & 31, 32, ld, ys, ss);
#pragma unroll
  for (int k = 0; k < kAxRows; k++) {
    ys[k] = warp_sum(ys[k]);
    ss[k] = warp_sum(ss[k]);
  }
}

template <bool kByRows>
__global__ void __launch_bounds__(kAxBlock, kByRows ? kAxRowBlocks : 1)
    k_ax(const float *x, float *__restrict__ y, float *__restrict__ sr, ViewGeo G, Dims D) {
  pdl_enter();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long w = (long long)blockIdx.x * kAxWarps + warp;
  if (w >= (kByRows ? ax_warps3(D) : nray(D))) return;  // the whole warp
  // plain loads: the previous kernel may write x while this one waits
  auto ld = [&](unsigned i) { return ASD_IN(i, nvox(D)) ? x[i] : 0.f; };
  if constexpr (kByRows) {
    int ia, ib0;
    ax_rows(D, w, ia, ib0);
    float ys[kAxRows], ss[kAxRows];
    ax_rows_sum(G, D, ia, ib0, ld, ys, ss);
    // lane k: row ib0 + k
    float yv = ys[0], sv = ss[0];
#pragma unroll
    for (int k = 1; k < kAxRows; k++) {
      yv = lane == k ? ys[k] : yv;
      sv = lane == k ? ss[k] : sv;
    }
    if (lane < kAxRows && ib0 + lane < D.nb) {
      const long long r = (long long)(ib0 + lane) * D.na + ia;
      y[r] = yv * G.scale;
      sr[r] = sv * G.scale;
    }
  } else {
    const unsigned ru = (unsigned)w, na = (unsigned)D.na;  // rays < 2^31
    float ys, ss;
    bool planar;
    const RayMarch R = ax_ray(G, D, (int)(ru % na), (int)(ru / na), planar);
    ax_lane_partial(R, planar, ld, ys, ss);
    ys = warp_sum(ys);
    ss = warp_sum(ss);
    if (lane == 0) {
      y[w] = ys * G.scale;
      sr[w] = ss * G.scale;
    }
  }
}

// Exact forward projection (siddon_setup, siddon_columns), a warp per `rpw`
// (1 to 32) rays: lane j sets up ray j (its FP64 arithmetic once per ray, not once per
// lane: the GPU's FP64 rate is a small fraction of its FP32 rate), then the
// warp walks its rays in turn, each ray's set-up broadcast from its lane
// and its columns dealt to the lanes, summed by the butterfly; lane j keeps
// ray j's totals.
__device__ __forceinline__ DSFloat ds_shfl(DSFloat v, int src) {
  DSFloat o;
  o.hi = __shfl_sync(0xffffffffu, v.hi, src);
  o.lo = __shfl_sync(0xffffffffu, v.lo, src);
  return o;
}

__device__ __forceinline__ SidRay sid_bcast(const SidRay &R, int src) {
  SidRay o;
#pragma unroll
  for (int a = 0; a < 2; a++) {
    o.pos0[a] = ds_shfl(R.pos0[a], src);
    o.r[a] = ds_shfl(R.r[a], src);
    o.n_ax[a] = __shfl_sync(0xffffffffu, R.n_ax[a], src);
  }
  o.ua = ds_shfl(R.ua, src);
  o.ub = ds_shfl(R.ub, src);
  o.Lu = __shfl_sync(0xffffffffu, R.Lu, src);
  o.du = __shfl_sync(0xffffffffu, R.du, src);
  o.nax = __shfl_sync(0xffffffffu, R.nax, src);
  o.nu = __shfl_sync(0xffffffffu, R.nu, src);
  o.full0 = __shfl_sync(0xffffffffu, R.full0, src);
  o.full1 = __shfl_sync(0xffffffffu, R.full1, src);
  o.su = __shfl_sync(0xffffffffu, R.su, src);
  o.sv = __shfl_sync(0xffffffffu, R.sv, src);
  o.sz = __shfl_sync(0xffffffffu, R.sz, src);
  o.hit = __shfl_sync(0xffffffffu, (int)R.hit, src) != 0;
  return o;
}

// Totals of rays r0 + lane (lane < rpw, nr - r0) for the whole warp.
template <class Loader>
__device__ __forceinline__ void siddon_warp_rays(const ViewGeo &G, const Dims &D,
                                                 long long r0, long long nr, int rpw,
                                                 Loader ld, float &my_y, float &my_s) {
  const int lane = threadIdx.x & 31;
  SidRay mine;
  const DSFloat z{0.f, 0.f};
  mine.pos0[0] = mine.pos0[1] = mine.r[0] = mine.r[1] = mine.ua = mine.ub = z;
  mine.Lu = 0.f;
  mine.du = mine.nax = mine.nu = mine.n_ax[0] = mine.n_ax[1] = mine.full0 = mine.full1 = 0;
  mine.su = mine.sv = mine.sz = 0u;
  mine.hit = false;
  const long long r = r0 + lane;
  if (lane < rpw && r < nr) mine = siddon_setup(G, D, G.y_det[r % D.na], G.z_det[r / D.na]);
  const int cnt = (int)min((long long)rpw, nr - r0);
  my_y = my_s = 0.f;
  for (int j = 0; j < cnt; j++) {
    const SidRay R = sid_bcast(mine, j);
    float ys = 0.f, ss = 0.f;
    siddon_columns(R, lane, 32, ld, ys, ss);
    ys = warp_sum(ys);
    ss = warp_sum(ss);
    if (lane == j) {
      my_y = ys;
      my_s = ss;
    }
  }
}

// Rays per warp of the exact kernels for `rays` rays in a launch.  A warp's
// set-up costs the same for one ray as for 32 (the FP64 pipe: about 0.7 us of
// an SM's time), and its rays follow one another at about 0.02 us a column, so
// the best count is near the root of rays over columns: largest power of two
// with rpw^2 <= 5/8 rays / columns.  us a view with 32 rays a warp, one, and
// this rule: 512^2 and 888 bins 328, 19.6, 19.6; eight of it 340, 65, 60; 64 of
// it 409, -, 280; 48^2 x 32 on 80 x 60 64, 37, 19; 96^2 x 64 on 160 x 128 96,
// -, 51; 160^2 x 128 on 256 x 200 215, -, 144.
static int sid_rays(long long rays, const Dims &d) {
  int rpw = 32;
  while (rpw > 1 && 8LL * rpw * rpw * max(d.nx, d.ny) > 5 * rays) rpw /= 2;
  return rpw;
}
static unsigned sid_blocks(long long rays, int rpw) {
  return (unsigned)((rays + kAxWarps * rpw - 1) / (kAxWarps * rpw));
}

__global__ void __launch_bounds__(kAxBlock)
    k_ax_siddon(const float *__restrict__ x, float *__restrict__ y,
                float *__restrict__ sr, ViewGeo G, Dims D, int rpw) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long nr = (long long)D.na * D.nb;
  const long long r0 = ((long long)blockIdx.x * kAxWarps + warp) * rpw;
  if (r0 >= nr) return;  // the whole warp
  float yv, sv;
  siddon_warp_rays(G, D, r0, nr, rpw,
                   [&](unsigned i) { return ASD_IN(i, nvox(D)) ? __ldg(x + i) : 0.f; }, yv, sv);
  const long long r = r0 + lane;
  if (lane < rpw && r < nr) {
    y[r] = yv * G.scale;
    sr[r] = sv * G.scale;
  }
}

// ------------------------------------------------------------------- Atx
// Shared staging of one block: the slopes of every ray its voxels see and the
// view's values on those rays.
template <bool kPlanar>
struct AtxShared {
  static constexpr int kA = kTabA;
  static constexpr int kC = kPlanar ? kTabA : kTabC;
  float4 tabA[kA];
  float4 tabC[kPlanar ? 1 : kC];
  float ys[kC];
  int4 win[kAtxThreads / 32];       // per warp: bins and rows its voxels see
  int flags[kAtxThreads / 32];      // per warp: what its share of the rays allows
};

// Footprint sum of one voxel (Ax_cone_gpu.cu:247-269) for every thread of
// the block: each block finds the detector window of its voxel tile, stages
// the window's ray slopes and view values in shared memory, and every lane of
// a warp then walks the same number of (bin) steps -- the warp's longest
// footprint -- with the face tests evaluated branch-free, so lanes seeing
// different rays do not serialise.  Each lane walks only the bins of its
// voxel's shadow (shadow_bins / shadow_bins3, inside the reference's window);
// the bins it skips have chords of exactly 0, which add nothing unless a view
// value is not finite, so a block whose window holds NaN/inf, an
// axis-parallel ray (whose reference chord is not geometric) or detector
// coordinates off the uniform grid the shadow assumes walks the whole
// window.  Pairs are accumulated in the reference's order (ib outer, ia
// inner).  A block whose window does not fit the staging arrays (extreme
// geometry) falls back to the direct per-pair computation.
// Must be called by every thread of the block.
template <bool kPlanar, class YLoad>
__device__ __forceinline__ void atx_block_sum(const ViewGeo &G, const Dims &D,
                                              bool valid, int ix, int iy,
                                              int iz, AtxShared<kPlanar> &sh,
                                              YLoad yl, float &acc,
                                              float &accl) {
  using Sh = AtxShared<kPlanar>;
  VoxelWin w;
  w.a0 = 0;
  w.a1 = -1;
  w.b0 = 0;
  w.b1 = -1;
  constexpr int kWarps = kAtxThreads / 32;
  bool has = false;
  if (valid) {
    w = voxel_window(G, D, ix, iy, iz);
    has = w.a0 <= w.a1 && w.b0 <= w.b1;
  }
  {
    // block window: warp-reduced, one slot per warp, every thread folds them
    const int big = 0x7fffffff;
    const int a0 = __reduce_min_sync(0xffffffffu, has ? w.a0 : big);
    const int a1 = __reduce_max_sync(0xffffffffu, has ? w.a1 : -1);
    const int b0 = __reduce_min_sync(0xffffffffu, has ? w.b0 : big);
    const int b1 = __reduce_max_sync(0xffffffffu, has ? w.b1 : -1);
    if ((threadIdx.x & 31) == 0) sh.win[threadIdx.x / 32] = make_int4(a0, a1, b0, b1);
  }
  // from here on memory that the stream's previous kernel may have written (the
  // detector coordinates among it)
  pdl_enter();
  // planar kernels verify the geometry they were chosen for (z_det == 0)
  const float z0 = kPlanar ? G.z_det[0] : 0.0f;
  __syncthreads();
  int4 bw = sh.win[0];
#pragma unroll
  for (int k = 1; k < kWarps; k++) {
    const int4 o = sh.win[k];
    bw = make_int4(min(bw.x, o.x), max(bw.y, o.y), min(bw.z, o.z), max(bw.w, o.w));
  }
  const int amin = bw.x, bmin = bw.z;
  const int nA = bw.y - amin + 1, nB = bw.w - bmin + 1;
  acc = 0.f;
  accl = 0.f;
  if (bw.y < 0) return;  // no voxel of the block sees the detector
  const bool fits = nA <= Sh::kA && (long long)nA * nB <= Sh::kC;
  // narrowing to the pixel shadow needs finite view values and rays with
  // both in-plane components (an axis-parallel ray's reference chord ignores
  // one coordinate and is 1 for every voxel of the window)
  bool narrow = true;
  bool allx = true, ally = true;  // every ray of the window x- / y-dominant
  if (fits) {  // z0 is on its way meanwhile
    narrow = G.dy_det > 0.0f && (kPlanar || G.dz_det > 0.0f);
    for (int k = threadIdx.x; k < nA; k += kAtxThreads) {
      const float yd = G.y_det[amin + k];
      const float4 A = ray_tab_a(G, yd);
      narrow = narrow && A.x != 0.0f && A.y != 0.0f &&
               on_grid(yd, amin + k, D.na, G.dy_det);
      const bool xf = fabsf(A.x) > fabsf(A.y);
      allx = allx && xf;
      ally = ally && !xf;
      sh.tabA[k] = A;
    }
    for (int k = threadIdx.x; k < nA * nB; k += kAtxThreads) {
      const int r = kPlanar ? 0 : k / nA, c = kPlanar ? k : k - r * nA;
      const long long yi = (long long)(bmin + r) * D.na + amin + c;
      const float v = ASD_IN(yi, nray(D)) ? yl(yi) : 0.f;
      narrow = narrow && isfinite(v);
      sh.ys[k] = v;
    }
    if (!kPlanar)
      for (int k = threadIdx.x; k < nB; k += kAtxThreads)
        narrow = narrow && on_grid(G.z_det[bmin + k], bmin + k, D.nb, G.dz_det);
    {
      const int f = (__all_sync(0xffffffffu, narrow) ? 1 : 0) |
                    (__all_sync(0xffffffffu, allx) ? 2 : 0) |
                    (__all_sync(0xffffffffu, ally) ? 4 : 0);
      if ((threadIdx.x & 31) == 0) sh.flags[threadIdx.x / 32] = f;
    }
    __syncthreads();
    int f = sh.flags[0];
#pragma unroll
    for (int k = 1; k < kWarps; k++) f &= sh.flags[k];
    narrow = f & 1;
    allx = f & 2;
    ally = f & 4;
    if (!kPlanar) {
      for (int k = threadIdx.x; k < nA * nB; k += kAtxThreads)
        sh.tabC[k] = ray_tab_c(sh.tabA[k % nA], G.z_det[bmin + k / nA]);
      __syncthreads();
    }
  }
  if (!fits || z0 != 0.0f) {
    if (valid) voxel_backproject(G, D, w, yl, acc, accl);
    return;
  }
  const float rx = G.cos_phi * (-G.SO) - w.xc;
  const float ry = G.sin_phi * (-G.SO) - w.yc;
  const float rz = 0.0f - w.zc;
  int lo = w.a0, hi = w.a1, blo = w.b0, bhi = w.b1;
  if (narrow && has) {
    int slo, shi, tlo, thi;
    if (kPlanar ? shadow_bins(G, D, w.xc, w.yc, slo, shi)
                : shadow_bins3(G, D, w.xc, w.yc, w.zc, slo, shi, tlo, thi)) {
      lo = max(lo, slo);
      hi = min(hi, shi);
      if (!kPlanar) {
        blo = max(blo, tlo);
        bhi = min(bhi, thi);
      }
    }
  }
  const int cntA = has && lo <= hi ? hi - lo + 1 : 0;
  const int cntB = has && blo <= bhi ? bhi - blo + 1 : 0;
  const int kA = __reduce_max_sync(0xffffffffu, cntA);
  const int kB = __reduce_max_sync(0xffffffffu, cntB);
  const int a_off = lo - amin;
  if (kPlanar && narrow && (allx || ally)) {
    // common case: no axis-parallel ray and one dominant axis for the whole
    // window; the chord needs no per-ray selection
    const int j0 = has ? a_off : 0;
    for (int ka = 0; ka < kA; ka++) {
      const bool on = ka < cntA;
      const int j = on ? j0 + ka : 0;
      const float4 A = sh.tabA[j];
      const float l = allx ? chord_planar_axis<true>(A, rx, ry)
                           : chord_planar_axis<false>(A, rx, ry);
      if (on) {
        acc += l * sh.ys[j];
        accl += l;
      }
    }
    return;
  }
  for (int kb = 0; kb < kB; kb++) {
    const bool onb = kb < cntB;
    const int ib = blo + kb;
    const float c = kPlanar ? 0.0f : G.z_det[onb ? ib : bmin] - 0.0f;
    const int row = (onb ? ib - bmin : 0) * nA + a_off;
    for (int ka = 0; ka < kA; ka++) {
      const bool on = onb && ka < cntA;
      const int j = on ? row + ka : 0;
      const float4 A = sh.tabA[on ? a_off + ka : 0];
      float l;
      if (kPlanar)
        l = chord_planar_bf(A, rx, ry, G.dz);
      else
        l = chord3_bf(A, sh.tabC[j], c, rx, ry, rz, G.dz);
      if (on) {
        acc += l * sh.ys[j];
        accl += l;
      }
    }
  }
}

// Both standalone projectors are launched so that they start while the
// stream's previous kernel drains, and wait for it before they touch memory:
// 60 views of a 512^2 image, 888 detector bins, Ax then Atx of each, 0.93 ms
// with ordinary launches and 0.76 with these.  Atx's block finds its window
// with one barrier and no atomics and agrees on the stored rays with another;
// its fan-beam form is bound by latency, not by the units (1024 blocks of a
// 512^2 image): 6 blocks per SM 0.70 ms, 5 0.75, 4 without the spills 0.76,
// 7 0.88.  Detectors so fine that a tile sees more bins than the block stages go
// per pair and are bound by the units, where the spills cost: 4 blocks (256^2 on
// 8192 bins 115 us with 6, 90 with 4; 64^2 on 4096 174 and 162).
template <bool kPlanar, int kBlocks>
__global__ void __launch_bounds__(kAtxThreads, kBlocks)
    k_atx(float *__restrict__ x, const float *yv, float *__restrict__ sc, ViewGeo G, Dims D) {
  __shared__ AtxShared<kPlanar> sh;
  int ix, iy, iz;
  const bool valid = tile_voxel(D, ix, iy, iz);
  float acc, accl;
  atx_block_sum<kPlanar>(G, D, valid, ix, iy, iz, sh,
                         [&](long long i) { return ASD_IN(i, nray(D)) ? yv[i] : 0.f; },
                         acc, accl);
  if (!valid) return;
  const unsigned idx = ((unsigned)iz * D.ny + iy) * D.nx + ix;
  if (!ASD_IN(idx, nvox(D))) return;
  x[idx] = acc * G.scale;
  sc[idx] = accl * G.scale;
}

// ------------------------------------------------------------- fused SART
__device__ __forceinline__ ViewGeo view_of(const Inst &I, int view) {
  ViewGeo g = I.g;
  const float2 t = I.trig[view];
  g.cos_phi = t.x;
  g.sin_phi = t.y;
  return g;
}

// Ray slope tables of every view (Inst::tabA) and the view flags, once per
// plan: grid (ceil(na/128), nv, instances) for the largest na and nv.
__global__ void __launch_bounds__(128)
    k_view_tables(const Inst *__restrict__ insts) {
  const Inst &I = insts[blockIdx.z];
  const Dims D = I.d;
  const int view = blockIdx.y;
  if (view >= I.nv) return;
  const int ia = blockIdx.x * 128 + threadIdx.x;
  const ViewGeo G = view_of(I, view);
  int f = 0;
  if (ia < D.na) {
    const float4 A = ray_tab_a(G, G.y_det[ia]);
    I.tabA[(long long)view * D.na + ia] = A;
    const bool xf = fabsf(A.x) > fabsf(A.y);
    f = (A.x == 0.0f || A.y == 0.0f ? kViewAxisParallel : 0) |
        (xf ? 0 : kViewNotX) | (xf ? kViewNotY : 0);
  }
  f = __reduce_or_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && f) atomicOr(I.vflags + view, f);
}

// ASD_POCS_cuda.m:117-123: [proj,sumR]=Ax(m); sumR(sumR==0)=1;
// cor0=P(:,ii)-proj; dd2+=||cor0||^2; cor=cor0./sumR.
// A ray's squared residual joins its own sum (Inst::ddr), which the end of
// the sweep adds up, and a residual that is not finite marks its view
// (Scalars::cor_bad), so a forward step has no block or grid reduction: its
// warps never wait for each other.  The sinogram value and the running sum
// are loaded before the march, whose latency covers theirs.  With a ticketed
// grid reduction per view instead, ten iterations of one 512^2 / 60-view
// slice took 13.0 ms (11.1 now), four of a batch of 64 23.9 ms (22.2) and 60
// views of a 256^3 volume 69.8 ms (64.4).
struct RayOut {
  float p;    // sinogram value
  double dd;  // Inst::ddr
};
// r: the ray's index ib * na + ia
__device__ __forceinline__ float ray_value(const Inst &I, int view, long long r, long long nr) {
  const long long pi = (long long)view * nr + r;
  return ASD_IN(pi, nr * I.nv) ? sino_at(I, pi) : 0.f;
}
__device__ __forceinline__ double ray_squares(const Inst &I, long long r, long long nr) {
  return ASD_IN(r, nr) ? I.ddr[r] : 0.0;
}
__device__ __forceinline__ RayOut ray_out_load(const Inst &I, int view, long long r,
                                               long long nr) {
  return RayOut{ray_value(I, view, r, nr), ray_squares(I, r, nr)};
}
// q: where cor keeps the ray; bad: Scalars::cor_bad or GroupState::bad
__device__ __forceinline__ void ray_out_store(const Inst &I, int *bad, int view, long long r,
                                              long long q, long long nr, const RayOut &o,
                                              float yv, float srv) {
  const float c0 = o.p - yv;
  const float cr = c0 / (srv == 0.f ? 1.f : srv);
  if (!ASD_IN(r, nr) || !ASD_IN(q, nr)) return;
  I.cor[q * I.cor_stride] = cr;
  I.ddr[r] = o.dd + (double)(c0 * c0);
  if (!isfinite(cr)) *bad = view + 1;
}

// The view's slopes of ray (ia, ib) for the backward step that follows (3-D).
__device__ __forceinline__ void ray_slopes(const Inst &I, const ViewGeo &G, const Dims &D,
                                           int view, int ia, int ib, long long q) {
  if (ASD_IN(q, nray(D)))
    I.tabC[q] = ray_tab_c(I.tabA[(long long)view * D.na + ia], G.z_det[ib]);
}

// For 3D geometry also writes the view's ray slopes (Inst::tabc_mode: a
// shared table's writer does so even after its own iterations have ended).
// By rows (ax_by_rows): a warp takes kAxRows rows of a detector column (lane k
// their k-th ray's value, residual and slopes), else one ray.
template <bool k3D, bool kByRows>
__global__ void __launch_bounds__(kAxBlock, kByRows ? kAxRowBlocks : 1)
    k_sart_ax(const Inst *__restrict__ insts, int view, const int *__restrict__ zmap) {
  const Inst &I = insts[zmap ? zmap[blockIdx.z] : blockIdx.z];
  const Dims D = I.d;
  const int lane = threadIdx.x & 31;
  const long long nr = nray(D), w = (long long)blockIdx.x * kAxWarps + (threadIdx.x >> 5);
  const bool have = view < I.nv && w < (kByRows ? ax_warps3(D) : nr);  // the whole warp
  ViewGeo G;
  int ia = 0, ib = 0;  // the warp's first ray
  RayMarch R;
  bool planar = false, own = false;
  long long r = 0;  // lane's own ray
  float p = 0.f;
  bool done = true;
  const float *m = nullptr;
  // The geometry is read before the wait, and after a sweep's first view the
  // sinogram too: whatever wrote that before the run (a kernel of the caller's
  // may, through asdpocs_plan_sinogram_ptr) is the kernel that view 0 waits for.
  if (have) {
    if (!kByRows) {
      m = I.m;
      // set, if at all, by the kernels between two sweeps
      if (view > 0) done = __ldcg(&I.s->done) != 0;
    }
    G = view_of(I, view);
    if (kByRows) {
      ax_rows(D, w, ia, ib);
    } else {
      ia = (int)((unsigned)w % (unsigned)D.na);
      ib = (int)((unsigned)w / (unsigned)D.na);
      R = ax_ray(G, D, ia, ib, planar);
    }
    own = lane < (kByRows ? kAxRows : 1) && ib + lane < D.nb;
    r = (long long)(ib + lane) * D.na + ia;
    if (own && view > 0) p = ray_value(I, view, r, nr);
  }
  pdl_enter();
  if (!have) return;
  if (own && view == 0) p = ray_value(I, view, r, nr);
  if (kByRows || view == 0) done = ((volatile int *)&I.s->done)[0] != 0;
  const bool tabc = k3D && (I.tabc_mode == kTabcShared || (!done && I.tabc_mode == kTabcOwn));
  const long long q = k3D && I.rays_t ? (long long)ia * D.nb + ib + lane : r;
  if (tabc && own) ray_slopes(I, G, D, view, ia, ib + lane, q);
  if (done) return;
  const double dd = own ? ray_squares(I, r, nr) : 0.0;
  if (kByRows) m = I.m;
  auto ld = [&](unsigned i) { return ASD_IN(i, nvox(D)) ? m[i] : 0.f; };
  float yv, sv;
  if constexpr (kByRows) {
    float ys[kAxRows], ss[kAxRows];
    ax_rows_sum(G, D, ia, ib, ld, ys, ss);
    yv = ys[0];
    sv = ss[0];
#pragma unroll
    for (int k = 1; k < kAxRows; k++) {
      yv = lane == k ? ys[k] : yv;
      sv = lane == k ? ss[k] : sv;
    }
  } else {
    ax_lane_partial(R, planar, ld, yv, sv);
    yv = warp_sum(yv);
    sv = warp_sum(sv);
  }
  if (own)
    ray_out_store(I, &I.s->cor_bad, view, r, q, nr, RayOut{p, dd}, yv * G.scale, sv * G.scale);
}

// k_sart_ax with the exact projection (siddon_warp_rays): a warp per `rpw` rays,
// lane j ray j's residual and normalisation.
template <bool k3D>
__global__ void __launch_bounds__(kAxBlock)
    k_sart_ax_exact(const Inst *__restrict__ insts, int view, const int *__restrict__ zmap,
                    int rpw) {
  pdl_enter();
  const Inst &I = insts[zmap ? zmap[blockIdx.z] : blockIdx.z];
  if (view >= I.nv) return;
  const bool done = ((volatile int *)&I.s->done)[0] != 0;
  const bool tabc = k3D && (I.tabc_mode == kTabcShared || (!done && I.tabc_mode == kTabcOwn));
  if (done && !tabc) return;
  const Dims D = I.d;
  const long long nr = nray(D);
  const ViewGeo G = view_of(I, view);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long r0 = ((long long)blockIdx.x * kAxWarps + warp) * rpw, r = r0 + lane;
  const bool own = lane < rpw && r < nr;
  const int ia = (int)(r % D.na), ib = (int)(r / D.na);
  const long long q = I.rays_t ? (long long)ia * D.nb + ib : r;
  if (tabc && own) ray_slopes(I, G, D, view, ia, ib, q);
  if (done || r0 >= nr) return;  // the whole warp
  float yv = 0.f, sv = 0.f;
  const float *m = I.m;
  siddon_warp_rays(G, D, r0, nr, rpw, [&](unsigned i) { return ASD_IN(i, nvox(D)) ? m[i] : 0.f; },
                   yv, sv);
  if (own)
    ray_out_store(I, &I.s->cor_bad, view, r, q, nr, ray_out_load(I, view, r, nr), yv * G.scale,
                  sv * G.scale);
}

// Planar chord for a window whose rays share dominant axis AX (1: x, 2: y;
// no axis-parallel ray), or any ray (AX == 0).
template <int AX>
__device__ __forceinline__ float chord_sel(const float4 A, float rx, float ry,
                                           float dz) {
  if (AX == 1) return chord_planar_axis<true>(A, rx, ry);
  if (AX == 2) return chord_planar_axis<false>(A, rx, ry);
  return chord_planar_bf(A, rx, ry, dz);
}

// Backward step over this block's tile group (see k_sart_atx).
// ---------------------------------------------------------------------------
// Chord tables of 2-D plans.  The chords of the backward step depend on the
// geometry and the view only, so a plan computes every view's chords once
// (k_atx_chords; one table for instances sharing geometry and view angles,
// else one per instance) and its backward steps read them instead of
// repeating the window, shadow and face tests of find_l for every group and
// iteration.  Per view the table holds, for voxel vi = iy * nx + ix of the
// N = nx * ny voxels:
//   head[vi]         (count << 24) | first ray, 0 for no pair; and the
//                    normalisation 1 / (chord sum) (float bits)
//   pair[p * N + vi] chords of pairs 2 p and 2 p + 1 < count (rays first + k)
// in that order, (2 + chK) * N words per view (chK is even, so that heads and
// pairs are 8-byte aligned).  The pairs, their chords and
// the chord sum are those of the narrow form of the backward steps
// (sart_atx_tiles, atx_shared_voxel), in the same order and from the same
// functions, so they give the same bits with or without the table.  Views
// with an axis-parallel ray have no table (their pairs need the full
// window); the steps also keep the direct form when a residual is not
// finite (0 * inf is not 0).
// ---------------------------------------------------------------------------
constexpr int kChordMaxSlots = 32;
// chord slots a thread loads with the table header, before it knows its count
constexpr int kChordPre = 4;

__host__ __device__ __forceinline__ size_t chord_view_words(const Dims &d, int K) {
  return (size_t)(2 + K) * (size_t)d.nx * (size_t)d.ny;
}

// SART update of a voxel (ASD_POCS_cuda.m:127-131): m += beta * Atx(cor) / sumC
// and positivity, the projector's common scale cancelled: accl is the voxel's
// chord sum, acc its weighted sum.  Every backward kernel uses these two, so
// a voxel's result does not depend on the kernel.  The reciprocal is the
// hardware's (1 ulp); max.NaN keeps NaN, as m(m<0)=0 does.
__device__ __forceinline__ float sart_norm(float accl) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(accl == 0.f ? 1.f : accl));
  return r;
}
__device__ __forceinline__ float sart_update(float m, float beta, float acc, float norm) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(__fmaf_rn(beta, acc * norm, m)), "f"(0.f));
  return r;
}
// Pair of a 2-D voxel: one rounding.
__device__ __forceinline__ void pair2(float &acc, float l, float y) { acc = __fmaf_rn(l, y, acc); }

// A voxel's table entries that do not depend on its header: head and the
// first kChordPre chords.
struct ChordPre {
  int cnt, first;
  float norm;
  float l[kChordPre];  // 0 past cnt
};
__device__ __forceinline__ ChordPre chord_load(const int *__restrict__ tab, size_t N, int K,
                                               unsigned vi) {
  static_assert(kChordPre % 2 == 0, "slots are read in pairs");
  ChordPre c;
  const int2 h = __ldg((const int2 *)tab + vi);
  const float2 *__restrict__ pair = (const float2 *)(tab + 2 * N) + vi;
#pragma unroll
  for (int p = 0; p < kChordPre / 2; p++) {
    const float2 v = 2 * p < K ? __ldg(pair + (size_t)p * N) : make_float2(0.f, 0.f);
    c.l[2 * p] = v.x;
    c.l[2 * p + 1] = v.y;
  }
  c.cnt = (int)((unsigned)h.x >> 24);
  c.first = h.x & 0xffffff;
  c.norm = __int_as_float(h.y);
#pragma unroll
  for (int k = 0; k < kChordPre; k++) c.l[k] = k < c.cnt ? c.l[k] : 0.f;
  return c;
}
__device__ __forceinline__ float chord_slot(const int *__restrict__ tab, size_t N, unsigned vi,
                                            int k) {
  return __ldg((const float *)(tab + 2 * N) + chord_word(N, vi, k));
}

// Asks for the chord table of the next view (the first after the last) in the
// L2: part `part` of `parts` of it, by one thread.  The tables of all views
// come from memory each sweep where they do not fit the L2, and the step waits
// for them: one slice of 512^2 (10.5 MB a view, 629 in all) 7.3 -> 6.6 ms for ten
// iterations, 6 and 24 slices of 256^2 (9.4 and 38 MB) 2.38 -> 2.24 and 5.76 ->
// 5.63 ms.  With 84 MB a view the L2 loses lines it still needs (8 slices of
// 512^2 7.8 -> 9.1 ms), and with 94 MB in all there is nothing to fetch (1.62 ->
// 1.64 ms).  The instances of a launch are taken to be of this one's size: in an
// uneven plan each decides for itself, and asks for its own table only.
constexpr size_t kPrefetchMax = (size_t)40 << 20, kPrefetchAll = (size_t)96 << 20;
__device__ __forceinline__ void prefetch_table(const Inst &I, const Dims &D, int view,
                                               unsigned part, unsigned parts) {
  const size_t bytes = chord_view_words(D, I.chK) * sizeof(int), next = bytes * gridDim.z;
  if (next > kPrefetchMax || next * I.nv < kPrefetchAll) return;
  const char *const t = (const char *)I.chtab + (view + 1 < I.nv ? view + 1 : 0) * bytes;
  const size_t chunk = (bytes / parts + 16) & ~(size_t)15;
  const char *lo = t + part * chunk, *hi = t + min((part + 1) * chunk, bytes);
  lo = (const char *)(((uintptr_t)lo + 15) & ~(uintptr_t)15);
  hi = (const char *)((uintptr_t)hi & ~(uintptr_t)15);
  if (lo < hi)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((unsigned)(hi - lo))
                 : "memory");
}

// Backward step over this block's `tiles` tiles from the view's chord table
// (2-D, narrow form; see sart_atx_tiles).  Everything but the residuals is
// loaded before the wait for the forward step: the table entries, and the
// image, which the forward step only reads and whose last writer had completed
// before that step began.  After it the residuals of every tile go out
// together with the word that says whether they are finite: one latency.
// Pairs past a voxel's own add 0 times a residual, which is finite here.
struct TabTiles {
  ChordPre c[kTilesPerBlock];
  float m[kTilesPerBlock];  // the image
};
__device__ __forceinline__ bool tab_voxel(const Dims &D, int tiles, int t, unsigned &vi) {
  const int ix = blockIdx.x * kTileX + threadIdx.x % kTileX;
  const int iy = (blockIdx.y * tiles + t) * kTileY + threadIdx.x / kTileX;
  const bool in = t < tiles && ix < D.nx && iy < D.ny;
  vi = in ? (unsigned)iy * D.nx + ix : 0u;
  return in;
}
__device__ __forceinline__ void tab_load(const Dims &D, const int *__restrict__ tab, int K,
                                         int tiles, const float *m, TabTiles &T) {
#pragma unroll
  for (int t = 0; t < kTilesPerBlock; t++) {
    if (t >= tiles) break;
    unsigned vi;
    tab_voxel(D, tiles, t, vi);
    const size_t N = (size_t)D.nx * D.ny;
    T.c[t] = chord_load(tab, N, K, vi);
    T.m[t] = ASD_IN(vi, N) ? __ldcg(m + vi) : 0.f;
  }
}
__device__ __forceinline__ void tab_residuals(const Dims &D, int tiles, const TabTiles &T,
                                              const float *cor,
                                              float (&y)[kTilesPerBlock][kChordPre]) {
  const long long M = nray(D);
#pragma unroll
  for (int t = 0; t < kTilesPerBlock; t++)
#pragma unroll
    for (int ka = 0; ka < kChordPre; ka++) {
      const int r = t < tiles ? T.c[t].first + (ka < T.c[t].cnt ? ka : 0) : 0;
      y[t][ka] = t < tiles && ASD_IN(r, M) ? cor[r] : 0.f;
    }
}
__device__ __forceinline__ void sart_atx_tiles_tab(const Inst &I, const Dims &D,
                                                   const int *__restrict__ tab, int K,
                                                   int tiles, const TabTiles &T, float beta,
                                                   const float (&y)[kTilesPerBlock][kChordPre]) {
  float *m = I.m;
  const float *cor = I.cor;
  const size_t N = (size_t)D.nx * D.ny;
  const long long M = nray(D);
#pragma unroll
  for (int t = 0; t < kTilesPerBlock; t++) {
    if (t >= tiles) break;
    unsigned vi;
    const bool in = tab_voxel(D, tiles, t, vi);
    const ChordPre &c = T.c[t];
    float acc = 0.f;
#pragma unroll
    for (int ka = 0; ka < kChordPre; ka++) pair2(acc, c.l[ka], y[t][ka]);
    for (int ka = kChordPre; ka < c.cnt; ka++)
      if (ASD_IN(ka, K) && ASD_IN(c.first + ka, M))
        pair2(acc, chord_slot(tab, N, vi, ka), cor[c.first + ka]);
    if (in && ASD_IN(vi, N)) m[vi] = sart_update(T.m[t], beta, acc, c.norm);
  }
}

template <bool kPlanar, int AX>
__device__ __forceinline__ void sart_atx_tiles(const Inst &I, const ViewGeo &G,
                                               const Dims &D,
                                               const float4 *__restrict__ tabA,
                                               bool narrow, int tiles) {
  const float beta = I.s->beta_f;
  const bool planar_ok = !kPlanar || G.z_det[0] == 0.0f;
  float *m = I.m;
  const float *__restrict__ cor = I.cor;
  const float4 *__restrict__ tabC = I.tabC;
  const float rx0 = G.cos_phi * (-G.SO), ry0 = G.sin_phi * (-G.SO);
  for (int t = 0; t < tiles; t++) {
    int x0, y0, iz;
    if (!group_tile(D.ny, D.nz, t, x0, y0, iz, tiles)) break;
    const int ix = x0 + threadIdx.x % kTileX, iy = y0 + threadIdx.x / kTileX;
    const bool valid = ix < D.nx && iy < D.ny;
    float acc = 0.f, accl = 0.f;
    VoxelWin w;
    bool has = false;
    if (valid) {
      w = voxel_window(G, D, ix, iy, iz);
      has = w.a0 <= w.a1 && w.b0 <= w.b1;
    }
    if (!planar_ok) {
      // planar kernel on a geometry with z_det != 0: direct per-pair form
      if (valid)
        voxel_backproject(G, D, w,
                          [&](long long i) { return ASD_IN(i, nray(D)) ? cor[i] : 0.f; }, acc,
                          accl);
    } else {
      int lo = has ? w.a0 : 0, hi = has ? w.a1 : -1;
      int blo = has ? w.b0 : 0, bhi = has ? w.b1 : -1;
      if (narrow && has) {
        int slo, shi, tlo, thi;
        if (kPlanar ? shadow_bins(G, D, w.xc, w.yc, slo, shi)
                    : shadow_bins3(G, D, w.xc, w.yc, w.zc, slo, shi, tlo, thi)) {
          lo = max(lo, slo);
          hi = min(hi, shi);
          if (!kPlanar) {
            blo = max(blo, tlo);
            bhi = min(bhi, thi);
          }
        }
      }
      const int cntA = has && lo <= hi ? hi - lo + 1 : 0;
      const int cntB = has && blo <= bhi ? bhi - blo + 1 : 0;
      const int kA = __reduce_max_sync(0xffffffffu, cntA);
      const int kB =
          kPlanar ? (kA > 0 ? 1 : 0) : __reduce_max_sync(0xffffffffu, cntB);
      const float rx = rx0 - (has ? w.xc : 0.f), ry = ry0 - (has ? w.yc : 0.f);
      const float rz = 0.0f - (has ? w.zc : 0.f);
      if (kPlanar) {
        for (int kb = 0; kb < kB; kb++) {
          const bool onb = kb < cntB;
          for (int ka = 0; ka < kA; ka++) {
            const bool on = onb && ka < cntA;
            const int ia = on ? lo + ka : 0;
            const float4 A = ASD_IN(ia, D.na) ? __ldg(tabA + ia) : make_float4(1.f, 1.f, 1.f, 1.f);
            const float yv = on && ASD_IN(ia, nray(D)) ? __ldg(cor + ia) : 0.f;
            const float l = chord_sel<AX>(A, rx, ry, G.dz);
            if (on) {
              pair2(acc, l, yv);
              accl += l;
            }
          }
        }
      } else {
        // the voxel's (row, column) pairs as one sequence (rows outer, the
        // reference's order), so a warp walks its longest sequence rather
        // than its widest row times its tallest column
        const int cnt = cntA * cntB;
        const int kN = __reduce_max_sync(0xffffffffu, cnt);
        int ka = 0, ib = blo;
        for (int k = 0; k < kN; k++) {
          const bool on = k < cnt;
          const int ia = on ? lo + ka : 0, ibs = on ? ib : 0;
          const int r = ibs * D.na + ia;
          const bool ok = ASD_IN(ibs, D.nb) && ASD_IN(ia, D.na) && ASD_IN(r, nray(D));
          const float c = (ok ? __ldg(G.z_det + ibs) : 0.f) - 0.0f;
          const float4 A = ok ? __ldg(tabA + ia) : make_float4(1.f, 1.f, 1.f, 1.f);
          const float4 Cs = ok ? __ldg(tabC + r) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float yv = on && ok ? __ldg(cor + r) : 0.f;
          const float l = AX == 0 ? chord3_bf(A, Cs, c, rx, ry, rz, G.dz)
                                  : chord3_axis<AX == 1>(A, Cs, rx, ry, rz, G.dz);
          if (on) {
            acc += l * yv;
            accl += l;
          }
          if (++ka == cntA) {
            ka = 0;
            ib++;
          }
        }
      }
    }
    const unsigned idx = ((unsigned)iz * D.ny + iy) * D.nx + ix;
    if (valid && ASD_IN(idx, nvox(D)))
      m[idx] = sart_update(m[idx], beta, acc, sart_norm(accl));
  }
}

// ASD_POCS_cuda.m:125-131: [bProj,sumC]=Atx(cor); sumC(sumC==0)=1;
// m = m + beta*(bProj./sumC); m(m<0)=0.
// Reads the view's ray tables and residuals through the L1 cache, so no
// block-wide staging or barrier is needed; each lane walks its voxel's shadow
// (or, when the view does not allow narrowing, the reference's window) in
// warp-uniform steps, pairs accumulated in the reference's order.  A view
// whose rays share one dominant in-plane axis and include no axis-parallel
// ray (the instance's view flags; a block-uniform branch) uses the
// axis-specialised chord.
// Bound by latency: a chain of dependent launches for one slice, too few loads
// in flight for a batch of slices of their own geometry.  Ten iterations of one
// 512^2 slice, 60 views: 8.13 ms with the images loaded after the wait and the
// residuals tile by tile, 7.3 with both as they are now and 2 blocks per SM, 7.5
// with 4 (spills); with the next table prefetched 6.6 (96 registers; two blocks
// then leave room for the forward step's, 110 registers 6.8).  Four iterations
// of 15 slices: 16.1 ms then, now 17.7 with 2 blocks per SM, 13.9 with 3, 12.1
// with 4, 11.9 with 5 (24 slices of 256^2: 7.9, 6.4, 5.8, 6.1), so kRegs is 96
// where the launch has no more than two blocks per SM and 64, for four,
// elsewhere; two tiles a block at 5 to 8 blocks 12.7 to 13.3 ms, one 17 to 18.
template <bool kPlanar, int kRegs>
__global__ void __launch_bounds__(kAtxThreads) __maxnreg__(kRegs)
    k_sart_atx(const Inst *__restrict__ insts, int view, const int *__restrict__ zmap,
               int tiles) {
  const Inst &I = insts[zmap ? zmap[blockIdx.z] : blockIdx.z];
  const Dims D = I.d;
  const bool have =
      view < I.nv && own_block(group_grid(D.nx, D.ny, D.nz, 1, tiles)).bid >= 0;
  const int *tab = nullptr;
  TabTiles T;
  int vf = 0;
  bool done = true;
  float beta = 0.f;
  const float *cor = nullptr;
  Scalars *s = nullptr;
  if (have) {  // before the wait: what the plan or kernels before the forward step wrote
    s = I.s;
    cor = I.cor;
    done = __ldcg(&s->done) != 0;
    beta = __ldcg(&s->beta_f);
    vf = I.vflags[view];
    if (kPlanar && I.chtab && !(vf & kViewAxisParallel) && I.g.z_det[0] == 0.0f) {
      tab = I.chtab + (size_t)view * chord_view_words(D, I.chK);
      tab_load(D, tab, I.chK, tiles, I.m, T);
      if (threadIdx.x == 0) {
        const OwnBlock b = own_block(group_grid(D.nx, D.ny, D.nz, 1, tiles));
        prefetch_table(I, D, view, b.bid, b.nblocks);
      }
    }
  }
  pdl_enter();
  if (done) return;
  if (tab) {
    float y[kTilesPerBlock][kChordPre];
    tab_residuals(D, tiles, T, cor, y);
    if (s->cor_bad != view + 1) {
      sart_atx_tiles_tab(I, D, tab, I.chK, tiles, T, beta, y);
      return;
    }
  }
  const bool finite = s->cor_bad != view + 1;
  const ViewGeo G = view_of(I, view);
  const float4 *tabA = I.tabA + (long long)view * D.na;
  const bool narrow =
      !(vf & kViewAxisParallel) && finite && (!kPlanar || G.z_det[0] == 0.0f);
  if (!(vf & (kViewAxisParallel | kViewNotX)))
    sart_atx_tiles<kPlanar, 1>(I, G, D, tabA, narrow, tiles);
  else if (!(vf & (kViewAxisParallel | kViewNotY)))
    sart_atx_tiles<kPlanar, 2>(I, G, D, tabA, narrow, tiles);
  else
    sart_atx_tiles<kPlanar, 0>(I, G, D, tabA, narrow, tiles);
}

// ---------------------------------------------------------------------------
// Cone-beam backward step in voxel columns (z-column form).  The lanes of a
// warp are consecutive voxels of one (x, y) column (lanes in groups of L for
// volumes of few slices), so what does not depend on z is the same for all of
// them: the footprint window's columns and magnification, the shadow's
// columns and corner magnifications (zcol_setup) and, for each detector
// column of the shadow, the in-plane part of the x and y face tests
// (col_faces).  A block computes these once for its W columns, one lane of its
// first warp per column, then one thread per (column, detector column), and keeps
// them in shared memory.  It runs over the slices that may have pairs (zcol_seen);
// the others' sums are 0.  Each voxel then
// finds its rows (zcol_shadow, or zcol_rows where a window clips the shadow)
// and evaluates the z parts of its pairs' face tests (col_hits).  Residuals
// and slopes are stored with the rays of a detector column one after the
// other (Inst::rays_t), so the warp's reads of a detector column are
// consecutive.
//
// The pairs of up to kZcCols detector columns by kZcRows rows are unrolled.
// Most pairs hit the two in-plane faces; the others (about one pair in seven
// crosses a z face) go to a list of the warp, whose items are then dealt to
// the lanes, so that a warp runs the z faces about once per voxel and not for
// every pair.  The chords go through shared memory and are accumulated in the
// reference's order (rows outer).  Voxels with more pairs, columns with three or more
// in-plane hits and shadows wider than kZcSlots take a plain loop, views that
// do not allow narrowing (an axis-parallel ray, a residual that is not
// finite) the per-voxel form over the reference's window.
// Sums pass through a tile of W columns by L voxels, so the image is read and
// written W voxels at a time.
// Instruction issue bounds it (81 % of cycles, 837 warp instructions per 32
// voxels): 0.451 ms for one 256^3 view on a 512^2 detector (ncu), against
// 0.618 with a thread per segment of a column (k_sart_atx_zwalk), which computes
// the in-plane part once per 8 voxels and the z faces for every pair, and 0.90
// per voxel.
// Grid: x tiles of W x y x segments of `seg` slices, instances.
// ---------------------------------------------------------------------------
constexpr int kZcThreads = 256, kZcWarps = kZcThreads / 32;
constexpr int kZcSlots = 6;  // detector columns of a shadow kept
static_assert(kZcRows <= 4 && kZcCols <= 8, "a pair's bit is 4 s + kb");

template <int W>
struct ZColShared {
  float4 z[kZcSlots][W];    // n1, n2, e12, bits
  float4 pts[kZcSlots][W];  // F1, F2 in-plane points
  float4 col[W];            // rx, ry, qmin, qmax
  float tb[W];              // window magnification
  int lo[W];                // first detector column
  int count[W];             // detector columns
  int flags[W];             // kZc*
  int seen[2];              // slices [seen[0], seen[1]) may have pairs
  float2 l[kZcCols * kZcRows][kZcThreads];  // a voxel's chords and their products
  unsigned short list[kZcWarps][32 * kZcCols * kZcRows];  // a warp's z-face pairs
  float acc[32][W + 1], accl[32][W + 1];
};
constexpr int kZcOk = 1, kZcWindow = 2, kZcInside = 4, kZcSpecial = 8;

// Launch shape: columns of a block (32 or 8), lanes of a column (32 to 2) and
// slices of a block, for a launch whose rays cross `seen` of its slices.  Lanes:
// what gives the least time for those, a voxel costing a tenth more with 8 lanes
// than with 32 or 16, two thirds more with 4 and three times as much with 2
// (512^2 x 100: 0.68 ms a view with 16 lanes, 0.71 with 8, 1.02 with 4; x 24 0.18
// with 8, x 4 0.067 with 4 and 0.077 with 8).  8 columns a block (and 32 lanes)
// where 32 leave SMs without a block; slices so that a launch has about four
// blocks per resident slot.  A view of a plan, 32 columns against 8: 128^2 x 48
// 31 us and 42, x 64 37 and 44, 64^2 x 32 14 and 12.
struct ZColShape {
  int W, L, seg;
  int lsh() const { return L == 32 ? 5 : L == 16 ? 4 : L == 8 ? 3 : L == 4 ? 2 : 1; }
};
inline ZColShape zcol_shape(const Dims &d, int batch, int seg, int seen) {
  ZColShape s{32, 32, 0};
  const long long lines = (long long)d.ny * batch;
  if ((d.nx + 31) / 32 * lines * ((d.nz + 31) / 32) < 152) s.W = 8;
  // a part of the slices begins anywhere in a group of lanes
  auto cost = [&](int L) {
    const int n = seen < d.nz ? seen + L / 2 : (seen + L - 1) / L * L;
    return (long long)n * (L >= 16 ? 20 : L == 8 ? 22 : L == 4 ? 33 : 60);
  };
  for (int L : {16, 8, 4, 2})
    if (s.W == 32 && cost(L) < cost(s.L)) s.L = L;
  const int least = std::max(s.L, 8);  // slices of a block
  const int chunks = (d.nz + least - 1) / least;
  const long long tiles = (d.nx + s.W - 1) / s.W * lines;
  const long long split = std::min<long long>(chunks, (152 * 16 + tiles - 1) / tiles);
  const long long per = seg > 0 ? (seg + least - 1) / least : (chunks + split - 1) / split;
  s.seg = (int)per * least;
  return s;
}
inline dim3 zcol_grid(const Dims &d, int batch, const ZColShape &s) {
  return dim3((unsigned)((d.nx + s.W - 1) / s.W) * (unsigned)d.ny *
                  (unsigned)((d.nz + s.seg - 1) / s.seg),
              1, batch);
}

// Sums of a warp's voxels with at most kZcCols detector columns (mA of them
// in the warp) and kZcRows rows each: the lane's pairs are columns s < cA and
// rows kb < cB from ray r0 (the others read rays nearby or the padding after
// the tables, whose values are finite, and have chord 0).  (c, zc0 + zl) of
// lane `src` come from v0 + src.
template <int W>
__device__ __forceinline__ void zcol_pairs(const ViewGeo &G, const Dims &D,
                                           const float4 *__restrict__ tabC,
                                           const float *__restrict__ yt, ZColShared<W> &sh, int v0,
                                           int zc0, int lsh, int c, int r0, int mA, int cA, int cB,
                                           float rz, float hz, bool steep, float &acc,
                                           float &accl) {
  constexpr int B = kZcRows;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const unsigned below = (1u << lane) - 1u;  // lanes before this one
  const long long room = nray(D) + zcol_pad(D);
  unsigned short *const list = sh.list[warp];
  unsigned todo = 0u, bit = 1u;  // pairs that do not hit both F1 and F2: bit 4 s + kb
#pragma unroll 1
  for (int s = 0; s < mA; s++) {
    const float4 q = sh.z[s][c];
    const unsigned bits = __float_as_uint(q.w);
    const int r = r0 + s * D.nb, rows = s < cA ? cB : 0;
    const float4 *const pc = tabC + r;
    const float *const py = yt + r;
    float4 Cs[B];
    float y[B];
#pragma unroll
    for (int kb = 0; kb < B; kb++) {
      const bool in = ASD_IN(r + kb, room);
      Cs[kb] = in ? __ldg(pc + kb) : make_float4(0.f, 0.f, 0.f, 0.f);
      y[kb] = in ? __ldg(py + kb) : 0.f;
    }
#pragma unroll
    for (int kb = 0; kb < B; kb++) {
      const bool on = kb < rows;
      const ColHits h = col_hits(bits, q.x, q.y, Cs[kb], rz, hz);
      const float e2 = h.z2 - h.z1, l2 = q.z + e2 * e2;
      const bool both = on && h.h1 && h.h2 && l2 >= kRootMin;
      const float l = both ? root_rn(l2) : 0.f;
      sh.l[kb * mA + s][t] = make_float2(l, l * y[kb]);
      todo |= on && !both && (steep || h.h1 || h.h2) ? bit << kb : 0u;
    }
    bit <<= 4;
  }
  // the other pairs into the warp's list, a lane's next one at a time
  int listed = 0;
  unsigned vote;
  while ((vote = __ballot_sync(0xffffffffu, todo != 0u)) != 0u) {
    if (todo) {
      list[listed + __popc(vote & below)] = (unsigned short)(lane | (__ffs((int)todo) - 1) << 5);
      todo &= todo - 1u;
    }
    listed += __popc(vote);
  }
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i - lane < listed; i += 32) {
    const int code = i < listed ? list[i] : 0, src = code & 31, k = code >> 5;
    const int rs = __shfl_sync(0xffffffffu, r0, src);
    if (i >= listed) continue;
    const int s = k >> 2, kb = k & 3, vs = v0 + src, cs = vs >> lsh;
    const int r = rs + s * D.nb + kb;
    if (!ASD_IN(r, nray(D))) continue;
    const float zr = 0.0f - zcol_height(G, D, zc0 + (vs & ((1 << lsh) - 1)));
    const float4 q = sh.z[s][cs], p = sh.col[cs], Cs = __ldg(tabC + r);
    const float yv = __ldg(yt + r);
    const ColHits h = col_hits(__float_as_uint(q.w), q.x, q.y, Cs, zr, hz);
    const float e2 = h.z2 - h.z1;
    const float l2 = h.h1 && h.h2 ? q.z + e2 * e2
                                  : chord3_zface2(sh.pts[s][cs], h, Cs, p.x, p.y, zr, hz);
    const float l = l2 > 0.f ? sqrtf(l2) : 0.f;
    sh.l[kb * mA + s][warp * 32 + src] = make_float2(l, l * yv);
  }
  __syncwarp();
  // rows outer, columns inner; 0 for a pair that is not there
  const float2 *p = &sh.l[0][t];
#pragma unroll 1
  for (int k = 0; k < mA; k++, p += B * kZcThreads)
#pragma unroll
    for (int j = 0; j < B; j++) {
      acc += p[j * kZcThreads].y;
      accl += p[j * kZcThreads].x;
    }
}

// Footprint sums of this block's columns; out(idx, acc, accl, was) takes a
// voxel's, was = old(idx) loaded before the block waits for its
// sums.  Every thread of the
// block calls it.
template <int W, class Old, class Out>
__device__ __forceinline__ void atx_zcol_walk(const ViewGeo &G, const Dims &D,
                                              const float4 *__restrict__ tabA,
                                              const float4 *__restrict__ tabC,
                                              const float *__restrict__ yt, bool narrow, int lsh,
                                              int seg, ZColShared<W> &sh, Old old, Out out) {
  const int L = 1 << lsh;
  const int xt = (D.nx + W - 1) / W, ns = (D.nz + seg - 1) / seg;
  if ((long long)blockIdx.x >= (long long)xt * D.ny * ns) return;
  const int x0 = (int)(blockIdx.x % xt) * W, iy = (int)(blockIdx.x / xt % D.ny);
  const int zb0 = (int)(blockIdx.x / xt / D.ny) * seg, zb1 = min(zb0 + seg, D.nz);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const float hz = G.dz / 2.0f;
  const long long M = nray(D);
  int za = zb0, zb = zb1;  // the slices that may have pairs
  if (narrow) {
    if (t < 32) {  // the columns' set-up, and their slices
      int s0 = zb1, s1 = zb0;
      if (t < W) {
        ZCol col;
        int cnt = 0, flags = kZcInside;
        col.rx = col.ry = col.qmin = col.qmax = col.tb = 0.f;
        if (x0 + t < D.nx) {
          col = zcol_setup(G, D, x0 + t, iy, true);
          cnt = zcol_count(col);
          flags = (col.ok ? kZcOk : 0) | (col.a0 <= col.a1 ? kZcWindow : 0) |
                  (zcol_shadow_inside(G, D, col, zb0, zb1) ? kZcInside : 0) |
                  (cnt > kZcSlots ? kZcSpecial : 0);
          if (cnt > 0) {
            zcol_seen(G, D, col, s0, s1);
            s0 = max(s0, zb0);
            s1 = min(s1, zb1);
          }
        }
        sh.col[t] = make_float4(col.rx, col.ry, col.qmin, col.qmax);
        sh.tb[t] = col.tb;
        sh.flags[t] = flags;
        sh.lo[t] = zcol_first(col, cnt);
        sh.count[t] = cnt;
      }
      s0 = __reduce_min_sync(0xffffffffu, s0);
      s1 = __reduce_max_sync(0xffffffffu, s1);
      if (t == 0) {
        sh.seen[0] = min(s0, s1);
        sh.seen[1] = s1;
      }
    }
    __syncthreads();
    za = sh.seen[0];
    zb = sh.seen[1];
    if (za < zb) {
      const int c = t % W, cnt = sh.count[c], lo = sh.lo[c];
      const float4 cd = sh.col[c];
      for (int k = t / W; k < min(cnt, kZcSlots); k += kZcThreads / W) {
        if (!ASD_IN(lo + k, D.na)) continue;
        const ColFaces f = col_faces(__ldg(tabA + lo + k), cd.x, cd.y);
        sh.pts[k][c] = make_float4(f.p1x, f.p1y, f.p2x, f.p2y);
        sh.z[k][c] = make_float4(f.n1, f.n2, f.e12, __uint_as_float(f.bits));
        if (f.bits & kCfMany) atomicOr(&sh.flags[c], kZcSpecial);
      }
      __syncthreads();
    }
  }
  // the others' sums are 0
  const int below = za - zb0, rest = below + (zb1 - zb);
  for (int v = t; v < rest * W; v += kZcThreads) {
    const int vz = v / W < below ? zb0 + v / W : zb + (v / W - below), vx = x0 + v % W;
    const unsigned idx = ((unsigned)vz * D.ny + iy) * D.nx + vx;
    if (vx < D.nx && ASD_IN(idx, nvox(D))) out(idx, 0.f, 0.f, old(idx));
  }
  // both z faces of a voxel can be hit, and so count without an in-plane
  // face, only if a ray climbs dz within a pixel; less than half of that
  // anywhere on the detector and the question never comes up
  const bool steep = !(D.nb * G.dz_det < G.dz * G.SD);
  const int zl = lane & (L - 1);
  for (int zc0 = za; zc0 < zb; zc0 += L) {
    // this thread's voxels of the chunk: every kZcThreads-th
    constexpr int kMine = W * 32 / kZcThreads;
    auto voxel = [&](int i, unsigned &idx) {
      const int v = t + i * kZcThreads, vz = zc0 + v / W, vx = x0 + v % W;
      idx = ((unsigned)vz * D.ny + iy) * D.nx + vx;
      return v < W * L && vx < D.nx && vz < zb && ASD_IN(idx, nvox(D));
    };
    // what depends on the lane's height only
    const int iz = zc0 + zl;
    const float zc = zcol_height(G, D, iz), rz = 0.0f - zc;
    float zlo, zhi;
    zcol_faces(G, zc, zlo, zhi);
    for (int v0 = warp * 32; v0 < W * L; v0 += kZcThreads) {  // warp-uniform
      const int c = (v0 + lane) >> lsh;
      const int ix = x0 + c;
      const bool valid = ix < D.nx && iz < zb;
      float acc = 0.f, accl = 0.f;
      if (!narrow) {
        // the per-voxel form over the reference's window
        if (valid) {
          const VoxelWin w = voxel_window(G, D, ix, iy, iz);
          const float rx = G.cos_phi * (-G.SO) - w.xc, ry = G.sin_phi * (-G.SO) - w.yc;
          for (int ib = w.b0; ib <= w.b1; ib++) {
            const float cz = (ASD_IN(ib, D.nb) ? __ldg(G.z_det + ib) : 0.f) - 0.0f;
            for (int ia = w.a0; ia <= w.a1; ia++) {
              const int r = ia * D.nb + ib;
              if (!(ASD_IN(ia, D.na) && ASD_IN(r, M))) continue;
              const float l =
                  chord3_bf(__ldg(tabA + ia), __ldg(tabC + r), cz, rx, ry, rz, G.dz);
              acc += l * __ldg(yt + r);
              accl += l;
            }
          }
        }
      } else {
        const float4 cd = sh.col[c];  // rx, ry, qmin, qmax
        const int flags = sh.flags[c];
        int blo, bhi;
        if (any_lane(!(flags & kZcInside))) {
          float zr;
          ZCol col;
          col.qmin = cd.z;
          col.qmax = cd.w;
          col.tb = sh.tb[c];
          col.ok = flags & kZcOk;
          col.a0 = 0;
          col.a1 = (flags & kZcWindow) ? 0 : -1;
          if (!zcol_rows(G, D, col, iz, zr, blo, bhi)) bhi = blo - 1;
        } else {
          float s0, s1;
          zcol_shadow(D, cd.z, cd.w, zlo, zhi, s0, s1);
          blo = max((int)ceilf(s0), 0);
          bhi = min((int)floorf(s1), D.nb - 1);
        }
        const int cB = valid && blo <= bhi ? bhi - blo + 1 : 0;
        const int cA = cB > 0 ? sh.count[c] : 0;
        const int mA = __reduce_max_sync(0xffffffffu, cA);
        const int mB = __reduce_max_sync(0xffffffffu, cA > 0 ? cB : 0);
        const int lo = sh.lo[c];
        const int r0 = zcol_first_ray(D, lo, blo);
        const bool special = cA > 0 && (flags & kZcSpecial);
        if (mA <= kZcCols && mB <= kZcRows && !any_lane(special)) {
          zcol_pairs<W>(G, D, tabC, yt, sh, v0, zc0, lsh, c, r0, mA, cA, cB, rz, hz, steep, acc,
                        accl);
        } else {
          for (int kb = 0; kb < cB; kb++)
            for (int s = 0; s < cA; s++) {
              const int r = r0 + s * D.nb + kb;
              if (!ASD_IN(r, M) || !ASD_IN(lo + s, D.na)) continue;
              const float4 Cs = __ldg(tabC + r);
              float l;
              if (flags & kZcSpecial) {
                l = chord3_bf(__ldg(tabA + lo + s), Cs, 0.0f, cd.x, cd.y, rz, G.dz);
              } else {
                const float4 q = sh.z[s][c], p = sh.pts[s][c];
                const ColFaces f{p.x, p.y, p.z, p.w, q.x, q.y, q.z, __float_as_uint(q.w)};
                l = chord3_col(f, Cs, cd.x, cd.y, rz, hz);
              }
              acc += l * __ldg(yt + r);
              accl += l;
            }
        }
      }
      sh.acc[zl][c] = acc;
      sh.accl[zl][c] = accl;
    }
    float was[kMine];
#pragma unroll
    for (int i = 0; i < kMine; i++) {
      unsigned idx;
      was[i] = voxel(i, idx) ? old(idx) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kMine; i++) {
      unsigned idx;
      const int v = t + i * kZcThreads;
      if (voxel(i, idx)) out(idx, sh.acc[v / W][v % W], sh.accl[v / W][v % W], was[i]);
    }
    __syncthreads();
  }
}

// SART backward step of cone-beam instances (see k_sart_atx) in z columns.
template <int W>
__global__ void __launch_bounds__(kZcThreads, 4)
    k_sart_atx_zcol(const Inst *__restrict__ insts, int view, int lsh, int seg,
                    const int *__restrict__ zmap) {
  __shared__ ZColShared<W> sh;
  pdl_enter();
  const Inst &I = insts[zmap ? zmap[blockIdx.z] : blockIdx.z];
  if (view >= I.nv || ((volatile int *)&I.s->done)[0]) return;
  const Dims D = I.d;
  const ViewGeo G = view_of(I, view);
  const bool narrow = !(I.vflags[view] & kViewAxisParallel) && I.s->cor_bad != view + 1;
  const float beta = I.s->beta_f;
  float *m = I.m;
  atx_zcol_walk<W>(G, D, I.tabA + (long long)view * D.na, I.tabC, I.cor, narrow, lsh, seg, sh,
                   [&](unsigned idx) { return m[idx]; },
                   [&](unsigned idx, float acc, float accl, float was) {
                     m[idx] = sart_update(was, beta, acc, sart_norm(accl));
                   });
}

// ---------------------------------------------------------------------------
// The same step with a thread per segment of a voxel column, walked down z, the
// 32 lanes of a warp neighbours along x (Inst::rays_t 0).  What does not depend on
// z is computed by every thread for its segment, in shared memory slots of its
// own, so no barrier is needed.  It is the better form of volumes of which a view
// crosses few slices (cone_form).  Pairs run as one sequence per voxel, rows
// outer, a warp walking its longest.
// Grid: x tiles of 32, y tiles of 8 x segments of `seg` slices, instances.
// ---------------------------------------------------------------------------
struct ZWalkShared {
  float4 pts[kZcSlots][kAtxThreads];  // F1, F2 in-plane points
  float4 z[kZcSlots][kAtxThreads];    // n1, n2, e12, bits
};
static_assert(sizeof(ZWalkShared) <= 48 << 10, "static shared memory");
// The longest of 32, 16, 8 and 4 slices that gives the launch 2^21 threads.
inline int zwalk_seg(long long voxels) {
  int seg = 32;
  while (seg > 4 && voxels / seg < (1LL << 21)) seg /= 2;
  return seg;
}

__global__ void __launch_bounds__(kAtxThreads, 4)
    k_sart_atx_zwalk(const Inst *__restrict__ insts, int view, int seg,
                     const int *__restrict__ zmap) {
  __shared__ ZWalkShared sh;
  pdl_enter();
  const Inst &I = insts[zmap ? zmap[blockIdx.z] : blockIdx.z];
  if (view >= I.nv || ((volatile int *)&I.s->done)[0]) return;
  const Dims D = I.d;
  const int ty = (D.ny + kTileY - 1) / kTileY, sg = blockIdx.y / ty;
  if ((int)blockIdx.x * kTileX >= D.nx || sg * seg >= D.nz) return;
  const ViewGeo G = view_of(I, view);
  const float4 *__restrict__ tabA = I.tabA + (long long)view * D.na;
  const float4 *__restrict__ tabC = I.tabC;
  const float *__restrict__ cor = I.cor;
  float *m = I.m;
  const bool narrow = !(I.vflags[view] & kViewAxisParallel) && I.s->cor_bad != view + 1;
  const float beta = I.s->beta_f, hz = G.dz / 2.0f;
  const int t = threadIdx.x;
  const int ix = blockIdx.x * kTileX + t % kTileX;
  const int iy = (blockIdx.y - sg * ty) * kTileY + t / kTileX;
  const int z0 = sg * seg, z1 = min(z0 + seg, D.nz);
  const bool valid = ix < D.nx && iy < D.ny;
  ZCol col;
  int cA = 0;
  col.lo = 0;
  col.rx = col.ry = 0.f;
  if (valid && narrow) {
    col = zcol_setup(G, D, ix, iy, true);
    cA = zcol_count(col);
    for (int k = 0; k < cA && cA <= kZcSlots; k++) {
      if (!ASD_IN(col.lo + k, D.na)) continue;
      const ColFaces f = col_faces(__ldg(tabA + col.lo + k), col.rx, col.ry);
      sh.pts[k][t] = make_float4(f.p1x, f.p1y, f.p2x, f.p2y);
      sh.z[k][t] = make_float4(f.n1, f.n2, f.e12, __uint_as_float(f.bits));
    }
  }
  for (int iz = z0; iz < z1; iz++) {
    const unsigned idx = ((unsigned)iz * D.ny + iy) * D.nx + ix;
    const bool in = valid && ASD_IN(idx, nvox(D));
    const float was = in ? m[idx] : 0.f;
    float acc = 0.f, accl = 0.f;
    if (!narrow) {
      // the per-voxel form over the reference's window
      if (in) {
        const VoxelWin w = voxel_window(G, D, ix, iy, iz);
        const float rx = G.cos_phi * (-G.SO) - w.xc, ry = G.sin_phi * (-G.SO) - w.yc;
        for (int ib = w.b0; ib <= w.b1; ib++)
          for (int ia = w.a0; ia <= w.a1; ia++) {
            const long long r = (long long)ib * D.na + ia;
            if (!(ASD_IN(ia, D.na) && ASD_IN(ib, D.nb))) continue;
            const float l = chord3_bf(__ldg(tabA + ia), __ldg(tabC + r), __ldg(G.z_det + ib) - 0.0f,
                                      rx, ry, 0.0f - w.zc, G.dz);
            acc += l * __ldg(cor + r);
            accl += l;
          }
      }
    } else {
      float zc = 0.f;
      int blo = 0, bhi = -1;
      const bool has = valid && zcol_rows(G, D, col, iz, zc, blo, bhi);
      const int cnt = has && blo <= bhi ? cA * (bhi - blo + 1) : 0;
      const int most = __reduce_max_sync(0xffffffffu, cnt);
      const float rz = 0.0f - zc;
      int ka = 0, ib = blo;
      for (int k = 0; k < most; k++) {
        const bool on = k < cnt;
        const int ia = on ? col.lo + ka : 0, r = (on ? ib : 0) * D.na + ia;
        if (!(ASD_IN(r, nray(D)) && ASD_IN(ia, D.na))) continue;
        const float4 Cs = __ldg(tabC + r);
        const float4 p = sh.pts[on ? min(ka, kZcSlots - 1) : 0][t];
        const float4 q = sh.z[on ? min(ka, kZcSlots - 1) : 0][t];
        const ColFaces f{p.x, p.y, p.z, p.w, q.x, q.y, q.z, __float_as_uint(q.w)};
        const float l = cA > kZcSlots || (f.bits & kCfMany)
                            ? chord3_bf(__ldg(tabA + ia), Cs, 0.0f, col.rx, col.ry, rz, G.dz)
                            : chord3_col(f, Cs, col.rx, col.ry, rz, hz);
        const float y = __ldg(cor + r);
        if (on) {
          acc += l * y;
          accl += l;
        }
        if (++ka == cA) {
          ka = 0;
          ib++;
        }
      }
    }
    if (in) m[idx] = sart_update(was, beta, acc, sart_norm(accl));
  }
}

// Ray tables of one view for the standalone backward step (launcher path), in
// the z-column step's ray order (ia * nb + ib): tabA[na], tabC[na*nb], the
// view's values yt[na*nb] and, in flag[0], whether the view forbids narrowing
// (flag[0] set unless every ray has both in-plane components, the bins lie
// on the uniform grid and every value is finite; flag[0] must be 0 before
// the launch).
__global__ void __launch_bounds__(256)
    k_view_tab3(const float *__restrict__ yv, float4 *tabA, float4 *tabC, float *yt, int *flag,
                ViewGeo G, Dims D) {
  const long long nr = (long long)D.na * D.nb;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  bool ok = true;
  if (q >= nr && q < nr + zcol_pad(D)) {
    tabC[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    yt[q] = 0.f;
  }
  if (q < nr) {
    const int ia = (int)(q / D.nb), ib = (int)(q % D.nb);
    const long long r = (long long)ib * D.na + ia;
    const float yd = G.y_det[ia], zd = G.z_det[ib];
    const float4 A = ray_tab_a(G, yd);
    if (ib == 0 && ASD_IN(ia, D.na)) tabA[ia] = A;
    const float v = ASD_IN(r, nr) ? yv[r] : 0.f;
    if (ASD_IN(q, nr)) {
      tabC[q] = ray_tab_c(A, zd);
      yt[q] = v;
    }
    ok = A.x != 0.0f && A.y != 0.0f && on_grid(yd, ia, D.na, G.dy_det) &&
         on_grid(zd, ib, D.nb, G.dz_det) && isfinite(v) && G.dy_det > 0.0f && G.dz_det > 0.0f;
  }
  if (!__all_sync(0xffffffffu, ok) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// Standalone cone-beam backward step (Ax_cone_gpu.cu:214-271) in z columns,
// from the tables of k_view_tab3.
template <int W>
__global__ void __launch_bounds__(kZcThreads, 4)
    k_atx_zcol(float *__restrict__ x, float *__restrict__ sc, const float4 *__restrict__ tabA,
               const float4 *__restrict__ tabC, const float *__restrict__ yt,
               const int *__restrict__ flag, ViewGeo G, Dims D, int lsh, int seg) {
  __shared__ ZColShared<W> sh;
  atx_zcol_walk<W>(G, D, tabA, tabC, yt, flag[0] == 0, lsh, seg, sh,
                   [](unsigned) { return 0.f; },
                   [&](unsigned idx, float acc, float accl, float) {
                     x[idx] = acc * G.scale;
                     sc[idx] = accl * G.scale;
                   });
}

// ---------------------------------------------------------------------------
// Shared-geometry backward step: when every instance of a plan has the same
// geometry and view angles, the chords of a (voxel, bin) pair are the same
// for all of them.  A block then handles one voxel tile for a group of
// kShareGroup instances: each lane computes the chords of its voxel's pairs
// once (kPairChunk at a time) and applies them to every instance of the
// group -- the backprojection becomes a sparse-matrix by dense-matrix
// product over the group.  Each instance accumulates its pairs in the
// reference's order, so the result is bit-identical to k_sart_atx.
// ---------------------------------------------------------------------------
constexpr int kShareGroup = kShareSlots;
// chords per round of the shared backward step's pair loop (1: 3 % faster
// than 2 for cone-beam groups, the same for fan beams)
constexpr int kPairChunk = 1;

// SART update of one voxel for the group's running instances (sart_update):
// m4 the group's images at the voxel, acc[b] slot b's weighted sum.
__device__ __forceinline__ void atx_shared_apply(float norm, const float *acc,
                                                 const GroupState &gs, unsigned active,
                                                 const float4 (&m4)[kShareGroup / 4],
                                                 float4 *mg) {
#pragma unroll
  for (int q = 0; q < kShareGroup / 4; q++) {
    if (!((active >> (4 * q)) & 0xFu)) continue;
    const float4 b4 = __ldg((const float4 *)gs.beta + q);
    float4 v = m4[q];
    const float *be = &b4.x;
    float *mv = &v.x;
#pragma unroll
    for (int j = 0; j < 4; j++)
      if ((active >> (4 * q + j)) & 1u) mv[j] = sart_update(mv[j], be[j], acc[4 * q + j], norm);
    mg[q] = v;
  }
}

// The voxel of this thread for the group (see k_sart_atx_shared).
template <bool kPlanar, int AX>
__device__ __forceinline__ void atx_shared_voxel(
    const ViewGeo &G, const Dims &D, const float4 *__restrict__ corg,
    const float4 *__restrict__ tabA, const float4 *__restrict__ tabC,
    bool planar_ok, bool narrow, const GroupState &gs, unsigned active, float *m_il) {
  int ix, iy, iz;
  const bool valid = tile_voxel(D, ix, iy, iz);
  VoxelWin w;
  bool has = false;
  if (valid) {
    w = voxel_window(G, D, ix, iy, iz);
    has = w.a0 <= w.a1 && w.b0 <= w.b1;
  }
  float acc[kShareGroup];
#pragma unroll
  for (int b = 0; b < kShareGroup; b++) acc[b] = 0.f;
  float accl = 0.f;
  if (!planar_ok) {
    // planar kernel on a geometry with z_det != 0: direct per-pair form
    if (valid) {
      const float xs = G.cos_phi * (-G.SO), ys0 = G.sin_phi * (-G.SO);
      for (int ib = w.b0; ib <= w.b1; ib++)
        for (int ia = w.a0; ia <= w.a1; ia++) {
          const float yd_ = G.y_det[ia];
          const float l = chord3(xs, ys0, 0.0f, G.cos_phi * G.OD - G.sin_phi * yd_,
                                 G.sin_phi * G.OD + G.cos_phi * yd_, G.z_det[ib],
                                 G.dz, w.xc, w.yc, w.zc);
          accl += l;
          const long long r = (long long)ib * D.na + ia;
#pragma unroll
          for (int q = 0; q < kShareGroup / 4; q++) {
            if (!((active >> (4 * q)) & 0xFu)) continue;
            const float4 c4 = ASD_IN(r, nray(D)) ? __ldg(corg + r * (kShareGroup / 4) + q)
                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
            acc[4 * q] += l * c4.x;
            acc[4 * q + 1] += l * c4.y;
            acc[4 * q + 2] += l * c4.z;
            acc[4 * q + 3] += l * c4.w;
          }
        }
    }
  } else {
    int lo = has ? w.a0 : 0, hi = has ? w.a1 : -1;
    int blo = has ? w.b0 : 0, bhi = has ? w.b1 : -1;
    if (narrow && has) {
      int slo, shi, tlo, thi;
      if (kPlanar ? shadow_bins(G, D, w.xc, w.yc, slo, shi)
                  : shadow_bins3(G, D, w.xc, w.yc, w.zc, slo, shi, tlo, thi)) {
        lo = max(lo, slo);
        hi = min(hi, shi);
        if (!kPlanar) {
          blo = max(blo, tlo);
          bhi = min(bhi, thi);
        }
      }
    }
    const int cntA = has && lo <= hi ? hi - lo + 1 : 0;
    const int cntB = has && blo <= bhi ? bhi - blo + 1 : 0;
    const int kA = __reduce_max_sync(0xffffffffu, cntA);
    const int kB =
        kPlanar ? (kA > 0 ? 1 : 0) : __reduce_max_sync(0xffffffffu, cntB);
    const float rx = G.cos_phi * (-G.SO) - (has ? w.xc : 0.f);
    const float ry = G.sin_phi * (-G.SO) - (has ? w.yc : 0.f);
    const float rz = 0.0f - (has ? w.zc : 0.f);
    for (int kb = 0; kb < kB; kb++) {
      const bool onb = kb < cntB;
      const int ib = blo + kb;
      const float c =
          kPlanar ? 0.0f : ((onb && ASD_IN(ib, D.nb)) ? __ldg(G.z_det + ib) : 1.0f) - 0.0f;
      const int row = onb ? ib * D.na : 0;
      for (int c0 = 0; c0 < kA; c0 += kPairChunk) {
        float l[kPairChunk];
        int idx[kPairChunk];
        bool on[kPairChunk];
#pragma unroll
        for (int j = 0; j < kPairChunk; j++) {
          const int ka = c0 + j;
          on[j] = onb && ka < cntA;
          const int ia = on[j] ? lo + ka : 0;
          idx[j] = row + ia;
          l[j] = 0.f;
          if (ka < kA) {  // warp-uniform
            const bool okr = ASD_IN(ia, D.na) && ASD_IN(row + ia, nray(D));
            const float4 A = okr ? __ldg(tabA + ia) : make_float4(1.f, 1.f, 1.f, 1.f);
            if (kPlanar)
              l[j] = chord_sel<AX>(A, rx, ry, G.dz);
            else if (AX == 0)
              l[j] = okr ? chord3_bf(A, __ldg(tabC + row + ia), c, rx, ry, rz, G.dz) : 0.f;
            else
              l[j] = okr ? chord3_axis<AX == 1>(A, __ldg(tabC + row + ia), rx, ry, rz, G.dz)
                         : 0.f;
          }
          if (on[j]) accl += l[j];
        }
#pragma unroll
        for (int j = 0; j < kPairChunk; j++) {
          if (on[j]) {
#pragma unroll
            for (int q = 0; q < kShareGroup / 4; q++) {
              // quads of the group with no running instance are skipped
              // (block-uniform); their accumulators are never read
              if (!((active >> (4 * q)) & 0xFu)) continue;
              const float4 c4 = ASD_IN(idx[j], nray(D))
                                    ? __ldg(corg + (long long)idx[j] * (kShareGroup / 4) + q)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
              const float *cv = &c4.x;
#pragma unroll
              for (int b = 0; b < 4; b++) {
                if (kPlanar)
                  pair2(acc[4 * q + b], l[j], cv[b]);
                else
                  acc[4 * q + b] += l[j] * cv[b];
              }
            }
          }
        }
      }
    }
  }
  if (!valid) return;
  const unsigned vi = ((unsigned)iz * D.ny + iy) * D.nx + ix;
  if (!ASD_IN(vi, nvox(D))) return;
  float4 *mg = (float4 *)m_il + (size_t)vi * (kShareGroup / 4);
  float4 m4[kShareGroup / 4];
#pragma unroll
  for (int q = 0; q < kShareGroup / 4; q++) m4[q] = mg[q];
  atx_shared_apply(sart_norm(accl), acc, gs, active, m4, mg);
}

// Pairs of this voxel: the reference's window narrowed to the voxel's shadow.
template <int AX>
__device__ __forceinline__ void chords_voxel(const ViewGeo &G, const Dims &D,
                                             const float4 *__restrict__ tabA,
                                             bool valid, int ix, int iy, int K,
                                             int *tab, int *kmax) {
  const VoxelWin w = voxel_window(G, D, ix, iy, 0);
  const bool has = valid && w.a0 <= w.a1 && w.b0 <= w.b1;
  int lo = has ? w.a0 : 0, hi = has ? w.a1 : -1;
  if (has) {
    int slo, shi;
    if (shadow_bins(G, D, w.xc, w.yc, slo, shi)) {
      lo = max(lo, slo);
      hi = min(hi, shi);
    }
  }
  const int cnt = has && lo <= hi ? hi - lo + 1 : 0;
  if (K == 0) {  // counting pass
    const int m = __reduce_max_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(kmax, m);
    return;
  }
  if (!valid) return;
  const size_t N = (size_t)D.nx * D.ny, vi = (size_t)iy * D.nx + ix;
  if (cnt > K) {  // cannot happen after the counting pass; the host drops the table
    atomicOr(kmax + 1, 1);
    return;
  }
  const float rx = G.cos_phi * (-G.SO) - w.xc;
  const float ry = G.sin_phi * (-G.SO) - w.yc;
  if (!ASD_IN(vi, N)) return;
  float accl = 0.f;
  for (int ka = 0; ka < cnt; ka++) {
    if (!(ASD_IN(lo + ka, D.na) && ASD_IN(ka, K))) continue;
    const float l = chord_sel<AX>(__ldg(tabA + lo + ka), rx, ry, G.dz);
    accl += l;
    ((float *)(tab + 2 * N))[chord_word(N, (unsigned)vi, ka)] = l;
  }
  ((int2 *)tab)[vi] =
      make_int2(cnt ? (int)(((unsigned)cnt << 24) | (unsigned)(w.b0 * D.na + lo)) : 0,
                __float_as_int(sart_norm(accl)));
}

// Counting (K == 0: the largest pair count into kmax[0]) or filling pass over
// every view of the instance insts[0] (the first of instances sharing
// geometry, or one instance): grid (x tiles, y tiles, views).
__global__ void __launch_bounds__(kAtxThreads)
    k_atx_chords(const Inst *__restrict__ insts, int K, int *tabs, int *kmax) {
  const Inst &I0 = insts[0];
  const Dims D = I0.d;
  const int view = blockIdx.z;
  if (view >= I0.nv) return;
  const ViewGeo G = view_of(I0, view);
  const int vf = I0.vflags[view];
  if ((vf & kViewAxisParallel) || G.z_det[0] != 0.0f) return;  // no table
  int ix, iy, iz;
  const bool valid = tile_voxel(D, ix, iy, iz);  // the whole warp goes on
  const float4 *__restrict__ tabA = I0.tabA + (long long)view * D.na;
  int *tab = tabs ? tabs + (size_t)view * chord_view_words(D, K) : nullptr;
  if (!(vf & kViewNotX))
    chords_voxel<1>(G, D, tabA, valid, ix, iy, K, tab, kmax);
  else if (!(vf & kViewNotY))
    chords_voxel<2>(G, D, tabA, valid, ix, iy, K, tab, kmax);
  else
    chords_voxel<0>(G, D, tabA, valid, ix, iy, K, tab, kmax);
}

// Backward step for a group of instances sharing geometry.  With a chord
// table (2-D) a thread's loads that depend on nothing but its position -- the
// table's head and first kChordPre chords, the group's image values -- go out
// together with the group's state, so that it waits for memory once before
// the residuals (the view's few kB, in L1), and no barrier is needed.  Pairs
// past a voxel's own add 0 times a residual, which is finite here.
// Memory latency bounds it (28 % issue).  A launch of 64 instances, 512^2:
// 53.5 us with the group's scalars gathered through shared memory between two
// barriers, one load per chord and a division per instance; 42.7 us now at 4
// blocks per SM, 41.3 at 5, 42.5 at 6; with the direct form out of line 43.8
// (5 blocks) to 54.8 (8 blocks).
// kPairs: a thread still loads its own voxel's table entries, but the image
// and the residuals are read with two lanes to a voxel, a quad of instances
// each, in two turns (the entries through shuffles): a load then takes whole
// 32-byte sectors, 16 of them in 512 contiguous bytes, where a lane that reads
// its two quads one after the other touches each sector twice.  34.8 us (4
// blocks 36.3, 3 42.8, 6 with the spills 41.0).  Groups of at most four
// instances, whose second quad is empty, keep the lane per voxel: 24 instances
// in groups of four 4.6 ms a run, 5.0 in pairs.
template <bool kPlanar, bool kPairs>
__global__ void __launch_bounds__(kAtxThreads, 5)
    k_sart_atx_shared(const Inst *__restrict__ insts, int batch, int view,
                      const int2 *__restrict__ gtab) {
  (void)batch;
  pdl_enter();
  const int g0 = gtab ? gtab[blockIdx.z].x : (int)blockIdx.z * kShareGroup;
  const Inst &I0 = insts[g0];
  if (view >= I0.nv) return;  // a group with fewer views
  const Dims D = I0.d;  // every instance of the group
  const GroupState &gs = *I0.grp;
  // the group's residuals, interleaved: ray r of slot b at corg[r*kShareGroup + b]
  const float4 *__restrict__ corg = (const float4 *)I0.cor;
  const int vf = I0.vflags[view];
  if (kPlanar && I0.chtab) {
    int ix, iy, iz;
    const bool valid = tile_voxel(D, ix, iy, iz);
    const size_t N = (size_t)D.nx * D.ny;
    const int K = I0.chK;
    const int *__restrict__ tab = I0.chtab + (size_t)view * chord_view_words(D, K);
    const unsigned vi = valid ? (unsigned)iy * D.nx + ix : 0u;
    const ChordPre c = chord_load(tab, N, K, vi);
    const bool use = !(vf & kViewAxisParallel) && I0.g.z_det[0] == 0.0f;
    if constexpr (kPairs) {
      // lane 2 j + q: quad q of voxel 16 h + j of the warp's row in turn h
      static_assert(kShareGroup == 8, "two quads");
      const int lane = threadIdx.x & 31, q = lane & 1;
      float4 *const mq = (float4 *)I0.m_il + q;
      const unsigned mine_vi = valid ? vi : 0xffffffffu;
      unsigned vh[2];
      float4 m4[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        vh[h] = __shfl_sync(0xffffffffu, mine_vi, 16 * h + (lane >> 1));
        m4[h] = vh[h] < N ? mq[(size_t)vh[h] * 2] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      const unsigned active = gs.active;
      if (!active) return;
      if (use && gs.bad != view + 1) {
        const unsigned mine = (active >> (4 * q)) & 0xFu;  // the quad's running instances
        const int kA = __reduce_max_sync(0xffffffffu, valid ? c.cnt : 0);
        const long long M = nray(D);
        const float4 *const cq = corg + q;
        const int head = c.cnt << 24 | c.first;
        int hd[2];
        float acc[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          hd[h] = __shfl_sync(0xffffffffu, head, 16 * h + (lane >> 1));
#pragma unroll
          for (int b = 0; b < 4; b++) acc[h][b] = 0.f;
        }
        auto pair = [&](float (&a)[4], int r, float l) {
          if (!mine || !ASD_IN(r, M)) return;
          const float4 c4 = __ldg(cq + (size_t)r * 2);
          pair2(a[0], l, c4.x);
          pair2(a[1], l, c4.y);
          pair2(a[2], l, c4.z);
          pair2(a[3], l, c4.w);
        };
#pragma unroll
        for (int ka = 0; ka < kChordPre; ka++) {
          if (ka >= kA) break;
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const float l = __shfl_sync(0xffffffffu, c.l[ka], 16 * h + (lane >> 1));
            pair(acc[h], (hd[h] & 0xffffff) + (ka < (int)((unsigned)hd[h] >> 24) ? ka : 0), l);
          }
        }
        for (int ka = kChordPre; ka < kA; ka++)
#pragma unroll
          for (int h = 0; h < 2; h++)
            if (ka < (int)((unsigned)hd[h] >> 24) && ASD_IN(ka, K) && vh[h] < N)
              pair(acc[h], (hd[h] & 0xffffff) + ka, chord_slot(tab, N, vh[h], ka));
        const float4 b4 = __ldg((const float4 *)gs.beta + q);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const float norm = __shfl_sync(0xffffffffu, c.norm, 16 * h + (lane >> 1));
          if (vh[h] >= N || !mine) continue;
          float4 v = m4[h];
          if (mine & 1u) v.x = sart_update(v.x, b4.x, acc[h][0], norm);
          if (mine & 2u) v.y = sart_update(v.y, b4.y, acc[h][1], norm);
          if (mine & 4u) v.z = sart_update(v.z, b4.z, acc[h][2], norm);
          if (mine & 8u) v.w = sart_update(v.w, b4.w, acc[h][3], norm);
          mq[(size_t)vh[h] * 2] = v;
        }
        return;
      }
    } else {
      float4 *mg = (float4 *)I0.m_il + (size_t)vi * (kShareGroup / 4);
      float4 m4[kShareGroup / 4];
#pragma unroll
      for (int q = 0; q < kShareGroup / 4; q++) m4[q] = mg[q];
      const unsigned active = gs.active;
      if (!active) return;
      if (use && gs.bad != view + 1) {
        const int kA = __reduce_max_sync(0xffffffffu, valid ? c.cnt : 0);
        const long long M = nray(D);
        float acc[kShareGroup];
#pragma unroll
        for (int b = 0; b < kShareGroup; b++) acc[b] = 0.f;
        auto pair = [&](int r, float l) {
          if (!ASD_IN(r, M)) return;
          const float4 *p = corg + (size_t)r * (kShareGroup / 4);
#pragma unroll
          for (int q = 0; q < kShareGroup / 4; q++) {
            if (!((active >> (4 * q)) & 0xFu)) continue;
            const float4 c4 = __ldg(p + q);
            pair2(acc[4 * q], l, c4.x);
            pair2(acc[4 * q + 1], l, c4.y);
            pair2(acc[4 * q + 2], l, c4.z);
            pair2(acc[4 * q + 3], l, c4.w);
          }
        };
#pragma unroll
        for (int ka = 0; ka < kChordPre; ka++) {
          if (ka >= kA) break;
          pair(c.first + (ka < c.cnt ? ka : 0), c.l[ka]);
        }
        for (int ka = kChordPre; ka < kA; ka++)
          if (ka < c.cnt && ASD_IN(ka, K)) pair(c.first + ka, chord_slot(tab, N, vi, ka));
        if (valid && ASD_IN(vi, N)) atx_shared_apply(c.norm, acc, gs, active, m4, mg);
        return;
      }
    }
  }
  const unsigned active = gs.active;
  if (!active) return;
  const ViewGeo G = view_of(I0, view);
  const float4 *__restrict__ tabA = I0.tabA + (long long)view * D.na;
  const float4 *__restrict__ tabC = I0.tabC;
  const bool planar_ok = !kPlanar || G.z_det[0] == 0.0f;
  const bool narrow = planar_ok && !(vf & kViewAxisParallel) && gs.bad != view + 1;
  if (!(vf & (kViewAxisParallel | kViewNotX)))
    atx_shared_voxel<kPlanar, 1>(G, D, corg, tabA, tabC, planar_ok, narrow, gs, active, I0.m_il);
  else if (!(vf & (kViewAxisParallel | kViewNotY)))
    atx_shared_voxel<kPlanar, 2>(G, D, corg, tabA, tabC, planar_ok, narrow, gs, active, I0.m_il);
  else
    atx_shared_voxel<kPlanar, 0>(G, D, corg, tabA, tabC, planar_ok, narrow, gs, active, I0.m_il);
}

// ---------------------------------------------------------------------------
// Shared-geometry forward step: one warp per ray for a group of kShareGroup
// instances.  The column march (cells and weights) is evaluated once per ray
// and each piece reads the group's voxel values with kShareGroup / 4 float4 loads
// from the interleaved images; every instance accumulates its pieces in the
// order of k_sart_ax and sums lanes with the same butterfly, and its
// epilogue is that of k_sart_ax, so its projection, residual, squares and
// flags are bit-identical to it.
// ---------------------------------------------------------------------------
// columns per round of loads in the shared forward step, and 64 registers for 8
// blocks per SM.  Cone beams: three pieces per column already keep six loads in
// flight (8 blocks 10 % faster than 6 at 128^3).  Fan beams, a launch of 64
// instances and four iterations of them (512^2): one column at 8 blocks 25.0 us
// and 15.2 ms; at 7 26.4 and 15.7, at 10 25.5 and 15.4; two columns at 6 blocks
// 26.9 and 16.1, at 8 26.6 and 16.1, at 10 25.9 and 15.5.
constexpr int kAxShareU = 1;
// quads of a group (4 instances each) per lane: one for fan beams, both for
// cone beams.  One: two lanes to a voxel, so that a load takes whole 32-byte
// sectors, and two warps to a ray, 16 of its columns each, so that the columns
// are still dealt to 32 lanes and added in the same order.  A launch of 64
// instances, 512^2 and 888 bins, waits for memory (42 % issue): at two columns
// a round 32.8 us with the two quads in blocks of their own, each taking half of
// every sector, 26.9 now; both quads in a lane 29.0.
template <bool k3D>
constexpr int kAxShareQ = k3D ? kShareGroup / 4 : 1;

// kU columns per round and kQ quads per lane are launch shapes that a plan's
// autotuner may change (asdpocs_plan_autotune_shapes): neither changes the
// order in which an instance's pieces are added, so every shape gives the
// same bits.
template <bool k3D, int kU, int kQ>
__global__ void __launch_bounds__(kAxBlock, 8)
    k_sart_ax_shared(const Inst *__restrict__ insts, int batch, int view,
                     const int2 *__restrict__ gtab) {
  constexpr int kQuads = kShareGroup / 4, kS = 4 * kQ;
  // kW lanes of a voxel (kQ quads each) and, so that a ray's columns are
  // still dealt to 32 lanes, kW warps of a ray
  constexpr int kW = kQuads / kQ, kRays = kAxWarps / kW;
  __shared__ float s_part[kW > 1 ? kRays : 1][kW][kS + 1][32];
  pdl_enter();
  const int gz = (int)blockIdx.z;                                    // the group
  const int g0 = gtab ? gtab[gz].x : gz * kShareGroup;
  const int gn = gtab ? gtab[gz].y : min(kShareGroup, batch - g0);
  const Inst &I0 = insts[g0];
  if (view >= I0.nv) return;
  const Dims D = I0.d;
  const long long nr = nray(D), r0 = (long long)blockIdx.x * kRays;
  const int lane = threadIdx.x & 31;
  const int rl = (threadIdx.x >> 5) / kW, wr = (threadIdx.x >> 5) % kW;
  const long long r = r0 + rl;
  const int q0 = lane % kW;                     // this lane's quads: q0, q0 + kW, ...
  const int col = wr * (32 / kW) + lane / kW;   // its columns: col, col + 32, ...
  const ViewGeo G = view_of(I0, view);
  // cone beam: the plan's one ray-slope table, refreshed by group 0 every
  // view whether or not its instances still run
  if (k3D && blockIdx.z == 0 && threadIdx.x < kRays && r0 + threadIdx.x < nr) {
    const long long rs = r0 + threadIdx.x;
    ray_slopes(I0, G, D, view, (int)(rs % D.na), (int)(rs / D.na), rs);
  }
  const unsigned active = I0.grp->active;
  if (!active) return;
  // lane kW * j + q0 of a ray's first warp: its j-th sum's instance
  const int slot = 4 * (q0 + kW * ((lane / kW) / 4)) + (lane / kW) % 4;
  const Inst &Ib = insts[g0 + min(slot, gn - 1)];
  const bool live = wr == 0 && r < nr && lane < kShareGroup && slot < gn && ((active >> slot) & 1u);
  RayOut o{0.f, 0.0};
  if (live) o = ray_out_load(Ib, view, r, nr);
  float v[kS + 1];  // the instances' sums, then the weights' sum
#pragma unroll
  for (int b = 0; b <= kS; b++) v[b] = 0.f;
  const float4 *__restrict__ mg = (const float4 *)I0.m_il;
  if (r < nr) {  // the whole warp
    const int ia = (int)(r % D.na), ib = (int)(r / D.na);
    const float zd = G.z_det[ib];
    const RayMarch R = ray_setup(G, D, G.y_det[ia], zd);
    const bool planar = D.nz == 1 && zd == 0.0f;
    // kU columns per round: their pieces first, then all their
    // (predicated) loads, then the accumulation in column and piece order
    auto march = [&](auto pieces) {
      constexpr int kP = decltype(pieces)::value;
      for (int iu0 = col; iu0 - col < R.nu; iu0 += 32 * kU) {
        unsigned id[kU][kP];
        float w[kU][kP];
        bool f[kU][kP];
        if constexpr (kP == 2) {
#pragma unroll
          for (int u = 0; u < kU; u++)
            column_pieces_planar(R, iu0 + u * 32, id[u], w[u], f[u]);
        } else {
          ColumnV cv[kU];
          ColumnZ cz[kU];
          bool some = false;
#pragma unroll
          for (int u = 0; u < kU; u++) {
            cv[u] = column_v(R, iu0 + u * 32);
            cz[u] = column_z(R, R.slope2, cv[u]);
            some = some || ((cv[u].lo || cv[u].hi) && (cz[u].lo || cz[u].hi));
          }
          if (!any_lane(some)) continue;
#pragma unroll
          for (int u = 0; u < kU; u++)
            column_pieces3(R, R.lfac, iu0 + u * 32, cv[u], cz[u], id[u], w[u], f[u]);
        }
        float4 x[kU][kP][kQ];
#pragma unroll
        for (int u = 0; u < kU; u++)
#pragma unroll
          for (int j = 0; j < kP; j++) {
            const float4 *p = mg + (size_t)id[u][j] * kQuads + q0;
            f[u][j] = f[u][j] && ASD_IN(id[u][j], nvox(D));
#pragma unroll
            for (int q = 0; q < kQ; q++)
              x[u][j][q] = (f[u][j] && ((active >> (4 * (q0 + kW * q))) & 0xFu))
                               ? __ldg(p + kW * q)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
        for (int u = 0; u < kU; u++)
#pragma unroll
          for (int j = 0; j < kP; j++) {
            if (!f[u][j]) continue;
#pragma unroll
            for (int q = 0; q < kQ; q++) {
              v[4 * q] = weight_fma(w[u][j], x[u][j][q].x, v[4 * q]);
              v[4 * q + 1] = weight_fma(w[u][j], x[u][j][q].y, v[4 * q + 1]);
              v[4 * q + 2] = weight_fma(w[u][j], x[u][j][q].z, v[4 * q + 2]);
              v[4 * q + 3] = weight_fma(w[u][j], x[u][j][q].w, v[4 * q + 3]);
            }
            v[kS] += w[u][j];
          }
      }
    };
    // fan beams (nz == nb == 1: the one detector row at z = 0) are planar
    if (!k3D || planar)
      march(std::integral_constant<int, 2>());
    else if constexpr (k3D)
      march(std::integral_constant<int, 3>());
  }
  // the butterfly of warp_sum over the 32 columns: the steps between a ray's
  // warps through shared memory, the others between lanes
  if constexpr (kW > 1) {
    static_assert(kW == 2, "one step between warps");
#pragma unroll
    for (int b = 0; b <= kS; b++) s_part[rl][wr][b][lane] = v[b];
    __syncthreads();
    if (wr) return;
#pragma unroll
    for (int b = 0; b <= kS; b++) v[b] += s_part[rl][1][b][lane];
  }
#pragma unroll
  for (int b = 0; b <= kS; b++)
#pragma unroll
    for (int o = 16; o >= kW; o >>= 1) v[b] += __shfl_xor_sync(0xffffffffu, v[b], o);
  float yb = 0.f;
#pragma unroll
  for (int b = 0; b < kS; b++)
    if (lane / kW == b) yb = v[b];
  if (live) ray_out_store(Ib, &I0.grp->bad, view, r, r, nr, o, yb * G.scale, v[kS] * G.scale);
}

// Rounds an FP32 sinogram to FP16 / BF16 storage (round to nearest, ties to
// even: the same bits as asdpocs_store_sinogram on the host).
__global__ void __launch_bounds__(256)
    k_store_sinogram(const float *__restrict__ src, void *dst, long long n, int fmt) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    if (fmt == ASDPOCS_STORE_F16)
      ((__half *)dst)[i] = __float2half_rn(src[i]);
    else
      ((__nv_bfloat16 *)dst)[i] = __float2bfloat16_rn(src[i]);
  }
}

// Copies the running instances of each shared-geometry group between their
// own images (m) and the group's interleaved images (m_il): pack before the
// SART sweep, unpack after it.  Grid (voxel blocks, 1, groups).
__global__ void __launch_bounds__(256)
    k_group_pack(const Inst *__restrict__ insts, int batch, int unpack,
                 const int2 *__restrict__ gtab) {
  __shared__ float *s_m[kShareGroup];
  __shared__ unsigned s_active;
  pdl_enter();
  const int g0 = gtab ? gtab[blockIdx.z].x : (int)blockIdx.z * kShareGroup;
  const int gn = gtab ? gtab[blockIdx.z].y : min(kShareGroup, batch - g0);
  if (threadIdx.x == 0) s_active = 0u;
  __syncthreads();
  if (threadIdx.x < gn) {
    const Inst &Ib = insts[g0 + threadIdx.x];
    s_m[threadIdx.x] = Ib.m;
    if (((volatile int *)&Ib.s->done)[0] == 0) atomicOr(&s_active, 1u << threadIdx.x);
  }
  __syncthreads();
  const unsigned active = s_active;
  if (!unpack && blockIdx.x == 0) {  // the sweep's group state
    GroupState &gs = *insts[g0].grp;
    if (threadIdx.x < gn) gs.beta[threadIdx.x] = insts[g0 + threadIdx.x].s->beta_f;
    if (threadIdx.x == 0) {
      gs.active = active;
      gs.bad = 0;
    }
  }
  const Dims D = insts[g0].d;
  const long long n = (long long)D.nx * D.ny * D.nz;
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (!active || v >= n) return;
  float4 *mg = (float4 *)insts[g0].m_il + v * (kShareGroup / 4);
#pragma unroll
  for (int q = 0; q < kShareGroup / 4; q++) {
    if (!((active >> (4 * q)) & 0xFu)) continue;
    float4 x = unpack ? mg[q] : make_float4(0.f, 0.f, 0.f, 0.f);
    float *xv = &x.x;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int b = 4 * q + j;
      if (b < gn && ((active >> b) & 1u)) {
        if (unpack)
          s_m[b][v] = xv[j];
        else
          xv[j] = s_m[b][v];
      }
    }
    if (!unpack) mg[q] = x;
  }
}

}  // namespace

// A caller's stream that is being captured gets ordinary launches.
static bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &c) == cudaSuccess) return c != cudaStreamCaptureStatusNone;
  cudaGetLastError();  // the launch that follows reports it
  return true;
}

// Whether a launch of `batch` instances takes kAxRows rays a warp.  One ray each
// where the warps of all rays are resident at once, or nearly (36 on each of 152
// SMs): a warp of four is four times as long then and saves nothing.  us a view of
// a plan, rows and rays: 64^3 on 128 x 16 4.5 and 3.4, x 40 5.3 and 4.4, x 48 5.5
// and 6.3, 32^3 on 64 x 64 4.1 and 3.6, 128 x 128 x 64 on 256 x 20 7.1 and 5.6, x 24
// 7.1 and 7.6, 256 x 256 x 64 on 512 x 8 9.5 and 7.8, x 16 11.0 and 11.9.
static bool ax_by_rows(const Dims &d, int batch) {
  return d.nz > 1 && d.nb > 2 && (long long)d.na * d.nb * batch > 152 * 36;
}

// Blocks of the forward kernels that take an instance at a time.
static unsigned ax_blocks(const Dims &d, bool rows) {
  const long long warps = rows ? ax_warps3(d) : (long long)d.na * d.nb;
  return (unsigned)((warps + kAxWarps - 1) / kAxWarps);
}

cudaError_t launch_ax(const float *x, float *y, float *sr, const ViewGeo &g,
                      const Dims &d, cudaStream_t st) {
  const long long nr = (long long)d.na * d.nb;
  if (nr == 0) return cudaSuccess;
  const PdlScope scope(!capturing(st));
  const bool rows = ax_by_rows(d, 1);
  auto k = rows ? k_ax<true> : k_ax<false>;
  return launch_iter(k, dim3(ax_blocks(d, rows)), dim3(kAxBlock), st, x, y, sr, g, d);
}

cudaError_t launch_atx(float *x, const float *y, float *sc, const ViewGeo &g,
                       const Dims &d, cudaStream_t st) {
  const dim3 grid = tile_grid(d.nx, d.ny, d.nz, 1);
  const PdlScope scope(!capturing(st));
  // bins that a tile sees, about: its diagonal at the magnification of the corner
  // nearest the source
  const float corner = 0.5f * sqrtf((float)d.nx * d.nx + (float)d.ny * d.ny);
  const bool fine = (kTileX + kTileY / 2) * g.SD > kTabA * (g.SO - corner) * g.dy_det;
  auto k = !(d.nz == 1 && d.nb == 1) ? k_atx<false, 3> : fine ? k_atx<true, 4> : k_atx<true, 6>;
  return launch_iter(k, grid, dim3(kAtxThreads), st, x, y, sc, g, d);
}

cudaError_t launch_store_sinogram(const float *src, void *dst, size_t n, int fmt,
                                  cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (fmt == ASDPOCS_STORE_F32)
    return cudaMemcpyAsync(dst, src, n * 4, cudaMemcpyDeviceToDevice, st);
  const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 152 * 64);
  k_store_sinogram<<<blocks, 256, 0, st>>>(src, dst, (long long)n, fmt);
  return cudaGetLastError();
}

static size_t zcol_align(size_t b) { return (b + 255) & ~(size_t)255; }

bool zcol_fits(const Dims &d) {
  return d.nz > 1 && ((long long)d.na + kZcCols) * d.nb + kZcRows < (1LL << 31);
}

int seen_slices(const ViewGeo &g, const Dims &d) {
  const float n = d.nb * g.dz_det * g.SO / (g.SD * g.dz) + 2.0f;
  return n >= 2.0f && n < (float)d.nz ? (int)n : d.nz;
}

// The set-up of a voxel column is shared by its crossed slices, and a block of
// columns waits for it, so the walk is the better form where a view crosses few
// slices: in launches of more blocks than are resident at once (152 SMs, four
// each) up to one for every 512 blocks with all slices crossed, and up to 23 with
// a part of them, whose groups of lanes are not full; in smaller launches up to 5
// with a part of them.  us a view of a plan, columns and walk, n^2 x nz:
//   all crossed: 256 x 4 23 and 24, x 8 26 and 32, 512 x 4 67 and 47, x 8 80 and 69,
//     x 12 117 and 97, x 16 119 and 120, x 32 200 and 235, 128 x 8 12 and 18;
//   part of them (seen): 256 x 24 (9) 45 and 35, 256 x 64 (21) 64 and 65, 512 x 32
//     (21) 188 and 173, 512 x 100 (32) 302 and 317, 128 x 32 (5) 18 and 14, 128 x 48
//     (16) 21 and 26.
ConeForm cone_form(const Dims &d, int batch, int seen) {
  if (!zcol_fits(d)) return kConeVoxels;
  const long long blocks = (long long)((d.nx + 31) / 32) * d.ny * batch;
  const bool large = blocks > 152 * 4;
  const bool few = seen < d.nz ? seen < (large ? 24 : 6) : large && 512LL * seen <= blocks;
  return few ? kConeWalk : kConeColumns;
}

// One view by itself needs its ray tables first, two launches more: about 1.4
// million pairs of a voxel and a bin (the bins across a voxel at the axis, by the
// rows).  us a view on device buffers, columns and per voxel, n^2 x nz (million
// pairs): 64 x 64 (0.8) 20 and 17; 91 x 81 x 70 (1.2) 29 and 25; 98 x 88 x 59 (1.3)
// 27 and 28; 93 x 83 x 52 (1.6) 28 and 28; 101 x 101 x 48 (1.9) 28 and 37; 128 x 64
// (3.2) 40 and 56.  Few slices as for a plan: 256 x 8 28 and 28, x 16 38 and 52; 512 x
// 6 75 and 68, x 8 75 and 92; part of the slices (seen): 256 x 24 (9) 45 and 34, 256
// x 64 (8) 44 and 47, 512 x 24 (9) 115 and 126, x 16 (7) 88 and 78.
bool atx_columns(const ViewGeo &g, const Dims &d) {
  const int seen = seen_slices(g, d);
  const float q = g.SD / g.SO;
  const float pairs = (float)d.nx * d.ny * seen * fmaxf(q / g.dy_det, 1.0f) *
                      fmaxf(q * g.dz / g.dz_det, 1.0f);
  // volumes beyond a launch's rows are refused in either form (launch_atx)
  return zcol_fits(d) && tile_rows(d.ny, d.nz) <= kMaxGridRows &&
         seen >= (seen < d.nz ? 12 : 8) && pairs >= 1.4e6f;
}

size_t ray_table_pad(const Dims &d) { return zcol_fits(d) ? (size_t)zcol_pad(d) : 0; }

size_t atx_zcol_scratch_bytes(const Dims &d) {
  const size_t M = (size_t)d.na * d.nb + (size_t)zcol_pad(d);
  return zcol_align((size_t)d.na * sizeof(float4)) + zcol_align(M * sizeof(float4)) +
         zcol_align(M * sizeof(float)) + 256;
}

cudaError_t launch_atx_zcol(float *x, const float *y, float *sc, const ViewGeo &g,
                            const Dims &d, void *scratch, cudaStream_t st) {
  const long long nr = (long long)d.na * d.nb + zcol_pad(d);
  char *b = (char *)scratch;
  float4 *tabA = (float4 *)b;
  float4 *tabC = (float4 *)(b + zcol_align((size_t)d.na * sizeof(float4)));
  float *yt = (float *)((char *)tabC + zcol_align((size_t)nr * sizeof(float4)));
  int *flag = (int *)((char *)yt + zcol_align((size_t)nr * sizeof(float)));
  // launches that report their own errors only, in the ordinary way (neither
  // kernel waits for the one before it)
  const PdlScope scope(false);
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), st);
  if (e == cudaSuccess)
    e = launch_iter(k_view_tab3, dim3((unsigned)((nr + 255) / 256)), dim3(256), st, y, tabA, tabC,
                    yt, flag, g, d);
  const ZColShape s = zcol_shape(d, 1, 0, seen_slices(g, d));
  if (e == cudaSuccess)
    e = launch_iter(s.W == 32 ? k_atx_zcol<32> : k_atx_zcol<8>, zcol_grid(d, 1, s),
                    dim3(kZcThreads), st, x, sc, tabA, tabC, yt, flag, g, d, s.lsh(), s.seg);
  return e;
}

cudaError_t launch_sart_ax(const Inst *insts, int batch, const Dims &d,
                           int view, cudaStream_t st, bool exact, const int *zmap) {
  cudaError_t e;
  const long long nr = (long long)d.na * d.nb;
  const bool rows = ax_by_rows(d, batch);
  const dim3 grid(ax_blocks(d, rows), 1, batch);
  const int rpw = sid_rays(nr * batch, d);
  const dim3 grid_ex(sid_blocks(nr, rpw), 1, batch);
  const bool p3 = d.nz > 1 || d.nb > 1;
  if (exact) {
    if (p3)
      e = launch_iter(k_sart_ax_exact<true>, grid_ex, dim3(kAxBlock), st, insts, view, zmap, rpw);
    else
      e = launch_iter(k_sart_ax_exact<false>, grid_ex, dim3(kAxBlock), st, insts, view, zmap, rpw);
  } else {
    if (rows)
      e = launch_iter(k_sart_ax<true, true>, grid, dim3(kAxBlock), st, insts, view, zmap);
    else if (p3)
      e = launch_iter(k_sart_ax<true, false>, grid, dim3(kAxBlock), st, insts, view, zmap);
    else
      e = launch_iter(k_sart_ax<false, false>, grid, dim3(kAxBlock), st, insts, view, zmap);
  }
  return e;
}

cudaError_t launch_ax_siddon(const float *x, float *y, float *sr, const ViewGeo &g,
                             const Dims &d, cudaStream_t st) {
  const long long nr = (long long)d.na * d.nb;
  if (nr == 0) return cudaSuccess;
  const int rpw = sid_rays(nr, d);
  k_ax_siddon<<<sid_blocks(nr, rpw), kAxBlock, 0, st>>>(x, y, sr, g, d, rpw);
  return cudaGetLastError();
}

cudaError_t launch_sart_atx(const Inst *insts, int batch, const Dims &d,
                            int view, cudaStream_t st, ConeForm form, int zseg, int seen,
                            const int *zmap) {
  cudaError_t e;
  // fan beams: the fewest tiles a block (1, 2 or 4) that keep the launch within
  // two blocks per SM, so that they sit, their tables loaded, beside the forward
  // step's (512^2, ten iterations: 8.1 ms with 256 blocks of four tiles, 8.55
  // with 512 of two; 10.4 without the loads before the wait; 7.3 with the images
  // among them)
  int tiles = d.nz == 1 ? 1 : kTilesPerBlock;
  dim3 grid = group_grid(d.nx, d.ny, d.nz, batch, tiles);
  while (tiles < kTilesPerBlock && (long long)grid.x * grid.y * batch > 152 * 2) {
    tiles *= 2;
    grid = group_grid(d.nx, d.ny, d.nz, batch, tiles);
  }
  if (d.nz > 1 && form == kConeWalk) {
    const int seg = zseg > 0 ? zseg : zwalk_seg((long long)d.nx * d.ny * d.nz * batch);
    const dim3 g((d.nx + kTileX - 1) / kTileX,
                 (d.ny + kTileY - 1) / kTileY * ((d.nz + seg - 1) / seg), batch);
    e = launch_iter(k_sart_atx_zwalk, g, dim3(kAtxThreads), st, insts, view, seg, zmap);
  } else if (d.nz > 1 && form == kConeColumns) {
    const ZColShape s = zcol_shape(d, batch, zseg, seen > 0 ? std::min(seen, d.nz) : d.nz);
    e = launch_iter(s.W == 32 ? k_sart_atx_zcol<32> : k_sart_atx_zcol<8>, zcol_grid(d, batch, s),
                    dim3(kZcThreads), st, insts, view, s.lsh(), s.seg, zmap);
  } else if (d.nz > 1 || d.nb > 1)
    e = launch_iter(k_sart_atx<false, 64>, grid, dim3(kAtxThreads), st, insts, view, zmap, tiles);
  else if ((long long)grid.x * grid.y * batch <= 152 * 2)
    e = launch_iter(k_sart_atx<true, 96>, grid, dim3(kAtxThreads), st, insts, view, zmap, tiles);
  else
    e = launch_iter(k_sart_atx<true, 64>, grid, dim3(kAtxThreads), st, insts, view, zmap, tiles);
  return e;
}

cudaError_t launch_sart_atx_shared(const Inst *insts, int batch,
                                   const Dims &d, int view, cudaStream_t st,
                                   const int2 *gtab, int ngroups, int fewest) {
  cudaError_t e;
  if (!gtab) fewest = min(batch, kShareGroup);
  dim3 grid = tile_grid(d.nx, d.ny, d.nz, 1);
  grid.z = gtab ? ngroups : (batch + kShareGroup - 1) / kShareGroup;
  if (d.nz > 1 || d.nb > 1)
    e = launch_iter(k_sart_atx_shared<false, false>, grid, dim3(kAtxThreads), st, insts, batch,
                    view, gtab);
  else if (fewest > 4)
    e = launch_iter(k_sart_atx_shared<true, true>, grid, dim3(kAtxThreads), st, insts, batch,
                    view, gtab);
  else
    e = launch_iter(k_sart_atx_shared<true, false>, grid, dim3(kAtxThreads), st, insts, batch,
                    view, gtab);
  return e;
}

template <bool k3D, int kU, int kQ>
static cudaError_t sart_ax_shared_as(const Inst *insts, int batch, long long rays,
                                     unsigned groups, int view, cudaStream_t st,
                                     const int2 *gtab) {
  constexpr int kRays = kAxWarps / (kShareGroup / 4 / kQ);
  return launch_iter(k_sart_ax_shared<k3D, kU, kQ>,
                     dim3((unsigned)((rays + kRays - 1) / kRays), 1, groups), dim3(kAxBlock), st,
                     insts, batch, view, gtab);
}

template <bool k3D>
static cudaError_t sart_ax_shared_shape(const Inst *insts, int batch, long long rays,
                                        unsigned groups, int view, cudaStream_t st, int u,
                                        int q, const int2 *gtab) {
  u = u ? u : kAxShareU;
  q = q ? q : kAxShareQ<k3D>;
  if (u == 1 && q == 1)
    return sart_ax_shared_as<k3D, 1, 1>(insts, batch, rays, groups, view, st, gtab);
  if (u == 2 && q == 1)
    return sart_ax_shared_as<k3D, 2, 1>(insts, batch, rays, groups, view, st, gtab);
  if (u == 1 && q == 2)
    return sart_ax_shared_as<k3D, 1, 2>(insts, batch, rays, groups, view, st, gtab);
  if (u == 2 && q == 2)
    return sart_ax_shared_as<k3D, 2, 2>(insts, batch, rays, groups, view, st, gtab);
  return cudaErrorInvalidValue;
}

cudaError_t launch_sart_ax_shared(const Inst *insts, int batch, const Dims &d,
                                  int view, cudaStream_t st, int u, int q,
                                  const int2 *gtab, int ngroups) {
  const long long rays = (long long)d.na * d.nb;
  const unsigned groups =
      gtab ? (unsigned)ngroups : (unsigned)((batch + kShareGroup - 1) / kShareGroup);
  if (d.nz > 1 || d.nb > 1)
    return sart_ax_shared_shape<true>(insts, batch, rays, groups, view, st, u, q, gtab);
  return sart_ax_shared_shape<false>(insts, batch, rays, groups, view, st, u, q, gtab);
}

cudaError_t launch_group_pack(const Inst *insts, int batch, const Dims &d,
                              int unpack, cudaStream_t st, const int2 *gtab, int ngroups) {
  cudaError_t e;
  const long long n = (long long)d.nx * d.ny * d.nz;
  const dim3 grid((unsigned)((n + 255) / 256), 1,
                  gtab ? ngroups : (batch + kShareGroup - 1) / kShareGroup);
  e = launch_iter(k_group_pack, grid, dim3(256), st, insts, batch, unpack, gtab);
  return e;
}

cudaError_t launch_atx_chords(const Inst *insts, const Dims &d, int nv, int K,
                              int *tabs, int *kmax, cudaStream_t st) {
  if (K < 0 || K > kChordMaxSlots || (K > 0 && !tabs) || d.nz != 1 || d.nb != 1)
    return cudaErrorInvalidValue;
  dim3 grid = tile_grid(d.nx, d.ny, 1, nv);
  k_atx_chords<<<grid, kAtxThreads, 0, st>>>(insts, K, tabs, kmax);
  return cudaGetLastError();
}

size_t atx_chord_words(const Dims &d, int nv, int K) {
  return chord_view_words(d, K) * (size_t)nv;
}

int atx_chord_max_slots() { return kChordMaxSlots; }

cudaError_t launch_view_tables(const Inst *insts, int batch, const Dims &d,
                               int nv, cudaStream_t st) {
  k_view_tables<<<dim3((d.na + 127) / 128, nv, batch), 128, 0, st>>>(insts);
  return cudaGetLastError();
}

#ifdef ASDPOCS_CHECKED
ASD_CHECKED_READER(checked_take_proj)
#endif

int reduce_blocks_for(const Dims &d) { return atx_blocks(d); }

}  // namespace asd
