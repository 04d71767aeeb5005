// Host build of the z-column backward step's addressing and sums (the
// __host__ __device__ functions of csrc/projector.cuh that k_atx_zcol and
// k_sart_atx_zcol call) -- TEST INFRASTRUCTURE.
//   dm_zcol_walk -- a view walked warp by warp, 32 / L voxel columns of L
//              slices each: the tables with the rays of a detector column one
//              after the other, followed by zcol_pad zeros, every lane reading
//              the rays of the warp's most detector columns whether it has
//              pairs there or not.  Returns the number of reads past the
//              padding (skipped); x and sc, where given, take the sums.
// Compiled with -ffp-contract=off so the host compiler fuses nothing.
#include <vector>

#include "../../asd_pocs_mex_cuda_demo_gb300/csrc/projector.cuh"

using namespace asd;

extern "C" long long dm_zcol_walk(float *x, const float *yv, float *sc, float c, float s,
                                  const float *yd, const float *zd, float SO, float OD,
                                  float scale, float ddy, float ddz, float dz, int nx, int ny,
                                  int nz, int na, int nb, int L) {
  const ViewGeo G = with_constants(ViewGeo{c, s, SO, OD, scale, ddy, ddz, dz, yd, zd});
  const Dims D{nx, ny, nz, na, nb};
  const long long M = (long long)na * nb, room = M + zcol_pad(D);
  std::vector<float4> tA(na), tC(room, make_float4(0.f, 0.f, 0.f, 0.f));
  std::vector<float> yt(room, 0.f);
  for (int ia = 0; ia < na; ia++) {
    tA[ia] = ray_tab_a(G, yd[ia]);
    // views without an axis-parallel ray only (the others take the per-voxel form)
    if (tA[ia].x == 0.0f || tA[ia].y == 0.0f) return -1;
    for (int ib = 0; ib < nb; ib++) {
      tC[(long long)ia * nb + ib] = ray_tab_c(tA[ia], zd[ib]);
      if (yv) yt[(long long)ia * nb + ib] = yv[(long long)ib * na + ia];
    }
  }
  long long bad = 0;
  const float hz = dz / 2.0f;
  const int cols = 32 / L;  // voxel columns of a warp
  struct Lane {
    ZCol col;
    int cA, cB, r0;
    float rz;
    bool own;
  } w[32];
  for (int iy = 0; iy < ny; iy++)
    for (int x0 = 0; x0 < nx; x0 += cols)
      for (int z0 = 0; z0 < nz; z0 += L) {
        int mA = 0, mB = 0;
        bool many = false;
        for (int l = 0; l < 32; l++) {
          Lane &q = w[l];
          const int ix = x0 + l / L, iz = z0 + l % L;
          q.own = ix < nx && iz < nz;
          q.cA = q.cB = q.r0 = 0;
          if (ix >= nx) continue;
          q.col = zcol_setup(G, D, ix, iy, true);
          const int count = zcol_count(q.col);
          float zc;
          int blo, bhi;
          if (!zcol_rows(G, D, q.col, iz, zc, blo, bhi)) bhi = blo - 1;
          q.rz = 0.0f - zc;
          q.cB = q.own && blo <= bhi ? bhi - blo + 1 : 0;
          q.cA = q.cB > 0 ? count : 0;
          int s0, s1;  // a voxel with pairs lies in its column's range of slices
          zcol_seen(G, D, q.col, s0, s1);
          bad += q.cA > 0 && (iz < s0 || iz >= s1);
          q.r0 = zcol_first_ray(D, zcol_first(q.col, count), blo);
          mA = q.cA > mA ? q.cA : mA;
          mB = q.cA > 0 && q.cB > mB ? q.cB : mB;
          for (int k = 0; k < q.cA && !many; k++)
            many = col_faces(tA[q.col.lo + k], q.col.rx, q.col.ry).bits & kCfMany;
        }
        const bool unrolled = mA <= kZcCols && mB <= kZcRows && !many;
        for (int l = 0; l < 32; l++) {
          const Lane &q = w[l];
          float acc = 0.f, accl = 0.f;
          if (unrolled && !yv) {  // every lane's reads
            for (int k = 0; k < mA; k++)
              for (int kb = 0; kb < kZcRows; kb++) {
                const long long r = (long long)q.r0 + (long long)k * nb + kb;
                bad += r < 0 || r >= room;
              }
          }
          if (!yv || !q.own) continue;
          // rows outer, columns inner; a lane's missing pairs add 0 times what it reads
          for (int kb = 0; kb < (unrolled ? kZcRows : q.cB); kb++)
            for (int k = 0; k < (unrolled ? mA : q.cA); k++) {
              const long long r = (long long)q.r0 + (long long)k * nb + kb;
              if (r < 0 || r >= room) {
                bad++;
                continue;
              }
              float chord = 0.f;
              if (k < q.cA && kb < q.cB) {
                const int ia = q.col.lo + k;
                const ColFaces f = col_faces(tA[ia], q.col.rx, q.col.ry);
                chord = f.bits & kCfMany
                            ? chord3_bf(tA[ia], tC[r], 0.0f, q.col.rx, q.col.ry, q.rz, dz)
                            : chord3_col(f, tC[r], q.col.rx, q.col.ry, q.rz, hz);
              }
              acc += chord * yt[r];
              accl += chord;
            }
          const long long idx = ((long long)(z0 + l % L) * ny + iy) * nx + x0 + l / L;
          x[idx] = acc * scale;
          sc[idx] = accl * scale;
        }
      }
  return bad;
}
