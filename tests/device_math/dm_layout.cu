// Host build of two more parts of csrc/projector.cuh -- TEST INFRASTRUCTURE.
//   dm_ax_rows -- Ax of a volume by rows of a detector column, as the forward
//              kernels of many rays run it (ray_columns_rows, 32 lanes), or a
//              ray at a time (ray_columns_fast<1>), lanes joined by the warp's
//              butterfly;
//   dm_atx_chords -- a fan-beam view's chord table in the layout of chord_word,
//              filled and read back as the plans' steps do.
// Compiled with -ffp-contract=off so the host compiler fuses nothing.
#include <string.h>

#include <vector>

#include "../../asd_pocs_mex_cuda_demo_gb300/csrc/projector.cuh"

using namespace asd;

static float butterfly(float (&v)[32]) {
  for (int o = 16; o > 0; o >>= 1) {
    float w[32];
    for (int l = 0; l < 32; l++) w[l] = v[l] + v[l ^ o];
    memcpy(v, w, sizeof v);
  }
  return v[0];
}

extern "C" void dm_ax_rows(const float *x, float *y, float *sr, float c, float s,
                           const float *yd, const float *zd, float SO, float OD, float scale,
                           float dz, int nx, int ny, int nz, int na, int nb, int rows) {
  constexpr int K = 4;
  const ViewGeo G = with_constants(ViewGeo{c, s, SO, OD, scale, 0.f, 0.f, dz, yd, zd});
  const Dims D{nx, ny, nz, na, nb};
  auto ld = [&](unsigned i) { return x[i]; };
  for (int ia = 0; ia < na; ia++)
    for (int ib0 = 0; ib0 < nb; ib0 += K) {
      float ty[K][32], ts[K][32], slope2[K], lfac[K];
      for (int k = 0; k < K; k++) {
        const RayMarch Rk = ray_setup(G, D, yd[ia], zd[ib0 + k < nb ? ib0 + k : nb - 1]);
        slope2[k] = Rk.slope2;
        lfac[k] = Rk.lfac;
      }
      for (int l = 0; l < 32; l++) {
        float ys[K] = {0.f, 0.f, 0.f, 0.f}, ss[K] = {0.f, 0.f, 0.f, 0.f};
        const RayMarch R = ray_setup(G, D, yd[ia], zd[ib0]);
        if (rows)
          ray_columns_rows<K>(R, slope2, lfac, l, 32, ld, ys, ss);
        else
          for (int k = 0; k < K && ib0 + k < nb; k++)
            ray_columns_fast<1>(ray_setup(G, D, yd[ia], zd[ib0 + k]), l, 32, ld, ys[k], ss[k]);
        for (int k = 0; k < K; k++) {
          ty[k][l] = ys[k];
          ts[k][l] = ss[k];
        }
      }
      for (int k = 0; k < K && ib0 + k < nb; k++) {
        y[(long long)(ib0 + k) * na + ia] = butterfly(ty[k]) * scale;
        sr[(long long)(ib0 + k) * na + ia] = butterfly(ts[k]) * scale;
      }
    }
}

// Returns the slots used (even), or -1 for a view with an axis-parallel ray.
extern "C" int dm_atx_chords(float *x, const float *yv, float *sc, float c, float s,
                             const float *yd, float SO, float OD, float scale, float ddy, int nx,
                             int ny, int na) {
  const float zd = 0.0f;
  const ViewGeo G = with_constants(ViewGeo{c, s, SO, OD, scale, ddy, ddy, 1.0f, yd, &zd});
  const Dims D{nx, ny, 1, na, 1};
  std::vector<float4> tA(na);
  for (int ia = 0; ia < na; ia++) {
    tA[ia] = ray_tab_a(G, yd[ia]);
    if (tA[ia].x == 0.0f || tA[ia].y == 0.0f) return -1;
  }
  const size_t N = (size_t)nx * ny;
  auto pairs = [&](size_t vi, int &first, int &cnt, VoxelWin &w) {
    w = voxel_window(G, D, (int)(vi % nx), (int)(vi / nx), 0);
    int lo = w.a0, hi = w.b0 <= w.b1 ? w.a1 : w.a0 - 1, slo, shi;
    if (shadow_bins(G, D, w.xc, w.yc, slo, shi)) {
      lo = lo > slo ? lo : slo;
      hi = hi < shi ? hi : shi;
    }
    cnt = lo <= hi ? hi - lo + 1 : 0;
    first = cnt ? w.b0 * na + lo : 0;
  };
  int K = 0, first, cnt;
  VoxelWin w;
  for (size_t vi = 0; vi < N; vi++) {
    pairs(vi, first, cnt, w);
    K = cnt > K ? cnt : K;
  }
  K += K & 1;
  // a word past the table, and words that no voxel fills, would show in the sums
  std::vector<float> tab((2 + K) * N, __int_as_float_hd(0x7fc00000));
  for (size_t vi = 0; vi < N; vi++) {
    pairs(vi, first, cnt, w);
    const float rx = G.cos_phi * (-G.SO) - w.xc, ry = G.sin_phi * (-G.SO) - w.yc;
    float sum = 0.f;
    for (int k = 0; k < cnt; k++) {
      const float l = chord_planar_bf(tA[first % na + k], rx, ry, 1.0f);
      if (2 * N + chord_word(N, (unsigned)vi, k) >= tab.size()) return -2;
      tab[2 * N + chord_word(N, (unsigned)vi, k)] = l;
      sum += l;
    }
    const int head = cnt << 24 | first;
    memcpy(&tab[2 * vi], &head, 4);
    tab[2 * vi + 1] = sum;
  }
  for (size_t vi = 0; vi < N; vi++) {
    int head;
    memcpy(&head, &tab[2 * vi], 4);
    float acc = 0.f;
    for (int k = 0; k < (int)((unsigned)head >> 24); k++)
      acc += tab[2 * N + chord_word(N, (unsigned)vi, k)] * yv[(head & 0xffffff) + k];
    x[vi] = acc * scale;
    sc[vi] = tab[2 * vi + 1] * scale;
  }
  return K;
}
