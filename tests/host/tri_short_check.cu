// Host driver for tests/test_tri_short_host.py: the short FP64 forms of the
// N-view and algebraic estimators beside the general ones
// (csrc/gbtri_track.cuh), as host code; no GPU is used.
//
// Input:  int64 nt, int64 ncam, double P[ncam][12], int64 off[nt+1],
//         uint32 cam[no], double xy[no][2]
// Output: double general[2][nt][4], short[2][nt][4], taken[2][nt] (1 where
//         the short form accepted the track); N-view, then algebraic.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "gbtri_track.cuh"

struct HostViews {
  const double* P;
  const uint32_t* cam;
  const double* xy;
  int64_t b;
  __host__ __device__ void operator()(int j, const double** Pj, double* x, double* y) const {
    *Pj = P + 12 * (int64_t)cam[b + j];
    *x = xy[2 * (b + j)];
    *y = xy[2 * (b + j) + 1];
  }
};

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  FILE* in = fopen(argv[1], "rb");
  FILE* out = fopen(argv[2], "wb");
  if (!in || !out) return 2;
  int64_t nt, ncam;
  if (fread(&nt, 8, 1, in) != 1 || fread(&ncam, 8, 1, in) != 1) return 2;
  std::vector<double> P(12 * ncam);
  std::vector<int64_t> off(nt + 1);
  if (fread(P.data(), 8, P.size(), in) != P.size() || fread(off.data(), 8, off.size(), in) != off.size()) return 2;
  const int64_t no = off[nt];
  std::vector<uint32_t> cam(no);
  std::vector<double> xy(2 * no);
  if (fread(cam.data(), 4, cam.size(), in) != cam.size() || fread(xy.data(), 8, xy.size(), in) != xy.size()) return 2;
  std::vector<double> general(8 * nt, 0.0), brief(8 * nt, 0.0), taken(2 * nt, 0.0);
  for (int64_t t = 0; t < nt; ++t) {
    const HostViews v{P.data(), cam.data(), xy.data(), off[t]};
    const int n = (int)(off[t + 1] - off[t]);
    gbba::nview_track<double, true>(v, n, &general[4 * t]);
    gbba::algebraic_track<double>(v, n, &general[4 * (nt + t)]);
    taken[t] = gbba::nview_track_short(v, n, &brief[4 * t]) ? 1.0 : 0.0;
    taken[nt + t] = gbba::algebraic_track_short(v, n, &brief[4 * (nt + t)]) ? 1.0 : 0.0;
  }
  fwrite(general.data(), 8, general.size(), out);
  fwrite(brief.data(), 8, brief.size(), out);
  fwrite(taken.data(), 8, taken.size(), out);
  fclose(out);
  return 0;
}
