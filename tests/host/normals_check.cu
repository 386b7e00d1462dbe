// normals_check.cu -- where unit_normals_mask (mhc_sweep.cuh) says that the
// initial outer normals along an axis are exactly (-1, 1), the general
// formula (outer_normals) gives exactly those for every cell of the mesh:
// 2D and 3D meshes of odd sizes, origins far from a tiny mesh included (where
// the mask must not be set).  Exit status 0 when that holds.
#include <cstdio>
#include "mhc_sweep.cuh"
using namespace mhc;

template <int DIM, int D>
bool all_unit(const Mesh& M) {
  const int n[3] = {M.ncx, M.ncy, M.ncz};
  constexpr int A0 = D == 0 ? 1 : 0, A1 = D == 2 ? 1 : 2;
  for (int p = 0; p < n[D]; ++p)
    for (int a = 0; a < n[A0]; ++a)
      for (int b = 0; b < n[A1]; ++b) {
        double back, front;
        outer_normals<DIM, D>(M, p, a, b, back, front);
        if (back != -1. || front != 1.) return false;
      }
  return true;
}

int main() {
  long checked = 0, bad = 0, set = 0, unset = 0;
  const double origins[] = {0., -0.5, 1.0 / 3.0, 1e3, 1e6, -1e9};
  const double lengths[] = {1.0, 0.1, 1.2, 1e-6, 1e-3, 7e4};
  const int sizes[][3] = {{5, 3, 4}, {31, 7, 9}, {1, 17, 2}, {64, 33, 1}, {97, 5, 11}};
  for (double o : origins)
    for (double L : lengths)
      for (auto& s : sizes)
        for (int dim = 2; dim <= 3; ++dim) {
          Mesh M{};
          M.dim = dim;
          M.ncx = s[0]; M.ncy = s[1]; M.ncz = dim == 3 ? s[2] : 1;
          M.o[0] = o; M.o[1] = -o; M.o[2] = 0.5 * o;
          M.h[0] = L / s[0]; M.h[1] = 0.3 * L / s[1]; M.h[2] = dim == 3 ? 2. * L / s[2] : 0.;
          const int mask = unit_normals_mask(M);
          const bool unit[3] = {dim == 2 ? all_unit<2, 0>(M) : all_unit<3, 0>(M),
                                dim == 2 ? all_unit<2, 1>(M) : all_unit<3, 1>(M), dim == 3 && all_unit<3, 2>(M)};
          for (int D = 0; D < dim; ++D) {
            const bool m = (mask >> D) & 1;
            if (m && !unit[D] && bad++ < 10) printf("o=%g L=%g n=%d,%d,%d D=%d\n", o, L, s[0], s[1], s[2], D);
            ++checked;
            if (m) ++set;
            else if (!unit[D]) ++unset;
          }
        }
  printf("checked %ld axes, mismatches %ld, set %ld, not unit %ld\n", checked, bad, set, unset);
  return bad != 0 || set == 0 || unset == 0;
}
