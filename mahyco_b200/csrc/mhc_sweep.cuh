// mhc_sweep.cuh -- one direction of the ADI remap (cells, then nodes).
//
// Two forms of the same arithmetic: the x sweeps (and every sweep of the wide
// stencils) one warp per line, without shared memory or barriers; the y and z
// sweeps of the classical limiters through a shared-memory tile that turns
// their strided lines into runs of consecutive x.
//
// A warp holds 32 consecutive cells along the sweep direction, one per
// lane; every intermediate of the reference -- phi, face gradient, limited
// cell gradient, upwind face value, face flux -- is computed once per cell
// or face and handed to the neighbour lane by a shuffle.  The 4 warps of a
// block hold neighbouring transverse columns, so for the y and z sweeps the
// block reads whole 32-byte sectors of every row it touches.
//
// Arithmetic and operation order are those of computeGradPhiFace,
// computeGradPhiCell, computeUpwindFaceQuantitiesForProjection and
// computeUremap (RemapADIService.cc:119-575, UtilesRemap.cc:108-120,
// 325-357); face quantities of the Lagrangian mesh (PrepareRemap.cc:18-59)
// are rebuilt from the node positions.  The initial face normals of the
// cartesian grid are unit axis vectors, so dot(., n) is the D component.
#pragma once
#include <vector>

#include "mhc_kernels.cuh"

namespace mhc {

struct SweepArgs {
  const double* Uin;
  double* Uout;
  int first;
  int limiter;
  int simple_pente;   // projection-simple-pente (generalised limiters)
  int first_remap;    // first remap of the run: every cell counts as pure
  int part, parts;    // classical limiters: this block sweeps the part-th share of the variables
};

// the variables [v0, v1) of a share of NV (SHARE: a launch over one case whose
// blocks split the variables; otherwise all of them)
template <int NV, bool SHARE>
__device__ __forceinline__ void share_of(const SweepArgs& A, int& v0, int& v1) {
  v0 = SHARE ? NV * A.part / A.parts : 0;
  v1 = SHARE ? NV * (A.part + 1) / A.parts : NV;
}

// face node q (in the order of the reference face, smallest node id first)
// of the face normal to D whose lowest node is (i, j, k)
template <int DIM, int D>
__host__ __device__ __forceinline__ void face_node_ijk2(int i, int j, int k, int q, int& a, int& b, int& cz) {
  a = i; b = j; cz = k;
  if (DIM == 2) {
    if (D == 0) b += q; else a += q;
    return;
  }
  int s1 = (q == 1 || q == 2), s2 = (q == 2 || q == 3);
  if (D == 0) { b += s1; cz += s2; }
  else if (D == 1) { a += s1; cz += s2; }
  else { a += s1; b += s2; }
}


constexpr int SW_LANES = 32; // cells along D per warp
#ifndef MHC_SW_ROWS
#define MHC_SW_ROWS 4
#endif
constexpr int SW_ROWS = MHC_SW_ROWS;  // warps (transverse rows) per block
constexpr int SW_THREADS = SW_LANES * SW_ROWS;
constexpr int XOUT = 27;     // cells written per warp (lanes 2 .. 28)
constexpr int XOUT_W = 26;   // wide stencils (3 halo lanes each side): lanes 3 .. 28

// ---------------------------------------------------------------------------
// Initial-grid quantities of the outer normals, one coordinate at a time.
// Node coordinate A of the initial grid depends on the node index along A
// only, so the sums of the reference (cell centre over the local nodes,
// face centre over the face nodes, in their orders) are rebuilt from the
// two coordinate values c0 (offset 0) and c1 (offset 1).
// ---------------------------------------------------------------------------
template <int DIM>
__host__ __device__ __forceinline__ double grid_coord(const Mesh& M, int A, int idx) {
  return (DIM == 2 && A == 2) ? 0. : M.o[A] + idx * M.h[A];
}

// component A of the initial cell centre (wc * sum over local nodes)
template <int DIM, int A>
__host__ __device__ __forceinline__ double cc0_comp(const Mesh& M, int idx) {
  if (DIM == 2 && A == 2) return 0.;
  const double c0 = grid_coord<DIM>(M, A, idx), c1 = grid_coord<DIM>(M, A, idx + 1);
  double s = 0.;
#pragma unroll
  for (int l = 0; l < (DIM == 3 ? 8 : 4); ++l) {
    int da, db, dc;
    local_node_offset(l, da, db, dc);
    s += (A == 0 ? da : (A == 1 ? db : dc)) ? c1 : c0;
  }
  return (DIM == 2 ? .25 : .125) * s;
}

// component A of the initial centre of a face normal to D (sum over the
// face nodes of wf * coordinate)
template <int DIM, int D, int A>
__host__ __device__ __forceinline__ double fc0_comp(const Mesh& M, int idx) {
  if (DIM == 2 && A == 2) return 0.;
  const double wf = DIM == 2 ? .5 : .25;
  const double c0 = grid_coord<DIM>(M, A, idx), c1 = grid_coord<DIM>(M, A, idx + 1);
  double s = 0.;
#pragma unroll
  for (int q = 0; q < (DIM == 3 ? 4 : 2); ++q) {
    int a, b, cz;
    face_node_ijk2<DIM, D>(0, 0, 0, q, a, b, cz);
    const int off = A == 0 ? a : (A == 1 ? b : cz);
    s = s + wf * ((A == D) ? c0 : (off ? c1 : c0));
  }
  return s;
}

// D component of the unit outer normal: diff_D / |diff| with the sum of
// squares in x, y, z order
template <int D>
__host__ __device__ __forceinline__ double unit_comp(double dD, double t0, double t1) {
  // t0, t1: transverse differences in increasing axis order
  double ss;
  if (D == 0) ss = dD * dD + t0 * t0 + t1 * t1;
  else if (D == 1) ss = t0 * t0 + dD * dD + t1 * t1;
  else ss = t0 * t0 + t1 * t1 + dD * dD;
  return dD / sqrt(ss);
}

// D components of the outer normals of a cell's back and front faces along D
// (index p along D, ta and tb the transverse indices in increasing axis order)
template <int DIM, int D>
__host__ __device__ __forceinline__ void outer_normals(const Mesh& M, int p, int ta, int tb, double& ondB,
                                                       double& ondF) {
  constexpr int A0 = D == 0 ? 1 : 0, A1 = D == 2 ? 1 : 2;
  const double t0 = fc0_comp<DIM, D, A0>(M, ta) - cc0_comp<DIM, A0>(M, ta);
  const double t1 = fc0_comp<DIM, D, A1>(M, tb) - cc0_comp<DIM, A1>(M, tb);
  const double cc0 = cc0_comp<DIM, D>(M, p);
  ondB = unit_comp<D>(fc0_comp<DIM, D, D>(M, p) - cc0, t0, t1);
  ondF = unit_comp<D>(fc0_comp<DIM, D, D>(M, p + 1) - cc0, t0, t1);
}

// Whether outer_normals is exactly (-1, 1) for every cell of the mesh: with
// the largest transverse squares a, b of the mesh, d^2 + a + b rounds to d^2
// for every face (rounding is monotonic, so it does for the smaller squares
// too) and the root and quotient give 1.  Holds unless the origin is so far
// from a tiny mesh that the rounding of its coordinates shows.  The sweeps
// then skip the normals: about 110 of their 390 FP64 operations per cell in
// 3D with one material (Mesh::unit_normals, evaluated once per case).
// cc: the initial cell centres along every axis (cc0_comp).
template <int DIM, int D>
inline bool outer_normals_unit(const Mesh& M, const std::vector<double> (&cc)[3]) {
  constexpr int A0 = D == 0 ? 1 : 0, A1 = D == 2 ? 1 : 2;
  const int n[3] = {M.ncx, M.ncy, M.ncz};
  double a = 0., b = 0.;
  for (int i = 0; i < n[A0]; ++i) {
    const double t = fc0_comp<DIM, D, A0>(M, i) - cc[A0][i];
    if (!(t * t <= a)) a = t * t;
  }
  for (int i = 0; i < n[A1]; ++i) {
    const double t = fc0_comp<DIM, D, A1>(M, i) - cc[A1][i];
    if (!(t * t <= b)) b = t * t;
  }
  for (int p = 0; p < n[D]; ++p) {
    for (int front = 0; front < 2; ++front) {
      const double d = fc0_comp<DIM, D, D>(M, p + front) - cc[D][p], dd = d * d;
      const double ss = D == 0 ? dd + a + b : (D == 1 ? a + dd + b : a + b + dd);
      if (ss != dd || d / std::sqrt(dd) != (front ? 1. : -1.)) return false;
    }
  }
  return true;
}
template <int DIM>
inline int unit_normals_of(const Mesh& M) {
  std::vector<double> cc[3];
  cc[0].resize(M.ncx);
  cc[1].resize(M.ncy);
  cc[2].resize(M.ncz);
  for (int i = 0; i < M.ncx; ++i) cc[0][i] = cc0_comp<DIM, 0>(M, i);
  for (int j = 0; j < M.ncy; ++j) cc[1][j] = cc0_comp<DIM, 1>(M, j);
  for (int k = 0; k < M.ncz; ++k) cc[2][k] = cc0_comp<DIM, 2>(M, k);
  int m = (outer_normals_unit<DIM, 0>(M, cc) ? 1 : 0) | (outer_normals_unit<DIM, 1>(M, cc) ? 2 : 0);
  if constexpr (DIM == 3) m |= outer_normals_unit<3, 2>(M, cc) ? 4 : 0;
  return m;
}
inline int unit_normals_mask(const Mesh& M) { return M.dim == 2 ? unit_normals_of<2>(M) : unit_normals_of<3>(M); }

// the same in the sweeps
template <int DIM, int D>
__device__ __forceinline__ void sweep_normals(const Mesh& M, int p, int ta, int tb, double& ondB, double& ondF) {
  if ((M.unit_normals >> D) & 1) {
    ondB = -1.;
    ondF = 1.;
  } else {
    outer_normals<DIM, D>(M, p, ta, tb, ondB, ondF);
  }
}

// face-node slot q (face_node_ijk2 order) of local node l of a cell, and
// whether l sits on the front plane along D
template <int DIM, int D>
__device__ __forceinline__ void local_to_plane(int l, int& q, int& front) {
  int da, db, dc;
  local_node_offset(l, da, db, dc);
  int s1, s2;
  if (D == 0) { front = da; s1 = db; s2 = dc; }
  else if (D == 1) { front = db; s1 = da; s2 = dc; }
  else { front = dc; s1 = da; s2 = db; }
  if (DIM == 2) s2 = 0;
  q = s2 ? (s1 ? 2 : 3) : (s1 ? 1 : 0);
}

// Lagrangian plane data: the D coordinates of the face nodes, and the face
// centre, normal velocity and length of the face (PrepareRemap.cc:18-59)
template <int DIM> struct Plane {
  double xd[DIM == 3 ? 4 : 2];
  double fc, un, L;
};

template <int DIM, int D>
__device__ __forceinline__ void load_plane(const Mesh& M, const Fields& F, int i, int j, int k, Plane<DIM>& P) {
  constexpr int NQ = DIM == 3 ? 4 : 2;
  const double wf = DIM == 2 ? .5 : .25;
  const double* vD = F.fv[D];  // the node velocities, or (CSTS) their means at n and n+1
  long long fn[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    int a, b, cz;
    face_node_ijk2<DIM, D>(i, j, k, q, a, b, cz);
    fn[q] = node_id(M, a, b, cz);
  }
  double vm = 0.;
  P.fc = 0.;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    P.xd[q] = __ldg(F.Xn[D] + fn[q]);
    P.fc = P.fc + wf * P.xd[q];
    vm = vm + __ldg(vD + fn[q]);
  }
  P.un = wf * vm;
  if (DIM == 3) {
    R3 x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[q].x = D == 0 ? P.xd[q] : __ldg(F.Xn[0] + fn[q]);
      x[q].y = D == 1 ? P.xd[q] : __ldg(F.Xn[1] + fn[q]);
      x[q].z = D == 2 ? P.xd[q] : __ldg(F.Xn[2] + fn[q]);
    }
    const R3 v1 = x[2] - x[0], v2 = x[3] - x[1];
    if (D == 0) P.L = 0.5 * fabs(produit(v1.y, v2.z, v1.z, v2.y));
    else if (D == 1) P.L = 0.5 * fabs(produit(v2.x, v1.z, v2.z, v1.x));
    else P.L = 0.5 * fabs(produit(v1.x, v2.y, v1.y, v2.x));
  } else {
    const double* Xt = F.Xn[1 - D];
    P.L = fabs(__ldg(Xt + fn[1]) - __ldg(Xt + fn[0]));
  }
}

// Lagrangian cell centre along D from its back (B) and front (Fr) planes,
// summed in local node order
template <int DIM, int D>
__device__ __forceinline__ double centre_from_planes(const Plane<DIM>& B, const Plane<DIM>& Fr) {
  double s = 0.;
#pragma unroll
  for (int l = 0; l < (DIM == 3 ? 8 : 4); ++l) {
    int q, front;
    local_to_plane<DIM, D>(l, q, front);
    s += front ? Fr.xd[q] : B.xd[q];
  }
  return (DIM == 2 ? .25 : .125) * s;
}

// ---------------------------------------------------------------------------
// Lane layout of a sweep along D over an nx x ny x nz array of cells or
// nodes.  The array is cut into lines along D; consecutive lines are
// concatenated so that every warp window holds `out` written elements plus
// `hl` halo elements before them (2, or 3 for the wide stencils) and the
// rest after them, whatever the line length.
//  * D = 0: lines are consecutive in memory; window w = vbx * SW_ROWS + row
//    covers flat positions [w*out - hl, w*out - hl + 32).
//  * D = 1, 2: warp `row` of the block owns x column ta = vbx * SW_ROWS +
//    row and walks the lines of that column (slow transverse index tb, then
//    p along D) in windows vby; the 4 warps of a block hold neighbouring x
//    columns at the same positions, so each row of the block is one or two
//    32-byte sectors, and consecutive blocks (vbx fastest) hold the
//    neighbouring columns, so the SMs that run them at the same time read
//    whole DRAM bursts together.
// Returns false when the lane holds nothing; p is the index along D and
// (ta, tb) the transverse indices in increasing axis order.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ bool sweep_lane(int nx, int ny, int nz, int out, int hl, int vbx, int vby, int lane,
                                           int row, int& i, int& j, int& k, int& p, int& ta, int& tb) {
  i = j = k = p = ta = tb = 0;
  // positions in unsigned 32-bit arithmetic (a case has < 2^31 cells)
  if (D == 0) {
    const int g = (vbx * SW_ROWS + row) * out - hl + lane;
    if (g < 0 || g >= nx * ny * nz) return false;
    const unsigned r = (unsigned)g / (unsigned)nx;
    i = (int)((unsigned)g - r * (unsigned)nx);
    k = (int)(r / (unsigned)ny);
    j = (int)(r - (unsigned)k * (unsigned)ny);
    p = i; ta = j; tb = k;
    return true;
  }
  const int nd = D == 1 ? ny : nz, nb = D == 1 ? nz : ny;
  ta = vbx * SW_ROWS + row;
  const int g = vby * out - hl + lane;
  if (ta >= nx || g < 0 || g >= nb * nd) return false;
  tb = (int)((unsigned)g / (unsigned)nd);
  p = g - tb * nd;
  i = ta;
  if (D == 1) { j = p; k = tb; }
  else { j = tb; k = p; }
  return true;
}

// the whole warp holds nothing (warp-uniform test, before any shuffle)
template <int D>
__device__ __forceinline__ bool sweep_warp_empty(int nx, int ny, int nz, int out, int hl, int vbx, int vby, int row) {
  if (D == 0) return (vbx * SW_ROWS + row) * out - hl >= nx * ny * nz;
  const int nd = D == 1 ? ny : nz, nb = D == 1 ? nz : ny;
  return vbx * SW_ROWS + row >= nx || vby * out - hl >= nb * nd;
}

// D coordinates of the face nodes of the node plane whose lowest node is
// (i, j, k)
template <int DIM, int D>
__device__ __forceinline__ void load_plane_xd(const Mesh& M, const Fields& F, int i, int j, int k, Plane<DIM>& P) {
#pragma unroll
  for (int q = 0; q < (DIM == 3 ? 4 : 2); ++q) {
    int a, b, cz;
    face_node_ijk2<DIM, D>(i, j, k, q, a, b, cz);
    P.xd[q] = __ldg(F.Xn[D] + node_id(M, a, b, cz));
  }
}

// all coordinates of the face nodes of the node plane whose lowest node is
// (i, j, k); z = 0 in 2D
template <int DIM, int D>
__device__ __forceinline__ void load_plane_full(const Mesh& M, const Fields& F, int i, int j, int k,
                                                double (&x)[DIM == 3 ? 4 : 2][3]) {
#pragma unroll
  for (int q = 0; q < (DIM == 3 ? 4 : 2); ++q) {
    int a, b, cz;
    face_node_ijk2<DIM, D>(i, j, k, q, a, b, cz);
    const long long n = node_id(M, a, b, cz);
    x[q][0] = __ldg(F.Xn[0] + n);
    x[q][1] = __ldg(F.Xn[1] + n);
    x[q][2] = DIM == 3 ? __ldg(F.Xn[2] + n) : 0.;
  }
}

__device__ __forceinline__ double norm3(double a, double b, double c) { return sqrt(a * a + b * b + c * c); }

// Width of the lane's cell along D (m_h_cell_lagrange,
// RemapADIService.cc:141-143): distance from the Lagrangian cell centre to
// the centres of its inner faces of direction D, back face first.  Every
// lane of the warp calls it (the front plane comes from lane + 1).
template <int DIM, int D>
__device__ __forceinline__ double lane_cell_width(const Mesh& M, const Fields& F, bool ok, int i, int j, int k,
                                                  int p, int nd) {
  constexpr int NQ = DIM == 3 ? 4 : 2;
  constexpr unsigned FULL = 0xffffffffu;
  double b[NQ][3], f[NQ][3];
  if (ok) load_plane_full<DIM, D>(M, F, i, j, k, b);
  else {
#pragma unroll
    for (int q = 0; q < NQ; ++q) b[q][0] = b[q][1] = b[q][2] = 0.;
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int a = 0; a < 3; ++a) f[q][a] = __shfl_down_sync(FULL, b[q][a], 1);
  // the front plane is loaded at the end of a line, and by the last lane,
  // whose next cell lies outside the warp
  if (ok && (p == nd - 1 || (threadIdx.x % SW_LANES) == SW_LANES - 1))
    load_plane_full<DIM, D>(M, F, D == 0 ? i + 1 : i, D == 1 ? j + 1 : j, D == 2 ? k + 1 : k, f);
  if (!ok) return 0.;
  const double wf = DIM == 2 ? .5 : .25, wc = DIM == 2 ? .25 : .125;
  double cc[3], fb[3], ff[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double s = 0.;
#pragma unroll
    for (int l = 0; l < (DIM == 3 ? 8 : 4); ++l) {
      int q, front;
      local_to_plane<DIM, D>(l, q, front);
      s += front ? f[q][a] : b[q][a];
    }
    cc[a] = wc * s;
    fb[a] = ff[a] = 0.;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      fb[a] = fb[a] + wf * b[q][a];
      ff[a] = ff[a] + wf * f[q][a];
    }
  }
  double h = 0.;
  if (p > 0) h += norm3(fb[0] - cc[0], fb[1] - cc[1], fb[2] - cc[2]);
  if (p < nd - 1) h += norm3(ff[0] - cc[0], ff[1] - cc[1], ff[2] - cc[2]);
  return h;
}

// ---------------------------------------------------------------------------
// One variable of a classical cell sweep, one cell per lane along D: value,
// face gradient, limited gradient, upwind face value and flux, the neighbours'
// by shuffles.  What the lane knows about its cell and its two faces is set
// once; the variables then come in a rolled loop, which leaves registers for
// 8 blocks of 4 warps per SM (the sweeps are bound by the latency of their
// FP64 chains: 6 blocks of the same code are 9 % slower).  The quotients by
// the cell's divisor and by the distance of the centres share a reciprocal
// each (SharedDivisor); a warp with an operand out of its range divides.  A
// warp whose values are all zero (an absent material) or all equal (a flat
// field) leaves out what would come out as zero.
// ---------------------------------------------------------------------------
template <int DIM, int D, int LIM>
struct CellLane {
  bool ok, face_b, up_left;
  bool odd;               // a factor is not finite, or a divisor out of range: nothing is left out
  SharedDivisor den, dx;  // the cell's divisor; distance to the centre of the cell behind
  double fu;              // (ordre-projection - 1) x distance from the upwind cell's centre to the back face
  double cB, cF;          // outer normal x normal velocity x length x deltat of the back / front face, 0 at the ends
  double ondB, ondF;
  // generalised limiters
  int limiter, simple_pente;
  bool first, last;       // ends of the line
  double hw, hw_l, hw_r;

  // the lane's faces: un, L of the back face and fc its centre, xc / xc_l the
  // centres of the own cell and of the one behind
  __device__ __forceinline__ void set_faces(double dt, int order2, double fc, double xc, double xc_l, double un,
                                            double L, double divisor) {
    constexpr unsigned FULL = 0xffffffffu;
    const bool face_f = __shfl_down_sync(FULL, face_b, 1) && (threadIdx.x % SW_LANES) < 31;
    const double un_r = __shfl_down_sync(FULL, un, 1), L_r = __shfl_down_sync(FULL, L, 1);
    const double dxb = xc - xc_l;
    up_left = un * dxb > 0.0;
    fu = order2 * (fc - (up_left ? xc_l : xc));
    cB = face_b ? ondB * un * L * dt : 0.;
    cF = face_f ? ondF * un_r * L_r * dt : 0.;
    den.set(divisor);
    dx.set(face_b ? dxb : 1.);
    constexpr double TOP = 1.7976931348623157e308;
    odd = den.y == 0. || dx.y == 0. || !(fabs(fu) <= TOP && fabs(cB) <= TOP && fabs(cF) <= TOP);
  }

  // fluxes of the variable of value u (0 on lanes without a cell) through the
  // back and front faces, out of the cell; false: all zero in this warp
  __device__ __forceinline__ bool fluxes(double u, double& fB, double& fF) const {
    constexpr unsigned FULL = 0xffffffffu;
    fB = fF = 0.;
    if (!__any_sync(FULL, u != 0. || odd)) return false;
    bool fine = true;
    double phi = den.q(u, fine);
    if (__any_sync(FULL, !fine)) phi = div_rn(u, den.b);
    const double phi_l = __shfl_up_sync(FULL, phi, 1);
    const double diff = phi - phi_l;
    double up = up_left ? phi_l : phi;  // upwind value
    if (__any_sync(FULL, (LIM != LIM_ORDER1 && face_b && diff != 0.) || odd)) {
      fine = true;
      double gf = face_b ? dx.q(diff, fine) : 0.;
      if (__any_sync(FULL, !fine)) gf = face_b ? div_rn(diff, dx.b) : 0.;
      const double gf_r = __shfl_down_sync(FULL, gf, 1);
      double gr;
      if constexpr (LIM == LIM_GEN) {
        // back / front neighbours, the cell itself at the line ends
        const double phi_r = __shfl_down_sync(FULL, phi, 1);
        const double ym = first ? phi : phi_l, yp = last ? phi : phi_r;
        gr = ok ? generalized_gradient(limiter, gf_r, gf, yp, ym, hw, hw_r, hw_l, simple_pente) : 0.;
      } else {
        gr = LIM != LIM_ORDER1 ? limited_gradient_t<LIM == LIM_ORDER1 ? 0 : LIM>(gf, gf_r) : 0.;
      }
      const double gr_l = __shfl_up_sync(FULL, gr, 1);
      up = up + fu * (up_left ? gr_l : gr);
    }
    const double pf = face_b ? up : 0.;
    const double pf_r = __shfl_down_sync(FULL, pf, 1);
    fB = cB * pf;
    fF = cF * pf_r;
    return true;
  }
  // dual mass flux of a mass variable
  __device__ __forceinline__ double dual(double fB, double fF) const { return 0.5 * fB * ondB + 0.5 * fF * ondF; }
};

// ---------------------------------------------------------------------------
// Cell sweep along D with warp shuffles.  A warp holds 32 consecutive cells
// along D (lane l: cell x0 - 2 + l), loads the back node plane of each and
// takes the front plane from lane l+1; stencil neighbours come from lanes
// l-1 / l+1.  Lanes 2 .. XOUT+1 write.  Virtual block: x = window index
// along D, y = group of SW_ROWS rows.  Rows are the transverse cells with
// the lowest transverse axis fastest, so the warps of a block read
// neighbouring columns and share L1 sectors.
// ---------------------------------------------------------------------------
// XV: further projected variables after the pseudo-viscosity (the
// deviator and plastic strains of an elasto-plastic case), remapped like it
template <int DIM, int NE, int D, int LIM, bool SHARE, int XV = 0>
__device__ __forceinline__ void body_sweep_cells_lanes(const Mesh& M, const Fields& F, const SweepArgs& A,
                                                       int vbx, int vby) {
  constexpr int NV = 3 * NE + 1 + XV;
  constexpr int NQ = DIM == 3 ? 4 : 2;
  constexpr unsigned FULL = 0xffffffffu;
  const long long N = M.ncell;
  const int lane = threadIdx.x % SW_LANES, row = threadIdx.x / SW_LANES;
  const int nd = D == 0 ? M.ncx : (D == 1 ? M.ncy : M.ncz);
  if (sweep_warp_empty<D>(M.ncx, M.ncy, M.ncz, XOUT, 2, vbx, vby, row)) return;  // whole warp leaves together
  int i, j, k, p, ta, tb;
  const bool ok = sweep_lane<D>(M.ncx, M.ncy, M.ncz, XOUT, 2, vbx, vby, lane, row, i, j, k, p, ta, tb);
  const bool out = ok && lane >= 2 && lane < 2 + XOUT;
  const double dt = F.s->dt;
  const int order2 = LIM == LIM_ORDER1 ? 0 : 1;  // ordre-projection - 1
  const double* __restrict__ Uin = A.Uin;
  // back node plane of the own cell; the front plane is the back plane of
  // the next lane, except at the end of a line
  Plane<DIM> back;
  if (ok) load_plane<DIM, D>(M, F, i, j, k, back);
  else {
#pragma unroll
    for (int q = 0; q < NQ; ++q) back.xd[q] = 0.;
    back.fc = back.un = back.L = 0.;
  }
  Plane<DIM> front;
#pragma unroll
  for (int q = 0; q < NQ; ++q) front.xd[q] = __shfl_down_sync(FULL, back.xd[q], 1);
  if (ok && p == nd - 1)
    load_plane_xd<DIM, D>(M, F, D == 0 ? i + 1 : i, D == 1 ? j + 1 : j, D == 2 ? k + 1 : k, front);
  CellLane<DIM, D, LIM> K;
  K.ok = ok;
  long long c = 0;
  double den = 1., xc = 0.;
  K.ondB = K.ondF = 0.;
  if (ok) {
    c = cell_id(M, i, j, k);
    if (A.first) {
      den = __ldg(F.V + c);
    } else {
      den = 0.;
#pragma unroll
      for (int q = 0; q < NE; ++q) den += __ldg(Uin + q * N + c);
    }
    xc = centre_from_planes<DIM, D>(back, front);
    if (out) sweep_normals<DIM, D>(M, p, ta, tb, K.ondB, K.ondF);
  }
  int v0, v1;
  share_of<NV, SHARE>(A, v0, v1);
  const double* src = Uin + v0 * N + c;
  double u = ok ? __ldg(src) : 0.;
  if constexpr (LIM == LIM_GEN) {
    // widths of the own and neighbouring cells
    K.hw = lane_cell_width<DIM, D>(M, F, ok, i, j, k, p, nd);
    K.hw_l = __shfl_up_sync(FULL, K.hw, 1);
    K.hw_r = __shfl_down_sync(FULL, K.hw, 1);
    if (p == 0) K.hw_l = K.hw;
    if (p == nd - 1) K.hw_r = K.hw;
    K.limiter = A.limiter;
    K.simple_pente = A.simple_pente;
    K.first = p == 0;
    K.last = p == nd - 1;
  }
  const double fc = back.fc, un = back.un, L = back.L;  // back face of the cell
  const bool ok_l = __shfl_up_sync(FULL, ok, 1) && lane > 0 && p > 0;  // same line
  const double xc_l = __shfl_up_sync(FULL, xc, 1);
  K.face_b = ok && ok_l;                       // face between p-1 and p
  K.set_faces(dt, order2, fc, xc, xc_l, un, L, den);
  double* dst = A.Uout + v0 * N + c;
#pragma unroll 1
  for (int v = v0; v < v1; ++v) {
    // the next variable's value is on its way during this one's arithmetic
    src += N;
    const double u_next = (ok && v + 1 < v1) ? __ldg(src) : 0.;
    double fB, fF;
    K.fluxes(u, fB, fF);
    if (out) {
      double uo = u - (fB + fF);
      if (v >= NE && v < 3 * NE && uo < 0.) uo = 0.;  // masses and energies stay >= 0
      *dst = uo;
      if (v >= NE && v < 2 * NE) F.mflux[(v - NE) * N + c] = K.dual(fB, fF);
    }
    dst += N;
    u = u_next;
  }
}

// ---------------------------------------------------------------------------
// Pente-borne fluxes (UtilesRemap.cc:84-96 INTY, 190-312 computeY0 /
// computexgxd / computeygyd, 417-832 computeFluxPP / computeFluxPPPure):
// the flux of one variable out of a cell through its back (type 0) or front
// (type 1) face is the integral, over the length swept in deltat, of a
// three-piece reconstruction bounded by the neighbours.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void pb_y0(int id, double yp, double ym, double h0, double hp, double hm, int simple_pente,
                                      double& y0p, double& y0m) {
  y0p = 0.; y0m = 0.;
  if (id == 3 || id == 0) {
    y0p = yp; y0m = ym;
  } else if (id == 4 || id == 1) {
    y0p = ((h0 + hm) * yp + h0 * ym) / (2 * h0 + hm);
    y0m = ((h0 + hp) * ym + h0 * yp) / (2 * h0 + hp);
  } else if (id == 5 || id == 2) {
    const double a = amin(yp, ym), b = amax(yp, ym);
    double xp = (h0 * h0 + 3 * h0 * hm + 2 * hm * hm) * yp;
    double xm = (h0 * h0 + 3 * h0 * hp + 2 * hp * hp) * ym;
    xp += (h0 * h0 - h0 * hp - 2 * hp * hp + 2 * h0 * hm) * ym;
    xm += (h0 * h0 - h0 * hm - 2 * hm * hm + 2 * h0 * hp) * yp;
    xp /= (2 * h0 * h0 + 5 * h0 * hm + 2 * hm * hm - h0 * hp - 2 * hp * hp);
    xm /= (2 * h0 * h0 + 5 * h0 * hp + 2 * hp * hp - h0 * hm - 2 * hm * hm);
    y0p = amin(amax(xp, a), b);
    y0m = amin(amax(xm, a), b);
  } else if (id == 7) {
    y0p = (yp + ym) / 2.;
    y0m = (yp + ym) / 2.;
  } else if (id == 6) {
    y0p = ((h0 + hm + hp) * yp + h0 * ym) / (2 * h0 + hm + hp);
    y0m = ((h0 + hm + hp) * ym + h0 * yp) / (2 * h0 + hm + hp);
  }
  if (simple_pente) { y0p = yp; y0m = ym; }
}

// the fluxes of one variable out of a cell through its back (Fb) and front
// (Ff) faces, swept lengths pb and pf.  At an extremum (flat regions, absent
// materials) the flux is y0 times the swept length (formule 16), decided
// before the reconstruction, which those cells never read.  The three pieces
// are a rolled loop, as the variables of the sweep are: unrolled, the warps
// of a sweep waited for instructions (8.5 of 14 stalled cycles).
__device__ __forceinline__ void pb_fluxes(double y0, double yp, double ym, double h0, double hp, double hm,
                                          double grad, double pb, double pf, int lim, int simple_pente, double thr,
                                          double& Fb, double& Ff) {
  double y0p, y0m;
  pb_y0(lim, yp, ym, h0, hp, hm, simple_pente, y0p, y0m);
  // breaks of the reconstruction; half a cell where the divisor vanishes
  const double xd = +h0 * (fabs(y0p - yp) > thr ? pb_ratio_mid(y0 - yp, y0p - yp) : 1. / 2.);
  const double xg = -h0 * (fabs(y0m - ym) > thr ? pb_ratio_mid(y0 - ym, y0m - ym) : 1. / 2.);
  const double xtd = y0 + h0 / 2 * grad, xtg = y0 - h0 / 2 * grad;
  const double ad = amin(yp, 2. * y0m - ym), bd = amax(yp, 2. * y0m - ym);
  const double ag = amin(ym, 2. * y0p - yp), bg = amax(ym, 2. * y0p - yp);
  const double yd = amin(amax(xtd, ad), bd), yg = amin(amax(xtg, ag), bg);
  // upper and lower ends of the swept length of each face
  const double b1 = -h0 / 2. + pb, b0 = -h0 / 2., f1 = h0 / 2., f0 = h0 / 2. - pf;
  double x0 = -h0 / 2., v0 = ym, x1 = xg, v1 = yg, sb = 0., sf = 0.;
#pragma unroll 1
  for (int piece = 0; piece < 3; ++piece) {
    // integral of the piece (x0, v0) - (x1, v1) up to X (INTY)
    const double dx = x1 - x0, dv = v1 - v0;
    auto inty = [&](double X) {
      double flux = 0.;
      if (fabs(dx) > thr) {
        const double eta = pb_ratio01(X - x0, dx);
        flux = (v0 + 0.5 * eta * dv) * dx * eta;
      }
      return flux;
    };
    const double db = inty(b1) - inty(b0), df = inty(f1) - inty(f0);
    sb = piece == 0 ? db : sb + db;
    sf = piece == 0 ? df : sf + df;
    x0 = x1; v0 = v1;
    x1 = piece == 0 ? xd : h0 / 2.;
    v1 = piece == 0 ? yd : yp;
  }
  Fb = smax(sb, 0.);
  Ff = smax(sf, 0.);
}

// ---------------------------------------------------------------------------
// Cell sweep along D with the pente-borne fluxes (computeGradPhiCell,
// computeUpwindFaceQuantitiesForProjection, computeUremap with
// projection-pente-borne, RemapADIService.cc:196-266, 314-318, 419-530).
// The lane layout of the classical sweep (2 halo lanes).  Every lane computes
// the fluxes out of its cell through both faces; the value of the face
// between lanes l-1 and l is front(l-1) - back(l).  The projected values
// (phi) are the volume fraction, density and specific internal energy per
// environment and the pseudo-viscosity, read from phi_pb on the first sweep
// of a remap and rebuilt from the projected quantities on the others.
//
// Bound by the latency of its divisions and by its code size: one rolled loop
// over the variables, extrema (flat regions) before any division, and a
// division of the piecewise integrals only where the swept length ends inside
// a piece.  350 x 150 cells, three environments, superbeeG: 92.8 us a sweep
// before (variables and pieces unrolled, every quotient divided), 32.5 now.
// ---------------------------------------------------------------------------
template <int DIM, int NE, int D>
__device__ __forceinline__ void body_sweep_cells_pb(const Mesh& M, const Fields& F, const mhc_case_params& P,
                                                    const SweepArgs& A, int vbx, int vby) {
  constexpr int NV = 3 * NE + 1;
  constexpr int NQ = DIM == 3 ? 4 : 2;
  constexpr unsigned FULL = 0xffffffffu;
  const long long N = M.ncell;
  const int lane = threadIdx.x % SW_LANES, row = threadIdx.x / SW_LANES;
  const int nd = D == 0 ? M.ncx : (D == 1 ? M.ncy : M.ncz);
  if (sweep_warp_empty<D>(M.ncx, M.ncy, M.ncz, XOUT, 2, vbx, vby, row)) return;  // whole warp leaves together
  int i, j, k, p, ta, tb;
  const bool ok = sweep_lane<D>(M.ncx, M.ncy, M.ncz, XOUT, 2, vbx, vby, lane, row, i, j, k, p, ta, tb);
  const bool out = ok && lane >= 2 && lane < 2 + XOUT;
  const double dt = F.s->dt;
  const double thr = P.remap_threshold;
  const int fix = P.projection_pente_borne_debar_fix;
  const double* __restrict__ Uin = A.Uin;
  // per-thread slots: fluxes of the volumes and masses through both faces,
  // then the updated variables (indexed by the rolled loops below)
  __shared__ double pb_slots[(4 * NE + NV) * SW_THREADS];
  double* const s_vol = pb_slots + threadIdx.x;
  double* const s_mass = s_vol + 2 * NE * SW_THREADS;
  double* const s_out = s_vol + 4 * NE * SW_THREADS;
  Plane<DIM> back;
  if (ok) load_plane<DIM, D>(M, F, i, j, k, back);
  else {
#pragma unroll
    for (int q = 0; q < NQ; ++q) back.xd[q] = 0.;
    back.fc = back.un = back.L = 0.;
  }
  Plane<DIM> front;
#pragma unroll
  for (int q = 0; q < NQ; ++q) front.xd[q] = __shfl_down_sync(FULL, back.xd[q], 1);
  if (ok && p == nd - 1)
    load_plane_xd<DIM, D>(M, F, D == 0 ? i + 1 : i, D == 1 ? j + 1 : j, D == 2 ? k + 1 : k, front);
  long long c = 0;
  double sv = 0., xc = 0., ondB = 0., ondF = 0.;
  uint8_t mask = 0;
  if (ok) {
    c = cell_id(M, i, j, k);
    mask = F.mask[c];
    if (!A.first) {
#pragma unroll
      for (int q = 0; q < NE; ++q) sv += __ldg(Uin + q * N + c);
    }
    xc = centre_from_planes<DIM, D>(back, front);
    sweep_normals<DIM, D>(M, p, ta, tb, ondB, ondF);
  }
  // projected value of variable v in the lane's cell: kept from the Lagrange
  // phase on the first sweep, rebuilt from the projected quantities on the
  // others (the pseudo-viscosity is not rebuilt)
  auto phi_of = [&](int v) -> double {
    if (!ok) return 0.;
    if (A.first || v == NV - 1) return __ldg(F.phi_pb + v * N + c);
    const double u = __ldg(Uin + v * N + c);
    const double d = v < NE ? sv : __ldg(Uin + (v - NE) * N + c);
    return (v < NE || d != 0.) ? div_rn(u, d) : 0.;
  };
  // cell widths, the cell itself beyond the line ends
  const double hw = lane_cell_width<DIM, D>(M, F, ok, i, j, k, p, nd);
  double hw_l = __shfl_up_sync(FULL, hw, 1), hw_r = __shfl_down_sync(FULL, hw, 1);
  if (p == 0) hw_l = hw;
  if (p == nd - 1) hw_r = hw;
  // pure neighbourhood (projection-pente-borne-mixte): purity codes -2 mixed,
  // else the last environment with a positive volume fraction (-1: none)
  bool pure = false;
  if (P.projection_pente_borne_mixte) {
    int code = 0;
    if (ok && !A.first_remap) {
      int cnt = 0;
      code = -1;
#pragma unroll 1
      for (int q = 0; q < NE; ++q)
        if ((!A.first || ((mask >> q) & 1)) && phi_of(q) > 0.) { ++cnt; code = q; }
      if (cnt > 1) code = -2;
    }
    int code_l = __shfl_up_sync(FULL, code, 1), code_r = __shfl_down_sync(FULL, code, 1);
    if (p == 0) code_l = code;
    if (p == nd - 1) code_r = code;
    pure = code != -2 && code_l != -2 && code_r != -2 && code == code_l && code == code_r;
  }
  const int lim_g = (P.projection_limiteur_pure_id == 1 && pure) ? P.projection_limiteur_pure_id : A.limiter;
  const int lim_y = pure ? P.projection_limiteur_pure_id : A.limiter;
  const double un = back.un, L = back.L;  // back face of the cell
  const bool ok_l = __shfl_up_sync(FULL, ok, 1) && lane > 0 && p > 0;  // same line
  const double xc_l = __shfl_up_sync(FULL, xc, 1);
  const bool face_b = ok && ok_l;
  const bool face_f = __shfl_down_sync(FULL, face_b, 1) && lane < 31;
  const double un_r = __shfl_down_sync(FULL, un, 1), L_r = __shfl_down_sync(FULL, L, 1);
  const double dxb = xc - xc_l;
  // outgoing normal velocities and swept lengths of the back / front faces
  const double vb = ondB * un, vf = ondF * un_r;
  const double ppv_b = 0.5 * (vb + fabs(vb)) * dt, ppv_f = 0.5 * (vf + fabs(vf)) * dt;
  constexpr bool FRONT_FIRST = DIM == 2 && D == 0;
  // one rolled loop: the volume fluxes (step t < NE) come before anything is
  // updated, since the de-barring fix 1 divides by their sums; then every
  // variable in order, the volumes' fluxes read back
  double sfb = 0., sff = 0.;
  bool zb = false, zf = false;
#pragma unroll 1
  for (int t = 0; t < NV + NE; ++t) {
    const bool ahead = t < NE;
    const int v = ahead ? t : t - NE;
    double Fb, Ff, y0 = 0.;
    if (ahead || v >= NE) {
      y0 = phi_of(v);
      const double y_l = __shfl_up_sync(FULL, y0, 1), y_r = __shfl_down_sync(FULL, y0, 1);
      const double ym = p > 0 ? y_l : y0, yp = p < nd - 1 ? y_r : y0;
      const bool extremum = ((yp - y0) * (ym - y0)) >= 0.;
      Fb = ok ? y0 * ppv_b : 0.;
      Ff = ok ? y0 * ppv_f : 0.;
      if (__any_sync(FULL, ok && !extremum)) {
        const double gf = face_b ? div_rn(y0 - y_l, dxb) : 0.;
        const double gf_r = __shfl_down_sync(FULL, gf, 1);
        if (ok && !extremum) {
          const double gr = lim_g < 3
                                ? limited_gradient(lim_g, gf, gf_r)
                                : generalized_gradient(lim_g, gf_r, gf, yp, ym, hw, hw_r, hw_l, A.simple_pente);
          pb_fluxes(y0, yp, ym, hw, hw_r, hw_l, gr, ppv_b, ppv_f, lim_y, A.simple_pente, thr, Fb, Ff);
        }
      }
    } else {
      Fb = s_vol[v * SW_THREADS];
      Ff = s_vol[(NE + v) * SW_THREADS];
    }
    if (ahead) {
      s_vol[v * SW_THREADS] = Fb;
      s_vol[(NE + v) * SW_THREADS] = Ff;
      sfb += Fb;
      sff += Ff;
      if (t == NE - 1) {
        zb = (fix == 1 && !(fabs(sfb) > thr)) || ppv_b == 0.;
        zf = (fix == 1 && !(fabs(sff) > thr)) || ppv_f == 0.;
      }
      continue;
    }
    if (v >= NE && v < 2 * NE) {
      const int q = v - NE;
      const double vol_b = s_vol[q * SW_THREADS], vol_f = s_vol[(NE + q) * SW_THREADS];
      if (fix == 1 && !pure) { Fb = (Fb / sfb) * vol_b; Ff = (Ff / sff) * vol_f; }
      if (fix == 2 && !pure) { Fb = y0 * vol_b; Ff = y0 * vol_f; }
      s_mass[q * SW_THREADS] = Fb;
      s_mass[(NE + q) * SW_THREADS] = Ff;
    } else if (v >= 2 * NE && v < 3 * NE) {
      const int q = v - 2 * NE;
      const double mass_b = s_mass[q * SW_THREADS], mass_f = s_mass[(NE + q) * SW_THREADS];
      if (fix == 1) { Fb = (Fb / sfb) * mass_b; Ff = (Ff / sff) * mass_f; }
      if (fix == 2) { Fb = y0 * mass_b; Ff = y0 * mass_f; }
    }
    if (zb) Fb = 0.;
    if (zf) Ff = 0.;
    const double Ff_l = __shfl_up_sync(FULL, Ff, 1);
    const double pf = face_b ? Ff_l - Fb : 0.;  // face value: front flux of l-1 minus back flux of l
    const double pf_r = __shfl_down_sync(FULL, pf, 1);
    if (out) {
      const double fB = face_b ? ondB * L * pf : 0.;
      const double fF = face_f ? ondF * L_r * pf_r : 0.;
      double sumf = 0., du = 0.;
      if (FRONT_FIRST) {
        if (face_f) { sumf += fF; du += 0.5 * fF * ondF; }
        if (face_b) { sumf += fB; du += 0.5 * fB * ondB; }
      } else {
        if (face_b) { sumf += fB; du += 0.5 * fB * ondB; }
        if (face_f) { sumf += fF; du += 0.5 * fF * ondF; }
      }
      s_out[v * SW_THREADS] = __ldg(Uin + v * N + c) - sumf;
      if (v >= NE && v < 2 * NE) F.mflux[(v - NE) * N + c] = du;
    }
  }
  if (!out) return;
  // truncation of tiny volumes, masses and energies (with the dual
  // projection only, not in a sans-lagrange advection), then the clip of
  // negative masses and energies
  const bool trunc = !P.sans_lagrange;
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    double a = s_out[q * SW_THREADS], m = s_out[(NE + q) * SW_THREADS], e = s_out[(2 * NE + q) * SW_THREADS];
    if (trunc && a < 1. * thr) { a = 0.; m = 0.; e = 0.; }
    if (trunc && m < 1. * thr) { a = 0.; m = 0.; e = 0.; }
    if (trunc && e < 1. * thr) { a = 0.; m = 0.; e = 0.; }
    if (m < 0.) m = 0.;
    if (e < 0.) e = 0.;
    A.Uout[q * N + c] = a;
    A.Uout[(NE + q) * N + c] = m;
    A.Uout[(2 * NE + q) * N + c] = e;
  }
  A.Uout[(NV - 1) * N + c] = s_out[(NV - 1) * SW_THREADS];
}

// ---------------------------------------------------------------------------
// Third-order face value (Remap-ordre-3.cc:16-188: evaluate_grad,
// evaluate_ystar, evaluate_fm / evaluate_fp, the TVD interval bound of
// ComputeFluxOrdre3).  y[0..5], h[0..5]: values and widths of the cells
// b-2 .. f+2 around the face, repeated at the line ends; vdt = face normal
// velocity x deltat.
// ---------------------------------------------------------------------------
// Everything that depends on the widths and the swept length alone is made
// once per face (O3Face) and used by every variable: the expressions keep
// their trees, so each value rounds as the reference's.  Only the gradients
// and the interface value of the upwind side are evaluated (the reference
// reads no others).
struct O3Grad {
  double a, b, c;  // g = a (b (yp - y0) + c (y0 - ym))
  __device__ __forceinline__ void set(double hm, double h0, double hp) {
    a = h0 / (hm + h0 + hp);
    b = (2. * hm + h0) / (h0 + hp);
    c = (h0 + 2. * hp) / (hm + h0);
  }
  __device__ __forceinline__ double at(double ym, double y0, double yp) const {
    return a * (b * (yp - y0) + c * (y0 - ym));
  }
};
struct O3Star {
  double a, bp, bm, w, s;
  __device__ __forceinline__ void set(double hmm, double hm, double hp, double hpp) {
    a = (2. * hp * hm) / (hm + hp) * ((hmm + hm) / (2. * hm + hp) - (hpp + hp) / (2. * hp + hm));
    bp = -hm * (hmm + hm) / (2. * hm + hp);
    bm = hp * (hp + hpp) / (hm + 2. * hp);
    w = hm / (hm + hp);
    s = 1. / (hmm + hm + hp + hpp);
  }
  __device__ __forceinline__ double at(double ym, double yp, double gm, double gp) const {
    const double dy = yp - ym;
    return ym + w * dy + s * (a * dy + (bp * gp + bm * gm));
  }
};
struct O3Face {
  int side;         // 1: vdt > 0 (upwind cell b), -1: vdt < 0 (upwind cell f), 0: no flux
  O3Grad g1, g2, g; // cells b, f and the one behind the upwind cell
  O3Star s0, su;    // the face, and the other interface of the upwind cell
  double k1, k2, kx;
  __device__ __forceinline__ void set(const double (&h)[6], double vdt) {
    side = vdt > 0. ? 1 : (vdt < 0. ? -1 : 0);
    const bool up = side > 0;
    g1.set(h[1], h[2], h[3]);
    g2.set(h[2], h[3], h[4]);
    g.set(up ? h[0] : h[3], up ? h[1] : h[4], up ? h[2] : h[5]);
    s0.set(h[1], h[2], h[3], h[4]);
    su.set(up ? h[0] : h[2], up ? h[1] : h[3], up ? h[2] : h[4], up ? h[3] : h[5]);
    const double x = up ? vdt : -vdt, hu = up ? h[2] : h[3];
    k1 = 0.5 * x / hu;
    k2 = 1. - 2. / 3. * x / hu;
    // upwind extrapolation of the TVD bound
    const double nu = vdt / hu;
    kx = (up ? 1. - nu : 1. + nu) / nu;
  }
  __device__ __forceinline__ double at(const double (&y)[6]) const {
    if (side == 0) return 0.;
    const bool up = side > 0;
    const double ga = g1.at(y[1], y[2], y[3]), gb = g2.at(y[2], y[3], y[4]);
    const double gc = g.at(up ? y[0] : y[3], up ? y[1] : y[4], up ? y[2] : y[5]);
    const double i0 = s0.at(y[2], y[3], ga, gb);
    const double iu = su.at(up ? y[1] : y[3], up ? y[2] : y[4], up ? gc : gb, up ? ga : gc);
    const double yu = up ? y[2] : y[3];  // upwind value
    const double sl = up ? iu : i0, sr = up ? i0 : iu;
    const double du = sr - sl, u6 = 6. * (yu - 0.5 * (sl + sr));
    const double t = k1 * (du - k2 * u6);
    double v = up ? i0 - t : i0 + t;
    // TVD bound: [y_b, y_f] intersected with the upwind extrapolation
    const double e = kx * (yu - (up ? y[1] : y[4]));
    const double x = up ? yu + e : yu - e;
    const double i1a = amin(y[2], y[3]), i1b = amax(y[2], y[3]);
    const double i2a = amin(yu, x), i2b = amax(yu, x);
    double lo = 0., hi = 0.;
    if (!(i1b < i2a || i2b < i1a)) {
      lo = amax(i1a, i2a);
      hi = amin(i1b, i2b);
    }
    if (v < lo) v = lo;
    if (v > hi) v = hi;
    return v;
  }
};

// ---------------------------------------------------------------------------
// Cell sweep along D with the third-order face values
// (computeUpwindFaceQuantitiesForProjection, RemapADIService.cc:319-380):
// the same lane layout with 3 halo lanes on each side (lane l: cell
// x0 - 3 + l, lanes 3 .. 28 write).  Faces between two cells that are not
// both pure in the same material (EstMixte / EstPure, which equal the
// volume-fraction signs of the cell values read here; every cell is pure in
// material 0 before the first remap of the run) take their mass and energy
// values from the volume value with the upwind cell's density and specific
// energy.
//
// Bound by its instructions: the face's coefficients (about 30 divisions) are
// made once for all variables and the variables are a rolled loop, one
// division each.  101 x 37 x 35 cells, two environments: 94 us (x) and 98 us
// (y, z) a sweep with every variable unrolled and evaluating both upwind
// sides, 36 and 43 us now.
// ---------------------------------------------------------------------------
template <int DIM, int NE, int D>
__device__ __forceinline__ void body_sweep_cells_o3(const Mesh& M, const Fields& F, const SweepArgs& A, int vbx,
                                                    int vby) {
  constexpr int NV = 3 * NE + 1;
  constexpr int NQ = DIM == 3 ? 4 : 2;
  constexpr int HL = 3;
  constexpr unsigned FULL = 0xffffffffu;
  const long long N = M.ncell;
  const int lane = threadIdx.x % SW_LANES, row = threadIdx.x / SW_LANES;
  const int nd = D == 0 ? M.ncx : (D == 1 ? M.ncy : M.ncz);
  if (sweep_warp_empty<D>(M.ncx, M.ncy, M.ncz, XOUT_W, HL, vbx, vby, row)) return;  // whole warp leaves together
  int i, j, k, p, ta, tb;
  const bool ok = sweep_lane<D>(M.ncx, M.ncy, M.ncz, XOUT_W, HL, vbx, vby, lane, row, i, j, k, p, ta, tb);
  const bool out = ok && lane >= HL && lane < HL + XOUT_W;
  const double dt = F.s->dt;
  const double* __restrict__ Uin = A.Uin;
  Plane<DIM> back;
  if (ok) load_plane<DIM, D>(M, F, i, j, k, back);
  else {
#pragma unroll
    for (int q = 0; q < NQ; ++q) back.xd[q] = 0.;
    back.fc = back.un = back.L = 0.;
  }
  // per-thread slots of the rolled variable loop: the value of the back face
  // and of its two cells, of the volumes, then of the masses
  __shared__ double o3_slots[3 * NE * SW_THREADS];
  double* const s_face = o3_slots + threadIdx.x;
  long long c = 0;
  double den = 1., ondB = 0., ondF = 0.;
  if (ok) {
    c = cell_id(M, i, j, k);
    if (A.first) {
      den = __ldg(F.V + c);
    } else {
      den = 0.;
#pragma unroll
      for (int q = 0; q < NE; ++q) den += __ldg(Uin + q * N + c);
    }
    if (out) {
      sweep_normals<DIM, D>(M, p, ta, tb, ondB, ondF);
    }
  }
  // widths of the stencil b-2 .. f+2 of the back face (f = this cell)
  const double hw = lane_cell_width<DIM, D>(M, F, ok, i, j, k, p, nd);
  const bool m2 = p >= 2, m3 = p >= 3, p1 = p + 1 < nd, p2 = p + 2 < nd;
  double h[6];
  {
    const double a1 = __shfl_up_sync(FULL, hw, 1), a2 = __shfl_up_sync(FULL, hw, 2),
                 a3 = __shfl_up_sync(FULL, hw, 3), b1 = __shfl_down_sync(FULL, hw, 1),
                 b2 = __shfl_down_sync(FULL, hw, 2);
    h[2] = a1; h[1] = m2 ? a2 : h[2]; h[0] = m3 ? a3 : h[1];
    h[3] = hw; h[4] = p1 ? b1 : h[3]; h[5] = p2 ? b2 : h[4];
  }
  // purity code: -2 mixed, else the last material with a positive volume
  // fraction (-1: none)
  int code = 0;
  if (ok && !A.first_remap) {
    int cnt = 0;
    code = -1;
#pragma unroll 1
    for (int q = 0; q < NE; ++q)
      if (div_rn(__ldg(Uin + q * N + c), den) > 0.) { ++cnt; code = q; }
    if (cnt > 1) code = -2;
  }
  const int code_l = __shfl_up_sync(FULL, code, 1);
  const bool pure_nb = code_l == code && code != -2;
  const double un = back.un, L = back.L;  // back face of the cell
  const bool ok_l = __shfl_up_sync(FULL, ok, 1) && lane > 0 && p > 0;  // same line
  const bool face_b = ok && ok_l;
  const bool face_f = __shfl_down_sync(FULL, face_b, 1) && lane < 31;
  const double un_r = __shfl_down_sync(FULL, un, 1), L_r = __shfl_down_sync(FULL, L, 1);
  const double vdt = un * dt;
  O3Face face;
  face.set(h, vdt);
  constexpr bool FRONT_FIRST = DIM == 2 && D == 0;
  unsigned corr = 0;  // bit e: the mass and energy of environment e follow its volume value
  double u = ok ? __ldg(Uin + c) : 0.;
  // rolled: with the variables unrolled the warps waited for instructions
#pragma unroll 1
  for (int v = 0; v < NV; ++v) {
    const double u_next = (ok && v + 1 < NV) ? __ldg(Uin + (v + 1) * N + c) : 0.;
    const double phi = ok ? div_rn(u, den) : 0.;
    double y[6];
    {
      const double a1 = __shfl_up_sync(FULL, phi, 1), a2 = __shfl_up_sync(FULL, phi, 2),
                   a3 = __shfl_up_sync(FULL, phi, 3), b1 = __shfl_down_sync(FULL, phi, 1),
                   b2 = __shfl_down_sync(FULL, phi, 2);
      y[2] = a1; y[1] = m2 ? a2 : y[2]; y[0] = m3 ? a3 : y[1];
      y[3] = phi; y[4] = p1 ? b1 : y[3]; y[5] = p2 ? b2 : y[4];
    }
    double pf = face_b ? face.at(y) : 0.;
    if (v < 3 * NE) {
      const int e = v < NE ? v : (v < 2 * NE ? v - NE : v - 2 * NE);
      double* const sf = s_face + 3 * e * SW_THREADS;
      if (v >= NE && v < 2 * NE) {
        const double yb = sf[SW_THREADS], yf = sf[2 * SW_THREADS];
        const bool cb = vdt > 0. && yb != 0. && y[2] != 0.;
        const bool cf = vdt < 0. && yf != 0. && y[3] != 0.;
        if (!pure_nb && (cb || cf)) {
          corr |= 1u << e;
          pf = (cb ? (y[2] / yb) : (y[3] / yf)) * sf[0];
        }
      } else if (v >= 2 * NE) {
        if ((corr >> e) & 1) pf = (vdt > 0. ? (y[2] / sf[SW_THREADS]) : (y[3] / sf[2 * SW_THREADS])) * sf[0];
      }
      sf[0] = pf;
      sf[SW_THREADS] = y[2];
      sf[2 * SW_THREADS] = y[3];
    }
    const double pf_r = __shfl_down_sync(FULL, pf, 1);
    if (out) {
      const double fB = face_b ? ondB * un * L * dt * pf : 0.;
      const double fF = face_f ? ondF * un_r * L_r * dt * pf_r : 0.;
      double sumf = 0., dual = 0.;
      if (FRONT_FIRST) {
        if (face_f) { sumf += fF; dual += 0.5 * fF * ondF; }
        if (face_b) { sumf += fB; dual += 0.5 * fB * ondB; }
      } else {
        if (face_b) { sumf += fB; dual += 0.5 * fB * ondB; }
        if (face_f) { sumf += fF; dual += 0.5 * fF * ondF; }
      }
      double uo = u - sumf;
      if (v >= NE && v < 3 * NE && uo < 0.) uo = 0.;  // masses and energies stay >= 0
      A.Uout[v * N + c] = uo;
      if (v >= NE && v < 2 * NE) F.mflux[(v - NE) * N + c] = dual;
    }
    u = u_next;
  }
}

// ---------------------------------------------------------------------------
// Cell sweep along D = 1, 2 through a shared-memory tile, classical limiters
// and first order.  A block holds SWT_COLS neighbouring x columns and one
// window of 32 positions along D (the concatenated lines of the lane layout:
// 2 halo cells, XOUT written, the rest after them).
//  1. Load: thread t takes column t % SWT_COLS and position t / SWT_COLS, so
//     the SWT_COLS threads of one position read consecutive x cells (every
//     global load and store is a contiguous 64-byte run); each thread
//     stages its cell's projected quantities, divisor, Lagrangian centre
//     along D and back-face centre, normal velocity and length.
//  2. Sweep: warp w takes column w, lane = position along D, and runs the
//     arithmetic of body_sweep_cells_lanes, in the same order, from the
//     staged values (neighbours by shuffles); results go back to the tile.
//  3. Store: the load layout again, written cells only.
// The staged front-plane coordinates of a cell are loaded, not shuffled, so
// the cell centre is the same sum of the same node coordinates.
//
// For meshes of every size: a y or z sweep of 384^3 cells takes 2.3 ms here,
// 2.6 ms with one thread per line chunk and the stencil carried in registers
// (3 blocks per SM), 5.6 ms with a warp per line.
// ---------------------------------------------------------------------------
constexpr int SWT_COLS = 8;                     // x columns (warps) per block
constexpr int SWT_THREADS = SWT_COLS * SW_LANES;
constexpr int SWT_PITCH = SWT_COLS + 1;         // padded row: two wavefronts per warp access
constexpr int SWT_FIELD = SW_LANES * SWT_PITCH;  // doubles per staged quantity

// staged quantities: NV projected values, divisor, centre, face centre,
// normal velocity, face length (outputs reuse the first NV + NE slots)
__host__ __device__ constexpr int swt_slots(int ne) { return 3 * ne + 1 + 5; }
__host__ __device__ constexpr int swt_smem_bytes(int ne) { return swt_slots(ne) * SWT_FIELD * 8; }

template <int DIM, int NE, int D, int LIM, bool SHARE>
__device__ __forceinline__ void body_sweep_cells_tile(const Mesh& M, const Fields& F, const SweepArgs& A, int vbx,
                                                      int vby, double* __restrict__ sm) {
  static_assert(D >= 1, "x sweeps use the lane layout");
  constexpr int NV = 3 * NE + 1;
  constexpr int S_DEN = NV, S_XC = NV + 1, S_FC = NV + 2, S_UN = NV + 3, S_L = NV + 4;
  constexpr unsigned FULL = 0xffffffffu;
  const long long N = M.ncell;
  const int nd = D == 1 ? M.ncy : M.ncz, nb = D == 1 ? M.ncz : M.ncy;
  const int x0 = vbx * SWT_COLS;
  const int g0 = vby * XOUT - 2;  // first position of the window (2 halo cells)
  const double* __restrict__ Uin = A.Uin;
  int v0, v1;
  share_of<NV, SHARE>(A, v0, v1);
  // -- 1. load (row layout); the volumes make the divisor of every share
  {
    const int col = threadIdx.x % SWT_COLS, pos = threadIdx.x / SWT_COLS;
    const int i = x0 + col, g = g0 + pos;
    if (i < M.ncx && g >= 0 && g < nb * nd) {
      const int tb = (int)((unsigned)g / (unsigned)nd), p = g - tb * nd;
      const int j = D == 1 ? p : tb, k = D == 1 ? tb : p;
      Plane<DIM> back, front;
      load_plane<DIM, D>(M, F, i, j, k, back);
      load_plane_xd<DIM, D>(M, F, i, D == 1 ? j + 1 : j, D == 2 ? k + 1 : k, front);
      const long long c = cell_id(M, i, j, k);
      double* s = sm + pos * SWT_PITCH + col;
      double den = 0.;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (v >= NE && (v < v0 || v >= v1)) continue;
        const double u = __ldg(Uin + v * N + c);
        s[v * SWT_FIELD] = u;
        if (v < NE) den += u;
      }
      if (A.first) den = __ldg(F.V + c);
      s[S_DEN * SWT_FIELD] = den;
      s[S_XC * SWT_FIELD] = centre_from_planes<DIM, D>(back, front);
      s[S_FC * SWT_FIELD] = back.fc;
      s[S_UN * SWT_FIELD] = back.un;
      s[S_L * SWT_FIELD] = back.L;
    }
  }
  __syncthreads();
  // -- 2. sweep (warp w: column x0 + w, lane: position along D)
  const int lane = threadIdx.x % SW_LANES, w = threadIdx.x / SW_LANES;
  const int ta = x0 + w;
  if (ta < M.ncx && g0 < nb * nd) {  // warp-uniform
    const int g = g0 + lane;
    const bool ok = g >= 0 && g < nb * nd;
    int tb = 0, p = 0;
    if (ok) {
      tb = (int)((unsigned)g / (unsigned)nd);
      p = g - tb * nd;
    }
    const bool out = ok && lane >= 2 && lane < 2 + XOUT;
    const double dt = F.s->dt;
    const int order2 = LIM == LIM_ORDER1 ? 0 : 1;  // ordre-projection - 1
    double* s = sm + lane * SWT_PITCH + w;
    CellLane<DIM, D, LIM> K;
    K.ok = ok;
    double den = 1., xc = 0., fc = 0., un = 0., L = 0.;
    K.ondB = K.ondF = 0.;
    if (ok) {
      den = s[S_DEN * SWT_FIELD];
      xc = s[S_XC * SWT_FIELD];
      fc = s[S_FC * SWT_FIELD];
      un = s[S_UN * SWT_FIELD];
      L = s[S_L * SWT_FIELD];
      if (out) sweep_normals<DIM, D>(M, p, ta, tb, K.ondB, K.ondF);
    }
    const bool ok_l = __shfl_up_sync(FULL, ok, 1) && lane > 0 && p > 0;  // same line
    const double xc_l = __shfl_up_sync(FULL, xc, 1);
    K.face_b = ok && ok_l;                       // face between p-1 and p
    K.set_faces(dt, order2, fc, xc, xc_l, un, L, den);
#pragma unroll 1
    for (int v = v0; v < v1; ++v) {
      const double u = ok ? s[v * SWT_FIELD] : 0.;
      double fB, fF;
      const bool some = K.fluxes(u, fB, fF);
      if (out) {
        if (some) {
          double uo = u - (fB + fF);
          if (v >= NE && v < 3 * NE && uo < 0.) uo = 0.;  // masses and energies stay >= 0
          s[v * SWT_FIELD] = uo;                          // the lane's own slots: read above
        }
        if (v >= NE && v < 2 * NE) s[(S_XC + v - NE) * SWT_FIELD] = K.dual(fB, fF);
      }
    }
  }
  __syncthreads();
  // -- 3. store (row layout), written positions only
  {
    const int col = threadIdx.x % SWT_COLS, pos = threadIdx.x / SWT_COLS;
    const int i = x0 + col, g = g0 + pos;
    if (pos >= 2 && pos < 2 + XOUT && i < M.ncx && g < nb * nd) {
      const int tb = (int)((unsigned)g / (unsigned)nd), p = g - tb * nd;
      const long long c = cell_id(M, i, D == 1 ? p : tb, D == 1 ? tb : p);
      const double* s = sm + pos * SWT_PITCH + col;
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (v >= v0 && v < v1) A.Uout[v * N + c] = s[v * SWT_FIELD];
#pragma unroll
      for (int e = 0; e < NE; ++e)
        if (NE + e >= v0 && NE + e < v1) F.mflux[e * N + c] = s[(S_XC + e) * SWT_FIELD];
    }
  }
  __syncthreads();  // the tile is reused by the block's next work item
}

// ---------------------------------------------------------------------------
// Node part: RemapADIService::computeDualUremap (DualPhaseRemap.cc:38-258,
// classical limiter) with the same lane layout.  Lane l holds node
// x0 - 2 + l along D; lanes 2 .. NOUT+1 write.  The mass flux through the
// back half-plane of a node is the flux through the front half-plane of the
// node behind it, summed over the same cells in the same order, so each
// lane sums its front cells once and hands the sum to lane l+1.
// ---------------------------------------------------------------------------
constexpr int NOUT = 28;    // nodes written per warp (lanes 2 .. 29)
constexpr int NOUT_W = 26;  // generalised limiters (widths need 2 more nodes): lanes 3 .. 28

struct DualArgs {
  const double* Uin;   // null on the first sweep (U built from m and v)
  double* Uout;
  int order;
  int limiter;
  int simple_pente;    // projection-simple-pente (generalised limiters)
  int done_dirs;       // bit d: direction d already swept this cycle
  int energy;          // conservation-energie-totale: the kinetic energy is projected too
};

__device__ __forceinline__ bool node_inner_dir(const Mesh& M, int i, int j, int k, int d) {
  int id = d == 0 ? i : (d == 1 ? j : k);
  int nn = d == 0 ? M.nnx : (d == 1 ? M.nny : M.nnz);
  return id > 0 && id < nn - 1;
}

// ---------------------------------------------------------------------------
// One variable of a node sweep, one node per lane along D: its value, the
// limited gradient and the two fluxes, the neighbours' by shuffles.  The
// swept velocity component comes first (its values give the upwind lengths of
// the others), then the other two, then, where the total energy is conserved,
// the kinetic energy (no gradient); nothing else reads the kinetic energy, so
// it is left out otherwise.  The quotients by the node mass and by
// the distance of the nodes share a reciprocal each.
// ---------------------------------------------------------------------------
template <int D, int LIM>
struct NodeLane {
  bool ok, inner, was_inner, has_r;  // has_r: the next node is on the same line, in the warp
  bool odd;                          // an upwind length is not finite, or the distance out of range
  SharedDivisor mass, dx;            // projected mass before the sweep; distance to the next node
  double x, x_l, x_r, ffm, bfm, dt;
  double geo_f, geo_b;
  int order2;
  // generalised limiters
  int limiter, simple_pente;
  double h0, hm, hp;

  // positions and mass fluxes of the neighbours (every lane of the warp)
  __device__ __forceinline__ void set_line(double position, double front_flux, double m, int id, int nn) {
    constexpr unsigned FULL = 0xffffffffu;
    x = position;
    ffm = front_flux;
    x_l = __shfl_up_sync(FULL, x, 1);
    x_r = __shfl_down_sync(FULL, x, 1);
    // the mass flux through the back half-plane of a node is the front one
    // of the node behind it
    bfm = __shfl_up_sync(FULL, ffm, 1);
    has_r = ok && (threadIdx.x % SW_LANES) < 31 && id < nn - 1;
    mass.set(was_inner ? m : 1.);
    dx.set(has_r ? x_r - x : 1.);
    if constexpr (LIM == LIM_GEN) {
      // dual cell widths (UtilesRemap.cc:51-63); a missing second neighbour
      // gives a zero width
      const double x_ll = __shfl_up_sync(FULL, x, 2), x_rr = __shfl_down_sync(FULL, x, 2);
      const bool bb = id >= 2, ff = id + 2 < nn;
      h0 = hm = hp = 0.;
      h0 = 0.5 * (x_r - x_l);
      if (!bb) {
        if (ff) hp = 0.5 * (x_rr - x);
      } else if (!ff) {
        hm = 0.5 * (x - x_ll);
      } else {
        hm = 0.5 * (x - x_ll);
        hp = 0.5 * (x_rr - x);
      }
    }
  }
  // the node's value of a variable: U / mass of a node that a sweep of this
  // remap moved, the node's own value (v) otherwise
  __device__ __forceinline__ double value(double U, double v) const {
    constexpr unsigned FULL = 0xffffffffu;
    bool fine = true;
    double ph = was_inner ? mass.q(U, fine) : v;
    if (__any_sync(FULL, !fine) && was_inner) ph = div_rn(U, mass.b);
    return ph;
  }
  // the update of U for a variable of value ph: component t of the order D,
  // then the others (t = 0 sets the upwind lengths), t = 3 the kinetic energy
  __device__ __forceinline__ double update(int t, double ph, double U) {
    constexpr unsigned FULL = 0xffffffffu;
    const double ph_l = __shfl_up_sync(FULL, ph, 1), ph_r = __shfl_down_sync(FULL, ph, 1);
    if (t == 0) {
      const double ufront = 0.5 * (ph + ph_r), uback = 0.5 * (ph_l + ph);
      const int signfront = (ufront > 0) ? 1 : -1, signback = (uback > 0) ? 1 : -1;
      geo_f = (signfront * (x_r - x) - dt * ufront);
      geo_b = (signback * (x - x_l) - dt * uback);
      constexpr double TOP = 1.7976931348623157e308;
      odd = dx.y == 0. || !(fabs(geo_f) <= TOP && fabs(geo_b) <= TOP);
    }
    const bool fr = ffm < 0., bk = bfm > 0.;
    double FV = fr ? ph_r : ph, BV = bk ? ph_l : ph;
    const double diff = has_r ? ph_r - ph : 0.;
    // a warp without differences has no gradients
    if (__any_sync(FULL, (LIM != LIM_ORDER1 && t < 3 && diff != 0.) || odd)) {
      // the backward difference of a node is the forward difference of the
      // node before it (same operands)
      bool fine = true;
      double gfw = has_r ? dx.q(diff, fine) : 0.;
      if (__any_sync(FULL, !fine)) gfw = has_r ? div_rn(diff, dx.b) : 0.;
      const double gbw = __shfl_up_sync(FULL, gfw, 1);
      double g = 0.;
      if (LIM != LIM_ORDER1 && inner && t < 3) {  // limited gradients of inner nodes only
        if constexpr (LIM == LIM_GEN) g = generalized_gradient(limiter, gfw, gbw, ph_r, ph_l, h0, hp, hm, simple_pente);
        else g = limited_gradient_t<LIM == LIM_ORDER1 ? 0 : LIM>(gbw, gfw);
      }
      const double g_l = __shfl_up_sync(FULL, g, 1), g_r = __shfl_down_sync(FULL, g, 1);
      FV = FV + order2 * (0.5 * (fr ? g_r : g) * geo_f);
      BV = BV + order2 * (0.5 * (bk ? g_l : g) * geo_b);
    }
    double W = U + (bfm * BV - ffm * FV);
    if (t < 3 && fabs(W) < 1.e-300) W = 0.;
    return W;
  }
};

// mass flux through the front half-plane of node (i, j, k): the faces of the
// node plane in face id order, then the environments
template <int DIM, int NE, int D>
__device__ __forceinline__ double front_mass_flux(const Mesh& M, const Fields& F, int i, int j, int k, int id) {
  const long long N = M.ncell;
  const int ndc = D == 0 ? M.ncx : (D == 1 ? M.ncy : M.ncz);
  double ffm = 0.;
  if (id >= ndc) return ffm;
  const double w = DIM == 2 ? .5 : .25;
  // the cells behind and in front of the node along the transverse axes
  constexpr bool T2 = DIM == 3;
  const int t1 = D == 0 ? j : i, n1 = D == 0 ? M.ncy : M.ncx, t2 = D == 2 ? j : k, n2 = D == 2 ? M.ncy : M.ncz;
  const unsigned s1 = D == 0 ? (unsigned)M.ncx : 1u, s2 = D == 2 ? (unsigned)M.ncx : (unsigned)M.ncx * (unsigned)M.ncy;
  const bool lo1 = t1 > 0, hi1 = t1 < n1, lo2 = !T2 || t2 > 0, hi2 = T2 && t2 < n2;
  // id of the cell in front along both (2D: along the first)
  const unsigned cf = (unsigned)i + (unsigned)M.ncx * ((unsigned)j + (T2 ? (unsigned)M.ncy * (unsigned)k : 0u));
  const unsigned c2 = T2 ? cf - s2 : cf;
  auto add = [&](bool in, unsigned c) {
    if (!in) return;
#pragma unroll
    for (int q = 0; q < NE; ++q) ffm += w * __ldg(F.mflux + q * N + c);
  };
  add(lo1 && lo2, c2 - s1);
  add(hi1 && lo2, c2);
  if (T2) {
    add(lo1 && hi2, cf - s1);
    add(hi1 && hi2, cf);
  }
  return ffm;
}

// a direction swept before moved node (i, j, k)
template <int DIM>
__device__ __forceinline__ bool node_was_inner(const Mesh& M, const DualArgs& A, int i, int j, int k) {
  bool was = false;
#pragma unroll
  for (int d = 0; d < DIM; ++d)
    if (((A.done_dirs >> d) & 1) && node_inner_dir(M, i, j, k, d)) was = true;
  return was;
}

template <int DIM, int NE, int D, int LIM>
__device__ __forceinline__ void body_sweep_nodes_lanes(const Mesh& M, const Fields& F, const DualArgs& A,
                                                       int vbx, int vby) {
  constexpr unsigned FULL = 0xffffffffu;
  const long long NN = M.nnode;
  const int lane = threadIdx.x % SW_LANES, row = threadIdx.x / SW_LANES;
  const int nn = D == 0 ? M.nnx : (D == 1 ? M.nny : M.nnz);
  constexpr int HL = LIM == LIM_GEN ? 3 : 2;
  constexpr int NO = LIM == LIM_GEN ? NOUT_W : NOUT;
  if (sweep_warp_empty<D>(M.nnx, M.nny, M.nnz, NO, HL, vbx, vby, row)) return;  // whole warp leaves together
  int i, j, k, id, ta, tb;
  NodeLane<D, LIM> K;
  K.ok = sweep_lane<D>(M.nnx, M.nny, M.nnz, NO, HL, vbx, vby, lane, row, i, j, k, id, ta, tb);
  K.inner = K.ok && id > 0 && id < nn - 1;
  const bool out = K.ok && lane >= HL && lane < HL + NO;
  K.was_inner = false;
  K.dt = F.s->dt;
  K.order2 = LIM == LIM_ORDER1 ? 0 : A.order - 1;  // ordre-projection - 1
  K.limiter = A.limiter;
  K.simple_pente = A.simple_pente;
  long long n = 0;
  double m = 1., x = 0., ffm = 0.;
  if (K.ok) {
    n = node_id(M, i, j, k);
    x = __ldg(F.Xn[D] + n);
    K.was_inner = node_was_inner<DIM>(M, A, i, j, k);
    m = A.Uin ? __ldg(A.Uin + 3 * NN + n) : __ldg(F.mn + n);
    ffm = front_mass_flux<DIM, NE, D>(M, F, i, j, k, id);
  }
  K.set_line(x, ffm, m, id, nn);
  double vel[3] = {0., 0., 0.}, mom[3] = {0., 0., 0.};
  if (K.ok) {
    if (!K.was_inner || !A.Uin || A.energy) {
      vel[0] = __ldg(F.vx + n);
      vel[1] = __ldg(F.vy + n);
      vel[2] = __ldg(F.vz + n);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) mom[q] = A.Uin ? __ldg(A.Uin + q * NN + n) : m * vel[q];
  }
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    constexpr int order[3] = {D, D == 0 ? 1 : 0, D == 2 ? 1 : 2};  // swept component first
    const int q = order[t];
    const double W = K.update(t, K.value(mom[q], vel[q]), mom[q]);
    if (out) A.Uout[q * NN + n] = K.inner ? W : mom[q];
  }
  if (A.energy) {
    const double vv = vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2];
    const double U = !K.ok ? 0. : (A.Uin ? __ldg(A.Uin + 4 * NN + n) : 0.5 * m * vv);
    const double W = K.update(3, K.value(U, 0.5 * vv), U);
    if (out) A.Uout[4 * NN + n] = K.inner ? W : U;
  }
  if (out) A.Uout[3 * NN + n] = K.inner ? m + (K.bfm - K.ffm) : m;
}

// ---------------------------------------------------------------------------
// Node sweep along D = 1, 2 through a shared-memory tile, classical limiters
// and first order (the layout of body_sweep_cells_tile): the load layout
// stages, per node, its position along D, the mass flux through its front
// half-plane, its mass, and per variable the projected dual U and the value
// that the limited reconstruction uses; warp w then runs the arithmetic of
// body_sweep_nodes_lanes on column w, in the same order, and the store
// layout writes the updated variables of the written nodes (NOUT per
// window).
// ---------------------------------------------------------------------------
// staged: x, front mass flux, mass, then U and value of every variable
constexpr int SWTN_SLOTS = 11;
constexpr int SWTN_SMEM_BYTES = SWTN_SLOTS * SWT_FIELD * 8;

template <int DIM, int NE, int D, int LIM>
__device__ __forceinline__ void body_sweep_nodes_tile(const Mesh& M, const Fields& F, const DualArgs& A, int vbx,
                                                      int vby, double* __restrict__ sm) {
  static_assert(D >= 1, "x sweeps use the lane layout");
  constexpr int S_X = 0, S_FFM = 1, S_M = 2, S_U = 3, S_V = 7;
  const long long NN = M.nnode;
  const int nn = D == 1 ? M.nny : M.nnz, nb = D == 1 ? M.nnz : M.nny;
  const int x0 = vbx * SWT_COLS;
  const int g0 = vby * NOUT - 2;  // first position of the window (2 halo nodes)
  const int nc = A.energy ? 4 : 3;
  // -- 1. load (row layout)
  {
    const int col = threadIdx.x % SWT_COLS, pos = threadIdx.x / SWT_COLS;
    const int i = x0 + col, g = g0 + pos;
    if (i < M.nnx && g >= 0 && g < nb * nn) {
      const int tb = (int)((unsigned)g / (unsigned)nn), id = g - tb * nn;
      const int j = D == 1 ? id : tb, k = D == 1 ? tb : id;
      const long long n = node_id(M, i, j, k);
      double* s = sm + pos * SWT_PITCH + col;
      const double m = A.Uin ? __ldg(A.Uin + 3 * NN + n) : __ldg(F.mn + n);
      const double v[3] = {__ldg(F.vx + n), __ldg(F.vy + n), __ldg(F.vz + n)};
      s[S_X * SWT_FIELD] = __ldg(F.Xn[D] + n);
      s[S_FFM * SWT_FIELD] = front_mass_flux<DIM, NE, D>(M, F, i, j, k, id);
      s[S_M * SWT_FIELD] = m;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        s[(S_V + q) * SWT_FIELD] = v[q];
        s[(S_U + q) * SWT_FIELD] = A.Uin ? __ldg(A.Uin + q * NN + n) : m * v[q];
      }
      if (nc == 4) {
        const double vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        s[(S_V + 3) * SWT_FIELD] = 0.5 * vv;
        s[(S_U + 3) * SWT_FIELD] = A.Uin ? __ldg(A.Uin + 4 * NN + n) : 0.5 * m * vv;
      }
    }
  }
  __syncthreads();
  // -- 2. sweep (warp w: column x0 + w, lane: position along D)
  const int lane = threadIdx.x % SW_LANES, w = threadIdx.x / SW_LANES;
  if (x0 + w < M.nnx && g0 < nb * nn) {  // warp-uniform
    const int g = g0 + lane;
    NodeLane<D, LIM> K;
    K.ok = g >= 0 && g < nb * nn;
    const int tb = K.ok ? (int)((unsigned)g / (unsigned)nn) : 0, id = K.ok ? g - tb * nn : 0;
    K.inner = K.ok && id > 0 && id < nn - 1;
    K.was_inner = K.ok && node_was_inner<DIM>(M, A, x0 + w, D == 1 ? id : tb, D == 1 ? tb : id);
    K.dt = F.s->dt;
    K.order2 = LIM == LIM_ORDER1 ? 0 : A.order - 1;  // ordre-projection - 1
    const bool out = K.ok && lane >= 2 && lane < 2 + NOUT;
    double* s = sm + lane * SWT_PITCH + w;
    double m = 1., x = 0., ffm = 0.;
    if (K.ok) {
      m = s[S_M * SWT_FIELD];
      x = s[S_X * SWT_FIELD];
      ffm = s[S_FFM * SWT_FIELD];
    }
    K.set_line(x, ffm, m, id, nn);
    auto component = [&](int t, int q) {
      const double U = K.ok ? s[(S_U + q) * SWT_FIELD] : 0., v = K.ok ? s[(S_V + q) * SWT_FIELD] : 0.;
      const double W = K.update(t, K.value(U, v), U);
      if (out && K.inner) s[(S_U + q) * SWT_FIELD] = W;  // the lane's own slots; outer nodes keep their U
    };
    component(0, D);  // swept component first
    component(1, 0);
    component(2, D == 2 ? 1 : 2);
    if (nc == 4) component(3, 3);
    if (out && K.inner) s[S_M * SWT_FIELD] = m + (K.bfm - K.ffm);
  }
  __syncthreads();
  // -- 3. store (row layout), written positions only
  {
    const int col = threadIdx.x % SWT_COLS, pos = threadIdx.x / SWT_COLS;
    const int i = x0 + col, g = g0 + pos;
    if (pos >= 2 && pos < 2 + NOUT && i < M.nnx && g < nb * nn) {
      const int tb = (int)((unsigned)g / (unsigned)nn), id = g - tb * nn;
      const long long n = node_id(M, i, D == 1 ? id : tb, D == 1 ? tb : id);
      const double* s = sm + pos * SWT_PITCH + col;
#pragma unroll
      for (int q = 0; q < 3; ++q) A.Uout[q * NN + n] = s[(S_U + q) * SWT_FIELD];
      A.Uout[3 * NN + n] = s[S_M * SWT_FIELD];
      if (nc == 4) A.Uout[4 * NN + n] = s[(S_U + 3) * SWT_FIELD];
    }
  }
  __syncthreads();  // the tile is reused by the block's next work item
}

}  // namespace mhc
