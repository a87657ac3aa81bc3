// recon_sym.cu -- linear reconstruction with two Gauss points per direction, by parity.
//
// Every face point of a cell (and, for GLM-MHD, every interior point) has mirror
// images under the reflections x -> -x, y -> -y, z -> -z of the cell, the stencil
// is invariant under them, and the weights of mirrored points are mirrored copies
// (the stencil build copies them, so they agree bit for bit).  The reflections
// diagonalise the contraction: with the stencil values combined into sums and
// differences over each orbit of mirrored cells (33 combinations in 3D, 13 in 2D),
// the 8 (4) points of one face direction follow from 32 (12) products, split over
// the 8 (4) parities, and a butterfly.  The weights of a point sum to 1, so the sums
// run over differences to the cell's value: rounding then scales with the local
// variation, and uniform gas comes back exactly.  Per cell and variable that is
// 58 + 3 x (32 + 32) = 250 FP64 operations in 3D for the 24 face points, where the
// direct sum takes 24 x 33 = 792, and 76 against 104 in 2D.  The FP64 tensor
// instruction (m8n8k4) runs at the rate of the plain FP64 pipe, so the operation
// count decides, and the direct sum on it was the longest kernel of a stage.
//
// In 3D one thread takes one variable of a cell (a thread per cell ran at 255
// registers and 8 warps per SM, waiting for its own results two thirds of the time),
// and blocks march along z through a chunk of planes with a ring of TMA-staged state
// planes, so that a plane is loaded and its limiter footprint computed once per block
// instead of once for each of the planes that read it.  In 2D a block takes one 32 x 8
// tile with one thread per cell.
//
// Bound by the issue rate (the point test and the indicator cost more instructions than
// the contraction) and by the block's two barriers per plane.  Per launch, the direct sum
// on the FP64 tensor instruction before: Euler 256^3 7.5 -> 5.0 ms, Navier-Stokes 160^3
// 1.89 -> 1.30 ms, GLM-MHD 96^3 1.45 -> 0.72 ms, Euler 1024^2 0.186 -> 0.111 ms, GLM-MHD
// 1024^2 0.48 -> 0.30 ms.
//
// Special-relativistic hydrodynamics keeps the direct sum (recon_tma_kernel): its limiter
// compares with bounds that hold the cell's own value, so the rounding of the sum in
// uniform gas decides theta there, and the flags that follow from it are the
// reference's only with the reference's kind of sum.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "kernels.cuh"
#include "launch.h"
#include "plane_ring.h"
#include "recon_common.cuh"
#include "tma.cuh"

namespace kfvm {

// Stencil combinations, in the order of the weights (fill_sym_weights), of differences to the
// cell's value (the value itself comes first).  They come grouped by parity: even in
// all axes, odd in x, odd in y, (odd in z, in x and y, in x and z, in y and z, in all).
// In 3D the combinations within a plane (x and y) are formed once per plane, as
// differences to the cell's own value in that plane, and serve the three planes of cells
// that read it: 9 loads and 20 operations per plane and variable instead of 27 and 36.
struct SymPlane {
  double x1s, x1d, y1s, y1d, xys, xyx, xyy, xyo;  // (+-1, 0), (0, +-1), (+-1, +-1): sum, odd in x, in y, in both
};
template <int TX>
__device__ __forceinline__ SymPlane sym_plane(const double *u, double c) {
  SymPlane p;
  double a = u[1] - c, b = u[-1] - c;
  p.x1s = a + b;
  p.x1d = a - b;
  a = u[TX] - c, b = u[-TX] - c;
  p.y1s = a + b;
  p.y1d = a - b;
  const double pp = u[TX + 1] - c, mp = u[TX - 1] - c, pm = u[-TX + 1] - c, mm = u[-TX - 1] - c;
  const double e = pp + pm, f = pp - pm, g = mp + mm, h = mp - mm;
  p.xys = e + g;
  p.xyx = e - g;
  p.xyy = f + h;
  p.xyo = f - h;
  return p;
}
// of the planes below (m), of (o) and above (p) the cell; c..: the column's values
// (differences refer to c0, so a plane's own reference enters with its multiplicity)
template <int TX>
__device__ __forceinline__ void sym_combine(const double *u, const SymPlane &m, const SymPlane &o, const SymPlane &p,
                                            double cm2, double cm1, double c0, double cp1, double cp2,
                                            double (&s)[33]) {
  auto pair = [&](double a, double b, double &sum, double &dif) {
    sum = a + b;
    dif = a - b;
  };
  s[0] = c0;
  s[1] = o.x1s, s[11] = o.x1d, s[2] = o.y1s, s[16] = o.y1d;
  s[7] = o.xys, s[13] = o.xyx, s[18] = o.xyy, s[26] = o.xyo;
  pair(cp1 - c0, cm1 - c0, s[3], s[21]);
  pair(cp2 - c0, cm2 - c0, s[6], s[22]);
  pair(u[2] - c0, u[-2] - c0, s[4], s[12]);
  pair(u[2 * TX] - c0, u[-2 * TX] - c0, s[5], s[17]);
  pair(p.x1s, m.x1s, s[8], s[23]);
  pair(p.x1d, m.x1d, s[14], s[28]);
  pair(p.y1s, m.y1s, s[9], s[24]);
  pair(p.y1d, m.y1d, s[19], s[30]);
  pair(p.xys, m.xys, s[10], s[25]);
  pair(p.xyx, m.xyx, s[15], s[29]);
  pair(p.xyy, m.xyy, s[20], s[31]);
  pair(p.xyo, m.xyo, s[27], s[32]);
  s[8] = fma(2.0, s[3], s[8]);
  s[9] = fma(2.0, s[3], s[9]);
  s[10] = fma(4.0, s[3], s[10]);
  s[23] = fma(2.0, s[21], s[23]);
  s[24] = fma(2.0, s[21], s[24]);
  s[25] = fma(4.0, s[21], s[25]);
}
// in 2D: ld(dx, dy) is the difference at that offset, and the value itself at (0, 0)
template <class Ld>
__device__ __forceinline__ void sym_combine(Ld ld, double (&s)[13]) {
  s[0] = ld(0, 0);
  double a = ld(1, 0), b = ld(-1, 0);
  s[1] = a + b;
  s[6] = a - b;
  a = ld(0, 1), b = ld(0, -1);
  s[2] = a + b;
  s[9] = a - b;
  a = ld(2, 0), b = ld(-2, 0);
  s[3] = a + b;
  s[7] = a - b;
  a = ld(0, 2), b = ld(0, -2);
  s[4] = a + b;
  s[10] = a - b;
  const double pp = ld(1, 1), pm = ld(1, -1), mp = ld(-1, 1), mm = ld(-1, -1);
  const double e = pp + pm, f = pp - pm, g = mp + mm, h = mp - mm;
  s[5] = e + g;
  s[8] = e - g;
  s[11] = f + h;
  s[12] = f - h;
}

// The 8 (4) points of a group from its weights (w[0] is not used): f[o], bit d of o set where the point
// lies on the positive side of axis d.
__device__ __forceinline__ void sym_points(const double *w, const double (&s)[33], double (&f)[8]) {
  auto dot = [&](int b, int n) {
    double r = w[b] * s[b];
#pragma unroll
    for (int t = 1; t < 11; t++)
      if (t < n) r = fma(w[b + t], s[b + t], r);
    return r;
  };
  const double E = dot(1, 10), X = dot(11, 5), Y = dot(16, 5), Z = dot(21, 5);
  const double XY = dot(26, 2), XZ = dot(28, 2), YZ = dot(30, 2), A = dot(32, 1);
#pragma unroll
  for (int tz = 0; tz < 2; tz++) {
    const double e = tz ? E + Z : E - Z, x = tz ? X + XZ : X - XZ, y = tz ? Y + YZ : Y - YZ, a = tz ? XY + A : XY - A;
    const double e0 = e - y, e1 = e + y, x0 = x - a, x1 = x + a;
    f[4 * tz] = s[0] + (e0 - x0);
    f[4 * tz + 1] = s[0] + (e0 + x0);
    f[4 * tz + 2] = s[0] + (e1 - x1);
    f[4 * tz + 3] = s[0] + (e1 + x1);
  }
}
__device__ __forceinline__ void sym_points(const double *w, const double (&s)[13], double (&f)[4]) {
  auto dot = [&](int b, int n) {
    double r = w[b] * s[b];
#pragma unroll
    for (int t = 1; t < 6; t++)
      if (t < n) r = fma(w[b + t], s[b + t], r);
    return r;
  };
  const double E = dot(1, 5), X = dot(6, 3), Y = dot(9, 3), A = w[12] * s[12];
  const double e0 = E - Y, e1 = E + Y, x0 = X - A, x1 = X + A;
  f[0] = s[0] + (e0 - x0);
  f[1] = s[0] + (e0 + x0);
  f[2] = s[0] + (e1 - x1);
  f[3] = s[0] + (e1 + x1);
}

// quadrature index of point o on the faces of axis d (the lower transverse axis
// first), and in the interior
template <int DIM>
__host__ __device__ __forceinline__ constexpr int sym_face_q(int d, int o) {
  const int x = o & 1, y = (o >> 1) & 1, z = (o >> 2) & 1;
  if (DIM == 2) return d == 0 ? y : x;
  return d == 0 ? 2 * y + z : (d == 1 ? 2 * x + z : 2 * x + y);
}
template <int DIM>
__device__ __forceinline__ constexpr int sym_inner_q(int o) {
  const int x = o & 1, y = (o >> 1) & 1, z = (o >> 2) & 1;
  return DIM == 2 ? 2 * x + y : (2 * x + y) * 2 + z;
}

// The limiter's bounds of a cell.
struct SymBounds {
  double minDens, maxDens, minEint;
};
// What a cell's thread needs besides its stencil values in 2D.
struct SymCell {
  SymBounds bd;
  int64_t c;        // cell index
  int64_t fidx[2];  // its low face per axis
  int64_t fstr[2];  // from there to the high face
};

// One cell in 2D: ld(v, dx, dy) gives variable v at an offset.  Writes the face states
// (and the interior points), the indicator and the cell's status.
//
// A cell whose states do not lie inside the limiter's bounds with a margin of
// rounding goes to the heavy pass, which decides exactly (theta stays 1 there when
// the states are inside after all), so the kinetic energy needs no IEEE division here.
template <int EQ, class Ld>
__device__ __forceinline__ void sym_cell(Ld ld, const SymW &w, const Grid &g, const SymCell &cl, int wantInd,
                                         double *const (&F)[2], float *const (&W)[2], double *__restrict__ src,
                                         uint8_t *__restrict__ status, double2 *__restrict__ lamvel) {
  using E = Eos<EQ>;
  constexpr int DIM = 2, NV = E::NV, NQF = 2, NP = 4, NS = 13;
  bool inside = true;
  double lam = 0.0, vel = 0.0;
  auto combine = [&](int v, double (&s)[NS]) {
    const double c = ld(v, 0, 0);
    sym_combine([&](int dx, int dy) { return dx == 0 && dy == 0 ? c : ld(v, dx, dy) - c; }, s);
  };
  // the points of face direction d for variable v, stored; f[o] as sym_points
  auto points = [&](int d, int v, const double (&s)[NS], double (&f)[NP]) {
    sym_points(w.a[d], s, f);
    const int64_t nf = g.nface[d];
    double *lo = F[d] + (int64_t)(NQF * NV + v) * nf + cl.fidx[d], *hi = F[d] + (int64_t)v * nf + cl.fidx[d] + cl.fstr[d];
#pragma unroll
    for (int q = 0; q < NQF; q++) {
#pragma unroll
      for (int o = 0; o < NP; o++)
        if (sym_face_q<DIM>(d, o) == q) {
          if ((o >> d) & 1) *hi = f[o];
          else *lo = f[o];
        }
      lo += NV * nf;
      hi += NV * nf;
    }
  };
  auto store_ind = [&](int d, int o, float x) {
    const int hi = (o >> d) & 1, q = sym_face_q<DIM>(d, o);
    W[d][(int64_t)((hi ? 0 : NQF) + q) * g.nface[d] + cl.fidx[d] + (hi ? cl.fstr[d] : 0)] = x;
  };
  if constexpr (EQ != EQ_GLM) {
    // momenta (their squares), density (kinetic energy, power of the indicator), energy
    double acc[DIM * NP];
    double pw[DIM * NP];
#pragma unroll
    for (int t = 0; t < DIM * NP; t++) acc[t] = 0.0;
#pragma unroll 1
    for (int v = MOMX; v <= MOMZ; v++) {
      double s[NS], f[NP];
      combine(v, s);
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        points(d, v, s, f);
#pragma unroll
        for (int o = 0; o < NP; o++) acc[d * NP + o] = fma(f[o], f[o], acc[d * NP + o]);
      }
    }
    {
      double s[NS], f[NP];
      combine(DENS, s);
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        points(d, DENS, s, f);
#pragma unroll
        for (int o = 0; o < NP; o++) {
          double &a = acc[d * NP + o];
          inside = inside && f[o] > cl.bd.minDens && f[o] < cl.bd.maxDens && f[o] > 0.0;
          a = 0.5 * a * rcp_nr(f[o]);
          if (wantInd) pw[d * NP + o] = E::template weno_power<DIM>(g.gamma, f[o]);
        }
      }
    }
    {
      double s[NS], f[NP];
      combine(ETOT, s);
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        points(d, ETOT, s, f);
#pragma unroll
        for (int o = 0; o < NP; o++) {
          const double a = acc[d * NP + o], ei = f[o] - a;
          inside = inside && ei - cl.bd.minEint > 8.9e-16 * (fabs(a) + fabs(ei)) + 1e-300;
          if (wantInd) store_ind(d, o, E::template weno_from_power<DIM>((g.gamma - 1.0) * ei, pw[d * NP + o]));
        }
      }
    }
  } else {
    // nine variables: one group of points at a time (the partial sums of all groups
    // would not fit in registers), the combinations formed again for each
#pragma unroll
    for (int d = 0; d <= DIM; d++) {
      // sums over the variables as they come: momenta, magnetic field, psi, density, energy
      double m2[NP], b2[NP], mx[NP], bx[NP], ps[NP], ir[NP];
      double pw[NP];
#pragma unroll
      for (int o = 0; o < NP; o++) m2[o] = b2[o] = mx[o] = bx[o] = ps[o] = ir[o] = 0.0, pw[o] = 0;
#pragma unroll 1
      for (int n = 0; n < NV; n++) {
        const int v = n < 3 ? MOMX + n : (n < 7 ? MAGX + n - 3 : (n == 7 ? DENS : ETOT));
        double s[NS], f[NP];
        combine(v, s);
        if (d < DIM) {
          points(d, v, s, f);
        } else {
          sym_points(w.a[d], s, f);
#pragma unroll
          for (int o = 0; o < NP; o++) src[(int64_t)(sym_inner_q<DIM>(o) * NV + v) * g.n + cl.c] = f[o];
        }
#pragma unroll
        for (int o = 0; o < NP; o++) {
          if (v >= MOMX && v <= MOMZ) {
            m2[o] = fma(f[o], f[o], m2[o]);
            if (v == MOMX) mx[o] = f[o];
          } else if (v >= MAGX && v <= MAGZ) {
            b2[o] = fma(f[o], f[o], b2[o]);
            if (v == MAGX) bx[o] = f[o];
          } else if (v == PSI) {
            ps[o] = 0.5 * f[o] * f[o];
          } else if (v == DENS) {
            inside = inside && f[o] > cl.bd.minDens && f[o] < cl.bd.maxDens && f[o] > 0.0;
            ir[o] = rcp_nr(f[o]);
            if (wantInd && d < DIM) pw[o] = E::template weno_power<DIM>(g.gamma, f[o]);
          } else {
            const double other = 0.5 * b2[o] + 0.5 * m2[o] * ir[o] + ps[o], ei = f[o] - other;
            inside = inside && ei - cl.bd.minEint > 8.9e-16 * (fabs(other) + fabs(ei)) + 1e-300;
            if (d < DIM) {
              const double p = (g.gamma - 1.0) * ei;
              if (wantInd) store_ind(d, o, E::template weno_from_power<DIM>(p, pw[o]));
              // SpeedEstimate_K<MHD_GLM> (MHD_GLM_K.H:213-310): x components on every face
              const double asq = g.gamma * p * ir[o], absq = asq + b2[o] * ir[o], blsq = bx[o] * bx[o] * ir[o];
              const double vv = fabs(mx[o] * ir[o]);
              const double l = sqrt_nr(0.5 * (absq + sqrt_nr(absq * absq - 4.0 * asq * blsq))) + vv;
              vel = vv > vel ? vv : vel;
              lam = l > lam ? l : lam;
            }
          }
        }
      }
    }
    lamvel[cl.c] = make_double2(lam, vel);
  }
  status[cl.c] = inside ? 1 : 0;
}

// Limiter footprint of a state plane (the block's cells and a one-cell ring): internal
// energy, squared sound speed (NaN where it is negative: the minimum skips it, as it
// skips the square root's NaN) and 1 / rho.
template <int EQ>
__device__ __forceinline__ void sym_foot(const double *u, int stride, double gam, double *e, double *c2, double *ir) {
  constexpr int NV = Eos<EQ>::NV;
  double st[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) st[v] = u[v * stride];
  const double r = rcp_nr(st[DENS]), ei = Eos<EQ>::eint_r(st, r), c = gam * ((gam - 1.0) * ei) * r;
  *e = ei;
  *c2 = c >= 0.0 ? c : __longlong_as_double(0x7ff8000000000000ll);
  *ir = r;
}

// extrema over a cell's neighbourhood
struct SymExt {
  double rMax, rMin, eMin, c2Min;
};
// PositivityPreserve_K bounds (Common_K.H:331-380) from the neighbourhood's extrema
// and twice the velocity divergence
__device__ __forceinline__ SymBounds sym_bounds(const SymExt &x, double div2) {
  const double snd = sqrt_nr(x.c2Min), divV = div2 / 2.0;
  double kappa = 0.2;
  // (the IEEE quotient: cold gas has snd = 0, and +-infinity decides)
  const double eta = fmin(1.0, fmax(0.0, -(kappa * snd + divV) / (kappa * snd)));
  kappa *= (1.0 - eta);
  return {x.rMin * (1.0 - kappa), x.rMax * (1.0 + kappa), x.eMin * (1.0 - kappa)};
}

// Where the points of a cell go, as byte offsets from the cell's low face at variable v
// and point 0 of the upper slot: [direction][point]; for the indicators likewise.  Host
// constants, so that a store costs one 64-bit addition of address arithmetic.
struct SymOff {
  int64_t f[3][8], w[3][8];
};

// ---------------------------------------------------------------------------
// 3D: a block is a row of 32 cells, one warp per variable, and marches along z over a ring
// of planes.  The warps exchange the point states through shared memory and share the
// points among them for the limiter test and the indicator.
template <int EQ>
struct Sym3 {
  static constexpr int NV = Eos<EQ>::NV, BX = 32, THREADS = BX * NV;
  static constexpr int TX = BX + 2 * kRad, TY = 1 + 2 * kRad, TN = TX * TY;       // state plane of one variable
  static constexpr int PX = BX + 2, PN = PX * 3;                                  // its footprint
  // Each thread keeps the combinations of planes k - 1 and k, so the ring holds planes k to
  // k + 2 and the one in flight.  GLM-MHD's nine warps leave 96 registers a thread, too
  // few for that: it forms them again from a ring that holds plane k - 1 too.
  static constexpr bool KEEP = EQ != EQ_GLM;
  static constexpr int RING = KEEP ? 4 : 5, PLANE = (NV * TN + 15) / 16 * 16;     // planes start on 128 bytes
  static constexpr int NG = EQ == EQ_GLM ? 4 : 3;          // point groups: x, y, z faces, interior
  static constexpr int GP = EQ == EQ_GLM ? 2 : 3;          // groups exchanged at a time
  static constexpr int EX = GP * 8 * NV * BX;              // exchanged point states
  static constexpr int RED = EQ == EQ_GLM ? NV * 2 * BX : 0;
  static constexpr int QN = 5 + 3;                         // bound ingredients, bounds
  static constexpr int OFF_F = RING * PLANE * 8, OFF_X = OFF_F + 2 * 3 * PN * 8, OFF_Q = OFF_X + EX * 8;
  static constexpr int OFF_R = OFF_Q + QN * BX * 8, OFF_M = OFF_R + RED * 8;
  static constexpr int OFF_BAR = OFF_M + (NV + 1) / 2 * 8, BYTES = OFF_BAR + RING * 8;
  static constexpr int RESIDENT = EQ == EQ_GLM ? 2 : 3;    // 96 and 128 registers a thread
  static_assert((TX * 8) % 16 == 0, "TMA box inner extent");
  static_assert(RESIDENT * (BYTES + 1024) <= 228 * 1024, "shared memory of the resident blocks");
};

template <int EQ>
__global__ void __launch_bounds__(Sym3<EQ>::THREADS, Sym3<EQ>::RESIDENT)
    recon_sym3_kernel(const __grid_constant__ CUtensorMap umap, const __grid_constant__ Grid g,
                      const __grid_constant__ SymW w, const __grid_constant__ SymOff off, int zc, int wantInd,
                      double *__restrict__ F0, double *__restrict__ F1, double *__restrict__ F2,
                      float *__restrict__ W0, float *__restrict__ W1, float *__restrict__ W2,
                      double *__restrict__ src, uint8_t *__restrict__ status, double2 *__restrict__ lamvel,
                      double *__restrict__ bnd, DevScalars *sc) {
  pdl_begin();
  using L = Sym3<EQ>;
  using E = Eos<EQ>;
  constexpr int NV = L::NV, TX = L::TX, TN = L::TN, PX = L::PX, PN = L::PN;
  constexpr double big = 1.7976931348623157e308;
  extern __shared__ __align__(128) uint8_t smem[];
  double *ring = reinterpret_cast<double *>(smem);
  double *foot = reinterpret_cast<double *>(smem + L::OFF_F);  // [plane parity][e | c2 | ir][PN]
  const uint32_t bar = smem_u32(smem + L::OFF_BAR);
  const int tid = threadIdx.x, lane = tid & 31, v = tid >> 5;
  double *ex = reinterpret_cast<double *>(smem + L::OFF_X) + lane;       // [point][v][lane]
  // [rho max, rho min, e min, c^2 min, 2 div v][lane], then the bounds [3][lane]
  double *quant = reinterpret_cast<double *>(smem + L::OFF_Q) + lane;
  double *red = reinterpret_cast<double *>(smem + L::OFF_R) + lane;      // GLM speeds [v][2][lane]
  unsigned *mask = reinterpret_cast<unsigned *>(smem + L::OFF_M);
  // the rows of cells are numbered along blockIdx.x: a grid may have more than 65535 of them in y
  const unsigned nbx = (unsigned)(g.nx + L::BX - 1) / L::BX;
  const int j = (int)(blockIdx.x / nbx), i0 = (int)((blockIdx.x - (unsigned)j * nbx) * L::BX);
  const int k0 = (int)blockIdx.z * zc, k1 = k0 + zc < (int)g.nz ? k0 + zc : (int)g.nz;
  using Ring = PlaneRing<L::RING>;
  const int last = k1 + 1;
  auto issue = [&](int p) {
    const int s = Ring::slot(k0, p);
    mbar_arrive_expect_tx(bar + 8 * s, (uint32_t)(NV * TN * 8));
    tma_load_4d(smem_u32(ring + s * L::PLANE), &umap, i0, j, p + kRad, 0, bar + 8 * s);
  };
  auto wait = [&](int p) { return mbar_wait(bar + 8 * Ring::slot(k0, p), Ring::parity(k0, p)); };
  if (tid == 0) {
    for (int s = 0; s < L::RING; s++) mbar_init(bar + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    global_acquire_for_copies();
    for (int p = k0 - 2; p <= Ring::started(k0, last); p++) issue(p);
  }
  __syncthreads();
  const int own = 2 * TX + lane + 2, pown = PX + lane + 1;
  auto fill_foot = [&](const double *u, int par) {
    double *f = foot + par * (3 * PN);
    for (int t = tid; t < PN; t += L::THREADS) {
      const int a = t % PX, b = t / PX;
      sym_foot<EQ>(u + (b + 1) * TX + a + 1, TN, g.gamma, f + t, f + PN + t, f + 2 * PN + t);
    }
  };
  // The warps share the ingredients of the bounds: for a plane, warp 0 the
  // extrema of the density over 3 x 3 cells, warp 1 the minimum of the internal energy,
  // warp 2 that of the squared sound speed, warp 3 the x and y part of (twice) the
  // velocity divergence and the velocity along z.  (The comparisons skip NaN, as fmin does.)
  auto survey = [&](const double *u, int par, double &a, double &b) {
    const double *f = foot + par * (3 * PN);
    if (v == 0) {
      const double *r = u + DENS * TN + own;
      a = -big, b = big;
#pragma unroll
      for (int y = -1; y <= 1; y++)
#pragma unroll
        for (int x = -1; x <= 1; x++) {
          const double t = r[y * TX + x];
          a = t > a ? t : a;
          b = t < b ? t : b;
        }
    } else if (v <= 2) {
      const double *e = f + (v - 1) * PN + pown;
      a = big;
#pragma unroll
      for (int y = -1; y <= 1; y++)
#pragma unroll
        for (int x = -1; x <= 1; x++) {
          const double t = e[y * PX + x];
          a = t < a ? t : a;
        }
    } else if (v == 3) {
      const double *ir = f + 2 * PN + pown, *mx = u + MOMX * TN + own, *my = u + MOMY * TN + own;
      a = (mx[1] * ir[1] - mx[-1] * ir[-1]) + (my[TX] * ir[PX] - my[-TX] * ir[-PX]);
      b = u[MOMZ * TN + own] * ir[0];
    }
  };
  // surveys of planes p - 2 .. p joined into the ingredients of plane p - 1
  double am = 0.0, ac = 0.0, bm = 0.0, bc = 0.0;
  auto join = [&](double ap, double bp) {
    if (v == 0) {
      const double a = am > ac ? am : ac, b = bm < bc ? bm : bc;
      quant[0] = a > ap ? a : ap;
      quant[32] = b < bp ? b : bp;
    } else if (v <= 2) {
      const double a = am < ac ? am : ac;
      quant[(v + 1) * 32] = a < ap ? a : ap;
    } else if (v == 3) {
      quant[4 * 32] = ac + (bp - bm);
    }
    am = ac, ac = ap, bm = bc, bc = bp;
  };
  const int i = i0 + lane;
  const bool live = i < g.nx;
  bool ok = wait(k0 - 2) && wait(k0 - 1) && wait(k0) && wait(k0 + 1);
  const double *p0 = ring + L::PLANE;  // planes k0 - 1 .. k0 + 1 are in slots 1 .. 3
  if (ok) {
    fill_foot(p0, 0);
    fill_foot(p0 + L::PLANE, 1);
  }
  ok = __syncthreads_and(ok);
  // this thread's variable: the column's values in planes k - 2 .. k + 1 and the
  // combinations of planes k - 1 and k
  double cm2 = 0.0, cm1 = 0.0, c0 = 0.0, cp1 = 0.0;
  SymPlane qm{}, qo{};
  if (ok) {
    survey(p0, 0, am, bm);
    survey(p0 + L::PLANE, 1, ac, bc);
    const double *u = ring + v * TN + own;
    cm2 = u[0];
    cm1 = u[L::PLANE];
    c0 = u[2 * L::PLANE];
    cp1 = u[3 * L::PLANE];
    if constexpr (L::KEEP) {
      qm = sym_plane<TX>(u + L::PLANE, cm1);
      qo = sym_plane<TX>(u + 2 * L::PLANE, c0);
    }
  }
  smem_release_to_copies();  // (the column's values above are used much later)
  __syncthreads();
  if (L::KEEP && ok && tid == 0) issue(k0 + 2);  // into the slot of plane k0 - 2
  if (ok) fill_foot(p0 + 2 * L::PLANE, 0);
  ok = __syncthreads_and(ok);
  if (ok) {
    double ap = 0.0, bp = 0.0;
    survey(p0 + 2 * L::PLANE, 0, ap, bp);
    join(ap, bp);
  }
  // the cell's low face per axis, one plane on each iteration (a z face has the index of
  // the cell above it; fewer than 2^32 of each: a grid has at most 2^29 cells)
  unsigned wb[3];
#pragma unroll
  for (int d = 0; d < 3; d++) wb[d] = (unsigned)(((int64_t)k0 * g.fdim[d][1] + j) * g.fdim[d][0] + i);
  double *const F[3] = {F0, F1, F2};
  // the status of a plane's cell, once its points are all tested (and the GLM speed maxima)
  auto finish = [&](unsigned cc) {
    if (v != 0 || !live) return;
    unsigned m = 0xffffffffu;
#pragma unroll
    for (int t = 0; t < NV; t++) m &= mask[t];
    status[cc] = (m >> lane) & 1u;
    if constexpr (EQ == EQ_GLM) {
      double lam = 0.0, vel = 0.0;
#pragma unroll
      for (int t = 0; t < NV; t++) {
        lam = fmax(lam, red[(2 * t) * 32]);
        vel = fmax(vel, red[(2 * t + 1) * 32]);
      }
      lamvel[cc] = make_double2(lam, vel);
    }
  };
  // ring slots of planes k - 1 .. k + 2 (in doubles from the ring's start)
  int sm = L::PLANE, s0 = 2 * L::PLANE, sp = 3 * L::PLANE, sq = 4 % L::RING * L::PLANE;
#pragma unroll 1
  for (int k = k0; k < k1; k++) {
    const int par = (k - k0) & 1;
    ok = ok && wait(k + 2);
    if (ok && k + 1 < k1) fill_foot(ring + sq, 1 - par);
    smem_release_to_copies();
    if (!__syncthreads_and(ok)) {
      // a plane never arrived: record it, give the copies in flight a bounded time
      // to land, and leave
      if (tid == 0) {
        atomicExch(&sc->fault, 1u);
        for (int p = Ring::flying_from(k0, k); p <= Ring::flying_to(k, last); p++) wait(p);
      }
      return;
    }
    if (tid == 0 && k + 3 <= last) issue(k + 3);  // into the slot of plane k - 1 (KEEP) or k - 2
    if (k > k0) finish(wb[2] - (unsigned)(g.nx * g.ny));
    double ap = 0.0, bp = 0.0;
    if (k + 1 < k1) survey(ring + sq, 1 - par, ap, bp);
    if (v == ETOT) {
      const SymBounds bd = sym_bounds(SymExt{quant[0], quant[32], quant[64], quant[96]}, quant[128]);
      quant[5 * 32] = bd.minDens > 0.0 ? bd.minDens : 0.0;
      quant[6 * 32] = bd.maxDens;
      quant[7 * 32] = bd.minEint;
      if (live) {
        bnd[wb[2]] = bd.minDens;  // for the heavy pass
        bnd[g.n + wb[2]] = bd.maxDens;
        bnd[2 * g.n + wb[2]] = bd.minEint;
      }
    }
    // ---- the contraction of this warp's variable
    const double *u = ring + v * TN + own;
    const double cp2 = u[sq];
    const SymPlane qp = sym_plane<TX>(u + sp, cp1);
    if constexpr (!L::KEEP) {
      qm = sym_plane<TX>(u + sm, cm1);
      qo = sym_plane<TX>(u + s0, c0);
    }
    double s[33];
    sym_combine<TX>(u + s0, qm, qo, qp, cm2, cm1, c0, cp1, cp2, s);
    if constexpr (L::KEEP) qm = qo, qo = qp;
    cm2 = cm1, cm1 = c0, c0 = cp1, cp1 = cp2;
    bool inside = true;
    double lam = 0.0, vel = 0.0, minDens, maxDens, minEint;
#pragma unroll
    for (int ph = 0; ph < L::NG; ph += L::GP) {
#pragma unroll
      for (int gr = 0; gr < L::GP; gr++) {
        const int d = ph + gr;
        double f[8];
        sym_points(w.a[d], s, f);
        double *x = ex + (gr * 8 * NV + v) * 32;
#pragma unroll
        for (int o = 0; o < 8; o++) x[o * NV * 32] = f[o];
        if (!live) continue;
        if (d < 3) {
          char *fb = reinterpret_cast<char *>(F[d] + (int64_t)v * g.nface[d] + wb[d]);
#pragma unroll
          for (int o = 0; o < 8; o++) *reinterpret_cast<double *>(fb + off.f[d][o]) = f[o];
        } else {
#pragma unroll
          for (int o = 0; o < 8; o++) src[(int64_t)(sym_inner_q<3>(o) * NV + v) * g.n + wb[2]] = f[o];
        }
      }
      // ---- the points of these groups, shared among the warps
      __syncthreads();
      if (ph == 0) {
        minDens = quant[5 * 32], maxDens = quant[6 * 32], minEint = quant[7 * 32];
        if (k + 1 < k1) join(ap, bp);  // plane k's ingredients have been read
      }
#pragma unroll 1
      for (int p = v; p < L::GP * 8; p += NV) {
        const double *x = ex + p * NV * 32;
        const int d = ph + (p >> 3);
        const double rho = x[DENS * 32], ux = x[MOMX * 32], uy = x[MOMY * 32], uz = x[MOMZ * 32];
        const double ir = rcp_nr(rho);
        double other = 0.5 * (ux * ux + uy * uy + uz * uz) * ir, b2 = 0.0, bx = 0.0;
        if constexpr (EQ == EQ_GLM) {
          bx = x[MAGX * 32];
          const double by = x[MAGY * 32], bz = x[MAGZ * 32], psi = x[PSI * 32];
          b2 = bx * bx + by * by + bz * bz;
          other = 0.5 * b2 + other + 0.5 * psi * psi;
        }
        const double ei = x[ETOT * 32] - other;
        // not inside unless clear of rounding: the heavy pass then decides exactly
        // (theta stays 1 there when the states are inside after all), so the kinetic
        // energy needs no IEEE division
        inside = inside && rho > minDens && rho < maxDens &&
                 ei - minEint > 8.9e-16 * (fabs(other) + fabs(ei)) + 1e-300;
        if (L::NG == 3 || d < 3) {
          const double pr = (g.gamma - 1.0) * ei;
          if (wantInd && live) {
            float *Wd = (d == 0 ? W0 + wb[0] : (d == 1 ? W1 + wb[1] : W2 + wb[2]));
            Wd[off.w[d][p & 7]] = E::template weno_store<3>(g.gamma, rho, pr);
          }
          if constexpr (EQ == EQ_GLM) {
            // SpeedEstimate_K<MHD_GLM> (MHD_GLM_K.H:213-310): x components on every face
            const double asq = g.gamma * pr * ir, absq = asq + b2 * ir, blsq = bx * bx * ir;
            const double vv = fabs(ux * ir);
            const double l = sqrt_nr(0.5 * (absq + sqrt_nr(absq * absq - 4.0 * asq * blsq))) + vv;
            vel = vv > vel ? vv : vel;
            lam = l > lam ? l : lam;
          }
        }
      }
      if (ph + L::GP < L::NG) __syncthreads();
    }
    const unsigned in = __ballot_sync(0xffffffffu, inside);
    if (lane == 0) mask[v] = in;
    if constexpr (EQ == EQ_GLM) {
      red[(2 * v) * 32] = lam;
      red[(2 * v + 1) * 32] = vel;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) wb[d] += (unsigned)(g.fdim[d][0] * g.fdim[d][1]);
    sm = s0, s0 = sp, sp = sq, sq = sq == (L::RING - 1) * L::PLANE ? 0 : sq + L::PLANE;
  }
  __syncthreads();
  finish(wb[2] - (unsigned)(g.nx * g.ny));
}

// ---------------------------------------------------------------------------
// 2D: one 32 x 8 tile per block
template <int EQ>
struct Sym2 {
  static constexpr int NV = Eos<EQ>::NV, BX = 32, BY = 8, THREADS = BX * BY;
  static constexpr int TX = BX + 2 * kRad, TY = BY + 2 * kRad, TN = TX * TY;
  static constexpr int PX = BX + 2, PY = BY + 2, PN = PX * PY;
  static constexpr int RESIDENT = 2;
  static_assert((TX * 8) % 16 == 0, "TMA box inner extent");
};

template <int EQ>
__global__ void __launch_bounds__(Sym2<EQ>::THREADS, Sym2<EQ>::RESIDENT)
    recon_sym2_kernel(const __grid_constant__ CUtensorMap umap, const __grid_constant__ Grid g,
                      const __grid_constant__ SymW w, int wantInd, double *__restrict__ F0, double *__restrict__ F1,
                      float *__restrict__ W0, float *__restrict__ W1, double *__restrict__ src,
                      uint8_t *__restrict__ status, double2 *__restrict__ lamvel, double *__restrict__ bnd,
                      DevScalars *sc) {
  pdl_begin();
  using L = Sym2<EQ>;
  constexpr int NV = L::NV, TX = L::TX, TN = L::TN, PX = L::PX, PN = L::PN;
  __shared__ __align__(128) double tile[NV * TN];
  __shared__ double foot[3 * PN];
  __shared__ uint64_t sbar;
  const uint32_t bar = smem_u32(&sbar);
  const int tid = threadIdx.x, lane = tid & 31, ty = tid >> 5;
  const int i0 = (int)(blockIdx.x * L::BX), j0 = (int)(blockIdx.y * L::BY);
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_arrive_expect_tx(bar, (uint32_t)sizeof(tile));
    global_acquire_for_copies();
    tma_load_4d(smem_u32(tile), &umap, i0, j0, 0, 0, bar);
  }
  __syncthreads();
  if (!mbar_wait(bar, 0)) {
    // (each thread for itself: its cell stays unwritten, whatever the others saw)
    atomicExch(&sc->fault, 1u);
    mbar_wait(bar, 0);  // a bounded time for the copy to land
    return;
  }
  for (int t = tid; t < PN; t += L::THREADS) {
    const int a = t % PX, b = t / PX;
    sym_foot<EQ>(tile + (b + 1) * TX + a + 1, TN, g.gamma, foot + t, foot + PN + t, foot + 2 * PN + t);
  }
  __syncthreads();
  const int64_t i = i0 + lane, j = j0 + ty;
  if (i >= g.nx || j >= g.ny) return;
  const int pown = (ty + 1) * PX + lane + 1;
  const double *u = tile + (ty + 2) * TX + lane + 2;
  constexpr double big = 1.7976931348623157e308;
  SymExt x{-big, big, big, big};
#pragma unroll
  for (int b = -1; b <= 1; b++)
#pragma unroll
    for (int a = -1; a <= 1; a++) {
      const double r = u[DENS * TN + b * TX + a];
      x.rMax = fmax(x.rMax, r);
      x.rMin = fmin(x.rMin, r);
      x.eMin = fmin(x.eMin, foot[pown + b * PX + a]);
      x.c2Min = fmin(x.c2Min, foot[PN + pown + b * PX + a]);
    }
  const double *ir = foot + 2 * PN + pown, *mx = u + MOMX * TN, *my = u + MOMY * TN;
  const double div2 = (mx[1] * ir[1] - mx[-1] * ir[-1]) + (my[TX] * ir[PX] - my[-TX] * ir[-PX]);
  SymCell cl;
  cl.bd = sym_bounds(x, div2);
  cl.c = j * g.nx + i;
#pragma unroll
  for (int d = 0; d < 2; d++) {
    cl.fidx[d] = j * g.fdim[d][0] + i;
    cl.fstr[d] = d == 0 ? 1 : g.fdim[1][0];
  }
  bnd[cl.c] = cl.bd.minDens;  // for the heavy pass
  bnd[g.n + cl.c] = cl.bd.maxDens;
  bnd[2 * g.n + cl.c] = cl.bd.minEint;
  double *const F[2] = {F0, F1};
  float *const W[2] = {W0, W1};
  sym_cell<EQ>([&](int v, int dx, int dy) { return u[v * TN + dy * TX + dx]; }, w, g, cl, wantInd, F, W, src, status,
               lamvel);
}

// ---------------------------------------------------------------------------
// host

// Parity weights of the full stencil (SymW) for two Gauss points.  For the point of a
// group on the positive side of every axis with weights W(c), the combination of
// parity e over the orbit of a stencil cell r >= 0 with m nonzero coordinates has the
// weight sum over signs t of (product of t_i, i in e) W(t r) / 2^m.  Returns nonzero if
// the weights of a group's points are not mirror images of each other.
int fill_sym_weights(const kfvm_stencil &st, bool interior, SymW &out) {
  const int dim = st.dim, C = st.n_cells, np = 1 << dim;
  std::memset(&out, 0, sizeof(out));
  auto find = [&](int x, int y, int z) {
    for (int c = 0; c < C; c++)
      if (st.off[0][c] == x && st.off[1][c] == y && (dim == 2 || st.off[2][c] == z)) return c;
    return -1;
  };
  // representatives of the combinations in the kernel's order, and the parities' bits
  static const int r3[11][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {2, 0, 0}, {0, 2, 0},
                                {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}};
  static const int r2[6][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {2, 0, 0}, {0, 2, 0}, {1, 1, 0}};
  static const int e3[8] = {0, 1, 2, 4, 3, 5, 6, 7}, e2[4] = {0, 1, 2, 3};
  const int nr = dim == 3 ? 11 : 6;
  for (int gr = 0; gr < dim + (interior ? 1 : 0); gr++) {
    auto weight = [&](int o, int c) {  // stencil cell c, point o (bit d: positive side of axis d)
      const int x = o & 1, y = (o >> 1) & 1, z = (o >> 2) & 1;
      if (gr == dim) return st.cell_w[0][dim == 2 ? 2 * x + y : (2 * x + y) * 2 + z][c];
      const int q = dim == 2 ? (gr == 0 ? y : x) : (gr == 0 ? 2 * y + z : (gr == 1 ? 2 * x + z : 2 * x + y));
      return st.face_w[0][2 * gr + ((o >> gr) & 1)][q][c];
    };
    for (int o = 0; o < np; o++)
      for (int c = 0; c < C; c++) {
        int m[3];
        for (int d = 0; d < 3; d++) m[d] = d < dim ? (int)st.off[d][c] * ((o >> d) & 1 ? 1 : -1) : 0;
        const int cm = find(m[0], m[1], m[2]);
        if (cm < 0 || weight(o, c) != weight(np - 1, cm)) return 1;
      }
    int n = 0;
    for (int e = 0; e < np; e++) {
      const int bits = dim == 3 ? e3[e] : e2[e];
      for (int r = 0; r < nr; r++) {
        const int *rep = dim == 3 ? r3[r] : r2[r];
        int nz = 0;
        bool odd = true;  // odd parities need a nonzero coordinate
        for (int d = 0; d < dim; d++) {
          nz += rep[d] != 0;
          odd = odd && (!((bits >> d) & 1) || rep[d] != 0);
        }
        if (!odd) continue;
        long double a = 0.0L;
        for (int t = 0; t < np; t++) {
          int p[3] = {rep[0], rep[1], rep[2]}, sgn = 1;
          bool skip = false;
          for (int d = 0; d < dim; d++)
            if (!((t >> d) & 1)) {
              if (rep[d] == 0) skip = true;  // each member of the orbit once
              p[d] = -p[d];
              if ((bits >> d) & 1) sgn = -sgn;
            }
          if (!skip) a += sgn * (long double)weight(np - 1, find(p[0], p[1], p[2]));
        }
        out.a[gr][n++] = (double)(a / (1 << nz));
      }
    }
  }
  return 0;
}

int recon_sym_state_map(CUtensorMap *map, const double *U, const Grid &g, int dim, int nv) {
  const uint64_t planes = (uint64_t)(g.pvol / (g.px * g.py));
  const uint64_t dims[4] = {(uint64_t)g.px, (uint64_t)g.py, planes, (uint64_t)nv};
  const uint64_t strides[3] = {(uint64_t)g.px * 8, (uint64_t)(g.px * g.py) * 8, (uint64_t)g.pvol * 8};
  const int rows = dim == 2 ? Sym2<EQ_HYDRO>::TY : Sym3<EQ_HYDRO>::TY;
  const uint32_t box[4] = {(uint32_t)Sym3<EQ_HYDRO>::TX, (uint32_t)rows, 1u, (uint32_t)nv};
  return encode_tensor_map_8b(map, U, 4, dims, strides, box);
}

// A chunk costs about 2.5 planes' time besides its own planes (the first loads and
// footprints), and the blocks run in waves of the resident ones: the chunk count with the
// least waves times chunk cost.  The choice depends little on that cost: with 0.5 and 1.5
// planes nine sizes from 32^3 to 256 x 256 x 40 take the same times within 6 %, with 3.5
// 160^3 takes 1.42 instead of 1.28 ms, with 8 the grid of 97 x 75 x 51 0.22 instead of 0.17.
int recon_sym_planes(int eq, const Grid &g, int nsm) {
  const int64_t cols = (g.nx + Sym3<EQ_HYDRO>::BX - 1) / Sym3<EQ_HYDRO>::BX * g.ny;
  const int64_t slots = (int64_t)nsm * (eq == EQ_GLM ? Sym3<EQ_GLM>::RESIDENT : Sym3<EQ_HYDRO>::RESIDENT);
  int64_t zc = g.nz;
  double best = 1e300;
  for (int64_t n = 1; n <= g.nz; n++) {
    const int64_t len = (g.nz + n - 1) / n, waves = (cols * ((g.nz + len - 1) / len) + slots - 1) / slots;
    const double cost = (double)waves * ((double)len + 2.5);
    if (cost < best) {
      best = cost;
      zc = len;
    }
  }
  return (int)zc;
}

template <int EQ>
static cudaError_t sym3(const ReconSymArgs &a, const CUtensorMap &umap, const Grid &g, const SymW &w, cudaStream_t s) {
  using L = Sym3<EQ>;
  static const cudaError_t attr =
      cudaFuncSetAttribute(recon_sym3_kernel<EQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES);
  if (attr != cudaSuccess) return attr;
  SymOff off;
  for (int d = 0; d < 3; d++)
    for (int o = 0; o < 8; o++) {
      const int hi = (o >> d) & 1, q = (hi ? 0 : 4) + sym_face_q<3>(d, o);
      const int64_t str = hi ? (d == 0 ? 1 : (d == 1 ? g.fdim[1][0] : g.fdim[2][0] * g.fdim[2][1])) : 0;
      off.f[d][o] = (q * L::NV * g.nface[d] + str) * 8;
      off.w[d][o] = q * g.nface[d] + str;
    }
  const dim3 grid((unsigned)((g.nx + L::BX - 1) / L::BX * g.ny), 1u, (unsigned)((g.nz + a.planes - 1) / a.planes));
  return launch_chain(g.chain, recon_sym3_kernel<EQ>, grid, dim3(L::THREADS), L::BYTES, s, umap, g, w, off, a.planes, a.wantInd,
                      a.F[0], a.F[1], a.F[2], a.W[0], a.W[1], a.W[2], a.src, a.status, a.lamvel, a.bnd, a.sc);
}

template <int EQ>
static cudaError_t sym2(const ReconSymArgs &a, const CUtensorMap &umap, const Grid &g, const SymW &w, cudaStream_t s) {
  using L = Sym2<EQ>;
  const dim3 grid((unsigned)((g.nx + L::BX - 1) / L::BX), (unsigned)((g.ny + L::BY - 1) / L::BY));
  return launch_chain(g.chain, recon_sym2_kernel<EQ>, grid, dim3(L::THREADS), 0, s, umap, g, w, a.wantInd, a.F[0], a.F[1], a.W[0],
                      a.W[1], a.src, a.status, a.lamvel, a.bnd, a.sc);
}

cudaError_t launch_recon_sym(int dim, int eq, const ReconSymArgs &a, const CUtensorMap &umap, const Grid &g,
                             const SymW &w, cudaStream_t s) {
  if (dim == 2) {
    if (eq == EQ_HYDRO) return sym2<EQ_HYDRO>(a, umap, g, w, s);
    if (eq == EQ_NS) return sym2<EQ_NS>(a, umap, g, w, s);
    if (eq == EQ_GLM) return sym2<EQ_GLM>(a, umap, g, w, s);
  } else {
    if (eq == EQ_HYDRO) return sym3<EQ_HYDRO>(a, umap, g, w, s);
    if (eq == EQ_NS) return sym3<EQ_NS>(a, umap, g, w, s);
    if (eq == EQ_GLM) return sym3<EQ_GLM>(a, umap, g, w, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace kfvm
