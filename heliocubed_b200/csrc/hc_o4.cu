// Fourth-order Berta pointwise-WENOZ operator on batched ghosted boxes,
// src/BoxOp_BertaCubedSphereImplem.H:1737-2076 with the Roe glue of
// src/BoxOp_RoeCubedSphere.H:29-145 and the Powell terms of
// src/BoxOp_DivBcleaning.H:35-172.  FP64.
//
// Kernels per evaluation, each one launch over every box and (for the face
// kernels) all three directions of a batch:
//   o4PrimAvgKernel, o4ThetaRawKernel, o4PointKernel: detector and point values
//   o4FaceReconKernel: both states of every face
//   o4FaceRiemannKernel: point flux sums and dissipation
//   o4FaceAvgKernel: face averages and their radial-area products
//   o4FaceFinalKernel: mapped final flux of every face
//   o4CellKernel: flux divergence and Powell source into rhs
// and on a side stream o4PowellAvgKernel, o4PowellFluxKernel, o4PowellDivKernel.
// Every intermediate covers what a later kernel reads of the box the reference
// computes it on.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "hc_device.cuh"
#include "hc_level.h"

namespace hc {
namespace {

struct Box3 {
  int lo[3], hi[3];
  __host__ __device__ Box3 grow(int g) const { Box3 b = *this; for (int d = 0; d < 3; ++d) { b.lo[d] -= g; b.hi[d] += g; } return b; }
  __host__ __device__ Box3 growTrans(int d, int g) const {
    Box3 b = *this;
    for (int t = 0; t < 3; ++t) if (t != d) { b.lo[t] -= g; b.hi[t] += g; }
    return b;
  }
  __host__ __device__ Box3 extrude(int d) const { Box3 b = *this; b.hi[d] += 1; return b; }
  __host__ __device__ int n(int d) const { return hi[d] - lo[d] + 1; }
  __host__ __device__ long size() const { return (long)n(0) * n(1) * n(2); }
};

__host__ __device__ inline Reg regOf(const Box3& b) {
  Reg r;
  for (int d = 0; d < 3; ++d) { r.lo[d] = b.lo[d]; r.n[d] = b.n(d); }
  r.N = b.size();
  return r;
}

// Offset of (i, j, k) in an array laid out on region r.  Every array of a
// box holds fewer than 2^31 points per component (o4BatchCreate rejects
// larger boxes), so the offset is formed in 32-bit arithmetic, which the
// compiler shares between the neighbours of a stencil.
__device__ __forceinline__ long roff(const Reg& r, int i, int j, int k) {
  return (long)((i - r.lo[0]) + r.n[0] * ((j - r.lo[1]) + r.n[1] * (k - r.lo[2])));
}

// Offsets of the face arrays inside a direction's face scratch (units of
// F.N).  Vector components of the flux sums, dissipations and averages are
// kept along (normal, next, next but one) native direction; the flux sum of
// the normal field vanishes and has no array.  Arrays share places with what
// nothing reads any more: the final fluxes (Cartesian components) that of the
// flux sums and pressures, the area products that of the left states, and
// the dissipation that of the right states (a face's states are in its
// thread's hands before the thread writes the face's dissipation).
enum FaceArr { F_FS = 0, F_PS = 7, F_FX = 0, F_L = 8, F_X = 8, F_T3 = 15, F_R = 16, F_QD = 16, F_THF = 24, F_BP = 25,
               F_SPD = 26, F_BF = 27 };
static_assert(F_BF + 1 == kO4FaceArrays && F_T3 == F_X + 7, "face arrays");
// F_FS array of component c in (rho, m_n, m_1, m_2, E, B_n, B_1, B_2) order (c != 5), also of F_X.
__host__ __device__ constexpr int fluxSlot(int c) { return c < 5 ? c : c - 1; }

struct Ctx {
  O4Args a;
  int d;
  Box3 V, G, GR, GD, F, V0, V1;
  Reg gr, fr, v1r, vr;
};

// Regions the operator's kernels loop over (host and device agree through
// this one table): the work lists of a batch are built from it.  The face
// regions are walked for all three directions by one launch.
enum RegionId { RG_G = 0, RG_GR, RG_V, RG_V1, RG_F, RG_PB, RG_V0, RG_PF, RG_COUNT };
__host__ __device__ constexpr bool faceRegion(int id) { return id >= RG_F; }
__host__ __device__ inline Box3 regionOf(const Ctx& c, int id) {
  switch (id) {
    case RG_G: return c.G;
    case RG_GR: return c.GR;
    case RG_V: return c.V;
    case RG_V1: return c.V1;
    case RG_F: return c.F;
    case RG_PB: return c.V0.growTrans(c.d, 1);
    case RG_V0: return c.V0;
    default: {  // Powell fluxes: the faces of V1, and their radial neighbours for the area product
      Box3 b = c.V1.extrude(c.d);
      if (c.d != 0) { b.lo[0] -= 1; b.hi[0] += 1; }
      return b;
    }
  }
}
// Whether at most one coordinate of a cell lies outside the valid box grown
// by g: the corners of the ghosted box, which no face stencil reaches (the
// stencils are long along one direction only), are not computed.
__device__ __forceinline__ bool crossShaped(const Box3& V, int g, int i, int j, int k) {
  const bool a = i < V.lo[0] - g || i > V.hi[0] + g, b = j < V.lo[1] - g || j > V.hi[1] + g,
             c = k < V.lo[2] - g || k > V.hi[2] + g;
  return !((a && b) || (a && c) || (b && c));
}
// Points a CTA takes per pass: the face averages give up one thread at each
// end, whose averages only serve their neighbours.
constexpr int kAvgPoints = 126;
__host__ __device__ constexpr int passPoints(int id) { return id == RG_PB ? kAvgPoints : 128; }

// One CTA's work: flat points begin .. end - 1 of one region of box `box`,
// direction `dir`; with march > 0 its points are columns of that many faces.
struct WorkChunk {
  int box, dir, march;
  long begin, end;
};

// The face averages and final fluxes march along an angular direction
// transverse to the faces (k, or j for the faces of k): a thread takes
// `march` faces and keeps the values of the row behind and of its row in
// registers, so a row is read from L2 once and not once per neighbour.
__host__ __device__ constexpr bool marches(int id) { return id == RG_PB || id == RG_V0; }
__host__ __device__ constexpr int marchDim(int d) { return d == 2 ? 1 : 2; }
__host__ __device__ inline long columns(const Box3& b, int d, int march) {
  const int t = marchDim(d);
  return (long)b.n(0) * b.n(3 - t) * ((b.n(t) + march - 1) / march);
}
// Points per CTA of a work list: its total points over about 148 x 16 CTAs,
// rounded up to whole passes of the CTA and held within 1 to 16 passes, so
// one launch has as many CTAs whatever the box sizes.
inline long chunkPoints(long total, long pass) {
  const long target = (total + 148L * 16 - 1) / (148L * 16);
  const long passes = (target + pass - 1) / pass;
  return pass * (passes < 1 ? 1 : passes > 16 ? 16 : passes);
}

// The box the face arrays of every direction are laid out on: the face
// boxes G.extrude(d).grow(-3) together.
Box3 faceBox(const Box3& G) {
  Box3 FB = G.grow(-3);
  for (int q = 0; q < 3; ++q) FB.hi[q] += 1;
  return FB;
}

Ctx makeCtx(const O4Args& a, int d) {
  Ctx c;
  c.a = a;
  c.d = d;
  for (int q = 0; q < 3; ++q) { c.V.lo[q] = a.vlo[q]; c.V.hi[q] = a.vhi[q]; }
  c.G = c.V.grow(a.ghost);
  c.GR = c.G.grow(-1);
  c.GD = c.G.grow(-2);
  c.V0 = c.V.extrude(d);
  c.V1 = c.V.grow(1);
  // faces whose states something reads: one beyond the valid box along the
  // normal (the Powell fluxes of V1), two across (the averages' neighbours)
  c.F = c.V1.extrude(d).growTrans(d, 1);
  c.gr = regOf(c.G);
  // face scratch is laid out on the largest face box over the directions
  c.fr = regOf(faceBox(c.G));
  c.v1r = regOf(c.V1);
  c.vr = a.rr.N ? a.rr : regOf(c.V);
  return c;
}

// ---- geometry access -------------------------------------------------------
// Position of angular (j, k) of a panel in the metric tables.
__device__ __forceinline__ long angular(const O4Geo& g, long plane, int j, int k) {
  const int n = g.na + 2 * g.ext + 1;
  return (plane * n + (k + g.ext)) * n + (j + g.ext);
}
__device__ __forceinline__ const double* faceRec(const O4Geo& g, int block, int d, int j, int k) {
  return d == 0 ? g.face0 + angular(g, block, j, k) * kO4FaceRec0
                : g.face12 + angular(g, block * 2 + (d - 1), j, k) * kO4FaceRec12;
}
__device__ __forceinline__ const double* roeRec(const O4Geo& g, int block, int d, int j, int k) {
  return g.frames + angular(g, block * 3 + d, j, k) * kO4RoeRec;
}
__device__ __forceinline__ const double* cellBasis(const O4Geo& g, int block, int j, int k) {
  const long n = g.na + 2 * g.ext + 1;
  return g.cell + (((long)block * n + (k + g.ext)) * n + (j + g.ext)) * 9;
}
__device__ __forceinline__ double4 radialRow(const O4Geo& g, int i) { return g.radial[i + kO4Rad]; }
__device__ __forceinline__ double adjDr(const O4Geo& g, int d, int i) {
  const double4 r = radialRow(g, i);
  return d == 0 ? r.x : r.y;
}
__device__ __forceinline__ Rn radialPoint(const O4Geo& g, int d, int i) {
  if (d == 0) return adjDr(g, 0, i);
  const Rn a = adjDr(g, d, i);
  return mad(-1.0 / 24.0, mad(-2.0, a, adjDr(g, d, i + 1)) + adjDr(g, d, i - 1), a);
}

// ---- pointwise pieces -----------------------------------------------------
// Divisions by 4 pi and 8 pi are multiplications by the rounded reciprocals
// (a one-ulp difference from the reference's x / 8.0 / M_PI).
constexpr double kInv4Pi = 0.25 / kPi, kInv8Pi = 0.125 / kPi;
// f_sphToPrim + energies + pressure (src/BoxOp_BertaCubedSphereImplem.H:212-340)
__device__ __forceinline__ void sphToPrim(const double u[8], const double* A, double gamma, double w[8]) {
  const Rn rho = dmax(u[0], kRHO00), inv = rcpDensity(rho);
  w[0] = rho;
  Rn ke = 0.0, me = 0.0;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    w[1 + e] = inv * u[1 + e];
    w[5 + e] = u[5 + e];
  }
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const Rn v = dot3(A[3 * e], w[1], A[3 * e + 1], w[2], A[3 * e + 2], w[3]);
    const Rn b = dot3(A[3 * e], w[5], A[3 * e + 1], w[6], A[3 * e + 2], w[7]);
    ke = mad(v, v, ke);
    me = mad(b, b, me);
  }
  const Rn p = (mad(-0.5 * rho, ke, u[4]) - kInv8Pi * me) * (gamma - 1.0);
  w[4] = p < 0.0 ? 0.0 : p.v;
}

// bertaNormalizeWenoStencil (:747-773)
template <int N>
__device__ __forceinline__ double normalizeStencil(double (&v)[N]) {
  double scale = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) scale = dmax(scale, fabs(v[i]));
  if (scale == 0.0) {
    for (int i = 0; i < N; ++i) if (v[i] != 0.0) return v[i];
    return scale;
  }
  if (scale > 0.0) {
    if (scale >= 2.2250738585072014e-308) {
      const double inverse = 1.0 / scale;
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] *= inverse;
    } else {
      for (int i = 0; i < N; ++i) v[i] /= scale;
    }
  }
  return scale;
}

// f_wenoz_pointwise_faceF (:782-878), one component, cells W[i-3..i+2]: the
// fifth-order states of both sides of the face.
//
// The two sides share the differences of the six cells: with d_q = v[q+1] -
// v[q] and s_q = d_q - d_{q-1}, four times the smoothness indicators are
// (13/3) s^2 + b^2 (b = 3 d1 - d0, d1 + d2, 3 d2 - d3 on the left side,
// mirrored on the right), the squares of s are common, and the candidate
// states are c + e / 8 with e = 7 d1 - 3 d0, d1 + 3 d2, 5 d2 - d3.  With
// a_k = d_k (1 + tau / D_k), D_k = beta_k + eps, the state is sum a_k q_k /
// sum a_k; the a_k are replaced by the proportional d_k (D_k + tau)
// prod_{j != k} D_j, and both sides' quotients come from one reciprocal.
// The weights do not change with the scale of the stencil (eps guards 0 / 0
// only), so the stencil is scaled by the power of two of its largest value,
// formed from the exponents in integer arithmetic: |v| < 2, every weight
// lies in [6e-119, 1e9], and neither the product of the sums nor its
// reciprocal, nor the quotients formed before they are scaled back, under- or
// overflow (values below 8e307, whose differences are finite).  A zero
// stencil gives zeros; a NaN or infinity gives NaN.
// The reconstruction is bound by instruction issue; sharing takes about 95
// FP64 instructions per component and face where two separate sides with
// divisions took 170 (64 x 32^2 x 6: 89 -> 70 us per direction).
__device__ __forceinline__ void wenozFace(const double v[6], double& L, double& R) {
  int top = 0;
#pragma unroll
  for (int q = 0; q < 6; ++q) top = max(top, __double2hiint(v[q]) & 0x7fffffff);
  const int e = min(max(top >> 20, 1), 2045);  // 2^(e - 1023) <= largest |v|
  const Rn inv = __hiloint2double((2046 - e) << 20, 0);
  // 2^(e - 1023) / 8
  const double scale8 = e > 3 ? __hiloint2double((e - 3) << 20, 0) : __hiloint2double(e << 20, 0) * 0.125;
  const Rn d0 = (Rn(v[1]) - v[0]) * inv, d1 = (Rn(v[2]) - v[1]) * inv, d2 = (Rn(v[3]) - v[2]) * inv,
           d3 = (Rn(v[4]) - v[3]) * inv, d4 = (Rn(v[5]) - v[4]) * inv;
  const double eps = 4.0e-40;
  auto square = [&](Rn s) { return mad((13.0 / 3.0) * s, s, eps); };
  const Rn t1 = square(d1 - d0), t2 = square(d2 - d1), t3 = square(d3 - d2), t4 = square(d4 - d3);
  auto side = [](Rn D0, Rn D1, Rn D2, Rn e0, Rn e1, Rn e2, Rn& num, Rn& den) {
    const Rn tau = fabs((D0 - D2).v), D02 = D0 * D2;
    const Rn w0 = (D0 + tau) * (D1 * D2), w1 = (D1 + tau) * (10.0 * D02), w2 = (D2 + tau) * (5.0 * (D0 * D1));
    num = dot3(w0, e0, w1, e1, w2, e2);
    den = w0 + w1 + w2;
  };
  auto plus = [](Rn t, Rn x) { return mad(x, x, t); };
  Rn nl, dl, nr, dr;
  side(plus(t1, mad(3.0, d1, -d0)), plus(t2, d1 + d2), plus(t3, mad(3.0, d2, -d3)), mad(-3.0, d0, 7.0 * d1),
       mad(3.0, d2, d1), mad(5.0, d2, -d3), nl, dl);
  // mirrored; its e carry the opposite sign
  side(plus(t4, mad(3.0, d3, -d4)), plus(t3, d3 + d2), plus(t2, mad(3.0, d2, -d1)), mad(-3.0, d4, 7.0 * d3),
       mad(3.0, d2, d3), mad(5.0, d2, -d1), nr, dr);
  // the quotients first: the reciprocal of a constant stencil is near 1e234
  const Rn q = rcpN(dl * dr);
  L = mad(nl * dr * q, scale8, v[2]);
  R = mad(-(nr * dl) * q, scale8, v[3]);
}

// f_weno3_pointwise_faceF (:881-946), one component, cells W[i-2..i+1].
__device__ __forceinline__ void weno3Face(const double in[4], double dx2, double& L, double& R) {
  // a_k = d_k (1 + tau / (beta_k + eps)), both sides' quotients from one
  // reciprocal; eps = dx^2 is a size of the normalised stencil, so the
  // stencil is normalised by its largest value.
  double v[4] = {in[0], in[1], in[2], in[3]};
  const double scale = normalizeStencil(v);
  if (scale == 0.0) { L = R = 0.0; return; }
  const Rn d0 = Rn(v[1]) - v[0], d1 = Rn(v[2]) - v[1], d2 = Rn(v[3]) - v[2];
  const Rn B0 = mad(d0, d0, dx2), B1 = mad(d1, d1, dx2), B2 = mad(d2, d2, dx2);
  auto side = [](Rn Bp, Rn Bm, Rn jump, Rn q0, Rn q1, Rn& num, Rn& den) {
    const Rn tau = jump * jump, w0 = 3.0 * ((Bp + tau) * Bm), w1 = (Bm + tau) * Bp;
    num = mad(w0, q0, w1 * q1);
    den = w0 + w1;
  };
  Rn nl, dl, nr, dr;
  const Rn mid = 0.5 * (Rn(v[1]) + v[2]);
  side(B1, B0, d1 - d0, mid, mad(0.5, d0, v[1]), nl, dl);
  side(B1, B2, d2 - d1, mid, mad(-0.5, d2, v[2]), nr, dr);
  const Rn q = scale * Rn(rcpN(dl * dr));
  L = nl * dr * q;
  R = nr * dl * q;
}

__device__ __forceinline__ double minmod3(double a, double b, double c) {
  if (a > 0.0 && b > 0.0 && c > 0.0) return dmin(a, dmin(b, c));
  if (a < 0.0 && b < 0.0 && c < 0.0) return dmax(a, dmax(b, c));
  return 0.0;
}

// f_plm_pointwise_faceF (:949-991), one component, cells W[i-2..i+1].
__device__ __forceinline__ void plmFallbackFace(const double in[4], double& L, double& R) {
  const double theta = 1.5;
  const double dm = in[1] - in[0], dp = in[2] - in[1], dc = 0.5 * (in[2] - in[0]);
  L = in[1] + 0.5 * minmod3(theta * dm, dc, theta * dp);
  const double rdm = in[2] - in[1], rdp = in[3] - in[2], rdc = 0.5 * (in[3] - in[1]);
  R = in[2] - 0.5 * minmod3(theta * rdm, rdc, theta * rdp);
}

__device__ __forceinline__ bool usablePrimitive(const double w[8]) {
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 8; ++c) ok = ok && isfinite(w[c]);
  return ok && w[0] >= kRHO00 && w[4] >= 0.0;
}

// Pairs of a face's record in the frame table.  The second half is read
// after the solver (volatile: not merged with an earlier read), so it does
// not occupy registers while the solver runs.
__device__ __forceinline__ double2 roeLoad2(const double* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

// ---- stencils on scratch arrays --------------------------------------------
struct View {
  const double* p;
  Reg r;
  __device__ double operator()(int c, int i, int j, int k) const { return p[c * r.N + roff(r, i, j, k)]; }
};


__device__ __forceinline__ double lapCell(const View& f, int c, int i, int j, int k) {
  return (f(c, i - 1, j, k) + f(c, i + 1, j, k)) + (f(c, i, j - 1, k) + f(c, i, j + 1, k)) +
         (f(c, i, j, k - 1) + f(c, i, j, k + 1)) - 6.0 * f(c, i, j, k);
}

// Order in which a work list's flat points cover a region (radial index
// fastest): a CTA's contiguous points then march along the direction its
// stencil reaches, and the rows that its next pass needs are in L1.
//   WALK_J  j, then k
//   WALK_K  k, then j
//   WALK_JK k over strips of kStrip rows of j, strip by strip (both)
enum Walk { WALK_J = 0, WALK_K, WALK_JK };
constexpr int kStrip = 8;

// Point t of region b: regions hold fewer than 2^31 points (o4BatchCreate
// rejects larger boxes), so the index split runs in 32-bit unsigned
// arithmetic.
__device__ __forceinline__ void pointOf(const Box3& b, int walk, unsigned t, int& i, int& j, int& k) {
  const unsigned n0 = (unsigned)b.n(0), n1 = (unsigned)b.n(1), n2 = (unsigned)b.n(2);
  unsigned q = t / n0;
  i = b.lo[0] + (int)(t - q * n0);
  unsigned row, col;
  if (walk == WALK_JK) {
    const unsigned strip = q / (kStrip * n2), first = strip * kStrip;
    const unsigned rows = n1 - first < (unsigned)kStrip ? n1 - first : (unsigned)kStrip;
    q -= first * n2;
    col = q / rows;
    row = first + (q - col * rows);
  } else if (walk == WALK_K) {
    row = q / n2;
    col = q - row * n2;
  } else {
    col = q / n1;
    row = q - col * n1;
  }
  j = b.lo[1] + (int)row;
  k = b.lo[2] + (int)col;
}

// Column u of region b for faces of direction d: its first point, and the
// number of faces.
__device__ __forceinline__ int columnOf(const Box3& b, int d, int march, unsigned u, int p[3]) {
  const bool alongK = marchDim(d) == 2;
  const unsigned n0 = (unsigned)b.n(0), no = (unsigned)b.n(alongK ? 1 : 2);
  const unsigned q = u / n0, seg = q / no;
  p[0] = b.lo[0] + (int)(u - q * n0);
  const int other = b.lo[alongK ? 1 : 2] + (int)(q - seg * no), first = b.lo[alongK ? 2 : 1] + (int)seg * march;
  p[1] = alongK ? other : first;
  p[2] = alongK ? first : other;
  const int left = b.hi[alongK ? 2 : 1] - first + 1;
  return left < march ? left : march;
}

__device__ __forceinline__ void prefetch(const double* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// Thread -> (i, j, k) over the chunk's points of region b of the chunk's box.
template <class F>
__device__ __forceinline__ void forRegion(const Box3& b, int walk, const WorkChunk& w, F f) {
  const unsigned n = (unsigned)b.n(0) * (unsigned)b.n(1) * (unsigned)b.n(2);
  const unsigned end = w.end < (long)n ? (unsigned)w.end : n;
  for (unsigned t = (unsigned)w.begin + threadIdx.x; t < end; t += 128u) {
    int i, j, k;
    pointOf(b, walk, t, i, j, k);
    f(i, j, k);
  }
}

// Roe dissipation unless the device flag switches a Roe context to Rusanov
// (the CME insertion window, exec/main.cpp:406-420).
__device__ __forceinline__ bool roeNow(const O4Geo& G) { return G.roe && !(G.rusanov && *G.rusanov); }

// ---- kernels ------------------------------------------------------------------
// 1. detector primitives of the averages, V(<U>) (:1776).
__global__ void o4PrimAvgKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + 0];
  const O4Args& a = c.a;
  forRegion(c.G, WALK_JK, wc, [&](int i, int j, int k) {
    if (!crossShaped(c.V, 4, i, j, k)) return;  // what the flags below read
    double u[8], w[8];
    const double* U = a.U + roff(a.ur, i, j, k);
#pragma unroll
    for (int q = 0; q < 8; ++q) u[q] = U[q * a.ur.N];
    sphToPrim(u, cellBasis(a.G, a.block0, j, k), a.G.gamma, w);
    double* W = a.WA + roff(c.gr, i, j, k);
#pragma unroll
    for (int q = 0; q < 8; ++q) W[q * c.gr.N] = w[q];
  });
}

// 2. raw Jameson flag on G.grow(-1) (:347-402): per direction the largest of
// three curvatures |q+ - 2 q + q-| / (|q+| + 2 |q| + |q-| + 1e-40) of the
// density, the pressure and the magnetic pressure.  The scales are far from
// the ends of the range of doubles except where a field vanishes; there the
// sum is 1e-40, whose reciprocal is exact enough.
__global__ void __launch_bounds__(128) o4ThetaRawKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + 0];
  const O4Args& a = c.a;
  const long N = c.gr.N;
  const int st[3] = {1, c.gr.n[0], c.gr.n[0] * c.gr.n[1]};
  auto magp = [&](const double* W) -> Rn {
    const double bx = __ldg(W + 5 * N), by = __ldg(W + 6 * N), bz = __ldg(W + 7 * N);
    return 0.5 * dot3(bx, bx, by, by, bz, bz);
  };
  auto eta = [](Rn m, Rn q, Rn p) -> Rn {
    const Rn num = fabs(mad(-2.0, q, p + m).v);
    return num * rcpN(mad(2.0, fabs(q.v), Rn(fabs(p.v)) + fabs(m.v)) + 1.0e-40);
  };
  forRegion(c.GR, WALK_JK, wc, [&](int i, int j, int k) {
    if (!crossShaped(c.V, 3, i, j, k)) return;  // what the dilation reads
    const long o = roff(c.gr, i, j, k);
    const double* W = a.WA + o;
    const Rn r0 = __ldg(W), p0 = __ldg(W + 4 * N), m0 = magp(W);
    Rn sum = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double *lo = W - st[d], *hi = W + st[d];
      const double er = eta(__ldg(lo), r0, __ldg(hi)), ep = eta(__ldg(lo + 4 * N), p0, __ldg(hi + 4 * N)),
                   em = eta(magp(lo), m0, magp(hi));
      const Rn et = dmax(er, dmax(ep, em));
      sum = mad(et, et, sum);
    }
    a.thr[o] = sqrt(sum.v) < a.G.eta_d ? 1.0 : 0.0;
  });
}

// 3. dilated theta (0 outside G.grow(-2)), theta-aware average-to-point and
// point primitives on G (:404-507, 696-741, 212-275).
__global__ void o4PointKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + 0];
  const O4Args& a = c.a;
  forRegion(c.GR, WALK_JK, wc, [&](int i, int j, int k) {
    if (!crossShaped(c.V, 2, i, j, k)) return;  // what the reconstruction reads
    const long N = c.gr.N, o = roff(c.gr, i, j, k);
    const double* R = a.thr;
    double t = 0.0;
    const bool inD = i >= c.GD.lo[0] && i <= c.GD.hi[0] && j >= c.GD.lo[1] && j <= c.GD.hi[1] && k >= c.GD.lo[2] &&
                     k <= c.GD.hi[2];
    if (inD) {
      t = R[o];
      t = dmin(t, R[roff(c.gr, i - 1, j, k)]);
      t = dmin(t, R[roff(c.gr, i + 1, j, k)]);
      t = dmin(t, R[roff(c.gr, i, j - 1, k)]);
      t = dmin(t, R[roff(c.gr, i, j + 1, k)]);
      t = dmin(t, R[roff(c.gr, i, j, k - 1)]);
      t = dmin(t, R[roff(c.gr, i, j, k + 1)]);
    }
    View U{a.U, a.ur};
    double u[8], w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) u[q] = U(q, i, j, k);
    // the neighbours are loaded whatever the flag, with the flags' own loads
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const double point = fma(lapCell(U, q, i, j, k), -1.0 / 24.0, u[q]);
      u[q] = t > 0.5 ? point : u[q];
    }
    sphToPrim(u, cellBasis(a.G, a.block0, j, k), a.G.gamma, w);
    double* W = a.WP + o;
#pragma unroll
    for (int q = 0; q < 8; ++q) W[q * N] = w[q];
    // stored last: a store ahead of the state loads would hold them back
    // until the dilation's loads return
    a.th[o] = t;
  });
}

__device__ __forceinline__ double* faceArr(const Ctx& c, int arr) { return c.a.face[c.d] + arr * c.fr.N; }
// Asynchronous copy of one double to shared memory.
__device__ __forceinline__ void copyAsync(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// Strides of the two directions transverse to d in an array laid out on r,
// lower direction first.
__device__ __forceinline__ int2 transverse(const Reg& r, int d) {
  return make_int2(d == 0 ? r.n[0] : 1, d == 2 ? r.n[0] : r.n[0] * r.n[1]);
}
__device__ __forceinline__ int stride(const Reg& r, int d) { return d == 0 ? 1 : d == 1 ? r.n[0] : r.n[0] * r.n[1]; }

// Component array of place q of the (rho, m_n, m_1, m_2, E, B_n, B_1, B_2)
// order along direction d.
__device__ __forceinline__ int place(int q, int d) {
  const int first = q > 4 ? 5 : 1;
  if (q == 0 || q == 4) return q;
  const int e = d + q - first;
  return first + (e > 2 ? e - 3 : e);
}

// 4a. Reconstruction (WENOZ / WENO3 / PLM) of the eight components on both
// sides of every face of F, and the face's flag; the Riemann kernel clamps.
//
// One thread per face, one launch for the three directions.  The kernel
// holds two components at a time: with the Riemann solver in the same kernel
// it took 128 registers, and 16 warps an SM are too few for the latency of
// the FP64 chains (64 x 32^2 x 6, three directions: 325 us against 163 + 130).
// Pairs of components in a loop: all eight unrolled overflow the instruction
// cache (225 us), one at a time costs the registers' rotation (229 us).
template <int MB>
__global__ void __launch_bounds__(128, MB) o4FaceReconKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const int d = wc.dir;
  const Ctx& c = tab[wc.box * 3 + d];
  const O4Args& a = c.a;
  const long NG = c.gr.N, NF = c.fr.N;
  const int st = stride(c.gr, d);
  const double dx2 = a.G.dx[d] * a.G.dx[d];
  forRegion(c.F, d == 2 ? WALK_K : WALK_J, wc, [&](int i, int j, int k) {
    const long o = roff(c.gr, i, j, k);
    const double* W = a.WP + o;
    double v[6], nx[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) nx[m] = __ldg(W + (m - 3) * st);
    double th[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) th[m] = __ldg(a.th + o + (m - 3) * st);
    const double thF = dmin(th[2], th[3]);
    const bool smooth = dmin(dmin(th[0], th[1]), dmin(thF, dmin(th[4], th[5]))) > 0.5;
    double* out = faceArr(c, F_L) + roff(c.fr, i, j, k);
    out[(F_THF - F_L) * NF] = thF;
    auto states = [&](const double (&x)[6]) {
      double l, r;
      if (smooth) {
        wenozFace(x, l, r);
      } else {
        const double y[4] = {x[1], x[2], x[3], x[4]};
        if (a.G.fallback == 0) weno3Face(y, dx2, l, r);
        else plmFallbackFace(y, l, r);
      }
      out[0] = l;
      out[(F_R - F_L) * NF] = r;
      out += NF;
    };
    // the next component's cells are loaded while one is reconstructed
#pragma unroll 1
    for (int q = 0; q < 8; q += 2) {
      W += NG;
#pragma unroll
      for (int m = 0; m < 6; ++m) v[m] = __ldg(W + (m - 3) * st);
      states(nx);
      if (q < 6) {
        W += NG;
#pragma unroll
        for (int m = 0; m < 6; ++m) nx[m] = __ldg(W + (m - 3) * st);
      }
      states(v);
    }
  });
}

// 4b. Riemann problem of every face of F: Roe repair, point flux sum,
// total-pressure sum, centred normal B, and the point dissipation: factored
// Roe (src/BoxOp_RoeCubedSphere.H:73-98, mappedRoe8WaveDissipation +
// factoredRoe8WaveDissipation, src/MHD_Roe8Wave.H:634-740) on the final
// faces plus one transverse ring, or the Rusanov jump and the face's speed
// bound (src/BoxOp_BertaCubedSphereImplem.H:1665-1720).
//
// The next pass's states are copied to shared memory while this pass is
// solved (cp.async, each thread its own column, no barrier), its frame record
// prefetched.
//
// One 3 x 3 matrix (F A of the frame table) turns both states into the face
// frame, where the energies, fluxes and the Roe solver use them; one matrix
// (|n| adj A F^T / det A^2) takes the dissipation back.
template <bool ROE, int MB>
__global__ void __launch_bounds__(128, MB) o4FaceRiemannKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const int d = wc.dir;
  const Ctx& c = tab[wc.box * 3 + d];
  const O4Args& a = c.a;
  const bool roe = ROE && roeNow(a.G);
  const long NF = c.fr.N;
  const int blk = a.block0;
  // states of this pass and the next, a column per thread
  __shared__ double sh[2][16][128];
  const Box3 F = c.F;
  auto fetch = [&](unsigned t, int slot) {
    int i, j, k;
    pointOf(F, WALK_J, t, i, j, k);
    const double* src = faceArr(c, F_L) + roff(c.fr, i, j, k);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      copyAsync(&sh[slot][q][threadIdx.x], src + place(q, d) * NF);
      copyAsync(&sh[slot][8 + q][threadIdx.x], src + (F_R - F_L + place(q, d)) * NF);
    }
    const double* R = roeRec(a.G, blk, d, j, k);
    prefetch(R);
    prefetch(R + 16);
  };
  const unsigned end = (unsigned)wc.end;
  int slot = 0;
  if ((unsigned)wc.begin + threadIdx.x < end) fetch((unsigned)wc.begin + threadIdx.x, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (unsigned t = (unsigned)wc.begin + threadIdx.x; t < end; t += 128u, slot ^= 1) {
    if (t + 128u < end) fetch(t + 128u, slot ^ 1);
    asm volatile("cp.async.commit_group;\n cp.async.wait_group 1;" ::: "memory");
    int i, j, k;
    pointOf(F, WALK_J, t, i, j, k);
    double* const base = faceArr(c, 0) + roff(c.fr, i, j, k);
    double l[8], r[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) { l[q] = sh[slot][q][threadIdx.x]; r[q] = sh[slot][8 + q][threadIdx.x]; }
    l[0] = dmax(l[0], kRHO00); r[0] = dmax(r[0], kRHO00);
    l[4] = dmax(l[4], 1.0e-12); r[4] = dmax(r[4], 1.0e-12);
    const Rn area = radialPoint(a.G, d, i);
    // only faces whose reconstructed states are unusable read the adjacent
    // cells' average primitives (most faces never do)
    if (roe && !(usablePrimitive(l) && usablePrimitive(r))) {
      const long o = roff(c.gr, i, j, k);
      const int st = stride(c.gr, d);
      double cl[8], cr[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double* W = a.WA + place(q, d) * c.gr.N + o;
        cl[q] = W[-st];
        cr[q] = W[0];
      }
      if (usablePrimitive(cl) && usablePrimitive(cr)) {
#pragma unroll
        for (int q = 0; q < 8; ++q) { l[q] = cl[q]; r[q] = cr[q]; }
        base[F_THF * NF] = 0.0;
      }
    }
    base[F_BP * NF] = 0.5 * (Rn(l[5]) + r[5]);
    const int along = d == 0 ? i : d == 1 ? j : k;
    if (along < c.V.lo[d] || along > c.V.hi[d] + 1) continue;  // a face of the Powell flux only
    const double* R = roeRec(a.G, blk, d, j, k);
    double f[10];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const double2 v = roeLoad2(R + 2 * q);
      f[2 * q] = v.x;
      f[2 * q + 1] = v.y;
    }
    double loc[2][8];
    Rn fs[7], ps = 0.0, energy[2];
    const double enthalpy = a.G.gamma * a.G.invGm1;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const double* w = side == 0 ? l : r;
      double* q = loc[side];
      q[0] = w[0];
      q[4] = w[4];
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        q[1 + e] = dot3(f[3 * e], w[1], f[3 * e + 1], w[2], f[3 * e + 2], w[3]);
        q[5 + e] = dot3(f[3 * e], w[5], f[3 * e + 1], w[6], f[3 * e + 2], w[7]);
      }
      // energies (EnergyW, src/BoxOp_Utilities.H:447-520) and f_primflux
      // (src/BoxOp_EulerCubedSphere.H:195-225)
      const Rn ke = 0.5 * Rn(w[0]) * dot3(q[1], q[1], q[2], q[2], q[3], q[3]);
      const Rn me = kInv8Pi * dot3(q[5], q[5], q[6], q[6], q[7], q[7]);
      const Rn vb = dot3(q[1], q[5], q[2], q[6], q[3], q[7]);
      const Rn mass = Rn(w[0]) * w[1], bn = -kInv4Pi * Rn(w[5]);
      Rn g[7];
      g[0] = mass;
#pragma unroll
      for (int e = 0; e < 3; ++e) g[1 + e] = mad(bn, w[5 + e], mass * w[1 + e]);
      g[4] = mad(bn, vb, (mad(2.0, me, ke) + enthalpy * Rn(w[4])) * w[1]);
#pragma unroll
      for (int e = 1; e < 3; ++e) g[4 + e] = mad(w[1], w[5 + e], -(Rn(w[1 + e]) * w[5]));
#pragma unroll
      for (int q7 = 0; q7 < 7; ++q7) fs[q7] = side == 0 ? g[q7] : fs[q7] + g[q7];
      ps = side == 0 ? me + w[4] : ps + (me + w[4]);
      energy[side] = mad(w[4], a.G.invGm1, ke + me);
    }
#pragma unroll
    for (int q = 0; q < 7; ++q) base[(F_FS + q) * NF] = fs[q];
    base[F_PS * NF] = ps;
    const Box3 PB = regionOf(c, RG_PB);
    if (i < PB.lo[0] || i > PB.hi[0] || j < PB.lo[1] || j > PB.hi[1] || k < PB.lo[2] || k > PB.hi[2]) continue;
    if (roe) {
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        loc[side][0] = fmax(loc[side][0], kRHO00);
        loc[side][4] = fmax(loc[side][4], 0.0);
      }
      double diss[8];
      if (!roe8Body<true>(diss, loc[0], loc[1], a.G.gamma, a.G.entropy, a.G.invGm1))
        rusanovDissipation(diss, loc[0], loc[1], a.G.gamma, a.G.invGm1);
      double g[12];  // g[1 .. 9] the matrix back, g[10] = |n| / det A
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const double2 v = roeLoad2(R + 8 + 2 * q);
        g[2 * q] = v.x;
        g[2 * q + 1] = v.y;
      }
      base[F_QD * NF] = area * (Rn(g[10]) * diss[0]);
      base[(F_QD + 4) * NF] = area * (Rn(g[10]) * diss[4]);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        base[(F_QD + 1 + e) * NF] = area * dot3(g[1 + 3 * e], diss[1], g[2 + 3 * e], diss[2], g[3 + 3 * e], diss[3]);
        base[(F_QD + 5 + e) * NF] = area * dot3(g[1 + 3 * e], diss[5], g[2 + 3 * e], diss[6], g[3 + 3 * e], diss[7]);
      }
    } else {
      base[F_QD * NF] = area * (Rn(r[0]) - l[0]);
      base[(F_QD + 4) * NF] = area * (energy[1] - energy[0]);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        base[(F_QD + 1 + e) * NF] = area * mad(r[0], r[1 + e], -(Rn(l[0]) * l[1 + e]));
        base[(F_QD + 5 + e) * NF] = area * (Rn(r[5 + e]) - l[5 + e]);
      }
      // fast speed of the mean state, from the field along the radial basis
      // vector; the mean normal velocity; |A_d|
      double bm[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) bm[e] = 0.5 * (Rn(loc[0][5 + e]) + loc[1][5 + e]);
      double ar[3];  // the matrix' radial column: place (3 - d) % 3 of the (d, d1, d2) order
#pragma unroll
      for (int e = 0; e < 3; ++e) ar[e] = d == 0 ? f[3 * e] : d == 1 ? f[3 * e + 2] : f[3 * e + 1];
      const Rn bn = dot3(ar[0], bm[0], ar[1], bm[1], ar[2], bm[2]), b2 = dot3(bm[0], bm[0], bm[1], bm[1], bm[2], bm[2]);
      const double rho = dmax(0.5 * (Rn(l[0]) + r[0]), kRHO00);
      const double p = dmax(0.5 * (Rn(l[4]) + r[4]), 0.0);
      const Rn rs = rsqrtN(rho), ce2 = a.G.gamma * Rn(p) * (rs * rs);
      const Rn aa = mad(kInv4Pi * b2, rs * rs, ce2);
      const Rn bb = Rn(fabs(bn.v)) * sqrtN(ce2) * rs * 0.56418958354775628694807945156077;  // 1 / sqrt(pi)
      const Rn af = 0.5 * (Rn(sqrtN(dmax(0.0, aa + bb))) + sqrtN(dmax(0.0, aa - bb)));
      base[F_SPD * NF] = mad(af, sqrt(dot3(f[0], f[0], f[3], f[3], f[6], f[6]).v), fabs(0.5 * (Rn(l[1]) + r[1])));
    }
  }
}

// 5. Theta-aware point-to-average of the flux sum and the total pressure, and
// (7) their products with the radial areas: with the areas s(i) varying
// radially only, X = s <F> + (1/12) D_r s D_r <F> on the final faces plus one
// transverse ring (D_r s = 0 for d = 0, whose transverse directions are
// angular).  The reference maps first and multiplies by the area after;
// the metric factors of the mapping do not vary radially, so the two
// commute, and the mapping then takes flux and dissipation together.
//
// One thread per column of faces.  The radial neighbours' averages are the
// neighbouring threads' (shared memory; the first and last thread of the
// CTA only serve as neighbours).  Bound by the latency of L2: 64^3, three
// directions, 182 us marching against 257 with a thread per face, which read
// every transverse row again for each neighbour (L1 held none of them).
__global__ void __launch_bounds__(128, 6) o4FaceAvgKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  __shared__ double sh[2][8][128];
  const WorkChunk wc = wk[blockIdx.x];
  const int d = wc.dir, tid = threadIdx.x;
  const Ctx& c = tab[wc.box * 3 + d];
  const O4Geo& G = c.a.G;
  const Box3 PB = regionOf(c, RG_PB);
  const long NF = c.fr.N;
  // strides of the marching and of the other transverse direction
  const int st = stride(c.fr, marchDim(d)), so = d == 0 ? stride(c.fr, 1) : 1;
  const long u = wc.begin + tid - 1;
  const bool in = u >= 0 && u < columns(PB, d, wc.march);
  int p[3] = {0, 0, 0};
  const int steps = in ? columnOf(PB, d, wc.march, (unsigned)u, p) : 0;
  const int i = p[0];
  // outputs: the CTA's inner threads, below the chunk's end, radially on final faces
  const bool mine = in && tid >= 1 && tid <= kAvgPoints && u < wc.end && i >= c.V0.lo[0] && i <= c.V0.hi[0];
  double* base = in ? faceArr(c, 0) + roff(c.fr, p[0], p[1], p[2]) : nullptr;
  const Rn s = adjDr(G, d, i), ds = (Rn(adjDr(G, d, i + 1)) - adjDr(G, d, i - 1)) * (1.0 / 48.0);
  // the pressure sum follows the seven flux sums
  double fm[8], f0[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    fm[e] = in ? __ldg(base + (F_FS + e) * NF - st) : 0.0;
    f0[e] = in ? __ldg(base + (F_FS + e) * NF) : 0.0;
  }
#pragma unroll 1
  for (int step = 0; step < wc.march; ++step) {
    Rn fa[8];
    if (step < steps) {
      const bool sm = __ldg(base + F_THF * NF) > 0.5;
      double fp[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) fp[e] = __ldg(base + (F_FS + e) * NF + st);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const double* F = base + (F_FS + e) * NF;
        const Rn pt = f0[e], march = Rn(fm[e]) + fp[e], other = Rn(__ldg(F - so)) + __ldg(F + so);
        const Rn lap = mad(-4.0, pt, other + march);
        fa[e] = sm ? mad(lap, 1.0 / 24.0, pt) : pt;
        fm[e] = f0[e];
        f0[e] = fp[e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) fa[e] = 0.0;
    }
    if (d != 0) {
      double (*row)[128] = sh[step & 1];
#pragma unroll
      for (int e = 0; e < 8; ++e) row[e][tid] = fa[e];
      __syncthreads();
      if (mine && step < steps) {
#pragma unroll
        for (int e = 0; e < 8; ++e) base[(F_X + e) * NF] = mad(Rn(row[e][tid + 1]) - row[e][tid - 1], ds, s * fa[e]);
      }
    } else if (mine && step < steps) {
#pragma unroll
      for (int e = 0; e < 8; ++e) base[(F_X + e) * NF] = s * fa[e];
    }
    base += st;
  }
}

// 6, 8. Final flux of every face: mapped flux with its transverse products,
// pressure force, averaged dissipation.  Flux and dissipation are mapped by
// the same metric averages M = <det A A>, so their difference is mapped
// once: F = (1/2) [M Z + sum_t (1/12) D_t M D_t Y] with Z = X - sigma <Q>,
// D_t Y = D_t X - D_t Q (Roe, sigma = 1; Q the point dissipation) or D_t X
// (Rusanov, sigma the speed bound).  D_t M vanishes radially, so directions
// 1 and 2 have one transverse product and direction 0 two.  The record
// holds the halved M, det and normal and their angular differences / 48.
//
// One thread per column of faces, no barrier.  Bound by the latency of L2:
// 64^3, three directions, 475 us with a thread per face (about 75 taps), 398
// marching, 351 with the next row's prefetch; three component groups in
// separate CTAs, which raised the warps from 12 to 32 an SM, were slower, 2.2
// times the instructions, and so was taking the other direction's taps
// through shared memory, 467 us.  The walk over face slabs staged by TMA that
// this and the averages replace ran at 10-20 % of the warp slots between its
// barriers (833 us).
template <bool D0>
__device__ __forceinline__ void finalColumn(const Ctx& c, const RegArgs& rg, const Box3& V0, int d, int march, unsigned u) {
  const O4Args& a = c.a;
  const bool roe = roeNow(a.G);
  const long NF = c.fr.N;
  int p[3];
  const int steps = columnOf(V0, d, march, u, p), t = marchDim(d);
  const int st = stride(c.fr, t), so = D0 ? stride(c.fr, 1) : 1;
  double* base = faceArr(c, 0) + roff(c.fr, p[0], p[1], p[2]);
  const long row = t == 2 ? a.G.na + 2 * a.G.ext + 1 : 1;  // record step along the march
  const double* M = faceRec(a.G, a.block0, d, p[1], p[2]);
  // seam register and caller's flux
  const Reg r0 = regOf(V0);
  double* const reg = a.seamReg ? a.seamReg : rg.reg;
  const long nrna = (long)a.G.na * a.G.nr;
  // row behind and row of the march: area products X (7) and T3, dissipation Q
  double xm[8], x0[8], qm[8], q0[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const double *X = base + (F_X + e) * NF, *Q = base + (F_QD + e) * NF;
    xm[e] = __ldg(X - st);
    x0[e] = __ldg(X);
    qm[e] = __ldg(Q - st);
    q0[e] = __ldg(Q);
  }
#pragma unroll 1
  for (int step = 0; step < steps; ++step) {
    const bool sm = __ldg(base + F_THF * NF) > 0.5;
    const double sigma = roe ? 1.0 : __ldg(base + F_SPD * NF);
    double xp[8], qp[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      xp[e] = __ldg(base + (F_X + e) * NF + st);
      qp[e] = __ldg(base + (F_QD + e) * NF + st);
    }
    // the next step's rows on their way to L1 (395 -> 351 us; the averages,
    // at twice the warps, got slower with it)
    if (step + 1 < steps) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        prefetch(base + (F_X + e) * NF + 2 * st);
        prefetch(base + (F_QD + e) * NF + 2 * st);
      }
    }
    // Z and the transverse differences of Y of place q: along the march (m)
    // and, for direction 0, along j (o)
    auto load = [&](int q, Rn& z, Rn& ym, Rn& yo) {
      const double* Q = base + (F_QD + q) * NF;
      const Rn pt = q0[q], lo = __ldg(Q - so), hi = __ldg(Q + so);
      const Rn lap = mad(-4.0, pt, (lo + hi) + (Rn(qm[q]) + qp[q]));
      z = -(sigma * (sm ? mad(lap, 1.0 / 24.0, pt) : pt));
      ym = 0.0;
      yo = 0.0;
      if (q != 5) {  // the normal field has no flux
        const int e = fluxSlot(q);
        z = z + x0[e];
        ym = Rn(xp[e]) - xm[e];
        if (D0) yo = Rn(__ldg(base + (F_X + e) * NF + so)) - __ldg(base + (F_X + e) * NF - so);
      }
      if (roe) {
        ym = ym - (Rn(qp[q]) - qm[q]);
        if (D0) yo = yo - (hi - lo);
      }
    };
    // record places: the differences along j come first for direction 0
    constexpr int dm = D0 ? 26 : 13, dj = 13;
    Rn fx[8];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      Rn z, ym, yo;
      load(4 * e, z, ym, yo);
      fx[4 * e] = mad(__ldg(M + 9), z, Rn(__ldg(M + dm + 9)) * ym);
      if (D0) fx[4 * e] = mad(__ldg(M + dj + 9), yo, fx[4 * e]);
    }
#pragma unroll
    for (int b = 1; b < 8; b += 4)
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        Rn z, ym, yo;
        load(b + e, z, ym, yo);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const Rn first = e == 0 ? Rn(__ldg(M + 3 * r)) * z : mad(__ldg(M + 3 * r + e), z, fx[b + r]);
          fx[b + r] = mad(__ldg(M + dm + 3 * r + e), ym, first);
          if (D0) fx[b + r] = mad(__ldg(M + dj + 3 * r + e), yo, fx[b + r]);
        }
      }
    // pressure force
    const Rn pm = Rn(xp[7]) - xm[7];
    const Rn po = D0 ? Rn(__ldg(base + F_T3 * NF + so)) - __ldg(base + F_T3 * NF - so) : Rn(0.0);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      fx[1 + r] = fx[1 + r] + mad(__ldg(M + 10 + r), x0[7], Rn(__ldg(M + dm + 10 + r)) * pm);
      if (D0) fx[1 + r] = mad(__ldg(M + dj + 10 + r), po, fx[1 + r]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      base[(F_FX + q) * NF] = fx[q];
      xm[q] = x0[q];
      x0[q] = xp[q];
      qm[q] = q0[q];
      q0[q] = qp[q];
    }
    if (a.flux[d]) {
      double* out = a.flux[d] + roff(r0, p[0], p[1], p[2]);
#pragma unroll
      for (int q = 0; q < 8; ++q) out[q * r0.N] = fx[q];
    }
    if (!D0 && reg) {
      const int f = d == 1 ? p[1] : p[2];
      if (f == 0 || f == a.G.na) {
        const double w = a.seamReg ? rg.w * (a.seamCfl / *a.seamInvMax) : rg.wDev ? rg.w * (rg.cfl / *rg.wDev) : rg.w;
        double* S = reg + (((long)a.block0 * 2 + (d - 1)) * 2 + (f == 0 ? 0 : 1)) * 8 * nrna +
                    (long)(d == 1 ? p[2] : p[1]) * a.G.nr + p[0];
#pragma unroll
        for (int q = 0; q < 8; ++q) S[q * nrna] = mad(w, fx[q], S[q * nrna]);
      }
    }
    base += st;
    M += row * (D0 ? kO4FaceRec0 : kO4FaceRec12);
    if (t == 2) ++p[2]; else ++p[1];
  }
}

template <int MB>
__global__ void __launch_bounds__(128, MB) o4FaceFinalKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + wc.dir];
  const unsigned u = (unsigned)wc.begin + threadIdx.x;
  if ((long)u >= wc.end) return;
  if (wc.dir == 0) finalColumn<true>(c, rg, c.V0, 0, wc.march, u);
  else finalColumn<false>(c, rg, c.V0, wc.dir, wc.march, u);
}

// 9, 12b. Flux divergence of the three directions and the Powell source
// (DivBPowell2's cell products) into rhs, one pass over the cells.  A launch that
// starts from rhs 0 (rg.fresh) neither clears nor reads it, and in the RK4
// step of a whole level the stage update (rg.rk) follows in registers, so the
// stage rhs is not stored at all.  Bound by HBM and its latency: 64^3 with the
// update 985 MB in 238 us, 4.1 TB/s, 63 % of the measured copy rate.
__global__ void __launch_bounds__(128) o4CellKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + 0];
  const O4Args& a = c.a;
  const long NF = c.fr.N;
  const double dt = rg.rk.stage < 0 ? 0.0 : rg.rk.invDtMax ? rg.rk.cfl / *rg.rk.invDtMax : rg.rk.dtv;
  forRegion(c.V, WALK_JK, wc, [&](int i, int j, int k) {
    double* R = a.rhs + roff(c.vr, i, j, k);
    const long fo = roff(c.fr, i, j, k);
    Rn kv[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) kv[q] = rg.fresh ? 0.0 : R[q * c.vr.N];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const Rn coef = -a.scale / a.G.dx[d];
      const int st = stride(c.fr, d);
      const double* F = a.face[d] + F_FX * NF + fo;
#pragma unroll
      for (int q = 0; q < 8; ++q) kv[q] = mad(coef, Rn(__ldg(F + q * NF + st)) - __ldg(F + q * NF), kv[q]);
    }
    if (a.G.powell) {
      const long o = roff(c.v1r, i, j, k), N = c.v1r.N;
      const double* MJ = a.mj + o;
      const Rn m0 = MJ[0];
      Rn dm[3];
#pragma unroll
      for (int t = 0; t < 3; ++t) dm[t] = (Rn(MJ[stride(c.v1r, t)]) - MJ[-stride(c.v1r, t)]) * (1.0 / 48.0);
#pragma unroll
      for (int q = 1; q < 8; ++q) {
        const double* K = a.ka + (q - 1) * N + o;
        Rn value = m0 * K[0];
#pragma unroll
        for (int t = 0; t < 3; ++t) value = mad(dm[t], Rn(__ldg(K + stride(c.v1r, t))) - __ldg(K - stride(c.v1r, t)), value);
        kv[q] = kv[q] + value;
      }
    }
    if (rg.rk.stage < 0) {
#pragma unroll
      for (int q = 0; q < 8; ++q) R[q * c.vr.N] = kv[q];
    } else {
      const long N = c.vr.N, at = (long)a.block0 * 8 * N + roff(c.vr, i, j, k);
      rkUpdate(rg.rk, dt, at, N, kv);
    }
  });
}

// 10. Powell face flux (DivBPowell1, src/BoxOp_DivBcleaning.H:35-74): <det A>
// times the fourth-order face average of the normal field with its angular
// product (<det A> does not vary radially), or the reconstruction's centred
// field where the face is not smooth.
__global__ void o4PowellFluxKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const int d = wc.dir;
  const Ctx& c = tab[wc.box * 3 + d];
  const O4Args& a = c.a;
  forRegion(regionOf(c, RG_PF), WALK_J, wc, [&](int i, int j, int k) {
    const long NF = c.fr.N;
    double* base = faceArr(c, 0) + roff(c.fr, i, j, k);
    const double* M = faceRec(a.G, a.block0, d, j, k);
    Rn out;
    if (base[F_THF * NF] <= 0.5) {
      out = M[9] * Rn(base[F_BP * NF]);
    } else {
      const double* U = a.U + (5 + d) * a.ur.N + roff(a.ur, i, j, k);
      const int st = stride(a.ur, d);
      auto bface = [&](const double* u) -> Rn {
        return mad(7.0 / 12.0, Rn(u[-st]) + u[0], (-1.0 / 12.0) * (Rn(u[-2 * st]) + u[st]));
      };
      const int2 tr = transverse(a.ur, d);
      const int ta = d == 0 ? tr.x : tr.y;
      out = mad(M[22], bface(U + ta) - bface(U - ta), M[9] * bface(U));
      if (d == 0) out = mad(M[35], bface(U + tr.y) - bface(U - tr.y), out);
    }
    base[F_BF * NF] = 2.0 * out;
  });
}

// 11. -J div B on V1: radial-area products of the Powell face fluxes and
// their divergence, the three directions at once.
__global__ void o4PowellDivKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + 0];
  const O4Args& a = c.a;
  forRegion(c.V1, WALK_JK, wc, [&](int i, int j, int k) {
    const long fo = roff(c.fr, i, j, k);
    const double* B0 = a.face[0] + F_BF * c.fr.N + fo;
    Rn mj = (-1.0 / a.G.dx[0]) * mad(B0[1], adjDr(a.G, 0, i + 1), -(Rn(B0[0]) * adjDr(a.G, 0, i)));
    const Rn s = adjDr(a.G, 1, i), ds = (Rn(adjDr(a.G, 1, i + 1)) - adjDr(a.G, 1, i - 1)) * (1.0 / 48.0);
#pragma unroll
    for (int d = 1; d < 3; ++d) {
      const double* B = a.face[d] + F_BF * c.fr.N + fo;
      const int st = stride(c.fr, d);
      const Rn flux = s * (Rn(B[st]) - B[0]), slope = (Rn(B[st + 1]) - B[1]) - (Rn(B[st - 1]) - B[-1]);
      mj = mad(-1.0 / a.G.dx[d], mad(ds, slope, flux), mj);
    }
    a.mj[roff(c.v1r, i, j, k)] = mj;
  });
}

// 12a. Averages of DivBPowell2's cell coefficients (src/BoxOp_DivBcleaning.H:
// 80-172) on V1: K = (0, B, v . B, v) / (4 pi, 4 pi, 1) of the point
// primitives in the cell basis, <K> = K + lap K / 24, formed from the seven
// cells' primitives (the density coefficient is zero and has no array).
__global__ void o4PowellAvgKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + 0];
  const O4Args& a = c.a;
  forRegion(c.V1, WALK_JK, wc, [&](int i, int j, int k) {
    const long NG = c.gr.N;
    const double* W = a.WP + roff(c.gr, i, j, k);
    Rn sum[7], mid[7];
#pragma unroll
    for (int n = 0; n < 7; ++n) {
      // the cell itself, then its neighbours in i, j, k
      const int t = (n - 1) / 2, sgn = (n & 1) ? 1 : -1;
      const double* w = n == 0 ? W : W + sgn * stride(c.gr, t);
      const double* A = cellBasis(a.G, a.block0, n > 0 && t == 1 ? j + sgn : j, n > 0 && t == 2 ? k + sgn : k);
      Rn K[7], vb = 0.0;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        K[4 + e] = dot3(A[3 * e], w[NG], A[3 * e + 1], w[2 * NG], A[3 * e + 2], w[3 * NG]);
        K[e] = kInv4Pi * dot3(A[3 * e], w[5 * NG], A[3 * e + 1], w[6 * NG], A[3 * e + 2], w[7 * NG]);
        vb = mad(K[4 + e], K[e], vb);
      }
      K[3] = vb;
#pragma unroll
      for (int q = 0; q < 7; ++q) {
        if (n == 0) mid[q] = K[q];
        else sum[q] = n == 1 ? K[q] : sum[q] + K[q];
      }
    }
    double* KA = a.ka + roff(c.v1r, i, j, k);
#pragma unroll
    for (int q = 0; q < 7; ++q) KA[q * c.v1r.N] = mad(mad(-6.0, mid[q], sum[q]), 1.0 / 24.0, mid[q]);
  });
}

// Gravity_Euler (src/BoxOp_Gravity.H:84-164) on the valid boxes: with
// dr = D_r (dr/dxi0) the fourth-order cell products <rho dr>, <rho V_r dr>
// (<ab> = <a><b> + (1/12) sum_d D_d a D_d b; dr varies only radially), then
// rhs(m_d) += -GM faceProduct(<det A A>(d, 0), <rho dr>, 0) and
// rhs(E) += -GM faceProduct(<det A>, <rho V_r dr>, 0), faceProduct over the
// two angular directions.
__global__ void o4GravityKernel(const Ctx* __restrict__ tab, const RegArgs rg, const WorkChunk* __restrict__ wk) {
  const WorkChunk wc = wk[blockIdx.x];
  const Ctx& c = tab[wc.box * 3 + 0];
  const O4Args& a = c.a;
  const double minusGM = -kGrav * kMsun;
  forRegion(c.V, WALK_JK, wc, [&](int i, int j, int k) {
    const View U{a.U, a.ur};
    const int blk = a.block0;
    const double dr0 = radialRow(a.G, i).z;
    const double da = 0.5 * radialRow(a.G, i + 1).z - 0.5 * radialRow(a.G, i - 1).z;
    const int pj[5] = {j, j + 1, j - 1, j, j}, pk[5] = {k, k, k, k + 1, k - 1};
    double rd[5], re[5];
    const double* M = faceRec(a.G, blk, 0, j, k);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const double d0 = 0.5 * U(0, i + 1, pj[q], pk[q]) - 0.5 * U(0, i - 1, pj[q], pk[q]);
      const double d1 = 0.5 * U(1, i + 1, pj[q], pk[q]) - 0.5 * U(1, i - 1, pj[q], pk[q]);
      rd[q] = dr0 * U(0, i, pj[q], pk[q]) + da * d0 * (1.0 / 12.0);
      re[q] = dr0 * U(1, i, pj[q], pk[q]) + da * d1 * (1.0 / 12.0);
    }
    // the record holds half the averages and their angular differences / 48
    auto faceP = [&](int e, const double* v) {
      return 2.0 * (M[e] * v[0] + M[13 + e] * (v[1] - v[2]) + M[26 + e] * (v[3] - v[4]));
    };
    double* R = a.rhs + roff(c.vr, i, j, k);
#pragma unroll
    for (int d = 0; d < 3; ++d) R[(1 + d) * c.vr.N] += faceP(3 * d, rd) * minusGM;
    R[4 * c.vr.N] += faceP(9, re) * minusGM;
  });
}


}  // namespace

size_t o4CarveScratch(O4Args& a, double* sp) {
  Box3 V;
  for (int q = 0; q < 3; ++q) { V.lo[q] = a.vlo[q]; V.hi[q] = a.vhi[q]; }
  const Box3 G = V.grow(a.ghost);
  const size_t NG = (size_t)G.size(), NF = (size_t)faceBox(G).size(), N1 = (size_t)V.grow(1).size(), nb = (size_t)a.nbox;
  size_t off = 0;
  auto take = [&](double*& dst, size_t n) {
    if (sp) dst = sp + off;
    off += (n + 31) / 32 * 32;  // 256-byte boundaries
  };
  take(a.WA, nb * 8 * NG);
  take(a.WP, nb * 8 * NG);
  take(a.th, nb * NG);
  take(a.thr, nb * NG);
  for (int d = 0; d < 3; ++d) take(a.face[d], nb * kO4FaceArrays * NF);
  take(a.mj, nb * N1);
  take(a.ka, nb * 7 * N1);
  return off;
}

size_t o4ScratchDoubles(int nbox, const int vlo[3], const int vhi[3], int ghost) {
  O4Args a{};
  a.nbox = nbox;
  a.ghost = ghost;
  for (int q = 0; q < 3; ++q) { a.vlo[q] = vlo[q]; a.vhi[q] = vhi[q]; }
  return o4CarveScratch(a, nullptr);
}

// A batch: per box and direction the Ctx of a one-box O4Args, in device
// memory (the kernels' argument).
struct O4Batch {
  int nbox = 0;
  Ctx* dev = nullptr;
  bool roe = false, powell = false;
  // work lists: per region, chunks of every box's region (of every direction
  // for the face regions), all in one device array
  WorkChunk* chunks = nullptr;
  long chunkOff[RG_COUNT] = {};
  int chunkCount[RG_COUNT] = {};
  int var[kO4TunedKernels] = {0, 0, 0};  // register-cap variant of the tuned kernels
  // DivBPowell2's coefficients (from the point primitives) and the Powell
  // face fluxes and divergence (from the reconstruction's flags and normal
  // field) run on a side stream, joined before the cell pass.
  cudaStream_t side = nullptr;
  cudaEvent_t pointEv = nullptr, reconEv = nullptr, joinEv = nullptr;
};

// Minimum resident CTAs per SM (the register cap) of each variant of the
// tuned kernels: reconstruction, Riemann problem, final flux.  Variant 0 is
// the default.
constexpr int kO4MinBlocks[kO4TunedKernels][kO4Variants] = {{6, 8, 7}, {4, 3, 5}, {3, 4, 5}};

void o4BatchSetVariants(O4Batch* B, const int v[kO4TunedKernels]) {
  for (int q = 0; q < kO4TunedKernels; ++q) B->var[q] = v[q] >= 0 && v[q] < kO4Variants ? v[q] : 0;
}

int o4VariantMinBlocks(int kernel, int variant) {
  return kernel >= 0 && kernel < kO4TunedKernels && variant >= 0 && variant < kO4Variants ? kO4MinBlocks[kernel][variant]
                                                                                          : 0;
}

O4Batch* o4BatchCreate(const O4Args* boxes, int nbox, cudaError_t* err) {
  *err = cudaSuccess;
  if (nbox <= 0 || nbox > 65535) {
    *err = cudaErrorInvalidValue;
    return nullptr;
  }
  for (int b = 0; b < nbox; ++b)
    if (boxes[b].ur.N >= 0x7fffffffL) {  // roff forms offsets in 32 bits
      *err = cudaErrorInvalidValue;
      return nullptr;
    }
  O4Batch* B = new O4Batch;
  B->nbox = nbox;
  std::vector<Ctx> host((size_t)nbox * 3);
  for (int b = 0; b < nbox; ++b) {
    O4Args one = boxes[b];
    one.nbox = 1;
    for (int d = 0; d < 3; ++d) host[(size_t)b * 3 + d] = makeCtx(one, d);
  }
  B->roe = boxes[0].G.roe;
  B->powell = boxes[0].G.powell;
  std::vector<WorkChunk> work;
  for (int id = 0; id < RG_COUNT; ++id) {
    B->chunkOff[id] = (long)work.size();
    const long pass = passPoints(id);
    const int nd = faceRegion(id) ? 3 : 1;
    long total = 0;
    for (size_t q = 0; q < (size_t)nbox * 3; ++q) {
      if ((int)(q % 3) >= nd) continue;
      const long n = regionOf(host[q], id).size();
      if (n >= 0x7fffffffL) {  // forRegion splits indices in 32 bits
        *err = cudaErrorInvalidValue;
        o4BatchDestroy(B);
        return nullptr;
      }
      total += n;
    }
    if (marches(id)) {
      // columns as long as leaves every SM about 1024 threads, at most 16
      // faces: a column's first row costs two more
      const int march = (int)std::max(1L, std::min(16L, total / (148L * 1024)));
      for (int d = 0; d < nd; ++d)
        for (int b = 0; b < nbox; ++b) {
          const long n = columns(regionOf(host[(size_t)b * 3 + d], id), d, march);
          for (long u = 0; u < n; u += pass) work.push_back(WorkChunk{b, d, march, u, std::min(u + pass, n)});
        }
    } else {
      const long chunk = chunkPoints(total, pass);
      for (int d = 0; d < nd; ++d)
        for (int b = 0; b < nbox; ++b) {
          const long n = regionOf(host[(size_t)b * 3 + d], id).size();
          for (long t = 0; t < n; t += chunk) work.push_back(WorkChunk{b, d, 0, t, std::min(t + chunk, n)});
        }
    }
    const long count = (long)work.size() - B->chunkOff[id];
    if (count > 0x7fffffffL) {
      *err = cudaErrorInvalidValue;
      o4BatchDestroy(B);
      return nullptr;
    }
    B->chunkCount[id] = (int)count;
  }
  *err = cudaMalloc(&B->dev, sizeof(Ctx) * host.size());
  if (*err == cudaSuccess) *err = cudaMemcpy(B->dev, host.data(), sizeof(Ctx) * host.size(), cudaMemcpyHostToDevice);
  if (*err == cudaSuccess && !work.empty()) {
    *err = cudaMalloc(&B->chunks, sizeof(WorkChunk) * work.size());
    if (*err == cudaSuccess)
      *err = cudaMemcpy(B->chunks, work.data(), sizeof(WorkChunk) * work.size(), cudaMemcpyHostToDevice);
  }
  if (*err == cudaSuccess && B->powell) {
    *err = cudaStreamCreateWithFlags(&B->side, cudaStreamNonBlocking);
    for (cudaEvent_t* ev : {&B->pointEv, &B->reconEv, &B->joinEv})
      if (*err == cudaSuccess) *err = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
  }
  if (*err != cudaSuccess) {
    o4BatchDestroy(B);
    return nullptr;
  }
  return B;
}

void o4BatchDestroy(O4Batch* B) {
  if (!B) return;
  if (B->dev) cudaFree(B->dev);
  if (B->chunks) cudaFree(B->chunks);
  for (cudaEvent_t ev : {B->pointEv, B->reconEv, B->joinEv})
    if (ev) cudaEventDestroy(ev);
  if (B->side) cudaStreamDestroy(B->side);
  delete B;
}

void o4SplitArgs(const O4Args& a, std::vector<O4Args>& out) {
  const Ctx c = makeCtx(a, 0);
  out.assign(a.nbox, a);
  for (int b = 0; b < a.nbox; ++b) {
    O4Args& o = out[b];
    o.nbox = 1;
    o.block0 = a.block0 + b;
    o.U = a.U + (long)b * a.uStride;
    o.rhs = a.rhs + (long)b * a.rhsStride;
    for (int d = 0; d < 3; ++d) {
      if (a.flux[d]) o.flux[d] = a.flux[d] + (long)b * 8 * c.V.extrude(d).size();
      o.face[d] = a.face[d] + (long)b * kO4FaceArrays * c.fr.N;
    }
    o.WA = a.WA + (long)b * 8 * c.gr.N;
    o.WP = a.WP + (long)b * 8 * c.gr.N;
    o.th = a.th + (long)b * c.gr.N;
    o.thr = a.thr + (long)b * c.gr.N;
    o.mj = a.mj + (long)b * c.v1r.N;
    o.ka = a.ka + (long)b * 7 * c.v1r.N;
  }
}

cudaError_t launchO4BatchGravity(const O4Batch* B, cudaStream_t s) {
  const RegArgs none;
  if (B->chunkCount[RG_V] == 0) return cudaSuccess;
  o4GravityKernel<<<B->chunkCount[RG_V], 128, 0, s>>>(B->dev, none, B->chunks + B->chunkOff[RG_V]);
  return cudaGetLastError();
}

cudaError_t launchO4Batch(const O4Batch* B, const RegArgs* reg, cudaStream_t s) {
  const RegArgs none;
  const RegArgs rg = reg ? *reg : none;
  cudaError_t e = cudaSuccess;
  using Kernel = void (*)(const Ctx*, const RegArgs, const WorkChunk*);
  auto launch = [&](Kernel kernel, RegionId region, cudaStream_t st) {
    if (e != cudaSuccess || B->chunkCount[region] == 0) return;
    kernel<<<(unsigned)B->chunkCount[region], 128, 0, st>>>(B->dev, rg, B->chunks + B->chunkOff[region]);
    e = cudaGetLastError();
  };
  // the side stream's next kernels run after everything queued on s so far
  auto fork = [&](cudaEvent_t ev) {
    if (e == cudaSuccess) e = cudaEventRecord(ev, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(B->side, ev, 0);
  };
  static constexpr Kernel recon[kO4Variants] = {o4FaceReconKernel<kO4MinBlocks[0][0]>,
                                                o4FaceReconKernel<kO4MinBlocks[0][1]>,
                                                o4FaceReconKernel<kO4MinBlocks[0][2]>};
  static constexpr Kernel riemann[2][kO4Variants] = {
      {o4FaceRiemannKernel<false, kO4MinBlocks[1][0]>, o4FaceRiemannKernel<false, kO4MinBlocks[1][1]>,
       o4FaceRiemannKernel<false, kO4MinBlocks[1][2]>},
      {o4FaceRiemannKernel<true, kO4MinBlocks[1][0]>, o4FaceRiemannKernel<true, kO4MinBlocks[1][1]>,
       o4FaceRiemannKernel<true, kO4MinBlocks[1][2]>}};
  static constexpr Kernel final[kO4Variants] = {o4FaceFinalKernel<kO4MinBlocks[2][0]>,
                                                o4FaceFinalKernel<kO4MinBlocks[2][1]>,
                                                o4FaceFinalKernel<kO4MinBlocks[2][2]>};
  launch(o4PrimAvgKernel, RG_G, s);
  launch(o4ThetaRawKernel, RG_GR, s);
  launch(o4PointKernel, RG_GR, s);
  if (B->powell) {
    fork(B->pointEv);
    launch(o4PowellAvgKernel, RG_V1, B->side);
  }
  launch(recon[B->var[0]], RG_F, s);
  launch(riemann[B->roe ? 1 : 0][B->var[1]], RG_F, s);
  if (B->powell) {
    fork(B->reconEv);
    launch(o4PowellFluxKernel, RG_PF, B->side);
    launch(o4PowellDivKernel, RG_V1, B->side);
    if (e == cudaSuccess) e = cudaEventRecord(B->joinEv, B->side);
  }
  launch(o4FaceAvgKernel, RG_PB, s);
  launch(final[B->var[2]], RG_V0, s);
  if (B->powell && e == cudaSuccess) e = cudaStreamWaitEvent(s, B->joinEv, 0);
  launch(o4CellKernel, RG_V, s);
  return e;
}

}  // namespace hc
