// Plain FP64 / complex<double> assembly.
//
// K1-K3 + K5, the quadrature loop: for each quadrature point the Jacobian,
// its inverse and determinant (gmsh getJacobians, src/term/Assembler.cpp:131-139),
// the coefficient programs at the physical point (EquationEvaluator::initialize,
// src/term/evaluator/EquationEvaluator.h:155-168), the map of the reference
// gradients with J^-T (FieldEvaluator<Form1>, src/term/evaluator/FieldEvaluator.h:67-70)
// and Ke += w det (c L)^T conj(R) (BilinearTerm::evaluate,
// src/term/BilinearTerm.cpp:314-326) with the AFrequency factors
// (src/term/Assembler.cpp:283-295), and b_e += w det conj(phi) f
// (LinearTerm::evaluate, src/term/LinearTerm.cpp:182-191).
//
// GB300's FP64 pipe takes 64 cycles per warp instruction and scheduler,
// whether one lane is active or 32, so what counts is the number of FP64
// warp instructions and how full their lanes are. Hence:
//  - At each point the functions are mapped once, to physical gradients (or
//    curls and values) and, scaled by w det c, to what they are multiplied
//    by; an entry is then a plain dot product. Both functions of a product are
//    physical: through det J^-1 J^-T in reference coordinates the mapping
//    would cost a little less, but on flat elements the large entries of that
//    matrix cancel, and an entry's error grows as the square of the aspect
//    ratio instead of the ratio (1:1,000: 5e-10 instead of 3e-13).
//  - Blocks work on several elements, and every phase spreads its items over
//    all threads: elements (Jacobians), (element, point) pairs (D, the coefficients),
//    (element, point, function) triples (H, the mapped functions), and
//    (element, entry) pairs (the sums).
//    The entries of all elements of a block are numbered through, so that
//    small element matrices fill the lanes too.
//
// The element matrices and vectors then go through the deterministic CSR
// reduction of gather.cu.
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace femg {

constexpr int kQuadThreads = 128;
constexpr int kQuadMaxElems = 64;             // elements per block
constexpr size_t kQuadSmem = 30 * 1024;       // shared memory of a block: seven blocks per SM
// per element: det, J^-1, then J / det (HCurl), or J where the points' geometry
// follows from it (modified elements)
constexpr int kGeomDet = 0, kGeomJi = 1, kGeomJd = 10, kGeomJ = 10;
__host__ __device__ constexpr int quadGeom(int affine, int own, bool hcurl) { return !affine ? 0 : own || hcurl ? 19 : 10; }

// Shape and switches of one launch
struct QuadArgs {
  int NE;          // elements per block
  int QD, QC;      // points per chunk of D, and of H within it
  int nd;          // doubles per point of D: coefficients, then the point's own geometry
  int nEnt;        // entries accumulated per element: the upper triangle, or all n x nc
  int comps;       // mask of the test functions' physical components that contribute
  int flat;        // planar elements as they are: J is a 2 x 2 matrix beside the normal
  int own;         // the geometry differs from point to point (curved or modified elements)
  int ng;          // doubles per element of the geometry
  int tensor;      // kQuadSym, kQuadHcurl: coefficients are symmetric tensors
  int uniform;     // the scalar bilinear coefficients are constant on each element
  int realSource;  // the scalar sources are real
  int needX;       // some coefficient or modificator reads the physical point
};

// Kinds of element matrices. The components of a function: H1, the physical
// gradient and the value (4); HCurl, curl and value (6). Coefficients of a
// point, all times w det: kQuadSym and kQuadHcurl one per term kind, or the six
// entries (00 11 22 01 02 12) of a tensor; kQuadFull M (9), b' (3), v (3), m.
enum { kQuadSym = 0, kQuadHcurl = 1, kQuadFull = 2 };
__host__ __device__ constexpr int quadComps(int kind) { return kind == kQuadHcurl ? 6 : 4; }
__host__ __device__ constexpr int quadCoefs(int kind, bool tensor) {
  return kind == kQuadFull ? 16 : !tensor ? 2 : kind == kQuadHcurl ? 12 : 7;
}

// Offsets (in doubles) of a block's shared memory
struct QuadLayout {
  int X, geom, coef, D, src, be, H, pairs, orient, total;
};
// ng: doubles per element, nd, nh: per point of D and H, n: right-hand side entries
__host__ __device__ inline QuadLayout quadLayout(int NE, int QD, int QC, int nn, int n, int ng, int nd, int nh, bool be, int nPairs) {
  QuadLayout L;
  int o = 0;
  L.be = o;  // double2
  o += be ? 2 * NE * n : 0;
  L.X = o;
  o += NE * nn * 3;
  L.geom = o;
  o += NE * ng;
  L.coef = o;
  o += NE * 6;
  L.D = o;
  o += NE * QD * nd;
  L.src = o;
  o += be ? NE * QD * 8 : 0;
  L.H = o;
  o += NE * QC * nh;
  L.pairs = o;
  o += (nPairs * 2 + 7) / 8;
  L.orient = o;
  o += NE;  // two ints per element
  L.total = o;
  return L;
}

// One copy of the coefficient interpreter per file (it is large), called
// where a coefficient is not constant
__device__ __noinline__ double2 evalExprCall(const DevExpr *ex, int64_t e, const double *x, const double *phi, int nb, int q, int nq) {
  return evalExpr(*ex, e, x, phi, nb, q, nq);
}
__device__ __noinline__ double evalRealCall(const DevExpr *ex, int64_t e, const double *x, const double *phi, int nb, int q, int nq) {
  return evalExprReal(*ex, e, x, phi, nb, q, nq);
}
struct CoefPoint {
  int64_t e;
  const double *x, *phi;
  int nb, q, nq;
};
__device__ __forceinline__ double2 evalAt(const DevExpr &ex, const CoefPoint &c) {
  if (ex.cls == kExprConst) return ex.cval;
  if (ex.real) return make_double2(evalRealCall(&ex, c.e, c.x, c.phi, c.nb, c.q, c.nq), 0.0);
  return evalExprCall(&ex, c.e, c.x, c.phi, c.nb, c.q, c.nq);
}
// a coefficient times its module factor; real ones, which are told apart by
// their bits (a comparison of doubles would take the FP64 pipe), by one product
__device__ __forceinline__ bool zeroBits(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ double2 scaled(double2 factor, double2 v) {
  if (zeroBits(factor.y) && zeroBits(v.y)) return make_double2(factor.x * v.x, 0.0);
  return cmul(factor, v);
}
// A = c0 I + factor c D of tensor term `term` (coefTensor of common.cuh with
// the shared interpreter)
__device__ inline void tensorAt(const DevTerms *terms, int term, const DevExpr *D, int g, const CoefPoint &c, double2 c0, double2 *A) {
  for (int k = 0; k < 6; ++k) A[k] = k < 3 ? c0 : make_double2(0.0, 0.0);
  if (term < 0 || terms->t[term].mod != g) return;
  const double2 fc = cmul(terms->t[term].factor, evalAt(terms->t[term].coef, c));
  for (int k = 0; k < 6; ++k) A[k] = cadd(A[k], cmul(fc, evalAt(D[k], c)));
}
// summed scalar coefficients of group g: c[0] grad-grad (curl-curl), c[1]
// mass; elastic fields: c[0] lambda, c[1] mass, c[2] mu
__device__ inline void scalarCoefs(const DevTerms *terms, int g, const CoefPoint &cp, double2 *c) {
  c[0] = c[1] = c[2] = make_double2(0.0, 0.0);
  for (int t = 0; t < terms->n; ++t) {
    const DevTerm &T = terms->t[t];
    if (T.mod != g) continue;
    if (T.kind == FG_TERM_GRAD_GRAD || T.kind == FG_TERM_ELASTIC) c[0] = cadd(c[0], scaled(T.factor, evalAt(T.coef, cp)));
    else if (T.kind == FG_TERM_MASS) c[1] = cadd(c[1], scaled(T.factor, evalAt(T.coef, cp)));
    if (T.kind == FG_TERM_ELASTIC) c[2] = cadd(c[2], scaled(T.factor, evalAt(T.coef2, cp)));
  }
}

// J / det
__device__ inline void overDet(const double *J, double det, double *Jd) {
  const double id = 1.0 / det;
  for (int k = 0; k < 9; ++k) Jd[k] = J[k] * id;
}

// J, its inverse and determinant from the nodes of a planar 2D element: J is
// [[a b 0], [c d 0], [0 0 s]] with s = +-1 the normal, so no square root, and
// one division
__device__ inline double planarMaps(int nn, bool p1, const double *X, const double *dN, double *J, double *Ji) {
  double a = 0.0, b = 0.0, c = 0.0, d = 0.0;  // dx/du dy/du dx/dv dy/dv
  if (p1) {
    a = X[3] - X[0];
    b = X[4] - X[1];
    c = X[6] - X[0];
    d = X[7] - X[1];
  } else {
    for (int k = 0; k < nn; ++k) {
      a += X[3 * k] * dN[3 * k];
      b += X[3 * k + 1] * dN[3 * k];
      c += X[3 * k] * dN[3 * k + 1];
      d += X[3 * k + 1] * dN[3 * k + 1];
    }
  }
  const double nz = a * d - b * c, s = copysign(1.0, nz), det = fabs(nz), id = 1.0 / det, sid = s * id;
  for (int k = 0; k < 9; ++k) J[k] = Ji[k] = 0.0;
  J[0] = a;
  J[1] = b;
  J[3] = c;
  J[4] = d;
  J[8] = s;
  Ji[0] = d * sid;
  Ji[1] = -c * sid;
  Ji[3] = -b * sid;
  Ji[4] = a * sid;
  Ji[8] = s;
  return det;
}

// Nodes and, for affine elements, the geometry of the block's elements
template <bool HCURL>
__device__ inline void quadElements(const PlanDev &p, const DevTerms *terms, const QuadArgs &a, int64_t e0, int live, double *X,
                                    double *geom, int *orient) {
  // the term list (its first 16 KB: the scalar terms) towards L1 while the
  // nodes come in: small meshes are bound by the latency of such loads
  static_assert(sizeof(DevTerms) >= 128 * kQuadThreads, "one 128-byte line per thread");
  asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char *>(terms) + 128 * threadIdx.x));
  for (int t = threadIdx.x; t < live * p.nn * 3; t += kQuadThreads)
    X[t] = p.xyz[3 * (int64_t)p.enodes[e0 * p.nn + t / 3] + t % 3];
  for (int t = threadIdx.x; t < live; t += kQuadThreads) {
    orient[2 * t] = p.orient ? p.orient[e0 + t] : 0;
    orient[2 * t + 1] = p.orientU ? p.orientU[e0 + t] : 0;
  }
  __syncthreads();
  if (p.affine) {
    for (int t = threadIdx.x; t < live; t += kQuadThreads) {
      double *g = geom + t * a.ng;
      double J[9], det;
      if (p.planar) {
        det = planarMaps(p.nn, p.p1geom != 0, X + t * p.nn * 3, p.geoGrad, J, g + kGeomJi);
      } else {
        det = p.p1geom ? jacobianP1(p.dim, X + t * p.nn * 3, J) : jacobian(p.dim, p.nn, X + t * p.nn * 3, p.geoGrad, J);
        jacobianInverse(J, det, g + kGeomJi);
      }
      g[kGeomDet] = det;
      if (a.own)
        for (int k = 0; k < 9; ++k) g[kGeomJ + k] = J[k];
      else if (HCURL)
        overDet(J, det, g + kGeomJd);
    }
    __syncthreads();
  }
}

// det and the physical point x of one (element, point) for the terms of
// modificator group g. own (null where the element's geometry holds, see
// QuadArgs): the point's J^-1 and J / det
template <bool HCURL>
__device__ inline double quadPoint(const PlanDev &p, const DevTerms *terms, int g, int q, const double *X, const double *geom,
                                   bool needX, double *own, double *x) {
  x[0] = x[1] = x[2] = 0.0;
  if (needX)
    for (int k = 0; k < p.nn; ++k) {
      const double v = p.geoVal[q * p.nn + k];
      x[0] += v * X[3 * k];
      x[1] += v * X[3 * k + 1];
      if (!p.planar || !zeroBits(X[2])) x[2] += v * X[3 * k + 2];
    }
  if (!own) return geom[kGeomDet];
  double J[9], det;
  if (p.affine) {
    for (int k = 0; k < 9; ++k) J[k] = geom[kGeomJ + k];
    det = geom[kGeomDet];
  } else if (p.planar) {
    det = planarMaps(p.nn, false, X, p.geoGrad + (size_t)q * p.nn * 3, J, own);
  } else {
    det = jacobian(p.dim, p.nn, X, p.geoGrad + (size_t)q * p.nn * 3, J);
  }
  const DevJacMod &m = terms->mods[g];
  if (m.kind != FG_JACMOD_NONE && !applyJacMod(m, x, J, det)) atomicOr(p.jmErr, 1);
  if (m.kind != FG_JACMOD_NONE || p.affine || !p.planar) jacobianInverse(J, det, own);
  if (HCURL) overDet(J, det, own + 9);
  return det;
}

// Upper-triangle entry k -> (i << 8 | j), i <= j, row-major
__device__ inline void fillPairs(uint16_t *pairs, int n) {
  const int nEnt = n * (n + 1) / 2;
  for (int k = threadIdx.x; k < nEnt; k += kQuadThreads) {
    int i = 0, rem = k;
    while (rem >= n - i) {
      rem -= n - i;
      ++i;
    }
    pairs[k] = (uint16_t)(i << 8 | (i + rem));
  }
}

// The physical gradient J^-T g (M = J^-1), or curl J g / det (M = J / det).
// flat: planar elements, the components of `comps` alone
__device__ __forceinline__ void mapVector(const double *M, double g0, double g1, double g2, bool flat, int comps, double *o) {
  if (flat) {
    o[0] = o[1] = o[2] = 0.0;
    if (comps & 3) {
      o[0] = M[0] * g0 + M[3] * g1;
      o[1] = M[1] * g0 + M[4] * g1;
    }
    if (comps & 4) o[2] = M[8] * g2;
    return;
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) o[r] = M[r] * g0 + M[3 + r] * g1 + M[6 + r] * g2;
}
// h = c g, c a scalar or the six entries of a symmetric tensor
__device__ __forceinline__ void scaleVector(const double *c, bool tensor, const double *g, double *h) {
  if (tensor) {
    h[0] = c[0] * g[0] + c[3] * g[1] + c[4] * g[2];
    h[1] = c[3] * g[0] + c[1] * g[1] + c[5] * g[2];
    h[2] = c[4] * g[0] + c[5] * g[1] + c[2] * g[2];
  } else {
#pragma unroll
    for (int r = 0; r < 3; ++r) h[r] = c[0] * g[r];
  }
}

// The element matrices and vectors of blocks of NE elements.
//   kQuadSym:   scalar H1, symmetric: G_i . (w det A G_j) + phi_i (w det m phi_j)
//               with the physical gradients G = J^-T grad phi
//   kQuadHcurl: HCurl values P = J^-T v and curls C = J c / det
//               (FieldEvaluator<Form1/Form2>, src/term/evaluator/FieldEvaluator.h:59-105):
//               C_i . (w det A C_j) + P_i . (w det B P_j)
//   kQuadFull:  scalar H1, terms whose element matrix is not symmetric (a
//               general TensorFunction, VectorFunction terms) or a two-field
//               plan (BilinearTerm with _field[0] != _field[1],
//               src/term/BilinearTerm.cpp:304-343; test functions from the
//               test tables, unknown functions from the unknown field's):
//               Ke[i][j] = G_i . w det (M G_j + b' phi_j) + phi_i w det (v . G_j + m phi_j).
// H holds, per point, the unknown functions' rows (what is multiplied, per
// part) and the test functions' rows.
// CPLX: complex D. SPLIT: complex coefficients that are constant on each
// element: the real integrals of the two term kinds are summed apart and
// combined at the end, half the FP64 work of complex D. MASKED: some components
// vanish or have no term (a.comps); otherwise all contribute.
// Bound by the FP64 pipe: 82,944 tetrahedra of order 3 (24 points, real,
// constant on each element) take 3.91 ms, of which the entries' products
// alone are 2.7 ms at one warp instruction per 64 cycles and scheduler; a warp
// per element, with the geometry and coefficients on its first lane, took
// 9.93 ms, and one function of each product left in reference coordinates
// 3.72 ms (13 instructions to map a function instead of 10), at the loss of
// accuracy told at the top. Order 2 with complex coefficients that vary inside
// the elements (55,566 tetrahedra): 1.22 ms, with a warp per element 7.93.
// HCurl of order 1 (34,992 tetrahedra): 1.67 ms, 5.32. Seven blocks per SM in
// 72 registers: the phases of one block fill the barriers of the others, which
// costs spills of 0.5 (real kQuadSym) to 2.4 KB a thread (complex kQuadHcurl,
// MASKED), most around the (element, point) phase. Three blocks in 168
// registers took 4.12, 1.42 and 1.76 ms, five 3.92, 1.42 and 1.72, six 3.90,
// 1.40 and 1.67, eight 3.93, 1.21 and 1.67. A call of kQuadFull on 10,368
// order-3 tetrahedra: 2.37 ms with seven, 2.33 with three, 2.17 with six, 2.32
// with eight; of complex kQuadHcurl 0.584, 0.590, 0.584 and 0.586.
template <int KIND, bool CPLX, bool SPLIT, bool MASKED, int MAXE>
__global__ void __launch_bounds__(kQuadThreads, MAXE > 10 ? 2 : 7)
    k_element_fp64(const PlanDev p, const DevTerms *__restrict__ terms, const QuadArgs a, double *__restrict__ ke, double2 *__restrict__ be) {
  constexpr int R = quadComps(KIND);
  constexpr int NC = CPLX ? 2 : 1;           // parts of the coefficients
  constexpr int NA = (CPLX || SPLIT) ? 2 : 1;  // sums per entry
  extern __shared__ __align__(16) double qsm[];
  const int n = p.nb, nU = p.nbU, tid = threadIdx.x;
  const int S = R * (NC * nU + n);  // doubles of H per point: unknown functions, then test functions
  const QuadLayout L = quadLayout(a.NE, a.QD, a.QC, p.nn, n, a.ng, a.nd, S, be != nullptr, KIND == kQuadFull ? 0 : a.nEnt);
  double *X = qsm + L.X, *geom = qsm + L.geom, *D = qsm + L.D, *src = qsm + L.src, *H = qsm + L.H;
  double2 *bs = reinterpret_cast<double2 *>(qsm + L.be);
  double *coef = qsm + L.coef;
  uint16_t *pairs = reinterpret_cast<uint16_t *>(qsm + L.pairs);
  int *orient = reinterpret_cast<int *>(qsm + L.orient);
  const int64_t e0 = (int64_t)blockIdx.x * a.NE;
  const int live = (int)min((int64_t)a.NE, p.E - e0);
  gridTrigger();
  if (KIND != kQuadFull && ke) fillPairs(pairs, n);
  quadElements<KIND == kQuadHcurl>(p, terms, a, e0, live, X, geom, orient);
  if (be)
    for (int t = tid; t < live * n; t += kQuadThreads) bs[t] = make_double2(0.0, 0.0);

  // this thread's entries: the test and unknown functions' places in H (below
  // 48 KB / 8 each), in one register
  double acc[NA][MAXE];
  uint32_t off[MAXE];
  int mine = 0;
#pragma unroll
  for (int m = 0; m < MAXE; ++m) {
#pragma unroll
    for (int c = 0; c < NA; ++c) acc[c][m] = 0.0;
    off[m] = 0;
    const int k = tid + kQuadThreads * m;
    if (ke && k < live * a.nEnt) {
      const int el = k / a.nEnt, r = k - el * a.nEnt;
      const int i = KIND == kQuadFull ? r / nU : pairs[r] >> 8, j = KIND == kQuadFull ? r % nU : pairs[r] & 255;
      off[m] = (uint32_t)(el * a.QC * S + j) << 16 | (uint32_t)(el * a.QC * S + R * NC * nU + i);
      mine = m + 1;
    }
  }
  const int nCoef = quadCoefs(KIND, a.tensor != 0);
  const bool flat = MASKED && a.flat;
  const int nG = terms->nMod > 1 ? terms->nMod : 1;
  for (int g = 0; g < nG; ++g) {
    if (a.uniform && ke)
      for (int t = tid; t < live; t += kQuadThreads) {
        double2 c[3];
        const CoefPoint cp = {e0 + t, X, nullptr, 0, 0, p.nq};
        scalarCoefs(terms, g, cp, c);
        for (int k = 0; k < 2; ++k) {
          coef[6 * t + 2 * k] = c[k].x;
          coef[6 * t + 2 * k + 1] = c[k].y;
        }
      }
    __syncthreads();
    for (int d0 = 0; d0 < p.nq; d0 += a.QD) {
      const int dn = min(a.QD, p.nq - d0);
      // D (and the source) of every (element, point)
      for (int t = tid; t < live * dn; t += kQuadThreads) {
        const int el = t / dn, qd = t - el * dn, q = d0 + qd;
        double x[3];
        double *d = D + (size_t)(el * a.QD + qd) * a.nd;
        const double wd = p.w[q] * quadPoint<KIND == kQuadHcurl>(p, terms, g, q, X + el * p.nn * 3, geom + el * a.ng, a.needX != 0,
                                                                 a.own ? d + nCoef * NC : nullptr, x);
        CoefPoint cp = {e0 + el, x, nullptr, 0, q, p.nq};
        if (KIND != kQuadHcurl) {  // field-node coefficients read the point's row of the basis table
          cp.phi = p.bval + ((size_t)orient[2 * el] * p.nq + q) * n;
          cp.nb = n;
        }
        double2 c[3];
        if (SPLIT || !ke) {
          c[0] = c[1] = make_double2(1.0, 0.0);
        } else if (a.uniform) {
          c[0] = make_double2(coef[6 * el], coef[6 * el + 1]);
          c[1] = make_double2(coef[6 * el + 2], coef[6 * el + 3]);
        } else {
          scalarCoefs(terms, g, cp, c);
        }
        if (!ke) {
          // the right-hand side alone: no coefficients
        } else if (KIND != kQuadFull) {
          if (a.tensor) {
            double2 A[6], B[6];
            tensorAt(terms, terms->tensorTerm, terms->tensor, g, cp, c[0], A);
            if (KIND == kQuadHcurl) tensorAt(terms, terms->tensorMassTerm, terms->tensorMass, g, cp, c[1], B);
#pragma unroll
            for (int part = 0; part < NC; ++part) {
              double *dp = d + part * nCoef;
              for (int k = 0; k < 6; ++k) {
                dp[k] = wd * (part ? A[k].y : A[k].x);
                if (KIND == kQuadHcurl) dp[6 + k] = wd * (part ? B[k].y : B[k].x);
              }
              if (KIND == kQuadSym) dp[6] = wd * (part ? c[1].y : c[1].x);
            }
          } else {
#pragma unroll
            for (int part = 0; part < NC; ++part) {
              d[2 * part] = wd * (part ? c[0].y : c[0].x);
              d[2 * part + 1] = wd * (part ? c[1].y : c[1].x);
            }
          }
        } else {
          double2 A6[6], M[9], v[3], vb[3];
          tensorAt(terms, terms->tensorTerm, terms->tensor, g, cp, c[0], A6);  // c_gg I (+ the symmetric tensor term)
          const int sym[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
          for (int k = 0; k < 9; ++k) M[k] = A6[sym[k]];
          if (terms->tensorFullTerm >= 0 && terms->t[terms->tensorFullTerm].mod == g) {
            const DevTerm &T = terms->t[terms->tensorFullTerm];
            const double2 fc = cmul(T.factor, evalAt(T.coef, cp));
            for (int k = 0; k < 9; ++k) M[k] = cadd(M[k], cmul(fc, evalAt(terms->tensorFull[k], cp)));
          }
          for (int k = 0; k < 3; ++k) v[k] = vb[k] = make_double2(0.0, 0.0);
          if (terms->advectTerm >= 0 && terms->t[terms->advectTerm].mod == g) {
            const DevTerm &T = terms->t[terms->advectTerm];
            const double2 fc = cmul(T.factor, evalAt(T.coef, cp));
            for (int k = 0; k < 3; ++k) v[k] = cmul(fc, evalAt(terms->advect[k], cp));
          }
          if (terms->vecGradTerm >= 0 && terms->t[terms->vecGradTerm].mod == g) {
            const DevTerm &T = terms->t[terms->vecGradTerm];
            const double2 fc = cmul(T.factor, evalAt(T.coef, cp));
            for (int k = 0; k < 3; ++k) vb[k] = cmul(fc, evalAt(terms->vecGrad[k], cp));
          }
#pragma unroll
          for (int part = 0; part < NC; ++part) {
            double *dp = d + part * nCoef;
            auto re = [&](double2 z) { return part ? z.y : z.x; };
            for (int k = 0; k < 9; ++k) dp[k] = wd * re(M[k]);
            for (int k = 0; k < 3; ++k) {
              dp[9 + k] = wd * re(vb[k]);
              dp[12 + k] = wd * re(v[k]);
            }
            dp[15] = wd * re(c[1]);
          }
        }
        if (be) {
          double2 f = make_double2(0.0, 0.0);
          for (int k = 0; k < terms->n; ++k)
            if (terms->t[k].kind == FG_TERM_SOURCE && terms->t[k].mod == g) f = cadd(f, evalAt(terms->t[k].coef, cp));
          double *s = src + (size_t)(el * a.QD + qd) * 8;
          s[0] = wd * f.x;
          s[1] = wd * f.y;
          if (KIND == kQuadFull) {
            double2 sg[3] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
            if (terms->srcGradTerm >= 0 && terms->t[terms->srcGradTerm].mod == g) {
              const double2 fc = evalAt(terms->t[terms->srcGradTerm].coef, cp);
              for (int k = 0; k < 3; ++k) sg[k] = cmul(fc, evalAt(terms->srcGrad[k], cp));
            }
            for (int r = 0; r < 3; ++r) {
              s[2 + r] = wd * sg[r].x;
              s[5 + r] = wd * sg[r].y;
            }
          }
        }
      }
      __syncthreads();
      // b_e[i] += w det conj(phi_i) f (+ the vector source against gradients)
      if (be)
        for (int t = tid; t < live * n; t += kQuadThreads) {
          const int el = t / n, i = t - el * n;
          double2 b = bs[t];
          for (int qd = 0; qd < dn; ++qd) {
            const size_t row = ((size_t)orient[2 * el] * p.nq + d0 + qd) * n + i;
            const double *s = src + (size_t)(el * a.QD + qd) * 8;
            const double ph = p.bval[row];
            b.x += s[0] * ph;
            if (!a.realSource) b.y += s[1] * ph;
            if (KIND == kQuadFull && terms->srcGradTerm >= 0) {
              const double *gr = p.bgrad + 3 * row;
              const double *Ji = a.own ? D + (size_t)(el * a.QD + qd) * a.nd + nCoef * NC : geom + el * a.ng + kGeomJi;
              double G[3];
              mapVector(Ji, gr[0], gr[1], gr[2], false, 7, G);
              b.x += s[2] * G[0] + s[3] * G[1] + s[4] * G[2];
              b.y += s[5] * G[0] + s[6] * G[1] + s[7] * G[2];
            }
          }
          bs[t] = b;
        }
      if (!ke) __syncthreads();  // the sources are read before the next ones are written
      for (int q0 = d0; ke && q0 < d0 + dn; q0 += a.QC) {
        const int qn = min(a.QC, d0 + dn - q0);
        if (q0 > d0) __syncthreads();  // H has been read
        // H of every (element, point, function): the unknown functions, which
        // are the test functions too but in two-field plans
        const int nF = KIND == kQuadFull && p.coupled ? nU + n : nU;
        for (int t = tid; t < live * qn * nF; t += kQuadThreads) {
          const int ep = t / nF, f = t - ep * nF, el = ep / qn, qc = ep - el * qn, q = q0 + qc;
          const bool testOnly = KIND == kQuadFull && f >= nU;
          const double *d = D + (size_t)(el * a.QD + q - d0) * a.nd;
          const double *Ji = a.own ? d + nCoef * NC : geom + el * a.ng + kGeomJi;
          double *h = H + (size_t)(el * a.QC + qc) * S;
          const size_t row = testOnly ? ((size_t)orient[2 * el] * p.nq + q) * n + f - nU : ((size_t)orient[2 * el + 1] * p.nq + q) * nU + f;
          const double *gr = (testOnly ? p.bgrad : p.bgradU) + 3 * row;
          const double *va = testOnly ? p.bval : p.bvalU;
          double *ht = h + R * NC * nU + (testOnly ? f - nU : f);
          h += f;
          double G[3], v[3];
          if (KIND == kQuadHcurl) {
            const double *Jd = a.own ? Ji + 9 : geom + el * a.ng + kGeomJd;
            if (!MASKED || (a.comps & 7)) mapVector(Jd, gr[0], gr[1], gr[2], flat, a.comps, G);
            if (!MASKED || (a.comps & 56)) mapVector(Ji, va[3 * row], va[3 * row + 1], va[3 * row + 2], flat, a.comps >> 3, v);
          } else {
            if (KIND == kQuadFull || !MASKED || (a.comps & 7)) mapVector(Ji, gr[0], gr[1], gr[2], flat, KIND == kQuadFull ? 7 : a.comps, G);
            v[0] = va[row];
          }
          if (KIND != kQuadFull || testOnly || !p.coupled) {
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (!MASKED || (a.comps >> r & 1)) ht[r * n] = r < 3 ? G[r] : v[r - 3];
          }
          if (testOnly) continue;
#pragma unroll
          for (int part = 0; part < NC; ++part) {
            const double *dp = d + part * nCoef;
            double o[6];
            if (KIND == kQuadFull) {
#pragma unroll
              for (int r = 0; r < 3; ++r) o[r] = dp[3 * r] * G[0] + dp[3 * r + 1] * G[1] + dp[3 * r + 2] * G[2] + dp[9 + r] * v[0];
              o[3] = dp[12] * G[0] + dp[13] * G[1] + dp[14] * G[2] + dp[15] * v[0];
            } else {
              if (!MASKED || (a.comps & 7)) scaleVector(dp, a.tensor != 0, G, o);
              if (KIND == kQuadSym) o[3] = dp[nCoef - 1] * v[0];
              else if (!MASKED || (a.comps & 56)) scaleVector(dp + nCoef / 2, a.tensor != 0, v, o + 3);
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (!MASKED || (a.comps >> r & 1)) h[(part * R + r) * nU] = o[r];
          }
        }
        __syncthreads();
        // Ke[i][j] += t_i . H_j. The next D may be written meanwhile: it is
        // read after the barrier that follows.
        for (int qc = 0; qc < qn; ++qc) {
          const double *Hq = H + (size_t)qc * S;
#pragma unroll
          for (int m = 0; m < MAXE; ++m)
            if (m < mine) {
              const double *ti = Hq + (off[m] & 0xFFFFu), *h = Hq + (off[m] >> 16);
#pragma unroll
              for (int r = 0; r < R; ++r) {
                if (MASKED && !(a.comps >> r & 1)) continue;
                const double t = ti[r * n];
                if (SPLIT) {
                  acc[r < 3 ? 0 : NA - 1][m] = fma(t, h[r * nU], acc[r < 3 ? 0 : NA - 1][m]);
                } else {
                  acc[0][m] = fma(t, h[r * nU], acc[0][m]);
                  if (CPLX) acc[NA - 1][m] = fma(t, h[(R + r) * nU], acc[NA - 1][m]);
                }
              }
            }
        }
      }
    }
  }
  // Ke layout [E][ncomp][n][nc], row = local test index, column = local unknown index
  const int nn2 = n * nU;
#pragma unroll
  for (int m = 0; m < MAXE; ++m)
    if (m < mine) {
      const int k = tid + kQuadThreads * m, el = k / a.nEnt, r = k - el * a.nEnt;
      double re = acc[0][m], im = acc[NA - 1][m];
      if (SPLIT) {
        const double *c = coef + 6 * el;
        const double sg = re, sm = im;
        re = c[0] * sg + c[2] * sm;
        im = c[1] * sg + c[3] * sm;
      }
      double *K = ke + (size_t)(e0 + el) * NA * nn2;
      if (KIND == kQuadFull) {
        K[r] = re;
        if (NA == 2) K[nn2 + r] = im;
      } else {
        const int i = pairs[r] >> 8, j = pairs[r] & 255;
        K[i * n + j] = re;
        K[j * n + i] = re;
        if (NA == 2) {
          K[nn2 + i * n + j] = im;
          K[nn2 + j * n + i] = im;
        }
      }
    }
  if (be)
    for (int t = tid; t < live * n; t += kQuadThreads) be[(size_t)e0 * n + t] = bs[t];
}

// Compound (3-component) field with the isotropic Tensor4 term
// integral(C * grad(dof(u)), grad(tf(u))) and the mass term: the Tensor4
// evaluator of the reference (src/term/evaluator/EquationEvaluator.h:1267-1276,
// CompoundFieldEvaluator<Form1,3> src/term/evaluator/FieldEvaluator.h:171-182)
// with C_ijkl = lambda d_ij d_kl + mu (d_ik d_jl + d_il d_jk) gives, for the
// test DOF (i, a) and the unknown DOF (j, b) (local index = basis * 3 + component),
//   Ke = w det [ lambda dj_b di_a + mu d_ab (gi . gj) + mu dj_a di_b ] + w det c_m d_ab phi_i phi_j
// with g = J^-T grad phi. Items are scalar basis pairs (i <= j) with their
// 3x3 blocks; the element matrix is symmetric. With coefficients constant on
// each element (UNIFORM) only T_ab = sum w det gi_a gj_b and the mass are
// summed, 10 products per pair and point, and
//   Ke_ab = lambda T_ab + mu T_ba + d_ab (mu tr T + c_m mass)
// is formed once; otherwise the lambda- and mu-weighted sums are kept apart
// (19 products, twice for complex coefficients). a.comps: 1 the elastic
// term, 2 the mass term. Bound by the FP64 pipe: order 2, 20,250 tetrahedra,
// Lame coefficients per element: 0.475 ms (with the weighted terms formed for
// every entry, a warp per element, it took 3.15 ms); three blocks per SM in
// place of four took 0.492.
template <bool UNIFORM, bool CPLX, int MAXP>
__global__ void __launch_bounds__(kQuadThreads, UNIFORM ? 4 : 2)
    k_element_elastic_fp64(const PlanDev p, const DevTerms *__restrict__ terms, const QuadArgs a, double *__restrict__ ke,
                           double2 *__restrict__ be) {
  constexpr int NC = (!UNIFORM && CPLX) ? 2 : 1;
  constexpr int ND = 10 + (UNIFORM ? 0 : 3 * NC);  // J^-1, w det; lambda, mu, c_m times w det
  constexpr int NH = UNIFORM ? 7 : 3 + 7 * NC;     // g, then w det g and w det phi, or per part lambda g, mu g, c_m phi
  constexpr int NS = UNIFORM ? 10 : 19 * NC;       // sums per pair
  extern __shared__ __align__(16) double qsm[];
  const int ns = p.nb, n = 3 * ns, tid = threadIdx.x;
  const QuadLayout L = quadLayout(a.NE, a.QD, a.QC, p.nn, 0, a.ng, ND, NH * ns, false, a.nEnt);
  double *X = qsm + L.X, *geom = qsm + L.geom, *D = qsm + L.D, *H = qsm + L.H, *coef = qsm + L.coef;
  uint16_t *pairs = reinterpret_cast<uint16_t *>(qsm + L.pairs);
  int *orient = reinterpret_cast<int *>(qsm + L.orient);
  const int64_t e0 = (int64_t)blockIdx.x * a.NE;
  const int live = (int)min((int64_t)a.NE, p.E - e0);
  gridTrigger();
  fillPairs(pairs, ns);
  quadElements<false>(p, terms, a, e0, live, X, geom, orient);
  double acc[MAXP][NS];
  int offI[MAXP], offJ[MAXP], rowI[MAXP], mine = 0;
#pragma unroll
  for (int m = 0; m < MAXP; ++m) {
#pragma unroll
    for (int c = 0; c < NS; ++c) acc[m][c] = 0.0;
    offI[m] = offJ[m] = rowI[m] = 0;
    const int k = tid + kQuadThreads * m;
    if (k < live * a.nEnt) {
      const int el = k / a.nEnt, pr = pairs[k - el * a.nEnt];
      offI[m] = el * a.QC * NH * ns + (pr >> 8);
      offJ[m] = el * a.QC * NH * ns + (pr & 255);
      rowI[m] = orient[2 * el] * p.nq * ns + (pr >> 8);
      mine = m + 1;
    }
  }
  const bool elastic = a.comps & 1, mass = a.comps & 2;
  const int nG = terms->nMod > 1 ? terms->nMod : 1;
  for (int g = 0; g < nG; ++g) {
    if (UNIFORM) {
      for (int t = tid; t < live; t += kQuadThreads) {
        double2 c[3];
        const CoefPoint cp = {e0 + t, X, nullptr, 0, 0, p.nq};
        scalarCoefs(terms, g, cp, c);
        for (int k = 0; k < 3; ++k) {
          coef[6 * t + 2 * k] = c[k].x;
          coef[6 * t + 2 * k + 1] = c[k].y;
        }
      }
      __syncthreads();
    }
    for (int d0 = 0; d0 < p.nq; d0 += a.QD) {
      const int dn = min(a.QD, p.nq - d0);
      for (int t = tid; t < live * dn; t += kQuadThreads) {
        const int el = t / dn, qd = t - el * dn, q = d0 + qd;
        double x[3];
        double *d = D + (size_t)(el * a.QD + qd) * ND;
        const double wd = p.w[q] * quadPoint<false>(p, terms, g, q, X + el * p.nn * 3, geom + el * a.ng, a.needX != 0,
                                                    a.own ? d : nullptr, x);
        if (!a.own)
          for (int k = 0; k < 9; ++k) d[k] = geom[el * a.ng + kGeomJi + k];
        d[9] = wd;
        if (!UNIFORM) {
          double2 c[3];
          const CoefPoint cp = {e0 + el, x, p.bval + ((size_t)orient[2 * el] * p.nq + q) * ns, ns, q, p.nq};
          scalarCoefs(terms, g, cp, c);
          d[10] = wd * c[0].x;
          d[11] = wd * c[2].x;
          d[12] = wd * c[1].x;
          if (NC == 2) {
            d[ND - 3] = wd * c[0].y;
            d[ND - 2] = wd * c[2].y;
            d[ND - 1] = wd * c[1].y;
          }
        }
      }
      __syncthreads();
      for (int q0 = d0; q0 < d0 + dn; q0 += a.QC) {
        const int qn = min(a.QC, d0 + dn - q0);
        if (q0 > d0) __syncthreads();  // H has been read
        for (int t = tid; t < live * qn * ns; t += kQuadThreads) {
          const int ep = t / ns, j = t - ep * ns, el = ep / qn, qc = ep - el * qn;
          const size_t row = ((size_t)orient[2 * el] * p.nq + q0 + qc) * ns + j;
          const double *d = D + (size_t)(el * a.QD + q0 + qc - d0) * ND;
          double *h = H + (size_t)(el * a.QC + qc) * NH * ns + j;
          const double g0 = p.bgrad[3 * row], g1 = p.bgrad[3 * row + 1], g2 = p.bgrad[3 * row + 2], ph = p.bval[row];
#pragma unroll
          for (int r = 0; r < 3; ++r) {
            if (!elastic) continue;
            const double G = d[r] * g0 + d[3 + r] * g1 + d[6 + r] * g2;
            h[r * ns] = G;
            if (UNIFORM) {
              h[(3 + r) * ns] = d[9] * G;
            } else {
#pragma unroll
              for (int part = 0; part < NC; ++part) {
                h[(3 + 7 * part + r) * ns] = d[10 + 3 * part] * G;
                h[(6 + 7 * part + r) * ns] = d[11 + 3 * part] * G;
              }
            }
          }
          if (UNIFORM) {
            h[6 * ns] = d[9] * ph;
          } else {
#pragma unroll
            for (int part = 0; part < NC; ++part) h[(9 + 7 * part) * ns] = d[12 + 3 * part] * ph;
          }
        }
        __syncthreads();
        for (int qc = 0; qc < qn; ++qc) {
          const double *Hq = H + (size_t)qc * NH * ns;
          const double *bv = p.bval + (size_t)(q0 + qc) * ns;
#pragma unroll
          for (int m = 0; m < MAXP; ++m)
            if (m < mine) {
              const double *hi = Hq + offI[m], *hj = Hq + offJ[m];
              if (elastic) {
                const double gi[3] = {hi[0], hi[ns], hi[2 * ns]};
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                  if (UNIFORM) {
                    const double w = hj[(3 + b) * ns];
#pragma unroll
                    for (int c = 0; c < 3; ++c) acc[m][3 * c + b] = fma(gi[c], w, acc[m][3 * c + b]);
                  } else {
#pragma unroll
                    for (int part = 0; part < NC; ++part) {
                      const double l = hj[(3 + 7 * part + b) * ns], u = hj[(6 + 7 * part + b) * ns];
#pragma unroll
                      for (int c = 0; c < 3; ++c) {
                        double &al = acc[m][(19 * part + 3 * c + b) % NS], &au = acc[m][(19 * part + 9 + 3 * c + b) % NS];
                        al = fma(gi[c], l, al);
                        au = fma(gi[c], u, au);
                      }
                    }
                  }
                }
              }
              if (mass) {
                const double ph = bv[rowI[m]];
                if (UNIFORM) {
                  acc[m][9] = fma(ph, hj[6 * ns], acc[m][9]);
                } else {
#pragma unroll
                  for (int part = 0; part < NC; ++part) {
                    double &am = acc[m][(19 * part + 18) % NS];
                    am = fma(ph, hj[(9 + 7 * part) * ns], am);
                  }
                }
              }
            }
        }
      }
    }
  }
  constexpr int ncomp = CPLX ? 2 : 1;
#pragma unroll
  for (int m = 0; m < MAXP; ++m)
    if (m < mine) {
      const int k = tid + kQuadThreads * m, el = k / a.nEnt, pr = pairs[k - el * a.nEnt], i = pr >> 8, j = pr & 255;
      double *K = ke + (size_t)(e0 + el) * ncomp * n * n;
#pragma unroll
      for (int part = 0; part < ncomp; ++part) {
        double lam = 1.0, mu = 1.0, cm = 1.0;
        if (UNIFORM) {
          lam = coef[6 * el + part];
          cm = coef[6 * el + 2 + part];
          mu = coef[6 * el + 4 + part];
        }
        // the lambda-, mu- and mass-weighted sums
        const double *sl = acc[m] + (UNIFORM ? 0 : (19 * part) % NS), *su = UNIFORM ? sl : sl + 9;
        const double diag = mu * (su[0] + su[4] + su[8]) + cm * (UNIFORM ? sl[9] : sl[(18) % NS]);
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            double v = lam * sl[3 * c + b] + mu * su[3 * b + c];
            if (c == b) v += diag;
            const int ii = 3 * i + c, jj = 3 * j + b;  // test (i, c), unknown (j, b)
            K[(size_t)part * n * n + ii * n + jj] = v;
            K[(size_t)part * n * n + jj * n + ii] = v;
          }
      }
    }
  if (be)
    for (int t = tid; t < live * n; t += kQuadThreads) be[(size_t)e0 * n + t] = make_double2(0.0, 0.0);
}

// Elements per block and points per chunk: the fewest FP64 instructions that
// an SM's fullest warps run one after the other. A block takes, per point,
// one product per table component for every entry of a thread (comps), hCost
// instructions per round of (element, point, function) triples of a chunk,
// dCost per round of (element, point) pairs, about as long as kBarrier
// instructions at each barrier, and about 60 for the elements' geometry; an
// SM runs blocks / SMs of them, of which those that are resident at once hide
// each other's gaps (kBusy: how busy one alone keeps the pipe), the last ones,
// fewer than an SM holds, less well. So small meshes get few elements per
// block, large ones what fills the rounds best. D is formed for QD points at a
// time, H for QC of these. (The search takes 0.1 to 3 us of the host's time.)
// Measured on 54 calls (triangles of order 1 to 5, tetrahedra of order 1 to 4
// and HCurl elements, three sizes each) with every number of elements: the
// rule's choice takes 1.6% longer than the best one on average, 22% at most;
// without the last blocks' part 3.3% and 37%, and without the overlap
// (kBusy 1) 512 triangles of order 6 take 232 us a call instead of 170. kBusy
// from 0.3 to 0.4 and barriers of 2 to 12 instructions make no difference.
static bool quadShape(const PlanDev &p, int nEnt, int n, int nF, int nd, int nh, bool be, int nPairs, int maxItems, int comps,
                      int hCost, int dCost, int blocksPerSm, QuadArgs *a) {
  constexpr int kBarrier = 4;
  constexpr double kBusy = 0.35;
  const int64_t sms = smCount();
  auto bytes = [&](int NE, int QD, int QC) { return (size_t)quadLayout(NE, QD, QC, p.nn, n, a->ng, nd, nh, be, nPairs).total * 8; };
  auto parts = [](int of, int by) { return (of + by - 1) / by; };
  auto rounds = [&](int items) { return parts(items, kQuadThreads); };
  double best = 0.0, idles[8] = {1.0};
  for (int k = 1; k < 8; ++k) idles[k] = idles[k - 1] * (1.0 - kBusy);
  a->NE = 0;
  for (int NE = 1; NE <= kQuadMaxElems && NE * nEnt <= kQuadThreads * maxItems; NE += NE < 24 ? 1 : 4) {
    // shared memory without D and H, and a point of each
    const int rest = (int)bytes(NE, 0, 0), dPoint = (int)bytes(NE, 1, 0) - rest, hPoint = NE * nh * 8;
    const int room = (int)kQuadSmem - rest;
    if (room < dPoint + hPoint) break;
    if (NE > 1 && (NE > 24 ? NE - 4 : NE - 1) * sms >= p.E) break;  // more elements per block would leave SMs without any
    const int64_t blocks = (p.E + NE - 1) / NE, perSm = (blocks + sms - 1) / sms;
    const int64_t tail = perSm % blocksPerSm;
    double each = (double)(perSm - tail) / (1.0 - idles[blocksPerSm]);
    if (tail) each += (double)tail / (1.0 - idles[tail]);
    const double fixed = (double)(rounds(NE * nEnt) * p.nq * comps + 60);
    if (a->NE && each * fixed >= best) continue;  // (without the chunks already as long)
    const int fewest = parts(p.nq, std::min(p.nq, (room - hPoint) / dPoint));
    for (int c = fewest; c <= fewest + 2 && c <= p.nq; ++c) {
      const int QD = parts(p.nq, c), nD = parts(p.nq, QD);
      const int most = std::min(std::min(QD, 16), (room - QD * dPoint) / hPoint);
      for (int h = parts(QD, most), end = std::min(h + 1, QD); h <= end; ++h) {
        const int QC = parts(QD, h), nH = parts(QD, QC);
        const int chunks = nD * (nH * rounds(NE * QC * nF) * hCost + rounds(NE * QD) * dCost + kBarrier * (1 + nH));
        const double cost = each * (fixed + chunks);
        if (a->NE == 0 || cost < best) {
          best = cost;
          a->NE = NE;
          a->QD = QD;
          a->QC = QC;
        }
      }
    }
  }
  if (a->NE == 0) {
    // the widest element matrices: one element and one point at a time
    a->NE = a->QD = a->QC = 1;
    if (nEnt > kQuadThreads * maxItems || bytes(1, 1, 1) > 48 * 1024) return false;
  }
  a->nEnt = nEnt;
  return true;
}

// What the launch's switches need to know of the terms
struct TermUse {
  bool grad = false, mass = false, pointBilinear = false, pointSource = false, realSource = true;
};
static TermUse termUse(const DevTerms &terms) {
  TermUse u;
  auto scan = [](const DevExpr *ex, int count, bool &point) {
    for (int k = 0; k < count; ++k) point = point || ex[k].cls == kExprPoint;
  };
  for (int t = 0; t < terms.n; ++t) {
    const DevTerm &T = terms.t[t];
    switch (T.kind) {
      case FG_TERM_SOURCE:
        scan(&T.coef, 1, u.pointSource);
        u.realSource = u.realSource && T.coef.real;
        continue;
      case FG_TERM_SOURCE_GRAD:
        scan(&T.coef, 1, u.pointSource);
        scan(terms.srcGrad, 3, u.pointSource);
        continue;
      case FG_TERM_MASS:
      case FG_TERM_MASS_TENSOR: u.mass = true; break;
      case FG_TERM_ADVECTION: u.mass = true; break;  // tested by values
      default: u.grad = true;
    }
    scan(&T.coef, 1, u.pointBilinear);
    if (T.kind == FG_TERM_ELASTIC) scan(&T.coef2, 1, u.pointBilinear);
    if (T.kind == FG_TERM_GRAD_GRAD_TENSOR) scan(terms.tensor, 6, u.pointBilinear);
    if (T.kind == FG_TERM_MASS_TENSOR) scan(terms.tensorMass, 6, u.pointBilinear);
    if (T.kind == FG_TERM_GRAD_GRAD_TENSOR_FULL) scan(terms.tensorFull, 9, u.pointBilinear);
    if (T.kind == FG_TERM_ADVECTION) scan(terms.advect, 3, u.pointBilinear);
    if (T.kind == FG_TERM_VECTOR_GRAD_TEST) scan(terms.vecGrad, 3, u.pointBilinear);
  }
  return u;
}

static int quadFail() {
  setLastError("FP64 element kernel: more basis functions or nodes per element than a block's shared memory holds");
  return FG_ERR_UNSUPPORTED;
}

template <int KIND, bool CPLX, bool SPLIT, bool MASKED, int MAXE>
static int quadLaunch(const PlanDev &p, const DevTerms *dterms, QuadArgs a, int nEnt, int coefCost, double *ke, double2 *be, cudaStream_t s) {
  constexpr int NC = CPLX ? 2 : 1;
  const int nPairs = KIND == kQuadFull ? 0 : nEnt, nh = quadComps(KIND) * (NC * p.nbU + p.nb);
  a.nd = quadCoefs(KIND, a.tensor != 0) * NC + (a.own ? (KIND == kQuadHcurl ? 18 : 9) : 0);
  const int map = a.flat ? 5 : 9, scale = a.tensor ? 15 : 3;
  const int nF = p.coupled ? p.nb + p.nbU : p.nbU;  // functions mapped per point
  const int hCost = KIND == kQuadSym ? map + (scale + 1) * NC : KIND == kQuadHcurl ? 2 * (map + scale * NC) : map + 16 * NC * p.nbU / nF;
  if (!quadShape(p, nEnt, p.nb, nF, a.nd, nh, be != nullptr, nPairs, MAXE, quadComps(KIND) * NC, hCost, a.nd + coefCost, MAXE > 10 ? 2 : 7, &a))
    return quadFail();
  const size_t smem = (size_t)quadLayout(a.NE, a.QD, a.QC, p.nn, p.nb, a.ng, a.nd, nh, be != nullptr, nPairs).total * 8;
  k_element_fp64<KIND, CPLX, SPLIT, MASKED, MAXE>
      <<<(unsigned)((p.E + a.NE - 1) / a.NE), kQuadThreads, smem, s>>>(p, dterms, a, ke, be);
  countLaunch();
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}

// The kernel of one kind for these terms. ke null: the right-hand side alone.
template <int KIND, int MAXE>
static int quadKind(const PlanDev &p, const DevTerms &terms, const DevTerms *dterms, int nEnt, double *ke, double2 *be, cudaStream_t s) {
  const TermUse u = termUse(terms);
  QuadArgs a;
  std::memset(&a, 0, sizeof(a));
  const int full = (1 << quadComps(KIND)) - 1;
  a.own = !p.affine || terms.hasJacMod;
  a.ng = quadGeom(p.affine, a.own, KIND == kQuadHcurl);
  a.flat = p.planar && !terms.hasJacMod;
  a.tensor = KIND != kQuadFull && (terms.tensorTerm >= 0 || terms.tensorMassTerm >= 0);
  a.comps = p.tableComps & ((u.grad ? 7 : 0) | (u.mass ? full & ~7 : 0));
  // mapping mixes a vector's components, but for planar elements those of the
  // plane with the normal one
  const int inPlane = a.flat ? 3 : 7;
  for (int v = 0; v < (KIND == kQuadHcurl ? 6 : 3); v += 3)
    if (a.comps >> v & inPlane) a.comps |= inPlane << v;
  a.uniform = !u.pointBilinear;
  a.realSource = u.realSource;
  a.needX = (ke && u.pointBilinear) || (be && u.pointSource) || terms.hasJacMod;
  const bool masked = a.comps != full, cplx = terms.complexKe != 0;
  // about what a point's coefficients take
  const int coefCost = (ke && u.pointBilinear ? 80 : 10) + (be ? (u.realSource ? 40 : 100) : 0);
  // complex sums of real integrals: one group of terms, no tensors
  const bool split = KIND != kQuadFull && cplx && a.uniform && terms.nMod <= 1 && terms.tensorTerm < 0 && terms.tensorMassTerm < 0;
#define FG_QUAD(C, S)                                                                              \
  (masked ? quadLaunch<KIND, C, S, true, MAXE>(p, dterms, a, nEnt, coefCost, ke, be, s)                      \
          : quadLaunch<KIND, C, S, false, MAXE>(p, dterms, a, nEnt, coefCost, ke, be, s))
  if constexpr (KIND != kQuadFull) {
    if (split) return FG_QUAD(false, true);
  }
  return cplx ? FG_QUAD(true, false) : FG_QUAD(false, false);
#undef FG_QUAD
}

template <bool UNIFORM, bool CPLX, int MAXP>
static int quadElastic(const PlanDev &p, const DevTerms *dterms, QuadArgs a, int nEnt, double *ke, double2 *be, cudaStream_t s) {
  constexpr int NC = (!UNIFORM && CPLX) ? 2 : 1, ND = 10 + (UNIFORM ? 0 : 3 * NC), NH = UNIFORM ? 7 : 3 + 7 * NC;
  const int sums = UNIFORM ? 10 : 19 * NC;
  a.nd = ND;
  if (!quadShape(p, nEnt, 0, p.nb, ND, NH * p.nb, false, nEnt, MAXP, sums, 9 + NH, ND + (UNIFORM ? 0 : 80), UNIFORM ? 4 : 2, &a)) return quadFail();
  const size_t smem = (size_t)quadLayout(a.NE, a.QD, a.QC, p.nn, 0, a.ng, ND, NH * p.nb, false, nEnt).total * 8;
  k_element_elastic_fp64<UNIFORM, CPLX, MAXP><<<(unsigned)((p.E + a.NE - 1) / a.NE), kQuadThreads, smem, s>>>(p, dterms, a, ke, be);
  countLaunch();
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}

static int launchElementKernels(fg_plan *plan, const DevTerms &terms, const DevTerms *dterms, double *ke, double *be, cudaStream_t s) {
  const PlanDev &p = plan->d;
  if (p.E == 0) return FG_OK;
  double2 *be2 = (double2 *)be;
  if (terms.nonSym) {
    const int nEnt = p.nb * p.nbU;
    if (nEnt > 39 * 32) {
      setLastError("FP64 full element kernel: more than 35 basis functions per element");
      return FG_ERR_UNSUPPORTED;
    }
    ProfScope prof("k_element_full_fp64", s);
    return quadKind<kQuadFull, 10>(p, terms, dterms, nEnt, ke, be2, s);
  }
  if (factoredFp64Applies(plan, terms)) {
    int st = launchFactoredFp64(plan, terms, dterms, ke, s);
    if (st) return st;
    if (be) {
      if (p.form == FG_FORM_1) {
        setLastError("HCurl fields take no source terms");
        return FG_ERR_UNSUPPORTED;
      }
      return launchRhsFp64(plan, terms, dterms, be, s);
    }
    return FG_OK;
  }
  const int nEnt = p.nb * (p.nb + 1) / 2;
  if (p.form == FG_FORM_1) {
    ProfScope prof("k_element_hcurl_fp64", s);
    // one thread's entries: 10 reach 50 functions, 17 the limit of 64
    if (nEnt <= 10 * kQuadThreads) return quadKind<kQuadHcurl, 10>(p, terms, dterms, nEnt, ke, nullptr, s);
    return quadKind<kQuadHcurl, 17>(p, terms, dterms, nEnt, ke, nullptr, s);
  }
  if (p.mult != 1 || terms.hasElastic) {
    if (p.mult != 3 || terms.hasSource) {
      setLastError("FP64 element kernel: compound fields take the elastic and mass terms only");
      return FG_ERR_UNSUPPORTED;
    }
    if (nEnt > 8 * 32) {
      setLastError("FP64 elastic kernel: more than 21 scalar basis functions per element");
      return FG_ERR_UNSUPPORTED;
    }
    const TermUse u = termUse(terms);
    QuadArgs a;
    std::memset(&a, 0, sizeof(a));
    a.comps = (u.grad ? 1 : 0) | (u.mass ? 2 : 0);
    a.needX = u.pointBilinear || terms.hasJacMod;
    a.own = !p.affine || terms.hasJacMod;
    a.ng = quadGeom(p.affine, a.own, false);
    // the element's sums are scaled once at the end: one group of terms
    a.uniform = !u.pointBilinear && terms.nMod <= 1;
    const bool cplx = terms.complexKe != 0;
    ProfScope prof("k_element_elastic_fp64", s);
    if (a.uniform)
      return cplx ? quadElastic<true, true, 4>(p, dterms, a, nEnt, ke, be2, s) : quadElastic<true, false, 4>(p, dterms, a, nEnt, ke, be2, s);
    return cplx ? quadElastic<false, true, 2>(p, dterms, a, nEnt, ke, be2, s) : quadElastic<false, false, 2>(p, dterms, a, nEnt, ke, be2, s);
  }
  if (nEnt > 20 * 32) {
    setLastError("FP64 element kernel: more than 35 basis functions per element");
    return FG_ERR_UNSUPPORTED;
  }
  ProfScope prof("k_element_fp64", s);
  return quadKind<kQuadSym, 10>(p, terms, dterms, nEnt, ke, be2, s);
}

// FP64 element right-hand sides of the source terms into be ([E][n] complex):
// the quadrature kernel without its element matrices
int launchRhsFp64(fg_plan *plan, const DevTerms &terms, const DevTerms *dterms, double *be, cudaStream_t s) {
  const PlanDev &p = plan->d;
  if (p.E == 0) return FG_OK;
  ProfScope prof("k_rhs_fp64", s);
  return quadKind<kQuadSym, 10>(p, terms, dterms, p.nb, nullptr, (double2 *)be, s);
}

// With Jacobian modificators the kernels flag integration points outside a
// shell; the flag is read back here (the reference throws from apply()).
int launchElementFp64(fg_plan *plan, const DevTerms &terms, const DevTerms *dterms, double *ke, double *be, cudaStream_t s) {
  const PlanDev &p = plan->d;
  if (!terms.hasJacMod || p.E == 0) return launchElementKernels(plan, terms, dterms, ke, be, s);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  FG_CUDA(cudaStreamIsCapturing(s, &cs));
  if (cs != cudaStreamCaptureStatusNone) {
    setLastError("Jacobian modificators: the shell-radius check reads a device word back, which a stream capture cannot");
    return FG_ERR_UNSUPPORTED;
  }
  FG_CUDA(cudaMemsetAsync(p.jmErr, 0, sizeof(int), s));
  int st = launchElementKernels(plan, terms, dterms, ke, be, s);
  if (st) return st;
  FG_CUDA(cudaMemcpyAsync(plan->jmErrHost, p.jmErr, sizeof(int), cudaMemcpyDeviceToHost, s));
  FG_CUDA(cudaStreamSynchronize(s));
  if (*plan->jmErrHost) {
    setLastError("Jacobian modificator: an integration point lies outside the shell [r_min, r_max]");
    return FG_ERR_ARG;
  }
  return FG_OK;
}

int prepareOutputs(fg_plan *plan, double *csr_values, double *rhs, Outputs *o) {
  if (!csr_values) {
    setLastError("csr_values must not be NULL");
    return FG_ERR_ARG;
  }
  o->hostValues = !isDevicePointer(csr_values);
  if (plan->accumulate && (o->hostValues || (rhs && !isDevicePointer(rhs)))) {
    setLastError("accumulating assembly adds into device outputs: csr_values and rhs must be device memory");
    return FG_ERR_ARG;
  }
  o->values = csr_values;
  if (o->hostValues) {
    int st = ensureDevice((void **)&plan->values, &plan->valuesBytes, plan->d.nnz * 16);
    if (st) return st;
    o->values = plan->values;
  }
  o->rhs = rhs;
  if (rhs) {
    o->hostRhs = !isDevicePointer(rhs);
    if (o->hostRhs) {
      int st = ensureDevice((void **)&plan->rhs, &plan->rhsBytes, plan->d.nRows * 16);
      if (st) return st;
      o->rhs = plan->rhs;
    }
  }
  return FG_OK;
}

int finishOutputs(fg_plan *plan, const Outputs &o, double *csr_values, double *rhs, cudaStream_t s) {
  if (o.hostValues && !o.valuesCopied) FG_CUDA(cudaMemcpyAsync(csr_values, o.values, plan->d.nnz * 16, cudaMemcpyDeviceToHost, s));
  if (o.valuesCopied) FG_CUDA(cudaStreamSynchronize(plan->copyStream));
  if (rhs && o.hostRhs) FG_CUDA(cudaMemcpyAsync(rhs, o.rhs, plan->d.nRows * 16, cudaMemcpyDeviceToHost, s));
  if (o.hostValues || (rhs && o.hostRhs)) FG_CUDA(cudaStreamSynchronize(s));
  return FG_OK;
}

}  // namespace femg

using namespace femg;

extern "C" int fg_assemble_fp64(fg_plan *plan, const fg_term_desc *terms, int32_t n_terms, double frequency, const double *dirichlet,
                                double *csr_values, double *rhs, void *stream) {
  if (!plan) return FG_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  DevTerms dt;
  const DevTerms *dterms = nullptr;
  int st = resolveTerms(plan, terms, n_terms, frequency, &dt, &dterms, s);
  if (st) return st;
  if ((st = coupledLiftCheck(plan, rhs))) return st;
  const double *uD = nullptr;
  if ((st = uploadDirichlet(plan, dirichlet, &uD, s))) return st;
  Outputs o;
  if ((st = prepareOutputs(plan, csr_values, rhs, &o))) return st;
  const PlanDev &p = plan->d;
  const int ncomp = dt.complexKe ? 2 : 1;
  if ((st = ensureDevice((void **)&plan->ke, &plan->keBytes, (size_t)p.E * ncomp * p.n * p.nc * sizeof(double)))) return st;
  double *be = nullptr;
  if (dt.hasSource && rhs) {
    if ((st = ensureDevice((void **)&plan->be, &plan->beBytes, (size_t)p.E * p.n * 16))) return st;
    be = plan->be;
  }
  if (p.E > 0) {
    if ((st = launchElementFp64(plan, dt, dterms, plan->ke, be, s))) return st;
  }
  if ((st = gatherToOutputs(plan, plan->ke, dt.complexKe, 0, keRect(p.n, p.nc), be, uD, o, csr_values, s))) return st;
  return finishOutputs(plan, o, csr_values, rhs, s);
}
