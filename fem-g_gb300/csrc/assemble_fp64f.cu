// FP64 element matrices by factorization, on the CUDA cores.
//
// For affine elements with element-constant bilinear coefficients the
// quadrature sum of BilinearTerm::evaluate (src/term/BilinearTerm.cpp:304-343)
// factors exactly into per-element factors and per-orientation reference
// tensors (the same identity the tensor-core path uses):
//   scalar H1:  Ke[i][j] = sum_ab c det K_ab T_ab[i][j] + c_m det M[i][j],  K = J^-1 J^-T,
//   HCurl:      Ke[i][j] = sum_ab (c / det) (J^T J)_ab Tc_ab[i][j] + c_m det K_ab Tv_ab[i][j],
// with T summed over the quadrature points in FP64 once per orientation. All
// arithmetic stays FP64, but GB300's narrow FP64 pipe does 2 kp FLOPs per
// entry (kp = 7 or 12) instead of about 8 nq: 17x fewer for order 3 with
// Gauss6. Selected per plan (FG_FP64_FACTORED); the plain method is the
// quadrature loop. Curved elements, point-dependent coefficients and compound
// fields keep the quadrature kernels.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "common.cuh"

namespace femg {

constexpr int kFacTile = 64;  // elements per tile (one orientation)

struct FactoredState {
  int built = 0;
  int kp = 0;        // factors: 7 (scalar H1) or 12 (HCurl)
  double *T = nullptr;       // [nOrient][kp][n*n] reference tensors
  int32_t *perm = nullptr;   // rank -> element, ranks sorted by orientation
  int4 *tiles = nullptr;     // (orientation, first rank, count, -)
  int nTiles = 0;
};

// Geometry factors of an element in FP64 and its summed coefficients:
//   scalar H1: d[0..5] det J^-1 J^-T (00 11 22 01 02 12), d[6] det,
//   HCurl:     d[0..5] J^T J / det, d[6..11] det J^-1 J^-T;
// c[0] multiplies the first six, c[1] the others. With the cofactors C,
// det J^-1 J^-T = (C^T C) / det: one division, since a lane's FP64
// instructions cost as much as a full warp's.
__device__ inline void elementFactors(const PlanDev &p, const DevTerms *__restrict__ terms, int64_t e, double *d, double2 *c) {
  double X[kMaxNodes * 3];
  const int nx = p.p1geom ? p.dim + 1 : p.nn;
  for (int k = 0; k < nx; ++k)
    for (int r = 0; r < 3; ++r) X[3 * k + r] = p.xyz[3 * (int64_t)p.enodes[e * p.nn + k] + r];
  double J[9];
  const double det = p.p1geom ? jacobianP1(p.dim, X, J) : jacobian(p.dim, p.nn, X, p.geoGrad, J);
  auto Jm = [&](int r, int cc) { return J[3 * cc + r]; };
  double C[9];  // C[3a + r] = (adj J)(a, r)
  C[0] = Jm(1, 1) * Jm(2, 2) - Jm(1, 2) * Jm(2, 1);
  C[1] = Jm(0, 2) * Jm(2, 1) - Jm(0, 1) * Jm(2, 2);
  C[2] = Jm(0, 1) * Jm(1, 2) - Jm(0, 2) * Jm(1, 1);
  C[3] = Jm(1, 2) * Jm(2, 0) - Jm(1, 0) * Jm(2, 2);
  C[4] = Jm(0, 0) * Jm(2, 2) - Jm(0, 2) * Jm(2, 0);
  C[5] = Jm(0, 2) * Jm(1, 0) - Jm(0, 0) * Jm(1, 2);
  C[6] = Jm(1, 0) * Jm(2, 1) - Jm(1, 1) * Jm(2, 0);
  C[7] = Jm(0, 1) * Jm(2, 0) - Jm(0, 0) * Jm(2, 1);
  C[8] = Jm(0, 0) * Jm(1, 1) - Jm(0, 1) * Jm(1, 0);
  const double id = 1.0 / det;
  const int ab[6][2] = {{0, 0}, {1, 1}, {2, 2}, {0, 1}, {0, 2}, {1, 2}};
  for (int k = 0; k < 6; ++k) {
    const int a = ab[k][0], b = ab[k][1];
    const double K = (C[3 * a] * C[3 * b] + C[3 * a + 1] * C[3 * b + 1] + C[3 * a + 2] * C[3 * b + 2]) * id;
    if (p.form == FG_FORM_1) {
      d[k] = (J[3 * a] * J[3 * b] + J[3 * a + 1] * J[3 * b + 1] + J[3 * a + 2] * J[3 * b + 2]) * id;
      d[6 + k] = K;
    } else {
      d[k] = K;
    }
  }
  if (p.form != FG_FORM_1) d[6] = det;
  double xc[3] = {0.0, 0.0, 0.0};
  c[0] = c[1] = make_double2(0.0, 0.0);
  for (int t = 0; t < terms->n; ++t) {
    const DevTerm &T = terms->t[t];
    if (T.kind == FG_TERM_GRAD_GRAD) c[0] = cadd(c[0], cmul(T.factor, evalExpr(T.coef, e, xc)));
    else if (T.kind == FG_TERM_MASS) c[1] = cadd(c[1], cmul(T.factor, evalExpr(T.coef, e, xc)));
  }
}

// One tile of elements of one orientation per block: the elements' factors
// and the upper triangle of the orientation's reference tensors in shared
// memory, then EC elements at a time: their upper-triangle entries, numbered
// through over the threads, into a stage that holds the full matrices, and
// the stage to memory in 16-byte pieces. Real coefficients go into the
// factors (kp products an entry); complex ones multiply the real sums of the
// two term kinds (kp + 4 in place of 2 kp).
// Bound by the FP64 pipe (64 cycles per warp instruction and scheduler):
// 162,000 order-3 tetrahedra, 7 products for 210 entries, are 0.38 ms of it
// and take 0.472 ms (0.791 with all 400 entries formed).
template <bool CPLX>
__global__ void __launch_bounds__(256) k_element_factored_fp64(const PlanDev p, const DevTerms *__restrict__ terms,
                                                               const double *__restrict__ T, const int32_t *__restrict__ perm,
                                                               const int4 *__restrict__ tiles, int kp, int EC, double *__restrict__ ke) {
  constexpr int ncomp = CPLX ? 2 : 1;
  extern __shared__ __align__(16) double fsm[];
  const int n = p.n, nn2 = n * n, np = n * (n + 1) / 2, tid = threadIdx.x;
  const int fLd = kp + 4;                       // factors, then the two complex coefficients
  double *stage = fsm;                          // [EC][ncomp][nn2]
  double *Ts = stage + EC * ncomp * nn2 + (EC * nn2 & 1);  // [kp][np]
  double *F = Ts + kp * np;                     // [kFacTile][fLd]
  uint16_t *pairs = reinterpret_cast<uint16_t *>(F + kFacTile * fLd);  // [np] i << 8 | j
  gridTrigger();
  const int4 tile = tiles[blockIdx.x];
  const double *To = T + (size_t)tile.x * kp * nn2;
  for (int k = tid; k < np; k += 256) {
    int i = 0, rem = k;
    while (rem >= n - i) {
      rem -= n - i;
      ++i;
    }
    pairs[k] = (uint16_t)(i << 8 | (i + rem));
    for (int q = 0; q < kp; ++q) Ts[q * np + k] = To[(size_t)q * nn2 + i * n + i + rem];
  }
  if (tid < tile.z) {
    double *f = F + tid * fLd;
    double2 c[2];
    elementFactors(p, terms, perm[tile.y + tid], f, c);
    if (CPLX) {
      f[kp] = c[0].x;
      f[kp + 1] = c[0].y;
      f[kp + 2] = c[1].x;
      f[kp + 3] = c[1].y;
    } else {
      for (int k = 0; k < kp; ++k) f[k] *= k < 6 ? c[0].x : c[1].x;
    }
  }
  __syncthreads();
  for (int e0 = 0; e0 < tile.z; e0 += EC) {
    const int ne = min(EC, tile.z - e0);
    for (int k = tid; k < ne * np; k += 256) {
      const int el = k / np, r = k - el * np;
      const double *f = F + (e0 + el) * fLd, *t = Ts + r;
      double g = 0.0, m = 0.0;
#pragma unroll
      for (int q = 0; q < 6; ++q) g = fma(f[q], t[q * np], g);
      if (!CPLX) m = g;  // one chain: no sum of two to form
      for (int q = 6; q < kp; ++q) m = fma(f[q], t[q * np], m);
      const int i = pairs[r] >> 8, j = pairs[r] & 255;
      double *K = stage + el * ncomp * nn2;
      if (CPLX) {
        const double re = f[kp] * g + f[kp + 2] * m, im = f[kp + 1] * g + f[kp + 3] * m;
        K[i * n + j] = K[j * n + i] = re;
        K[nn2 + i * n + j] = K[nn2 + j * n + i] = im;
      } else {
        K[i * n + j] = K[j * n + i] = m;
      }
    }
    __syncthreads();
    if ((ncomp * nn2) % 2 == 0) {
      const int half = ncomp * nn2 / 2;
      for (int k = tid; k < ne * half; k += 256) {
        const int el = k / half, r = k - el * half;
        reinterpret_cast<double2 *>(ke + (size_t)perm[tile.y + e0 + el] * ncomp * nn2)[r] = reinterpret_cast<double2 *>(stage)[k];
      }
    } else {
      for (int k = tid; k < ne * nn2; k += 256) {
        const int el = k / nn2, r = k - el * nn2;
        ke[(size_t)perm[tile.y + e0 + el] * nn2 + r] = stage[k];
      }
    }
    __syncthreads();
  }
}

// Shared memory of a block (54 KB measured best on 162,000 order-3
// tetrahedra: 0.472 ms, against 0.528 at 36 KB and 0.495 at 72 and 108), and
// the elements per round: those that fill the
// threads best, among what keeps four blocks on an SM
static size_t factoredSmem(int n, int kp, int ncomp, int EC) {
  const size_t nn2 = (size_t)n * n, np = (size_t)n * (n + 1) / 2;
  return (EC * ncomp * nn2 + 1 + kp * np + (size_t)kFacTile * (kp + 4)) * 8 + (np * 2 + 7) / 8 * 8;
}
constexpr size_t kFacSmem = 54 * 1024;
constexpr size_t kFacSmemMax = 220 * 1024;  // (a block may hold 227 KB)
static int factoredRound(int n, int kp, int ncomp) {
  const int np = n * (n + 1) / 2;
  int best = 1;
  double fill = 0.0;
  for (int EC = 1; EC <= kFacTile && (EC == 1 || factoredSmem(n, kp, ncomp, EC) <= kFacSmem); ++EC) {
    const int rounds = (kFacTile + EC - 1) / EC;  // the last one may be partial
    const int last = kFacTile - (rounds - 1) * EC;
    const int slots = (rounds - 1) * ((EC * np + 255) / 256) + (last * np + 255) / 256;
    const double f = (double)kFacTile * np / (256.0 * slots);
    if (f > fill + 0.005) {
      fill = f;
      best = EC;
    }
  }
  return best;
}

static FactoredState *factoredState(fg_plan *plan) {
  if (!plan->fp64f) plan->fp64f = new FactoredState();
  return (FactoredState *)plan->fp64f;
}

// Reference tensors per orientation (FP64) and the orientation-sorted tiles.
static int prepareFactored(fg_plan *plan) {
  FactoredState *f = factoredState(plan);
  if (f->built) return FG_OK;
  const PlanDev &p = plan->d;
  const int nb = p.nb, nq = p.nq, n2 = nb * nb;
  const bool hc = p.form == FG_FORM_1;
  f->kp = hc ? 12 : 7;
  std::vector<double> w(nq), bval((size_t)p.nOrient * nq * nb * (hc ? 3 : 1)), bgrad((size_t)p.nOrient * nq * nb * 3);
  FG_CUDA(cudaMemcpy(w.data(), p.w, w.size() * 8, cudaMemcpyDeviceToHost));
  FG_CUDA(cudaMemcpy(bval.data(), p.bval, bval.size() * 8, cudaMemcpyDeviceToHost));
  FG_CUDA(cudaMemcpy(bgrad.data(), p.bgrad, bgrad.size() * 8, cudaMemcpyDeviceToHost));
  const int ab[6][2] = {{0, 0}, {1, 1}, {2, 2}, {0, 1}, {0, 2}, {1, 2}};
  std::vector<double> T((size_t)p.nOrient * f->kp * n2, 0.0);
  for (int o = 0; o < p.nOrient; ++o)
    for (int i = 0; i < nb; ++i)
      for (int j = 0; j < nb; ++j) {
        double *t = &T[(size_t)o * f->kp * n2 + (size_t)i * nb + j];
        for (int q = 0; q < nq; ++q) {
          const double *gi = &bgrad[(((size_t)o * nq + q) * nb + i) * 3], *gj = &bgrad[(((size_t)o * nq + q) * nb + j) * 3];
          for (int k = 0; k < 6; ++k) {
            const int a = ab[k][0], b = ab[k][1];
            t[(size_t)k * n2] += w[q] * (gj[a] * gi[b] + (a != b ? gj[b] * gi[a] : 0.0));
          }
          if (hc) {
            const double *vi = &bval[(((size_t)o * nq + q) * nb + i) * 3], *vj = &bval[(((size_t)o * nq + q) * nb + j) * 3];
            for (int k = 0; k < 6; ++k) {
              const int a = ab[k][0], b = ab[k][1];
              t[(size_t)(6 + k) * n2] += w[q] * (vj[a] * vi[b] + (a != b ? vj[b] * vi[a] : 0.0));
            }
          } else {
            t[(size_t)6 * n2] += w[q] * bval[((size_t)o * nq + q) * nb + i] * bval[((size_t)o * nq + q) * nb + j];
          }
        }
      }
  std::vector<int32_t> orient((size_t)p.E, 0);
  if (p.orient && p.E) FG_CUDA(cudaMemcpy(orient.data(), p.orient, (size_t)p.E * 4, cudaMemcpyDeviceToHost));
  std::vector<int32_t> perm((size_t)p.E);
  std::iota(perm.begin(), perm.end(), 0);
  std::stable_sort(perm.begin(), perm.end(), [&](int32_t a, int32_t b) { return orient[a] < orient[b]; });
  std::vector<int4> tiles;
  for (int64_t r = 0; r < p.E;) {
    const int o = orient[perm[r]];
    int64_t e = r;
    while (e < p.E && e - r < kFacTile && orient[perm[e]] == o) ++e;
    tiles.push_back(make_int4(o, (int)r, (int)(e - r), 0));
    r = e;
  }
  FG_CUDA(cudaMalloc(&f->T, std::max<size_t>(T.size(), 1) * 8));
  FG_CUDA(cudaMemcpy(f->T, T.data(), T.size() * 8, cudaMemcpyHostToDevice));
  FG_CUDA(cudaMalloc(&f->perm, std::max<size_t>(perm.size(), 1) * 4));
  if (!perm.empty()) FG_CUDA(cudaMemcpy(f->perm, perm.data(), perm.size() * 4, cudaMemcpyHostToDevice));
  FG_CUDA(cudaMalloc(&f->tiles, std::max<size_t>(tiles.size(), 1) * sizeof(int4)));
  if (!tiles.empty()) FG_CUDA(cudaMemcpy(f->tiles, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice));
  f->nTiles = (int)tiles.size();
  f->built = 1;
  return FG_OK;
}

bool factoredFp64Applies(const fg_plan *plan, const DevTerms &terms) {
  const PlanDev &p = plan->d;
  if (plan->fp64Method != FG_FP64_FACTORED) return false;
  if (!p.affine || p.mult != 1 || terms.hasElastic || terms.hasJacMod || terms.nonSym || terms.tensorTerm >= 0 ||
      terms.tensorMassTerm >= 0)
    return false;
  for (int t = 0; t < terms.n; ++t)
    if (terms.t[t].kind != FG_TERM_SOURCE && terms.t[t].coef.cls == kExprPoint) return false;
  // the upper triangles of an orientation's reference tensors and one element
  // have to fit a block's shared memory: all H1 elements, HCurl ones up to 61
  // functions (real) or 57 (complex)
  return factoredSmem(p.n, p.form == FG_FORM_1 ? 12 : 7, terms.complexKe ? 2 : 1, 1) <= kFacSmemMax;
}

bool factoredFp64Ready(const fg_plan *plan) {
  const FactoredState *f = (const FactoredState *)plan->fp64f;
  return f && f->built;
}

// The tables are built when the method is chosen (fg_plan_set_fp64_method),
// so a launch allocates nothing and issues no blocking copy.
int launchFactoredFp64(fg_plan *plan, const DevTerms &terms, const DevTerms *dterms, double *ke, cudaStream_t s) {
  if (!factoredFp64Ready(plan)) {
    setLastError("FP64 factored kernel: the plan's reference tensors are not built");
    return FG_ERR_ARG;
  }
  FactoredState *f = factoredState(plan);
  const PlanDev &p = plan->d;
  if (f->nTiles == 0) return FG_OK;
  const bool cplx = terms.complexKe != 0;
  const int EC = factoredRound(p.n, f->kp, cplx ? 2 : 1);
  const size_t smem = factoredSmem(p.n, f->kp, cplx ? 2 : 1, EC);  // within the limit by factoredFp64Applies
  auto kern = cplx ? k_element_factored_fp64<true> : k_element_factored_fp64<false>;
  static SmemAllowance allowed[2];
  FG_CUDA(allowSmem(kern, smem, allowed[cplx]));
  ProfScope prof("k_element_factored_fp64", s);
  kern<<<f->nTiles, 256, smem, s>>>(p, dterms, f->T, f->perm, f->tiles, f->kp, EC, ke);
  countLaunch();
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}

}  // namespace femg

extern "C" int fg_plan_set_fp64_method(fg_plan *plan, int32_t method) {
  if (!plan || (method != FG_FP64_QUADRATURE && method != FG_FP64_FACTORED)) {
    femg::setLastError("fg_plan_set_fp64_method: invalid arguments");
    return FG_ERR_ARG;
  }
  // the reference tensors and element tiles are built here, once, so that
  // assemble calls (fg_assemble_fp64_static included) allocate nothing for them
  if (method == FG_FP64_FACTORED && plan->d.E > 0) {
    const int st = femg::prepareFactored(plan);
    if (st) return st;
  }
  plan->fp64Method = method;
  return FG_OK;
}

extern "C" int fg_plan_set_accumulate(fg_plan *plan, int32_t accumulate) {
  if (!plan || (accumulate != 0 && accumulate != 1)) {
    femg::setLastError("fg_plan_set_accumulate: invalid arguments");
    return FG_ERR_ARG;
  }
  plan->accumulate = accumulate;
  return FG_OK;
}

extern "C" void fp64fDestroy(fg_plan *plan) {
  femg::FactoredState *f = (femg::FactoredState *)plan->fp64f;
  if (!f) return;
  cudaFree(f->T);
  cudaFree(f->perm);
  cudaFree(f->tiles);
  delete f;
  plan->fp64f = nullptr;
}
