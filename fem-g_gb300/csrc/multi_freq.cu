// Multi-frequency assembly: the system of the AFrequency module at n_freq
// angular frequencies from one integration of the element matrices.
//
// The reference assembles one frequency per assemble() call: every term with a
// time derivative is scaled by the module factor of the formulation's current
// frequency, -omega^2 for dt2 and -i omega for dt1, before the element matrix
// is summed (src/term/Assembler.cpp:263-305; AFrequencyModule,
// src/system/MatrixModule.cpp:100-171). The terms split into at most three
// groups by time derivative, K (none), C (dt) and M (dt2), whose element
// matrices do not depend on the frequency. They are integrated once (FP64
// element kernels, or the mixed-precision factor rows and one tensor-core
// contraction over all groups), and one row-owner reduction accumulates the
// group sums of each CSR row in shared memory and writes every frequency's
//   values_f = K + (-i omega_f) C + (-omega_f^2) M
// and right-hand side (sources, plus the Dirichlet lifting of each group
// scaled the same way). The reduction visits the element rows in the order
// of the single-frequency gather, so each group sum is deterministic.
#include <algorithm>
#include <cstring>
#include <functional>

#include "multi_gather.cuh"

namespace femg {

static int launchGatherMulti(fg_plan *plan, const MultiIn &in, bool isFloat, cudaStream_t s) {
  const PlanDev &p = plan->d;
  if (p.nRows == 0) return FG_OK;
  MultiLaunch a;
  a.in = in;
  a.p = &p;
  a.s = s;
  // the single-frequency shape of one group; several groups' sums take as
  // many times the shared memory, and complex groups come column by column
  // (VW = 1), which keeps the rare kernels few
  a.g = gatherShape(p, p.maxRowLen, 0, isFloat, in.lay, 8);
  GatherShape &g = a.g;
  if (in.anyCplx) {
    const int nb = g.blocks3 ? p.nc / 3 : p.nc;
    g.VW = 1;
    g.J = g.blocks3 || nb <= 24 ? 3 : 5;
    g.lanes.L = g.blocks3 ? nb : (nb + g.J - 1) / g.J;
    g.lanes.R = 32 / g.lanes.L;
  }
  const size_t size = isFloat ? 4 : 8;
  const size_t cfBytes = (size_t)multiHeadBytes(in.F, in.G, (int)size);
  const size_t rowBytes = (size_t)std::max(p.maxRowLen, 1) * (in.anyCplx ? 2 : 1) * in.G * size;
  // a row of the visiting order has to fit with this many rows per warp
  const int limit = p.n <= 6 ? 16 : p.n <= 12 ? 8 : p.n <= 24 ? 4 : p.n <= 48 ? 2 : 1;
  if ((size_t)multiFactorBytes(in.F, in.G, (int)size) + rowBytes * limit > 200 * 1024) {
    setLastError("multi-frequency gather: CSR row too long for shared memory");
    return FG_ERR_UNSUPPORTED;
  }
  // warps per block: 4; 8 took 0 to 8% longer on 30 sweeps and separate
  // matrices, scalar and of three components, in FP32 and FP64. 4 or 2 rows per
  // warp in place of 6 took 13 and 33% longer (48,000 order-2 tetrahedra of
  // three components, 8 frequencies).
  // Lanes that write a row, by the mean row: on 39,200 order-1 triangles (7
  // entries a row), 3 frequencies in FP32, 8 lanes took 51 us a call, 16 58 and
  // 32 62; on 16,464 order-2 tetrahedra (27), 6 frequencies, 63, 61 and 64; on
  // 6,000 of order 3 (49) 118, 105 and 105, in FP64 446, 448 and 434
  g.wpb = 4;
  const double mean = (double)p.nnz / (double)p.nRows;
  g.lanes.lgOL = mean < 12.0 ? 3 : mean < 40.0 ? 4 : 5;
  g.lanes.OL = 1 << g.lanes.lgOL;
  while (g.lanes.R > 1 && cfBytes + rowBytes * g.lanes.R * g.wpb > 100 * 1024) --g.lanes.R;
  while (g.wpb > 1 && cfBytes + rowBytes * g.lanes.R * g.wpb > 200 * 1024) g.wpb >>= 1;  // (a block may hold 227 KB)
  g.smem = cfBytes + rowBytes * g.lanes.R * g.wpb;
  g.rowsPerBlock = g.wpb * g.lanes.R;
  const int64_t groups = ((int64_t)p.nRows + g.rowsPerBlock - 1) / g.rowsPerBlock;
  a.blocks = std::min<int64_t>(groups, (int64_t)smCount() * kGatherWarpsPerSm / g.wpb);
  ProfScope prof("k_gather_multi", s);
  countLaunch();
  return isFloat ? launchMultiF32(a) : launchMultiF64(a);
}

struct MultiState {
  DevTerms terms[kMaxGroups];
  DevTerms *dev[kMaxGroups] = {nullptr, nullptr, nullptr};
  std::vector<void *> arrays[kMaxGroups];
  double *ke[kMaxGroups] = {nullptr, nullptr, nullptr};
  size_t keBytes[kMaxGroups] = {0, 0, 0};
  double2 *coef = nullptr;                   // [kMaxFreq][kMaxGroups] value factors, then as many lifting factors
  double2 **ptrs = nullptr;                  // device tables: value arrays, then right-hand sides
  double *values = nullptr, *rhs = nullptr;  // staging for host outputs
  size_t valuesBytes = 0, rhsBytes = 0;
};

static MultiState *multiState(fg_plan *plan) {
  if (!plan->multi) plan->multi = new MultiState();
  return (MultiState *)plan->multi;
}

}  // namespace femg

using namespace femg;

extern "C" void multiDestroy(fg_plan *plan) {
  MultiState *m = (MultiState *)plan->multi;
  if (!m) return;
  for (int g = 0; g < kMaxGroups; ++g) {
    for (void *p : m->arrays[g]) cudaFree(p);
    cudaFree(m->dev[g]);
    cudaFree(m->ke[g]);
  }
  cudaFree(m->coef);
  cudaFree(m->ptrs);
  cudaFree(m->values);
  cudaFree(m->rhs);
  delete m;
  plan->multi = nullptr;
}

namespace {

// Splits the terms by time derivative, integrates each group once (unit
// factor) and runs the fused reduction. coefOf(dts, G, coef, rcoef) fills
// the [F][G] value factors and [R][G] lifting factors. values[f] /
// rhs[r]: host or device arrays ([nnz] / [nRows]); rhs may be null.
int runGroups(fg_plan *plan, const fg_term_desc *terms, int32_t n_terms, int32_t mixed, const double *dirichlet, int F,
              double *const *values, int R, double *const *rhs, cudaStream_t s,
              const std::function<int(const int *, int, double2 *, double2 *)> &coefOf) {
  MultiState *m = multiState(plan);
  const PlanDev &p = plan->d;
  if (p.coupled) {
    setLastError("several frequencies / separate matrices: two-field plans are assembled with fg_assemble_fp64");
    return FG_ERR_UNSUPPORTED;
  }
  if (plan->accumulate) {
    setLastError("several frequencies / separate matrices: the plan accumulates; assemble one frequency at a time");
    return FG_ERR_UNSUPPORTED;
  }
  if (p.lscale) {
    setLastError("several frequencies / separate matrices: plans with linked DOFs are assembled one frequency at a time");
    return FG_ERR_UNSUPPORTED;
  }
  // groups by time derivative; the factors are applied in the reduction
  int dts[kMaxGroups], G = 0;
  fg_term_desc grp[kMaxTerms];
  for (int d = FG_DT_NONE; d <= FG_DT_2; ++d) {
    int cnt = 0;
    for (int t = 0; t < n_terms; ++t) {
      if (terms[t].dt < FG_DT_NONE || terms[t].dt > FG_DT_2) {
        setLastError("unknown time derivative");
        return FG_ERR_ARG;
      }
      if (terms[t].kind == FG_TERM_SOURCE && terms[t].dt != FG_DT_NONE) {
        setLastError("a linear term cannot carry a time derivative");
        return FG_ERR_ARG;
      }
      if (terms[t].dt == d) {
        grp[cnt] = terms[t];
        grp[cnt].dt = FG_DT_NONE;
        ++cnt;
      }
    }
    if (!cnt) continue;
    int st = uploadTerms(plan, grp, cnt, 0.0, &m->terms[G], m->arrays[G]);
    if (st) return st;
    if (!m->dev[G]) FG_CUDA(cudaMalloc(&m->dev[G], sizeof(DevTerms)));
    FG_CUDA(cudaMemcpyAsync(m->dev[G], &m->terms[G], sizeof(DevTerms), cudaMemcpyHostToDevice, s));
    dts[G++] = d;
  }
  std::vector<double2> coef((size_t)2 * kMaxFreq * kMaxGroups, make_double2(0.0, 0.0));
  int st = coefOf(dts, G, coef.data(), coef.data() + (size_t)kMaxFreq * kMaxGroups);
  if (st) return st;
  if (!m->coef) FG_CUDA(cudaMalloc(&m->coef, coef.size() * sizeof(double2)));
  FG_CUDA(cudaMemcpyAsync(m->coef, coef.data(), coef.size() * sizeof(double2), cudaMemcpyHostToDevice, s));
  const double *uD = nullptr;
  if ((st = uploadDirichlet(plan, dirichlet, &uD, s))) return st;
  // outputs: device arrays in place, host arrays through staging buffers
  std::vector<double2 *> dv(F), dr(R, nullptr);
  std::vector<char> hv(F, 0), hr(R, 0);
  size_t stageV = 0, stageR = 0;
  for (int f = 0; f < F; ++f) {
    hv[f] = !isDevicePointer(values[f]);
    stageV += hv[f];
  }
  for (int r = 0; r < R; ++r) {
    hr[r] = rhs[r] && !isDevicePointer(rhs[r]);
    stageR += hr[r];
  }
  if (stageV && (st = ensureDevice((void **)&m->values, &m->valuesBytes, stageV * p.nnz * 16))) return st;
  if (stageR && (st = ensureDevice((void **)&m->rhs, &m->rhsBytes, stageR * p.nRows * 16))) return st;
  for (int f = 0, k = 0; f < F; ++f) dv[f] = hv[f] ? (double2 *)(m->values + 2 * p.nnz * k++) : (double2 *)values[f];
  for (int r = 0, k = 0; r < R; ++r) dr[r] = hr[r] ? (double2 *)(m->rhs + 2 * p.nRows * k++) : (double2 *)rhs[r];
  const bool anyRhs = R > 0 && rhs[0];
  if (!m->ptrs) FG_CUDA(cudaMalloc(&m->ptrs, 2 * kMaxFreq * sizeof(double2 *)));
  std::vector<double2 *> table(2 * kMaxFreq, nullptr);
  std::copy(dv.begin(), dv.end(), table.begin());
  std::copy(dr.begin(), dr.end(), table.begin() + kMaxFreq);
  FG_CUDA(cudaMemcpyAsync(m->ptrs, table.data(), table.size() * sizeof(double2 *), cudaMemcpyHostToDevice, s));
  // source terms are linear terms without time derivative: group of dt 0
  const int g0 = dts[0] == FG_DT_NONE ? 0 : -1;
  double *be = nullptr;
  const bool source = g0 == 0 && m->terms[0].hasSource && anyRhs;
  if (source) {
    if ((st = ensureDevice((void **)&plan->be, &plan->beBytes, (size_t)p.E * p.n * 16))) return st;
    be = plan->be;
  }
  MultiIn in;
  std::memset(&in, 0, sizeof(in));
  in.G = G;
  in.F = F;
  for (int g = 0; g < G; ++g) {
    bool re = true, im = true;
    for (int f = 0; f < F; ++f) {
      re = re && coef[(size_t)f * G + g].y == 0.0;
      im = im && coef[(size_t)f * G + g].x == 0.0;
    }
    in.realFactor[g] = re;
    in.imagFactor[g] = im && !re;
  }
  in.allReal = 1;
  for (int g = 0; g < G; ++g) in.allReal = in.allReal && in.realFactor[g];
  in.R = anyRhs ? R : 0;
  in.coef = m->coef;
  in.rcoef = m->coef + (size_t)kMaxFreq * kMaxGroups;
  in.be = (const double2 *)be;
  in.uD = (const double2 *)uD;
  in.values = m->ptrs;
  in.rhs = anyRhs ? m->ptrs + kMaxFreq : nullptr;
  const size_t nn = (size_t)p.n * p.n;
  bool isFloat = false;
  if (!mixed) {
    in.lay = keFull(p.n);
    for (int g = 0; g < G; ++g) {
      const int ncomp = m->terms[g].complexKe ? 2 : 1;
      if ((st = ensureDevice((void **)&m->ke[g], &m->keBytes[g], (size_t)p.E * ncomp * nn * sizeof(double)))) return st;
      if (p.E > 0)
        if ((st = launchElementFp64(plan, m->terms[g], m->dev[g], m->ke[g], g == g0 && source ? be : nullptr, s))) return st;
      in.ke[g] = m->ke[g];
      in.stride[g] = (int64_t)(ncomp * nn);
      in.cplx[g] = ncomp == 2;
    }
  } else {
    int ncomp = 1;
    for (int g = 0; g < G; ++g) {
      if (m->terms[g].complexKe) ncomp = 2;
      for (int t = 0; t < m->terms[g].n; ++t)
        if ((m->terms[g].t[t].kind != FG_TERM_SOURCE && m->terms[g].t[t].coef.cls == kExprPoint) || m->terms[g].hasJacMod ||
            m->terms[g].tensorPoint || m->terms[g].nonSym) {
          setLastError("mixed path: bilinear coefficients must be constant per element, without Jacobian modificators");
          return FG_ERR_UNSUPPORTED;
        }
    }
    if ((st = prepareMixed(plan, ncomp, G))) return st;
    if ((st = mixedCheckTimeout(plan, false))) return st;
    if (source)
      if ((st = launchRhsFp64(plan, m->terms[0], m->dev[0], be, s))) return st;
    if (p.E > 0) {
      const DevTerms *devs[kMaxGroups] = {m->dev[0], m->dev[1], m->dev[2]};
      uint32_t tensorMask = 0;
      for (int g = 0; g < G; ++g)
        if (m->terms[g].tensorTerm >= 0) tensorMask |= 1u << g;
      if ((st = launchMixedElement(plan, devs, G, tensorMask, s))) return st;
    }
    const float *ke = mixedKe(plan, &in.lay);
    const size_t ld = (size_t)in.lay.ld;
    for (int g = 0; g < G; ++g) {
      in.ke[g] = ke + (size_t)g * ncomp * ld;
      in.stride[g] = (int64_t)((size_t)G * ncomp * ld);
      in.cplx[g] = ncomp == 2 && m->terms[g].complexKe;
    }
    isFloat = true;
  }
  in.anyCplx = 0;
  for (int g = 0; g < G; ++g) in.anyCplx |= in.cplx[g] ? 1 : 0;
  if ((st = launchGatherMulti(plan, in, isFloat, s))) return st;
  if (mixed)
    if ((st = mixedRecordError(plan, s))) return st;
  bool anyHost = false;
  for (int f = 0; f < F; ++f)
    if (hv[f]) {
      FG_CUDA(cudaMemcpyAsync(values[f], dv[f], p.nnz * 16, cudaMemcpyDeviceToHost, s));
      anyHost = true;
    }
  for (int r = 0; r < R; ++r)
    if (hr[r]) {
      FG_CUDA(cudaMemcpyAsync(rhs[r], dr[r], p.nRows * 16, cudaMemcpyDeviceToHost, s));
      anyHost = true;
    }
  if (anyHost) {
    FG_CUDA(cudaStreamSynchronize(s));
    if (mixed) return mixedCheckTimeout(plan, true);
  }
  return FG_OK;
}

}  // namespace

extern "C" int fg_assemble_multi_freq(fg_plan *plan, const fg_term_desc *terms, int32_t n_terms, const double *omegas, int32_t n_freq,
                                      int32_t mixed, const double *dirichlet, double *csr_values, double *rhs, void *stream) {
  if (!plan) return FG_ERR_ARG;
  if (!terms || n_terms <= 0 || n_terms > kMaxTerms || !omegas || n_freq <= 0 || n_freq > kMaxFreq || !csr_values) {
    setLastError("fg_assemble_multi_freq: terms, 1..64 frequencies and csr_values are required");
    return FG_ERR_ARG;
  }
  const PlanDev &p = plan->d;
  std::vector<double *> v(n_freq), r(n_freq);
  for (int f = 0; f < n_freq; ++f) {
    v[f] = csr_values + 2 * p.nnz * (size_t)f;
    r[f] = rhs ? rhs + 2 * p.nRows * (size_t)f : nullptr;
  }
  // AFrequency factors (src/term/Assembler.cpp:283-295), on values and liftings alike
  auto coefOf = [&](const int *dts, int G, double2 *coef, double2 *rcoef) {
    for (int f = 0; f < n_freq; ++f)
      for (int g = 0; g < G; ++g) {
        const double w = omegas[f];
        const double2 c = dts[g] == FG_DT_2 ? make_double2(-w * w, 0.0) : dts[g] == FG_DT_1 ? make_double2(0.0, -w) : make_double2(1.0, 0.0);
        coef[(size_t)f * G + g] = c;
        rcoef[(size_t)f * G + g] = c;
      }
    return FG_OK;
  };
  return runGroups(plan, terms, n_terms, mixed, dirichlet, n_freq, v.data(), rhs ? n_freq : 0, r.data(), (cudaStream_t)stream, coefOf);
}

extern "C" int fg_assemble_separate(fg_plan *plan, const fg_term_desc *terms, int32_t n_terms, int32_t mixed, const double *dirichlet,
                                    double *k_values, double *c_values, double *m_values, double *rhs, void *stream) {
  if (!plan) return FG_ERR_ARG;
  if (!terms || n_terms <= 0 || n_terms > kMaxTerms) {
    setLastError("fg_assemble_separate: terms are required");
    return FG_ERR_ARG;
  }
  bool have[3] = {false, false, false};
  for (int t = 0; t < n_terms; ++t)
    if (terms[t].kind != FG_TERM_SOURCE && terms[t].dt >= FG_DT_NONE && terms[t].dt <= FG_DT_2) have[terms[t].dt] = true;
  double *out[3] = {k_values, c_values, m_values};
  for (int d = 0; d < 3; ++d) {
    if (have[d] && !out[d]) {
      setLastError("fg_assemble_separate: the formulation has a matrix whose output array is NULL");
      return FG_ERR_ARG;
    }
  }
  // value array f <- group f (the groups present, in the order K, C, M); the
  // right-hand side lifts with K alone (src/term/Assembler.cpp:306-347)
  auto coefOf = [&](const int *dts, int G, double2 *coef, double2 *rcoef) {
    for (int f = 0; f < G; ++f)
      for (int g = 0; g < G; ++g) coef[(size_t)f * G + g] = make_double2(f == g ? 1.0 : 0.0, 0.0);
    for (int g = 0; g < G; ++g) rcoef[g] = make_double2(dts[g] == FG_DT_NONE ? 1.0 : 0.0, 0.0);
    return FG_OK;
  };
  // a source without K terms still makes a group of dt 0
  bool sourceOnlyK = false;
  for (int t = 0; t < n_terms; ++t)
    if (terms[t].kind == FG_TERM_SOURCE) sourceOnlyK = !have[0];
  if (sourceOnlyK && !k_values) {
    setLastError("fg_assemble_separate: source terms need k_values (the stiffness group carries the right-hand side)");
    return FG_ERR_ARG;
  }
  std::vector<double *> vv;
  for (int d = 0; d < 3; ++d)
    if (have[d] || (d == FG_DT_NONE && sourceOnlyK)) vv.push_back(out[d]);
  double *r[1] = {rhs};
  return runGroups(plan, terms, n_terms, mixed, dirichlet, (int)vv.size(), vv.data(), rhs ? 1 : 0, r, (cudaStream_t)stream, coefOf);
}
