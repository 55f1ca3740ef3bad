// The CSR reduction (device code in gather.cuh): shapes and launches.
#include <algorithm>
#include <cstring>

#include "gather.cuh"

namespace femg {

constexpr size_t kGatherSmemMax = 200 * 1024;   // shared memory of a block
constexpr size_t kGatherSmemGood = 100 * 1024;  // ... up to which two blocks share an SM

// Rows per warp with which a CSR row has to fit the shared memory. The limit
// on row lengths follows from it; long rows run with fewer rows per warp.
static int limitRows(int nc, bool vec4) {
  if (vec4) return 32 / (nc / 4);
  return nc <= 6 ? 16 : nc <= 12 ? 8 : nc <= 40 ? 4 : nc <= 48 ? 2 : 1;
}

// Warps per block: 4 took 0.423 ms on 384,000 order-3 tetrahedra (FP32
// element matrices) where 8 took 0.443, and 0.091 against 0.108 ms on 55,566
// order-2 ones (complex FP64, the general kernel without a bound). With 64 warps per SM in the grid; 128 took 4%
// and a block per row group 12% longer (the pipeline starts anew in every
// block), 32 left the second example at 0.108.
// Columns come by vectors of VW values (16 bytes at most) where the rows of
// the element matrices keep them aligned. J vectors per lane: one, so that
// most rows share a warp (32 / L), but three from 12 vectors per row on (30
// columns: 6 rows of 5 lanes instead of 2 of 15), and 3 or 5 single columns.
// Rows of four columns take pieces of two: a row of one lane leaves a warp 32
// rows, and few warps (16,464 order-1 tetrahedra 16.2 us against 12.5, 384,000
// of them 30.7 against 27.0; with three components 26.6 against 20.4). At most
// eight rows where they add to what is there: it is read row after row at the
// end (three components on 16,464 order-1 tetrahedra 77 us a call, with 16 rows
// 86; one component on 82,944 of them 51.5 and 54.6), but in complex FP64, where
// eight take longer (63.7 and 59.5).
GatherShape gatherShape(const PlanDev &p, int maxRowLen, int kcplx, int isFloat, KeLayout lay, int wpb, bool acc) {
  GatherShape g;
  const int nc = p.nc;
  g.blocks3 = lay.kind == kKeBlocks3;
  if (g.blocks3) {
    const int nb = nc / 3;
    g.VW = nb % 4 == 0 && nb > 4 ? 4 : nb % 2 == 0 ? 2 : 1;
    g.J = 3;
    g.lanes.L = (nb + g.VW - 1) / g.VW;
  } else {
    g.VW = isFloat && nc % 4 == 0 && nc > 4 && lay.ld % 4 == 0 ? 4 : nc % 2 == 0 && lay.ld % 2 == 0 ? 2 : 1;
    const int pieces = (nc + g.VW - 1) / g.VW;
    g.J = g.VW == 4 ? 1 : g.VW == 2 ? (pieces >= 12 ? 3 : 1) : (nc <= 24 ? 3 : 5);
    g.lanes.L = (pieces + g.J - 1) / g.J;
  }
  g.lanes.R = 32 / g.lanes.L;
  if (acc && (isFloat || !kcplx)) g.lanes.R = std::min(g.lanes.R, 8);
  const size_t rowBytes = (size_t)std::max(maxRowLen, 1) * (kcplx ? 2 : 1) * (isFloat ? 4 : 8);
  const bool vec4 = isFloat && !kcplx && !g.blocks3 && nc % 4 == 0 && nc <= 32 && p.slotBytes == 1;
  g.ok = rowBytes * limitRows(nc, vec4) <= kGatherSmemMax;
  g.wpb = wpb > 0 ? wpb : 4;
  while (g.lanes.R > 1 && rowBytes * g.lanes.R * g.wpb > kGatherSmemGood) --g.lanes.R;
  if (wpb <= 0)
    while (g.wpb > 1 && rowBytes * g.lanes.R * g.wpb > kGatherSmemMax) g.wpb >>= 1;
  g.smem = rowBytes * g.lanes.R * g.wpb;
  g.ok = g.ok && g.smem <= kGatherSmemMax;
  g.rowsPerBlock = g.wpb * g.lanes.R;
  // lanes that write a finished row: 16 (8 where rows are shorter than that);
  // 32 measured 1 to 2% slower, on the 20-column tetrahedra up to 3%
  const double mean = p.nRows ? (double)p.nnz / (double)p.nRows : 0.0;
  g.lanes.lgOL = mean >= 12.0 ? 4 : 3;
  g.lanes.OL = 1 << g.lanes.lgOL;
  return g;
}

// The rows of visit records [v0, v1) (all rows: 0, nRows).
static int launchGatherRange(const PlanDev &p, const double *ke, int keComplex, int keIsFloat, KeLayout lay, const double *be,
                             const double *dirichletDev, double *values, double *rhs, int64_t v0, int64_t v1, bool acc,
                             cudaStream_t s) {
  if (v1 <= v0) return FG_OK;
  if (p.lscale && !keComplex) {
    setLastError("gather: linked DOFs need complex element matrices");
    return FG_ERR_UNSUPPORTED;
  }
  GatherLaunch a;
  std::memset(&a, 0, sizeof(a));
  a.g = gatherShape(p, p.maxRowLen, keComplex, keIsFloat, lay, 0, acc);
  if (!a.g.ok) {
    setLastError("gather: CSR row too long for shared memory");
    return FG_ERR_UNSUPPORTED;
  }
  a.slotBytes = p.slotBytes;
  a.kcplx = keComplex;
  a.acc = acc;
  a.mode = gatherMode(p, be);
  const int64_t groups = (v1 - v0 + a.g.rowsPerBlock - 1) / a.g.rowsPerBlock;
  a.blocks = std::max<int64_t>(1, std::min<int64_t>(groups, (int64_t)smCount() * kGatherWarpsPerSm / a.g.wpb));
  a.capped = a.blocks < groups;
  // complex FP32 in 16-byte pieces: on large plans the general kernel, 16
  // warps per SM in place of 28 (order 3, 105,456 tetrahedra 350 us a call and
  // 368, 48,000 179 and 182; 10,368, which fit the grid, 69 and 62)
  if (keIsFloat && keComplex && a.g.VW == 4 && !a.g.blocks3 && a.capped && !acc && a.mode == kGatherClean) a.mode = kGatherGeneral;
  // small systems only: blocks that come to an SM beside the contraction's run
  // with its division of L1 and shared memory, and 384,000 order-3 tetrahedra
  // took 0.773 ms a call instead of 0.632. Nor where the contraction runs over
  // more than one tile of 128 rows per SM, which the waiting blocks sit
  // through: three components on 16,464 order-1 tetrahedra 86 us a call against
  // 74, on 48,000 184 against 152; one component, 129 tiles, 26 against 35
  const int64_t rows = keIsFloat ? p.E * (a.g.blocks3 ? 9 : 1) * (keComplex ? 2 : 1) : 0;
  a.early = groups <= (int64_t)smCount() * kGatherWarpsPerSm / a.g.wpb && rows <= (int64_t)smCount() * 128;
  a.s = s;
  a.p = &p;
  a.ke = ke;
  a.be = (const double2 *)be;
  a.uD = (const double2 *)dirichletDev;
  a.values = (double2 *)values;
  a.rhs = (double2 *)rhs;
  a.lay = lay;
  a.v0 = v0;
  a.v1 = v1;
  ProfScope prof(a.g.VW == 4 && !a.g.blocks3 ? "k_gather_v4" : "k_gather", s);
  countLaunch();
  return keIsFloat ? launchGatherF32(a) : launchGatherF64(a);
}

int launchGather(fg_plan *plan, const double *ke, int keComplex, int keIsFloat, KeLayout lay, const double *be,
                 const double *dirichletDev, double *values, double *rhs, cudaStream_t s) {
  return launchGatherRange(plan->d, ke, keComplex, keIsFloat, lay, be, dirichletDev, values, rhs, 0, (int64_t)plan->d.nRows,
                           plan->accumulate != 0, s);
}

// Host values: the reduction runs range by range; after each range an event
// lets the copy stream bring that range's CSR slice to the host while the
// next range reduces (the copy, not the reduction, bounds a host-output call).
int gatherToOutputs(fg_plan *plan, const double *ke, int keComplex, int keIsFloat, KeLayout lay, const double *be,
                    const double *dirichletDev, Outputs &o, double *csr_values, cudaStream_t s) {
  const size_t nc = plan->outChunkRow.size() > 1 ? plan->outChunkRow.size() - 1 : 0;
  if (!o.hostValues || nc < 2)
    return launchGather(plan, ke, keComplex, keIsFloat, lay, be, dirichletDev, o.values, o.rhs, s);
  if (!plan->copyStream) {
    FG_CUDA(cudaStreamCreateWithFlags(&plan->copyStream, cudaStreamNonBlocking));
    plan->copyEvents.assign(nc, nullptr);
    for (auto &ev : plan->copyEvents) FG_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  }
  for (size_t c = 0; c < nc; ++c) {
    const uint64_t r0 = plan->outChunkRow[c], r1 = plan->outChunkRow[c + 1];
    int st = launchGatherRange(plan->d, ke, keComplex, keIsFloat, lay, be, dirichletDev, o.values, o.rhs, (int64_t)r0, (int64_t)r1, false, s);
    if (st) return st;
    FG_CUDA(cudaEventRecord(plan->copyEvents[c], s));
    FG_CUDA(cudaStreamWaitEvent(plan->copyStream, plan->copyEvents[c], 0));
    const uint64_t a0 = plan->hAi[r0], a1 = plan->hAi[r1];
    if (a1 > a0)
      FG_CUDA(cudaMemcpyAsync(csr_values + 2 * a0, o.values + 2 * a0, (a1 - a0) * 16, cudaMemcpyDeviceToHost, plan->copyStream));
  }
  o.valuesCopied = true;
  return FG_OK;
}

int launchGatherBatch(const GatherJob *jobsDev, int nJobs, int64_t blocks, int slotBytes, int kcplx, int keIsFloat,
                      const GatherShape &g, int mode, cudaStream_t s) {
  if (blocks <= 0) return FG_OK;
  countLaunch();
  GatherLaunch a;
  std::memset(&a, 0, sizeof(a));
  a.g = g;
  a.slotBytes = slotBytes;
  a.kcplx = kcplx;
  a.blocks = blocks;
  a.s = s;
  a.mode = mode;
  a.jobs = jobsDev;
  a.nJobs = nJobs;
  ProfScope prof(g.VW == 4 && !g.blocks3 ? "k_gather_batch_v4" : "k_gather_batch", s);
  return keIsFloat ? launchGatherF32(a) : launchGatherF64(a);
}

// The records of the visiting order (gather.cuh): per list entry the packed
// (element, local row), then the slots of its element row. A thread per word.
__global__ void k_records(const uint8_t *__restrict__ slot, int slotRowBytes, int usedBytes, const uint32_t *__restrict__ visitElem,
                          int64_t words, int n, int recWords, uint32_t *__restrict__ rec) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= words) return;
  const int64_t k = t / recWords;
  const int w = (int)(t - k * recWords);
  const uint32_t packed = visitElem[k];
  uint32_t out = packed;
  if (w > 0) {
    const uint8_t *row = slot + ((size_t)(packed >> 6) * n + (packed & 63)) * slotRowBytes;
    out = 0;
    for (int b = 0; b < 4; ++b) out |= (uint32_t)(4 * (w - 1) + b < usedBytes ? row[4 * (w - 1) + b] : 0xFF) << (8 * b);
  }
  rec[t] = out;
}

int buildRecords(const PlanDev &p, const uint32_t *visitElem, int64_t entries, uint32_t *rec) {
  if (entries == 0) return FG_OK;
  const int recWords = p.recLd / 4;
  const int64_t words = entries * recWords;
  k_records<<<(unsigned)((words + 255) / 256), 256>>>((const uint8_t *)p.slot, p.slotLd * p.slotBytes, p.nc * p.slotBytes, visitElem,
                                                      words, p.n, recWords, rec);
  countLaunch();
  FG_CUDA(cudaGetLastError());
  // the kernel's own stream alone: a wait for the device would end captures
  // that other streams have under way
  FG_CUDA(cudaStreamSynchronize(nullptr));
  return FG_OK;
}

}  // namespace femg
