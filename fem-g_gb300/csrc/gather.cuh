// K4 + K5: deterministic row-owner reduction of element matrices and vectors
// into the CSR values and the right-hand side (device code; gather.cu picks
// the shapes, gather_f32.cu and gather_f64.cu hold the instances).
//
// Replaces MatrixFactory::addValues (src/system/MatrixFactory.cpp:233-448:
// lower_bound per entry + OpenMP atomics) and VectorFactory::addValues /
// addValuesDC (src/system/VectorFactory.cpp:122-210). Each CSR row is owned
// by a sub-warp of L lanes; the sub-warp walks the row's (element, local test
// index) list in element order, and every lane adds its columns of that
// element row into a shared accumulator at the slots precomputed by
// fg_plan_create. Entries are separated by __syncwarp, so each CSR value is
// summed in the same order on every run. Rows are visited sorted by their
// number of contributing elements, so the sub-warps of a warp run loops of
// equal length. Dirichlet lifting reads the transposed element entry, as
// addValuesDC does (values[j*n + i] * valuesDC[J],
// src/system/VectorFactory.cpp:184).
//
// The reduction is bound by the latency of its loads, not by their number, so
// they are taken off each other's path:
//  - A list entry and the slots of its element row sit in one record, and the
//    records lie in visiting order: a row's records are a contiguous stream
//    whose addresses are known from the row's visit record alone.
//  - Records are loaded two steps ahead and element rows one step ahead,
//    across row boundaries: the first element rows of the next CSR row are in
//    flight while the current row is summed and written. Most rows have two
//    (faces) to five (edges) entries, so a pipeline that starts anew on every
//    row is mostly empty. A step takes two entries where registers allow.
//  - A lane's columns come by 16- or 8-byte loads where the row length allows.
//  - The finished rows are written by OL lanes each, which also clear the
//    accumulator for the next rows.
// 384,000 order-3 tetrahedra, FP32 element matrices: 0.423 ms, 2.36 GB of DRAM
// traffic at 5.6 TB/s (0.570 ms with a row's loads started anew on every row,
// scalar adds through atomics and narrow stores); 162,000 of them in FP64
// 0.241 ms (0.365); 55,566 order-2 ones, complex FP64 with element vectors 0.081
// ms (0.106).
#pragma once
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace femg {

constexpr uint32_t kRecNone = 0xFFFFFFFFu;  // packed (element, local row) of no entry

// VW values of type KT, naturally aligned to the whole vector (16 bytes at
// most), by ordinary (coherent) loads: the kernel that writes the element
// matrices may still run when this one starts, so they are not read-only over
// this kernel's life, which ld.global.nc (__ldg) asks for. asm, so that a load
// is known to be from global memory and can be placed among the shared-memory
// adds; it stays behind gridWait() because its address comes from afterWait().
template <typename KT, int VW>
__device__ __forceinline__ void loadValues(const KT *p, KT *out) {
  const size_t g = __cvta_generic_to_global(p);
  if constexpr (sizeof(KT) == 4) {
    if constexpr (VW == 4) asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(out[0]), "=f"(out[1]), "=f"(out[2]), "=f"(out[3]) : "l"(g));
    else if constexpr (VW == 2) asm("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(out[0]), "=f"(out[1]) : "l"(g));
    else asm("ld.global.f32 %0, [%1];" : "=f"(out[0]) : "l"(g));
  } else {
    if constexpr (VW == 2) asm("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(out[0]), "=d"(out[1]) : "l"(g));
    else asm("ld.global.f64 %0, [%1];" : "=d"(out[0]) : "l"(g));
  }
}

// VW slots, packed in one or two words
template <typename SlotT, int VW>
struct SlotWords {
  static constexpr int kBytes = VW * (int)sizeof(SlotT), kWords = kBytes > 4 ? 2 : 1;
  uint32_t w[kWords];
  __device__ __forceinline__ void load(const uint8_t *r) {
    if constexpr (kBytes == 8) {
      w[0] = __ldg(reinterpret_cast<const uint32_t *>(r));
      w[1] = __ldg(reinterpret_cast<const uint32_t *>(r + 4));
    } else if constexpr (kBytes == 4) {
      w[0] = __ldg(reinterpret_cast<const uint32_t *>(r));
    } else if constexpr (kBytes == 2) {
      w[0] = __ldg(reinterpret_cast<const uint16_t *>(r));
    } else {
      w[0] = __ldg(r);
    }
  }
  __device__ __forceinline__ uint32_t at(int t) const {
    const int b = t * (int)sizeof(SlotT);
    return __byte_perm(w[b / 4], 0, sizeof(SlotT) == 1 ? 0x4440 + b % 4 : 0x4400 + 0x11 * (b % 4) + 0x10);
  }
};

// The rows of visit records [v0, v1) handled by block `blk` of `nblk`.
// FULL layout: lane lt of a row's L lanes owns the pieces lt + L c (c < J) of
// VW columns. BLOCKS (compound fields on the tensor-core path): it owns the
// scalar columns VW lt .. VW lt + VW - 1 of the three component blocks
// (J = 3), which are 3 VW consecutive DOF columns and so consecutive slots.
// MODE: kGatherClean and kGatherOpen are for plans without linked DOFs and
// fixed columns whose element rows have no two columns in one slot
// (p.plainSlots), and no element vectors: half the registers of
// kGatherGeneral. kGatherClean: every slot is a column of the row
// (p.cleanSlots); kGatherOpen: some columns are not stored (upper storage).
template <typename SlotT, bool KCPLX, typename KT, int VW, int J, bool BLOCKS, bool ACC, int MODE>
__device__ __forceinline__ void gatherRows(const PlanDev &p, const KT *ke, const double2 *be, const double2 *uD,
                                           double2 *__restrict__ values, double2 *__restrict__ rhs, const GatherLanes g,
                                           KeLayout lay, int64_t blk, int64_t nblk, int64_t v0, int64_t v1) {
  constexpr int SS = KCPLX ? 2 : 1;
  constexpr bool SIMPLE = MODE != kGatherGeneral;
  constexpr int U = VW * J * (int)sizeof(KT) * SS <= 16 ? 2 : 1;  // entries per step
  constexpr uint32_t kIgnore = sizeof(SlotT) == 1 ? 0xFEu : kSlotIgnore, kFixed = sizeof(SlotT) == 1 ? 0xFFu : kSlotFixed;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int L = g.L, R = g.R;
  const int sub = lane / L, lt = lane - sub * L;
  const bool laneLive = sub < R;
  const int lo = lane & (g.OL - 1);  // among the lanes writing a row
  KT *Aw = reinterpret_cast<KT *>(smraw) + warp * R * p.maxRowLen * SS;  // this warp's rows
  KT *A = Aw + (laneLive ? sub : 0) * p.maxRowLen * SS;
  const int n = p.n, nc = p.nc, nb = BLOCKS ? p.nb : nc;
  const uint32_t ld = (uint32_t)lay.ld;  // entries per component
  const bool clean = MODE == kGatherClean || (!SIMPLE && p.cleanSlots != 0), plain = SIMPLE || p.plainSlots != 0;
  const uint8_t *recs = p.rec;
  const uint32_t recLd = (uint32_t)p.recLd;
  bool ok[J];  // the lane's pieces that exist
  int col[J];  // their offset in an element row
#pragma unroll
  for (int c = 0; c < J; ++c) {
    const int q = BLOCKS ? lt : lt + L * c;
    ok[c] = laneLive && VW * q < nb;
    col[c] = (BLOCKS ? c * nb * nb : 0) + VW * q;
  }

  struct Step {  // U entries: their records and element-row values
    uint32_t packed[U];
    SlotWords<SlotT, VW> sw[U][J];
  };
  auto loadRec = [&](uint32_t first, int k, int cnt, Step &s) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s.packed[u] = kRecNone;
      if (k + u < cnt) {
        const uint8_t *r = recs + (size_t)(first + k + u) * recLd;
        s.packed[u] = __ldg(reinterpret_cast<const uint32_t *>(r));
#pragma unroll
        for (int c = 0; c < J; ++c)
          if (ok[c]) s.sw[u][c].load(r + 4 + SlotWords<SlotT, VW>::kBytes * (BLOCKS ? 3 * lt + c : lt + L * c));
      }
    }
  };
  auto loadKe = [&](const Step &s, KT (&vr)[U][J * VW], KT (&vi)[U][KCPLX ? J * VW : 1], double2 (&vb)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s.packed[u] != kRecNone) {
        const uint32_t e = s.packed[u] >> 6, i = s.packed[u] & 63;
        uint32_t row = i * (uint32_t)nc;
        if (BLOCKS) {
          const uint32_t ib = i / 3, a = i - 3 * ib;
          row = (a * 3 * nb + ib) * nb;
        }
        if (!SIMPLE && be && lt == 0) {
          double b[2];
          loadValues<double, 2>(&be[(size_t)e * n + i].x, b);
          vb[u] = make_double2(b[0], b[1]);
        }
        const KT *K = ke + ((uint64_t)e * (SS * ld) + row);
#pragma unroll
        for (int c = 0; c < J; ++c)
          if (ok[c]) {
            loadValues<KT, VW>(K + col[c], &vr[u][c * VW]);
            if constexpr (KCPLX) loadValues<KT, VW>(K + ld + col[c], &vi[u][c * VW]);
          }
      }
  };

  const int64_t stride = nblk * wpb * R;
  const int64_t first = v0 + (blk * wpb + warp) * R + sub;
  auto visitAt = [&](int64_t idx) { return laneLive && idx < v1 ? __ldg(&p.visit[idx]) : make_uint4(0, 0, 0, 0); };
  for (int s = lane; s < R * p.maxRowLen * SS; s += 32) Aw[s] = (KT)0;
  // the pipeline: values of the current step, records of the next one
  uint4 v = visitAt(first), vN = visitAt(first + stride);
  Step cur, nxt;
  KT vr[U][J * VW], vi[U][KCPLX ? J * VW : 1];
  double2 vb[U];  // the element vectors' entries (first lane of a row)
  loadRec(v.z, 0, (int)(v.w >> 16), cur);
  loadRec(v.z, U, (int)(v.w >> 16), nxt);
  gridWait();  // the kernel that writes the element matrices and vectors
  ke = afterWait(ke);
  be = afterWait(be);
  uD = afterWait(uD);
  if (ACC) {  // what the values and right-hand sides held before this plan
    values = afterWait(values);
    rhs = afterWait(rhs);
  }
  loadKe(cur, vr, vi, vb);
  __syncwarp();
  for (int64_t base = v0 + (blk * wpb + warp) * R; base < v1; base += stride) {
    const int64_t idx = base + sub;
    const bool live = laneLive && idx < v1;
    const uint4 vNN = visitAt(idx + 2 * stride);
    const int len = (int)(v.w & 0xFFFFu), cnt = (int)(v.w >> 16), cntN = (int)(vN.w >> 16);
    // rows without entries take one empty step, which carries the pipeline on
    const int steps = max(1, ((int)__reduce_max_sync(0xffffffffu, (unsigned)cnt) + U - 1) / U);
    Step nextRow;
    loadRec(vN.z, 0, cntN, nextRow);
    if (ACC) {  // what the rows hold, towards L2 while they are summed
#pragma unroll 1
      for (int r = lane >> g.lgOL; r - (lane >> g.lgOL) < R; r += 32 >> g.lgOL) {
        const int rc = r < R ? r : 0;
        const int rLen = __shfl_sync(0xffffffffu, len, rc * L);
        const uint32_t start = __shfl_sync(0xffffffffu, v.y, rc * L);
        // eight values to a line of 128 bytes
        if (r < R)
          for (int s = 8 * lo; s < rLen + 7; s += 8 * g.OL)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(values + ((size_t)start + min(s, rLen - 1))));
      }
    }
    double2 dc = make_double2(0.0, 0.0), bsum = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int st = 0; st < steps; ++st) {
      const bool last = st + 1 == steps;
      if (last) nxt = nextRow;
      KT vrN[U][J * VW], viN[U][KCPLX ? J * VW : 1];
      double2 vbN[U];
      loadKe(nxt, vrN, viN, vbN);
      Step after;
      if (last) loadRec(vN.z, U, cntN, after);
      else loadRec(v.z, (st + 2) * U, cnt, after);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (cur.packed[u] != kRecNone) {
          const uint32_t e = cur.packed[u] >> 6, i = cur.packed[u] & 63;
          // linked DOFs (complex element matrices only): the row scales by the
          // conjugate of its coefficient, each column by its own
          const bool linked = !SIMPLE && KCPLX && p.lscale != nullptr;
          double2 cI = make_double2(1.0, 0.0);
          if (linked) {
            cI = p.lscale[(size_t)e * n + i];
            cI.y = -cI.y;
          }
          if (!SIMPLE && be && lt == 0) {
            bsum = cadd(bsum, linked ? cmul(cI, vb[u]) : vb[u]);
          }
#pragma unroll
          for (int c = 0; c < J; ++c) {
            if (!ok[c]) continue;
#pragma unroll
            for (int w = 0; w < VW; ++w) {
              const int flat = BLOCKS ? 3 * w + c : c * VW + w;  // the lane's slots in DOF column order
              const uint32_t s = cur.sw[u][flat / VW].at(flat % VW);
              const int j = BLOCKS ? 3 * (VW * lt + w) + c : VW * (lt + L * c) + w;  // DOF column
              if (clean || s < kIgnore) {
                KT ar = vr[u][c * VW + w], ai = KCPLX ? vi[u][KCPLX ? c * VW + w : 0] : (KT)0;
                if (linked) {
                  const double2 cc = cmul(cI, p.lscale[(size_t)e * n + j]);
                  const KT tr = ar * (KT)cc.x - ai * (KT)cc.y;
                  ai = ar * (KT)cc.y + ai * (KT)cc.x;
                  ar = tr;
                }
                // an element row's columns sit in distinct slots unless the
                // plan says otherwise; successive element rows are ordered by
                // the __syncwarp below
                KT *at = A + (int)s * SS;
                if constexpr (SIMPLE && KCPLX) {  // both parts by one access
                  using Pair = typename std::conditional<sizeof(KT) == 4, float2, double2>::type;
                  Pair sum = *reinterpret_cast<Pair *>(at);
                  sum.x += ar;
                  sum.y += ai;
                  *reinterpret_cast<Pair *>(at) = sum;
                } else if (plain) {
                  at[0] += ar;
                  if (KCPLX) at[1] += ai;
                } else {
                  atomicAdd(at, ar);
                  if (KCPLX) atomicAdd(at + 1, ai);
                }
              } else if (!SIMPLE && s == kFixed) {
                // (a two-field plan with fixed columns has as many columns as rows)
                const KT *Kt = ke + (size_t)e * SS * ld;
                const int o = keOffset(lay, nc, j, (int)i);
                double2 t = make_double2((double)Kt[o], KCPLX ? (double)Kt[ld + o] : 0.0);
                if (linked) t = cmul(cI, t);
                dc = cadd(dc, cmul(t, uD[p.edofU[(size_t)e * nc + j]]));
              }
            }
          }
        }
        __syncwarp();
      }
      cur = nxt;
      nxt = after;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!SIMPLE) vb[u] = vbN[u];
#pragma unroll
        for (int k = 0; k < J * VW; ++k) {
          vr[u][k] = vrN[u][k];
          if constexpr (KCPLX) vi[u][k] = viN[u][k];
        }
      }
    }
    // ACC: add into the values (several buckets sharing rows) instead of overwriting them
#pragma unroll 1
    for (int r = lane >> g.lgOL; r - (lane >> g.lgOL) < R; r += 32 >> g.lgOL) {
      const int rc = r < R ? r : 0;
      const int rLen = __shfl_sync(0xffffffffu, len, rc * L);
      const uint32_t start = __shfl_sync(0xffffffffu, v.y, rc * L);
      KT *Ar = Aw + (rc * p.maxRowLen + lo) * SS;
      double2 *out = values + ((size_t)start + lo);
#pragma unroll 2
      for (int s = r < R ? rLen - lo : 0; s > 0; s -= g.OL, Ar += g.OL * SS, out += g.OL) {
        double2 val = make_double2(widen(Ar[0]), KCPLX ? widen(Ar[SS - 1]) : 0.0);
        Ar[0] = (KT)0;
        if (KCPLX) Ar[SS - 1] = (KT)0;
        if (ACC) val = cadd(*out, val);
        *out = val;
      }
    }
    if (rhs) {
      double2 tot = bsum;
      if (!SIMPLE && uD) {  // the sub-warp's lifted terms, summed on its first lane
        tot = cadd(tot, dc);
        for (int t = 1; t < L; ++t) {
          const int src = laneLive ? sub * L + t : lane;
          tot.x += __shfl_sync(0xffffffffu, dc.x, src);
          tot.y += __shfl_sync(0xffffffffu, dc.y, src);
        }
      }
      if (live && lt == 0) rhs[v.x] = ACC ? cadd(rhs[v.x], tot) : tot;
    }
    __syncwarp();
    v = vN;
    vN = vNN;
  }
}

// Blocks of 256 threads per SM the compiler makes room for: four (64
// registers) where a lane holds few bytes of an element row and the kernel is
// a lean one, else two, which leaves the others as many warps as their loads
// need: with four blocks they spill (35 columns: complex FP32 127 us a call on
// 6,000 order-4 tetrahedra, two 99.8; complex FP64 370 and 293), without a
// bound the general kernel takes up to 174 registers (35 columns in complex
// FP64 with element vectors 526 us, two 424, three 689).
// The lean kernels against the general one, which took these calls before:
// complex 35 columns in FP32 (10,368 tetrahedra) 288 us a call, now 147; upper
// storage on 48,000 order-3 tetrahedra 139 and 101, outputs added to 244 and
// 160.
constexpr int gatherBlocksPerSm(int laneBytes, int mode) {
  return mode == kGatherGeneral ? 2 : laneBytes <= 24 ? 4 : 2;
}

template <typename SlotT, bool KCPLX, typename KT, int VW, int J, bool BLOCKS, bool ACC, int MODE>
__global__ void __launch_bounds__(256, gatherBlocksPerSm(VW * J * (int)sizeof(KT) * (KCPLX ? 2 : 1), MODE))
    k_gather(const PlanDev p, const KT *ke, const double2 *be, const double2 *uD, double2 *__restrict__ values,
             double2 *__restrict__ rhs, const GatherLanes g, KeLayout lay, int64_t v0, int64_t v1) {
  gatherRows<SlotT, KCPLX, KT, VW, J, BLOCKS, ACC, MODE>(p, ke, be, uD, values, rhs, g, lay, blockIdx.x, gridDim.x, v0, v1);
}

// Many plans in one launch: job q owns blocks [blockStart, blockStart + nBlocks)
template <typename SlotT, bool KCPLX, typename KT, int VW, int J, bool BLOCKS, int MODE>
__global__ void __launch_bounds__(256, gatherBlocksPerSm(VW * J * (int)sizeof(KT) * (KCPLX ? 2 : 1), MODE))
    k_gather_batch(const GatherJob *__restrict__ jobs, int nJobs, const GatherLanes g) {
  int lo = 0, hi = nJobs - 1;
  while (lo < hi) {  // last job whose blockStart <= blockIdx.x
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].blockStart <= (int64_t)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const GatherJob &Jb = jobs[lo];
  gatherRows<SlotT, KCPLX, KT, VW, J, BLOCKS, false, MODE>(Jb.p, (const KT *)Jb.ke, Jb.be, Jb.uD, Jb.values, Jb.rhs, g, Jb.lay,
                                                             (int64_t)blockIdx.x - Jb.blockStart, Jb.nBlocks, 0, (int64_t)Jb.p.nRows);
}

// One launch: a single plan (jobs null) or a batch class
struct GatherLaunch {
  GatherShape g;
  int slotBytes, kcplx;
  bool acc;
  int mode;
  bool early;  // may start before the element kernel ends
  int64_t blocks;
  bool capped;  // fewer blocks than row groups
  cudaStream_t s;
  // a single plan
  const PlanDev *p;
  const void *ke;
  const double2 *be, *uD;
  double2 *values, *rhs;
  KeLayout lay;
  int64_t v0, v1;
  // a batch class
  const GatherJob *jobs;
  int nJobs;
};

template <typename SlotT, bool KCPLX, typename KT, int VW, int J, bool BLOCKS, int MODE>
int launchGatherBatchKernel(const GatherLaunch &a) {
  auto kern = k_gather_batch<SlotT, KCPLX, KT, VW, J, BLOCKS, MODE>;
  static SmemAllowance allowed;
  FG_CUDA(allowSmem(kern, a.g.smem, allowed));
  kern<<<(unsigned)a.blocks, 32u * (unsigned)a.g.wpb, a.g.smem, a.s>>>(a.jobs, a.nJobs, a.g.lanes);
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}
template <typename SlotT, bool KCPLX, typename KT, int VW, int J, bool BLOCKS, bool ACC, int MODE>
int launchGatherKernel(const GatherLaunch &a) {
  auto kern = k_gather<SlotT, KCPLX, KT, VW, J, BLOCKS, ACC, MODE>;
  static SmemAllowance allowed;
  FG_CUDA(allowSmem(kern, a.g.smem, allowed));
  int64_t blocks = a.blocks;
  if (a.capped) {
    // whole rounds of the blocks that are resident at once: with 28 warps per
    // SM of 64 in the grid the last round was a quarter full (complex order 3,
    // 48,000 tetrahedra 190 us a call, with 56 in the grid 182)
    int resident = 0;
    FG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, 32 * a.g.wpb, a.g.smem));
    const int warps = std::max(resident, 1) * a.g.wpb;
    blocks = (int64_t)smCount() * std::max(resident, 1) * std::max(1, (kGatherWarpsPerSm + warps / 2) / warps);
  }
  FG_CUDA(launchDependent(a.early, kern, (unsigned)blocks, 32u * (unsigned)a.g.wpb, a.g.smem, a.s, *a.p, (const KT *)a.ke, a.be, a.uD,
                          a.values, a.rhs, a.g.lanes, a.lay, a.v0, a.v1));
  return FG_OK;
}
template <typename SlotT, bool KCPLX, typename KT, int VW, int J, bool BLOCKS>
int launchGatherShape(const GatherLaunch &a) {
#define FG_GATHER_MODE(M)                                                              \
  (a.jobs  ? launchGatherBatchKernel<SlotT, KCPLX, KT, VW, J, BLOCKS, M>(a)            \
   : a.acc ? launchGatherKernel<SlotT, KCPLX, KT, VW, J, BLOCKS, true, M>(a)           \
           : launchGatherKernel<SlotT, KCPLX, KT, VW, J, BLOCKS, false, M>(a))
  switch (a.mode) {
    case kGatherClean: return FG_GATHER_MODE(kGatherClean);
    case kGatherOpen: return FG_GATHER_MODE(kGatherOpen);
    default: return FG_GATHER_MODE(kGatherGeneral);
  }
#undef FG_GATHER_MODE
}

int launchGatherF32(const GatherLaunch &a);
int launchGatherF64(const GatherLaunch &a);

}  // namespace femg
