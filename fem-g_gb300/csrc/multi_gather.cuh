// The CSR reduction of several term groups and frequencies at once (device
// code; multi_freq.cu picks the shapes, multi_f32.cu and multi_f64.cu hold the
// instances). 48,000 order-2 Navier tetrahedra at 8 frequencies: 0.580 ms for
// 2.2 GB of values written (1.28 ms without the pipeline, an atomic per group
// and column and a table lookup and two widenings per value written). The
// launch bound is left to the compiler: at 64 or 80 registers it spills, and
// the same launch takes 0.887 or 0.835 ms.
// The pipeline is the one of gather.cuh: records of the visiting
// order two steps ahead, the groups' element rows one step ahead, across row
// boundaries. Each slot has one sum per group (two when some group is
// complex); a finished row is written once per frequency, by OL lanes.
#pragma once
#include <type_traits>

#include "gather.cuh"

namespace femg {

constexpr int kMaxGroups = 3;
constexpr int kMaxFreq = 64;

struct MultiIn {
  const void *ke[kMaxGroups];    // element matrices of group g (KT)
  int64_t stride[kMaxGroups];    // KT entries from one element to the next
  int cplx[kMaxGroups];          // group g has an imaginary part (at +n*n)
  int realFactor[kMaxGroups];    // the factors of group g are real for every output
  int imagFactor[kMaxGroups];    // ... purely imaginary for every output
  int G, F, R;
  int allReal;                   // the factors of every group are real for every output
  int anyCplx;                   // some group has an imaginary part: two accumulators per group and slot, else one
  KeLayout lay;                  // element-matrix layout (ld entries per component)
  const double2 *coef;           // [F][G] factors of the value arrays
  const double2 *rcoef;          // [R][G] factors of the liftings in the right-hand sides
  const double2 *be;             // [E][n] element right-hand sides or null
  const double2 *uD;             // Dirichlet values or null
  double2 *const *values;        // F value arrays [nnz] (device table)
  double2 *const *rhs;           // R right-hand sides [nRows] (device table), or null
};

// A block's shared memory begins with the factors and the value arrays'
// addresses; the accumulators follow
__host__ __device__ inline int multiFactorBytes(int F, int G, int size) { return (F * G * 2 * size + 15) / 16 * 16; }
__host__ __device__ inline int multiHeadBytes(int F, int G, int size) { return multiFactorBytes(F, G, size) + (F * 8 + 15) / 16 * 16; }

// GM: at most so many groups (2, or 3 with the number read at run time);
// CPLX: some group has an imaginary part; SIMPLE: as in gather.cuh, two real groups
template <typename SlotT, typename KT, int VW, int J, bool BLOCKS, int GM, bool CPLX, bool SIMPLE>
__global__ void __launch_bounds__(256) k_gather_multi(const PlanDev p, const MultiIn in, const GatherLanes g) {
  constexpr int U = VW * J * (int)sizeof(KT) * GM * (CPLX ? 2 : 1) <= 16 ? 2 : 1;  // entries per step
  constexpr uint32_t kIgnore = sizeof(SlotT) == 1 ? 0xFEu : kSlotIgnore, kFixed = sizeof(SlotT) == 1 ? 0xFFu : kSlotFixed;
  constexpr int gStep = CPLX ? 2 : 1;
  const int G = GM == 2 ? 2 : in.G, F = in.F;
  extern __shared__ __align__(16) unsigned char smraw[];
  KT *cf = reinterpret_cast<KT *>(smraw);  // [F][G][2] factors in the accumulation type
  const bool allReal = !CPLX && in.allReal;  // then [F][G] real factors
  for (int k = threadIdx.x; k < F * G; k += blockDim.x) {
    if (allReal) {
      cf[k] = (KT)in.coef[k].x;
    } else {
      cf[2 * k] = (KT)in.coef[k].x;
      cf[2 * k + 1] = (KT)in.coef[k].y;
    }
  }
  double2 **out = reinterpret_cast<double2 **>(smraw + multiFactorBytes(F, G, sizeof(KT)));  // [F] value arrays
  for (int k = threadIdx.x; k < F; k += blockDim.x) out[k] = in.values[k];
  const int cfBytes = multiHeadBytes(F, G, sizeof(KT));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int L = g.L, R = g.R;
  const int sub = lane / L, lt = lane - sub * L;
  const bool laneLive = sub < R;
  const int lo = lane & (g.OL - 1);  // among the lanes writing a row
  const int perSlot = gStep * G;
  KT *Aw = reinterpret_cast<KT *>(smraw + cfBytes) + warp * R * p.maxRowLen * perSlot;
  KT *A = Aw + (laneLive ? sub : 0) * p.maxRowLen * perSlot;
  const int n = p.n, nb = BLOCKS ? p.nb : n;
  const int ld = in.lay.ld;  // entries per component
  const bool clean = SIMPLE || p.cleanSlots != 0, plain = SIMPLE || p.plainSlots != 0;
  const uint32_t recLd = (uint32_t)p.recLd;
  bool ok[J];
  int col[J];
#pragma unroll
  for (int c = 0; c < J; ++c) {
    const int q = BLOCKS ? lt : lt + L * c;
    ok[c] = laneLive && VW * q < nb;
    col[c] = (BLOCKS ? c * nb * nb : 0) + VW * q;
  }
  struct Step {
    uint32_t packed[U];
    SlotWords<SlotT, VW> sw[U][J];
  };
  struct Values {
    KT r[U][GM][J * VW], i[U][CPLX ? GM : 1][CPLX ? J * VW : 1];
  };
  auto loadRec = [&](uint32_t first, int k, int cnt, Step &s) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s.packed[u] = kRecNone;
      if (k + u < cnt) {
        const uint8_t *r = p.rec + (size_t)(first + k + u) * recLd;
        s.packed[u] = __ldg(reinterpret_cast<const uint32_t *>(r));
#pragma unroll
        for (int c = 0; c < J; ++c)
          if (ok[c]) s.sw[u][c].load(r + 4 + SlotWords<SlotT, VW>::kBytes * (BLOCKS ? 3 * lt + c : lt + L * c));
      }
    }
  };
  auto loadKe = [&](const Step &s, Values &v) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s.packed[u] != kRecNone) {
        const int64_t e = s.packed[u] >> 6;
        const int i = (int)(s.packed[u] & 63);
        int row = i * n;
        if (BLOCKS) {
          const int ib = (int)((unsigned)i / 3u), a = i - 3 * ib;
          row = (a * 3 * nb + ib) * nb;
        }
#pragma unroll
        for (int gr = 0; gr < GM; ++gr) {
          if (gr >= G) break;
          const KT *K = (const KT *)in.ke[gr] + e * in.stride[gr] + row;
#pragma unroll
          for (int c = 0; c < J; ++c)
            if (ok[c]) {
              loadValues<KT, VW>(K + col[c], &v.r[u][gr][c * VW]);
              if constexpr (CPLX) {
                if (in.cplx[gr]) loadValues<KT, VW>(K + ld + col[c], &v.i[u][gr][c * VW]);
              }
            }
        }
      }
  };
  for (int s = lane; s < R * p.maxRowLen * perSlot; s += 32) Aw[s] = (KT)0;
  __syncthreads();
  const int64_t nRows = (int64_t)p.nRows;
  const int64_t stride = (int64_t)gridDim.x * wpb * R;
  const int64_t base0 = ((int64_t)blockIdx.x * wpb + warp) * R;
  auto visitAt = [&](int64_t idx) { return laneLive && idx < nRows ? __ldg(&p.visit[idx]) : make_uint4(0, 0, 0, 0); };
  uint4 v = visitAt(base0 + sub), vN = visitAt(base0 + sub + stride);
  Step cur, nxt;
  Values val;
  loadRec(v.z, 0, (int)(v.w >> 16), cur);
  loadRec(v.z, U, (int)(v.w >> 16), nxt);
  loadKe(cur, val);
  for (int64_t base = base0; base < nRows; base += stride) {
    const int64_t idx = base + sub;
    const bool live = laneLive && idx < nRows;
    const uint4 vNN = visitAt(idx + 2 * stride);
    const int len = (int)(v.w & 0xFFFFu), cnt = (int)(v.w >> 16), cntN = (int)(vN.w >> 16);
    const int steps = max(1, ((int)__reduce_max_sync(0xffffffffu, (unsigned)cnt) + U - 1) / U);
    Step nextRow;
    loadRec(vN.z, 0, cntN, nextRow);
    double2 dc[GM];
#pragma unroll
    for (int gr = 0; gr < GM; ++gr) dc[gr] = make_double2(0.0, 0.0);
    double2 bsum = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int st = 0; st < steps; ++st) {
      const bool last = st + 1 == steps;
      if (last) nxt = nextRow;
      Values valN;
      loadKe(nxt, valN);
      Step after;
      if (last) loadRec(vN.z, U, cntN, after);
      else loadRec(v.z, (st + 2) * U, cnt, after);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (cur.packed[u] != kRecNone) {
          const int64_t e = cur.packed[u] >> 6;
          const int i = (int)(cur.packed[u] & 63);
          if (!SIMPLE && in.be && lt == 0) bsum = cadd(bsum, in.be[e * n + i]);
#pragma unroll
          for (int c = 0; c < J; ++c) {
            if (!ok[c]) continue;
#pragma unroll
            for (int w = 0; w < VW; ++w) {
              const int flat = BLOCKS ? 3 * w + c : c * VW + w;
              const uint32_t s = cur.sw[u][flat / VW].at(flat % VW);
              if constexpr (SIMPLE) {
                // two real groups: their sums by one access
                using Pair = typename std::conditional<sizeof(KT) == 4, float2, double2>::type;
                Pair *at = reinterpret_cast<Pair *>(A) + (int)s;
                Pair sum = *at;
                sum.x += val.r[u][0][c * VW + w];
                sum.y += val.r[u][1][c * VW + w];
                *at = sum;
              } else if (clean || s < kIgnore) {
                // distinct slots per lane within an element row unless the
                // plan says otherwise; rows are separated by the __syncwarp below
#pragma unroll
                for (int gr = 0; gr < GM; ++gr) {
                  if (gr >= G) break;
                  KT *at = A + (int)s * perSlot + gStep * gr;
                  if (plain) at[0] += val.r[u][gr][c * VW + w];
                  else atomicAdd(at, val.r[u][gr][c * VW + w]);
                  if constexpr (CPLX) {
                    if (in.cplx[gr]) {
                      if (plain) at[1] += val.i[u][gr][c * VW + w];
                      else atomicAdd(at + 1, val.i[u][gr][c * VW + w]);
                    }
                  }
                }
              } else if (!SIMPLE && s == kFixed) {
                // lifting with the transposed entry (VectorFactory::addValuesDC)
                const int j = BLOCKS ? 3 * (VW * lt + w) + c : VW * (lt + L * c) + w;
                const int o = keOffset(in.lay, n, j, i);
                const double2 uj = in.uD[p.edof[e * n + j]];
#pragma unroll
                for (int gr = 0; gr < GM; ++gr) {
                  if (gr >= G) break;
                  const KT *K = (const KT *)in.ke[gr] + e * in.stride[gr];
                  const double2 kv = make_double2((double)K[o], in.cplx[gr] ? (double)K[ld + o] : 0.0);
                  dc[gr] = cadd(dc[gr], cmul(kv, uj));
                }
              }
            }
          }
        }
        __syncwarp();
      }
      cur = nxt;
      nxt = after;
      val = valN;
    }
#pragma unroll 1
    for (int r = lane >> g.lgOL; r - (lane >> g.lgOL) < R; r += 32 >> g.lgOL) {
      const int rc = r < R ? r : 0;
      const int rLen = __shfl_sync(0xffffffffu, len, rc * L);
      const uint32_t start = __shfl_sync(0xffffffffu, v.y, rc * L);
      KT *Ar = Aw + rc * p.maxRowLen * perSlot;
#pragma unroll 1
      for (int s = lo; s < (r < R ? rLen : 0); s += g.OL) {
        KT ar[GM], ai[GM];
#pragma unroll
        for (int gr = 0; gr < GM; ++gr) {
          ar[gr] = ai[gr] = (KT)0;
          if (gr < G) {
            KT *sum = Ar + s * perSlot + gStep * gr;
            ar[gr] = sum[0];
            sum[0] = (KT)0;
            if constexpr (CPLX) {
              if (in.cplx[gr]) ai[gr] = sum[1];
              sum[1] = (KT)0;
            }
          }
        }
        const size_t at = (size_t)start + s;
        if (allReal) {
          // real sums and real factors (sweeps without damping, separate
          // matrices): no imaginary parts to form
#pragma unroll 2
          for (int f = 0; f < F; ++f) {
            KT re = (KT)0;
#pragma unroll
            for (int gr = 0; gr < GM; ++gr)
              if (gr < G) re += cf[f * G + gr] * ar[gr];
            out[f][at] = make_double2(widen(re), 0.0);
          }
          continue;
        }
#pragma unroll 1
        for (int f = 0; f < F; ++f) {
          KT re = (KT)0, im = (KT)0;
#pragma unroll
          for (int gr = 0; gr < GM; ++gr) {
            if (gr >= G) break;
            const KT cr = cf[2 * (f * G + gr)], ci = cf[2 * (f * G + gr) + 1];
            // real sums and real or imaginary factors (the usual case) skip the
            // zero products: they cost FP64 issue slots on the FP64 path
            if (in.realFactor[gr]) re += cr * ar[gr];
            else if (in.imagFactor[gr]) im += ci * ar[gr];
            else {
              re += cr * ar[gr];
              im += ci * ar[gr];
            }
            if (CPLX && in.cplx[gr]) {
              re -= ci * ai[gr];
              im += cr * ai[gr];
            }
          }
          out[f][at] = make_double2(widen(re), widen(im));
        }
      }
    }
    if (in.rhs) {
      // without fixed columns every right-hand side is the element vectors'
      // sum, and zero without those: the products by the frequencies' factors
      // would cost FP64 instructions on every row (a quarter of the pipe's
      // time, and of the kernel's, at 8 frequencies)
      if (SIMPLE || !in.uD) {
        if (live && lt == 0)
          for (int r = 0; r < in.R; ++r) in.rhs[r][v.x] = bsum;
      } else {
        double2 tot[GM];
#pragma unroll
        for (int gr = 0; gr < GM; ++gr) {
          tot[gr] = dc[gr];
          for (int t = 1; t < L; ++t) {
            const int src = laneLive ? sub * L + t : lane;
            tot[gr].x += __shfl_sync(0xffffffffu, dc[gr].x, src);
            tot[gr].y += __shfl_sync(0xffffffffu, dc[gr].y, src);
          }
        }
        if (live && lt == 0)
          for (int r = 0; r < in.R; ++r) {
            double2 b = bsum;
#pragma unroll
            for (int gr = 0; gr < GM; ++gr)
              if (gr < G) b = cadd(b, cmul(in.rcoef[r * G + gr], tot[gr]));
            in.rhs[r][v.x] = b;
          }
      }
    }
    __syncwarp();
    v = vN;
    vN = vNN;
  }
}

struct MultiLaunch {
  GatherShape g;
  MultiIn in;
  const PlanDev *p;
  int64_t blocks;
  cudaStream_t s;
};

template <typename SlotT, typename KT, int VW, int J, bool BLOCKS, int GM, bool CPLX, bool SIMPLE = false>
int launchMultiShape(const MultiLaunch &a) {
  auto kern = k_gather_multi<SlotT, KT, VW, J, BLOCKS, GM, CPLX, SIMPLE>;
  static SmemAllowance allowed;
  FG_CUDA(allowSmem(kern, a.g.smem, allowed));
  kern<<<(unsigned)a.blocks, 32 * a.g.wpb, a.g.smem, a.s>>>(*a.p, a.in, a.g.lanes);
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}
// real groups: two, or any number
template <typename SlotT, typename KT, int VW, int J, bool BLOCKS>
int launchMultiReal(const MultiLaunch &a) {
  if (a.in.G != 2) return launchMultiShape<SlotT, KT, VW, J, BLOCKS, 3, false>(a);
  return gatherMode(*a.p, a.in.be) == kGatherClean ? launchMultiShape<SlotT, KT, VW, J, BLOCKS, 2, false, true>(a)
                                     : launchMultiShape<SlotT, KT, VW, J, BLOCKS, 2, false>(a);
}

int launchMultiF32(const MultiLaunch &a);
int launchMultiF64(const MultiLaunch &a);

}  // namespace femg
