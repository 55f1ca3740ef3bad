// GPU DOF numbering: DofsManager::reorderWithHilbert(true)
// (src/dofs/DofsManager.cpp:118-331) with the Hilbert sort of
// src/reorder/Hilbert.cpp:174-288.
//
// Keys: float coordinates scaled into the box exactly as the host does it,
// an unfused float multiply then add (__fmul_rn, __fadd_rn) truncated to an
// integer per axis, walked through the Hilbert state tables (2D: 32 bits
// per axis, 3D: 21). The order is the stable order of the keys: a radix sort
// of (key, input index) by eight bits a pass, least first, each pass stable.
// The numbering sorts every DOF by one more pass over its class (Unknown,
// Unknown bubble, other), so that the host neither picks out nor spreads the
// DOFs: on 195,112 DOFs, 0.63 ms a call in place of 2.4. A radix sort is 18 to
// 29 launches whatever the size; up to kBlockSort items are sorted by one
// block instead.
#include <algorithm>
#include <cmath>
#include <vector>

#include "../host/dofs.h"
#include "common.cuh"

namespace femg {

constexpr int kRadixThreads = 256, kRadixWarps = 8;
constexpr int kRadixTile = 4096, kRadixTileSmall = 1024;  // 512 or 128 consecutive items per warp
constexpr uint32_t kRadixSmall = 65536;  // up to so many items: small tiles, whose counts the scatter scans itself
constexpr uint32_t kBlockSort = 8192;  // up to so many: one block

struct HilbertDev {
  uint8_t code[24][8];
  uint8_t next[24][8];
};

// Keys of the points pts [n][stride], index i beside each. cls (may be null):
// the class of DOF i by its assemble type. count (may be null): for the sort by
// one block, the classes go with the indices, and DOFs that get no number are
// left out (the order of the others does not matter to that sort)
__global__ void k_hilbert_keys(int dim, uint64_t n, const float *__restrict__ pts, int stride, float3 scale, float3 scaleMin,
                               const HilbertDev tab, uint64_t *__restrict__ keys, uint32_t *__restrict__ idx,
                               const int32_t *__restrict__ type, uint8_t *__restrict__ cls, uint32_t *__restrict__ count) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float sc[3] = {scale.x, scale.y, scale.z}, sm[3] = {scaleMin.x, scaleMin.y, scaleMin.z};
  uint32_t u[3] = {0, 0, 0};
  for (int j = 0; j < dim; ++j) u[j] = __float2uint_rz(__fadd_rn(__fmul_rn(pts[i * stride + j], sc[j]), sm[j]));
  const int begBit = (64 / dim) - 1;
  uint64_t h = 0;
  unsigned ed = 0;
  for (int m = begBit; m >= 0; --m) {
    unsigned l = 0;
    for (int c = dim - 1; c >= 0; --c) l ^= ((u[c] >> m) & 1u) << c;
    h <<= dim;
    h ^= tab.code[ed][l];
    ed = tab.next[ed][l];
  }
  const uint32_t c = !cls ? 0u : type[i] == FG_AT_UNKNOWN ? 0u : type[i] == FG_AT_UNKNOWN_BUBBLE ? 1u : 2u;
  if (count) {
    if (c == 2u) return;
    const uint32_t at = atomicAdd(count, 1u);
    keys[at] = h;
    idx[at] = c << 30 | (uint32_t)i;
    return;
  }
  keys[i] = h;
  idx[i] = (uint32_t)i;
  if (cls) cls[i] = (uint8_t)c;
}

struct SortItem {
  uint64_t key;
  uint32_t idx;  // class << 30 | index
};
__device__ __forceinline__ void sortPair(SortItem &a, SortItem &b, bool up) {
  const uint32_t ca = a.idx >> 30, cb = b.idx >> 30;
  // no two items are equal but the padding
  const bool after = ca != cb ? ca > cb : a.key != b.key ? a.key > b.key : a.idx > b.idx;
  if (after == up) {
    const SortItem t = a;
    a = b;
    b = t;
  }
}

// Sort of up to kBlockSort items by (class, key, index) in one block: a bitonic
// network over `padded` (a power of two) items in shared memory, two strides
// at a time; then the order itself, or numbers from 1 on. Shared memory skips a
// place after every 16 items, which takes most of the small strides' bank
// conflicts away.
__device__ __forceinline__ uint32_t sortPlace(uint32_t i) { return i + (i >> 4); }
__global__ void __launch_bounds__(1024) k_sort_block(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ idx, uint32_t n,
                                                    uint32_t padded, uint32_t *__restrict__ perm, uint64_t *__restrict__ num) {
  extern __shared__ __align__(16) uint64_t sk[];
  uint32_t *si = reinterpret_cast<uint32_t *>(sk + sortPlace(padded));
  for (uint32_t t = threadIdx.x; t < padded; t += blockDim.x) {
    sk[sortPlace(t)] = t < n ? keys[t] : ~0ull;
    si[sortPlace(t)] = t < n ? idx[t] : 0xFFFFFFFFu;  // after every item
  }
  __syncthreads();
  for (uint32_t lgk = 1; (1u << lgk) <= padded; ++lgk) {
    const uint32_t k = 1u << lgk;
    uint32_t lgj = lgk;  // the strides below 2^lgj are left
    if (lgk & 1) {       // an odd number of them: the largest by itself
      --lgj;
      const uint32_t j = 1u << lgj;
      for (uint32_t t = threadIdx.x; t < padded / 2; t += blockDim.x) {
        const uint32_t lo = 2 * t - (t & (j - 1)), pl = sortPlace(lo), ph = sortPlace(lo + j);
        SortItem a = {sk[pl], si[pl]}, b = {sk[ph], si[ph]};
        sortPair(a, b, (lo & k) == 0);
        sk[pl] = a.key, si[pl] = a.idx;
        sk[ph] = b.key, si[ph] = b.idx;
      }
      __syncthreads();
    }
    for (; lgj > 0; lgj -= 2) {
      const uint32_t q = 1u << (lgj - 2);  // strides 2q, then q
      for (uint32_t t = threadIdx.x; t < padded / 4; t += blockDim.x) {
        const uint32_t lo = 4 * t - 3 * (t & (q - 1));
        const bool up = (lo & k) == 0;
        SortItem v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = {sk[sortPlace(lo + c * q)], si[sortPlace(lo + c * q)]};
        sortPair(v[0], v[2], up);
        sortPair(v[1], v[3], up);
        sortPair(v[0], v[1], up);
        sortPair(v[2], v[3], up);
#pragma unroll
        for (int c = 0; c < 4; ++c) sk[sortPlace(lo + c * q)] = v[c].key, si[sortPlace(lo + c * q)] = v[c].idx;
      }
      __syncthreads();
    }
  }
  for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) {
    const uint32_t i = si[sortPlace(t)] & 0x3FFFFFFFu;
    if (perm) perm[t] = i;
    else num[i] = t + 1;
  }
}

// The digit of item k in a pass: eight bits of its key, or its DOF's class
struct RadixDigit {
  const uint64_t *keys;
  const uint32_t *idx;
  const uint8_t *cls;  // not null: the pass over the classes
  int shift;
  __device__ __forceinline__ uint32_t at(uint64_t k) const { return cls ? cls[idx[k]] : (uint32_t)(keys[k] >> shift) & 0xFFu; }
};

// Digit counts of a tile into hist[digit][tile]
__global__ void __launch_bounds__(kRadixThreads) k_radix_count(const RadixDigit d, uint64_t n, uint32_t tile, uint32_t tiles, uint32_t *__restrict__ hist) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t end = min(n, ((uint64_t)blockIdx.x + 1) * tile);
  for (uint64_t k = (uint64_t)blockIdx.x * tile + threadIdx.x; k < end; k += kRadixThreads) atomicAdd(&h[d.at(k)], 1u);
  __syncthreads();
  hist[(uint64_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of each digit's counts over the tiles, in place; totals[digit]
__global__ void __launch_bounds__(kRadixThreads) k_radix_scan(uint32_t *__restrict__ hist, uint32_t tiles, uint32_t *__restrict__ totals) {
  __shared__ uint32_t warpSum[kRadixWarps];
  uint32_t *row = hist + (uint64_t)blockIdx.x * tiles;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (uint32_t b = 0; b < tiles; b += kRadixThreads) {
    const uint32_t k = b + threadIdx.x, v = k < tiles ? row[k] : 0u;
    uint32_t inc = v;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += o;
    }
    if (lane == 31) warpSum[warp] = inc;
    __syncthreads();
    uint32_t before = carry, all = 0;
    for (int w = 0; w < kRadixWarps; ++w) {
      if (w < warp) before += warpSum[w];
      all += warpSum[w];
    }
    if (k < tiles) row[k] = before + inc - v;
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// The items of a tile to their places: after all items of smaller digits,
// those of the digit in earlier tiles, in earlier warps of this one (a warp
// has consecutive items) and earlier in the warp (32 at a time, the equal
// digits of which are matched). SMALL: hist holds the tiles' counts as they
// are, and there are few enough of them to be summed here.
template <bool SMALL>
__global__ void __launch_bounds__(kRadixThreads)
    k_radix_scatter(const RadixDigit d, uint64_t n, uint32_t tiles, const uint32_t *__restrict__ hist, const uint32_t *__restrict__ totals,
                    uint64_t *__restrict__ keysOut, uint32_t *__restrict__ idxOut) {
  __shared__ uint32_t place[kRadixWarps][256];
  __shared__ uint32_t warpSum[kRadixWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int w = 0; w < kRadixWarps; ++w) place[w][tid] = 0;
  __syncthreads();
  constexpr int kTile = SMALL ? kRadixTileSmall : kRadixTile, kPer = kTile / kRadixWarps;
  const uint64_t w0 = (uint64_t)blockIdx.x * kTile + (uint64_t)warp * kPer;
  for (int r = 0; r < kPer; r += 32)
    if (w0 + r + lane < n) atomicAdd(&place[warp][d.at(w0 + r + lane)], 1u);
  // exclusive scan of the digits' totals, one digit per thread
  uint32_t total = 0, earlier = 0;  // of the digit, and in earlier tiles
  if (SMALL) {
#pragma unroll 4
    for (uint32_t t = 0; t < tiles; ++t) {
      const uint32_t c = hist[(uint64_t)tid * tiles + t];
      total += c;
      earlier += t < blockIdx.x ? c : 0u;
    }
  } else {
    total = totals[tid];
    earlier = hist[(uint64_t)tid * tiles + blockIdx.x];
  }
  uint32_t inc = total;
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += o;
  }
  if (lane == 31) warpSum[warp] = inc;
  __syncthreads();
  uint32_t at = inc - total + earlier;
  for (int w = 0; w < warp; ++w) at += warpSum[w];
  for (int w = 0; w < kRadixWarps; ++w) {
    const uint32_t c = place[w][tid];
    place[w][tid] = at;
    at += c;
  }
  __syncthreads();
  for (int r = 0; r < kPer; r += 32) {
    const uint64_t k = w0 + r + lane;
    const bool live = k < n;
    const uint32_t digit = live ? d.at(k) : 256u;
    const uint32_t same = __match_any_sync(0xffffffffu, digit);
    if (live) {
      const uint32_t to = place[warp][digit] + __popc(same & ((1u << lane) - 1u));
      keysOut[to] = d.keys[k];
      idxOut[to] = d.idx[k];
    }
    __syncwarp();
    if (live && lane == __ffs(same) - 1) place[warp][digit] += __popc(same);
    __syncwarp();
  }
}

// DOF idx[k] gets number k + 1, k < count (Unknown DOFs, then bubbles)
__global__ void k_number(const uint32_t *__restrict__ idx, uint64_t n, const uint8_t *__restrict__ cls, uint64_t *__restrict__ num) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n && cls[idx[k]] < 2) num[idx[k]] = k + 1;
}

// Stable Hilbert order of n points (float [n][stride], in host memory) in the
// box [mn, mx]: into perm; or, with the assemble types, the numbers of the
// DOFs, `sorted` of which get one, into num.
// One block up to kBlockSort items: 25 DOFs 149 us a call and 281 by the radix
// sort of 4,096-item tiles, 5,101 DOFs to number among 10,201 234 and 427; at
// 9,000 points, 16,384 places of the network, it would be past the radix
// sort, which took 263 there by small tiles and 390 by large ones. Those are
// worth it up to kRadixSmall (60,000 points 318 and 405), beyond which the sum
// over the tiles' counts in every block grows too long.
static int hilbertOrderGpu(int dim, uint64_t n, const float *pts, int stride, const float *mn, const float *mx, uint32_t *perm,
                           const int32_t *type, uint64_t *num, uint64_t sorted) {
  if (n == 0) return FG_OK;
  // scale as the host sort computes it (float)
  const unsigned nbrBits = 64 / dim;
  const unsigned twoPow = 1u << (nbrBits - 1);
  float sc[3] = {0, 0, 0}, sm[3] = {0, 0, 0};
  for (int i = 0; i < dim; ++i) {
    sc[i] = (float)twoPow / (mx[i] - mn[i]);
    sm[i] = -mn[i] * sc[i];
  }
  HilbertDev tab;
  hilbertTableData(dim, &tab.code[0][0], &tab.next[0][0]);
  const bool small = n <= kRadixSmall;
  const uint32_t tile = small ? kRadixTileSmall : kRadixTile, tiles = (uint32_t)((n + tile - 1) / tile);
  size_t bytes = 0;
  auto part = [&](size_t b) {
    const size_t at = bytes;
    bytes += (b + 255) / 256 * 256;
    return at;
  };
  const size_t oPts = part(n * stride * sizeof(float)), oType = part(type ? n * 4 : 0), oCls = part(type ? n : 0),
               oNum = part(type ? n * 8 : 0), oK0 = part(n * 8), oK1 = part(n * 8), oI0 = part(n * 4), oI1 = part(n * 4),
               oHist = part((size_t)256 * tiles * 4), oTotals = part(256 * 4), oCount = part(4);
  const bool oneBlock = sorted <= kBlockSort && n <= (uint64_t(1) << 30);
  uint8_t *base = nullptr;
  if (cudaMalloc(&base, bytes) != cudaSuccess) {
    cudaGetLastError();
    setLastError("hilbert order: device allocation failed");
    return FG_ERR_OOM;
  }
  uint64_t *keys[2] = {(uint64_t *)(base + oK0), (uint64_t *)(base + oK1)};
  uint32_t *idx[2] = {(uint32_t *)(base + oI0), (uint32_t *)(base + oI1)};
  uint32_t *hist = (uint32_t *)(base + oHist), *totals = (uint32_t *)(base + oTotals);
  uint8_t *cls = type ? base + oCls : nullptr;
  auto run = [&]() -> cudaError_t {
    cudaError_t e = cudaMemcpyAsync(base + oPts, pts, n * stride * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && type) e = cudaMemcpyAsync(base + oType, type, n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && type) e = cudaMemcpyAsync(base + oNum, num, n * 8, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return e;
    const unsigned nb = (unsigned)((n + 255) / 256);
    uint32_t *count = oneBlock ? (uint32_t *)(base + oCount) : nullptr;
    if (count && (e = cudaMemsetAsync(count, 0, 4)) != cudaSuccess) return e;
    k_hilbert_keys<<<nb, 256>>>(dim, n, (const float *)(base + oPts), stride, make_float3(sc[0], sc[1], sc[2]),
                                make_float3(sm[0], sm[1], sm[2]), tab, keys[0], idx[0], (const int32_t *)(base + oType), cls, count);
    if (oneBlock) {
      uint32_t padded = 64;
      while (padded < sorted) padded <<= 1;
      const size_t smem = (size_t)(padded + padded / 16) * 12;
      static SmemAllowance allowed;
      if ((e = allowSmem(k_sort_block, smem, allowed)) != cudaSuccess) return e;
      k_sort_block<<<1, std::min(1024u, padded / 2), smem>>>(keys[0], idx[0], (uint32_t)sorted, padded, type ? nullptr : idx[1],
                                                            (uint64_t *)(base + oNum));
      countLaunch(2);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      return type ? cudaMemcpy(num, base + oNum, n * 8, cudaMemcpyDeviceToHost) : cudaMemcpy(perm, idx[1], n * 4, cudaMemcpyDeviceToHost);
    }
    const int passes = 8 + (type ? 1 : 0);
    for (int q = 0; q < passes; ++q) {
      const int a = q & 1;
      const RadixDigit d = {keys[a], idx[a], q == 8 ? cls : nullptr, 8 * q};
      k_radix_count<<<tiles, kRadixThreads>>>(d, n, tile, tiles, hist);
      if (small) {
        k_radix_scatter<true><<<tiles, kRadixThreads>>>(d, n, tiles, hist, totals, keys[a ^ 1], idx[a ^ 1]);
      } else {
        k_radix_scan<<<256, kRadixThreads>>>(hist, tiles, totals);
        k_radix_scatter<false><<<tiles, kRadixThreads>>>(d, n, tiles, hist, totals, keys[a ^ 1], idx[a ^ 1]);
      }
    }
    const uint32_t *order = idx[passes & 1];
    if (type) k_number<<<nb, 256>>>(order, n, cls, (uint64_t *)(base + oNum));
    countLaunch(1 + (small ? 2 : 3) * passes + (type ? 1 : 0));
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return type ? cudaMemcpy(num, base + oNum, n * 8, cudaMemcpyDeviceToHost) : cudaMemcpy(perm, order, n * 4, cudaMemcpyDeviceToHost);
  };
  const cudaError_t e = run();
  cudaFree(base);
  if (e == cudaSuccess) return FG_OK;
  cudaGetLastError();
  setLastError(std::string("hilbert order: ") + cudaGetErrorString(e));
  return FG_ERR_CUDA;
}

}  // namespace femg

using namespace femg;

extern "C" int fg_hilbert_order(int32_t dim, uint64_t n, const float *pts, const float *mn, const float *mx, uint32_t *perm) {
  if ((dim != 2 && dim != 3) || (n > 0 && (!pts || !mn || !mx || !perm)) || n >= (uint64_t(1) << 32) - 1) {
    setLastError("fg_hilbert_order: invalid arguments");
    return FG_ERR_ARG;
  }
  int dev = 0;
  if (cudaGetDeviceCount(&dev) != cudaSuccess || dev == 0) {
    cudaGetLastError();
    setLastError("fg_hilbert_order: no CUDA device");
    return FG_ERR_NO_DEVICE;
  }
  return hilbertOrderGpu(dim, n, pts, dim, mn, mx, perm, nullptr, nullptr, n);
}

extern "C" int fg_hilbert_numbering(int32_t dim, const double *bbox, uint64_t n_dofs, const float *xyz, const int32_t *assemble_type,
                                    uint64_t *num_dof) {
  if ((dim != 2 && dim != 3) || !bbox || (n_dofs > 0 && (!xyz || !assemble_type || !num_dof))) {
    setLastError("fg_hilbert_numbering: invalid arguments");
    return FG_ERR_ARG;
  }
  // the DOFs that get a number, as far as it matters: without any, no device
  // is needed
  uint64_t nUnknown = 0;
  for (uint64_t i = 0; i < n_dofs && nUnknown <= kBlockSort; ++i)
    nUnknown += assemble_type[i] == FG_AT_UNKNOWN || assemble_type[i] == FG_AT_UNKNOWN_BUBBLE;
  if (nUnknown == 0) return FG_OK;
  // the box widened by a relative 1e-6, as the reference does (DofsManager.cpp)
  float mn[3], mx[3];
  for (int c = 0; c < dim; ++c) {
    mn[c] = (float)(bbox[c] - 0.000001 * std::fabs(bbox[c]));
    mx[c] = (float)(bbox[3 + c] + 0.000001 * std::fabs(bbox[3 + c]));
  }
  if (n_dofs >= (uint64_t(1) << 32) - 1) {
    setLastError("fg_hilbert_numbering: more than 2^32 - 2 DOFs");
    return FG_ERR_ARG;
  }
  int dev = 0;
  if (cudaGetDeviceCount(&dev) != cudaSuccess || dev == 0) {
    cudaGetLastError();
    setLastError("fg_hilbert_numbering: no CUDA device");
    return FG_ERR_NO_DEVICE;
  }
  return hilbertOrderGpu(dim, n_dofs, xyz, 3, mn, mx, nullptr, assemble_type, num_dof, nUnknown);
}
