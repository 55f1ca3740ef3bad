// GPU symbolic assembly of the CSR pattern of one element bucket.
//
// Replaces MatrixFactory::addPattern (src/system/MatrixFactory.cpp:459-539)
// and finalizePattern (:188-213) for a bucket whose test and unknown DOFs
// are the same field: row I (a test DOF of assemble type Unknown, Unknown
// bubble or Unknown global) holds the sorted, unique unknown DOFs of every
// element that has I; Fixed DOFs take no column; within one element the
// bubble rows after the first alias the first one (their pattern is its).
// Linked DOFs are rows and columns of their masters; a linked bubble's
// master is a bubble row of another element, whose bubble rows then share
// one pattern with the linked element's.
//
// No global sort: per element the row counts and the bubble aliases, per row
// its list of (element, local row) entries, then a warp per row gathers the
// candidate columns of its elements into shared memory, sorts them with a
// bitonic network and keeps the first of every run, once to count and once
// to write. The result does not depend on the order of the entries, so it
// is the reference's pattern bit for bit.
//
// The element DOF map is converted and checked on the device, and the row
// starts and row pointers come from device scans; the host reads five words
// and the two results. The columns go to plain host memory: page-locking 73 MB
// (9.2 M nonzeros) and giving it back took 4.7 ms of 7.0, and its pages are
// instead touched by all cores while the device writes the columns. 41,154
// order-3 tetrahedra: 2.0 ms a call.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <unordered_set>
#include <vector>

#include "common.cuh"

namespace femg {

constexpr uint32_t kPatNone = 0xFFFFFFFFu;

__device__ __forceinline__ bool patRow(uint8_t t) { return t == FG_AT_UNKNOWN || t == FG_AT_UNKNOWN_BUBBLE || t == FG_AT_UNKNOWN_GLOBAL; }

// What the host needs of the device's passes
struct PatInfo {
  unsigned long long total;  // of the last scan
  uint32_t maxCount;         // largest value scanned
  int bad;                   // an index out of range
  int linkedBubbles;         // some linked bubble
  int pad;
};

// The element DOF map as the passes below read it: rows' indices in 32 bits
// (0 for other types) and the assemble types in bytes. A linked DOF is a row
// and a column of its master (MatrixFactory.cpp:468-470, :481-483); a linked
// bubble is a bubble row of its master's (:505).
__global__ void k_pat_convert(const uint64_t *__restrict__ idx, const int32_t *__restrict__ type, int64_t count, uint64_t nRows,
                              const uint64_t *__restrict__ linkedRow, uint64_t nLinked, uint32_t *__restrict__ ed,
                              uint8_t *__restrict__ et, PatInfo *__restrict__ info) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  // an entry out of range is marked and takes no part in what follows
  et[k] = FG_AT_UNDEFINED;
  ed[k] = 0u;
  int t = type[k];
  uint64_t v = idx[k];
  if (t == FG_AT_LINKED || t == FG_AT_LINKED_BUBBLE) {
    if (!linkedRow || v >= nLinked) {
      atomicOr(&info->bad, 1);
      return;
    }
    v = linkedRow[v];
    if (t == FG_AT_LINKED_BUBBLE) atomicOr(&info->linkedBubbles, 1);
    t = t == FG_AT_LINKED ? FG_AT_UNKNOWN : FG_AT_UNKNOWN_BUBBLE;
  }
  const bool row = t == FG_AT_UNKNOWN || t == FG_AT_UNKNOWN_BUBBLE || t == FG_AT_UNKNOWN_GLOBAL;
  if (row && v >= nRows) {
    atomicOr(&info->bad, 1);
    return;
  }
  // (a value outside the enumeration is no row, whatever its low byte)
  et[k] = t >= FG_AT_UNDEFINED && t <= FG_AT_LINKED_BUBBLE ? (uint8_t)t : (uint8_t)FG_AT_UNDEFINED;
  if (row) ed[k] = (uint32_t)v;
}

// Exclusive scan of in[n] into out[n + 1] (64 bits), the total and the largest
// value into info: sums of tiles, a scan of those by one block, and the tiles.
constexpr int kScanThreads = 256, kScanTile = 2048;
__device__ __forceinline__ uint64_t blockExclusive(uint64_t v, uint64_t *total) {  // over kScanThreads threads
  __shared__ uint64_t warpSum[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t inc = v;
  for (int off = 1; off < 32; off <<= 1) {
    const uint64_t o = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += o;
  }
  __syncthreads();  // an earlier call's sums have been read
  if (lane == 31) warpSum[warp] = inc;
  __syncthreads();
  uint64_t before = 0, all = 0;
  for (int w = 0; w < kScanThreads / 32; ++w) {
    if (w < warp) before += warpSum[w];
    all += warpSum[w];
  }
  *total = all;
  return before + inc - v;
}
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const uint32_t *__restrict__ in, uint64_t n, uint64_t *__restrict__ sums,
                                                           PatInfo *__restrict__ info) {
  uint64_t sum = 0, all;
  uint32_t top = 0;
  for (uint64_t k = (uint64_t)blockIdx.x * kScanTile + threadIdx.x; k < min(n, ((uint64_t)blockIdx.x + 1) * kScanTile); k += kScanThreads) {
    sum += in[k];
    top = max(top, in[k]);
  }
  blockExclusive(sum, &all);
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && top) atomicMax(&info->maxCount, top);
  if (threadIdx.x == 0) sums[blockIdx.x] = all;
}
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(uint64_t *__restrict__ sums, uint64_t tiles, PatInfo *__restrict__ info) {
  uint64_t carry = 0;
  for (uint64_t b = 0; b < tiles; b += kScanThreads) {
    const uint64_t k = b + threadIdx.x;
    uint64_t all;
    const uint64_t ex = blockExclusive(k < tiles ? sums[k] : 0, &all);
    if (k < tiles) sums[k] = carry + ex;
    carry += all;
  }
  if (threadIdx.x == 0) info->total = carry;
}
__global__ void __launch_bounds__(kScanThreads) k_scan_write(const uint32_t *__restrict__ in, uint64_t n, const uint64_t *__restrict__ sums,
                                                            uint64_t *__restrict__ out) {
  constexpr int kPer = kScanTile / kScanThreads;  // consecutive values per thread
  const uint64_t k0 = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kPer;
  uint32_t v[kPer];
  uint64_t sum = 0, all;
  for (int i = 0; i < kPer; ++i) {
    v[i] = k0 + i < n ? in[k0 + i] : 0u;
    sum += v[i];
  }
  uint64_t at = sums[blockIdx.x] + blockExclusive(sum, &all);
  for (int i = 0; i < kPer; ++i) {
    if (k0 + i < n) out[k0 + i] = at;
    at += v[i];
    if (k0 + i + 1 == n) out[n] = at;
  }
}

// Row counts and bubble aliases, thread per element. preAliased: the
// aliases came from the host (linked bubbles: the bubble rows of a master
// element and of the element linked to it share one list), and an element's
// first bubble entry counts on the list's row.
__global__ void k_pat_count(const uint32_t *__restrict__ edof, const uint8_t *__restrict__ etype, int64_t E, int n,
                            uint32_t *__restrict__ cnt, uint32_t *__restrict__ alias, bool preAliased) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  uint32_t first = kPatNone;
  for (int i = 0; i < n; ++i) {
    const uint8_t t = etype[e * n + i];
    if (!patRow(t)) continue;
    uint32_t I = edof[e * n + i];
    if (t == FG_AT_UNKNOWN_BUBBLE) {
      if (first != kPatNone) {
        if (!preAliased) alias[I] = first;
        continue;
      }
      first = I;
      if (preAliased && alias[I] != kPatNone) I = alias[I];
    }
    atomicAdd(&cnt[I], 1u);
  }
}

// (element, local row) entries of every row, in any order
__global__ void k_pat_fill(const uint32_t *__restrict__ edof, const uint8_t *__restrict__ etype, int64_t E, int n,
                           const uint64_t *__restrict__ rowStart, uint32_t *__restrict__ fill, uint32_t *__restrict__ rowElem,
                           const uint32_t *__restrict__ alias, bool preAliased) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  bool seenBubble = false;
  for (int i = 0; i < n; ++i) {
    const uint8_t t = etype[e * n + i];
    if (!patRow(t)) continue;
    uint32_t I = edof[e * n + i];
    if (t == FG_AT_UNKNOWN_BUBBLE) {
      if (seenBubble) continue;
      seenBubble = true;
      if (preAliased && alias[I] != kPatNone) I = alias[I];
    }
    rowElem[rowStart[I] + atomicAdd(&fill[I], 1u)] = (uint32_t)(e << 6) | (uint32_t)i;
  }
}

// Warp per row: candidate columns of the row's elements, bitonic sort in
// shared memory, unique. WRITE == false: rowLen[I] = number of columns;
// WRITE == true: the columns into aj[ai[I]...].
template <bool WRITE>
__global__ void k_pat_rows(const uint32_t *__restrict__ edof, const uint8_t *__restrict__ etype, int n,
                           const uint64_t *__restrict__ rowStart, const uint32_t *__restrict__ rowElem,
                           const uint32_t *__restrict__ alias, uint64_t nRows, int cap, int upper, uint32_t *__restrict__ rowLen,
                           const uint64_t *__restrict__ ai, uint64_t *__restrict__ aj) {
  extern __shared__ uint32_t patBuf[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *buf = patBuf + (size_t)warp * cap;
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t row = (uint64_t)blockIdx.x * (blockDim.x >> 5) + warp; row < nRows; row += warps) {
    if (alias[row] != kPatNone) continue;  // an aliased bubble row: filled from its first bubble
    const uint64_t s0 = rowStart[row];
    const int cnt = (int)(rowStart[row + 1] - s0);
    const int m = cnt * n;
    int size = 1;
    while (size < m) size <<= 1;
    for (int k = lane; k < size; k += 32) {
      uint32_t v = kPatNone;
      if (k < m) {
        const uint32_t pk = rowElem[s0 + k / n];
        const int64_t e = pk >> 6;
        const int j = k % n;
        // upper storage keeps the columns at or right of the entry's own row:
        // the row itself, or for bubbles the row of the element's first bubble
        if (patRow(etype[e * n + j]) && (!upper || edof[e * n + j] >= edof[e * n + (pk & 63)])) v = edof[e * n + j];
      }
      buf[k] = v;
    }
    __syncwarp();
    for (int blk = 2; blk <= size; blk <<= 1)
      for (int str = blk >> 1; str > 0; str >>= 1) {
        for (int t = lane; t < (size >> 1); t += 32) {
          const int i = 2 * str * (t / str) + (t % str), j = i + str;
          const bool up = (i & blk) == 0;
          const uint32_t a = buf[i], b = buf[j];
          if ((a > b) == up) {
            buf[i] = b;
            buf[j] = a;
          }
        }
        __syncwarp();
      }
    // unique values in ascending order (kPatNone sorts last)
    uint32_t count = 0;
    for (int base = 0; base < size; base += 32) {
      const int k = base + lane;
      const uint32_t v = k < size ? buf[k] : kPatNone;
      const bool keep = v != kPatNone && (k == 0 || buf[k - 1] != v);
      const unsigned mask = __ballot_sync(0xffffffffu, keep);
      if (WRITE && keep) aj[ai[row] + count + __popc(mask & ((1u << lane) - 1u))] = v;
      count += __popc(mask);
    }
    if (!WRITE && lane == 0) rowLen[row] = count;
    __syncwarp();
  }
}

__global__ void k_pat_alias_len(const uint32_t *__restrict__ alias, uint64_t nRows, uint32_t *__restrict__ rowLen) {
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < nRows && alias[r] != kPatNone) rowLen[r] = rowLen[alias[r]];
}

__global__ void k_pat_alias_copy(const uint32_t *__restrict__ alias, uint64_t nRows, const uint64_t *__restrict__ ai,
                                 uint64_t *__restrict__ aj) {
  const uint64_t r = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= nRows || alias[r] == kPatNone) return;
  const uint64_t src = ai[alias[r]], len = ai[r + 1] - ai[r];
  for (uint64_t k = lane; k < len; k += 32) aj[ai[r] + k] = aj[src + k];
}

}  // namespace femg

using namespace femg;

namespace {

struct DevBuf {
  void *p = nullptr;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
};

int devAlloc(DevBuf &b, size_t bytes) {
  if (cudaMalloc(&b.p, std::max<size_t>(bytes, 16)) != cudaSuccess) {
    cudaGetLastError();
    setLastError("fg_pattern_build: device allocation of " + std::to_string(bytes) + " bytes failed");
    return FG_ERR_OOM;
  }
  return FG_OK;
}

int scanCounts(const uint32_t *in, uint64_t n, uint64_t *sums, uint64_t *out, PatInfo *info) {
  FG_CUDA(cudaMemsetAsync(&info->maxCount, 0, sizeof(uint32_t)));
  if (n == 0) {
    FG_CUDA(cudaMemsetAsync(&info->total, 0, sizeof(info->total)));
    FG_CUDA(cudaMemsetAsync(out, 0, sizeof(uint64_t)));
    return FG_OK;
  }
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  k_scan_sums<<<(unsigned)tiles, kScanThreads>>>(in, n, sums, info);
  k_scan_tiles<<<1, kScanThreads>>>(sums, tiles, info);
  k_scan_write<<<(unsigned)tiles, kScanThreads>>>(in, n, sums, out);
  countLaunch(3);
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}

// With linked bubbles, the rows that share one list: the reference's element
// after element pointer assignment (MatrixFactory.cpp:505-535) puts every
// bubble row of a master element and of the element linked to it on the list
// of whichever bubble row was taken first; connecting the bubble rows of each
// element gives the same groups in any element order. Each group's list is
// kept on its smallest row.
std::vector<uint32_t> bubbleAliases(const std::vector<uint32_t> &ed, const std::vector<uint8_t> &et, int64_t E, int n, uint64_t nRows) {
  std::vector<uint32_t> root(nRows);
  for (uint64_t r = 0; r < nRows; ++r) root[r] = (uint32_t)r;
  auto find = [&](uint32_t r) {
    while (root[r] != r) r = root[r] = root[root[r]];
    return r;
  };
  for (int64_t e = 0; e < E; ++e) {
    uint32_t first = kPatNone;
    for (int i = 0; i < n; ++i) {
      const size_t k = (size_t)e * n + i;
      if (et[k] != FG_AT_UNKNOWN_BUBBLE) continue;
      if (first == kPatNone) {
        first = ed[k];
        continue;
      }
      const uint32_t a = find(first), b = find(ed[k]);
      if (a != b) root[std::max(a, b)] = std::min(a, b);
    }
  }
  std::vector<uint32_t> al(nRows, kPatNone);
  for (uint64_t r = 0; r < nRows; ++r)
    if (find((uint32_t)r) != r) al[r] = find((uint32_t)r);
  return al;
}

// Plain host memory for the columns (freed by fg_host_free), its pages made
// present by all cores
void *hostColumns(size_t bytes) {
  constexpr size_t kHuge = size_t(2) << 20;
  void *p = nullptr;
  if (bytes < 2 * kHuge) return std::malloc(std::max<size_t>(bytes, 8));
  if (posix_memalign(&p, kHuge, bytes) != 0) return nullptr;
  madvise(p, bytes, MADV_HUGEPAGE);  // a hint
  const size_t page = (size_t)std::max<long>(sysconf(_SC_PAGESIZE), 4096);
  const int64_t pages = (int64_t)((bytes + page - 1) / page);
#pragma omp parallel for schedule(static)
  for (int64_t k = 0; k < pages; ++k) static_cast<volatile char *>(p)[(size_t)k * page] = 0;
  return p;
}

// The columns that callers hold: plain memory, which fg_host_free must not
// tell from its page-locked buffers by what CUDA says of the address, as a
// caller may have page-locked them since
std::mutex g_columnsMutex;
std::unordered_set<void *> g_columns;

}  // namespace

bool femg::freePatternColumns(void *ptr) {
  {
    std::lock_guard<std::mutex> lk(g_columnsMutex);
    if (g_columns.erase(ptr) == 0) return false;
  }
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, ptr) != cudaSuccess) cudaGetLastError();
  else if (a.type == cudaMemoryTypeHost && cudaHostUnregister(ptr) != cudaSuccess) cudaGetLastError();
  std::free(ptr);
  return true;
}

extern "C" int fg_pattern_build(const uint64_t *elem_dof_idx, const int32_t *elem_dof_type, int64_t n_elements, int32_t n_dofs,
                                uint64_t n_rows, uint64_t *ai, uint64_t **aj, int32_t upper, const uint64_t *linked_row,
                                uint64_t n_linked) {
  if (!ai || !aj || n_elements < 0 || n_dofs <= 0 || n_dofs > 64 || (n_elements > 0 && (!elem_dof_idx || !elem_dof_type))) {
    setLastError("fg_pattern_build: invalid arguments");
    return FG_ERR_ARG;
  }
  *aj = nullptr;
  if (n_rows >= (uint64_t(1) << 32) - 1 || n_elements >= (int64_t(1) << 26)) {
    setLastError("fg_pattern_build: more than 2^32 - 2 rows or 2^26 elements");
    return FG_ERR_UNSUPPORTED;
  }
  int dev = 0;
  if (cudaGetDeviceCount(&dev) != cudaSuccess || dev == 0) {
    cudaGetLastError();
    setLastError("fg_pattern_build: no CUDA device");
    return FG_ERR_NO_DEVICE;
  }
  const int n = n_dofs;
  const int64_t E = n_elements;
  const size_t en = (size_t)E * n;
  if (!linked_row) n_linked = 0;
  // one device allocation for everything whose size is known here
  const uint64_t scanTiles = (n_rows + kScanTile - 1) / kScanTile;
  size_t bytes = 0;
  auto part = [&](size_t b) {
    const size_t at = bytes;
    bytes += (b + 255) / 256 * 256;
    return at;
  };
  const size_t oInfo = part(sizeof(PatInfo)), oIdx = part(en * 8), oType = part(en * 4), oLinked = part(n_linked * 8), oEd = part(en * 4),
               oEt = part(en), oCnt = part(n_rows * 4), oFill = part(n_rows * 4), oAlias = part(n_rows * 4), oLen = part(n_rows * 4),
               oStart = part((n_rows + 1) * 8), oAi = part((n_rows + 1) * 8), oSums = part(scanTiles * 8);
  DevBuf arena, dElem, dAj;
  int st;
  if ((st = devAlloc(arena, bytes))) return st;
  uint8_t *base = (uint8_t *)arena.p;
  PatInfo *info = (PatInfo *)(base + oInfo);
  uint32_t *ed = (uint32_t *)(base + oEd), *cnt = (uint32_t *)(base + oCnt), *fill = (uint32_t *)(base + oFill),
           *alias = (uint32_t *)(base + oAlias), *len = (uint32_t *)(base + oLen);
  uint8_t *et = base + oEt;
  uint64_t *rowStart = (uint64_t *)(base + oStart), *dai = (uint64_t *)(base + oAi), *sums = (uint64_t *)(base + oSums);
  PatInfo host;
  FG_CUDA(cudaMemsetAsync(info, 0, sizeof(PatInfo)));
  if (n_rows) {
    FG_CUDA(cudaMemsetAsync(cnt, 0, oAlias - oCnt));  // the counts and the fill positions
    FG_CUDA(cudaMemsetAsync(alias, 0xFF, n_rows * 4));
  }
  const unsigned eb = (unsigned)std::max<int64_t>(1, (E + 255) / 256);
  if (E > 0) {
    FG_CUDA(cudaMemcpyAsync(base + oIdx, elem_dof_idx, en * 8, cudaMemcpyHostToDevice));
    FG_CUDA(cudaMemcpyAsync(base + oType, elem_dof_type, en * 4, cudaMemcpyHostToDevice));
    if (n_linked) FG_CUDA(cudaMemcpyAsync(base + oLinked, linked_row, n_linked * 8, cudaMemcpyHostToDevice));
    k_pat_convert<<<(unsigned)((en + 255) / 256), 256>>>((const uint64_t *)(base + oIdx), (const int32_t *)(base + oType), (int64_t)en,
                                                         n_rows, n_linked ? (const uint64_t *)(base + oLinked) : nullptr, n_linked, ed,
                                                         et, info);
    countLaunch();
    FG_CUDA(cudaGetLastError());
  }
  bool preAliased = false;
  auto count = [&]() -> int {
    if (E > 0) {
      k_pat_count<<<eb, 256>>>(ed, et, E, n, cnt, alias, preAliased);
      countLaunch();
    }
    int s2 = scanCounts(cnt, n_rows, sums, rowStart, info);
    if (s2) return s2;
    FG_CUDA(cudaMemcpy(&host, info, sizeof(PatInfo), cudaMemcpyDeviceToHost));
    return FG_OK;
  };
  if ((st = count())) return st;
  if (host.bad) {
    setLastError("fg_pattern_build: a DOF index is not below n_rows (or a linked index not below n_linked)");
    return FG_ERR_INDEX;
  }
  if (host.linkedBubbles) {
    // rare: the groups on the host, and the counts again on the grouped rows
    std::vector<uint32_t> hEd(en);
    std::vector<uint8_t> hEt(en);
    FG_CUDA(cudaMemcpy(hEd.data(), ed, en * 4, cudaMemcpyDeviceToHost));
    FG_CUDA(cudaMemcpy(hEt.data(), et, en, cudaMemcpyDeviceToHost));
    const std::vector<uint32_t> al = bubbleAliases(hEd, hEt, E, n, n_rows);
    FG_CUDA(cudaMemcpy(alias, al.data(), n_rows * 4, cudaMemcpyHostToDevice));
    FG_CUDA(cudaMemsetAsync(cnt, 0, n_rows * 4));
    preAliased = true;
    if ((st = count())) return st;
  }
  if ((st = devAlloc(dElem, host.total * 4))) return st;
  if (E > 0) {
    k_pat_fill<<<eb, 256>>>(ed, et, E, n, rowStart, fill, (uint32_t *)dElem.p, alias, preAliased);
    countLaunch();
  }
  // shared memory per warp: the largest candidate list, rounded to a power of two
  int cap = 1;
  while ((uint64_t)cap < (uint64_t)host.maxCount * n) cap <<= 1;
  int wpb = 8;
  while (wpb > 1 && (size_t)cap * 4 * wpb > 96 * 1024) wpb >>= 1;
  const size_t smem = (size_t)cap * 4 * wpb;
  if (smem > 200 * 1024) {
    setLastError("fg_pattern_build: a row gathers more candidate columns than shared memory holds");
    return FG_ERR_UNSUPPORTED;
  }
  FG_CUDA(cudaFuncSetAttribute(k_pat_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  FG_CUDA(cudaFuncSetAttribute(k_pat_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const unsigned rb = (unsigned)std::min<uint64_t>(std::max<uint64_t>(1, (n_rows + wpb - 1) / wpb), (uint64_t)smCount() * 64);
  if (n_rows > 0) {
    k_pat_rows<false><<<rb, 32 * wpb, smem>>>(ed, et, n, rowStart, (const uint32_t *)dElem.p, alias, n_rows, cap, upper ? 1 : 0, len,
                                               nullptr, nullptr);
    k_pat_alias_len<<<(unsigned)((n_rows + 255) / 256), 256>>>(alias, n_rows, len);
    countLaunch(2);
    FG_CUDA(cudaGetLastError());
  }
  if ((st = scanCounts(len, n_rows, sums, dai, info))) return st;
  FG_CUDA(cudaMemcpy(&host, info, sizeof(PatInfo), cudaMemcpyDeviceToHost));
  const uint64_t nnz = host.total;
  if ((st = devAlloc(dAj, nnz * 8))) return st;
  if (n_rows > 0) {
    k_pat_rows<true><<<rb, 32 * wpb, smem>>>(ed, et, n, rowStart, (const uint32_t *)dElem.p, alias, n_rows, cap, upper ? 1 : 0, len, dai,
                                              (uint64_t *)dAj.p);
    k_pat_alias_copy<<<(unsigned)((n_rows + 7) / 8), 256>>>(alias, n_rows, dai, (uint64_t *)dAj.p);
    countLaunch(2);
    FG_CUDA(cudaGetLastError());
  }
  void *out = hostColumns(nnz * 8);  // while the device writes the columns
  if (!out) {
    setLastError("fg_pattern_build: host allocation failed");
    return FG_ERR_OOM;
  }
  if (cudaMemcpy(ai, dai, (n_rows + 1) * 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(out, dAj.p, nnz * 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
    cudaGetLastError();
    std::free(out);
    setLastError("fg_pattern_build: copy of the pattern failed");
    return FG_ERR_CUDA;
  }
  {
    std::lock_guard<std::mutex> lk(g_columnsMutex);
    g_columns.insert(out);
  }
  *aj = (uint64_t *)out;
  return FG_OK;
}
