// SpMV row classes and the stable radix sort used to transpose the operator.
#include "its_sparse.cuh"

namespace its {

// ---- row classes --------------------------------------------------------------------------
__host__ __device__ inline uint32_t rowClass(int64_t len) {
  for (int c = 0; c < kLongClass; ++c)
    if (len <= classMaxLen(c)) return (uint32_t)c;
  return kLongClass;
}
__global__ void kRowClass(int64_t n, const int64_t* __restrict__ rowptr, uint32_t* __restrict__ cls,
                          uint32_t* __restrict__ ids) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= n) return;
  cls[r] = rowClass(rowptr[r + 1] - rowptr[r]);
  ids[r] = (uint32_t)r;
}
// Class boundaries in the class-sorted list: entry i opens classes (cls[i-1], cls[i]].
__global__ void kClassBounds(int64_t n, const uint32_t* __restrict__ cls, int64_t* __restrict__ bounds) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i > n) return;
  const int64_t c = (i < n) ? (int64_t)cls[i] : kNumClasses;
  const int64_t prev = (i == 0) ? -1 : (int64_t)cls[i - 1];
  for (int64_t k = prev + 1; k <= c; ++k) bounds[k] = i;
}
__global__ void kSegCounts(int64_t nLong, const uint32_t* __restrict__ longRows, const int64_t* __restrict__ rowptr,
                           uint32_t* __restrict__ cnt) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= nLong) return;
  const int64_t l = rowptr[longRows[j] + 1] - rowptr[longRows[j]];
  cnt[j] = (uint32_t)((l + kSegLen - 1) / kSegLen);
}
// Long row j is cut into segments first[j] .. first[j+1]-1 of kSegLen entries each.
__global__ void kFillSegments(int64_t nLong, const uint32_t* __restrict__ longRows,
                              const uint32_t* __restrict__ first, const int64_t* __restrict__ rowptr,
                              uint32_t* __restrict__ segRow, int64_t* __restrict__ segBeg) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= nLong) return;
  const uint32_t row = longRows[j];
  const int64_t beg = rowptr[row];
  for (uint32_t s = first[j]; s < first[j + 1]; ++s) {
    segRow[s] = row;
    segBeg[s] = beg + (int64_t)(s - first[j]) * kSegLen;
  }
}

its_status buildSpmvPlan(its_ctx* ctx, int64_t n, const int64_t* rowptr, SpmvPlan* P) {
  *P = SpmvPlan();
  its_status st;
  DevBuf<uint32_t> cls, ids, sortedCls, tk, tv;
  DevBuf<int64_t> bounds;
  if ((st = cls.alloc(ctx, n)) != ITS_OK || (st = ids.alloc(ctx, n)) != ITS_OK ||
      (st = sortedCls.alloc(ctx, n)) != ITS_OK || (st = tk.alloc(ctx, n)) != ITS_OK ||
      (st = tv.alloc(ctx, n)) != ITS_OK || (st = bounds.alloc(ctx, kNumClasses + 1)) != ITS_OK)
    return st;
  if ((st = devAlloc(ctx, (void**)&P->rows, n * 4)) != ITS_OK) return st;
  kRowClass<<<gridFor(n, 256), 256, 0, ctx->stream>>>(n, rowptr, cls.p, ids.p);
  ITS_LAUNCHED(ctx);
  // one stable 8-bit pass groups the rows by class, ascending inside each class
  if ((st = radixSortPairs(ctx, cls.p, ids.p, sortedCls.p, P->rows, tk.p, tv.p, n, 3)) != ITS_OK) return st;
  kClassBounds<<<gridFor(n + 1, 256), 256, 0, ctx->stream>>>(n, sortedCls.p, bounds.p);
  ITS_LAUNCHED(ctx);
  int64_t hb[kNumClasses + 1];
  ITS_CU(ctx, cudaMemcpyAsync(hb, bounds.p, sizeof(hb), cudaMemcpyDeviceToHost, ctx->stream));
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  unsigned blk = 0;
  for (int c = 0; c < kNumClasses; ++c) {
    P->offset[c] = hb[c];
    P->count[c] = hb[c + 1] - hb[c];
    P->blockStart[c] = blk;
    if (c < kLongClass) {
      P->blocks[c] = (unsigned)((P->count[c] * classLanes(c) + kSpmvThreads - 1) / kSpmvThreads);
      blk += P->blocks[c];
    }
  }
  const int64_t nLong = P->nLong();
  if (nLong) {
    DevBuf<uint32_t> segCnt, tot;
    if ((st = segCnt.alloc(ctx, nLong)) != ITS_OK || (st = tot.alloc(ctx, 1)) != ITS_OK) return st;
    if ((st = devAlloc(ctx, (void**)&P->longFirstSeg, (nLong + 1) * 4)) != ITS_OK) return st;
    const uint32_t* longRows = P->rows + P->offset[kLongClass];
    kSegCounts<<<gridFor(nLong, 128), 128, 0, ctx->stream>>>(nLong, longRows, rowptr, segCnt.p);
    ITS_LAUNCHED(ctx);
    const uint32_t* sc = segCnt.p;
    auto fc = [sc] __device__(int64_t i) -> uint32_t { return sc[i]; };
    if ((st = scanExclusiveAlloc<uint32_t>(ctx, fc, nLong, StorePrefix<uint32_t>{P->longFirstSeg}, tot.p)) != ITS_OK)
      return st;
    ITS_CU(ctx, cudaMemcpyAsync(P->longFirstSeg + nLong, tot.p, 4, cudaMemcpyDeviceToDevice, ctx->stream));
    uint32_t nseg = 0;
    if ((st = readScalar(ctx, tot.p, &nseg)) != ITS_OK) return st;
    P->nSeg = nseg;
    if ((st = devAlloc(ctx, (void**)&P->segRow, nseg * 4)) != ITS_OK) return st;
    if ((st = devAlloc(ctx, (void**)&P->segBeg, nseg * 8)) != ITS_OK) return st;
    if ((st = devAlloc(ctx, (void**)&P->segPartial, nseg * 8)) != ITS_OK) return st;
    kFillSegments<<<gridFor(nLong, 128), 128, 0, ctx->stream>>>(nLong, longRows, P->longFirstSeg, rowptr, P->segRow,
                                                              P->segBeg);
    ITS_LAUNCHED(ctx);
  }
  P->blocks[kLongClass] = (unsigned)P->nSeg;
  P->blockStart[kLongClass] = blk;
  P->blockStart[kNumClasses] = blk + (unsigned)P->nSeg;
  return ITS_OK;
}

void releasePlan(its_ctx* ctx, SpmvPlan* P) {
  void* ptrs[] = {P->rows, P->longFirstSeg, P->segRow, P->segBeg, P->segPartial};
  for (void* p : ptrs) devFree(ctx, p);
  *P = SpmvPlan();
}

// ---- stable LSD radix sort (8-bit digits) ----------------------------------------------------
// Three launches per digit: a tile's digit counts (kRadixUpsweep), each digit's counts scanned over
// the tiles (kRadixScan, a block per digit), and the scatter (kRadixDownsweep). A tile is 256
// threads x ITEMS keys; a warp owns 32 x ITEMS consecutive ones and ranks them against its own
// counters, without the block, in (round, lane) order, which is their order in the input; the
// warps' counters are then added up per digit, and the tile is put in digit order in shared memory
// so that it leaves in runs. (Ranked round by round across the block, with four barriers a round,
// the scatter took 20 us for 196,681 pairs, in 48 tiles; 10^7 pairs take the same 64 us, bound by
// the 64-byte runs that go to 256 places.)
//
// The launches are dependent. A scatter ranks its keys while the counts are scanned: the keys were
// complete before the counting grid, which lets the scan start only after its own wait.
constexpr int kRsThreads = 256, kRsWarps = kRsThreads / 32;

template <int ITEMS>
__global__ void __launch_bounds__(kRsThreads) kRadixUpsweep(const uint32_t* keys, int64_t n, int shift, uint32_t* tileHist,
                                                            int64_t nb) {
  __shared__ uint32_t hist[kRsWarps / 2][256];  // a copy per warp pair: equal digits meet less often
  const int warp = threadIdx.x >> 5;
  for (int w = 0; w < kRsWarps / 2; ++w) hist[w][threadIdx.x] = 0;
  gridDependencyWait();
  gridDependents();
  const int64_t base = (int64_t)blockIdx.x * (kRsThreads * ITEMS) + threadIdx.x;
  uint32_t key[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int64_t i = base + j * kRsThreads;
    key[j] = i < n ? keys[i] : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if (base + j * kRsThreads < n) atomicAdd(&hist[warp >> 1][(key[j] >> shift) & 255u], 1u);
  __syncthreads();
  uint32_t c = 0;
#pragma unroll
  for (int w = 0; w < kRsWarps / 2; ++w) c += hist[w][threadIdx.x];
  tileHist[(int64_t)threadIdx.x * nb + blockIdx.x] = c;
}

// Block d: digit d's counts over the tiles, scanned in place; their total to totals[d].
__global__ void __launch_bounds__(kScanThreads) kRadixScan(uint32_t* tileHist, int64_t nb, uint32_t* totals) {
  uint32_t* row = tileHist + (int64_t)blockIdx.x * nb;
  uint32_t carry = 0;
  gridDependents();
  gridDependencyWait();
  for (int64_t i0 = 0; i0 < nb; i0 += kScanTile) {
    uint32_t v[kScanItems], s = 0;
    const int64_t at = i0 + (int64_t)threadIdx.x * kScanItems;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      v[k] = at + k < nb ? row[at + k] : 0u;
      s += v[k];
    }
    uint32_t total;
    uint32_t run = carry + blockExclusiveScan<uint32_t>(s, total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
      if (at + k < nb) {
        row[at + k] = run;
        run += v[k];
      }
    carry += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

template <int ITEMS>
__global__ void __launch_bounds__(kRsThreads, 6) kRadixDownsweep(const uint32_t* keys, const uint32_t* vals, int64_t n,
                                                              int shift, const uint32_t* tileOffsets, int64_t nb,
                                                              const uint32_t* totals, uint32_t* keysOut,
                                                              uint32_t* valsOut) {
  static_assert(kRsThreads == 256 && kScanThreads == 256, "a thread per digit");
  __shared__ uint32_t sKey[kRsThreads * ITEMS], sVal[kRsThreads * ITEMS];
  __shared__ uint32_t warpCnt[kRsWarps][256];
  __shared__ uint32_t sFirst[256];  // the digit's first place in the tile
  __shared__ uint32_t sDst[256];    // its first place in the output, less that
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t tile = (int64_t)blockIdx.x * (kRsThreads * ITEMS), mine = tile + warp * (32 * ITEMS) + lane;
  const int count = n - tile < kRsThreads * ITEMS ? (int)(n - tile) : kRsThreads * ITEMS;
  uint32_t key[ITEMS], rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const bool in = mine + 32 * j < n;
    key[j] = in ? __ldcg(keys + mine + 32 * j) : 0u;
  }
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) warpCnt[w][t] = 0;
  __syncthreads();
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    rank[j] = __match_any_sync(0xffffffffu, mine + 32 * j < n ? (key[j] >> shift) & 255u : 256u);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t digit = mine + 32 * j < n ? (key[j] >> shift) & 255u : 256u;
    const unsigned peers = rank[j];
    const uint32_t before = digit < 256u ? warpCnt[warp][digit] : 0u;
    rank[j] = before + __popc(peers & below);
    __syncwarp();
    if (digit < 256u && (peers & below) == 0u) warpCnt[warp][digit] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    uint32_t sum = 0, total;
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) {
      const uint32_t c = warpCnt[w][t];
      warpCnt[w][t] = sum;
      sum += c;
    }
    const uint32_t first = blockExclusiveScan<uint32_t>(sum, total);
    gridDependencyWait();
    gridDependents();
    const uint32_t global = blockExclusiveScan<uint32_t>(totals[t], total) + tileOffsets[(int64_t)t * nb + blockIdx.x];
    sFirst[t] = first;
    sDst[t] = global - first;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if (mine + 32 * j < n) {
      const uint32_t digit = (key[j] >> shift) & 255u, at = sFirst[digit] + warpCnt[warp][digit] + rank[j];
      sKey[at] = key[j];
      sVal[at] = vals ? vals[mine + 32 * j] : (uint32_t)(mine + 32 * j);
    }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int at = t + j * kRsThreads;
    if (at < count) {
      const uint32_t k = sKey[at], dst = sDst[(k >> shift) & 255u] + (uint32_t)at;
      keysOut[dst] = k;
      valsOut[dst] = sVal[at];
    }
  }
}

template <int ITEMS>
static its_status radixPass(its_ctx* ctx, const uint32_t* sk, const uint32_t* sv, uint32_t* dk, uint32_t* dv, int64_t n,
                            int shift, uint32_t* hist, int64_t nb) {
  uint32_t* totals = hist + 256 * nb;
  its_status st;
  // the first pass's keys may come from a copy
  if ((st = launchDependent(ctx, shift > 0, kRadixUpsweep<ITEMS>, (unsigned)nb, kRsThreads, 0, ctx->stream, sk, n, shift,
                            hist, nb)) != ITS_OK ||
      (st = launchDependent(ctx, true, kRadixScan, 256, kScanThreads, 0, ctx->stream, hist, nb, totals)) != ITS_OK)
    return st;
  return launchDependent(ctx, true, kRadixDownsweep<ITEMS>, (unsigned)nb, kRsThreads, 0, ctx->stream, sk, sv, n, shift,
                         (const uint32_t*)hist, nb, (const uint32_t*)totals, dk, dv);
}

its_status radixSortPairs(its_ctx* ctx, const uint32_t* keys, const uint32_t* vals, uint32_t* keysOut,
                          uint32_t* valsOut, uint32_t* tmpK, uint32_t* tmpV, int64_t n, int keyBits) {
  if (n <= 0) return ITS_OK;
  const int passes = keyBits <= 0 ? 1 : (keyBits + 7) / 8;
  // longer tiles leave in longer runs (10^7 pairs: 69 us a scatter with 4 per thread, 65 with 8, 66
  // with 16), short ones give every SM a block (196,681: 6.4 us with 4; 10^6: 12.5 and 12.6)
  const bool wide = n >= (1ll << 22);
  const int64_t per = (wide ? 8 : 4) * kRsThreads, nb = (n + per - 1) / per;
  its_status st;
  DevBuf<uint32_t> hist;
  if ((st = hist.alloc(ctx, 256 * nb + 256)) != ITS_OK) return st;
  const uint32_t* sk = keys;
  const uint32_t* sv = vals;
  for (int p = 0; p < passes; ++p) {
    const bool toOut = ((passes - p) & 1) == 1;
    uint32_t* dk = toOut ? keysOut : tmpK;
    uint32_t* dv = toOut ? valsOut : tmpV;
    st = wide ? radixPass<8>(ctx, sk, sv, dk, dv, n, 8 * p, hist.p, nb)
              : radixPass<4>(ctx, sk, sv, dk, dv, n, 8 * p, hist.p, nb);
    if (st != ITS_OK) return st;
    sk = dk;
    sv = dv;
  }
  return ITS_OK;
}

}  // namespace its
