// Tables of segments (one per octree, or per octree and band) for kernels that work on many octrees
// in one launch.
#pragma once
#include <cstring>
#include <vector>

#include "its_ctx.cuh"

namespace its {

// A segment table and its prefix. Up to kInlineSegs segments travel with the launch as a
// kernel parameter (no copy, nothing to wait for); a larger table is copied to the device once
// (from pageable memory, staged at the call) into keep, which the caller holds until the
// launches are queued.
constexpr int kInlineSegs = 16;
template <class Seg>
struct SegArgs {
  int nseg = 0;
  const Seg* dsegs = nullptr;
  const int64_t* dprefix = nullptr;
  unsigned long long* stamp = nullptr;  // when set: the device clock (ns) at the kernel's start
  Seg segs[kInlineSegs];
  int64_t prefix[kInlineSegs + 1];
  __device__ __forceinline__ const Seg& seg(int k) const { return dsegs ? dsegs[k] : segs[k]; }
  __device__ __forceinline__ int64_t pre(int k) const { return dsegs ? dprefix[k] : prefix[k]; }
  // last segment whose first item is <= i
  __device__ __forceinline__ int find(int64_t i) const {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pre(mid) <= i) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  }
};

template <class Seg>
its_status makeSegArgs(its_ctx* ctx, const std::vector<Seg>& segs, const std::vector<int64_t>& prefix,
                              SegArgs<Seg>& A, DevBuf<uint8_t>& keep) {
  A.nseg = (int)segs.size();
  if (A.nseg <= kInlineSegs) {
    for (int k = 0; k < A.nseg; ++k) {
      A.segs[k] = segs[k];
      A.prefix[k] = prefix[k];
    }
    A.prefix[A.nseg] = prefix[A.nseg];
    return ITS_OK;
  }
  const size_t a = segs.size() * sizeof(Seg), b = (segs.size() + 1) * sizeof(int64_t);
  std::vector<uint8_t> h(a + b);
  std::memcpy(h.data(), segs.data(), a);
  std::memcpy(h.data() + a, prefix.data(), b);
  its_status st;
  if ((st = keep.alloc(ctx, a + b)) != ITS_OK) return st;
  ITS_CU(ctx, cudaMemcpyAsync(keep.p, h.data(), a + b, cudaMemcpyHostToDevice, ctx->stream));
  A.dsegs = (const Seg*)keep.p;
  A.dprefix = (const int64_t*)(keep.p + a);
  return ITS_OK;
}

}  // namespace its
