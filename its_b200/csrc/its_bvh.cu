// Accelerated signed distance: a linear BVH over the triangles (Karras 2012: Morton codes of
// centroids, radix sort, binary radix tree, bottom-up boxes) answers
//   * the exact unsigned distance: nearest-first traversal with box lower bounds; a node is
//     skipped only when its box is farther than the best squared distance times (1 + 1e-12),
//     so the minimum is the same IEEE value the brute force finds (same per-triangle code);
//   * the sign from the fast winding number (Barill et al. 2018): a node farther than beta = 2
//     times its radius contributes the second-order expansion of its triangles' solid angles
//     about its area centroid (the area-weighted normal sum as a dipole, plus the tensor
//     M = sum_t an_t (c_t - c)^T), nearer nodes recurse, leaves add the exact solid angle.
//     libigl's signed_distance(FAST_WINDING_NUMBER), which the reference calls
//     (ThinShells.cpp:501), uses the same expansion order and accuracy scale; inside if w > 1/2.
#include <cmath>

#include "its_scan.cuh"
#include "its_sdf.cuh"
#include "its_sparse.cuh"
#include <vector>
#include <algorithm>

namespace its {

constexpr double kFwnBeta = 2.0;  // far-field test |q - c| > beta * r
constexpr int kBucket = 8;        // a subtree of at most this many triangles is one leaf of the wide tree

struct BvhDevice {
  int64_t nf = 0;
  int32_t* left = nullptr;   // internal nodes: child index; >= 0 internal, < 0 leaf -(k+1)
  int32_t* right = nullptr;
  int32_t* parent = nullptr; // 2F-1 entries: internal 0..F-2, leaves F-1..2F-2
  int32_t* range = nullptr;  // internal node i covers sorted leaves range[2i] .. range[2i+1]
  uint32_t* leafTri = nullptr;
  unsigned* flag = nullptr;
};

// What the walks read:
//   * WideNode, 256 bytes per wide node: up to eight subtrees of a binary node, each with its box
//     (FP32, rounded outward, so a distance to it is a lower bound of the exact box's) and its
//     code. The nearest-triangle walk reads one per visit, a lane per subtree, coalesced.
//   * FwnNode, one line per binary internal node: the fast winding number's expansion centre
//     (area-weighted centroid sum / area), squared radius (+inf for a node without area, which
//     the far-field test then never accepts), normal sum, the second-order tensor's trace,
//     diagonal and summed off-diagonal pairs (all that the expansion uses), and the children.
//   * the leaves' triangles in leaf order.
struct __align__(16) WideSlot {
  float lo[3], hi[3];
  int32_t code;    // a wide node's index, or the first leaf of a bucket
  int32_t leaves;  // 0: a wide node; 1..kBucket: a bucket of so many leaves; -1: empty
};
struct __align__(128) WideNode {
  WideSlot s[8];
};
static_assert(sizeof(WideNode) == 256, "eight slots of two 16-byte loads");
struct __align__(128) FwnNode {
  double c[3];
  double r2;
  double an[3];
  double tr;     // trace of M = sum_t an_t (c_t - c)^T about the node's centre c
  double dg[3];  // M's diagonal
  double of[3];  // M01 + M10, M02 + M20, M12 + M21
  int32_t child[2];
  int32_t pad[2];
};
static_assert(sizeof(FwnNode) == 128, "one line per node");
struct __align__(8) BoxF {  // a binary node's box, rounded outward
  float lo[3], hi[3];
};

// A subtree's sums on their way up: box, normal sum, area-weighted centroid sum, area, and
// sum over its triangles of an_t c_t^T (row-major).
struct NodeSums {
  double lo[3], hi[3], an[3], ac[3], area, sm[9];
};
constexpr int kSumWords = sizeof(NodeSums) / 8;
constexpr int kTriWords = 10;  // a leaf triangle's nine coordinates, padded to whole 16-byte loads

// Per block: the centroids' bounds, and the largest coordinate's size (its upper word: the exponent counts).
constexpr int kBoundWords = 7;
__global__ void kCentroidBounds(const double* __restrict__ V, const int32_t* __restrict__ F, int64_t nf,
                                double* __restrict__ partial) {
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
  int size = 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nf; t += (int64_t)gridDim.x * blockDim.x) {
    for (int a = 0; a < 3; ++a) {
      const double p0 = V[3 * F[3 * t] + a], p1 = V[3 * F[3 * t + 1] + a], p2 = V[3 * F[3 * t + 2] + a];
      const double c = (p0 + p1 + p2) / 3.0;
      mn[a] = fmin(mn[a], c);
      mx[a] = fmax(mx[a], c);
      size = max(size, max(__double2hiint(p0) & 0x7fffffff,
                           max(__double2hiint(p1) & 0x7fffffff, __double2hiint(p2) & 0x7fffffff)));
    }
  }
  for (int a = 0; a < 3; ++a)
    for (int o = 16; o > 0; o >>= 1) {
      mn[a] = fmin(mn[a], __shfl_down_sync(0xffffffffu, mn[a], o));
      mx[a] = fmax(mx[a], __shfl_down_sync(0xffffffffu, mx[a], o));
    }
  size = __reduce_max_sync(0xffffffffu, size);
  __shared__ double s[8][kBoundWords];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    for (int a = 0; a < 3; ++a) { s[w][a] = mn[a]; s[w][3 + a] = mx[a]; }
    s[w][6] = size;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
      for (int a = 0; a < 3; ++a) { mn[a] = fmin(mn[a], s[k][a]); mx[a] = fmax(mx[a], s[k][3 + a]); }
      size = max(size, (int)s[k][6]);
    }
    double* p = partial + kBoundWords * blockIdx.x;
    for (int a = 0; a < 3; ++a) { p[a] = mn[a]; p[3 + a] = mx[a]; }
    p[6] = size;
  }
}

__global__ void kMortonCodes(const double* __restrict__ V, const int32_t* __restrict__ F, int64_t nf, double3 lo,
                             double3 inv, uint32_t* __restrict__ codes, uint32_t* __restrict__ idx) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nf) return;
  const double c[3] = {(V[3 * F[3 * t]] + V[3 * F[3 * t + 1]] + V[3 * F[3 * t + 2]]) / 3.0,
                       (V[3 * F[3 * t] + 1] + V[3 * F[3 * t + 1] + 1] + V[3 * F[3 * t + 2] + 1]) / 3.0,
                       (V[3 * F[3 * t] + 2] + V[3 * F[3 * t + 1] + 2] + V[3 * F[3 * t + 2] + 2]) / 3.0};
  const double L[3] = {lo.x, lo.y, lo.z}, I[3] = {inv.x, inv.y, inv.z};
  uint32_t q[3];
  for (int a = 0; a < 3; ++a) {
    const double u = (c[a] - L[a]) * I[a];
    q[a] = (uint32_t)fmin(fmax(u * 1024.0, 0.0), 1023.0);
  }
  codes[t] = mortonEncode(q[0], q[1], q[2]);
  idx[t] = (uint32_t)t;
}

// Length of the common prefix of keys i and j (index bits break ties), -1 out of range.
__device__ inline int delta(const uint32_t* codes, int64_t n, int64_t i, int64_t j) {
  if (j < 0 || j >= n) return -1;
  const uint32_t a = codes[i], b = codes[j];
  if (a != b) return __clz(a ^ b);
  return 32 + __clzll((unsigned long long)(i ^ j));
}

__global__ void kBuildInternal(const uint32_t* __restrict__ codes, int64_t n, int32_t* __restrict__ left,
                               int32_t* __restrict__ right, int32_t* __restrict__ parent, int32_t* __restrict__ range) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int d = delta(codes, n, i, i + 1) - delta(codes, n, i, i - 1) >= 0 ? 1 : -1;
  const int dmin = delta(codes, n, i, i - d);
  int64_t lmax = 2;
  while (delta(codes, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int64_t l = 0;
  for (int64_t t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(codes, n, i, i + (l + t) * d) > dmin) l += t;
  const int64_t j = i + l * d;
  const int dnode = delta(codes, n, i, j);
  int64_t s = 0;
  for (int64_t t = (l + 1) >> 1;; t = (t + 1) >> 1) {
    if (delta(codes, n, i, i + (s + t) * d) > dnode) s += t;
    if (t == 1) break;
  }
  const int64_t g = i + s * d + (d < 0 ? d : 0);
  const int64_t lo = i < j ? i : j, hi = i < j ? j : i;
  const int32_t L = (lo == g) ? -(int32_t)(g + 1) : (int32_t)g;
  const int32_t R = (hi == g + 1) ? -(int32_t)(g + 2) : (int32_t)(g + 1);
  left[i] = L;
  right[i] = R;
  range[2 * i] = (int32_t)lo;
  range[2 * i + 1] = (int32_t)hi;
  parent[L < 0 ? (n - 1) + (-L - 1) : L] = (int32_t)i;
  parent[R < 0 ? (n - 1) + (-R - 1) : R] = (int32_t)i;
}

// The node's box times scale, a power of two, rounded outward.
__device__ __forceinline__ BoxF outwardBox(const NodeSums& S, double scale) {
  BoxF b;
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = __double2float_rd(__dmul_rd(S.lo[a], scale));
    b.hi[a] = __double2float_ru(__dmul_ru(S.hi[a], scale));
  }
  return b;
}
__device__ __forceinline__ void mergeSums(NodeSums& S, const NodeSums& O) {
  for (int a = 0; a < 3; ++a) {
    S.lo[a] = fmin(S.lo[a], O.lo[a]);
    S.hi[a] = fmax(S.hi[a], O.hi[a]);
    S.an[a] = S.an[a] + O.an[a];
    S.ac[a] = S.ac[a] + O.ac[a];
  }
  S.area = S.area + O.area;
  for (int e = 0; e < 9; ++e) S.sm[e] = S.sm[e] + O.sm[e];
}
__device__ __forceinline__ FwnNode fwnNode(const NodeSums& S, int32_t left, int32_t right) {
  FwnNode f;
  f.r2 = __longlong_as_double(0x7ff0000000000000ll);  // +inf: no far-field term without area
  for (int a = 0; a < 3; ++a) {
    f.an[a] = S.an[a];
    f.c[a] = S.area > 0.0 ? S.ac[a] / S.area : 0.0;
  }
  if (S.area > 0.0) {
    double r2 = 0.0;
    for (int a = 0; a < 3; ++a) {
      const double e = fmax(f.c[a] - S.lo[a], S.hi[a] - f.c[a]);
      r2 += e * e;
    }
    f.r2 = r2;
  }
  double m[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) m[3 * i + j] = S.sm[3 * i + j] - f.an[i] * f.c[j];
  f.tr = m[0] + m[4] + m[8];
  f.dg[0] = m[0];
  f.dg[1] = m[4];
  f.dg[2] = m[8];
  f.of[0] = m[1] + m[3];
  f.of[1] = m[2] + m[6];
  f.of[2] = m[5] + m[7];
  f.child[0] = left;
  f.child[1] = right;
  f.pad[0] = f.pad[1] = 0;
  return f;
}

// Leaf data, then climb: the second child to arrive at a node merges both and goes on. A block's
// leaves are consecutive, so a node whose range lies inside them is merged by the block's own
// threads, every node's sums in shared memory ([word][slot]: the leaves, then the inner nodes,
// whose indices lie in the block too, since Karras numbers a node by an end of its range). The
// tree's links come in beforehand, and the winding records are formed afterwards, a thread per
// node, so that a step of the climb is a merge and nothing else. The maximal subtrees of a block
// (a dozen of 128 leaves) are left for kClimbTop, their sums at their first leaf's place in raw
// and their node and first leaf listed in top. One thread per leaf climbing through global memory all the way, with
// the sums in arrays of their own and a packing pass over them, moved 0.9 GB and took 823 + 110
// us at 1,048,576 triangles; now 183 us and kClimbTop.
constexpr int kUpLeaves = 128;
__global__ void __launch_bounds__(kUpLeaves) kBottomUp(const double* __restrict__ V, const int32_t* __restrict__ F,
                                                       BvhDevice B, double scale, double* __restrict__ raw,
                                                       int2* __restrict__ top, unsigned* __restrict__ topCount,
                                                       BoxF* __restrict__ box, FwnNode* __restrict__ fwn,
                                                       double* __restrict__ tris) {
  __shared__ double sSum[kSumWords][2 * kUpLeaves];
  __shared__ unsigned sFlag[kUpLeaves];
  __shared__ int32_t sParent[2 * kUpLeaves], sLeft[kUpLeaves], sRight[kUpLeaves];
  __shared__ int2 sRange[kUpLeaves];
  __shared__ int sTops, sTopBase;
  const int64_t n = B.nf;
  const int64_t k0 = (int64_t)blockIdx.x * kUpLeaves;
  const int i = threadIdx.x;
  const int64_t k = k0 + i;
  const int64_t kEnd = k0 + kUpLeaves < n ? k0 + kUpLeaves : n;
  sFlag[i] = 0;
  if (i == 0) sTops = 0;
  sRange[i] = make_int2(-1, -1);
  if (k < n - 1) {
    sParent[kUpLeaves + i] = B.parent[k];
    sLeft[i] = B.left[k];
    sRight[i] = B.right[k];
    sRange[i] = ((const int2*)B.range)[k];
  }
  NodeSums S;
  const double* mine = (const double*)&S;
  if (k < n) {
    sParent[i] = B.parent[(n - 1) + k];
    const uint32_t t = B.leafTri[k];
    double p[3][3];
    for (int c = 0; c < 3; ++c) {
      const int64_t vi = F[3 * (int64_t)t + c];
      for (int a = 0; a < 3; ++a) p[c][a] = V[3 * vi + a];
    }
    double2* dst = (double2*)(tris + kTriWords * k);
    dst[0] = make_double2(p[0][0], p[0][1]);
    dst[1] = make_double2(p[0][2], p[1][0]);
    dst[2] = make_double2(p[1][1], p[1][2]);
    dst[3] = make_double2(p[2][0], p[2][1]);
    dst[4] = make_double2(p[2][2], 0.0);
    const double u[3] = {p[1][0] - p[0][0], p[1][1] - p[0][1], p[1][2] - p[0][2]};
    const double v[3] = {p[2][0] - p[0][0], p[2][1] - p[0][1], p[2][2] - p[0][2]};
    const double an[3] = {0.5 * (u[1] * v[2] - u[2] * v[1]), 0.5 * (u[2] * v[0] - u[0] * v[2]),
                          0.5 * (u[0] * v[1] - u[1] * v[0])};
    const double ar = sqrt(an[0] * an[0] + an[1] * an[1] + an[2] * an[2]);
    for (int a = 0; a < 3; ++a) {
      S.lo[a] = fmin(p[0][a], fmin(p[1][a], p[2][a]));
      S.hi[a] = fmax(p[0][a], fmax(p[1][a], p[2][a]));
      S.ac[a] = ar * (p[0][a] + p[1][a] + p[2][a]) / 3.0;
      S.an[a] = an[a];
    }
    for (int r = 0; r < 3; ++r)
      for (int j = 0; j < 3; ++j) S.sm[3 * r + j] = an[r] * ((p[0][j] + p[1][j] + p[2][j]) / 3.0);
    S.area = ar;
    box[(n - 1) + k] = outwardBox(S, scale);
  }
  __syncthreads();
  int place = -1;  // of the maximal subtree that this thread ends at
  int2 found = make_int2(0, 0);
  if (k < n) {
    int slot = i;
    int64_t first = k;
    while (true) {
      const int32_t par = sParent[slot];
      if (par < 0) break;  // the root
      const bool inside = par >= k0 && par < kEnd && sRange[par - k0].x >= k0 && sRange[par - k0].y < kEnd;
      if (!inside) {
        double* dst = raw + kSumWords * first;
#pragma unroll
        for (int w = 0; w < kSumWords; ++w) dst[w] = mine[w];
        place = atomicAdd(&sTops, 1);
        found = make_int2((int32_t)(slot < kUpLeaves ? (n - 1) + k0 + slot : k0 + slot - kUpLeaves), (int32_t)first);
        break;
      }
      const int pi = (int)(par - k0);
      if (slot < kUpLeaves) {  // an inner node's sums went in when it was merged
#pragma unroll
        for (int w = 0; w < kSumWords; ++w) sSum[w][slot] = mine[w];
      }
      __threadfence_block();
      if (atomicAdd(&sFlag[pi], 1u) == 0) break;  // first arrival: the sibling merges
      __threadfence_block();
      const int32_t l = sLeft[pi], r = sRight[pi];
      const int ls = l < 0 ? (int)(-(int64_t)l - 1 - k0) : (int)(l - k0) + kUpLeaves;
      const int rs = r < 0 ? (int)(-(int64_t)r - 1 - k0) : (int)(r - k0) + kUpLeaves;
      const int os = ls == slot ? rs : ls;
      NodeSums O;
      double* other = (double*)&O;
#pragma unroll
      for (int w = 0; w < kSumWords; ++w) other[w] = ((volatile double*)sSum[w])[os];
      mergeSums(S, O);
      slot = kUpLeaves + pi;
      first = sRange[pi].x;
#pragma unroll
      for (int w = 0; w < kSumWords; ++w) sSum[w][slot] = mine[w];
    }
  }
  __syncthreads();
  if (i == 0 && sTops) sTopBase = (int)atomicAdd(topCount, (unsigned)sTops);
  if (sRange[i].x >= k0 && sRange[i].y < kEnd) {
    NodeSums N;
    double* to = (double*)&N;
#pragma unroll
    for (int w = 0; w < kSumWords; ++w) to[w] = sSum[w][kUpLeaves + i];
    box[k] = outwardBox(N, scale);
    fwn[k] = fwnNode(N, sLeft[i], sRight[i]);
  }
  __syncthreads();
  if (place >= 0) top[sTopBase + place] = found;
}

// The nodes above the blocks' maximal subtrees, a thread per subtree: the first arrival's sums
// wait at its first leaf's place; a node's place is its left child's, whose sums the merging
// thread has read by then. A chain of global round trips, one node after another: a node's links
// come in while the sums before it go out (131 -> 108 us at 1,048,576 triangles).
__global__ void __launch_bounds__(128) kClimbTop(BvhDevice B, double scale, double* __restrict__ raw,
                                                 const int2* __restrict__ top,
                                                 const unsigned* __restrict__ topCount, BoxF* __restrict__ box,
                                                 FwnNode* __restrict__ fwn) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= *topCount) return;
  int64_t first = top[k].y;
  NodeSums S;
  double* mine = (double*)&S;
#pragma unroll
  for (int w = 0; w < kSumWords; ++w) mine[w] = raw[kSumWords * first + w];
  int32_t par = B.parent[top[k].x];
  while (par >= 0) {
    const int32_t r0 = B.range[2 * (int64_t)par], l = B.left[par], r = B.right[par], above = B.parent[par];
    __threadfence();
    if (atomicAdd(B.flag + par, 1u) == 0) return;  // first arrival: the sibling merges
    __threadfence();
    const int64_t rFirst = r < 0 ? -(int64_t)r - 1 : r;  // a right child's number is its first leaf's
    const volatile double* src = raw + kSumWords * (first == r0 ? rFirst : (int64_t)r0);
    NodeSums O;
    double* other = (double*)&O;
#pragma unroll
    for (int w = 0; w < kSumWords; ++w) other[w] = src[w];
    mergeSums(S, O);
    first = r0;
    volatile double* dst = raw + kSumWords * first;
#pragma unroll
    for (int w = 0; w < kSumWords; ++w) dst[w] = mine[w];
    box[par] = outwardBox(S, scale);
    fwn[par] = fwnNode(S, l, r);
    par = above;
  }
}

// The wide tree: for every binary node of more than kBucket leaves (and the root) its subtrees
// three levels down, where a subtree of at most kBucket leaves stays one slot; slots that stay
// free are filled by opening further subtrees. A wide node's index is its binary node's, and
// only those met from the root are ever read (a few per cent of 10^6 triangles' nodes: 8 MB).
__global__ void __launch_bounds__(128) kWideNodes(BvhDevice B, const BoxF* __restrict__ box,
                                                  WideNode* __restrict__ wide) {
  const int64_t n = B.nf;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (n > 1 ? n - 1 : 1)) return;
  auto leavesOf = [&](int32_t c) { return c < 0 ? 1 : B.range[2 * (int64_t)c + 1] - B.range[2 * (int64_t)c] + 1; };
  if (i > 0 && leavesOf((int32_t)i) <= kBucket) return;
  int32_t slot[8];
  int cnt[8];
  int k = 0;
  if (n == 1) {
    slot[0] = -1;
    cnt[0] = 1;
    k = 1;
  } else {
    slot[0] = B.left[i];
    slot[1] = B.right[i];
    cnt[0] = leavesOf(slot[0]);
    cnt[1] = leavesOf(slot[1]);
    k = 2;
    for (bool more = true; more && k < 8;) {
      more = false;
      const int have = k;
      for (int j = 0; j < have && k < 8; ++j) {
        if (cnt[j] <= kBucket) continue;
        const int32_t c = slot[j];
        slot[j] = B.left[c];
        cnt[j] = leavesOf(slot[j]);
        slot[k] = B.right[c];
        cnt[k] = leavesOf(slot[k]);
        ++k;
        more = true;
      }
    }
  }
  for (int j = 0; j < 8; ++j) {
    WideSlot w;
    for (int a = 0; a < 3; ++a) w.lo[a] = w.hi[a] = 0.0f;
    w.code = 0;
    w.leaves = -1;
    if (j < k) {
      const int32_t c = slot[j];
      const BoxF b = box[c < 0 ? (n - 1) + (-(int64_t)c - 1) : c];
      for (int a = 0; a < 3; ++a) {
        w.lo[a] = b.lo[a];
        w.hi[a] = b.hi[a];
      }
      const bool bucket = cnt[j] <= kBucket;
      w.code = bucket ? (c < 0 ? -c - 1 : B.range[2 * (int64_t)c]) : c;
      w.leaves = bucket ? cnt[j] : 0;
    }
    float4* dst = (float4*)&wide[i].s[j];
    dst[0] = ((const float4*)&w)[0];
    dst[1] = ((const float4*)&w)[1];
  }
}

// ---- the walks: eight lanes per query ------------------------------------------------------
// A warp walks four queries at a time, eight lanes each, in the Morton order of their positions:
// a group that has finished takes the next query from a counter while the others go on (queries
// differ tenfold in their visits: far from the surface many boxes are about equally near). A
// thread per query kept 7.6 of 32 lanes busy and waited on its dependent node loads: 7.57 ms at
// 196,681 queries against 1,048,576 triangles. A fixed run of 16 queries per warp left the SMs
// idle for 38 % of the nearest walk, waiting for the runs with many far queries.
constexpr int kWalkThreads = 128, kGroups = kWalkThreads / 8;
// The tree's keys are 30 bits of position and an index: at most 62 binary levels. A wide node
// spans at least three of them and leaves seven others on the stack. The winding walk takes eight
// nodes at a time (each may leave two) while its stack is short, else one at a time with none on
// their way, which adds at most one entry per level (short below 32, 64, 128, 256 or 400 entries,
// without the second buffer: 5.8, 4.6, 4.6, 5.0, 5.5 ms for the call: a longer stack takes shared
// memory from the L1 and the resident blocks). When it stops being short it has at most 72
// entries, and eight nodes on their way leave 16 more.
constexpr int kTreeLevels = 62, kNearStack = 7 * ((kTreeLevels + 2) / 3) + 8;
constexpr int kLeafRing = 32;  // leaves waiting in the winding walk, at most 23
constexpr int kWideFwn = 64, kFwnStack = kWideFwn + 24 + kTreeLevels + 2;

// The next query of each of the warp's groups that needs one, or -1.
__device__ __forceinline__ int64_t takeQuery(bool need, int lane, int64_t m, unsigned long long* counter) {
  const unsigned b = __ballot_sync(0xffffffffu, need && (lane & 7) == 0);
  if (!b) return -1;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(counter, (unsigned long long)__popc(b));
  base = __shfl_sync(0xffffffffu, base, 0);
  const int64_t q = (int64_t)base + __popc(b & ((1u << (lane & 24)) - 1u));
  return need && q < m ? q : -1;
}
// A leaf triangle.
__device__ __forceinline__ void loadTri(const double* __restrict__ tris, int64_t leaf, D3& a, D3& b, D3& c) {
  const double2* v = (const double2*)(tris + kTriWords * leaf);
  const double2 v0 = __ldg(v), v1 = __ldg(v + 1), v2 = __ldg(v + 2), v3 = __ldg(v + 3), v4 = __ldg(v + 4);
  a = D3{v0.x, v0.y, v1.x};
  b = D3{v1.y, v2.x, v2.y};
  c = D3{v3.x, v3.y, v4.x};
}

__device__ __forceinline__ double groupMin(double v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double groupSum(double v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Exact unsigned distance, nearest subtree first. A subtree is left out only when the lower
// bound of its box's squared distance (FP32, every operation rounded down) is beyond the best
// squared distance times (1 + 1e-12), so the minimum is the IEEE value the brute force finds.
// A bucket's triangles are tested together, one per lane.
//
// kScaled: boxes, queries and bounds times the power of two that brings the mesh's largest coordinate to
// 1/2 .. 1, where the squares stay within FP32's range. Unscaled, a mesh at 2^-80 or 2^80 had every bound
// 0 or infinite and every triangle tested (200,000 faces and points: 508 and 520 ms, scaled 3.1, as at
// scale 1). A kernel of its own: on ordinary meshes the multiplications cost 1 % of the call.
template <bool kScaled>
__global__ void __launch_bounds__(kWalkThreads, 6) kNearest(const double* __restrict__ P, int64_t m,
                                                         const uint32_t* __restrict__ order,
                                                         const WideNode* __restrict__ wide,
                                                         const double* __restrict__ tris, double scale, double slack,
                                                         double* __restrict__ out,
                                                         unsigned long long* __restrict__ counter) {
  __shared__ int2 sStack[kGroups][kNearStack];  // wide node, lower bound
  const int lane = threadIdx.x & 31, j = lane & 7, shift = lane & 24;
  int2* stack = sStack[threadIdx.x >> 3];
  int64_t qi = -1;
  bool drained = false;  // no query is left for this group
  gridDependents();
  D3 q{0, 0, 0};
  float qlo[3] = {0, 0, 0}, qhi[3] = {0, 0, 0};
  double best = 0.0;
  float bound = 0.0f;
  int sp = 0;
  while (true) {
    const int64_t got = takeQuery(qi < 0 && !drained, lane, m, counter);
    drained = drained || (qi < 0 && got < 0);
    if (got >= 0) {
      qi = order[got];
      q = D3{P[3 * qi], P[3 * qi + 1], P[3 * qi + 2]};
      const double x[3] = {q.x, q.y, q.z};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        qlo[a] = __double2float_rd(kScaled ? __dmul_rd(x[a], scale) : x[a]);
        qhi[a] = __double2float_ru(kScaled ? __dmul_ru(x[a], scale) : x[a]);
      }
      best = 1.7976931348623157e308;
      bound = __int_as_float(0x7f800000);
      if (j == 0) stack[0] = make_int2(0, 0);
      sp = 1;
    }
    if (!__any_sync(0xffffffffu, qi >= 0)) break;
    __syncwarp();
    // the topmost of the upper eight entries that is still within the bound
    int2 e = make_int2(0, 0);
    bool live = false;
    if (j < sp) {
      e = stack[sp - 1 - j];
      live = __int_as_float(e.y) <= bound;
    }
    const unsigned lv = (__ballot_sync(0xffffffffu, live) >> shift) & 0xffu;
    const int pick = lv ? __ffs(lv) - 1 : 7;
    const int node = __shfl_sync(0xffffffffu, e.x, pick, 8);
    sp = sp > pick + 1 ? sp - pick - 1 : 0;
    float d = 0.0f;
    WideSlot w;
    w.leaves = -1;
    if (lv) {
      const float4* src = (const float4*)&wide[node].s[j];
      ((float4*)&w)[0] = __ldg(src);
      ((float4*)&w)[1] = __ldg(src + 1);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float g = fmaxf(fmaxf(__fsub_rd(w.lo[a], qhi[a]), __fsub_rd(qlo[a], w.hi[a])), 0.0f);
        d = __fadd_rd(d, __fmul_rd(g, g));
      }
    }
    // buckets, the lowest slot first
    unsigned lf = (__ballot_sync(0xffffffffu, w.leaves > 0 && d <= bound) >> shift) & 0xffu;
    while (__any_sync(0xffffffffu, lf != 0)) {
      const int src = lf ? __ffs(lf) - 1 : 0;
      lf &= lf - 1;
      const int first = __shfl_sync(0xffffffffu, w.code, src, 8), count = __shfl_sync(0xffffffffu, w.leaves, src, 8);
      const float db = __shfl_sync(0xffffffffu, d, src, 8);
      const bool mine = qi >= 0 && count > 0 && j < count && db <= bound;
      double t2 = 1.7976931348623157e308;
      if (mine) {
        D3 a, b, c;
        loadTri(tris, (int64_t)first + j, a, b, c);
        t2 = fmin(t2, pointTriSqDist(q, a, b, c));
      }
      best = fmin(best, groupMin(t2));
      bound = __double2float_ru(kScaled ? __dmul_ru(best, slack) : best * (1.0 + 1e-12));
    }
    // wide nodes within the bound, the nearest on top
    const bool push = w.leaves == 0 && d <= bound;
    const unsigned pm = (__ballot_sync(0xffffffffu, push) >> shift) & 0xffu;
    int below = 0;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const float od = __shfl_sync(0xffffffffu, d, o, 8);
      below += ((pm >> o) & 1u) && (od > d || (od == d && o < j)) ? 1 : 0;
    }
    if (push) stack[sp + below] = make_int2(w.code, __float_as_int(d));
    sp += __popc(pm);
    __syncwarp();
    if (qi >= 0 && sp == 0) {
      if (j == 0) out[qi] = sqrt(best);
      qi = -1;
    }
  }
}

// Sixteen bytes from global to shared memory, without registers.
__device__ __forceinline__ void copyAsync16(void* to, const void* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}
__device__ __forceinline__ void copyAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All but the last N groups of this thread's copies are there.
template <int N>
__device__ __forceinline__ void copyAsyncWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The sign: the fast winding number's sum over the binary tree. A group takes up to eight nodes
// from the top of its stack, a lane each: a far node adds its expansion, a near one puts its
// inner children back on the stack and its leaves on a list, whose exact solid angles are formed
// eight at a time. The nodes accepted and opened are those of a walk one node at a time; the sum
// is over lanes. When leaves are summed depends on the warp's other groups, which queries those hold on
// a counter; so a query's k-th leaf is lane k mod 8's, added in that order to a sum of its own, and the
// result is the same from call to call (a group that waited for eight of its own: 2,330 -> 2,390 us at
// 200,000 faces). A node costs about 65 FP64 operations, a query 414 nodes and 17 leaves at a tube of
// 1,048,576 faces; a far node's 1/R is rsqrt's, one rounding error like the square root and the
// reciprocal before (2.06 -> 2.01 ms). Walks shared by clusters of 8 to 32 neighbouring queries down to
// the nodes that they disagree on read a third of the records and were no faster (1.82 to 2.3 ms):
// too few walks are in flight, over too much of the tree.
//
// The next eight records are fetched (cp.async, a line of 128 bytes by eight lanes) before the
// current ones are looked at, from what the stack holds then: waiting for L2 was three fifths of the walk's time.
// The second buffer takes the sixth block of an SM. Signed distance at 196,518 points and 1,048,576
// faces: 4.02 -> 3.22 ms; at 200,000 and 20,000 faces 1.16 -> 0.99 ms and 518 -> 467 us.
//
// The distances are not read: this grid starts in the places that the nearest walk's blocks leave,
// whose last walks are long (23 % of its time with a chip partly idle), and writes a byte per
// query; kSigns puts the signs on. Signed distance at 196,518 corners: 4.51 -> 4.08 ms; at 2,000
// faces 560 -> 444 us.
__global__ void __launch_bounds__(kWalkThreads, 5) kWinding(const double* __restrict__ P, int64_t m,
                                                         const uint32_t* __restrict__ order,
                                                         const FwnNode* __restrict__ W, const double* __restrict__ tris,
                                                         int64_t n, uint8_t* __restrict__ inside,
                                                         unsigned long long* __restrict__ counter) {
  __shared__ int32_t sStack[kGroups][kFwnStack];
  __shared__ double2 sRec[2][kGroups][64];  // eight records, twice; piece p of record r at p ^ r
  __shared__ int32_t sLeaves[kGroups][kLeafRing];  // fewer than eight are left before sixteen more can come
  const int lane = threadIdx.x & 31, j = lane & 7, shift = lane & 24;
  const unsigned below = (1u << j) - 1u;
  int32_t* stack = sStack[threadIdx.x >> 3];
  int32_t* leaves = sLeaves[threadIdx.x >> 3];
  int64_t qi = -1;
  bool drained = false;  // no query is left for this group
  D3 q{0, 0, 0};
  double w = 0.0, wl = 0.0;  // the far nodes' sum, the leaves'
  int sp = 0, buf = 0;
  int first = 0, nl = 0;  // the query's first leaf in waiting, and how many wait
  int here = 0, coming = 0;  // records in this buffer, and on their way to the other
  while (true) {
    const int64_t got = takeQuery(qi < 0 && !drained, lane, m, counter);
    drained = drained || (qi < 0 && got < 0);
    if (got >= 0) {
      qi = order[got];
      q = D3{P[3 * qi], P[3 * qi + 1], P[3 * qi + 2]};
      w = wl = 0.0;
      sp = n > 1 ? 1 : 0;
      nl = n > 1 ? 0 : 1;
      first = 0;
      if (j == 0) {
        stack[0] = 0;
        leaves[0] = 0;
      }
    }
    if (!__any_sync(0xffffffffu, qi >= 0)) break;
    __syncwarp();
    // the next records set out before these are looked at
    coming = sp > kWideFwn ? (here ? 0 : 1) : (sp < 8 ? sp : 8);
    const int32_t node = j < coming ? stack[sp - coming + j] : 0;
    sp -= coming;
    double2* to = sRec[buf ^ 1][threadIdx.x >> 3];
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const int32_t no = __shfl_sync(0xffffffffu, node, o, 8);
      if (o < coming) copyAsync16(&to[8 * o + (j ^ o)], (const double2*)(W + no) + j);
    }
    copyAsyncCommit();
    copyAsyncWait<1>();
    __syncwarp();
    const double2* rec = sRec[buf][threadIdx.x >> 3];
    bool near = false;
    int32_t c0 = 0, c1 = 0;
    if (j < here) {
      FwnNode nd;
#pragma unroll
      for (int p = 0; p < 8; ++p) ((double2*)&nd)[p] = rec[8 * j + (p ^ j)];
      const double d[3] = {nd.c[0] - q.x, nd.c[1] - q.y, nd.c[2] - q.z};
      const double R2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
      if (R2 > kFwnBeta * kFwnBeta * nd.r2) {  // the powers of 1/R from one reciprocal
        const double iR = rsqrt(R2);
        const double iR2 = iR * iR, iR3 = iR2 * iR, iR5 = iR3 * iR2;
        const double dmd = nd.dg[0] * d[0] * d[0] + nd.dg[1] * d[1] * d[1] + nd.dg[2] * d[2] * d[2] +
                           nd.of[0] * d[0] * d[1] + nd.of[1] * d[0] * d[2] + nd.of[2] * d[1] * d[2];
        w += (nd.an[0] * d[0] + nd.an[1] * d[1] + nd.an[2] * d[2]) * iR3 + (nd.tr * iR3 - 3.0 * dmd * iR5);
      } else {
        near = true;
        c0 = nd.child[0];
        c1 = nd.child[1];
      }
    }
    here = coming;
    buf ^= 1;
    const unsigned i0 = (__ballot_sync(0xffffffffu, near && c0 >= 0) >> shift) & 0xffu;
    const unsigned i1 = (__ballot_sync(0xffffffffu, near && c1 >= 0) >> shift) & 0xffu;
    const unsigned l0 = (__ballot_sync(0xffffffffu, near && c0 < 0) >> shift) & 0xffu;
    const unsigned l1 = (__ballot_sync(0xffffffffu, near && c1 < 0) >> shift) & 0xffu;
    if (near) {
      int at = sp + __popc(i0 & below) + __popc(i1 & below);
      int al = first + nl + __popc(l0 & below) + __popc(l1 & below);
      if (c0 >= 0) stack[at++] = c0;
      else leaves[al++ & (kLeafRing - 1)] = -c0 - 1;
      if (c1 >= 0) stack[at] = c1;
      else leaves[al & (kLeafRing - 1)] = -c1 - 1;
    }
    sp += __popc(i0) + __popc(i1);
    nl += __popc(l0) + __popc(l1);
    __syncwarp();
    // solid angles, once some group has eight leaves or nothing else to do; the others' along
    while (__any_sync(0xffffffffu, nl >= 8 || (sp == 0 && here == 0 && nl > 0))) {
      const int t = nl < 8 ? nl : 8, mine = (j - first) & 7;
      if (mine < t) {
        D3 a, b, c;
        loadTri(tris, leaves[(first + mine) & (kLeafRing - 1)], a, b, c);
        wl += solidAngle(q, a, b, c);
      }
      nl -= t;
      first += t;
      __syncwarp();
    }
    const bool done = qi >= 0 && sp == 0 && here == 0;  // its leaves are summed by now
    if (!__any_sync(0xffffffffu, done)) continue;
    const double total = groupSum(done ? w + wl : 0.0);
    if (done) {
      if (j == 0) inside[qi] = total / (4.0 * 3.14159265358979323846) > 0.5;
      qi = -1;
    }
  }
  gridDependencyWait();  // this kernel ends after the distances are written
}

__global__ void kSigns(const uint8_t* __restrict__ inside, double* __restrict__ out, int64_t m) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < m && inside[i]) out[i] = -out[i];
}

// Morton code of a query position in the triangles' centroid box (clamped), for the traversal order.
__global__ void kQueryCodes(const double* __restrict__ P, int64_t m, double3 lo, double3 inv,
                            uint32_t* __restrict__ codes, uint32_t* __restrict__ idx) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  const double L[3] = {lo.x, lo.y, lo.z}, I[3] = {inv.x, inv.y, inv.z};
  uint32_t qc[3];
  for (int a = 0; a < 3; ++a) {
    const double u = (P[3 * i + a] - L[a]) * I[a];
    qc[a] = (uint32_t)fmin(fmax(u * 1024.0, 0.0), 1023.0);
  }
  codes[i] = mortonEncode(qc[0], qc[1], qc[2]);
  idx[i] = (uint32_t)i;
}

its_status sdfBvh(its_ctx* ctx, const double* dP, int64_t m, const double* dV, const int32_t* dF, int64_t nf, double* dOut) {
  its_status st;
  const int64_t nodes = 2 * nf - 1, inner = nf > 1 ? nf - 1 : 1;
  BvhDevice B;
  B.nf = nf;
  DevBuf<int32_t> left, right, parent;
  DevBuf<uint32_t> codes, idx, sc, leafTri, tk, tv;
  DevBuf<unsigned> flag;
  DevBuf<int32_t> range;
  if ((st = left.alloc(ctx, nf)) != ITS_OK || (st = right.alloc(ctx, nf)) != ITS_OK ||
      (st = parent.alloc(ctx, nodes)) != ITS_OK || (st = codes.alloc(ctx, nf)) != ITS_OK ||
      (st = idx.alloc(ctx, nf)) != ITS_OK || (st = sc.alloc(ctx, nf)) != ITS_OK ||
      (st = leafTri.alloc(ctx, nf)) != ITS_OK || (st = tk.alloc(ctx, nf)) != ITS_OK ||
      (st = tv.alloc(ctx, nf)) != ITS_OK || (st = flag.zeros(ctx, nf)) != ITS_OK ||
      (st = range.alloc(ctx, 2 * nf)) != ITS_OK)
    return st;
  // centroid bounds for the Morton quantisation
  const unsigned pb = 256;
  DevBuf<double> part;
  if ((st = part.alloc(ctx, kBoundWords * pb)) != ITS_OK) return st;
  kCentroidBounds<<<pb, 256, 0, ctx->stream>>>(dV, dF, nf, part.p);
  ITS_LAUNCHED(ctx);
  std::vector<double> hp(kBoundWords * pb);
  ITS_CU(ctx, cudaMemcpyAsync(hp.data(), part.p, kBoundWords * pb * 8, cudaMemcpyDeviceToHost, ctx->stream));
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  double bl[3] = {1e300, 1e300, 1e300}, bh[3] = {-1e300, -1e300, -1e300};
  int size = 0;
  for (unsigned k = 0; k < pb; ++k) {
    const double* p = &hp[kBoundWords * k];
    for (int a = 0; a < 3; ++a) { bl[a] = std::min(bl[a], p[a]); bh[a] = std::max(bh[a], p[3 + a]); }
    size = std::max(size, (int)p[6]);
  }
  // Meshes between 2^-32 and 2^32 as they are: a distance of 1e-8 of them has an FP32 square, and so
  // has one across them. Others scaled (within 2^+-500, so that the scale's square is a number too).
  int exponent = size > 0 && size < 0x7ff00000 ? std::max(-500, std::min(500, 1022 - (size >> 20))) : 0;
  if (std::abs(exponent) <= 32) exponent = 0;
  const double scale = std::ldexp(1.0, exponent), slack = std::ldexp(1.0 + 1e-12, 2 * exponent);
  double inv[3];
  for (int a = 0; a < 3; ++a) inv[a] = bh[a] > bl[a] ? 1.0 / (bh[a] - bl[a]) : 0.0;
  kMortonCodes<<<gridFor(nf, 256), 256, 0, ctx->stream>>>(dV, dF, nf, make_double3(bl[0], bl[1], bl[2]),
                                                         make_double3(inv[0], inv[1], inv[2]), codes.p, idx.p);
  ITS_LAUNCHED(ctx);
  if ((st = radixSortPairs(ctx, codes.p, idx.p, sc.p, leafTri.p, tk.p, tv.p, nf, 30)) != ITS_OK) return st;
  B.left = left.p;
  B.right = right.p;
  B.parent = parent.p;
  B.leafTri = leafTri.p;
  B.flag = flag.p;
  B.range = range.p;
  ITS_CU(ctx, cudaMemsetAsync(parent.p, 0xFF, nodes * 4, ctx->stream));
  if (nf > 1) {
    kBuildInternal<<<gridFor(nf - 1, 256), 256, 0, ctx->stream>>>(sc.p, nf, left.p, right.p, parent.p, range.p);
    ITS_LAUNCHED(ctx);
  }
  DevBuf<double> raw, tris;
  DevBuf<int2> top;
  DevBuf<unsigned> topCount;
  DevBuf<unsigned long long> counters;
  DevBuf<BoxF> box;
  DevBuf<FwnNode> fwn;
  DevBuf<WideNode> wide;
  if ((st = raw.alloc(ctx, kSumWords * nf)) != ITS_OK || (st = tris.alloc(ctx, kTriWords * nf)) != ITS_OK ||
      (st = top.alloc(ctx, nf)) != ITS_OK || (st = topCount.zeros(ctx, 1)) != ITS_OK || (st = counters.zeros(ctx, 2)) != ITS_OK ||
      (st = box.alloc(ctx, nodes)) != ITS_OK || (st = fwn.alloc(ctx, inner)) != ITS_OK ||
      (st = wide.alloc(ctx, inner)) != ITS_OK)
    return st;
  kBottomUp<<<gridFor(nf, kUpLeaves), kUpLeaves, 0, ctx->stream>>>(dV, dF, B, scale, raw.p, top.p, topCount.p, box.p, fwn.p,
                                                               tris.p);
  ITS_LAUNCHED(ctx);
  if (nf > kUpLeaves) {
    kClimbTop<<<gridFor(nf, 128), 128, 0, ctx->stream>>>(B, scale, raw.p, top.p, topCount.p, box.p, fwn.p);
    ITS_LAUNCHED(ctx);
  }
  kWideNodes<<<gridFor(inner, 128), 128, 0, ctx->stream>>>(B, box.p, wide.p);
  ITS_LAUNCHED(ctx);
  // the queries in Morton order
  DevBuf<uint32_t> qc, qi, qsc, qorder, qtk, qtv;
  DevBuf<uint8_t> inside;
  if ((st = qc.alloc(ctx, m)) != ITS_OK || (st = qi.alloc(ctx, m)) != ITS_OK || (st = qsc.alloc(ctx, m)) != ITS_OK ||
      (st = qorder.alloc(ctx, m)) != ITS_OK || (st = qtk.alloc(ctx, m)) != ITS_OK || (st = qtv.alloc(ctx, m)) != ITS_OK ||
      (st = inside.alloc(ctx, m)) != ITS_OK)
    return st;
  kQueryCodes<<<gridFor(m, 256), 256, 0, ctx->stream>>>(dP, m, make_double3(bl[0], bl[1], bl[2]),
                                                       make_double3(inv[0], inv[1], inv[2]), qc.p, qi.p);
  ITS_LAUNCHED(ctx);
  if ((st = radixSortPairs(ctx, qc.p, qi.p, qsc.p, qorder.p, qtk.p, qtv.p, m, 30)) != ITS_OK) return st;
  const unsigned blocks = (unsigned)std::min<int64_t>(gridFor(m, kGroups), 6ll * ctx->numSMs);  // six fit an SM
  (exponent ? kNearest<true> : kNearest<false>)<<<blocks, kWalkThreads, 0, ctx->stream>>>(dP, m, qorder.p, wide.p, tris.p, scale, slack, dOut, counters.p);
  ITS_LAUNCHED(ctx);
  if ((st = launchDependent(ctx, true, kWinding, (unsigned)std::min<int64_t>(gridFor(m, kGroups), 5ll * ctx->numSMs), kWalkThreads, 0, ctx->stream, dP, m, qorder.p, fwn.p, tris.p,
                            nf, inside.p, counters.p + 1)) != ITS_OK)
    return st;
  kSigns<<<gridFor(m, 256), 256, 0, ctx->stream>>>(inside.p, dOut, m);
  ITS_LAUNCHED(ctx);
  return ITS_OK;
}

}  // namespace its
