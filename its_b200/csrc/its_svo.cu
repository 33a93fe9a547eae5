// Sparse voxel octree on the GPU (replaces SparseVoxelOctree::createOctree and
// constructNodeAtrributes, SVO.cu:366-1110 of the reference).
//
// Layout (structure of arrays, depth 0 = voxels first, root last; same node order as the
// reference's svoNodeArray):
//   * occupancy of the res^3 voxel grid is a Morton-indexed bitset (res^3/8 bytes) instead
//     of a dense uint32 array; surface voxels are compacted from it in Morton order;
//   * so is every coarser level's, and one scan ranks all levels' cells: no dense per-level arrays,
//     no sort, and parent, children and neighbours by bit tests and ranks;
//   * nodes: morton / parent / first-child / leaf flag / 27 neighbours;
//   * per-depth corner vertices are a bitmap over the (res_d+1)^3 corner lattice with a
//     popcount rank per 64-bit word, which gives the reference's sorted (x,y,z) vertex order
//     and an O(1) corner -> column lookup without hashing or tolerant compares;
//   * fine-node edges are a bitmap over (lattice point, axis) with the same rank.
#include <algorithm>
#include <cmath>
#include <vector>

#include "its_scan.cuh"
#include "its_rows.cuh"
#include "its_svo.cuh"

namespace its {

// ---- voxelisation: surfaceVoxelize (SVO.cu:366-493), one thread per triangle -------------
struct E2 { double a, b, d; };
__device__ inline E2 edgeTest(double a, double b, bool flip, double pa, double pb, double ua, double ub) {
  if (flip) { a = -a; b = -b; }
  double d = (-1.0 * (a * pa + b * pb)) + fmax0(ua * a);
  d = d + fmax0(ub * b);
  return E2{a, b, d};
}

__global__ void kVoxelize(const double* __restrict__ V, const int32_t* __restrict__ F, int64_t nf, int res,
                          double3 g, double3 u, unsigned long long* __restrict__ occ) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nf; t += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i0 = F[3 * t], i1 = F[3 * t + 1], i2 = F[3 * t + 2];
    const double v0x = V[3 * i0] - g.x, v0y = V[3 * i0 + 1] - g.y, v0z = V[3 * i0 + 2] - g.z;
    const double v1x = V[3 * i1] - g.x, v1y = V[3 * i1 + 1] - g.y, v1z = V[3 * i1 + 2] - g.z;
    const double v2x = V[3 * i2] - g.x, v2y = V[3 * i2 + 1] - g.y, v2z = V[3 * i2 + 2] - g.z;
    const double e0x = v1x - v0x, e0y = v1y - v0y, e0z = v1z - v0z;
    const double e1x = v2x - v1x, e1y = v2y - v1y, e1z = v2z - v1z;
    const double e2x = v0x - v2x, e2y = v0y - v2y, e2z = v0z - v2z;
    double nx = e0y * e1z - e0z * e1y, ny = e0z * e1x - e0x * e1z, nz = e0x * e1y - e0y * e1x;
    {
      double z = nx * nx;
      z = z + ny * ny;
      z = z + nz * nz;
      if (z > 0.0) {
        const double s = sqrt(z);
        nx = nx / s; ny = ny / s; nz = nz / s;
      }
    }
    const double bminx = dmin(v0x, dmin(v1x, v2x)), bminy = dmin(v0y, dmin(v1y, v2y)), bminz = dmin(v0z, dmin(v1z, v2z));
    const double bmaxx = dmax(v0x, dmax(v1x, v2x)), bmaxy = dmax(v0y, dmax(v1y, v2y)), bmaxz = dmax(v0z, dmax(v1z, v2z));
    const int gx0 = clampi((int)(bminx / u.x), 0, res - 1), gy0 = clampi((int)(bminy / u.y), 0, res - 1),
              gz0 = clampi((int)(bminz / u.z), 0, res - 1);
    const int gx1 = clampi((int)(bmaxx / u.x), 0, res - 1), gy1 = clampi((int)(bmaxy / u.y), 0, res - 1),
              gz1 = clampi((int)(bmaxz / u.z), 0, res - 1);
    const double cx = nx > 0.0 ? u.x : 0.0, cy = ny > 0.0 ? u.y : 0.0, cz = nz > 0.0 ? u.z : 0.0;
    double d1 = nx * (cx - v0x);
    d1 = d1 + ny * (cy - v0y);
    d1 = d1 + nz * (cz - v0z);
    double d2 = nx * ((u.x - cx) - v0x);
    d2 = d2 + ny * ((u.y - cy) - v0y);
    d2 = d2 + nz * ((u.z - cz) - v0z);
    const E2 xy0 = edgeTest(-1.0 * e0y, e0x, nz < 0.0, v0x, v0y, u.x, u.y);
    const E2 xy1 = edgeTest(-1.0 * e1y, e1x, nz < 0.0, v1x, v1y, u.x, u.y);
    const E2 xy2 = edgeTest(-1.0 * e2y, e2x, nz < 0.0, v2x, v2y, u.x, u.y);
    const E2 yz0 = edgeTest(-1.0 * e0z, e0y, nx < 0.0, v0y, v0z, u.y, u.z);
    const E2 yz1 = edgeTest(-1.0 * e1z, e1y, nx < 0.0, v1y, v1z, u.y, u.z);
    const E2 yz2 = edgeTest(-1.0 * e2z, e2y, nx < 0.0, v2y, v2z, u.y, u.z);
    const E2 zx0 = edgeTest(-1.0 * e0x, e0z, ny < 0.0, v0z, v0x, u.z, u.x);
    const E2 zx1 = edgeTest(-1.0 * e1x, e1z, ny < 0.0, v1z, v1x, u.z, u.x);
    const E2 zx2 = edgeTest(-1.0 * e2x, e2z, ny < 0.0, v2z, v2x, u.z, u.x);
    for (int z = gz0; z <= gz1; ++z)
      for (int y = gy0; y <= gy1; ++y)
        for (int x = gx0; x <= gx1; ++x) {
          const double px = (double)x * u.x, py = (double)y * u.y, pz = (double)z * u.z;
          double nd = nx * px;
          nd = nd + ny * py;
          nd = nd + nz * pz;
          if ((nd + d1) * (nd + d2) > 0.0) continue;
          if ((xy0.a * px + xy0.b * py) + xy0.d < 0.0) continue;
          if ((xy1.a * px + xy1.b * py) + xy1.d < 0.0) continue;
          if ((xy2.a * px + xy2.b * py) + xy2.d < 0.0) continue;
          if ((yz0.a * py + yz0.b * pz) + yz0.d < 0.0) continue;
          if ((yz1.a * py + yz1.b * pz) + yz1.d < 0.0) continue;
          if ((yz2.a * py + yz2.b * pz) + yz2.d < 0.0) continue;
          if ((zx0.a * pz + zx0.b * px) + zx0.d < 0.0) continue;
          if ((zx1.a * pz + zx1.b * px) + zx1.d < 0.0) continue;
          if ((zx2.a * pz + zx2.b * px) + zx2.d < 0.0) continue;
          const uint32_t m = mortonEncode((uint32_t)x, (uint32_t)y, (uint32_t)z);
          atomicOr(occ + (m >> 6), 1ull << (m & 63));
        }
  }
}

// Which of n consecutive runs i lies in.
__device__ __forceinline__ int levelOf(const int64_t* start, int n, int64_t i) {
  int L = 0;
#pragma unroll
  for (int k = 1; k < kMaxDepth; ++k) L += k < n && i >= start[k] ? 1 : 0;
  return L;
}

// ---- level build ---------------------------------------------------------------------------
// The occupancy of every level as Morton bitsets, the voxels' words first and each coarser level's
// after them (a cell is occupied when one of its eight children is). One scan over all the words
// ranks every level's cells at once, so that a node's parent, children and neighbours are a bit
// test and a rank away, for all levels in one launch each; only the levels' counts go to the host.
// (Level by level -- a scan, a read of its count and three fills each, then the neighbours from
// the top down -- an octree of 6 levels took 110 launches and 13 waits.)
struct Pyramid {
  int levels;  // log2(res) + 1
  int64_t word[kMaxDepth + 1];  // first word of each level
  const unsigned long long* bits;
  const uint32_t* rank;  // over all words
  __device__ __forceinline__ bool has(int L, uint32_t code) const {
    return (bits[word[L] + (code >> 6)] >> (code & 63)) & 1ull;
  }
  __device__ __forceinline__ uint32_t rankOf(int L, uint32_t code) const {  // cells of finer levels included
    const int64_t w = word[L] + (code >> 6);
    return rank[w] + (uint32_t)__popcll(bits[w] & ((1ull << (code & 63)) - 1ull));
  }
};
// Bit i of the result: byte i of the word is not 0.
__device__ __forceinline__ uint32_t bytesSet(unsigned long long w) {
  w |= w >> 4;
  w |= w >> 2;
  w |= w >> 1;
  w &= 0x0101010101010101ull;
  return (uint32_t)((w * 0x0102040810204080ull) >> 56);
}
// Levels first + 1 .. first + 3 from level first (as many as there are): a block takes 512 of its
// words, 64 of the next level's, 8, 1. A block alone with its level goes on to the top.
constexpr int kPyrThreads = 64;
__global__ void __launch_bounds__(kPyrThreads) kPyramid(unsigned long long* __restrict__ bits,
                                                        const __grid_constant__ Pyramid P, int first) {
  __shared__ unsigned long long s[2][kPyrThreads];
  int64_t from = (int64_t)blockIdx.x * 512;  // the block's first word of the current level
  const int t = threadIdx.x;
  for (int L = first; L + 1 < P.levels && (L < first + 3 || gridDim.x == 1); ++L) {
    const int64_t words = P.word[L + 1] - P.word[L], next = P.word[L + 2] - P.word[L + 1], to = from / 8;
    const unsigned long long* prev = s[(L - first + 1) & 1];
    const int outs = L == first ? 64 : (L == first + 1 ? 8 : 1);  // the block's words of level L + 1
    unsigned long long w = 0;
    if (t < outs) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int64_t i = from + 8 * t + k;
        const unsigned long long v = i >= words ? 0ull : (L == first ? bits[P.word[L] + i] : prev[8 * t + k]);
        w |= (unsigned long long)bytesSet(v) << (8 * k);
      }
    }
    s[(L - first) & 1][t] = w;
    if (t < outs && to + t < next) bits[P.word[L + 1] + to + t] = w;
    __syncthreads();
    from = to;
  }
}
// Every level's cells in Morton order, the voxels first.
__global__ void kEmitCells(const __grid_constant__ Pyramid P, int64_t words, uint32_t* __restrict__ cells) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= words) return;
  unsigned long long w = P.bits[i];
  if (!w) return;
  const uint32_t first = (uint32_t)((i - P.word[levelOf(P.word, P.levels, i)]) * 64);
  uint32_t r = P.rank[i];
  while (w) {
    cells[r++] = first + (uint32_t)(__ffsll((long long)w) - 1);
    w &= w - 1;
  }
}
// out[k] = the rank at word at[k]
struct Bounds {
  int n;
  int64_t at[2 * kMaxDepth];
};
__global__ void kRanksAt(const uint32_t* __restrict__ rank, Bounds B, uint32_t* __restrict__ out) {
  if ((int)threadIdx.x < B.n) out[threadIdx.x] = rank[B.at[threadIdx.x]];
}

// The octree's levels as the kernels below see them.
struct Levels {
  int depth, res;
  int64_t node[kMaxDepth + 1];  // first node of each depth
  int64_t cell[kMaxDepth + 1];  // first of the level's cells among all levels' cells
  int64_t vert[kMaxDepth + 1];  // first vertex of each depth
  int64_t vword[kMaxDepth + 1]; // first word of each depth's corner lattice
};
// Nodes (createNode_1/2, SVO.cu:560-638): the eight children of every cell of the level above.
__global__ void kNodes(const __grid_constant__ Pyramid P, const __grid_constant__ Levels V,
                       const uint32_t* __restrict__ cells, uint32_t* __restrict__ morton, uint32_t* __restrict__ parent,
                       uint32_t* __restrict__ child0, uint8_t* __restrict__ leaf) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= V.node[V.depth]) return;
  const int top = V.depth - 1, L = levelOf(V.node, V.depth, t);
  if (L == top) {  // the root
    morton[t] = cells[V.cell[top]];
    parent[t] = kNone;
    child0[t] = top > 0 ? (uint32_t)V.node[top - 1] : kNone;
    leaf[t] = top > 0 ? 0 : 1;
    return;
  }
  const int64_t i = t - V.node[L];
  const uint32_t up = cells[V.cell[L + 1] + (i >> 3)], code = (up << 3) | (uint32_t)(i & 7);
  morton[t] = code;
  parent[t] = L + 1 == top ? (uint32_t)V.node[top]
                           : (uint32_t)(V.node[L + 1] + 8 * (int64_t)(P.rankOf(L + 2, up >> 3) - V.cell[L + 2]) +
                                        (up & 7u));
  const bool inner = L > 0 && P.has(L, code);
  child0[t] = inner ? (uint32_t)(V.node[L - 1] + 8 * (int64_t)(P.rankOf(L, code) - V.cell[L])) : kNone;
  leaf[t] = inner ? 0 : 1;
}

// 27-neighbours (findNeighbors, SVO.cu:861-890): the node at offset d of the same depth, which exists
// when its parent cell is occupied.
__global__ void kNeighbors(const __grid_constant__ Pyramid P, const __grid_constant__ Levels V,
                           const uint32_t* __restrict__ morton, uint32_t* __restrict__ nb) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= V.node[V.depth] * 27) return;
  const int64_t t = idx / 27;
  const int s = (int)(idx - 27 * t), L = levelOf(V.node, V.depth, t);
  uint32_t r = kNone;
  if (L == V.depth - 1) {
    if (s == 13) r = (uint32_t)t;
  } else {
    uint32_t X, Y, Z;
    mortonDecode(morton[t], X, Y, Z);
    const int x = (int)X + s % 3 - 1, y = (int)Y + (s / 3) % 3 - 1, z = (int)Z + s / 9 - 1, side = V.res >> L;
    if (x >= 0 && y >= 0 && z >= 0 && x < side && y < side && z < side) {
      const uint32_t m = mortonEncode((uint32_t)x, (uint32_t)y, (uint32_t)z);
      if (P.has(L + 1, m >> 3))
        r = (uint32_t)(V.node[L] + 8 * (int64_t)(P.rankOf(L + 1, m >> 3) - V.cell[L + 1]) + (m & 7u));
    }
  }
  nb[idx] = r;
}

// ---- corner vertices (determineNodeVertex + sort + unique, SVO.cu:913-963, 1064-1096) -------
// All depths in one launch each.
__device__ __forceinline__ int64_t cornerBit(const Levels& V, int64_t idx, const uint32_t* __restrict__ morton) {
  const int64_t t = idx >> 3;
  const int k = (int)(idx & 7), L = levelOf(V.node, V.depth, t);
  const uint32_t M = (uint32_t)(V.res >> L) + 1u;
  uint32_t X, Y, Z;
  mortonDecode(morton[t], X, Y, Z);
  return V.vword[L] * 64 + ((X + (k & 1)) * M + (Y + ((k >> 1) & 1))) * M + (Z + ((k >> 2) & 1));
}
__global__ void kMarkCorners(const __grid_constant__ Levels V, const uint32_t* __restrict__ morton,
                             unsigned long long* bits) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= V.node[V.depth] * 8) return;
  const int64_t b = cornerBit(V, idx, morton);
  atomicOr(bits + (b >> 6), 1ull << (b & 63));
}
// The set bits' indices (of vertices within their depth's lattice) in order, their owners to come.
__global__ void kEmitBits(int64_t words, const unsigned long long* __restrict__ bits,
                          const uint32_t* __restrict__ rank, uint32_t* __restrict__ out, uint32_t* __restrict__ owner) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= words) return;
  unsigned long long w = bits[i];
  if (!w) return;
  uint32_t r = rank[i];
  while (w) {
    const int b = __ffsll((long long)w) - 1;
    if (owner) owner[r] = kNone;
    out[r++] = (uint32_t)(i * 64 + b);
    w &= w - 1;
  }
}
__global__ void kOwnerCorners(const __grid_constant__ Levels V, const uint32_t* __restrict__ morton,
                              const unsigned long long* __restrict__ bits, const uint32_t* __restrict__ rank,
                              uint32_t* owner) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= V.node[V.depth] * 8) return;
  const int64_t b = cornerBit(V, idx, morton);
  const uint32_t v = rank[b >> 6] + (uint32_t)__popcll(bits[b >> 6] & ((1ull << (b & 63)) - 1ull));
  atomicMin(owner + v, (uint32_t)(idx >> 3));
}
// Representative position of a corner: taken from its owner node, corner = origin (+ w),
// origin = g + w*X (the surviving entry of the reference's stable sort + unique).
// Also the vertex's packed key (lattice coordinates, depth, corner of the owner).
__global__ void kVertexPositions(const __grid_constant__ Levels V, double3 g, double w0, uint32_t* __restrict__ lin,
                                 const uint32_t* __restrict__ owner, const uint32_t* __restrict__ morton,
                                 double* __restrict__ pos, uint64_t* __restrict__ key) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v >= V.vert[V.depth]) return;
  const int L = levelOf(V.vert, V.depth, v);
  const uint32_t M = (uint32_t)(V.res >> L) + 1u, l = lin[v] - (uint32_t)(V.vword[L] * 64);
  const double w = w0 * (double)(1u << L);
  lin[v] = l;
  const uint32_t X = l / (M * M), Y = (l / M) % M, Z = l % M;
  uint32_t Xo, Yo, Zo;
  mortonDecode(morton[owner[v]], Xo, Yo, Zo);
  key[v] = encodeVertKey(X, Y, Z, L, Xo, Yo, Zo);
  const double bx = latticePos(g.x, w, Xo), by = latticePos(g.y, w, Yo), bz = latticePos(g.z, w, Zo);
  pos[3 * v] = (X != Xo) ? bx + w : bx;
  pos[3 * v + 1] = (Y != Yo) ? by + w : by;
  pos[3 * v + 2] = (Z != Zo) ? bz + w : bz;
}

// ---- fine-node edges (determineNodeEdge + sort + unique, SVO.cu:965-1008, 1098-1110) --------
// Edge key = lin(lower end)*3 + {z:0, y:1, x:2}: the reference's lexicographic order of
// (first point, second point).
__device__ __constant__ int8_t cEdgeCorners[12][2] = {{0, 2}, {2, 3}, {1, 3}, {0, 1}, {4, 6}, {6, 7},
                                                    {5, 7}, {4, 5}, {0, 4}, {2, 6}, {3, 7}, {1, 5}};
__device__ inline uint32_t fineEdgeKey(uint32_t X, uint32_t Y, uint32_t Z, int e, uint32_t M) {
  const int a = cEdgeCorners[e][0], b = cEdgeCorners[e][1];
  const uint32_t sx = X + (a & 1), sy = Y + ((a >> 1) & 1), sz = Z + ((a >> 2) & 1);
  const int diff = a ^ b;  // 1: x, 2: y, 4: z
  const uint32_t ord = diff == 4 ? 0u : (diff == 2 ? 1u : 2u);
  return ((sx * M + sy) * M + sz) * 3u + ord;
}
__global__ void kMarkEdges(int64_t count, const uint32_t* __restrict__ morton, uint32_t M,
                           unsigned long long* bits) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= count * 12) return;
  const int64_t t = idx / 12;
  const int e = (int)(idx % 12);
  uint32_t X, Y, Z;
  mortonDecode(morton[t], X, Y, Z);
  const uint32_t key = fineEdgeKey(X, Y, Z, e, M);
  atomicOr(bits + (key >> 6), 1ull << (key & 63));
}
__global__ void kOwnerEdges(int64_t count, const uint32_t* __restrict__ morton, uint32_t M,
                            const unsigned long long* __restrict__ bits, const uint32_t* __restrict__ rank,
                            uint32_t* owner) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= count * 12) return;
  const int64_t t = idx / 12;
  const int e = (int)(idx % 12);
  uint32_t X, Y, Z;
  mortonDecode(morton[t], X, Y, Z);
  const uint32_t key = fineEdgeKey(X, Y, Z, e, M);
  const unsigned long long w = bits[key >> 6];
  const uint32_t r = rank[key >> 6] + (uint32_t)__popcll(w & ((1ull << (key & 63)) - 1ull));
  atomicMin(owner + r, (uint32_t)t);
}
// The depth-0 nodes as a Morton bitset with its ranks: the eight children of every cell of level 1 (of
// a lone root: itself).
__global__ void kFineNodes(const __grid_constant__ Pyramid P, const __grid_constant__ Levels V, int64_t words,
                           unsigned long long* __restrict__ occ, uint32_t* __restrict__ rank) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= words) return;
  if (V.depth == 1) {
    occ[i] = P.bits[i];
    rank[i] = P.rank[i];
    return;
  }
  const int64_t at = P.word[1] + (i >> 3);
  const int shift = 8 * (int)(i & 7);
  const unsigned long long up = P.bits[at];
  unsigned long long b = (up >> shift) & 0xffull;  // bit j: the j-th byte of the word is full
  b = (b * 0x0101010101010101ull) & 0x8040201008040201ull;
  b = ((b + 0x7f7f7f7f7f7f7f7full) | b) & 0x8080808080808080ull;  // byte j's top bit
  occ[i] = (b >> 7) * 0xffull;
  rank[i] = 8u * (P.rank[at] + (uint32_t)__popcll(up & ((1ull << shift) - 1ull)) - (uint32_t)V.cell[1]);
}

// ---- getters -------------------------------------------------------------------------------------
__global__ void kNodeGeometry(int64_t count, int64_t start, double3 g, double w, const uint32_t* __restrict__ morton,
                              double* origin, double* width) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int64_t t = start + i;
  uint32_t X, Y, Z;
  mortonDecode(morton[t], X, Y, Z);
  if (origin) {
    origin[3 * t] = latticePos(g.x, w, X);
    origin[3 * t + 1] = latticePos(g.y, w, Y);
    origin[3 * t + 2] = latticePos(g.z, w, Z);
  }
  if (width) width[t] = w;
}
__global__ void kExpandChildren(int64_t n, const uint32_t* __restrict__ child0, uint32_t* childs) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * 8) return;
  const uint32_t c = child0[i >> 3];
  childs[i] = (c == kNone) ? kNone : c + (uint32_t)(i & 7);
}
__global__ void kEdgePositions(int64_t E, uint32_t M, double3 g, double w, const uint32_t* __restrict__ key,
                               const uint32_t* __restrict__ owner, const uint32_t* __restrict__ morton,
                               double* p0, double* p1) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= E) return;
  const uint32_t k = key[i];
  const uint32_t lin = k / 3, ord = k % 3;
  const uint32_t X = lin / (M * M), Y = (lin / M) % M, Z = lin % M;
  uint32_t Xo, Yo, Zo;
  mortonDecode(morton[owner[i]], Xo, Yo, Zo);
  const double bx = latticePos(g.x, w, Xo), by = latticePos(g.y, w, Yo), bz = latticePos(g.z, w, Zo);
  const uint32_t E1[3] = {X + (ord == 2), Y + (ord == 1), Z + (ord == 0)};
  const uint32_t S[3] = {X, Y, Z}, O[3] = {Xo, Yo, Zo};
  const double B[3] = {bx, by, bz};
  for (int a = 0; a < 3; ++a) {
    if (p0) p0[3 * i + a] = (S[a] != O[a]) ? B[a] + w : B[a];
    if (p1) p1[3 * i + a] = (E1[a] != O[a]) ? B[a] + w : B[a];
  }
}

}  // namespace its

// =====================================================================================
using namespace its;

static void svoRelease(its_svo* s) {
  if (!s) return;
  its::destroyPlan(s->plan);
  s->plan = nullptr;
  its_ctx* c = s->ctx;
  SvoDevice& d = s->d;
  void* ptrs[] = {d.voxels, d.nodeMorton, d.nodeParent, d.nodeChild0, d.nodeLeaf, d.nodeNb, d.vertLin, d.vertKey,
                  d.vertOwner, d.vertPos, d.ebits, d.erank, d.edgeKey, d.edgeOwner, d.fineOcc, d.fineRank,
                  d.nodeSampleCnt, d.nodeSamplePos, d.nodeSampleNrm, d.coincIds, d.rowParams, d.coincGeom};
  for (void* p : ptrs) devFree(c, p);
  devFree(c, d.vbits[0]);
  devFree(c, d.vrank[0]);
  d = SvoDevice();
}

namespace its {

its_status svoBuild(its_ctx* ctx, const double* dV, int64_t nv, const int32_t* dF, int64_t nf, int res,
                    const double origin[3], const double width[3], its_svo* s) {
  (void)nv;
  SvoDevice& d = s->d;
  d.res = res;
  for (int a = 0; a < 3; ++a) { d.origin[a] = origin[a]; d.unit[a] = width[a] / res; }
  const double3 g = make_double3(origin[0], origin[1], origin[2]);
  const double3 u = make_double3(d.unit[0], d.unit[1], d.unit[2]);
  its_status st;
  // device time of the build and of the learned fit's tables (reported by its_svo_get_info)
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  for (auto& e : ev) ITS_CU(ctx, cudaEventCreate(&e));
  struct EvFree {
    cudaEvent_t* e;
    ~EvFree() { for (int k = 0; k < 3; ++k) if (e[k]) cudaEventDestroy(e[k]); }
  } evFree{ev};
  ITS_CU(ctx, cudaEventRecord(ev[0], ctx->stream));

  // 1. voxelise into the finest level of the occupancy pyramid, then the coarser levels
  Pyramid P{};
  P.levels = 1;
  while ((res >> P.levels) > 0) ++P.levels;
  for (int L = 0; L < P.levels; ++L) {
    const int64_t side = res >> L;
    P.word[L + 1] = P.word[L] + (side * side * side + 63) / 64;
  }
  const int64_t pyrWords = P.word[P.levels];
  DevBuf<unsigned long long> pyr;
  DevBuf<uint32_t> pyrRank, counts;
  if ((st = pyr.zeros(ctx, pyrWords)) != ITS_OK || (st = pyrRank.alloc(ctx, pyrWords)) != ITS_OK ||
      (st = counts.alloc(ctx, 2 * kMaxDepth)) != ITS_OK)
    return st;
  P.bits = pyr.p;
  P.rank = pyrRank.p;
  if (nf > 0) {
    const int block = 128;
    const unsigned grid = (unsigned)std::min<int64_t>(gridFor(nf, block), (int64_t)ctx->numSMs * 64);
    kVoxelize<<<grid, block, 0, ctx->stream>>>(dV, dF, nf, res, g, u, pyr.p);
    ITS_LAUNCHED(ctx);
  }
  for (int L = 0; L + 1 < P.levels; L += 3) {
    const unsigned blocks = (unsigned)((P.word[L + 1] - P.word[L] + 511) / 512);
    kPyramid<<<blocks, kPyrThreads, 0, ctx->stream>>>(pyr.p, P, L);
    ITS_LAUNCHED(ctx);
    if (blocks == 1) break;
  }
  // 2. ranks and counts of every level's cells; the root's level is the first with one cell
  uint32_t host[2 * kMaxDepth];
  auto popc = [](const unsigned long long* bits) {
    return [bits] __device__(int64_t i) -> uint32_t { return (uint32_t)__popcll(bits[i]); };
  };
  {
    if ((st = scanExclusiveAlloc<uint32_t>(ctx, popc(pyr.p), pyrWords, StorePrefix<uint32_t>{pyrRank.p},
                                           counts.p + P.levels - 1)) != ITS_OK)
      return st;
    Bounds B{P.levels - 1, {}};
    for (int L = 0; L + 1 < P.levels; ++L) B.at[L] = P.word[L + 1];
    kRanksAt<<<1, 32, 0, ctx->stream>>>(pyrRank.p, B, counts.p);
    ITS_LAUNCHED(ctx);
    ITS_CU(ctx, cudaMemcpyAsync(host, counts.p, P.levels * 4, cudaMemcpyDeviceToHost, ctx->stream));
    ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  }
  d.numVoxels = host[0];
  if (d.numVoxels == 0) return setError(ctx, ITS_ERR_INVALID, "no surface voxel: the mesh does not meet the grid");
  Levels V{};
  V.res = res;
  for (int L = 0; L < P.levels; ++L) V.cell[L + 1] = host[L];
  int top = 0;  // root level
  while (V.cell[top + 1] - V.cell[top] > 1) ++top;
  d.depth = V.depth = top + 1;
  int64_t total = 0;
  for (int L = 0; L <= top; ++L) {
    d.levelStart[L] = total;
    d.levelCount[L] = (L < top) ? 8 * (V.cell[L + 2] - V.cell[L + 1]) : 1;
    total += d.levelCount[L];
  }
  d.levelStart[top + 1] = total;
  d.numNodes = total;
  for (int L = 0; L <= d.depth; ++L) V.node[L] = d.levelStart[L];
  // every level's cells in Morton order, the surface voxels first
  const int64_t cells = V.cell[P.levels];
  if ((st = devAlloc(ctx, (void**)&d.voxels, cells * sizeof(uint32_t))) != ITS_OK) return st;
  kEmitCells<<<gridFor(pyrWords, 256), 256, 0, ctx->stream>>>(P, pyrWords, d.voxels);
  ITS_LAUNCHED(ctx);
  // 3. nodes and their 27 neighbours
  if ((st = devAlloc(ctx, (void**)&d.nodeMorton, total * 4)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.nodeParent, total * 4)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.nodeChild0, total * 4)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.nodeLeaf, total)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.nodeNb, total * 27 * 4)) != ITS_OK) return st;
  kNodes<<<gridFor(total, 256), 256, 0, ctx->stream>>>(P, V, d.voxels, d.nodeMorton, d.nodeParent, d.nodeChild0,
                                                      d.nodeLeaf);
  ITS_LAUNCHED(ctx);
  kNeighbors<<<gridFor(total * 27, 256), 256, 0, ctx->stream>>>(P, V, d.nodeMorton, d.nodeNb);
  ITS_LAUNCHED(ctx);

  // 4. corner vertices per depth and fine-node edges: marked, ranked, counted
  for (int L = 0; L < d.depth; ++L) {
    const int64_t M = (int64_t)(res >> L) + 1;
    V.vword[L + 1] = V.vword[L] + (M * M * M + 63) / 64;
  }
  const int64_t vwords = V.vword[d.depth], nf0 = d.levelCount[0];
  const uint32_t M0 = (uint32_t)res + 1u;
  const int64_t ewords = (3ll * M0 * M0 * M0 + 63) / 64;
  if ((st = devAlloc(ctx, (void**)&d.vbits[0], vwords * 8)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.vrank[0], vwords * 4)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.ebits, ewords * 8)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.erank, ewords * 4)) != ITS_OK) return st;
  for (int L = 1; L < d.depth; ++L) {
    d.vbits[L] = d.vbits[0] + V.vword[L];
    d.vrank[L] = d.vrank[0] + V.vword[L];
  }
  ITS_CU(ctx, cudaMemsetAsync(d.vbits[0], 0, vwords * 8, ctx->stream));
  ITS_CU(ctx, cudaMemsetAsync(d.ebits, 0, ewords * 8, ctx->stream));
  kMarkCorners<<<gridFor(total * 8, 256), 256, 0, ctx->stream>>>(V, d.nodeMorton, d.vbits[0]);
  ITS_LAUNCHED(ctx);
  kMarkEdges<<<gridFor(nf0 * 12, 256), 256, 0, ctx->stream>>>(nf0, d.nodeMorton, M0, d.ebits);
  ITS_LAUNCHED(ctx);
  {
    if ((st = scanExclusiveAlloc<uint32_t>(ctx, popc(d.vbits[0]), vwords, StorePrefix<uint32_t>{d.vrank[0]},
                                           counts.p + d.depth - 1)) != ITS_OK ||
        (st = scanExclusiveAlloc<uint32_t>(ctx, popc(d.ebits), ewords, StorePrefix<uint32_t>{d.erank},
                                           counts.p + d.depth)) != ITS_OK)
      return st;
    Bounds B{d.depth - 1, {}};
    for (int L = 0; L + 1 < d.depth; ++L) B.at[L] = V.vword[L + 1];
    kRanksAt<<<1, 32, 0, ctx->stream>>>(d.vrank[0], B, counts.p);
    ITS_LAUNCHED(ctx);
    ITS_CU(ctx, cudaMemcpyAsync(host, counts.p, (d.depth + 1) * 4, cudaMemcpyDeviceToHost, ctx->stream));
    ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  }
  for (int L = 0; L < d.depth; ++L) V.vert[L + 1] = host[L];
  for (int L = 0; L < d.depth; ++L) {
    d.vertStart[L] = V.vert[L];
    d.vertCount[L] = V.vert[L + 1] - V.vert[L];
  }
  d.vertStart[d.depth] = d.numVerts = V.vert[d.depth];
  d.numEdges = host[d.depth];
  if ((st = devAlloc(ctx, (void**)&d.vertLin, d.numVerts * 4)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.vertOwner, d.numVerts * 4)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.vertPos, d.numVerts * 24)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.vertKey, d.numVerts * 8)) != ITS_OK) return st;
  kEmitBits<<<gridFor(vwords, 256), 256, 0, ctx->stream>>>(vwords, d.vbits[0], d.vrank[0], d.vertLin, d.vertOwner);
  ITS_LAUNCHED(ctx);
  kOwnerCorners<<<gridFor(total * 8, 256), 256, 0, ctx->stream>>>(V, d.nodeMorton, d.vbits[0], d.vrank[0], d.vertOwner);
  ITS_LAUNCHED(ctx);
  kVertexPositions<<<gridFor(d.numVerts, 256), 256, 0, ctx->stream>>>(V, g, d.unit[0], d.vertLin, d.vertOwner,
                                                                     d.nodeMorton, d.vertPos, d.vertKey);
  ITS_LAUNCHED(ctx);

  // 5. fine-node edges and the fine-node occupancy bitset
  if ((st = devAlloc(ctx, (void**)&d.edgeKey, (size_t)d.numEdges * 4)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.edgeOwner, (size_t)d.numEdges * 4)) != ITS_OK) return st;
  kEmitBits<<<gridFor(ewords, 256), 256, 0, ctx->stream>>>(ewords, d.ebits, d.erank, d.edgeKey, d.edgeOwner);
  ITS_LAUNCHED(ctx);
  kOwnerEdges<<<gridFor(nf0 * 12, 256), 256, 0, ctx->stream>>>(nf0, d.nodeMorton, M0, d.ebits, d.erank, d.edgeOwner);
  ITS_LAUNCHED(ctx);
  const int64_t gridWords = P.word[1];
  if ((st = devAlloc(ctx, (void**)&d.fineOcc, gridWords * 8)) != ITS_OK) return st;
  if ((st = devAlloc(ctx, (void**)&d.fineRank, gridWords * 4)) != ITS_OK) return st;
  kFineNodes<<<gridFor(gridWords, 256), 256, 0, ctx->stream>>>(P, V, gridWords, (unsigned long long*)d.fineOcc,
                                                              d.fineRank);
  ITS_LAUNCHED(ctx);
  // per-node sums of the face samples (features of the share network)
  ITS_CU(ctx, cudaEventRecord(ev[1], ctx->stream));
  if ((st = nodeSampleStats(ctx, d, dV, dF, nf)) != ITS_OK) return st;
  // the coincident vertices (the shares of the exact start)
  if ((st = devAlloc(ctx, (void**)&d.coincIds, std::max<int64_t>(d.numVerts, 1) * 8)) != ITS_OK) return st;
  if ((st = coincidentIds(ctx, d, d.coincIds, &d.numCoinc)) != ITS_OK) return st;
  if ((st = coincidentGeometry(ctx, d)) != ITS_OK) return st;
  // the row parameters of the matrix-free kernels, on the device for the octree's lifetime
  const RowParams hp = rowParams(d);
  if ((st = devAlloc(ctx, &d.rowParams, sizeof(RowParams))) != ITS_OK) return st;
  ITS_CU(ctx, cudaMemcpyAsync(d.rowParams, &hp, sizeof(RowParams), cudaMemcpyHostToDevice, ctx->stream));
  ITS_CU(ctx, cudaEventRecord(ev[2], ctx->stream));
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  cudaEventElapsedTime(&d.buildMs, ev[0], ev[2]);
  cudaEventElapsedTime(&d.learnedTablesMs, ev[1], ev[2]);
  return ITS_OK;
}

}  // namespace its

// ================================ C ABI ===============================================
extern "C" {

its_status its_svo_build(its_ctx* ctx, const double* verts, int64_t nverts, const int32_t* faces, int64_t nfaces,
                         int res, const double origin[3], const double width[3], its_svo** out) {
  if (!ctx || !out) return ITS_ERR_INVALID;
  *out = nullptr;
  if (!verts || !faces || nverts <= 0 || nfaces <= 0 || !origin || !width)
    return setError(ctx, ITS_ERR_INVALID, "its_svo_build: empty mesh or missing arguments");
  if (res < 1 || res > 1024 || (res & (res - 1)))
    return setError(ctx, ITS_ERR_INVALID, "its_svo_build: res must be a power of two in [1, 1024]");
  for (int a = 0; a < 3; ++a)
    if (!std::isfinite(origin[a]) || !(width[a] > 0.0) || !std::isfinite(width[a]))
      return setError(ctx, ITS_ERR_INVALID, "its_svo_build: bounding box must be finite with positive width");
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<double> V;
  InArg<int32_t> F;
  its_status st;
  if ((st = V.stage(ctx, verts, 3 * nverts)) != ITS_OK) return st;
  if ((st = F.stage(ctx, faces, 3 * nfaces)) != ITS_OK) return st;
  if ((st = validateMesh(ctx, V.d, nverts, F.d, nfaces)) != ITS_OK) return st;
  its_svo* s = new its_svo;
  s->ctx = ctx;
  st = svoBuild(ctx, V.d, nverts, F.d, nfaces, res, origin, width, s);
  if (st != ITS_OK) {
    svoRelease(s);
    delete s;
    return st;
  }
  *out = s;
  return ITS_OK;
}

its_status its_svo_free(its_svo* s) {
  if (!s) return ITS_OK;
  its_ctx* c = s->ctx;
  svoRelease(s);
  cudaStreamSynchronize(c->stream);
  delete s;
  return ITS_OK;
}

its_status its_svo_get_info(const its_svo* s, its_svo_info* info) {
  if (!s || !info) return ITS_ERR_INVALID;
  const SvoDevice& d = s->d;
  *info = its_svo_info{};
  info->res = d.res;
  info->depth = d.depth;
  info->num_voxels = d.numVoxels;
  info->num_fine_nodes = d.levelCount[0];
  info->num_nodes = d.numNodes;
  info->num_vertices = d.numVerts;
  info->num_edges = d.numEdges;
  for (int L = 0; L < d.depth && L < 16; ++L) {
    info->nodes_per_depth[L] = d.levelCount[L];
    info->vertices_per_depth[L] = d.vertCount[L];
  }
  for (int a = 0; a < 3; ++a) { info->origin[a] = d.origin[a]; info->unit[a] = d.unit[a]; }
  info->build_ms = d.buildMs;
  info->learned_tables_ms = d.learnedTablesMs;
  return ITS_OK;
}

its_status its_svo_get_voxels(its_svo* s, uint32_t* morton) {
  if (!s || !morton) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  ITS_CU(ctx, cudaMemcpyAsync(morton, s->d.voxels, s->d.numVoxels * 4, cudaMemcpyDefault, ctx->stream));
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_svo_get_nodes(its_svo* s, uint32_t* morton, uint32_t* parent, uint32_t* childs, uint8_t* is_leaf,
                             double* origin, double* width, uint32_t* neighbors) {
  if (!s) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  const SvoDevice& d = s->d;
  const int64_t N = d.numNodes;
  if (morton) ITS_CU(ctx, cudaMemcpyAsync(morton, d.nodeMorton, N * 4, cudaMemcpyDefault, ctx->stream));
  if (parent) ITS_CU(ctx, cudaMemcpyAsync(parent, d.nodeParent, N * 4, cudaMemcpyDefault, ctx->stream));
  if (is_leaf) ITS_CU(ctx, cudaMemcpyAsync(is_leaf, d.nodeLeaf, N, cudaMemcpyDefault, ctx->stream));
  if (neighbors) ITS_CU(ctx, cudaMemcpyAsync(neighbors, d.nodeNb, N * 27 * 4, cudaMemcpyDefault, ctx->stream));
  its_status st;
  if (childs) {
    OutArg<uint32_t> o;
    if ((st = o.stage(ctx, childs, N * 8)) != ITS_OK) return st;
    kExpandChildren<<<gridFor(N * 8, 256), 256, 0, ctx->stream>>>(N, d.nodeChild0, o.d);
    ITS_LAUNCHED(ctx);
    if ((st = o.finish(ctx)) != ITS_OK) return st;
    ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  }
  if (origin || width) {
    OutArg<double> o, w;
    if ((st = o.stage(ctx, origin, N * 3)) != ITS_OK) return st;
    if ((st = w.stage(ctx, width, N)) != ITS_OK) return st;
    const double3 g = make_double3(d.origin[0], d.origin[1], d.origin[2]);
    for (int L = 0; L < d.depth; ++L) {
      kNodeGeometry<<<gridFor(d.levelCount[L], 256), 256, 0, ctx->stream>>>(
          d.levelCount[L], d.levelStart[L], g, d.unit[0] * (double)(1u << L), d.nodeMorton, o.d, w.d);
      ITS_LAUNCHED(ctx);
    }
    if ((st = o.finish(ctx)) != ITS_OK) return st;
    if ((st = w.finish(ctx)) != ITS_OK) return st;
    ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  }
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_svo_get_vertices(its_svo* s, double* pos, uint32_t* owner) {
  if (!s) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  if (pos) ITS_CU(ctx, cudaMemcpyAsync(pos, s->d.vertPos, s->d.numVerts * 24, cudaMemcpyDefault, ctx->stream));
  if (owner) ITS_CU(ctx, cudaMemcpyAsync(owner, s->d.vertOwner, s->d.numVerts * 4, cudaMemcpyDefault, ctx->stream));
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_svo_get_edges(its_svo* s, double* p0, double* p1, uint32_t* owner) {
  if (!s) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  const SvoDevice& d = s->d;
  const int64_t E = d.numEdges;
  its_status st;
  if (owner) ITS_CU(ctx, cudaMemcpyAsync(owner, d.edgeOwner, E * 4, cudaMemcpyDefault, ctx->stream));
  if ((p0 || p1) && E > 0) {
    OutArg<double> a, b;
    if ((st = a.stage(ctx, p0, E * 3)) != ITS_OK) return st;
    if ((st = b.stage(ctx, p1, E * 3)) != ITS_OK) return st;
    kEdgePositions<<<gridFor(E, 256), 256, 0, ctx->stream>>>(E, (uint32_t)d.res + 1u,
                                                             make_double3(d.origin[0], d.origin[1], d.origin[2]),
                                                             d.unit[0], d.edgeKey, d.edgeOwner, d.nodeMorton, a.d, b.d);
    ITS_LAUNCHED(ctx);
    if ((st = a.finish(ctx)) != ITS_OK) return st;
    if ((st = b.finish(ctx)) != ITS_OK) return st;
  }
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

}  // extern "C"
