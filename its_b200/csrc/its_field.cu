#include <cmath>
// Field evaluation and marching cubes.
//
// * Points (ThinShells::cpLatentBSplineValue, ThinShells.cpp:655-755): a point's fine node
//   is found by binary search of its voxel's Morton code in the sorted depth-0 node list;
//   the field is sum(lambda * hat) over the 8 corners of that node and of every ancestor,
//   corners in order k = x|y<<1|z<<2, ancestors from fine to coarse (the reference's order).
// * Lattice (the MC input of MarchingCubes.cu:464-536 / CUDACompute.cu:435-510): the
//   reference sums lambda_j * hat_j over ALL n corner vertices for 8 duplicated corners per
//   voxel, O(8 R^3 n). Only the 8 corners of the depth-d cell holding p can be non-zero, so
//   each lattice point of the (R+1)^3 grid is evaluated once from at most 8 corners per depth,
//   their existence and column read from the per-depth lattice bitmaps: O(8 D) per point.
// * Marching cubes (MarchingCubes.cu:164-377): case index with bit i = f(corner i) < iso in
//   the reference's corner order, vertex counts from the case table, an exclusive scan of the
//   counts, and the triangle soup written in voxel order by the scan's own downsweep (no
//   compaction pass, no 18 R^3 preallocation).
#include <algorithm>
#include <cfloat>
#include <type_traits>
#include <vector>

#include "its_mc.cuh"
#include "its_tune.cuh"
#include "its_op.cuh"

namespace its {

struct EvalParams {
  int depth, res;
  double3 g;
  double w0;
  LatticeIndex lat[kMaxDepth];
  int64_t fineCount;
  const uint32_t* morton;
  const uint32_t* parent;
  const double* vertPos;
  const uint64_t* vertKey;  // packed lattice coordinates and the vertex's corner of its owner
  const unsigned long long* fineOcc;  // depth-0 nodes: Morton bitset and its word ranks
  const uint32_t* fineRank;
  double winv[kMaxDepth];  // RN(1 / w_d), for divRn
};

static EvalParams evalParams(const SvoDevice& d) {
  EvalParams P;
  P.depth = d.depth;
  P.res = d.res;
  P.g = make_double3(d.origin[0], d.origin[1], d.origin[2]);
  P.w0 = d.unit[0];
  for (int L = 0; L < kMaxDepth; ++L) P.lat[L] = L < d.depth ? d.lattice(L) : LatticeIndex{};
  P.fineCount = d.levelCount[0];
  P.morton = d.nodeMorton;
  P.parent = d.nodeParent;
  P.vertPos = d.vertPos;
  P.vertKey = d.vertKey;
  P.fineOcc = (const unsigned long long*)d.fineOcc;
  P.fineRank = d.fineRank;
  for (int L = 0; L < kMaxDepth; ++L) P.winv[L] = 1.0 / (P.w0 * (double)(1u << L));
  return P;
}

// Chain evaluation of one point; returns false when no fine node holds it.
__device__ inline bool evalChain(const EvalParams& P, const double* __restrict__ lambda, double px, double py,
                                 double pz, double& out) {
  const int dx = (int)((px - P.g.x) / P.w0), dy = (int)((py - P.g.y) / P.w0), dz = (int)((pz - P.g.z) / P.w0);
  if (dx < 0 || dy < 0 || dz < 0 || dx >= P.res || dy >= P.res || dz >= P.res) return false;
  uint32_t t = fineNodeOf(P.fineOcc, P.fineRank, mortonEncode((uint32_t)dx, (uint32_t)dy, (uint32_t)dz));
  if (t == kNone) return false;
  double sum = 0.0;
  for (int d = 0; d < P.depth && t != kNone; ++d) {
    uint32_t X, Y, Z;
    mortonDecode(P.morton[t], X, Y, Z);
    const double w = P.w0 * (double)(1u << d), wi = P.winv[d];
    const double bx = latticePos(P.g.x, w, X), by = latticePos(P.g.y, w, Y), bz = latticePos(P.g.z, w, Z);
    const LatticeIndex& L = P.lat[d];
    // hat3's three factors for the cell's two corner positions per axis (the 8 corners share
    // them); each term is hat3's value: 0 once a factor is not positive, else x * y * z
    const double fx[2] = {hat1r(px, bx, w, wi), hat1r(px, bx + w, w, wi)};
    const double fy[2] = {hat1r(py, by, w, wi), hat1r(py, by + w, w, wi)};
    const double fz[2] = {hat1r(pz, bz, w, wi), hat1r(pz, bz + w, w, wi)};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int ox = k & 1, oy = (k >> 1) & 1, oz = (k >> 2) & 1;
      const uint32_t col = latticeRank(L, ((X + ox) * L.M + (Y + oy)) * L.M + (Z + oz));
      const double h = (fx[ox] <= 0.0 || fy[oy] <= 0.0 || fz[oz] <= 0.0) ? 0.0 : fx[ox] * fy[oy] * fz[oz];
      sum += lambda[col] * h;
    }
    t = P.parent[t];
  }
  out = sum;
  return true;
}

__global__ void kEvalPoints(const __grid_constant__ EvalParams P, const double* __restrict__ lambda,
                            const double* __restrict__ pts, int64_t m, double* __restrict__ out,
                            uint8_t* __restrict__ missing) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  double v = 0.0;
  const bool ok = evalChain(P, lambda, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], v);
  out[i] = ok ? v : 0.0;
  if (missing) missing[i] = ok ? 0 : 1;
}

// min / max over the found points, count of missing ones; one partial per block.
__global__ void kIsoPartials(const __grid_constant__ EvalParams P, const double* __restrict__ lambda,
                             const double* __restrict__ pts, int64_t m, double* __restrict__ pmin,
                             double* __restrict__ pmax, unsigned long long* __restrict__ pmiss) {
  double lo = DBL_MAX, hi = -DBL_MAX;
  unsigned long long miss = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    double v;
    if (evalChain(P, lambda, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], v)) {
      lo = fmin(lo, v);
      hi = fmax(hi, v);
    } else {
      ++miss;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_down_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_down_sync(0xffffffffu, hi, o));
    miss += __shfl_down_sync(0xffffffffu, miss, o);
  }
  __shared__ double slo[8], shi[8];
  __shared__ unsigned long long smiss[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { slo[w] = lo; shi[w] = hi; smiss[w] = miss; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
      lo = fmin(lo, slo[k]);
      hi = fmax(hi, shi[k]);
      miss += smiss[k];
    }
    pmin[blockIdx.x] = lo;
    pmax[blockIdx.x] = hi;
    pmiss[blockIdx.x] = miss;
  }
}

// The field at any point: sum over every corner vertex of lambda * hat, restricted to the
// only terms that can be non-zero -- at each depth the 8 corners of the cell holding p that
// exist as vertices of that depth -- summed depth 0..D-1, corners k = x|y<<1|z<<2.
__device__ inline double fieldAt(const EvalParams& P, const double* __restrict__ lambda, double px, double py,
                                 double pz) {
  double sum = 0.0;
  for (int d = 0; d < P.depth; ++d) {
    const double w = P.w0 * (double)(1u << d), wi = P.winv[d];
    const LatticeIndex& L = P.lat[d];
    const int64_t lim = (int64_t)(P.res >> d);
    const int64_t cx = (int64_t)floor(divRn(px - P.g.x, w, wi)), cy = (int64_t)floor(divRn(py - P.g.y, w, wi)),
                  cz = (int64_t)floor(divRn(pz - P.g.z, w, wi));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int64_t Lx = cx + (k & 1), Ly = cy + ((k >> 1) & 1), Lz = cz + ((k >> 2) & 1);
      if (Lx < 0 || Ly < 0 || Lz < 0 || Lx > lim || Ly > lim || Lz > lim) continue;
      const uint32_t lin = (uint32_t)((Lx * L.M + Ly) * L.M + Lz);
      if (!latticeHas(L, lin)) continue;
      const uint32_t v = latticeRank(L, lin);
      sum += lambda[v] * hat3r(P.vertPos[3 * v], P.vertPos[3 * v + 1], P.vertPos[3 * v + 2], w, wi, px, py, pz);
    }
  }
  return sum;
}

constexpr int kBrickThreads = 256, kTileCap = 640;
// The FP64 field on the (R+1)^3 lattice in bricks of 32 x 4 x 8 points; a thread evaluates a column of
// 4 points along z. For each depth the brick's points fall in a small box of cells; the
// corners of that box (presence, coefficient, representative position) are staged in shared
// memory once, and every point then sums its 8 corners from there -- the same additions in
// the same order as fieldAt, so the result is bit-identical, without per-point lattice
// lookups. The x and y hat factors of a corner are shared by the thread's 4 points (equal
// inputs, equal IEEE results); all quotients use divRn. Depths whose corner box has no
// corner are skipped; depths whose box exceeds the tile (grids much coarser than the octree)
// fall back to per-point lookups.
// The cell at distance a from the lattice's first point; one outside the lattice's cells 0 .. lim touches no
// corner and is kept next to them, so that boxes stay small.
__device__ __forceinline__ int64_t cellOf(double a, double w, double wi, int64_t lim) {
  const int64_t c = (int64_t)floor(divRn(a, w, wi));
  return c < -2 ? -2 : (c > lim + 1 ? lim + 1 : c);
}

template <int kBrickX, int kBrickY, int kZPer>
__global__ void __launch_bounds__(kBrickThreads, 2)
    kEvalGridBricks(const __grid_constant__ EvalParams P, const double* __restrict__ lambda, double3 o, double3 vs,
                    int R, double* __restrict__ field) {
  constexpr int kBrickZ = (kBrickThreads / (kBrickX * kBrickY)) * kZPer;
  __shared__ double tLam[kTileCap], tPx[kTileCap], tPy[kTileCap], tPz[kTileCap];
  __shared__ unsigned char tHas[kTileCap];
  __shared__ int64_t box[6];  // first and last cell per axis at the current depth
  const int64_t M = (int64_t)R + 1;
  const int tid = threadIdx.x;
  const int64_t x0 = (int64_t)blockIdx.x * kBrickX, y0 = (int64_t)blockIdx.y * kBrickY,
                z0 = (int64_t)blockIdx.z * kBrickZ;
  const int64_t xi = x0 + (tid % kBrickX), yj = y0 + ((tid / kBrickX) % kBrickY);
  const int64_t zb = z0 + (int64_t)(tid / (kBrickX * kBrickY)) * kZPer;
  const bool inXY = xi < M && yj < M;
  const double px = o.x + (double)xi * vs.x, py = o.y + (double)yj * vs.y;
  const double gx = P.g.x, gy = P.g.y, gz = P.g.z;
  double pz[kZPer], sum[kZPer];
#pragma unroll
  for (int q = 0; q < kZPer; ++q) {
    pz[q] = o.z + (double)(zb + q) * vs.z;
    sum[q] = 0.0;
  }
  for (int d = 0; d < P.depth; ++d) {
    const double w = P.w0 * (double)(1u << d), wi = P.winv[d];
    const LatticeIndex& L = P.lat[d];
    const int64_t lim = (int64_t)(P.res >> d);
    if (tid < 6) {
      const int a = tid >> 1;
      const int64_t idx = (a == 0 ? x0 : a == 1 ? y0 : z0) +
                          ((tid & 1) ? (a == 0 ? kBrickX : a == 1 ? kBrickY : kBrickZ) - 1 : 0);
      const int64_t cl = idx < M ? idx : M - 1;
      const double oa = a == 0 ? o.x : a == 1 ? o.y : o.z, va = a == 0 ? vs.x : a == 1 ? vs.y : vs.z;
      const double ga = a == 0 ? P.g.x : a == 1 ? P.g.y : P.g.z;
      const double pa = oa + (double)cl * va;
      box[tid] = cellOf(pa - ga, w, wi, lim);
    }
    __syncthreads();
    const int64_t cx0 = box[0], cy0 = box[2], cz0 = box[4];
    const int nx = (int)(box[1] - cx0 + 2), ny = (int)(box[3] - cy0 + 2), nz = (int)(box[5] - cz0 + 2);
    // block-uniform (a lattice that runs backwards has no box)
    const bool tiled = nx > 1 && ny > 1 && nz > 1 && (int64_t)nx * ny * nz <= kTileCap;
    int any = 1;
    if (tiled) {
      int mine = 0;
      for (int t = tid; t < nx * ny * nz; t += kBrickThreads) {
        const int64_t Lx = cx0 + t / (ny * nz), Ly = cy0 + (t / nz) % ny, Lz = cz0 + t % nz;
        unsigned char has = 0;
        if (Lx >= 0 && Ly >= 0 && Lz >= 0 && Lx <= lim && Ly <= lim && Lz <= lim) {
          const uint32_t lin = (uint32_t)((Lx * L.M + Ly) * L.M + Lz);
          if (latticeHas(L, lin)) {
            const uint32_t v = latticeRank(L, lin);
            const double qx = P.vertPos[3 * v], qy = P.vertPos[3 * v + 1], qz = P.vertPos[3 * v + 2];
            tLam[t] = lambda[v];
            tPx[t] = qx;
            tPy[t] = qy;
            tPz[t] = qz;
            // bit 0: present; bits 1-3: the x / y / z coordinate is the lattice coordinate
            // g + w X, so the column's shared factor for that axis applies
            has = (unsigned char)(1 | (qx == latticePos(P.g.x, w, (uint32_t)Lx) ? 2 : 0) |
                                  (qy == latticePos(P.g.y, w, (uint32_t)Ly) ? 4 : 0) |
                                  (qz == latticePos(P.g.z, w, (uint32_t)Lz) ? 8 : 0));
          }
        }
        tHas[t] = has;
        mine |= has;
      }
      any = __syncthreads_or(mine);
    } else {
      __syncthreads();
    }
    if (any && inXY) {
      const int64_t cx = cellOf(px - gx, w, wi, lim), cy = cellOf(py - gy, w, wi, lim);
      // the lattice factors of this column's cell: x and y shared by its 4 points
      const double fx[2] = {hat1r(px, latticePos(P.g.x, w, (uint32_t)cx), w, wi),
                            hat1r(px, latticePos(P.g.x, w, (uint32_t)(cx + 1)), w, wi)};
      const double fy[2] = {hat1r(py, latticePos(P.g.y, w, (uint32_t)cy), w, wi),
                            hat1r(py, latticePos(P.g.y, w, (uint32_t)(cy + 1)), w, wi)};
#pragma unroll
      for (int q = 0; q < kZPer; ++q) {
        if (zb + q >= M) break;
        const double pzq = pz[q];
        const int64_t cz = cellOf(pzq - gz, w, wi, lim);
        const double fz[2] = {hat1r(pzq, latticePos(P.g.z, w, (uint32_t)cz), w, wi),
                              hat1r(pzq, latticePos(P.g.z, w, (uint32_t)(cz + 1)), w, wi)};
        double s = sum[q];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int ox = k & 1, oy = (k >> 1) & 1, oz = (k >> 2) & 1;
          double lam;
          unsigned f;
          int t = 0;
          uint32_t vv = 0;
          if (tiled) {
            t = ((int)(cx - cx0) + ox) * ny * nz + ((int)(cy - cy0) + oy) * nz + ((int)(cz - cz0) + oz);
            f = tHas[t];
            if (!f) continue;
            lam = tLam[t];
          } else {
            const int64_t Lx = cx + ox, Ly = cy + oy, Lz = cz + oz;
            if (Lx < 0 || Ly < 0 || Lz < 0 || Lx > lim || Ly > lim || Lz > lim) continue;
            const uint32_t lin = (uint32_t)((Lx * L.M + Ly) * L.M + Lz);
            if (!latticeHas(L, lin)) continue;
            vv = latticeRank(L, lin);
            lam = lambda[vv];
            f = 1u;  // positions from the vertex array
          }
          // hat3 as the reference forms it: x, y, z factors with early exits; a factor at the
          // lattice coordinate is the column's shared one (equal inputs, equal IEEE result)
          double hx, hy, hz;
          if (f & 2) hx = fx[ox];
          else hx = hat1r(px, tiled ? tPx[t] : P.vertPos[3 * (int64_t)vv], w, wi);
          if (hx <= 0.0) continue;
          if (f & 4) hy = fy[oy];
          else hy = hat1r(py, tiled ? tPy[t] : P.vertPos[3 * (int64_t)vv + 1], w, wi);
          if (hy <= 0.0) continue;
          if (f & 8) hz = fz[oz];
          else hz = hat1r(pzq, tiled ? tPz[t] : P.vertPos[3 * (int64_t)vv + 2], w, wi);
          if (hz <= 0.0) continue;
          s += lam * (hx * hy * hz);
        }
        sum[q] = s;
      }
    }
    __syncthreads();
  }
  if (inXY) {
#pragma unroll
    for (int q = 0; q < kZPer; ++q)
      if (zb + q < M) field[xi + M * (yj + M * (zb + q))] = sum[q];
  }
}

// The FP64 field again, separably. A corner vertex's position along one axis is one of two
// values: g + w X (the owner node's corner bit is 0 on that axis) or (g + w (X - 1)) + w (the
// bit is 1; SVO.cu:573-576 forms corners from the owner's origin). So the hat factor of a
// point and a corner along an axis is one of two values that depend only on the point's
// coordinate on that axis, the corner's lattice coordinate and that bit. kSepTables forms
// them once per grid coordinate and depth (the reference's hat arithmetic, quotients by
// divRn); each block copies its brick's slices and stages each corner of the brick's cell box
// at every depth as its coefficient and a flag byte (present, the three corner bits). A point
// then sums, for d = 0..D-1 and k = x|y<<1|z<<2, lambda * ((hx * hy) * hz) over its present
// corners -- fieldAt's additions in fieldAt's order, so the field is bit-identical, at a few
// table reads and three FP64 operations per term (the x*y factor is shared by a column's
// points where they lie in one cell).
constexpr int kSepX = 32, kSepY = 8, kSepThreads = kSepX * kSepY;
// Staged corners per depth and in all. Grids at least twice as fine as the octree need at most
// kSepTileCap; coarser ones (a point per finest cell: 34 x 10 x 10 corners a brick) get the larger
// pair, 72 KB of shared memory and three blocks per SM instead of four.
constexpr int kSepTileCap = 1024, kSepStageCap = 2048, kCoarseTileCap = 4608, kCoarseStageCap = 5632;
template <typename T> struct Pair { typedef double2 type; };
template <> struct Pair<float> { typedef float2 type; };

// The hat tables of every lattice coordinate of the grid, once per depth and axis (a grid of
// (R+1)^3 points has only 3 (R+1) coordinates per depth, which every brick would otherwise
// form again): tabC the coordinate's cell c = floor((p - g) / w), tabH its factors
// [corner side * 2 + corner bit] against the corner at c + side, whose position is g + w X for
// an owner bit 0 and (g + w (X - 1)) + w for an owner bit 1. Entry ((d * 3 + axis) * M + i).
__global__ void kSepTables(const __grid_constant__ EvalParams P, double3 o, double3 vs, int64_t M,
                           double* __restrict__ tabH, int* __restrict__ tabC) {
  const int64_t item = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (item >= (int64_t)P.depth * 3 * M) return;
  const int d = (int)(item / (3 * M)), a = (int)((item / M) % 3);
  const int64_t idx = item % M;
  const double w = P.w0 * (double)(1u << d), wi = P.winv[d];
  const double oa = a == 0 ? o.x : a == 1 ? o.y : o.z, va = a == 0 ? vs.x : a == 1 ? vs.y : vs.z;
  const double ga = a == 0 ? P.g.x : a == 1 ? P.g.y : P.g.z;
  const double pa = oa + (double)idx * va;
  const int64_t c = (int64_t)floor(divRn(pa - ga, w, wi));
  // a cell outside the depth's lattice touches no corner: kept next to it, so that boxes stay small
  const int64_t lim = (int64_t)(P.res >> d);
  const int64_t cc = c < -2 ? -2 : (c > lim + 1 ? lim + 1 : c);
  double h[4];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int64_t X = cc + side;
    const double pA = latticePos(ga, w, (uint32_t)(X < 0 ? 0 : X));
    const double pB = X >= 1 ? latticePos(ga, w, (uint32_t)(X - 1)) + w : pA;
    h[2 * side] = hat1r(pa, pA, w, wi);
    h[2 * side + 1] = hat1r(pa, pB, w, wi);
  }
  double2* dst = (double2*)(tabH + 4 * item);
  dst[0] = make_double2(h[0], h[1]);
  dst[1] = make_double2(h[2], h[3]);
  tabC[item] = (int)cc;
}

// One brick's hat tables and cell boxes: the hat factors and cells of the brick's coordinates
// for every depth ([corner side * 2 + corner bit]; hZ is [depth][that index][point], so a
// corner's factors for a thread's points lie side by side and come in pairs), and the corner
// boxes of every depth staged together in one pass (their lattice lookups are dependent loads:
// in one pass their latencies overlap).
template <typename T, int kSepZ, bool kCoarse>
struct alignas(16) SepStage {
  static constexpr int kTile = kCoarse ? kCoarseTileCap : kSepTileCap;
  static constexpr int kStage = kCoarse ? kCoarseStageCap : kSepStageCap;
  T hX[kMaxDepth][4][kSepX];  // [depth][corner side * 2 + corner bit][x]: a warp's x run reads side by side
  T hY[kMaxDepth][kSepY][4];
  T hZ[kMaxDepth][4][kSepZ];
  T tLam[kStage];
  int cX[kMaxDepth][kSepX], cY[kMaxDepth][kSepY], cZ[kMaxDepth][kSepZ];
  int tOff[kMaxDepth], tEnd[kMaxDepth];  // depth d's tile: [tOff[d], tEnd[d]); tOff -1: per-point
  int cOff[kMaxDepth], cEnd[kMaxDepth];  // its (x, y) columns: [cOff[d], cEnd[d])
  int bny[kMaxDepth], bnz[kMaxDepth];  // the box's corners along y and z
  int tAny[kMaxDepth], tOdd[kMaxDepth], tCols;  // any corner; a coefficient that is not finite (kCoarse)
  unsigned char tFlag[kStage];
  __device__ int boxOf(int d, int& nx, int& ny, int& nz) const {
    nx = cX[d][kSepX - 1] - cX[d][0] + 2;
    ny = cY[d][kSepY - 1] - cY[d][0] + 2;
    nz = cZ[d][kSepZ - 1] - cZ[d][0] + 2;
    return nx * ny * nz;
  }
};

// The brick's slices of kSepTables' tables (threads i = 0, n, 2n, ... of the calling group).
template <typename T, int kSepZ, bool kCoarse>
__device__ void sepTables(SepStage<T, kSepZ, kCoarse>& S, int D, int64_t M, int64_t x0, int64_t y0, int64_t z0,
                          const double* __restrict__ tabH, const int* __restrict__ tabC, int i, int n) {
  constexpr int kCoords = kSepX + kSepY + kSepZ, kBatch = 4;  // a thread's items in batches, loads first
  const int total = kCoords * D;
  for (int item0 = i; item0 < total; item0 += kBatch * n) {
    double2 h01[kBatch], h23[kBatch];
    int c[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int item = item0 + u * n;
      if (item >= total) break;
      const int d = item / kCoords, j = item % kCoords;
      const int a = j < kSepX ? 0 : (j < kSepX + kSepY ? 1 : 2);
      const int k = a == 0 ? j : (a == 1 ? j - kSepX : j - kSepX - kSepY);
      int64_t idx = (a == 0 ? x0 : a == 1 ? y0 : z0) + k;
      if (idx > M - 1) idx = M - 1;  // clamped to the grid
      const int64_t r = ((int64_t)d * 3 + a) * M + idx;
      h01[u] = __ldg((const double2*)(tabH + 4 * r));
      h23[u] = __ldg((const double2*)(tabH + 4 * r) + 1);
      c[u] = __ldg(tabC + r);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int item = item0 + u * n;
      if (item >= total) break;
      const int d = item / kCoords, j = item % kCoords;
      const int a = j < kSepX ? 0 : (j < kSepX + kSepY ? 1 : 2);
      const int k = a == 0 ? j : (a == 1 ? j - kSepX : j - kSepX - kSepY);
      if (a == 2) {
        S.hZ[d][0][k] = (T)h01[u].x;
        S.hZ[d][1][k] = (T)h01[u].y;
        S.hZ[d][2][k] = (T)h23[u].x;
        S.hZ[d][3][k] = (T)h23[u].y;
      } else if (a == 0) {
        S.hX[d][0][k] = (T)h01[u].x;
        S.hX[d][1][k] = (T)h01[u].y;
        S.hX[d][2][k] = (T)h23[u].x;
        S.hX[d][3][k] = (T)h23[u].y;
      } else {
        T* dst = S.hY[d][k];
        dst[0] = (T)h01[u].x;
        dst[1] = (T)h01[u].y;
        dst[2] = (T)h23[u].x;
        dst[3] = (T)h23[u].y;
      }
      (a == 0 ? S.cX[d] : a == 1 ? S.cY[d] : S.cZ[d])[k] = c[u];
    }
  }
}

// Where each depth's box goes (a box over the capacity: per-point lookups), by one warp: lane d
// sizes depth d's box, then every lane runs the greedy placement in depth order on the
// shuffled sizes (registers only) and lane d keeps depth d's place.
template <typename T, int kSepZ, bool kCoarse>
__device__ void sepPlace(SepStage<T, kSepZ, kCoarse>& S, int D, int lane) {
  int n = 0, c = 0, ny = 0, nz = 0;
  if (lane < D) {
    int nx;
    n = S.boxOf(lane, nx, ny, nz);
    c = nx > 1 && ny > 1 && nz > 1 ? nx * ny : 0;
  }
  int off = 0, cols = 0, myOff = -1, myCol = 0, myEnd = 0, myColEnd = 0;
  for (int d = 0; d < D; ++d) {
    const int nd = __shfl_sync(0xffffffffu, n, d), cd = __shfl_sync(0xffffffffu, c, d);
    // (a lattice that runs backwards has no box)
    const bool fits = cd > 0 && nd > 0 && nd <= S.kTile && off + nd <= S.kStage;
    if (lane == d) {
      myOff = fits ? off : -1;
      myCol = cols;
    }
    if (fits) {
      off += (nd + 1) & ~1;  // boxes start at even entries: a column's z pairs are aligned
      cols += cd;
    }
    if (lane == d) {
      myEnd = off;
      myColEnd = cols;
    }
  }
  if (lane < D) {
    S.tOff[lane] = myOff;
    S.tEnd[lane] = myEnd;
    S.cOff[lane] = myCol;
    S.cEnd[lane] = myColEnd;
    S.bny[lane] = ny;
    S.bnz[lane] = nz;
    S.tAny[lane] = 0;
    S.tOdd[lane] = 0;
  }
  if (lane == 0) S.tCols = cols;
}

// The corners of every depth's cell box: coefficient and flag byte (bit 0 present, bits 1-3
// the owner corner bits); tAny[d]: whether depth d has any. A thread per (x, y) column of a
// box, eight z entries at a time: their lattice indices are consecutive, so they lie in one or
// two words of the lattice bits, and the loads of those words, then of the present corners'
// coefficients and keys, go out together. The box entry (x, y, z) sits at (x ny + y) nz + z.
template <typename T, int kSepZ, bool kCoarse>
__device__ void sepStageBoxes(SepStage<T, kSepZ, kCoarse>& S, const EvalParams& P, const double* __restrict__ lambda, int i,
                              int n) {
  for (int e = i; e < S.tCols; e += n) {
    // the columns lie in depth order (a depth without a tile: an empty range): e's depth is the
    // number of depths whose columns end at or before it
    int d = 0;
#pragma unroll
    for (int j = 0; j < kMaxDepth; ++j) d += (j < P.depth && e >= S.cEnd[j]) ? 1 : 0;
    const int ny = S.bny[d], nz = S.bnz[d];
    const int col = e - S.cOff[d], ix = col / ny, iy = col - ix * ny;
    const LatticeIndex& L = P.lat[d];
    const int lim = P.res >> d;
    const int Lx = S.cX[d][0] + ix, Ly = S.cY[d][0] + iy;
    const bool inBox = Lx >= 0 && Ly >= 0 && Lx <= lim && Ly <= lim;
    const uint32_t colBase = inBox ? ((uint32_t)Lx * L.M + (uint32_t)Ly) * L.M : 0u;
    bool any = false;
    for (int z8 = 0; z8 < nz; z8 += 8) {
      const int zA = S.cZ[d][0] + z8;
      const int zLo = zA < 0 ? 0 : zA, zHi = min(min(zA + 7, S.cZ[d][0] + nz - 1), lim);
      unsigned long long wLo = 0, wHi = 0;
      uint32_t rLo = 0, rHi = 0, wIdx = 0;
      const bool live = inBox && zLo <= zHi;
      if (live) {
        wIdx = (colBase + (uint32_t)zLo) >> 6;
        const uint32_t wLast = (colBase + (uint32_t)zHi) >> 6;
        wLo = L.bits[wIdx];
        rLo = L.rank[wIdx];
        if (wLast != wIdx) {
          wHi = L.bits[wLast];
          rHi = L.rank[wLast];
        }
      }
      uint32_t v[8];
      unsigned hasMask = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int Lz = zA + j;
        v[j] = 0;
        if (live && Lz >= zLo && Lz <= zHi) {
          const uint32_t lin = colBase + (uint32_t)Lz;
          const bool lo = (lin >> 6) == wIdx;
          const unsigned long long word = lo ? wLo : wHi;
          if ((word >> (lin & 63)) & 1ull) {  // latticeHas / latticeRank on the kept words
            v[j] = L.base + (lo ? rLo : rHi) + (uint32_t)__popcll(word & ((1ull << (lin & 63)) - 1ull));
            hasMask |= 1u << j;
          }
        }
      }
      double lv[8];
      uint32_t keyHi[8];  // the key's upper word: the owner corner bits 37-39 are its bits 5-7
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        lv[j] = 0.0;
        keyHi[j] = 0;
        if (hasMask >> j & 1u) {
          lv[j] = lambda[v[j]];
          keyHi[j] = ((const uint32_t*)P.vertKey)[2 * (size_t)v[j] + 1];
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (z8 + j >= nz) break;
        const int t = S.tOff[d] + col * nz + z8 + j;
        unsigned char f = 0;
        if (hasMask >> j & 1u) {
          S.tLam[t] = (T)lv[j];
          if (kCoarse && !isfinite((T)lv[j])) S.tOdd[d] = 1;
          f = (unsigned char)(1u | (((keyHi[j] >> 5) & 7u) << 1));
        }
        S.tFlag[t] = f;
      }
      any |= hasMask != 0;
    }
    if (any) S.tAny[d] = 1;  // benign race: every writer stores 1
  }
}

// The terms of G consecutive points q0.. of a thread's column that lie in one cell (box-relative
// z cell rz): each present corner's coefficient, bits and x*y factor are read once for them,
// and each point adds lambda * ((hx * hy) * hz) in corner order. colT[c]: the box entry of the
// (x, y) corner column c = x | y << 1 at z = 0.
template <int G, typename T, int kSepZ, bool kCoarse>
__device__ __forceinline__ void sepCellTerms(const SepStage<T, kSepZ, kCoarse>& S, int d, const T* hx, const T* hy,
                                             const T* lamT, const unsigned char* flagT, const int (&colT)[4], int rz,
                                             int q0, T (&sum)[kSepZ]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ox = k & 1, oy = (k >> 1) & 1, oz = k >> 2;
    const int t = colT[k & 3] + rz + oz;
    const unsigned f = flagT[t];
    if (!(f & 1u)) continue;
    const T lam = lamT[t];
    const T fxy = hx[kSepX * (2 * ox + ((f >> 1) & 1u))] * hy[2 * oy + ((f >> 2) & 1u)];
    const T* hz = S.hZ[d][2 * oz + ((f >> 3) & 1u)];
#pragma unroll
    for (int g = 0; g < G; ++g) sum[q0 + g] += lam * (fxy * hz[q0 + g]);
  }
}

// The terms of one thread's column of kSepZ points (brick column tx, ty) over every depth, in
// fieldAt's order: for d = 0..D-1 and k = x|y<<1|z<<2, lambda * ((hx * hy) * hz).
template <typename T, int kSepZ, bool kCoarse>
__device__ void sepTerms(const SepStage<T, kSepZ, kCoarse>& S, const EvalParams& P, const double* __restrict__ lambda,
                         int tx, int ty, T (&sum)[kSepZ]) {
#pragma unroll
  for (int q = 0; q < kSepZ; ++q) sum[q] = T(0);
  for (int d = 0; d < P.depth; ++d) {
    const int ny = S.bny[d], nz = S.bnz[d];
    if (S.tOff[d] < 0 || (kCoarse && S.tOdd[d])) {
      // The box does not fit the tile: each point looks its corners up, the four (x, y) corner
      // columns' two z neighbours in one or two words of the lattice bits, most of them empty. A
      // factor that is not positive ends its term here, as in the point-wise kernel, so that a
      // coefficient that is not finite stays within its own cells (where one is staged, a coarse
      // grid's depth comes this way too).
      const LatticeIndex& L = P.lat[d];
      const int lim = P.res >> d;
      const int cx = S.cX[d][tx], cy = S.cY[d][ty];
#pragma unroll
      for (int q = 0; q < kSepZ; ++q) {
        const int cz = S.cZ[d][q];
        unsigned has = 0;  // bit k: corner k is a vertex
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int Lx = cx + (c & 1), Ly = cy + (c >> 1);
          if (Lx < 0 || Ly < 0 || Lx > lim || Ly > lim) continue;
          const uint32_t col = ((uint32_t)Lx * L.M + (uint32_t)Ly) * L.M;
          if (cz >= 0 && cz <= lim && latticeHas(L, col + (uint32_t)cz)) has |= 1u << c;
          if (cz >= -1 && cz < lim && latticeHas(L, col + (uint32_t)(cz + 1))) has |= 16u << c;
        }
        T s = sum[q];
        while (has) {
          const int k = __ffs(has) - 1, ox = k & 1, oy = (k >> 1) & 1, oz = k >> 2;
          has &= has - 1;
          const uint32_t v = latticeRank(
              L, ((uint32_t)(cx + ox) * L.M + (uint32_t)(cy + oy)) * L.M + (uint32_t)(cz + oz));
          const unsigned f = (unsigned)(P.vertKey[v] >> 37) & 7u;  // the owner corner bits
          const T fx = S.hX[d][2 * ox + (f & 1u)][tx], fy = S.hY[d][ty][2 * oy + ((f >> 1) & 1u)],
                  fz = S.hZ[d][2 * oz + ((f >> 2) & 1u)][q];
          if (fx <= T(0) || fy <= T(0) || fz <= T(0)) continue;
          s += (T)lambda[v] * (fx * fy * fz);
        }
        sum[q] = s;
      }
    } else if (S.tAny[d]) {
      const int rx = S.cX[d][tx] - S.cX[d][0], ry = S.cY[d][ty] - S.cY[d][0];
      const T* hx = &S.hX[d][0][tx];  // hx[kSepX * e]: factor e of the thread's x
      const T* hy = S.hY[d][ty];
      const T* lamT = S.tLam + S.tOff[d];
      const unsigned char* flagT = S.tFlag + S.tOff[d];
      // A present corner adds lambda * ((hx * hy) * hz) even where a factor is 0: the term is
      // then +-0 (NaN for a non-finite coefficient), as fieldAt's sum over the corners adds it,
      // and a running sum that starts at +0 is never -0, so a +-0 term leaves it unchanged.
      if (nz == 2) {
        // Every point of the brick's z run lies in one cell (block-uniform): a corner is the
        // same vertex for all of the thread's points, so its coefficient, bits and x*y factor
        // are read once and its terms cost two products and a sum per point. The four (x, y)
        // corner columns' flag and coefficient pairs (z = 0, 1 side by side, at an even entry)
        // are read up front.
        typedef typename Pair<T>::type P2;
        unsigned fp[4];
        P2 lp[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int t0 = ((rx + (c & 1)) * ny + (ry + (c >> 1))) * 2;
          fp[c] = *(const unsigned short*)(flagT + t0);
          lp[c] = *(const P2*)(lamT + t0);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int ox = k & 1, oy = (k >> 1) & 1, oz = (k >> 2) & 1;
          const unsigned f = (fp[k & 3] >> (8 * oz)) & 0xffu;
          if (!(f & 1u)) continue;
          const T lam = oz ? lp[k & 3].y : lp[k & 3].x;
          const T fxy = hx[kSepX * (2 * ox + ((f >> 1) & 1u))] * hy[2 * oy + ((f >> 2) & 1u)];
          const T* hz = S.hZ[d][2 * oz + (int)((f >> 3) & 1u)];
#pragma unroll
          for (int q = 0; q < kSepZ; q += 2) {
            const typename Pair<T>::type h2 = *(const typename Pair<T>::type*)(hz + q);
            sum[q] += lam * (fxy * h2.x);
            sum[q + 1] += lam * (fxy * h2.y);
          }
        }
      } else {
        // The thread's z run spans several cells (the finest depths): the points are taken in
        // runs of four, two or one that lie in one cell (the runs are the same for the whole
        // block), so a corner's reads and x*y factor serve every point of its run.
        int colT[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) colT[c] = ((rx + (c & 1)) * ny + (ry + (c >> 1))) * nz;
        const int zc = S.cZ[d][0];
#pragma unroll
        for (int q0 = 0; q0 < kSepZ; q0 += 4) {
          const int ra = S.cZ[d][q0] - zc, rb = S.cZ[d][q0 + 1] - zc, rc = S.cZ[d][q0 + 2] - zc,
                    rd = S.cZ[d][q0 + 3] - zc;
          if (ra == rd) {
            sepCellTerms<4>(S, d, hx, hy, lamT, flagT, colT, ra, q0, sum);
          } else {
            if (ra == rb) {
              sepCellTerms<2>(S, d, hx, hy, lamT, flagT, colT, ra, q0, sum);
            } else {
              sepCellTerms<1>(S, d, hx, hy, lamT, flagT, colT, ra, q0, sum);
              sepCellTerms<1>(S, d, hx, hy, lamT, flagT, colT, rb, q0 + 1, sum);
            }
            if (rc == rd) {
              sepCellTerms<2>(S, d, hx, hy, lamT, flagT, colT, rc, q0 + 2, sum);
            } else {
              sepCellTerms<1>(S, d, hx, hy, lamT, flagT, colT, rc, q0 + 2, sum);
              sepCellTerms<1>(S, d, hx, hy, lamT, flagT, colT, rd, q0 + 3, sum);
            }
          }
        }
      }
    }
  }
}

// T = float is the precision form's FP32 field: the same tables (formed in FP64, rounded once)
// and the same terms, summed in FP32. One block per brick of kSepX x kSepY x kSepZ points.
template <typename T, int kSepZ, bool kCoarse>  // points per thread along z (the brick's depth)
__global__ void __launch_bounds__(kSepThreads, kCoarse ? 3 : 4)
    kEvalGridSep(const __grid_constant__ EvalParams P, const double* __restrict__ lambda,
                 const double* __restrict__ tabH, const int* __restrict__ tabC, int R, T* __restrict__ field) {
  extern __shared__ __align__(16) unsigned char sepRaw[];
  SepStage<T, kSepZ, kCoarse>& S = *(SepStage<T, kSepZ, kCoarse>*)sepRaw;
  const int64_t M = (int64_t)R + 1;
  const int tid = threadIdx.x, tx = tid % kSepX, ty = tid / kSepX;
  const int64_t x0 = (int64_t)blockIdx.x * kSepX, y0 = (int64_t)blockIdx.y * kSepY, z0 = (int64_t)blockIdx.z * kSepZ;
  const int64_t xi = x0 + tx, yj = y0 + ty;
  sepTables(S, P.depth, M, x0, y0, z0, tabH, tabC, tid, kSepThreads);
  __syncthreads();
  if (tid < 32) sepPlace(S, P.depth, tid);
  __syncthreads();
  sepStageBoxes(S, P, lambda, tid, kSepThreads);
  __syncthreads();
  if (xi < M && yj < M) {
    T sum[kSepZ];
    sepTerms(S, P, lambda, tx, ty, sum);
#pragma unroll
    for (int q = 0; q < kSepZ; ++q)
      if (z0 + q < M) field[xi + M * (yj + M * (z0 + q))] = sum[q];
  }
}

template <typename T, int kSepZ, bool kCoarse>
static its_status launchSep(its_ctx* ctx, const EvalParams& P, const double* lam, const double* tabH, const int* tabC,
                            int res, T* field) {
  const int64_t M = (int64_t)res + 1;
  const dim3 grid((unsigned)((M + kSepX - 1) / kSepX), (unsigned)((M + kSepY - 1) / kSepY),
                  (unsigned)((M + kSepZ - 1) / kSepZ));
  constexpr int bytes = (int)sizeof(SepStage<T, kSepZ, kCoarse>);
  if (bytes > 48 * 1024)
    ITS_CU(ctx, cudaFuncSetAttribute(kEvalGridSep<T, kSepZ, kCoarse>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  kEvalGridSep<T, kSepZ, kCoarse><<<grid, kSepThreads, bytes, ctx->stream>>>(P, lam, tabH, tabC, res, field);
  ITS_LAUNCHED(ctx);
  return ITS_OK;
}

// ---- marching cubes -----------------------------------------------------------------------
// kMcSigns reads the field once, flat and coalesced, and keeps one bit per lattice point
// (f < iso); everything after works on the bits, which stay in L2 (17 MB at 513^3), and on the
// field values of crossed voxels only. kMcCases: a thread takes ITEMS consecutive voxels, whose
// 4 corner rows are windows of ITEMS + 1 bits, writes the case bytes (most windows are all 0 or
// all 1) and counts the vertices; tiles with any are listed. The tiles' counts are scanned
// (scanSpine), and kMcEmit writes the listed tiles' triangles, a thread per vertex, in voxel
// order, as the reference's compaction does. Comparing in the classifying pass itself read
// every value four times through the L1 and formed each case from four ballots: 356 us for the
// 512^3 cases of an FP64 field, and a thread per crossed voxel in one block per tile 97 us for
// 1.25 M vertices; now 154 + 66 us and 38 us.
constexpr int kSignWords = 16;  // words of 32 lattice points per warp
template <typename T>
__global__ void __launch_bounds__(kScanThreads) kMcSigns(const T* __restrict__ field, int64_t total, double iso,
                                                         uint32_t* __restrict__ signs, unsigned* __restrict__ zero) {
  gridDependents();
  if (blockIdx.x == 0 && threadIdx.x == 0) *zero = 0u;  // the listed tiles' counter
  const int lane = threadIdx.x & 31;
  const int64_t w0 = ((int64_t)blockIdx.x * (kScanThreads / 32) + (threadIdx.x >> 5)) * kSignWords;
  const int64_t i0 = w0 * 32 + lane;
  T v[kSignWords];
  if ((w0 + kSignWords) * 32 <= total) {
#pragma unroll
    for (int j = 0; j < kSignWords; ++j) v[j] = field[i0 + 32 * j];
  } else {
#pragma unroll
    for (int j = 0; j < kSignWords; ++j) v[j] = i0 + 32 * j < total ? field[i0 + 32 * j] : field[total - 1];
  }
  uint32_t mine = 0;
#pragma unroll
  for (int j = 0; j < kSignWords; ++j) {
    const uint32_t b = __ballot_sync(0xffffffffu, (double)v[j] < iso);
    if (lane == j) mine = b;
  }
  if (lane < kSignWords) signs[w0 + lane] = mine;
}

// The bit of lattice point p, and the 32 bits from it on.
__device__ __forceinline__ unsigned signBit(const uint32_t* signs, int64_t p) {
  return (signs[p >> 5] >> (p & 31)) & 1u;
}
__device__ __forceinline__ uint32_t signWindow(const uint32_t* signs, int64_t p) {
  const uint32_t* w = signs + (p >> 5);
  return __funnelshift_r(w[0], w[1], (unsigned)(p & 31));
}
// Bits 0..3 of b, one per byte.
__device__ __forceinline__ uint32_t spread4(uint32_t b) { return ((b & 15u) * 0x00204081u) & 0x01010101u; }

// Division of v < 2^53 by d <= 2048: with m = ceil(2^64 / d), m d = 2^64 + e, e < d, so v m / 2^64 is
// v / d plus v e / (d 2^64), less than 1 / d: the same whole part.
struct FastDiv {
  unsigned long long m;
  int d;
  __device__ __forceinline__ int64_t operator()(int64_t v) const {
    return d == 1 ? v : (int64_t)__umul64hi((unsigned long long)v, m);
  }
};
static FastDiv fastDiv(int d) { return {d > 1 ? ~0ull / (unsigned)d + 1ull : 0ull, d}; }

// A warp takes kTiles consecutive tiles of 32 x ITEMS voxels, their windows loaded together. A run
// that crosses a row's end joins the windows of the two rows.
template <int ITEMS, int kTiles>
__global__ void __launch_bounds__(kScanThreads) kMcCases(const uint32_t* signs, int R, FastDiv byR,
                                                         uint8_t* __restrict__ cube, int64_t numTiles,
                                                         unsigned long long* __restrict__ tileSums,
                                                         uint32_t* __restrict__ listed, unsigned* __restrict__ numListed) {
  constexpr uint32_t kMask = (1u << ITEMS) - 1u;
  __shared__ unsigned char sCount[256];
  const int lane = threadIdx.x & 31;
  const int64_t nvox = (int64_t)R * R * R, M = (int64_t)R + 1;
  const int64_t tile0 = ((int64_t)blockIdx.x * (kScanThreads / 32) + (threadIdx.x >> 5)) * kTiles;
  sCount[threadIdx.x] = (unsigned char)(cMcCase[threadIdx.x] & 15ull);
  gridDependencyWait();
  gridDependents();
  uint32_t c[kTiles][4], n[kTiles][4];  // the corners at x and x + 1 of (y, z), (y+1, z), (y, z+1), (y+1, z+1)
  bool whole[kTiles];
#pragma unroll
  for (int t = 0; t < kTiles; ++t) {
    const int64_t base = ((tile0 + t) * 32 + lane) * ITEMS;
    whole[t] = base + ITEMS <= nvox && ITEMS <= R;
    if (!whole[t]) continue;
    const int64_t row = byR(base), z = byR(row), p = base + row + z * M;  // (z M + y) M + x
    const int left = (int)((row + 1) * R - base);                         // voxels left in the row
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = signWindow(signs, p + (k & 1 ? M : 0) + (k & 2 ? M * M : 0));
      c[t][k] = w & kMask;
      n[t][k] = (w >> 1) & kMask;
    }
    if (left < ITEMS) {
      const int64_t row2 = row + 1, z2 = byR(row2), p2 = row2 * R + row2 + z2 * M;
      const uint32_t keep = (1u << left) - 1u;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t w = signWindow(signs, p2 + (k & 1 ? M : 0) + (k & 2 ? M * M : 0));
        c[t][k] = (c[t][k] & keep) | (w << left & kMask);
        n[t][k] = (n[t][k] & keep) | ((w >> 1) << left & kMask);
      }
    }
  }
  __syncthreads();
  unsigned sums[kTiles];
#pragma unroll
  for (int t = 0; t < kTiles; ++t) {
    const int64_t base = ((tile0 + t) * 32 + lane) * ITEMS;
    unsigned cnt = 0;
    if (whole[t]) {
      uint32_t out[ITEMS / 4];
      const uint32_t some = c[t][0] | c[t][1] | c[t][2] | c[t][3] | n[t][0] | n[t][1] | n[t][2] | n[t][3];
      const uint32_t all = c[t][0] & c[t][1] & c[t][2] & c[t][3] & n[t][0] & n[t][1] & n[t][2] & n[t][3];
      if (some == 0u || all == kMask) {
#pragma unroll
        for (int j = 0; j < ITEMS / 4; ++j) out[j] = some ? 0xffffffffu : 0u;
      } else {
        // corner order 0 (0,0,0) 1 (0,1,0) 2 (1,1,0) 3 (1,0,0) 4 (0,0,1) 5 (0,1,1) 6 (1,1,1) 7 (1,0,1)
#pragma unroll
        for (int j = 0; j < ITEMS / 4; ++j) {
          const uint32_t v = spread4(c[t][0] >> (4 * j)) | spread4(c[t][1] >> (4 * j)) << 1 |
                             spread4(n[t][1] >> (4 * j)) << 2 | spread4(n[t][0] >> (4 * j)) << 3 |
                             spread4(c[t][2] >> (4 * j)) << 4 | spread4(c[t][3] >> (4 * j)) << 5 |
                             spread4(n[t][3] >> (4 * j)) << 6 | spread4(n[t][2] >> (4 * j)) << 7;
          out[j] = v;
          cnt += sCount[v & 255u] + sCount[(v >> 8) & 255u] + sCount[(v >> 16) & 255u] + sCount[v >> 24];
        }
      }
      uint8_t* dst = cube + base;
      if (!((uintptr_t)dst & (ITEMS - 1))) {  // base is a multiple of ITEMS: the caller's buffer decides
        if constexpr (ITEMS == 16) *(uint4*)dst = make_uint4(out[0], out[1], out[2], out[3]);
        else if constexpr (ITEMS == 8) *(uint2*)dst = make_uint2(out[0], out[1]);
        else *(uint32_t*)dst = out[0];
      } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) dst[j] = (uint8_t)(out[j >> 2] >> (8 * (j & 3)));
      }
    } else if (base < nvox) {
      int64_t x, y, z;
      voxelXYZ(base, R, x, y, z);
      for (int j = 0; j < ITEMS && base + j < nvox; ++j) {
        const int64_t q = (z * M + y) * M + x;
        const unsigned ci = signBit(signs, q) | signBit(signs, q + M) << 1 | signBit(signs, q + M + 1) << 2 |
                            signBit(signs, q + 1) << 3 | signBit(signs, q + M * M) << 4 |
                            signBit(signs, q + M * M + M) << 5 | signBit(signs, q + M * M + M + 1) << 6 |
                            signBit(signs, q + M * M + 1) << 7;
        cube[base + j] = (uint8_t)ci;
        cnt += sCount[ci];
        if (++x == R) {  // next row
          x = 0;
          if (++y == R) {
            y = 0;
            ++z;
          }
        }
      }
    }
    sums[t] = __reduce_add_sync(0xffffffffu, cnt);
  }
  if (lane == 0) {
    unsigned any = 0;
#pragma unroll
    for (int t = 0; t < kTiles; ++t) {
      if (tile0 + t < numTiles) tileSums[tile0 + t] = sums[t];
      any += sums[t] ? 1u : 0u;
    }
    if (any && listed) {  // in any order: every tile has its own place in the soup
      unsigned at = atomicAdd(numListed, any);
#pragma unroll
      for (int t = 0; t < kTiles; ++t)
        if (sums[t]) listed[at++] = (uint32_t)(tile0 + t);
    }
  }
}

// The listed tiles' triangles, a warp per tile. The tile's voxels with vertices are listed in voxel
// order (one scan of voxel and vertex counts packed in 32 bits), then its vertices are written, a
// lane each: a lane finds its voxel in the list, reads the two field values at its edge's ends
// and writes its point, so neighbouring lanes write neighbouring vertices.
template <typename T, int ITEMS>
__global__ void __launch_bounds__(kScanThreads) kMcEmit(McCaseT<T> mc, FastDiv byR, double3 o, double3 vs,
                                                        const uint8_t* cube,
                                                        const unsigned long long* tileOffsets,
                                                        const uint32_t* listed,
                                                        const unsigned* numListed,
                                                        double* __restrict__ tri, unsigned long long capacity) {
  constexpr int kTile = 32 * ITEMS;
  static_assert(15 * kTile < 65536, "voxel and vertex counts share 32 bits");
  __shared__ uint32_t sLists[kScanThreads / 32][kTile];  // place in the tile | first vertex << 16
  __shared__ uint8_t sCases[kScanThreads / 32][kTile];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, R = mc.R;
  uint32_t* sList = sLists[warp];
  uint8_t* sCase = sCases[warp];
  __shared__ uint32_t sWords[kScanThreads / 32][kTile / 4];
  __shared__ uint8_t sPlaces[kScanThreads / 32][kTile / 4];
  uint32_t* sWord = sWords[warp];
  uint8_t* sPlace = sPlaces[warp];
  __shared__ uint64_t sTable[256];  // per-lane indices: shared memory, not the constant cache
  sTable[threadIdx.x] = cMcCase[threadIdx.x];
  gridDependencyWait();
  __syncthreads();
  const int64_t nvox = (int64_t)R * R * R, M = (int64_t)R + 1;
  const unsigned n = *numListed, step = gridDim.x * (kScanThreads / 32);
  for (unsigned t = blockIdx.x * (kScanThreads / 32) + warp; t < n; t += step) {
    const uint32_t tile = listed[t];
    const int64_t tile0 = (int64_t)tile * kTile, base = tile0 + (int64_t)lane * ITEMS;
    const unsigned long long tileBase = tileOffsets[tile];
    // the words of four case bytes that are not all 0 or all 255, in voxel order
    uint32_t word[ITEMS / 4];
    if (base + ITEMS <= nvox && !((uintptr_t)(cube + base) & 3u)) {
#pragma unroll
      for (int j = 0; j < ITEMS / 4; ++j) word[j] = *(const uint32_t*)(cube + base + 4 * j);
    } else {
#pragma unroll
      for (int j = 0; j < ITEMS / 4; ++j) {
        word[j] = 0;
        for (int k = 0; k < 4; ++k)
          if (base + 4 * j + k < nvox) word[j] |= (uint32_t)cube[base + 4 * j + k] << (8 * k);
      }
    }
    uint32_t mixed = 0;
#pragma unroll
    for (int j = 0; j < ITEMS / 4; ++j) mixed += word[j] != 0u && word[j] != 0xffffffffu;
    uint32_t incl = mixed;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += up;
    }
    const uint32_t words = __shfl_sync(0xffffffffu, incl, 31);
    uint32_t at = incl - mixed;
    __syncwarp();  // the previous tile's lists have been read
#pragma unroll
    for (int j = 0; j < ITEMS / 4; ++j)
      if (word[j] != 0u && word[j] != 0xffffffffu) {
        sWord[at] = word[j];
        sPlace[at++] = (uint8_t)(lane * (ITEMS / 4) + j);
      }
    __syncwarp();
    // their voxels with vertices, a lane per byte
    uint32_t total = 0;  // vertices | voxels << 16
    for (uint32_t b0 = 0; b0 < 4 * words; b0 += 32) {
      const uint32_t b = b0 + lane;
      const uint32_t c = b < 4 * words ? (sWord[b >> 2] >> (8 * (b & 3))) & 255u : 0u;
      const uint32_t cnt = c != 0u && c != 255u ? ((unsigned)sTable[c] & 15u) + 65536u : 0u;
      uint32_t run = cnt;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, run, d);
        if (lane >= d) run += up;
      }
      const uint32_t first = total + run - cnt;
      if (cnt) {
        sList[first >> 16] = (4u * sPlace[b >> 2] + (b & 3u)) | first << 16;
        sCase[first >> 16] = (uint8_t)c;
      }
      total += __shfl_sync(0xffffffffu, run, 31);
    }
    __syncwarp();
    const unsigned nv = total & 65535u, nl = total >> 16;
    for (unsigned e = lane; e < nv; e += 32) {
      if (tileBase + e >= capacity) break;
      unsigned lo = 0, hi = nl;  // the last listed voxel whose first vertex is at or before e
      while (hi - lo > 1) {
        const unsigned mid = (lo + hi) / 2;
        if ((sList[mid] >> 16) <= e) lo = mid;
        else hi = mid;
      }
      const uint32_t item = sList[lo];
      const int64_t v = tile0 + (item & 65535u), row = byR(v), z = byR(row), x = v - row * R, y = row - z * R;
      const int edge = (int)((sTable[sCase[lo]] >> (4 * (e - (item >> 16) + 1))) & 15u);
      // the edge's corners (cMcEdge as nibbles) and their offsets (cMcCorner's columns as bits)
      const int a = (int)(0x321076543210ull >> (4 * edge)) & 15, b = (int)(0x765447650321ull >> (4 * edge)) & 15;
      const int oa[3] = {0xCC >> a & 1, 0x66 >> a & 1, 0xF0 >> a & 1},
                ob[3] = {0xCC >> b & 1, 0x66 >> b & 1, 0xF0 >> b & 1};
      const double vp[3] = {(double)x * vs.x + o.x, (double)y * vs.y + o.y, (double)z * vs.z + o.z};
      const double vsz[3] = {vs.x, vs.y, vs.z};
      double pa[3], pb[3], q[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        pa[k] = oa[k] ? vp[k] + vsz[k] : vp[k];
        pb[k] = ob[k] ? vp[k] + vsz[k] : vp[k];
      }
      const int64_t corner = (z * M + y) * M + x;
      const double sa = (double)mc.field[corner + (oa[2] * M + oa[1]) * M + oa[0]];
      const double sb = (double)mc.field[corner + (ob[2] * M + ob[1]) * M + ob[0]];
      vertexLerp(pa, pb, sa, sb, mc.iso, q);
      double* dst = tri + 3 * (tileBase + e);
      dst[0] = q[0];
      dst[1] = q[1];
      dst[2] = q[2];
    }
  }
}

// Dense-field launch shapes (bricks of BX x BY x BZ points, a thread per column of ZPER
// points); every shape computes the same bits, the autotuner picks the fastest.
template <int BX, int BY, int ZPER>
static its_status launchBricks(its_ctx* ctx, const EvalParams& P, const double* lam, double3 o, double3 vs, int res,
                               double* field) {
  constexpr int BZ = (kBrickThreads / (BX * BY)) * ZPER;
  const int64_t M = (int64_t)res + 1;
  const dim3 grid((unsigned)((M + BX - 1) / BX), (unsigned)((M + BY - 1) / BY), (unsigned)((M + BZ - 1) / BZ));
  kEvalGridBricks<BX, BY, ZPER><<<grid, kBrickThreads, 0, ctx->stream>>>(P, lam, o, vs, res, field);
  ITS_LAUNCHED(ctx);
  return ITS_OK;
}

// Corners per axis of the cell box that n consecutive lattice points span at the finest depth
// (one more than the exact bound, for the rounding of the cell quotients).
static double boxCorners(int n, double v, double w0) { return std::floor((n - 1) * std::fabs(v) / w0) + 3; }

template <typename T>
static its_status evalGridTuned(its_ctx* ctx, const SvoDevice& d, const double* lam, double3 o, double3 vs, int res,
                                T* field) {
  const EvalParams P = evalParams(d);
  // Every candidate computes the same bits for its type. Grids at least about twice as fine as the
  // octree (the brick's finest cell box fits the small tile): FP64, four brick shapes of the
  // point-wise kernel and the separable kernel with 4 or 8 points per thread along z; FP32, the
  // separable kernel's two shapes. Coarser grids: the separable kernel with the large tile, the
  // deeper brick by default where its box fits (torus of 99,000 faces, octree 256, grid 256: 3.52
  // ms point by point in bricks of 32 x 4 x 8).
  auto boxFits = [&](int z, int cap) {
    return boxCorners(kSepX, vs.x, d.unit[0]) * boxCorners(kSepY, vs.y, d.unit[0]) * boxCorners(z, vs.z, d.unit[0]) <=
           cap;
  };
  std::vector<int> cand;
  const bool coarse = !boxFits(4, kSepTileCap);
  if (!coarse) {
    if (sizeof(T) == 8) cand = {0, 1, 2, 3};
    cand.push_back(4);
    if (boxFits(8, kSepTileCap)) cand.push_back(5);
  } else {
    cand = {6};
    if (boxFits(8, kCoarseTileCap)) cand.push_back(7);
  }
  // the separable kernel's hat tables, formed once for all its launches here
  DevBuf<double> tabH;
  DevBuf<int> tabC;
  const int64_t M = (int64_t)res + 1, n = (int64_t)d.depth * 3 * M;
  its_status st = tabH.alloc(ctx, 4 * n);
  if (st == ITS_OK) st = tabC.alloc(ctx, n);
  if (st != ITS_OK) return st;
  kSepTables<<<gridFor(n, 256), 256, 0, ctx->stream>>>(P, o, vs, M, tabH.p, tabC.p);
  ITS_LAUNCHED(ctx);
  auto run = [&](int j) -> its_status {
    switch (cand[j]) {
      case 4: return launchSep<T, 4, false>(ctx, P, lam, tabH.p, tabC.p, res, field);
      case 5: return launchSep<T, 8, false>(ctx, P, lam, tabH.p, tabC.p, res, field);
      case 6: return launchSep<T, 4, true>(ctx, P, lam, tabH.p, tabC.p, res, field);
      case 7: return launchSep<T, 8, true>(ctx, P, lam, tabH.p, tabC.p, res, field);
    }
    if constexpr (sizeof(T) == 8) {
      switch (cand[j]) {
        case 1: return launchBricks<32, 8, 2>(ctx, P, lam, o, vs, res, field);
        case 2: return launchBricks<64, 4, 2>(ctx, P, lam, o, vs, res, field);
        case 3: return launchBricks<16, 4, 4>(ctx, P, lam, o, vs, res, field);
        default: return launchBricks<32, 4, 4>(ctx, P, lam, o, vs, res, field);
      }
    }
    return ITS_ERR_STATE;
  };
  // (a choice is a place in the list, and the box decides between two lists: a key for each)
  const std::string key = std::string("eval_grid/") + (sizeof(T) == 8 ? "f64" : "f32") + "/grid=" +
                          std::to_string(res) + "/octree=" + std::to_string(d.res) + "/depth=" + std::to_string(d.depth) +
                          (coarse ? "/coarse" : "");
  int choice = 0;
  st = tuneChoice(ctx, key, (int)cand.size(), (int)cand.size() - 1, run, &choice);
  if (st != ITS_OK) return st;
  return run(choice);
}

// divRn against the hardware-correct quotient (a test hook: out[i] = 1 where they differ).
__global__ void kCheckDivRn(const double* __restrict__ a, const double* __restrict__ b, int64_t n,
                            unsigned char* __restrict__ differ) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double y = 1.0 / b[i];
  const double q1 = divRn(a[i], b[i], y), q2 = a[i] / b[i];
  differ[i] = __double_as_longlong(q1) != __double_as_longlong(q2);
}

// ThinShells::getPointValGradient (ThinShells.cpp:1800-1866): a point outside the model box
// moves halfway towards its previous position until inside (at most 64 halvings; no move
// without previous positions), then the field and its gradient over its fine node's chain,
// with de_BaseFunction (BSpline.hpp:30-57) for the derivative factors.
__device__ __forceinline__ double deHat1(double x, double p, double w) {
  if (fabs(x - (p - w)) < 1e-9 || x < p - w || fabs(x - (p + w)) < 1e-9 || x > p + w) return 0.0;
  if (x <= p) return 1 / w;
  return -1 / w;
}

__global__ void kPointGradient(const __grid_constant__ EvalParams P, const double* __restrict__ lambda,
                               const double* __restrict__ pts, const double* __restrict__ before, int64_t m, double3 lo,
                               double3 hi, double* __restrict__ val, double* __restrict__ grad,
                               uint8_t* __restrict__ missing) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  double px = pts[3 * i], py = pts[3 * i + 1], pz = pts[3 * i + 2];
  if (before) {
    const double bx = before[3 * i], by = before[3 * i + 1], bz = before[3 * i + 2];
    for (int it = 0; it < 64; ++it) {
      if (!(px < lo.x || py < lo.y || pz < lo.z || px > hi.x || py > hi.y || pz > hi.z)) break;
      px = (px + bx) / 2.0;
      py = (py + by) / 2.0;
      pz = (pz + bz) / 2.0;
    }
  }
  double sum = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
  bool found = false;
  const int dx = (int)((px - P.g.x) / P.w0), dy = (int)((py - P.g.y) / P.w0), dz = (int)((pz - P.g.z) / P.w0);
  if (dx >= 0 && dy >= 0 && dz >= 0 && dx < P.res && dy < P.res && dz < P.res) {
    const uint32_t t0 = fineNodeOf(P.fineOcc, P.fineRank, mortonEncode((uint32_t)dx, (uint32_t)dy, (uint32_t)dz));
    if (t0 != kNone) {
      found = true;
      uint32_t t = t0;
      for (int d = 0; d < P.depth && t != kNone; ++d) {
        uint32_t X, Y, Z;
        mortonDecode(P.morton[t], X, Y, Z);
        const double w = P.w0 * (double)(1u << d);
        const double bx = latticePos(P.g.x, w, X), by = latticePos(P.g.y, w, Y), bz = latticePos(P.g.z, w, Z);
        const LatticeIndex& L = P.lat[d];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int ox = k & 1, oy = (k >> 1) & 1, oz = (k >> 2) & 1;
          const double cx = ox ? bx + w : bx, cy = oy ? by + w : by, cz = oz ? bz + w : bz;
          const double lam = lambda[latticeRank(L, ((X + ox) * L.M + (Y + oy)) * L.M + (Z + oz))];
          sum += lam * hat3(cx, cy, cz, w, px, py, pz);
          const double hx = hat1(px, cx, w), hy = hat1(py, cy, w), hz = hat1(pz, cz, w);
          gx += lam * (deHat1(px, cx, w) * hy * hz);
          gy += lam * (hx * deHat1(py, cy, w) * hz);
          gz += lam * (hx * hy * deHat1(pz, cz, w));
        }
        t = P.parent[t];
      }
    }
  }
  val[i] = sum;
  grad[3 * i] = gx;
  grad[3 * i + 1] = gy;
  grad[3 * i + 2] = gz;
  if (missing) missing[i] = found ? 0 : 1;
}

// Point queries (ThinShells::multiPointQuery, ThinShells.cpp:1183-1420, CUDA branch
// cuAcc::cpPointQuery, CUDACompute.cu:1070-1156): points outside the model box grown by one
// box width on every side take the outer iso value; the others the field. Label: 1 when the
// value >= outer, -1 when <= inner, else 0 (inside the shell).
__global__ void kPointQuery(const __grid_constant__ EvalParams P, const double* __restrict__ lambda,
                            const double* __restrict__ pts, int64_t m, double3 lo, double3 hi, double inner,
                            double outer, double* __restrict__ values, int8_t* __restrict__ labels) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  const double px = pts[3 * i], py = pts[3 * i + 1], pz = pts[3 * i + 2];
  const bool outside = px < lo.x || py < lo.y || pz < lo.z || px > hi.x || py > hi.y || pz > hi.z;
  const double v = outside ? outer : fieldAt(P, lambda, px, py, pz);
  if (values) values[i] = v;
  if (labels) labels[i] = (int8_t)(v >= outer ? 1 : (v <= inner ? -1 : 0));
}

}  // namespace its

using namespace its;

extern "C" {

its_status its_eval_points(its_svo* s, const double* lambda, const double* points, int64_t npoints, double* out,
                           uint8_t* missing) {
  if (!s || !lambda || (!points && npoints) || (!out && npoints) || npoints < 0) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  if (npoints == 0) return ITS_OK;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<double> L, P;
  OutArg<double> O;
  OutArg<uint8_t> Mi;
  its_status st;
  if ((st = L.stage(ctx, lambda, s->d.numVerts)) != ITS_OK) return st;
  if ((st = P.stage(ctx, points, 3 * npoints)) != ITS_OK) return st;
  if ((st = O.stage(ctx, out, npoints)) != ITS_OK) return st;
  if ((st = Mi.stage(ctx, missing, npoints)) != ITS_OK) return st;
  kEvalPoints<<<gridFor(npoints, 128), 128, 0, ctx->stream>>>(evalParams(s->d), L.d, P.d, npoints, O.d, Mi.d);
  ITS_LAUNCHED(ctx);
  if ((st = O.finish(ctx)) != ITS_OK) return st;
  if ((st = Mi.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_shell_iso_values(its_svo* s, const double* lambda, const double* points, int64_t npoints, double* inner,
                                double* outer, int64_t* num_missing) {
  if (!s || !lambda || !points || npoints <= 0 || !inner || !outer) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<double> L, P;
  its_status st;
  if ((st = L.stage(ctx, lambda, s->d.numVerts)) != ITS_OK) return st;
  if ((st = P.stage(ctx, points, 3 * npoints)) != ITS_OK) return st;
  const unsigned blocks = (unsigned)std::min<int64_t>(gridFor(npoints, 256), (int64_t)ctx->numSMs * 8);
  DevBuf<double> pmin, pmax;
  DevBuf<unsigned long long> pmiss;
  if ((st = pmin.alloc(ctx, blocks)) != ITS_OK) return st;
  if ((st = pmax.alloc(ctx, blocks)) != ITS_OK) return st;
  if ((st = pmiss.alloc(ctx, blocks)) != ITS_OK) return st;
  kIsoPartials<<<blocks, 256, 0, ctx->stream>>>(evalParams(s->d), L.d, P.d, npoints, pmin.p, pmax.p, pmiss.p);
  ITS_LAUNCHED(ctx);
  std::vector<double> hmin(blocks), hmax(blocks);
  std::vector<unsigned long long> hmiss(blocks);
  ITS_CU(ctx, cudaMemcpyAsync(hmin.data(), pmin.p, blocks * 8, cudaMemcpyDeviceToHost, ctx->stream));
  ITS_CU(ctx, cudaMemcpyAsync(hmax.data(), pmax.p, blocks * 8, cudaMemcpyDeviceToHost, ctx->stream));
  ITS_CU(ctx, cudaMemcpyAsync(hmiss.data(), pmiss.p, blocks * 8, cudaMemcpyDeviceToHost, ctx->stream));
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  double lo = DBL_MAX, hi = -DBL_MAX;
  unsigned long long miss = 0;
  for (unsigned k = 0; k < blocks; ++k) {
    lo = std::min(lo, hmin[k]);
    hi = std::max(hi, hmax[k]);
    miss += hmiss[k];
  }
  if (miss == (unsigned long long)npoints) return setError(ctx, ITS_ERR_INVALID, "no point lies in a fine node");
  *inner = lo;
  *outer = hi;
  if (num_missing) *num_missing = (int64_t)miss;
  return ITS_OK;
}

its_status its_point_query(its_svo* s, const double* lambda, const double* points, int64_t npoints,
                           const double box_origin[3], const double box_end[3], double inner, double outer,
                           double* values, int8_t* labels) {
  if (!s || !lambda || !box_origin || !box_end || npoints < 0 || (npoints && !points)) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  if (npoints == 0) return ITS_OK;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<double> L, P;
  OutArg<double> Va;
  OutArg<int8_t> La;
  its_status st;
  if ((st = L.stage(ctx, lambda, s->d.numVerts)) != ITS_OK) return st;
  if ((st = P.stage(ctx, points, 3 * npoints)) != ITS_OK) return st;
  if ((st = Va.stage(ctx, values, npoints)) != ITS_OK) return st;
  if ((st = La.stage(ctx, labels, npoints)) != ITS_OK) return st;
  // minRange = boxOrigin - boxWidth, maxRange = boxEnd + boxWidth (ThinShells.cpp:1198-1199)
  double lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    const double w = box_end[a] - box_origin[a];
    lo[a] = box_origin[a] - w;
    hi[a] = box_end[a] + w;
  }
  kPointQuery<<<gridFor(npoints, 128), 128, 0, ctx->stream>>>(evalParams(s->d), L.d, P.d, npoints,
                                                             make_double3(lo[0], lo[1], lo[2]),
                                                             make_double3(hi[0], hi[1], hi[2]), inner, outer, Va.d, La.d);
  ITS_LAUNCHED(ctx);
  if ((st = Va.finish(ctx)) != ITS_OK) return st;
  if ((st = La.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_point_value_gradient(its_svo* s, const double* lambda, const double* points, const double* before,
                                   int64_t npoints, const double box_origin[3], const double box_end[3], double* values,
                                   double* gradients, uint8_t* missing) {
  if (!s || !lambda || npoints < 0 || (npoints && (!points || !values || !gradients)) || !box_origin || !box_end)
    return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  if (npoints == 0) return ITS_OK;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<double> L, P, B;
  OutArg<double> Vo, G;
  OutArg<uint8_t> Mi;
  its_status st;
  if ((st = L.stage(ctx, lambda, s->d.numVerts)) != ITS_OK || (st = P.stage(ctx, points, 3 * npoints)) != ITS_OK ||
      (st = B.stage(ctx, before, before ? 3 * npoints : 0)) != ITS_OK || (st = Vo.stage(ctx, values, npoints)) != ITS_OK ||
      (st = G.stage(ctx, gradients, 3 * npoints)) != ITS_OK || (st = Mi.stage(ctx, missing, npoints)) != ITS_OK)
    return st;
  kPointGradient<<<gridFor(npoints, 128), 128, 0, ctx->stream>>>(
      evalParams(s->d), L.d, P.d, B.d, npoints, make_double3(box_origin[0], box_origin[1], box_origin[2]),
      make_double3(box_end[0], box_end[1], box_end[2]), Vo.d, G.d, Mi.d);
  ITS_LAUNCHED(ctx);
  if ((st = Vo.finish(ctx)) != ITS_OK || (st = G.finish(ctx)) != ITS_OK || (st = Mi.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_eval_grid(its_svo* s, const double* lambda, const double origin[3], const double width[3], int res,
                         double* field) {
  if (!s || !lambda || !origin || !width || !field || res < 1 || res > 2048) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  const int64_t M = (int64_t)res + 1, total = M * M * M;
  InArg<double> L;
  OutArg<double> F;
  its_status st;
  if ((st = L.stage(ctx, lambda, s->d.numVerts)) != ITS_OK) return st;
  if ((st = F.stage(ctx, field, total)) != ITS_OK) return st;
  const double3 o = make_double3(origin[0], origin[1], origin[2]);
  const double3 vs = make_double3(width[0] / res, width[1] / res, width[2] / res);
  if ((st = evalGridTuned<double>(ctx, s->d, L.d, o, vs, res, F.d)) != ITS_OK) return st;
  if ((st = F.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_eval_grid_f32(its_svo* s, const double* lambda, const double origin[3], const double width[3], int res,
                             float* field) {
  if (!s || !lambda || !origin || !width || !field || res < 1 || res > 2048) return ITS_ERR_INVALID;
  its_ctx* ctx = s->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  const int64_t M = (int64_t)res + 1, total = M * M * M;
  InArg<double> L;
  OutArg<float> F;
  its_status st;
  if ((st = L.stage(ctx, lambda, s->d.numVerts)) != ITS_OK) return st;
  if ((st = F.stage(ctx, field, total)) != ITS_OK) return st;
  const double3 o = make_double3(origin[0], origin[1], origin[2]);
  const double3 vs = make_double3(width[0] / res, width[1] / res, width[2] / res);
  if ((st = evalGridTuned<float>(ctx, s->d, L.d, o, vs, res, F.d)) != ITS_OK) return st;
  if ((st = F.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

// Counts the pairs (a[i], b[i]) whose quotient by divRn differs from a[i] / b[i] (device or
// host arrays). A self-check of the division the field kernels use.
its_status its_check_division(its_ctx* ctx, const double* a, const double* b, int64_t n, int64_t* mismatches) {
  if (!ctx || !a || !b || n <= 0 || !mismatches) return ITS_ERR_INVALID;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<double> A, B;
  its_status st;
  if ((st = A.stage(ctx, a, n)) != ITS_OK || (st = B.stage(ctx, b, n)) != ITS_OK) return st;
  DevBuf<unsigned char> diff;
  if ((st = diff.alloc(ctx, n)) != ITS_OK) return st;
  kCheckDivRn<<<gridFor(n, 256), 256, 0, ctx->stream>>>(A.d, B.d, n, diff.p);
  ITS_LAUNCHED(ctx);
  std::vector<unsigned char> h(n);
  ITS_CU(ctx, cudaMemcpyAsync(h.data(), diff.p, n, cudaMemcpyDeviceToHost, ctx->stream));
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  int64_t c = 0;
  for (int64_t i = 0; i < n; ++i) c += h[i];
  *mismatches = c;
  return ITS_OK;
}

}  // extern "C"

namespace {
template <typename FT>
its_status marchingCubesT(its_ctx* ctx, const FT* field, int res, const double origin[3], const double width[3],
                          double iso, uint8_t* cube_index, double* tri_verts, int64_t capacity, int64_t* num_verts) {
  if (!ctx) return ITS_ERR_INVALID;
  if (!field || !origin || !width || res < 1 || res > 2048 || !num_verts)
    return setError(ctx, ITS_ERR_INVALID, "its_marching_cubes: bad arguments");
  if (tri_verts && capacity < 0) return setError(ctx, ITS_ERR_INVALID, "negative capacity");
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  const int64_t M = (int64_t)res + 1, nvox = (int64_t)res * res * res;
  InArg<FT> F;
  OutArg<uint8_t> Cb;
  OutArg<double> T;
  its_status st;
  if ((st = F.stage(ctx, field, M * M * M)) != ITS_OK) return st;
  if ((st = Cb.stage(ctx, cube_index, nvox)) != ITS_OK) return st;
  if ((st = T.stage(ctx, tri_verts, tri_verts ? 3 * capacity : 0)) != ITS_OK) return st;
  McCaseT<FT> mc{F.d, res, iso};
  // case bytes: the caller's buffer when it is on the device, else scratch copied back
  DevBuf<uint8_t> cubeTmp;
  uint8_t* cubeD = Cb.d;
  if (!cubeD) {
    if ((st = cubeTmp.alloc(ctx, nvox)) != ITS_OK) return st;
    cubeD = cubeTmp.p;
  }
  // tiles of 32 lanes x ITEMS voxels; the autotuner picks ITEMS (same bits for every choice)
  const int itemsOf[3] = {8, 16, 4};
  const int64_t points = M * M * M, signBlocks = (points + 32 * kSignWords * (kScanThreads / 32) - 1) /
                                                 (32 * kSignWords * (kScanThreads / 32));
  const int64_t signWords = signBlocks * (kScanThreads / 32) * kSignWords + 1;  // a window reads the word after its own
  // one scratch for all: the total, the listed tiles' counter, the tiles' sums, their list, the signs
  // (with five allocations and ordinary launches 64^3 took 62 us, now 50)
  DevBuf<unsigned long long> scratch;
  unsigned long long *tot = nullptr, *sums = nullptr;
  unsigned* numListed = nullptr;
  uint32_t *listed = nullptr, *signs = nullptr;
  auto place = [&](int64_t nt) -> its_status {
    const int64_t ns = nt + spineTops(nt), nl = T.d ? (nt + 1) / 2 : 0, need = 2 + ns + nl + (signWords + 1) / 2;
    if ((int64_t)scratch.n < need && (st = scratch.alloc(ctx, need)) != ITS_OK) return st;
    tot = scratch.p;
    numListed = (unsigned*)(scratch.p + 1);
    sums = scratch.p + 2;
    listed = T.d ? (uint32_t*)(sums + ns) : nullptr;
    signs = (uint32_t*)(sums + ns + nl);
    return ITS_OK;
  };
  const double3 o3 = make_double3(origin[0], origin[1], origin[2]);
  const double3 v3 = make_double3(width[0] / res, width[1] / res, width[2] / res);
  auto runTiles = [&](auto itemsTag) -> its_status {
    constexpr int kItems = decltype(itemsTag)::value;
    const int64_t nt = (nvox + 32 * kItems - 1) / (32 * kItems);
    if ((st = place(nt)) != ITS_OK) return st;
    kMcSigns<FT><<<(unsigned)signBlocks, kScanThreads, 0, ctx->stream>>>(F.d, points, iso, signs, numListed);
    ITS_LAUNCHED(ctx);
    // four tiles per warp once that many keep every SM full of warps
    constexpr int kWarps = kScanThreads / 32;
    const bool four = nt >= 4ll * 64 * ctx->numSMs;
    const int64_t perBlock = (four ? 4 : 1) * kWarps;
    auto* cases = four ? kMcCases<kItems, 4> : kMcCases<kItems, 1>;
    if ((st = launchDependent(ctx, true, cases, (unsigned)((nt + perBlock - 1) / perBlock), kScanThreads, 0, ctx->stream,
                              (const uint32_t*)signs, res, fastDiv(res), cubeD, nt, sums, listed, numListed)) != ITS_OK)
      return st;
    if ((st = scanSpine<unsigned long long>(ctx, sums, nt, tot, sums + nt)) != ITS_OK) return st;
    if (!T.d) return ITS_OK;
    return launchDependent(ctx, true, kMcEmit<FT, kItems>,
                           (unsigned)std::min<int64_t>((nt + kWarps - 1) / kWarps, 8ll * ctx->numSMs), kScanThreads, 0,
                           ctx->stream, mc, fastDiv(res), o3, v3, (const uint8_t*)cubeD, (const unsigned long long*)sums,
                           (const uint32_t*)listed, (const unsigned*)numListed, T.d, (unsigned long long)capacity);
  };
  auto run = [&](int i) -> its_status {
    if (itemsOf[i] == 16) return runTiles(std::integral_constant<int, 16>());
    if (itemsOf[i] == 4) return runTiles(std::integral_constant<int, 4>());
    return runTiles(std::integral_constant<int, 8>());
  };
  const std::string key = std::string("marching_cubes/") + (sizeof(FT) == 8 ? "f64" : "f32") + "/res=" +
                          std::to_string(res) + (T.d ? "/soup" : "/cases");
  int choice = 0;
  // By default the shortest runs on small grids, so that every SM has warps, and longer ones as the
  // grid grows (us with 4, 8, 16 voxels per lane: 67^3 62, 70, 85; 128^3 79, 84, 96; 330^3 219, 190,
  // 200; 512^3 477, 376, 328).
  const int def = nvox < (1ll << 22) ? 2 : (nvox < (1ll << 26) ? 0 : 1);
  if ((st = tuneChoice(ctx, key, 3, def, run, &choice)) != ITS_OK) return st;
  if ((st = run(choice)) != ITS_OK) return st;
  unsigned long long total = 0;
  if ((st = readScalar(ctx, (const unsigned long long*)tot, &total)) != ITS_OK) return st;
  *num_verts = (int64_t)total;
  // only the vertices written leave the device (the rest of a host buffer is left untouched)
  T.count = 3 * (size_t)std::min<int64_t>(capacity, (int64_t)total);
  if ((st = Cb.finish(ctx)) != ITS_OK) return st;
  if ((st = T.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}
}  // namespace

extern "C" {

its_status its_marching_cubes(its_ctx* ctx, const double* field, int res, const double origin[3],
                              const double width[3], double iso, uint8_t* cube_index, double* tri_verts,
                              int64_t capacity, int64_t* num_verts) {
  return marchingCubesT<double>(ctx, field, res, origin, width, iso, cube_index, tri_verts, capacity, num_verts);
}

its_status its_marching_cubes_f32(its_ctx* ctx, const float* field, int res, const double origin[3],
                                  const double width[3], double iso, uint8_t* cube_index, double* tri_verts,
                                  int64_t capacity, int64_t* num_verts) {
  return marchingCubesT<float>(ctx, field, res, origin, width, iso, cube_index, tri_verts, capacity, num_verts);
}

}  // extern "C"
