// Cubic B-spline basis (its_cubic.cuh): the field at points and on a lattice, and the offset
// shell samples. No counterpart in the reference (degree-1 hats, corner-vertex samples).
#include <algorithm>
#include <cmath>

#include "its_cubic.cuh"
#include "its_scan.cuh"
#include "its_sparse.cuh"

namespace its {

__global__ void __launch_bounds__(128) kCubicEvalPoints(const __grid_constant__ CubicGen g,
                                                        const double* __restrict__ lambda,
                                                        const double* __restrict__ P, int64_t m,
                                                        double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  const double x[3] = {P[3 * i], P[3 * i + 1], P[3 * i + 2]};
  out[i] = g.eval(x, lambda);
}

// ---- the field on a lattice -------------------------------------------------------------------
// Lattice point (ix, iy, iz), x fastest, at o + i * vs, vs = width / res. A point's weights along an
// axis depend only on its coordinate there, so kCubicTables forms them once per grid coordinate
// and depth (the first of its four lattice points and their weights); a block takes a brick of
// 32 x 8 x kZ points, copies its slices and stages every depth's box of coefficients (0 where
// the lattice point is no vertex) in shared memory; a thread sums a column of kZ points, lattice
// columns (kx, ky) without a vertex left out, a coefficient read once for the points of its
// column that share a cell. The terms come in CubicGen's order with its products; those of absent
// vertices add +0 to a sum that is never -0, so the field is that of the point-wise evaluation bit
// for bit. At 129^3 points on an octree of 32 cells a side the point-wise kernel (bitmap, rank and
// weights per point and lattice point) took 1.10 ms, this one 0.17.
constexpr int kCubX = 32, kCubY = 8, kCubThreads = kCubX * kCubY;
constexpr int kCubMaxStage = 11264;  // staged coefficients: 88 KB, so that two blocks fit an SM

__global__ void kCubicTables(const __grid_constant__ CubicGen g, double3 o, double3 vs, int64_t M,
                             double* __restrict__ tabW, int* __restrict__ tabB) {
  const int64_t item = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (item >= (int64_t)g.depth * 3 * M) return;
  const int d = (int)(item / (3 * M)), a = (int)((item / M) % 3);
  const int64_t i = item % M;
  const double x[3] = {o.x + (double)i * vs.x, o.y + (double)i * vs.y, o.z + (double)i * vs.z};
  double u[3];
  g.pointU(x, d, u);
  const double f = floor(u[a]);
  const int64_t lim = g.lat[d].M;
  double w[4] = {0.0, 0.0, 0.0, 0.0};
  int base = -5;  // away from the lattice, or not a number: weights 0 on no lattice point
  if (f >= -3.0 && f <= (double)lim + 1.0) {
    base = (int)f - 1;
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = bspline3(u[a] - (double)(base + j));
  } else if (f > 0.0) {
    base = (int)lim + 1;
  }
  double2* dst = (double2*)(tabW + 4 * item);
  dst[0] = make_double2(w[0], w[1]);
  dst[1] = make_double2(w[2], w[3]);
  tabB[item] = base;
}

template <int kZ>
struct alignas(16) CubStage {
  double wX[kMaxDepth][4][kCubX], wY[kMaxDepth][kCubY][4], wZ[kMaxDepth][4][kZ];
  int bX[kMaxDepth][kCubX], bY[kMaxDepth][kCubY], bZ[kMaxDepth][kZ];
  int off[kMaxDepth], colOff[kMaxDepth + 1], ny[kMaxDepth], nz[kMaxDepth];  // off -1: no box
  int any[kMaxDepth], odd[kMaxDepth];  // some coefficient; one that is not finite
};

// The terms of lattice column (kx, ky) for the G points q0.. of a thread's column, which share a cell.
template <int G, int kZ>
__device__ __forceinline__ void cubicColumn(const CubStage<kZ>& S, int d, double wxy, const double* __restrict__ lam,
                                            int q0, double (&acc)[kZ]) {
#pragma unroll
  for (int jz = 0; jz < 4; ++jz) {
    const double l = lam[jz];
#pragma unroll
    for (int q = 0; q < G; ++q) acc[q0 + q] = acc[q0 + q] + wxy * S.wZ[d][jz][q0 + q] * l;
  }
}

template <int kZ>
__global__ void __launch_bounds__(kCubThreads, 3) kCubicEvalGrid(const __grid_constant__ CubicGen g,
                                                              const double* __restrict__ lambda, double3 o, double3 vs,
                                                              const double* __restrict__ tabW,
                                                              const int* __restrict__ tabB, int64_t M, int stageCap,
                                                              double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char cubRaw[];
  CubStage<kZ>& S = *(CubStage<kZ>*)cubRaw;
  double* tLam = (double*)(cubRaw + sizeof(CubStage<kZ>));
  unsigned char* tCol = (unsigned char*)(tLam + stageCap);  // per (x, y) column of a box: any vertex
  const int tid = threadIdx.x, tx = tid % kCubX, ty = tid / kCubX, D = g.depth;
  const int64_t first[3] = {(int64_t)blockIdx.x * kCubX, (int64_t)blockIdx.y * kCubY, (int64_t)blockIdx.z * kZ};
  constexpr int kCoords = kCubX + kCubY + kZ;
  for (int item = tid; item < kCoords * D; item += kCubThreads) {
    const int d = item / kCoords, j = item % kCoords;
    const int a = j < kCubX ? 0 : (j < kCubX + kCubY ? 1 : 2);
    const int k = a == 0 ? j : (a == 1 ? j - kCubX : j - kCubX - kCubY);
    const int64_t at = first[a] + k < M ? first[a] + k : M - 1;  // clamped to the grid
    const int64_t r = ((int64_t)d * 3 + a) * M + at;
    const double2 w01 = __ldg((const double2*)(tabW + 4 * r)), w23 = __ldg((const double2*)(tabW + 4 * r) + 1);
    const double w[4] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll
    for (int e = 0; e < 4; ++e) (a == 0 ? S.wX[d][e][k] : a == 1 ? S.wY[d][k][e] : S.wZ[d][e][k]) = w[e];
    (a == 0 ? S.bX[d] : a == 1 ? S.bY[d] : S.bZ[d])[k] = __ldg(tabB + r);
  }
  __syncthreads();
  if (tid == 0) {  // where each depth's box goes (a lattice that runs backwards has none)
    int off = 0, cols = 0;
    for (int d = 0; d < D; ++d) {
      const int nx = S.bX[d][kCubX - 1] - S.bX[d][0] + 4, ny = S.bY[d][kCubY - 1] - S.bY[d][0] + 4,
                nz = S.bZ[d][kZ - 1] - S.bZ[d][0] + 4;
      const bool fits = nx >= 4 && ny >= 4 && nz >= 4 && (int64_t)nx * ny * nz <= stageCap - off;
      S.off[d] = fits ? off : -1;
      S.colOff[d] = cols;
      S.ny[d] = ny;
      S.nz[d] = nz;
      S.any[d] = S.odd[d] = 0;
      if (fits) {
        off += nx * ny * nz;
        cols += nx * ny;
      }
    }
    S.colOff[D] = cols;
  }
  __syncthreads();
  for (int e = tid; e < S.colOff[D]; e += kCubThreads) {  // a thread per (x, y) column of a box
    int d = 0;
    while (e >= S.colOff[d + 1]) ++d;
    const LatticeIndex& L = g.lat[d];
    const int ny = S.ny[d], nz = S.nz[d], col = e - S.colOff[d];
    const int X = S.bX[d][0] + col / ny, Y = S.bY[d][0] + col % ny, Z0 = S.bZ[d][0], m = (int)L.M;
    double* dst = tLam + S.off[d] + col * nz;
    const bool in = X >= 0 && Y >= 0 && X < m && Y < m;
    const uint32_t base = in ? ((uint32_t)X * L.M + (uint32_t)Y) * L.M : 0u;
    bool some = false, odd = false;
    for (int z = 0; z < nz; ++z) {
      double l = 0.0;
      if (in && Z0 + z >= 0 && Z0 + z < m && latticeHas(L, base + (uint32_t)(Z0 + z))) {
        l = lambda[latticeRank(L, base + (uint32_t)(Z0 + z))];
        some = true;
        odd = odd || !isfinite(l);
      }
      dst[z] = l;
    }
    tCol[e] = some;
    if (some) S.any[d] = 1;  // benign races: every writer stores 1
    if (odd) S.odd[d] = 1;
  }
  __syncthreads();
  const int64_t xi = first[0] + tx, yj = first[1] + ty;
  if (xi >= M || yj >= M) return;
  double acc[kZ];
#pragma unroll
  for (int q = 0; q < kZ; ++q) acc[q] = 0.0;
  for (int d = 0; d < D; ++d) {
    if (S.off[d] < 0 || S.odd[d]) {  // point by point (a zero weight leaves its lattice points out)
      for (int q = 0; q < kZ; ++q) {
        if (first[2] + q >= M) break;
        const double x[3] = {o.x + (double)xi * vs.x, o.y + (double)yj * vs.y, o.z + (double)(first[2] + q) * vs.z};
        double s = 0.0;
#pragma unroll
        for (int e = 0; e < kZ; ++e) s = e == q ? acc[e] : s;
        g.rowDepth(d, [&](int dd, double* u) { g.pointU(x, dd, u); },
                   [&](int32_t c, double v) { s = s + v * lambda[c]; });
#pragma unroll
        for (int e = 0; e < kZ; ++e) acc[e] = e == q ? s : acc[e];
      }
      continue;
    }
    if (!S.any[d]) continue;
    const int ny = S.ny[d], nz = S.nz[d];
    const int rx = S.bX[d][tx] - S.bX[d][0], ry = S.bY[d][ty] - S.bY[d][0], z0 = S.bZ[d][0];
    const bool one = nz == 4;  // the brick's z run lies in one cell (block-uniform, as the runs below)
    for (int jx = 0; jx < 4; ++jx) {
      const double wx = S.wX[d][jx][tx];
#pragma unroll
      for (int jy = 0; jy < 4; ++jy) {
        const int col = (rx + jx) * ny + ry + jy;
        if (!tCol[S.colOff[d] + col]) continue;
        const double wxy = wx * S.wY[d][ty][jy];
        const double* lam = tLam + S.off[d] + col * nz;
        if (one) {
          cubicColumn<kZ>(S, d, wxy, lam, 0, acc);
        } else {
#pragma unroll
          for (int q = 0; q < kZ; q += 4) {
            const int a = S.bZ[d][q] - z0, b = S.bZ[d][q + 1] - z0, c = S.bZ[d][q + 2] - z0, e = S.bZ[d][q + 3] - z0;
            if (a == e) {
              cubicColumn<4>(S, d, wxy, lam + a, q, acc);
            } else {
              if (a == b) {
                cubicColumn<2>(S, d, wxy, lam + a, q, acc);
              } else {
                cubicColumn<1>(S, d, wxy, lam + a, q, acc);
                cubicColumn<1>(S, d, wxy, lam + b, q + 1, acc);
              }
              if (c == e) {
                cubicColumn<2>(S, d, wxy, lam + c, q + 2, acc);
              } else {
                cubicColumn<1>(S, d, wxy, lam + c, q + 2, acc);
                cubicColumn<1>(S, d, wxy, lam + e, q + 3, acc);
              }
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kZ; ++q)
    if (first[2] + q < M) out[xi + M * (yj + M * (first[2] + q))] = acc[q];
}

// Coefficients that a brick of z points deep stages, at most, over the depths; -1 where they may not
// all fit, or where the lattice does not run forwards.
static int cubicStage(const SvoDevice& d, double3 vs, int64_t M, int z) {
  double n = 0.0;
  for (int k = 0; k < d.depth; ++k) {
    const double w = d.unit[0] * (double)(1u << k), all = (double)(d.res >> k) + 11.0;  // (cells are clamped)
    auto side = [&](int points, double v) {
      return std::min(std::floor((double)(std::min<int64_t>(points, M) - 1) * v / w + 1e-6) + 5.0, all);
    };
    n += side(kCubX, vs.x) * side(kCubY, vs.y) * side(z, vs.z);
  }
  return vs.x > 0.0 && vs.y > 0.0 && vs.z > 0.0 && n <= (double)kCubMaxStage ? (int)n : -1;
}

template <int kZ>
static its_status cubicGrid(its_ctx* ctx, const SvoDevice& d, const double* lam, double3 o, double3 vs, int64_t M,
                            int cap, double* out) {
  const CubicGen g = cubicGen(d, nullptr);
  const int64_t n = (int64_t)d.depth * 3 * M;
  DevBuf<double> tabW;
  DevBuf<int> tabB;
  its_status st;
  if ((st = tabW.alloc(ctx, 4 * n)) != ITS_OK || (st = tabB.alloc(ctx, n)) != ITS_OK) return st;
  kCubicTables<<<gridFor(n, 256), 256, 0, ctx->stream>>>(g, o, vs, M, tabW.p, tabB.p);
  ITS_LAUNCHED(ctx);
  // (a box column holds at least four entries)
  auto bytes = [](int entries) { return (int)sizeof(CubStage<kZ>) + entries * 8 + entries / 4 + 16; };
  // The attribute is the function's, for every thread of the process: the most that any call asks for,
  // so that a call in another context cannot lower it between here and the launch.
  ITS_CU(ctx, cudaFuncSetAttribute(kCubicEvalGrid<kZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes(kCubMaxStage)));
  const dim3 grid((unsigned)((M + kCubX - 1) / kCubX), (unsigned)((M + kCubY - 1) / kCubY), (unsigned)((M + kZ - 1) / kZ));
  kCubicEvalGrid<kZ><<<grid, kCubThreads, bytes(cap), ctx->stream>>>(g, lam, o, vs, tabW.p, tabB.p, M, cap, out);
  ITS_LAUNCHED(ctx);
  return ITS_OK;
}

// Lattice point i (x fastest), one thread each: for lattices too coarse for bricks.
__global__ void __launch_bounds__(128) kCubicEvalLattice(const __grid_constant__ CubicGen g,
                                                         const double* __restrict__ lambda, double3 o, double3 vs,
                                                         int64_t M, double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= M * M * M) return;
  const int64_t ix = i % M, iy = (i / M) % M, iz = i / (M * M);
  const double x[3] = {o.x + (double)ix * vs.x, o.y + (double)iy * vs.y, o.z + (double)iz * vs.z};
  out[i] = g.eval(x, lambda);
}

// Start of each vertex's run in the vertex-sorted face corners (every pointer written once).
__global__ void kRunStarts(int64_t n, const uint32_t* __restrict__ keys, int64_t nv, int64_t* __restrict__ start) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i > n) return;
  const int64_t c = (i < n) ? (int64_t)keys[i] : nv;
  const int64_t prev = (i == 0) ? -1 : (int64_t)keys[i - 1];
  for (int64_t k = prev + 1; k <= c; ++k) start[k] = i;
}

// Unit area-weighted normal of every vertex (its faces' unnormalised normals summed in face
// order) and the two offset points with their targets.
__global__ void kOffsetSamples(const double* __restrict__ V, int64_t nv, const int32_t* __restrict__ F,
                               const int64_t* __restrict__ start, const uint32_t* __restrict__ corner, double eps,
                               double* __restrict__ pts, double* __restrict__ tgt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nv) return;
  double n[3] = {0.0, 0.0, 0.0};
  for (int64_t k = start[i]; k < start[i + 1]; ++k) {
    const int64_t f = corner[k] / 3;
    double p[3][3];
    for (int c = 0; c < 3; ++c)
      for (int a = 0; a < 3; ++a) p[c][a] = V[3 * (int64_t)F[3 * f + c] + a];
    const double u[3] = {p[1][0] - p[0][0], p[1][1] - p[0][1], p[1][2] - p[0][2]};
    const double v[3] = {p[2][0] - p[0][0], p[2][1] - p[0][1], p[2][2] - p[0][2]};
    n[0] = n[0] + (u[1] * v[2] - u[2] * v[1]);
    n[1] = n[1] + (u[2] * v[0] - u[0] * v[2]);
    n[2] = n[2] + (u[0] * v[1] - u[1] * v[0]);
  }
  double len = n[0] * n[0];
  len = len + n[1] * n[1];
  len = sqrt(len + n[2] * n[2]);
  double un[3] = {0.0, 0.0, 0.0};
  if (len > 0.0)
    for (int a = 0; a < 3; ++a) un[a] = n[a] / len;
  if (pts)
    for (int a = 0; a < 3; ++a) {
      pts[3 * i + a] = V[3 * i + a] + eps * un[a];
      pts[3 * (nv + i) + a] = V[3 * i + a] - eps * un[a];
    }
  if (tgt) {
    tgt[i] = eps;
    tgt[nv + i] = -eps;
  }
}

__global__ void kCornerKeys(const int32_t* __restrict__ F, int64_t n3, uint32_t* __restrict__ keys,
                            uint32_t* __restrict__ vals) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n3) return;
  keys[k] = (uint32_t)F[k];
  vals[k] = (uint32_t)k;
}

}  // namespace its

using namespace its;

extern "C" {

its_status its_eval_points_cubic(its_svo* svo, const double* lambda, const double* points, int64_t npoints,
                                 double* out) {
  if (!svo || !lambda || (npoints > 0 && (!points || !out)) || npoints < 0) return ITS_ERR_INVALID;
  its_ctx* ctx = svo->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  if (npoints == 0) return ITS_OK;
  InArg<double> L, P;
  OutArg<double> O;
  its_status st;
  if ((st = L.stage(ctx, lambda, svo->d.numVerts)) != ITS_OK || (st = P.stage(ctx, points, 3 * npoints)) != ITS_OK ||
      (st = O.stage(ctx, out, npoints)) != ITS_OK)
    return st;
  kCubicEvalPoints<<<gridFor(npoints, 128), 128, 0, ctx->stream>>>(cubicGen(svo->d, nullptr), L.d, P.d, npoints, O.d);
  ITS_LAUNCHED(ctx);
  if ((st = O.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_eval_grid_cubic(its_svo* svo, const double* lambda, const double origin[3], const double width[3],
                               int res, double* field) {
  if (!svo || !lambda || !origin || !width || !field || res < 1 || res > 2048) return ITS_ERR_INVALID;
  its_ctx* ctx = svo->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  const int64_t M = (int64_t)res + 1;
  InArg<double> L;
  OutArg<double> O;
  its_status st;
  if ((st = L.stage(ctx, lambda, svo->d.numVerts)) != ITS_OK || (st = O.stage(ctx, field, M * M * M)) != ITS_OK)
    return st;
  const double3 o = make_double3(origin[0], origin[1], origin[2]);
  const double3 vs = make_double3(width[0] / res, width[1] / res, width[2] / res);
  // Bricks where every depth's box fits, 8 points deep where two blocks per SM come of them, else 4
  // (65^3 points on an octree of 64: 101 us with 8, 76 with 4; 129^3 on one of 32: 175 and 207). Coarser
  // lattices point by point: a brick's threads would look the corners of a whole depth up for their
  // points, one after another (us by points and in bricks: 9^3 on an octree of 32 77 and 117, 33^3 on
  // 64 96 and 414, 65^3 on 256 277 and 640; where only the finest depth does not fit, bricks may win,
  // 129^3 on 256 1640 and 1030, or lose, 171^3 on 256 3590 and 4330).
  const int64_t deep = ((M + kCubX - 1) / kCubX) * ((M + kCubY - 1) / kCubY) * ((M + 7) / 8);
  const int cap8 = deep >= 2 * ctx->numSMs ? cubicStage(svo->d, vs, M, 8) : -1, cap4 = cubicStage(svo->d, vs, M, 4);
  if (cap8 >= 0) {
    st = cubicGrid<8>(ctx, svo->d, L.d, o, vs, M, cap8, O.d);
  } else if (cap4 >= 0) {
    st = cubicGrid<4>(ctx, svo->d, L.d, o, vs, M, cap4, O.d);
  } else {
    kCubicEvalLattice<<<gridFor(M * M * M, 128), 128, 0, ctx->stream>>>(cubicGen(svo->d, nullptr), L.d, o, vs, M, O.d);
    ITS_LAUNCHED(ctx);
  }
  if (st != ITS_OK) return st;
  if ((st = O.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

its_status its_offset_samples(its_ctx* ctx, const double* verts, int64_t nverts, const int32_t* faces, int64_t nfaces,
                              double eps, double* points, double* targets) {
  if (!ctx) return ITS_ERR_INVALID;
  if (!verts || nverts < 1 || nfaces < 0 || (nfaces > 0 && !faces) || !(eps == eps) || 3 * nfaces >= (1ll << 32) ||
      nverts >= (1ll << 32))
    return setError(ctx, ITS_ERR_INVALID, "its_offset_samples: bad arguments");
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  InArg<double> V;
  InArg<int32_t> F;
  OutArg<double> P, T;
  its_status st;
  if ((st = V.stage(ctx, verts, 3 * nverts)) != ITS_OK || (st = F.stage(ctx, faces, 3 * nfaces)) != ITS_OK ||
      (st = P.stage(ctx, points, 6 * nverts)) != ITS_OK || (st = T.stage(ctx, targets, 2 * nverts)) != ITS_OK)
    return st;
  if (nfaces > 0 && (st = validateMesh(ctx, V.d, nverts, F.d, nfaces)) != ITS_OK) return st;
  const int64_t n3 = 3 * nfaces;
  DevBuf<uint32_t> keys, vals, sk, sv, tk, tv;
  DevBuf<int64_t> start;
  if ((st = start.alloc(ctx, nverts + 1)) != ITS_OK) return st;
  if (n3 > 0) {
    if ((st = keys.alloc(ctx, n3)) != ITS_OK || (st = vals.alloc(ctx, n3)) != ITS_OK ||
        (st = sk.alloc(ctx, n3)) != ITS_OK || (st = sv.alloc(ctx, n3)) != ITS_OK || (st = tk.alloc(ctx, n3)) != ITS_OK ||
        (st = tv.alloc(ctx, n3)) != ITS_OK)
      return st;
    kCornerKeys<<<gridFor(n3, 256), 256, 0, ctx->stream>>>(F.d, n3, keys.p, vals.p);
    ITS_LAUNCHED(ctx);
    int bits = 1;
    while (bits < 32 && (1ll << bits) < nverts) ++bits;
    if ((st = radixSortPairs(ctx, keys.p, vals.p, sk.p, sv.p, tk.p, tv.p, n3, bits)) != ITS_OK) return st;
    kRunStarts<<<gridFor(n3 + 1, 256), 256, 0, ctx->stream>>>(n3, sk.p, nverts, start.p);
    ITS_LAUNCHED(ctx);
  } else {
    ITS_CU(ctx, cudaMemsetAsync(start.p, 0, (nverts + 1) * 8, ctx->stream));
  }
  kOffsetSamples<<<gridFor(nverts, 128), 128, 0, ctx->stream>>>(V.d, nverts, F.d, start.p, sv.p, eps, P.d, T.d);
  ITS_LAUNCHED(ctx);
  if ((st = P.finish(ctx)) != ITS_OK || (st = T.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

}  // extern "C"
