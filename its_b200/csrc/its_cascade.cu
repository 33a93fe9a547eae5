// Dense field on a lattice aligned with the octree, by prolongation.
//
// The field of MC::launch_computSDFKernel (MarchingCubes.cu:464-536, CUDACompute.cu:435-510)
// is F = sum over depths d of f_d, f_d(p) = sum over the depth-d corner vertices v of
// lambda_v * hat_v(p): on each depth-d lattice cell, the trilinear interpolant of the cell's
// corner coefficients (0 where the corner is not a vertex). When the output lattice is the
// octree's own box at res * 2^k points per axis, every output point sits on a dyadic point of
// every depth's lattice, and F can be built coarse to fine on dense per-depth lattices:
//   D_{root} = lambda at the root corners;   D_d = lambda at the depth-d corners + P(D_{d+1});
//   out = P^k(D_0),
// P the trilinear prolongation to the next finer lattice (a point between coarse points takes
// their mean: weights 1, 1/2, 1/4, 1/8 per point, exact in floating point). Each level is one
// pass over its lattice that reads an eighth as much: the cost is that of writing the output
// once (8 B per point), where evaluating every point from its cells at all depths
// (its_eval_grid, bit-identical to the reference's sums) is bound by hat arithmetic. The sums
// differ from the reference's by rounding only: the hats are centred on the exact lattice
// positions, the representative vertex positions of the octree differ from them by ulps.
#include <cmath>

#include "its_op.cuh"
#include "its_svo.cuh"

namespace its {

// Depth d's dense lattice: its first point and its points per axis.
template <typename T>
struct CascadeLevels {
  T* field[kMaxDepth];
  int M[kMaxDepth];
};

template <typename T>
__global__ void kScatterCorners(int64_t n, const uint64_t* __restrict__ vertKey, const double* __restrict__ lambda,
                                CascadeLevels<T> L) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v >= n) return;
  const VertCoord c = decodeVertKey(vertKey[v]);
  const int64_t M = L.M[c.d];
  L.field[c.d][c.X + M * (c.Y + M * (int64_t)c.Z)] = (T)lambda[v];
}

// fine = (kAdd ? fine : 0) + the trilinear prolongation of coarse by the factor 2^S (fine has
// Mf = (Mc - 1) 2^S + 1 points per axis, x fastest). A thread has one fine x and one coarse y
// interval and walks up `cells` coarse z intervals, 2^S x 2^S points each; the next plane of the
// coarse field, and the next old values, are on their way meanwhile. Threads run along the rows and
// on into the next interval's, so that a block's stores are runs of 256 points: bound by the writes.
// A thread per coarse x interval and fine (y, z) stored every 2^S-th point and read a cell's
// corners 18 times for the 8 points of S = 1; whole FP64 fields of 513 points per axis from 65, 129,
// 257 and 513: 612, 532, 526 and 942 us before, 221, 213, 335 and 685 now (1.08 GB: 166 us).
template <typename T, int S, bool kAdd>
__global__ void __launch_bounds__(256) kProlong(const T* coarse, int Mc, T* fine, int cells) {
  constexpr int F = 1 << S, kOld = kAdd ? F * F : 1;
  const int Mf = (Mc - 1) * F + 1;
  const unsigned column = blockIdx.x * 256 + threadIdx.x;
  const int yc = column / (unsigned)Mf, x = column - yc * Mf;
  const int zBegin = blockIdx.y * cells, zEnd = min(zBegin + cells, Mc);  // the last has one plane only
  gridDependencyWait();
  gridDependents();
  if (yc >= Mc) return;
  const int rx = x & (F - 1);
  const bool xr = rx != 0, yr = yc + 1 < Mc;
  const T wx1 = (T)rx / (T)F;  // exact: F is a power of two
  const int64_t outY = Mf, outZ = (int64_t)Mf * Mf, rowZ = (int64_t)Mc * Mc;
  const T* plane = coarse + (zBegin * rowZ + (int64_t)yc * Mc + (x >> S));
  T* out = fine + ((int64_t)zBegin * F * Mf + yc * F) * Mf + x;
  T lo[4], hi[4], up[4], old[kOld], oldUp[kOld];
  // corner x | y << 1 of a plane, where a point of the thread's takes it
  auto corners = [&](T (&c)[4], const T* p, bool in) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      c[k] = in && ((k & 1) == 0 || xr) && ((k & 2) == 0 || yr) ? p[(k & 1) + (k & 2 ? Mc : 0)] : T(0);
  };
  auto olds = [&](T (&o)[kOld], const T* p, int cz) {
    if constexpr (kAdd) {
#pragma unroll
      for (int k = 0; k < F * F; ++k)
        o[k] = (k % F == 0 || yr) && cz < Mc && (k < F || cz + 1 < Mc) ? p[(k % F) * outY + (k / F) * outZ] : T(0);
    }
  };
  corners(lo, plane, true);
  corners(hi, plane + rowZ, zBegin + 1 < Mc);
  olds(old, out, zBegin);
  for (int cz = zBegin; cz < zEnd; ++cz) {
    const bool more = cz + 1 < zEnd;
    corners(up, plane + 2 * rowZ, more && cz + 2 < Mc);
    olds(oldUp, out + F * outZ, more ? cz + 1 : Mc);
#pragma unroll
    for (int k = 0; k < F * F; ++k) {
      const int ry = k % F, rz = k / F;
      if ((ry > 0 && !yr) || (rz > 0 && cz + 1 >= Mc)) continue;
      const T wy1 = (T)ry / (T)F, wz1 = (T)rz / (T)F;
      // the field at the x interval's ends, interpolated in y and z
      T a0 = lo[0], a1 = lo[1];
      if (ry) {
        a0 = (T(1) - wy1) * a0 + wy1 * lo[2];
        a1 = (T(1) - wy1) * a1 + wy1 * lo[3];
      }
      if (rz) {
        T b0 = hi[0], b1 = hi[1];
        if (ry) {
          b0 = (T(1) - wy1) * b0 + wy1 * hi[2];
          b1 = (T(1) - wy1) * b1 + wy1 * hi[3];
        }
        a0 = (T(1) - wz1) * a0 + wz1 * b0;
        a1 = (T(1) - wz1) * a1 + wz1 * b1;
      }
      const T v = xr ? (T(1) - wx1) * a0 + wx1 * a1 : a0;
      out[ry * outY + rz * outZ] = kAdd ? old[kAdd ? k : 0] + v : v;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      lo[k] = hi[k];
      hi[k] = up[k];
    }
#pragma unroll
    for (int k = 0; k < kOld; ++k) old[k] = oldUp[k];
    plane += rowZ;
    out += F * outZ;
  }
}

// dependent: the previous operation in the stream is a kernel. A walk is as long as leaves the
// chip ten thousand threads per SM, several rounds, and at most 32 rows: longer ones write too
// many places at once (257 -> 513 points per axis, the whole field: 434, 370, 351, 335 us for
// 1, 2, 4, 8 intervals and 387 for 16; 129 -> 513: 224, 214, 230 for 1, 2, 4).
template <typename T, int S, bool kAdd>
static its_status prolong(its_ctx* ctx, bool dependent, const T* coarse, int Mc, T* fine) {
  const int64_t Mf = (int64_t)(Mc - 1) * (1 << S) + 1, columns = Mf * Mc, kMost = S == 1 ? 8 : S == 2 ? 2 : 1;
  const int cells = (int)std::min<int64_t>(std::max<int64_t>(columns * Mc / (ctx->numSMs * 10240), 1), kMost);
  const dim3 grid((unsigned)((columns + 255) / 256), (unsigned)((Mc + cells - 1) / cells));
  return launchDependent(ctx, dependent, kProlong<T, S, kAdd>, grid, 256, 0, ctx->stream, coarse, Mc, fine,
                         cells);
}

// Whether the lattice (origin, width, res) is the octree's box at res_octree * 2^s points: per
// axis the octree's origin and cell width (the octree sizes its cells by its first axis) to
// within 1e-6 of a cell. Boxes padded in single precision (BaseModel.cpp:24-51) have axes a
// few 1e-9 apart; the cascade's points are then the octree's lattice points, at most that far
// from the requested ones.
static bool alignedLattice(const SvoDevice& d, const double origin[3], const double width[3], int res, int* s) {
  const double u = d.unit[0];
  for (int a = 0; a < 3; ++a)
    if (fabs(origin[a] - d.origin[a]) > 1e-6 * u || fabs(width[a] / d.res - u) > 1e-6 * u) return false;
  for (int k = 0; k <= 3; ++k)
    if ((int64_t)d.res << k == res) {
      *s = k;
      return true;
    }
  return false;
}

template <typename T>
static its_status cascade(its_ctx* ctx, const SvoDevice& d, const double* lambda, int res, int s, T* out) {
  its_status st;
  const int D = d.depth;
  CascadeLevels<T> L = {};
  // with s == 0 the output is depth 0's lattice itself
  int64_t inner = 0;
  for (int k = 0; k < D; ++k) {
    L.M[k] = (d.res >> k) + 1;
    if (k > 0 || s > 0) inner += (int64_t)L.M[k] * L.M[k] * L.M[k];
  }
  DevBuf<T> lat;
  if ((st = lat.alloc(ctx, std::max<int64_t>(inner, 1))) != ITS_OK) return st;
  T* next = lat.p;
  for (int k = 0; k < D; ++k) {
    L.field[k] = k == 0 && s == 0 ? out : next;
    if (k > 0 || s > 0) next += (int64_t)L.M[k] * L.M[k] * L.M[k];
  }
  ITS_CU(ctx, cudaMemsetAsync(lat.p, 0, std::max<int64_t>(inner, 1) * sizeof(T), ctx->stream));
  if (s == 0) ITS_CU(ctx, cudaMemsetAsync(out, 0, (int64_t)L.M[0] * L.M[0] * L.M[0] * sizeof(T), ctx->stream));
  if (d.numVerts > 0) {
    kScatterCorners<T><<<gridFor(d.numVerts, 256), 256, 0, ctx->stream>>>(d.numVerts, d.vertKey, lambda, L);
    ITS_LAUNCHED(ctx);
  }
  bool kernelBefore = d.numVerts > 0;
  for (int k = D - 2; k >= 0; --k, kernelBefore = true)
    if ((st = prolong<T, 1, true>(ctx, kernelBefore, L.field[k + 1], L.M[k + 1], L.field[k])) != ITS_OK) return st;
  switch (s) {
    case 0: return ITS_OK;
    case 1: return prolong<T, 1, false>(ctx, kernelBefore, L.field[0], L.M[0], out);
    case 2: return prolong<T, 2, false>(ctx, kernelBefore, L.field[0], L.M[0], out);
    default: return prolong<T, 3, false>(ctx, kernelBefore, L.field[0], L.M[0], out);
  }
}

template <typename T>
static its_status evalGridFast(its_svo* sv, const double* lambda, const double origin[3], const double width[3],
                               int res, T* field) {
  if (!sv || !lambda || !origin || !width || !field || res < 1 || res > 2048) return ITS_ERR_INVALID;
  its_ctx* ctx = sv->ctx;
  ITS_CU(ctx, cudaSetDevice(ctx->device));
  int s = 0;
  if (!alignedLattice(sv->d, origin, width, res, &s)) {  // any other lattice: the exact field
    if (sizeof(T) == 8) return its_eval_grid(sv, lambda, origin, width, res, (double*)field);
    return its_eval_grid_f32(sv, lambda, origin, width, res, (float*)field);
  }
  const int64_t Mo = (int64_t)res + 1;
  InArg<double> L;
  OutArg<T> F;
  its_status st;
  if ((st = L.stage(ctx, lambda, sv->d.numVerts)) != ITS_OK || (st = F.stage(ctx, field, Mo * Mo * Mo)) != ITS_OK)
    return st;
  if ((st = cascade<T>(ctx, sv->d, L.d, res, s, F.d)) != ITS_OK) return st;
  if ((st = F.finish(ctx)) != ITS_OK) return st;
  ITS_CU(ctx, cudaStreamSynchronize(ctx->stream));
  return ITS_OK;
}

}  // namespace its

using namespace its;

extern "C" {

its_status its_eval_grid_fast(its_svo* svo, const double* lambda, const double origin[3], const double width[3],
                              int res, double* field) {
  return evalGridFast<double>(svo, lambda, origin, width, res, field);
}

its_status its_eval_grid_fast_f32(its_svo* svo, const double* lambda, const double origin[3], const double width[3],
                                  int res, float* field) {
  return evalGridFast<float>(svo, lambda, origin, width, res, field);
}

}  // extern "C"
