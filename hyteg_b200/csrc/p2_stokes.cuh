// Taylor-Hood coupling blocks (sm_100a) between the P1 pressure lattice (level L, size N) and the
// P2 velocity lattice (level L + 1, size M = 2N), one launch each:
//   p2DivKernel   q = sum_k D_k u_k at the pressure nodes
//   p2DivTKernel  v_k = D_k^T p (or += with ADD) at the velocity nodes
// Within a macro-cell every row is a constant stencil, per class inside the cell and per closure
// entry on its faces, edges and vertices (p2_stencil.h); the weights are per cell, [component][..].
// Interior nodes get their final value, closure nodes the cell's share, which is summed into the
// owners afterwards; with ADD the shares are added to those already in the closure slots, so one
// sum serves the velocity block and the gradient.
// The closure nodes come from the level's list (sorted by entry, so that a warp mostly runs one
// stencil), the interior ones from the triangle of a plane, one lane per node: rows walked by warps
// left two thirds of the lanes idle at N = 32. Bound by latency and L2 at the sizes met (P2 level 5:
// velocity vectors of 18 MB).
// Measured, 48 cells, P2 level 5, FP64: the block apply 0.685 ms with element gathers on the closure,
// separate interior launches and the gradient in scratch vectors, 0.380 ms so, 0.357 ms with every launch
// set up while its predecessor runs.
#pragma once

#include "kernels.cuh"

namespace hg {
namespace dev {

template <class T>
__device__ __forceinline__ void p2Acc3(T (&s)[6], const T* w, int stride, int I, const T* u0, const T* u1, const T* u2, int o) {
  const int h = I & 1;  // two partial sums per component
  s[h] += w[I] * __ldg(u0 + o);
  s[2 + h] += w[stride + I] * __ldg(u1 + o);
  s[4 + h] += w[2 * stride + I] * __ldg(u2 + o);
}

template <class T, int... DX, int... DY, int... DZ, int... I>
__device__ __forceinline__ T p2DivDot(p2s::List<p2s::O<DX, DY, DZ>...>, std::integer_sequence<int, I...>, const T* u0,
                                      const T* u1, const T* u2, const T* w, int stride, const int (&pbz)[5], int wv, int X,
                                      int Y, int Z) {
  T s[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
  (p2Acc3<T>(s, w, stride, I, u0, u1, u2, p2RowBase<DY, DZ>(pbz, wv, Y, Z) + X + DX), ...);
  return (s[0] + s[1]) + ((s[2] + s[3]) + (s[4] + s[5]));
}

template <class T>
__device__ __forceinline__ void p2Acc3T(T (&s)[3], const T* w, int stride, int I, T pv) {
  s[0] += w[I] * pv;
  s[1] += w[stride + I] * pv;
  s[2] += w[2 * stride + I] * pv;
}

template <class T, int... DX, int... DY, int... DZ, int... I>
__device__ __forceinline__ void p2DivTDot(p2s::List<p2s::O<DX, DY, DZ>...>, std::integer_sequence<int, I...>,
                                          const T* p, const T* w, int stride, const int (&pbz)[5], int wp, int x, int y,
                                          int z, T (&s)[3]) {
  (p2Acc3T<T>(s, w, stride, I, __ldg(p + p2RowBase<DY, DZ>(pbz, wp, y, z) + x + DX)), ...);
}

// First indices of the planes z - 2 .. z + 2 of a cell of lattice size n.
__device__ __forceinline__ void p2Planes(int (&pbz)[5], int n, int z) {
#pragma unroll
  for (int d = 0; d < 5; ++d) {
    const int zz = z - 2 + d;
    pbz[d] = (zz >= 0 && zz <= n) ? int(tetSize(n + 1) - tetSize(n + 1 - zz)) : 0;
  }
}

// Node t of a triangle with K nodes in its first row, K - 1 in the next, ...: row j, position i.
__device__ __forceinline__ void triangleNode(int K, int t, int& j, int& i) {
  const float b = float(2 * K + 1);
  j = max(0, min(int((b - sqrtf(fmaxf(b * b - 8.0f * float(t), 0.0f))) * 0.5f), K - 1));
  while (j > 0 && j * K - j * (j - 1) / 2 > t) --j;
  while (j < K - 1 && (j + 1) * K - (j + 1) * j / 2 <= t) ++j;
  i = t - (j * K - j * (j - 1) / 2);
}

// A closure pressure node reads the velocity nodes of its vertex-class entry KV.
template <class T, int KV>
__device__ __forceinline__ void p2DivClosure(T* q, const T* u0, const T* u1, const T* u2, const T* w, const int (&pbz)[5],
                                             int wv, int X, int Y, int Z) {
  using S = typename p2s::FaceList<KV>::type;
  constexpr int kFirst = p2s::kFaceFirst[KV], kLen = p2s::kFaceLen[KV], kTotal = p2s::kFaceTotal;
  *q = p2DivDot<T>(S{}, std::make_integer_sequence<int, kLen>{}, u0, u1, u2, w + kFirst, kTotal, pbz, wv, X, Y, Z);
}

// Grid: listBlocks blocks on the closure nodes, then (N >= 4) one per macro-cell and plane 1 .. N - 3.
template <class T>
__global__ void __launch_bounds__(kBlock) p2DivKernel(LevelDev lvp, LevelDev lvv, const T* __restrict__ WD,
                                                      const T* __restrict__ WC, const P2ClosureNode* __restrict__ list,
                                                      int nList, int listBlocks, T* __restrict__ q,
                                                      const T* __restrict__ u0, const T* __restrict__ u1,
                                                      const T* __restrict__ u2, unsigned mask) {
  waitForPredecessor(q, u0, u1, u2);
  const int N = lvp.N, wp = lvp.w, wv = lvv.w, M = lvv.N;
  int pbz[5];
  if ((int)blockIdx.x < listBlocks) {
    const int t = blockIdx.x * kBlock + threadIdx.x;
    if (t >= nList) return;
    const P2ClosureNode nd = list[t];
    const int X = 2 * nd.x, Y = 2 * nd.y, Z = 2 * nd.z;
    p2Planes(pbz, M, Z);
    const int64_t vb = lvv.cellOff[nd.cell];
    T* o = q + lvp.cellOff[nd.cell] + int(tetSize(wp) - tetSize(wp - nd.z)) + rowStart(wp - nd.z, nd.y) + nd.x;
    const T* w = WC + (int64_t)nd.cell * (3 * p2s::kFaceTotal);
    const T *a = u0 + vb, *b = u1 + vb, *c = u2 + vb;
    switch (nd.k < 16 ? nd.k & ~3 : nd.k < 28 ? nd.k & ~1 : nd.k) {
      case 0: p2DivClosure<T, 0>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 4: p2DivClosure<T, 4>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 8: p2DivClosure<T, 8>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 12: p2DivClosure<T, 12>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 16: p2DivClosure<T, 16>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 18: p2DivClosure<T, 18>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 20: p2DivClosure<T, 20>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 22: p2DivClosure<T, 22>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 24: p2DivClosure<T, 24>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 26: p2DivClosure<T, 26>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 28: p2DivClosure<T, 28>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 29: p2DivClosure<T, 29>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      case 30: p2DivClosure<T, 30>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
      default: p2DivClosure<T, 31>(o, a, b, c, w, pbz, wv, X, Y, Z); break;
    }
    return;
  }
  const int nPl = N - 3, r = blockIdx.x - listBlocks, c = r / nPl, z = 1 + r - c * nPl;
  if (!(lvp.cellType[c] & mask)) return;
  __shared__ T wts[195];
  for (int k = threadIdx.x; k < 195; k += kBlock) wts[k] = WD[(int64_t)c * 195 + k];
  __syncthreads();
  p2Planes(pbz, M, 2 * z);
  const int64_t vb = lvv.cellOff[c];
  T* o = q + lvp.cellOff[c] + int(tetSize(wp) - tetSize(wp - z));
  const int K = N - 2 - z;  // interior nodes of row y = 1
  for (int t = threadIdx.x; t < K * (K + 1) / 2; t += kBlock) {
    int j, i;
    triangleNode(K, t, j, i);
    const int x = 1 + i, y = 1 + j;
    o[rowStart(wp - z, y) + x] = p2DivDot<T>(p2s::S0{}, std::make_integer_sequence<int, p2s::kLen[0]>{}, u0 + vb, u1 + vb,
                                             u2 + vb, wts, 65, pbz, wv, 2 * x, 2 * y, 2 * z);
  }
}

template <class T, bool ADD>
__device__ __forceinline__ void p2Write3(T* v0, T* v1, T* v2, int64_t o, const T (&s)[3]) {
  if (ADD) {
    v0[o] += s[0];
    v1[o] += s[1];
    v2[o] += s[2];
  } else {
    v0[o] = s[0];
    v1[o] = s[1];
    v2[o] = s[2];
  }
}

template <class T, int K>
__device__ __forceinline__ void p2DivTClosure(const T* p, const T* w, const int (&pbz)[5], int wp, int x, int y, int z,
                                              T (&s)[3]) {
  using S = typename p2s::DivTFaceList<K>::type;
  constexpr int kFirst = p2s::kDivTFaceFirst[K], kLen = p2s::kDivTFaceLen[K], kTotal = p2s::kDivTFaceTotal;
  p2DivTDot<T>(S{}, std::make_integer_sequence<int, kLen>{}, p, w + kFirst, kTotal, pbz, wp, x, y, z, s);
}

template <class T, bool ADD, int PC>
__device__ __forceinline__ void p2DivTPlane(const T* wts, T* v0, T* v1, T* v2, const T* p, int64_t vb, const int (&pbz)[5],
                                            int wv, int wp, int M, int Z, int t0, int dt) {
  using S = typename p2s::DivTList<PC>::type;
  constexpr int kFirst = p2s::kDivTFirst[PC], kLen = p2s::kDivTLen[PC], kX = PC & 1 ? 1 : 2, kY = PC & 2 ? 1 : 2;
  const int room = M - 1 - Z - kX - kY, K = room < 0 ? 0 : room / 2 + 1;  // nodes of the class in its first row
#pragma unroll 1
  for (int t = t0; t < K * (K + 1) / 2; t += dt) {
    int j, i;
    triangleNode(K, t, j, i);
    const int X = kX + 2 * i, Y = kY + 2 * j;
    T s[3] = {T(0), T(0), T(0)};
    p2DivTDot<T>(S{}, std::make_integer_sequence<int, kLen>{}, p, wts + kFirst, 65, pbz, wp, X >> 1, Y >> 1, Z >> 1, s);
    p2Write3<T, ADD>(v0, v1, v2, vb + rowStart(wv - Z, Y) + X, s);
  }
}

// Grid: listBlocks blocks on the closure nodes, then (M >= 4) one per macro-cell and plane 1 .. M - 3,
// whose warps take the plane's four classes, two warps each.
template <class T, bool ADD>
__global__ void __launch_bounds__(kBlock) p2DivTKernel(LevelDev lvv, LevelDev lvp, const T* __restrict__ WT,
                                                       const T* __restrict__ WC, const P2ClosureNode* __restrict__ list,
                                                       int nList, int listBlocks, T* __restrict__ v0, T* __restrict__ v1,
                                                       T* __restrict__ v2, const T* __restrict__ p, unsigned mask) {
  waitForPredecessor(v0, v1, v2, p);
  const int M = lvv.N, wv = lvv.w, wp = lvp.w, Np = lvp.N;
  int pbz[5];
  if ((int)blockIdx.x < listBlocks) {
    const int t = blockIdx.x * kBlock + threadIdx.x;
    if (t >= nList) return;
    const P2ClosureNode nd = list[t];
    const int X = nd.x, Y = nd.y, Z = nd.z, x = X >> 1, y = Y >> 1, z = Z >> 1;
    p2Planes(pbz, Np, z);
    const T* pc = p + lvp.cellOff[nd.cell];
    const T* w = WC + (int64_t)nd.cell * (3 * p2s::kDivTFaceTotal);
    T s[3] = {T(0), T(0), T(0)};
    switch (nd.k) {
      case 0: p2DivTClosure<T, 0>(pc, w, pbz, wp, x, y, z, s); break;
      case 1: p2DivTClosure<T, 1>(pc, w, pbz, wp, x, y, z, s); break;
      case 2: p2DivTClosure<T, 2>(pc, w, pbz, wp, x, y, z, s); break;
      case 3: p2DivTClosure<T, 3>(pc, w, pbz, wp, x, y, z, s); break;
      case 4: p2DivTClosure<T, 4>(pc, w, pbz, wp, x, y, z, s); break;
      case 5: p2DivTClosure<T, 5>(pc, w, pbz, wp, x, y, z, s); break;
      case 6: p2DivTClosure<T, 6>(pc, w, pbz, wp, x, y, z, s); break;
      case 7: p2DivTClosure<T, 7>(pc, w, pbz, wp, x, y, z, s); break;
      case 8: p2DivTClosure<T, 8>(pc, w, pbz, wp, x, y, z, s); break;
      case 9: p2DivTClosure<T, 9>(pc, w, pbz, wp, x, y, z, s); break;
      case 10: p2DivTClosure<T, 10>(pc, w, pbz, wp, x, y, z, s); break;
      case 11: p2DivTClosure<T, 11>(pc, w, pbz, wp, x, y, z, s); break;
      case 12: p2DivTClosure<T, 12>(pc, w, pbz, wp, x, y, z, s); break;
      case 13: p2DivTClosure<T, 13>(pc, w, pbz, wp, x, y, z, s); break;
      case 14: p2DivTClosure<T, 14>(pc, w, pbz, wp, x, y, z, s); break;
      case 15: p2DivTClosure<T, 15>(pc, w, pbz, wp, x, y, z, s); break;
      case 16: p2DivTClosure<T, 16>(pc, w, pbz, wp, x, y, z, s); break;
      case 17: p2DivTClosure<T, 17>(pc, w, pbz, wp, x, y, z, s); break;
      case 18: p2DivTClosure<T, 18>(pc, w, pbz, wp, x, y, z, s); break;
      case 19: p2DivTClosure<T, 19>(pc, w, pbz, wp, x, y, z, s); break;
      case 20: p2DivTClosure<T, 20>(pc, w, pbz, wp, x, y, z, s); break;
      case 21: p2DivTClosure<T, 21>(pc, w, pbz, wp, x, y, z, s); break;
      case 22: p2DivTClosure<T, 22>(pc, w, pbz, wp, x, y, z, s); break;
      case 23: p2DivTClosure<T, 23>(pc, w, pbz, wp, x, y, z, s); break;
      case 24: p2DivTClosure<T, 24>(pc, w, pbz, wp, x, y, z, s); break;
      case 25: p2DivTClosure<T, 25>(pc, w, pbz, wp, x, y, z, s); break;
      case 26: p2DivTClosure<T, 26>(pc, w, pbz, wp, x, y, z, s); break;
      case 27: p2DivTClosure<T, 27>(pc, w, pbz, wp, x, y, z, s); break;
      case 28: p2DivTClosure<T, 28>(pc, w, pbz, wp, x, y, z, s); break;
      case 29: p2DivTClosure<T, 29>(pc, w, pbz, wp, x, y, z, s); break;
      case 30: p2DivTClosure<T, 30>(pc, w, pbz, wp, x, y, z, s); break;
      default: p2DivTClosure<T, 31>(pc, w, pbz, wp, x, y, z, s); break;
    }
    p2Write3<T, ADD>(v0, v1, v2, lvv.cellOff[nd.cell] + int(tetSize(wv) - tetSize(wv - Z)) + rowStart(wv - Z, Y) + X, s);
    return;
  }
  const int nPl = M - 3, r = blockIdx.x - listBlocks, c = r / nPl, Z = 1 + r - c * nPl;
  if (!(lvv.cellType[c] & mask)) return;
  __shared__ T wts[195];
  for (int k = threadIdx.x; k < 195; k += kBlock) wts[k] = WT[(int64_t)c * 195 + k];
  __syncthreads();
  p2Planes(pbz, Np, Z >> 1);
  const T* pc = p + lvp.cellOff[c];
  const int64_t vb = lvv.cellOff[c] + int(tetSize(wv) - tetSize(wv - Z));
  const int warp = threadIdx.x >> 5, t0 = (threadIdx.x & 31) + 32 * (warp >> 2), dt = kBlock / 4;
  switch ((warp & 3) | ((Z & 1) << 2)) {
    case 0: p2DivTPlane<T, ADD, 0>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
    case 1: p2DivTPlane<T, ADD, 1>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
    case 2: p2DivTPlane<T, ADD, 2>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
    case 3: p2DivTPlane<T, ADD, 3>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
    case 4: p2DivTPlane<T, ADD, 4>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
    case 5: p2DivTPlane<T, ADD, 5>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
    case 6: p2DivTPlane<T, ADD, 6>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
    default: p2DivTPlane<T, ADD, 7>(wts, v0, v1, v2, pc, vb, pbz, wv, wp, M, Z, t0, dt); break;
  }
}

}  // namespace dev
}  // namespace hg
