// P2 multicolour SOR (sm_100a): two launches per colour.
//
// 11 colours: the vertex class split in four, then the seven edge classes, from the DoF's
// barycentric weights in ascending vertex-ID order. Every colour updates from the values at its
// start, x += omega (b - A x) / diag(A). The colours of DoFs on different primitives are defined
// in different frames, and same-coloured vertices couple across some diagonals, so nothing is
// updated while rows of the colour are still read:
//   p2SorGatherKernel  reads x only: the cells' shares of the colour's closure rows, and the new
//                      values of its interior nodes, into a scratch vector;
//   p2SorUpdateKernel  sums the shares of every owner on a face, edge or vertex and updates it and
//                      its copies in the cell closures, and takes over the interior values.
// Both are bound by latency and launches up to P2 level 5, where a vector (18 MB) stays in L2. The
// lists below keep every lane of a warp on a node of the colour (rows walked by warps left two
// thirds idle at lattice 64), and the closure rows are constant stencils throughout: the element
// gather they replace took 31 to 36 us per colour for a chain of up to 24 micro-cells at a node on
// a cell's edge. Three launches per colour became two because the interior values no longer change
// while the closure rows are read; the extra copy costs 16 B per node of the colour.
// Measured: V(3,3) cycle at P2 level 5 on 48 cells, FP64: 8.10 ms before, 4.01 ms so, 3.65 ms
// with every launch set up while its predecessor runs.
#pragma once

#include "kernels.cuh"

namespace hg {
namespace dev {

// The interior nodes of one lattice level by parity class, the same for every macro-cell: X, Y, Z
// in ten bits each. The vertex class is listed by groups of four nodes consecutive in X (its
// colour changes by a constant 1, 2 or 3 mod 4 from one to the next).
// Class pc: node[node[pc]] .. node[node[pc + 1] - 1]; the first nine entries are these bounds.
constexpr int kP2NodeHead = 9;
// Per macro-cell: the class of each colour's interior nodes (-1: none, 0 for the vertex colours),
// and the vertex colour c0 + cx x + cy y + cz z mod 4 of the vertex node (2x, 2y, 2z).
struct P2CellColour {
  signed char cls[11];
  unsigned char c0, cx, cy, cz, pad;
};

// An owner DoF on a face, edge or vertex and its closure copies.
struct P2Owner {
  unsigned slot;
  int first;             // its copies: copies[first, first + count)
  unsigned short count, type;
};

// The nodes of entry e of class PC that carry colour sel: at most one per call of f, two when the
// vertex colour alternates between two values along X.
template <int PC, class F>
__device__ __forceinline__ void p2ForNodes(unsigned e, const P2CellColour& cc, int sel, int M, F f) {
  const int X = e & 1023, Y = (e >> 10) & 1023, Z = e >> 20;
  if (PC != 0) {
    f(X, Y, Z);
    return;
  }
  const int c = (cc.c0 + cc.cx * (X >> 1) + cc.cy * (Y >> 1) + cc.cz * (Z >> 1)) & 3;  // of the group's first node
  const int diff = (sel - c) & 3;
  if (cc.cx & 1) {
    const int x = X + 2 * ((diff * cc.cx) & 3);
    if (x + Y + Z <= M - 1) f(x, Y, Z);
  } else if (!(diff & 1)) {
    for (int x = X + diff; x <= X + 6 && x + Y + Z <= M - 1; x += 4) f(x, Y, Z);
  }
}

template <class T, int PC>
__device__ __forceinline__ void p2SorNodes(unsigned e, const P2CellColour& cc, int sel, const T* __restrict__ u,
                                           const T* __restrict__ f, T* __restrict__ out, const T* __restrict__ wt, int w,
                                           int M, T omega) {
  using S = typename p2s::Class<PC>::type;
  constexpr int kFirst = p2s::kFirst[PC], kCentre = p2s::kCentre[PC], kLen = p2s::kLen[PC];
  wt += kFirst;
  p2ForNodes<PC>(e, cc, sel, M, [&](int X, int Y, int Z) {
    int pbz[5];
#pragma unroll
    for (int d = 0; d < 5; ++d) {
      const int z = Z - 2 + d;
      pbz[d] = (z >= 0 && z <= M) ? int(tetSize(w) - tetSize(w - z)) : 0;
    }
    const int i = pbz[2] + rowStart(w - Z, Y) + X;
    const T s = p2StencilDot<T>(S{}, std::make_integer_sequence<int, kLen>{}, u, wt, pbz, w, X, Y, Z);
    out[i] = u[i] + omega * (f[i] - s) / wt[kCentre];
  });
}

// Grid: listBlocks blocks on the colour's closure nodes, then chunks blocks per macro-cell.
template <class T>
__global__ void __launch_bounds__(kBlock, 3) p2SorGatherKernel(LevelDev lv, const T* __restrict__ W,
                                                               const T* __restrict__ FW,
                                                               const P2ClosureNode* __restrict__ list, int nList,
                                                               int listBlocks, const unsigned* __restrict__ nodes,
                                                               const P2CellColour* __restrict__ cells, int sel, int chunks,
                                                               const T* __restrict__ x, const T* __restrict__ b,
                                                               T* __restrict__ ax, unsigned mask, T omega) {
  const int M = lv.N, w = lv.w;
  if ((int)blockIdx.x < listBlocks) {
    const int i = blockIdx.x * kBlock + threadIdx.x;
    const P2ClosureNode nd = list[min(i, nList - 1)];
    const int64_t base = lv.cellOff[nd.cell];
    waitForPredecessor(x, b, ax);
    if (i >= nList) return;
    const int X = nd.x, Y = nd.y, Z = nd.z;
    int pbz[5];
#pragma unroll
    for (int d = 0; d < 5; ++d) {
      const int z = Z - 2 + d;
      pbz[d] = (z >= 0 && z <= M) ? int(tetSize(w) - tetSize(w - z)) : 0;
    }
    ax[base + pbz[2] + rowStart(w - Z, Y) + X] =
        p2FaceDotAny<T>(nd.k, x + base, FW + (int64_t)nd.cell * p2s::kFaceTotal, pbz, w, X, Y, Z);
    return;
  }
  // the list entry is read before the wait, whether or not the cell has the colour
  const int q = blockIdx.x - listBlocks, c = q / chunks;
  const bool on = lv.cellType[c] & mask;
  const P2CellColour cc = cells[c];
  const int pc = cells[c].cls[sel];
  const unsigned end = nodes[max(pc, 0) + 1], t = nodes[max(pc, 0)] + (q - c * chunks) * kBlock + threadIdx.x;
  const unsigned e = t < end ? __ldg(nodes + t) : 0;
  const int64_t base = lv.cellOff[c];
  waitForPredecessor(x, b, ax);
  if (!on || pc < 0 || t >= end) return;
  const T* wc = W + (int64_t)c * p2s::kTotal;
  switch (pc) {
    case 0: p2SorNodes<T, 0>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
    case 1: p2SorNodes<T, 1>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
    case 2: p2SorNodes<T, 2>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
    case 3: p2SorNodes<T, 3>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
    case 4: p2SorNodes<T, 4>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
    case 5: p2SorNodes<T, 5>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
    case 6: p2SorNodes<T, 6>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
    default: p2SorNodes<T, 7>(e, cc, sel, x + base, b + base, ax + base, wc, w, M, omega); break;
  }
}

// Grid: ownerBlocks blocks on the colour's owners, then chunks blocks per macro-cell.
template <class T>
__global__ void __launch_bounds__(kBlock) p2SorUpdateKernel(LevelDev lv, const P2Owner* __restrict__ owners, int nOwners,
                                                            int ownerBlocks, const unsigned* __restrict__ copies,
                                                            const unsigned* __restrict__ nodes, const P2CellColour* __restrict__ cells, int sel,
                                                            int chunks, T* __restrict__ x, const T* __restrict__ b,
                                                            const T* __restrict__ ax, const T* __restrict__ diag,
                                                            unsigned mask, T omega) {
  if ((int)blockIdx.x < ownerBlocks) {
    const int t = blockIdx.x * kBlock + threadIdx.x;
    const P2Owner o = owners[min(t, nOwners - 1)];
    waitForPredecessor(x, b, ax, diag);
    if (t >= nOwners || !(o.type & mask)) return;
    const T x0 = x[o.slot], b0 = __ldg(b + o.slot), d0 = __ldg(diag + o.slot);
    T s = T(0);
    for (int k = o.first; k < o.first + o.count; ++k) s += __ldg(ax + copies[k]);
    const T v = x0 + omega * (b0 - s) / d0;
    x[o.slot] = v;
    // the owner's copies in the cell closures take the new value at once
    for (int k = o.first; k < o.first + o.count; ++k) x[copies[k]] = v;
    return;
  }
  const int M = lv.N, w = lv.w, q = blockIdx.x - ownerBlocks, c = q / chunks;
  const bool on = lv.cellType[c] & mask;
  const P2CellColour cc = cells[c];
  const int pc = cells[c].cls[sel];
  const unsigned end = nodes[max(pc, 0) + 1], t = nodes[max(pc, 0)] + (q - c * chunks) * kBlock + threadIdx.x;
  const unsigned e = t < end ? __ldg(nodes + t) : 0;
  const int64_t base = lv.cellOff[c];
  waitForPredecessor(x, b, ax, diag);
  if (!on || pc < 0 || t >= end) return;
  auto take = [&](int X, int Y, int Z) {
    const int64_t i = base + int(tetSize(w) - tetSize(w - Z)) + rowStart(w - Z, Y) + X;
    x[i] = __ldg(ax + i);
  };
  if (pc == 0) p2ForNodes<0>(e, cc, sel, M, take);
  else p2ForNodes<1>(e, cc, sel, M, take);
}

}  // namespace dev
}  // namespace hg
