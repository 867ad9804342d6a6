// P2 operator apply and residual on the closed macro-cells (sm_100a), one launch for everything.
//
// A level's work list (P2Item, the same for every macro-cell) holds three kinds of blocks:
//   interior tiles of 16 x 16 x 16 lattice nodes, staged in shared memory;
//   32 x 32 pieces of the cell's four faces;
//   the nodes on the cell's edges and vertices.
// Interior and face threads own a block of 2 x 2 x 2 (2 x 2) nodes, one of each parity class, and
// walk over the distinct lattice positions the block's stencils read: a position is loaded once
// and enters every row that uses it, so 89 loads serve the 230 products of eight nodes. The rows
// read one by one were bound by L1 wavefronts: each product loaded its value with a lane stride of
// two nodes. In the tile the even and the odd nodes of a row lie apart and the row stride of 20
// sets the four block rows of a warp on different banks, so every load is conflict-free; the
// weights are broadcast, two per load, and serve two blocks of a thread. 16^3 tiles (19^3 staged,
// 58 KB in FP64) leave two blocks of 256 threads per SM and waste the fewest threads at the sloped
// face (73 % of a cell's threads update a node at lattice 128, 55 % at 64, 34 % at 32).
// Measured, 48 cells, P2 level 6 (lattice 128, 16.6 M nodes), FP64, the whole apply with its halo
// exchanges: 0.707 ms with one launch for rows by parity class and one for the closure, 0.321 ms so.
#pragma once

#include "kernels.cuh"

namespace hg {
namespace dev {

enum P2ItemKind { P2_EDGES = 0, P2_TILE = 1, P2_FACE = 2 };
struct P2Item {
  int kind;
  int a, b, c;  // tile: origin (its first nodes are origin + 1); face: face, s0, t0; edges: first node
};

constexpr int kP2Tile = 16;                   // lattice nodes per tile edge
constexpr int kP2Region = kP2Tile + 3;        // staged nodes per edge: origin .. origin + 18
constexpr int kP2Stride = 20;                 // elements per staged row: even X, then odd X, ten each
constexpr int kP2FaceTile = 32;               // face nodes per piece edge
constexpr int kP2RowTab = kP2Region * kP2Region;

// Interior blocks. Node i of a block sits at origin + 1 + (bits of i), so its parity class is
// 7 - i (the block's origin is even). Entries by lattice position.
struct P2BlockEntry {
  signed char x, y, z;  // lattice position relative to the block's origin, 0 .. 4
  unsigned char node;
  unsigned char acc;    // the accumulator of the product
  bool first;           // first entry of its position
  short weight;         // index into the cell's weights p2s::kTotal
};
// The vertex class (65 products) is summed in four parts (7 .. 10), the edge classes of 27 products
// (nodes 1, 3, 4, 6) in two halves, those of 19 in one: more accumulators spill in FP64 (two halves
// everywhere: 335 us instead of 321 for the apply below). The positions of the nodes themselves come
// last, so that the diagonal, the largest product, is added late and the partial sums before it round
// less. Error against 64 bits, 48 cells, P2 level 5: FP64 6.2e-17, FP32 1.74e-8; with one chain per
// edge class in the order of the positions 6.9e-17 and 2.34e-8, with four parts for every row 6.3e-17
// and 1.80e-8.
constexpr int kP2Accs = 15;
__host__ __device__ constexpr bool p2Halves(int node) { return node == 1 || node == 3 || node == 4 || node == 6; }
__host__ __device__ constexpr int p2Second(int node) { return node == 1 ? 11 : node == 3 ? 12 : node == 4 ? 13 : 14; }

struct P2BlockTable {
  P2BlockEntry e[p2s::kTotal];
};

constexpr P2BlockTable makeP2BlockTable() {
  P2BlockTable t{};
  int n = 0, done[8] = {};
  for (const bool own : {false, true})
    for (int z = 0; z <= 4; ++z)
      for (int y = 0; y <= 4; ++y)
        for (int x = 0; x <= 4; ++x) {
          if (((x == 1 || x == 2) && (y == 1 || y == 2) && (z == 1 || z == 2)) != own) continue;
          bool first = true;
          for (int i = 0; i < 8; ++i) {
            const int pc = 7 - i, nx = 1 + (i & 1), ny = 1 + ((i >> 1) & 1), nz = 1 + (i >> 2);
            for (int k = 0; k < p2s::kLen[pc]; ++k)
              if (nx + p2s::kOff[pc][k][0] == x && ny + p2s::kOff[pc][k][1] == y && nz + p2s::kOff[pc][k][2] == z) {
                P2BlockEntry& q = t.e[n++];
                q.x = (signed char)x;
                q.y = (signed char)y;
                q.z = (signed char)z;
                q.node = (unsigned char)i;
                const bool second = p2Halves(i) && 2 * done[i]++ >= p2s::kLen[pc];
                q.acc = (unsigned char)(pc == 0 ? 7 + (k & 3) : second ? p2Second(i) : i);
                q.first = first;
                q.weight = (short)(p2s::kFirst[pc] + k);
                first = false;
              }
          }
        }
  return t;
}
constexpr P2BlockTable kP2Block = makeP2BlockTable();
// No accumulator takes more than 19 products, and every diagonal is among the products of the last eight
// positions.
constexpr bool p2SumsAreShort() {
  int taken[8][kP2Accs] = {}, left = 8;
  for (int e = p2s::kTotal - 1; e >= 0; --e) {
    const P2BlockEntry& q = kP2Block.e[e];
    const int i = q.node;
    if (++taken[i][q.acc] > 19) return false;
    const bool diagonal = q.x == 1 + (i & 1) && q.y == 1 + ((i >> 1) & 1) && q.z == 1 + (i >> 2);
    if (diagonal && left <= 0) return false;
    if (q.first) --left;
  }
  return true;
}
static_assert(p2SumsAreShort(), "P2 rows: summation order");
static __constant__ P2BlockTable kP2BlockDev = makeP2BlockTable();

// Face blocks: node i of face f at (s, t) = block origin + (bits of i); faces Z = 0: (X, Y),
// Y = 0: (X, Z), X = 0: (Y, Z), X + Y + Z = M: (Y, Z). Positions relative to node 0.
struct P2FaceEntry {
  signed char x, y, z;
  unsigned char node;
  unsigned char part;  // the products of a row are summed in two halves
  bool first;
  short weight;  // index into the cell's face weights p2s::kFaceTotal
};
constexpr int kP2FaceEntries = 92;  // of each face: its four classes
struct P2FaceTable {
  P2FaceEntry e[4][kP2FaceEntries];
};

__host__ __device__ constexpr int p2FaceNode(int f, int i, int axis) {  // offset of node i from node 0
  const int a = i & 1, b = i >> 1;
  if (f == 0) return axis == 0 ? a : axis == 1 ? b : 0;
  if (f == 1) return axis == 0 ? a : axis == 1 ? 0 : b;
  if (f == 2) return axis == 0 ? 0 : axis == 1 ? a : b;
  return axis == 0 ? -a - b : axis == 1 ? a : b;
}

constexpr P2FaceTable makeP2FaceTable() {  // the positions of the nodes themselves last, as above
  P2FaceTable t{};
  for (int f = 0; f < 4; ++f) {
    int n = 0, done[4] = {};
    // node 0 has odd (s, t): its class, and that of the others, as in p2ClosureEntry
    for (const bool own : {false, true})
      for (int z = -2; z <= 3; ++z)
        for (int y = -2; y <= 3; ++y)
          for (int x = -4; x <= 3; ++x) {
            bool node = false, first = true;
            for (int i = 0; i < 4; ++i)
              node = node || (p2FaceNode(f, i, 0) == x && p2FaceNode(f, i, 1) == y && p2FaceNode(f, i, 2) == z);
            if (node != own) continue;
            for (int i = 0; i < 4; ++i) {
              const int s = 1 + (i & 1), u = 1 + (i >> 1);  // parities of (s, t)
              int pc = 0;
              if (f == 0) pc = (s & 1) | ((u & 1) << 1);
              if (f == 1) pc = (s & 1) | ((u & 1) << 2);
              if (f == 2) pc = ((s & 1) << 1) | ((u & 1) << 2);
              if (f == 3) pc = ((s + u) & 1) | ((s & 1) << 1) | ((u & 1) << 2);
              int k = 4 * f;
              while (p2s::kFaceClass[k] != pc) ++k;
              for (int e = 0; e < p2s::kFaceLen[k]; ++e) {
                const auto& o = p2s::kFaceOff[k][e];
                if (p2FaceNode(f, i, 0) + o[0] != x || p2FaceNode(f, i, 1) + o[1] != y || p2FaceNode(f, i, 2) + o[2] != z)
                  continue;
                P2FaceEntry& q = t.e[f][n++];
                q.x = (signed char)x;
                q.y = (signed char)y;
                q.z = (signed char)z;
                q.node = (unsigned char)i;
                q.part = (unsigned char)(2 * done[i]++ / p2s::kFaceLen[k]);
                q.first = first;
                q.weight = (short)(p2s::kFaceFirst[k] + e);
                first = false;
              }
            }
          }
  }
  return t;
}
constexpr P2FaceTable kP2Face = makeP2FaceTable();

template <class T>
constexpr size_t p2TileSmem() {
  return sizeof(T) * (kP2RowTab * kP2Stride + p2s::kTotal + 2) + sizeof(int2) * kP2RowTab;
}

template <class T>
struct P2Vec;  // two weights per shared-memory load
template <>
struct P2Vec<double> {
  using type = double2;
};
template <>
struct P2Vec<float> {
  using type = float2;
};

// Entry E of a pair of blocks two lattice planes apart (blocks 0 and 1 of a thread).
template <class T, int E>
__device__ __forceinline__ void p2BlockEntry(const T* __restrict__ s, const T* __restrict__ wts,
                                             typename P2Vec<T>::type& w2, T (&v)[2], T (&acc)[2][kP2Accs]) {
  constexpr P2BlockEntry q = kP2Block.e[E];
  if constexpr (q.first) {
    constexpr int o = (q.z * kP2Region + q.y) * kP2Stride + (q.x & 1) * (kP2Stride / 2) + (q.x >> 1);
    v[0] = s[o];
    v[1] = s[o + 2 * kP2Region * kP2Stride];
  }
  if constexpr ((E & 1) == 0) w2 = *reinterpret_cast<const typename P2Vec<T>::type*>(wts + E);
  const T w = (E & 1) ? w2.y : w2.x;
  acc[0][q.acc] += w * v[0];
  acc[1][q.acc] += w * v[1];
}

template <class T, int... E>
__device__ __forceinline__ void p2BlockDot(std::integer_sequence<int, E...>, const T* __restrict__ s,
                                           const T* __restrict__ wts, T (&acc)[2][kP2Accs]) {
  typename P2Vec<T>::type w2;
  T v[2];
  (p2BlockEntry<T, E>(s, wts, w2, v, acc), ...);
}

// Row (Y + DY, Z + DZ) of the cell array, as an index of X = 0.
__device__ __forceinline__ int p2Row(int w, int Y, int Z) { return int(tetSize(w) - tetSize(w - Z)) + rowStart(w - Z, Y); }

template <class T, int F, int E>
__device__ __forceinline__ void p2FaceBlockEntry(const T* __restrict__ u, const T* __restrict__ fw, int w, int last, int X,
                                                 int Y, int Z, const int (&pbz)[6], T& v, T (&acc)[4][2]) {
  constexpr P2FaceEntry q = kP2Face.e[F][E];
  if constexpr (q.first) {
    // a partly empty block at the face's far side also walks over positions outside the cell: the
    // clamp keeps them inside the array (their nodes are not written)
    const int i = pbz[q.z + 2] + rowStart(w - Z - q.z, Y + q.y) + X + q.x;
    v = __ldg(u + min(unsigned(i), unsigned(last)));
  }
  acc[q.node][q.part] += __ldg(fw + q.weight) * v;
}

template <class T, int F, int... E>
__device__ __forceinline__ void p2FaceBlock(std::integer_sequence<int, E...>, const T* __restrict__ u,
                                            const T* __restrict__ fw, T* __restrict__ d, int w, int M, int s, int t) {
  const int X = F == 0 || F == 1 ? s : F == 2 ? 0 : M - s - t, Y = F == 0 ? t : F == 1 ? 0 : s, Z = F == 0 ? 0 : t;
  int pbz[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int z = Z - 2 + k;
    pbz[k] = z >= 0 && z <= M ? int(tetSize(w) - tetSize(w - z)) : 0;
  }
  const int last = int(tetSize(w)) - 1;
  T acc[4][2] = {}, v = T(0);
  (p2FaceBlockEntry<T, F, E>(u, fw, w, last, X, Y, Z, pbz, v, acc), ...);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int a = i & 1, b = i >> 1;
    if (s + a + t + b <= M - 1)
      d[p2Row(w, Y + p2FaceNode(F, i, 1), Z + p2FaceNode(F, i, 2)) + X + p2FaceNode(F, i, 0)] = acc[i][0] + acc[i][1];
  }
}

// An edge or vertex node's share (entries 16 .. 31 of the closure stencils).
template <class T>
__device__ __forceinline__ T p2RimDot(int k, const T* u, const T* fw, const int (&pbz)[5], int w, int X, int Y, int Z) {
  switch (k) {
    case 16: return p2FaceDot<T, 16>(u, fw, pbz, w, X, Y, Z);
    case 17: return p2FaceDot<T, 17>(u, fw, pbz, w, X, Y, Z);
    case 18: return p2FaceDot<T, 18>(u, fw, pbz, w, X, Y, Z);
    case 19: return p2FaceDot<T, 19>(u, fw, pbz, w, X, Y, Z);
    case 20: return p2FaceDot<T, 20>(u, fw, pbz, w, X, Y, Z);
    case 21: return p2FaceDot<T, 21>(u, fw, pbz, w, X, Y, Z);
    case 22: return p2FaceDot<T, 22>(u, fw, pbz, w, X, Y, Z);
    case 23: return p2FaceDot<T, 23>(u, fw, pbz, w, X, Y, Z);
    case 24: return p2FaceDot<T, 24>(u, fw, pbz, w, X, Y, Z);
    case 25: return p2FaceDot<T, 25>(u, fw, pbz, w, X, Y, Z);
    case 26: return p2FaceDot<T, 26>(u, fw, pbz, w, X, Y, Z);
    case 27: return p2FaceDot<T, 27>(u, fw, pbz, w, X, Y, Z);
    case 28: return p2FaceDot<T, 28>(u, fw, pbz, w, X, Y, Z);
    case 29: return p2FaceDot<T, 29>(u, fw, pbz, w, X, Y, Z);
    case 30: return p2FaceDot<T, 30>(u, fw, pbz, w, X, Y, Z);
    default: return p2FaceDot<T, 31>(u, fw, pbz, w, X, Y, Z);
  }
}

template <class T, int MODE>
__global__ void __launch_bounds__(kBlock, 2) p2ApplyKernel(LevelDev lv, const P2Item* __restrict__ items,
                                                           const T* __restrict__ W, const T* __restrict__ FW,
                                                           T* __restrict__ dst, const T* __restrict__ src,
                                                           const T* __restrict__ rhs, unsigned mask) {
  waitForPredecessor(dst, src, rhs);
  extern __shared__ __align__(16) unsigned char p2Smem[];
  const int c = blockIdx.x % lv.nCells;
  const P2Item it = items[blockIdx.x / lv.nCells];
  const int M = lv.N, w = lv.w, tid = threadIdx.x;
  const int64_t base = lv.cellOff[c];
  const T* __restrict__ u = src + base;
  T* __restrict__ d = dst + base;
  if (it.kind == P2_TILE) {
    if (!(lv.cellType[c] & mask)) return;
    T* sm = reinterpret_cast<T*>(p2Smem);
    T* wts = sm + kP2RowTab * kP2Stride;
    int2* rows = reinterpret_cast<int2*>(wts + p2s::kTotal + 2);  // per staged row: index of its first node, nodes
    const int x0 = it.a, y0 = it.b, z0 = it.c;
    for (int k = tid; k < p2s::kTotal; k += kBlock) wts[k] = W[(int64_t)c * p2s::kTotal + kP2BlockDev.e[k].weight];
    for (int r = tid; r < kP2RowTab; r += kBlock) {
      const int z = z0 + r / kP2Region, y = y0 + r % kP2Region;
      const int n = min(M - z - y - x0 + 1, kP2Region);
      rows[r] = make_int2(n > 0 ? p2Row(w, y, z) + x0 : 0, n);
    }
    __syncthreads();
    // the staged rows as one list of (row, x), the loads of a round before its stores
    constexpr int kStage = kP2RowTab * kP2Stride, kRound = 4;
    for (int i0 = tid; i0 < kStage; i0 += kRound * kBlock) {
      T v[kRound];
      int o[kRound];
#pragma unroll
      for (int k = 0; k < kRound; ++k) {
        const int i = i0 + k * kBlock, r = i / kP2Stride, x = i - r * kP2Stride;
        const int2 row = i < kStage ? rows[r] : make_int2(0, 0);
        o[k] = x < row.y ? r * kP2Stride + (x & 1) * (kP2Stride / 2) + (x >> 1) : -1;
        if (o[k] >= 0) v[k] = __ldg(u + row.x + x);
      }
#pragma unroll
      for (int k = 0; k < kRound; ++k)
        if (o[k] >= 0) sm[o[k]] = v[k];
    }
    __syncthreads();
    // threads 8 x 4 x 8: a warp covers 16 x 8 nodes, two blocks deep in z
    const int tx = tid & 7, ty = (tid >> 3) & 3, q = tid >> 5, by = ty + 4 * (q & 1), bz = 2 * (q >> 1);
    const int X = x0 + 1 + 2 * tx, Y = y0 + 1 + 2 * by, Z = z0 + 1 + 2 * bz;
    if (X + Y + Z > M - 1) return;
    T acc[2][kP2Accs];
#pragma unroll
    for (int k = 0; k < kP2Accs; ++k) acc[0][k] = acc[1][k] = T(0);
    p2BlockDot<T>(std::make_integer_sequence<int, p2s::kTotal>{}, sm + (2 * bz * kP2Region + 2 * by) * kP2Stride + tx, wts,
                  acc);
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int y = Y + (k & 1), z = Z + 2 * b + (k >> 1);
        const int g = p2Row(w, y, z) + X;
#pragma unroll
        for (int a = 0; a < 2; ++a)
          if (X + a + y + z <= M - 1) {
            const int i = a + 2 * k;
            const T s = i == 7        ? (acc[b][7] + acc[b][8]) + (acc[b][9] + acc[b][10])
                        : p2Halves(i) ? acc[b][i] + acc[b][p2Second(i)]
                                      : acc[b][i];
            d[g + a] = MODE == MODE_RESIDUAL ? rhs[base + g + a] - s : s;
          }
      }
  } else if (it.kind == P2_FACE) {
    const int s = it.b + 1 + 2 * (tid & 15), t = it.c + 1 + 2 * (tid >> 4);
    if (s + t > M - 1) return;
    const T* fw = FW + (int64_t)c * p2s::kFaceTotal;
    using S = std::make_integer_sequence<int, kP2FaceEntries>;
    switch (it.a) {
      case 0: p2FaceBlock<T, 0>(S{}, u, fw, d, w, M, s, t); break;
      case 1: p2FaceBlock<T, 1>(S{}, u, fw, d, w, M, s, t); break;
      case 2: p2FaceBlock<T, 2>(S{}, u, fw, d, w, M, s, t); break;
      default: p2FaceBlock<T, 3>(S{}, u, fw, d, w, M, s, t); break;
    }
  } else {
    // per edge its odd nodes, then its even ones, so that the lanes of a warp mostly run one entry
    const int e = it.a + tid;
    if (e >= 6 * (M - 1) + 4) return;
    int X = 0, Y = 0, Z = 0, entry;
    if (e >= 6 * (M - 1)) {
      const int v = e - 6 * (M - 1);
      X = v == 1 ? M : 0;
      Y = v == 2 ? M : 0;
      Z = v == 3 ? M : 0;
      entry = 28 + v;
    } else {
      const int k = e / (M - 1), r = e - k * (M - 1), t = r < M / 2 ? 2 * r + 1 : 2 * (r - M / 2) + 2;
      X = k == 0 ? t : k == 3 || k == 4 ? M - t : 0;
      Y = k == 1 || k == 3 ? t : k == 5 ? M - t : 0;
      Z = k == 2 || k == 4 || k == 5 ? t : 0;
      entry = 16 + 2 * k + (t & 1);
    }
    int pbz[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int z = Z - 2 + k;
      pbz[k] = z >= 0 && z <= M ? int(tetSize(w) - tetSize(w - z)) : 0;
    }
    d[pbz[2] + rowStart(w - Z, Y) + X] = p2RimDot<T>(entry, u, FW + (int64_t)c * p2s::kFaceTotal, pbz, w, X, Y, Z);
  }
}

}  // namespace dev
}  // namespace hg
