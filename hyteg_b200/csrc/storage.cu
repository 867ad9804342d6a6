// hg_storage: device arena, per-level work tables, operators, solvers and the C-ABI.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/hyteg_b200.h"
#include "discretization.hpp"
#include "kernels.cuh"
#include "p2_apply.cuh"
#include "p2_sor.cuh"
#include "p2_stokes.cuh"
#include "solvers.hpp"
#include "storage.hpp"

namespace hg {

thread_local std::string g_lastError;
static const int kAllGroups = (1 << G_COUNT) - 1;

void cudaCheck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    if (e == cudaErrorMemoryAllocation) {
      (void)cudaGetLastError();
      throw Error(HG_ERR_OOM, std::string(what) + ": " + cudaGetErrorString(e));
    }
    throw Error(HG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  }
}

void argCheck(bool ok, const std::string& msg) {
  if (!ok) throw Error(HG_ERR_ARG, msg);
}

DevBuf::~DevBuf() {
  if (p) cudaFree(p);
}
void* DevBuf::alloc(size_t n) {
  if (p) cudaFree(p);
  p = nullptr;
  bytes = n;
  if (!n) return p;
  cudaError_t e = cudaMalloc(&p, n);
  if (e == cudaErrorMemoryAllocation) {  // kept buffers go first
    (void)cudaGetLastError();
    int device = 0;
    cudaCheck(cudaGetDevice(&device), "cudaGetDevice");
    if (KeptBuffers::releaseAll(device)) e = cudaMalloc(&p, n);
  }
  cudaCheck(e, "cudaMalloc");
  return p;
}

// Every pool of the process; the mutex guards the list and the pools, which other storages' threads release.
static std::mutex keptMutex;
static std::vector<KeptBuffers*>& keptPools() {
  static auto* pools = new std::vector<KeptBuffers*>();
  return *pools;
}

KeptBuffers::KeptBuffers(int dev) : device(dev) {
  std::lock_guard<std::mutex> lock(keptMutex);
  keptPools().push_back(this);
}
KeptBuffers::~KeptBuffers() {
  std::lock_guard<std::mutex> lock(keptMutex);
  auto& pools = keptPools();
  pools.erase(std::find(pools.begin(), pools.end(), this));
  drop();
}
std::unique_ptr<DevBuf> KeptBuffers::take(int key) {
  std::lock_guard<std::mutex> lock(keptMutex);
  std::unique_ptr<DevBuf> b;
  for (size_t i = 0; i < free.size() && !b; ++i)
    if (free[i].first == key) {
      b = std::move(free[i].second);
      free.erase(free.begin() + (std::ptrdiff_t)i);
    }
  return b;
}
void KeptBuffers::give(int key, std::unique_ptr<DevBuf> buf) {
  std::lock_guard<std::mutex> lock(keptMutex);
  free.emplace_back(key, std::move(buf));
}
size_t KeptBuffers::drop() {
  size_t n = 0;
  for (auto& b : free) n += b.second->bytes;
  free.clear();
  return n;
}
size_t KeptBuffers::release() {
  std::lock_guard<std::mutex> lock(keptMutex);
  return drop();
}
size_t KeptBuffers::releaseAll(int device) {
  std::lock_guard<std::mutex> lock(keptMutex);
  size_t n = 0;
  for (KeptBuffers* p : keptPools())
    if (p->device == device) n += p->drop();
  return n;
}

template <class V>
static void* upload(std::vector<std::unique_ptr<DevBuf>>& keep, const std::vector<V>& h, cudaStream_t st) {
  keep.emplace_back(new DevBuf());
  void* d = keep.back()->alloc(std::max<size_t>(h.size(), 1) * sizeof(V));
  if (!h.empty()) cudaCheck(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(V), cudaMemcpyHostToDevice, st), "upload");
  return d;
}

static unsigned char dofType(int meshFlag) {
  // BoundaryCondition::create0123BC (src/hyteg/boundary/BoundaryConditions.cpp:26-33)
  switch (meshFlag) {
    case 1: return HG_DIRICHLET;
    case 2: return HG_NEUMANN;
    case 3: return HG_FREESLIP;
    default: return HG_INNER;
  }
}

template <class F>
static void allowSmem(F kernel, size_t bytes) {
  cudaCheck(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), "kernel shared memory");
}

Storage::Storage(const Topology& topo, int maxLevel) : disc(topo, maxLevel) {
  cudaCheck(cudaGetDevice(&device), "cudaGetDevice");
  kept.reset(new KeptBuffers(device));
  cudaCheck(cudaStreamCreateWithFlags(&ownStream, cudaStreamNonBlocking), "cudaStreamCreate");
  cudaCheck(cudaFuncSetAttribute(dev::cellSorWaveKernel<double, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)dev::waveSmemBytes<double, 0>(dev::kWaveMaxN)),
            "wave kernel shared memory");
  cudaCheck(cudaFuncSetAttribute(dev::cellSorWaveKernel<float, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)dev::waveSmemBytes<float, 0>(dev::kWaveMaxN)),
            "wave kernel shared memory");
  cudaCheck(cudaFuncSetAttribute(dev::cellSorWaveKernel<double, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)dev::waveSmemBytes<double, 1>(dev::kWaveMaxN)),
            "wave kernel shared memory");
  cudaCheck(cudaFuncSetAttribute(dev::cellSorWaveKernel<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)dev::waveSmemBytes<float, 1>(dev::kWaveMaxN)),
            "wave kernel shared memory");
  allowSmem(dev::cellSorResidentKernel<double>, dev::residentSmem<double>(dev::kResidentMaxN));
  allowSmem(dev::cellSorResidentKernel<float>, dev::residentSmem<float>(dev::kResidentMaxN));
  stream = ownStream;
  levels.resize(maxLevel + 1);
  for (int L = 0; L <= maxLevel; ++L) buildLevel(L);
  {
    const Topology& t = disc.topo();
    std::vector<double> vx;
    for (auto& v : t.verts)
      for (int d = 0; d < 3; ++d) vx.push_back(v.x[d]);
    std::vector<int> cv, fv, lv;
    for (auto& c : t.cells)
      for (int k = 0; k < 4; ++k) cv.push_back(c.v[k]);
    for (auto& f : t.faces)
      for (int k = 0; k < 3; ++k) fv.push_back(f.v[k]);
    for (auto& e : t.edges) {
      lv.push_back(e.v[0]);
      lv.push_back(e.v[1]);
    }
    for (size_t v = 0; v < t.verts.size(); ++v) {
      lv.push_back((int)v);
      lv.push_back((int)v);
    }
    geom.vx = (const double*)upload(geomKeep, vx, stream);
    geom.cellV = (const int*)upload(geomKeep, cv, stream);
    geom.faceV = (const int*)upload(geomKeep, fv, stream);
    geom.lowV = (const int*)upload(geomKeep, lv, stream);
  }
  scalars.alloc(64 * sizeof(double));
  cudaCheck(cudaMemsetAsync(scalars.p, 0, 64 * sizeof(double), stream), "memset");
  cudaCheck(cudaStreamSynchronize(stream), "sync");
}

Storage::~Storage() {
  p2gmgs.clear();
  gmgs.clear();
  ops.clear();
  fns.clear();
  levels.clear();
  if (ownStream) cudaStreamDestroy(ownStream);
}

static int64_t firstVertexSlot(const LevelLayout& lay) { return lay.off[KV].empty() ? lay.total : lay.off[KV][0]; }

// Calls f(destination, source) on the halo entries in the order of the level's table: group by group as
// generated, but the edge copies owned by vertices before the other edge copies.
template <class F>
static void forComm(const LevelLayout& lay, int g, F f) {
  const auto &d = lay.commDst[g], &s = lay.commSrc[g];
  if (g != G_EDGE) {
    for (size_t i = 0; i < d.size(); ++i) f(d[i], s[i]);
    return;
  }
  const int64_t first = firstVertexSlot(lay);
  for (const bool vertex : {true, false})
    for (size_t i = 0; i < d.size(); ++i)
      if ((s[i] >= first) == vertex) f(d[i], s[i]);
}

void Storage::buildLevel(int L) {
  const Topology& topo = disc.topo();
  const LevelLayout& lay = disc.level(L);
  LevelData& ld = levels[L];
  ld.lay = &lay;
  dev::LevelDev& lv = ld.lv;
  lv.L = L;
  lv.N = (int)lay.N;
  lv.w = (int)lay.w;
  lv.nCells = (int)topo.cells.size();
  lv.nFaces = (int)topo.faces.size();
  lv.nEdges = (int)topo.edges.size();
  lv.nLow = (int)(topo.edges.size() + topo.verts.size());
  const int64_t N = lay.N, w = lay.w;
  argCheck(lay.total < (int64_t(1) << 32), "level buffer exceeds 32-bit halo indices");

  std::vector<int64_t> lowOff;
  std::vector<int> lowFirst, lowCount;
  std::vector<unsigned char> cellType, faceType, lowType;
  for (auto& c : topo.cells) cellType.push_back(dofType(c.flag));
  for (auto& f : topo.faces) faceType.push_back(dofType(f.flag));
  for (size_t e = 0; e < topo.edges.size(); ++e) {
    lowOff.push_back(lay.off[KE][e]);
    lowFirst.push_back(1);
    lowCount.push_back((int)std::max<int64_t>(N - 1, 0));
    lowType.push_back(dofType(topo.edges[e].flag));
  }
  for (size_t v = 0; v < topo.verts.size(); ++v) {
    lowOff.push_back(lay.off[KV][v]);
    lowFirst.push_back(0);
    lowCount.push_back(1);
    lowType.push_back(dofType(topo.verts[v].flag));
  }
  ld.hostCellType = cellType;
  ld.hostFaceType = faceType;
  ld.hostLowType = lowType;

  lv.nCellBlocks = N >= 4 ? lv.nCells * (int)(N - 3) : 0;
  std::vector<dev::FaceBlock> fb;
  if (N >= 3)
    for (int f = 0; f < lv.nFaces; ++f)
      for (int y = 1; y < (int)w - 2; y += dev::kFaceRows) fb.push_back({f, y});
  std::vector<dev::FaceBlock> bands;
  if (N >= 3)
    for (int f = 0; f < lv.nFaces; ++f)
      for (int y = 1; y < (int)w - 2; y += dev::kFaceBand) bands.push_back({f, y});
  std::vector<dev::LowBlock> lb;
  for (int p = 0; p < lv.nLow; ++p) {
    if (p == lv.nEdges) lv.nLowEdgeBlocks = (int)lb.size();
    for (int s = lowFirst[p]; s < lowFirst[p] + lowCount[p]; s += dev::kBlock) lb.push_back({p, s});
  }
  if (lv.nEdges == lv.nLow) lv.nLowEdgeBlocks = (int)lb.size();

  std::vector<dev::Chunk> chunks;
  auto addChunks = [&](int64_t off, int64_t size, int type) {
    for (int64_t s = 0; s < size; s += 8192) chunks.push_back({off + s, (int)std::min<int64_t>(8192, size - s), type});
  };
  for (int c = 0; c < lv.nCells; ++c) addChunks(lay.off[KC][c], lay.size[KC][c], cellType[c]);
  for (int f = 0; f < lv.nFaces; ++f) addChunks(lay.off[KF][f], lay.size[KF][f], faceType[f]);
  for (int e = 0; e < lv.nEdges; ++e) addChunks(lay.off[KE][e], lay.size[KE][e], lowType[e]);
  for (size_t v = 0; v < topo.verts.size(); ++v) addChunks(lay.off[KV][v], lay.size[KV][v], lowType[lv.nEdges + v]);

  // halo table in the five destination groups
  std::vector<uint2> comm;
  size_t nComm = 0;
  for (int g : kCommOrder) nComm += lay.commDst[g].size();
  comm.reserve(nComm);
  for (int g : kCommOrder) {
    ld.commBegin[g] = (int64_t)comm.size();
    forComm(lay, g, [&](int64_t d, int64_t s) { comm.push_back(make_uint2((unsigned)d, (unsigned)s)); });
    ld.commCount[g] = (int64_t)comm.size() - ld.commBegin[g];
  }
  ld.commEdgeOther = ld.commBegin[G_EDGE];
  while (ld.commEdgeOther < ld.commBegin[G_EDGE] + ld.commCount[G_EDGE] &&
         (int64_t)comm[(size_t)ld.commEdgeOther].y >= firstVertexSlot(lay))
    ++ld.commEdgeOther;
  argCheck(comm.size() < (size_t(1) << 31), "halo table exceeds 32-bit ranges");
  // Each primitive's entries of a group are contiguous and the primitives follow one another (the
  // tables are generated primitive by primitive, and so are the arrays): the range of every
  // primitive's destination array in one walk over both.
  auto ranges = [&](int g, int kind, int nPrim) {
    std::vector<int2> r((size_t)nPrim, make_int2(0, 0));
    const auto &offs = lay.off[kind], &size = lay.size[kind];
    int p = 0, last = -1;
    // of the edge copies only those owned by vertices (the phases refresh the others before)
    const int64_t end = g == G_EDGE ? ld.commEdgeOther : ld.commBegin[g] + ld.commCount[g];
    for (int64_t i = ld.commBegin[g]; i < end; ++i) {
      const int64_t d = comm[(size_t)i].x;
      while (p < nPrim && d >= offs[(size_t)p] + size[(size_t)p]) ++p;
      argCheck(p < nPrim && d >= offs[(size_t)p], "halo entry outside its group's kind, or out of order");
      if (p != last) {
        r[(size_t)p].x = (int)i;
        last = p;
      }
      r[(size_t)p].y = (int)i + 1;
    }
    return r;
  };
  {
    std::vector<int2> low = ranges(G_EDGE, KE, lv.nEdges);
    std::vector<int2> vr = ranges(G_VERT, KV, (int)topo.verts.size());
    low.insert(low.end(), vr.begin(), vr.end());
    std::vector<int2> fr = ranges(G_FACE_BOUNDARY, KF, lv.nFaces);
    if (!low.empty()) ld.lowRange = (const int2*)upload(ld.keep, low, stream);
    if (!fr.empty()) ld.faceRange = (const int2*)upload(ld.keep, fr, stream);
    if (dev::residentLevel((int)N)) {
      // every cell has the same closure
      const int per = lv.nCells ? (int)(ld.commCount[G_CELL] / lv.nCells) : 0;
      std::vector<int2> cells;
      for (int c = 0; c < lv.nCells; ++c) {
        const int first = (int)ld.commBegin[G_CELL] + c * per;
        cells.push_back(make_int2(first, first + per));
        for (const int i : {first, first + per - 1})
          argCheck(comm[(size_t)i].x >= lay.off[KC][c] && comm[(size_t)i].x < lay.off[KC][c] + lay.size[KC][c],
                   "closure entry outside its cell");
      }
      ld.cellRange = (const int2*)upload(ld.keep, cells, stream);
      buildSplitRows(L);
    }
  }

  auto& keep = ld.keep;
  lv.cellOff = (const int64_t*)upload(keep, lay.off[KC], stream);
  lv.faceOff = (const int64_t*)upload(keep, lay.off[KF], stream);
  lv.lowOff = (const int64_t*)upload(keep, lowOff, stream);
  lv.lowFirst = (const int*)upload(keep, lowFirst, stream);
  lv.lowCount = (const int*)upload(keep, lowCount, stream);
  lv.cellType = (const unsigned char*)upload(keep, cellType, stream);
  lv.faceType = (const unsigned char*)upload(keep, faceType, stream);
  lv.lowType = (const unsigned char*)upload(keep, lowType, stream);
  lv.faceBlocks = (const dev::FaceBlock*)upload(keep, fb, stream);
  lv.nFaceBlocks = (int)fb.size();
  lv.faceBands = (const dev::FaceBlock*)upload(keep, bands, stream);
  lv.nFaceBands = (int)bands.size();
  lv.lowBlocks = (const dev::LowBlock*)upload(keep, lb, stream);
  lv.nLowBlocks = (int)lb.size();
  ld.comm = (uint2*)upload(keep, comm, stream);
  ld.chunks = (dev::Chunk*)upload(keep, chunks, stream);
  buildTiles(L);
  // single-pass SOR tiles: every (x, y) of the cell is in exactly one tile, tallest tiles first;
  // one list per precision (the tile heights differ)
  {
    const int tys[2][2] = {{dev::WaveGeom<double, 0>::TY, dev::WaveGeom<double, 1>::TY},
                           {dev::WaveGeom<float, 0>::TY, dev::WaveGeom<float, 1>::TY}};
    for (int pi = 0; pi < 2; ++pi)
      for (int gv = 0; gv < 2; ++gv) {
        const int ty = tys[pi][gv];
        std::vector<dev::WaveTile> wt;
        if (N >= 4)
          for (int c = 0; c < lv.nCells; ++c)
            for (int y0 = 0; y0 <= N; y0 += ty)
              for (int x0 = 0; x0 + y0 <= N; x0 += dev::kWaveTX) wt.push_back({c, x0, y0, (int)N - x0 - y0});
        std::stable_sort(wt.begin(), wt.end(),
                         [](const dev::WaveTile& a, const dev::WaveTile& b) { return a.pEnd > b.pEnd; });
        ld.waveTiles[pi][gv] = (dev::WaveTile*)upload(keep, wt, stream);
        ld.nWaveTiles[pi][gv] = (int)wt.size();
      }
    int64_t first = lay.total;
    for (int k : {KV, KE, KF})
      for (int64_t o : lay.off[k]) first = std::min(first, o);
    for (size_t c = 0; c < lay.off[KC].size(); ++c)
      argCheck(lay.off[KC][c] + lay.size[KC][c] <= first, "cell arrays must precede the other primitives");
    ld.nonCellBegin = first;
  }
  ld.nChunks = (int)chunks.size();
  const int nPartial = std::max(1, lv.nCellBlocks + lv.nFaceBlocks + lv.nLowBlocks);
  ld.partial.alloc(sizeof(double) * (size_t)(nPartial + 1));
  ld.arrived = (unsigned*)((double*)ld.partial.p + nPartial);
  cudaCheck(cudaMemsetAsync(ld.arrived, 0, sizeof(double), stream), "dot counter");
  cudaCheck(cudaStreamSynchronize(stream), "level upload");
}

// Cell-sweep work items: (cell, 30-column x 32-row block of strips, a few planes), the
// longest first inside groups of macro-cells whose two FP64 vectors fit into the L2 budget;
// the SOR colours of a group run back to back so that their re-reads hit L2.
void Storage::buildTiles(int L) {
  LevelData& ld = levels[L];
  const int64_t N = ld.lay->N, w = ld.lay->w;
  const int nCells = ld.lv.nCells;
  std::vector<dev::StripItem> items;
  const int64_t cellBytes = tet(w) * 8;
  ld.cellsPerGroup = (int)std::max<int64_t>(1, std::min<int64_t>(nCells, l2Budget / (2 * cellBytes)));
  ld.tileGroupBegin.assign(1, 0);
  for (int g0 = 0; N >= 4 && g0 < nCells; g0 += ld.cellsPerGroup) {
    std::vector<dev::StripItem> grp;
    for (int c = g0; c < std::min(nCells, g0 + ld.cellsPerGroup); ++c)
      for (int y0 = 1; y0 <= N - 3; y0 += dev::kStripRows)
        for (int x0 = 1; x0 <= N - 3; x0 += dev::kStripX) {
          const int zmax = (int)N - 1 - x0 - y0;  // last plane with an interior point in the block
          if (zmax < 1) continue;
          const int planes = dev::stripPlanes((int)N);
          for (int z0 = 1; z0 <= zmax; z0 += planes)
            grp.push_back({c, x0, y0, z0, std::min(zmax + 1, z0 + planes), 0, 0, 0});
        }
    std::stable_sort(grp.begin(), grp.end(),
                     [](const dev::StripItem& a, const dev::StripItem& b) { return (a.z1 - a.z0) > (b.z1 - b.z0); });
    items.insert(items.end(), grp.begin(), grp.end());
    ld.tileGroupBegin.push_back((int)items.size());
  }
  ld.tileBuf.reset(new DevBuf());
  ld.tiles = (dev::StripItem*)ld.tileBuf->alloc(std::max<size_t>(items.size(), 1) * sizeof(dev::StripItem));
  if (!items.empty())
    cudaCheck(cudaMemcpyAsync(ld.tiles, items.data(), items.size() * sizeof(dev::StripItem), cudaMemcpyHostToDevice,
                              stream),
              "strip items");
  ld.nTiles = (int)items.size();
  cudaCheck(cudaStreamSynchronize(stream), "strip items sync");
}

void Storage::setL2Budget(int64_t bytes) {
  argCheck(bytes > 0, "L2 budget must be positive");
  l2Budget = bytes;
  ++generation;
  for (int L = 0; L <= maxLevel(); ++L) buildTiles(L);
}

// ------------------------------------------------------------------------------------------
// functions
// ------------------------------------------------------------------------------------------
static int keptKey(int L, int prec) { return 2 * L + (prec == 4 ? 1 : 0); }

int Storage::borrowFunction(int L, int prec) {
  argCheck(L >= 0 && L <= maxLevel(), "invalid level range");
  argCheck(prec == 8 || prec == 4, "precision must be 8 or 4");
  std::unique_ptr<DevBuf> buf = kept->take(keptKey(L, prec));
  if (!buf) return createFunction(L, L, prec);
  std::unique_ptr<Function> f(new Function());
  f->minL = f->maxL = L;
  f->prec = prec;
  f->levels.push_back(std::move(buf));
  const int id = nextId++;
  fns[id] = std::move(f);
  return id;
}

void Storage::returnFunction(int id, bool give) {
  auto it = fns.find(id);
  if (it == fns.end()) return;
  Function& f = *it->second;
  if (give) kept->give(keptKey(f.minL, f.prec), std::move(f.levels[0]));
  fns.erase(it);
}

void Storage::cgUpdate(int L, unsigned mask, bool direction, const double* num, const double* den, int x, int r, int p,
                       int ap) {
  const LevelData& ld = levels[L];
  if (!ld.nChunks) return;
  auto run = [&](auto zero) {
    using T = decltype(zero);
    T *xd = direction ? nullptr : (T*)data(x, L), *ad = direction ? nullptr : (T*)data(ap, L);
    if (direction)
      launchNext(stream, dev::cgUpdateKernel<T, true>, ld.nChunks, dev::kBlock, 0, ld.chunks, mask, num, den, xd,
                 (T*)data(r, L), (T*)data(p, L), ad);
    else
      launchNext(stream, dev::cgUpdateKernel<T, false>, ld.nChunks, dev::kBlock, 0, ld.chunks, mask, num, den, xd,
                 (T*)data(r, L), (T*)data(p, L), ad);
  };
  if (fn(r).prec == 8) run(0.0);
  else run(0.0f);
  ++launches;
  cudaCheck(cudaGetLastError(), "CG update");
}

Function& Storage::fn(int id) {
  auto it = fns.find(id);
  argCheck(it != fns.end(), "unknown function handle");
  return *it->second;
}
void* Storage::data(int id, int L) {
  Function& f = fn(id);
  argCheck(L >= f.minL && L <= f.maxL, "level outside the function's level range");
  return f.levels[L - f.minL]->p;
}
int Storage::createFunction(int minL, int maxL, int prec) {
  argCheck(minL >= 0 && maxL <= maxLevel() && minL <= maxL, "invalid level range");
  argCheck(prec == 8 || prec == 4, "precision must be 8 or 4");
  std::unique_ptr<Function> f(new Function());
  f->minL = minL;
  f->maxL = maxL;
  f->prec = prec;
  for (int L = minL; L <= maxL; ++L) {
    f->levels.emplace_back(new DevBuf());
    const size_t bytes = (size_t)levels[L].lay->total * prec;
    f->levels.back()->alloc(bytes);
    cudaCheck(cudaMemsetAsync(f->levels.back()->p, 0, bytes, stream), "memset");
  }
  const int id = nextId++;
  fns[id] = std::move(f);
  return id;
}

static unsigned grid1d(int64_t n) { return (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 32); }

void Storage::communicate(int id, int L, int groupMask) {
  Function& f = fn(id);
  void* d = data(id, L);
  const LevelData& ld = levels[L];
  // one gather per contiguous run of selected groups in the table
  int k = 0;  // position in the table order
  while (k < G_COUNT) {
    if (!(groupMask & (1 << kCommOrder[k]))) {
      ++k;
      continue;
    }
    const int64_t begin = ld.commBegin[kCommOrder[k]];
    int64_t n = 0;
    while (k < G_COUNT && (groupMask & (1 << kCommOrder[k]))) n += ld.commCount[kCommOrder[k++]];
    if (n == 0) continue;
    if (f.prec == 8)
      launchNext(stream, dev::commGatherKernel<double>, grid1d(n), 256, 0, (double*)d, ld.comm + begin, n);
    else
      launchNext(stream, dev::commGatherKernel<float>, grid1d(n), 256, 0, (float*)d, ld.comm + begin, n);
    ++launches;
  }
  cudaCheck(cudaGetLastError(), "communicate");
}

template <class T>
void Storage::communicateSplit(T* buf, T* cells, int L, int groupMask) {
  buildSplit(L);
  const LevelData& ld = levels[L];
  const uint2* table = ld.commSplit;
  int k = 0;  // position in the table order
  while (k < G_COUNT) {
    if (!(groupMask & (1 << kCommOrder[k]))) {
      ++k;
      continue;
    }
    const int64_t begin = ld.commBegin[kCommOrder[k]];
    int64_t n = 0;
    while (k < G_COUNT && (groupMask & (1 << kCommOrder[k]))) n += ld.commCount[kCommOrder[k++]];
    if (n == 0) continue;
    launchNext(stream, dev::commGatherSplitKernel<T>, grid1d(n), 256, 0, buf, cells, table + begin, n, ld.nonCellBegin);
    ++launches;
  }
  cudaCheck(cudaGetLastError(), "communicate (split)");
}

// The interior rows of colour col of a closed macro-cell with w points per edge (x, y, z >= 1,
// x + y + z <= w - 2), each with its 15 slots at j = 0 in the colour-split order, and the
// colour's points as (row << kSplitJBits | j), in (z, y, j) order.
void splitTables(int64_t w, int col, std::vector<dev::SplitRow>& rows, std::vector<unsigned>& points) {
  const int64_t N = w - 1;
  argCheck(N <= 4096, "colour-split SOR: level too large");
  auto tet = [](int64_t a) { return a * (a + 1) * (a + 2) / 6; };
  auto tri = [](int64_t a) { return a * (a + 1) / 2; };
  auto rowStart = [&](int64_t z, int64_t y) {
    const int64_t W = w - z;
    return tet(w) - tet(W) + y * (W + 1) - y * (y + 1) / 2;
  };
  rows.clear();
  points.clear();
  for (int64_t z = 1; z <= N - 3; ++z) {
    const int64_t W = w - z;
    for (int64_t y = 1; y <= W - 3; ++y) {
      const int m = (int)(W - y);
      const int q = (int)((((col - 2 * y - 3 * z) % 4) + 4) % 4);
      const int j0 = q == 0 ? 1 : 0, jEnd = m - 2 - q >= 0 ? (m - 2 - q) / 4 : -1;
      if (jEnd < j0) continue;
      const int qE = (q + 1) & 3, qW = (q + 3) & 3, jE = q == 3 ? 1 : 0, jW = q == 0 ? -1 : 0;
      const int64_t r0 = rowStart(z, y), rN = r0 + m, rS = r0 - (m + 1);
      const int64_t rT = r0 + tri(W) - y, rTS = rT - m, rB = r0 - tri(W + 1) + y, rBN = rB + (m + 1);
      auto sub = [](int mm, int qq) { return (int64_t)dev::splitSub(mm, qq); };
      dev::SplitRow r;
      const int64_t v[16] = {r0 + sub(m, q),          r0 + sub(m, qE) + jE,      r0 + sub(m, qW) + jW,
                             rN + sub(m - 1, q),      rS + sub(m + 1, q),        rN + sub(m - 1, qW) + jW,
                             rS + sub(m + 1, qE) + jE, rT + sub(m - 1, q),       rT + sub(m - 1, qW) + jW,
                             rTS + sub(m, q),         rTS + sub(m, qE) + jE,     rB + sub(m + 1, q),
                             rB + sub(m + 1, qE) + jE, rBN + sub(m, q),          rBN + sub(m, qW) + jW,
                             0};
      for (int k = 0; k < 16; ++k) r.i[k] = (int)v[k];
      argCheck(rows.size() < (size_t(1) << (32 - dev::kSplitJBits)), "colour-split SOR: too many rows");
      const unsigned id = (unsigned)rows.size();
      rows.push_back(r);
      for (int j = j0; j <= jEnd; ++j) points.push_back(id << dev::kSplitJBits | (unsigned)j);
    }
  }
}

// Position of every point of a closed macro-cell with w points per edge in the colour-split order (a
// permutation inside each row).
static std::vector<int> splitPermutation(int64_t w) {
  auto tet = [](int64_t a) { return a * (a + 1) * (a + 2) / 6; };
  std::vector<int> perm((size_t)tet(w));
  int64_t r0 = 0;
  for (int64_t z = 0; z < w; ++z)
    for (int64_t y = 0; y < w - z; ++y) {
      const int m = (int)(w - z - y);
      for (int x = 0; x < m; ++x) perm[(size_t)(r0 + x)] = (int)(r0 + dev::splitSub(m, x & 3) + (x >> 2));
      r0 += m;
    }
  return perm;
}

// Per colour the interior rows (their 15 slots at j = 0) and points (row << 10 | j) that
// cellSorSplitKernel and cellSorResidentKernel walk, the same for every macro-cell of the level, and for
// the latter the permutation: one buffer, from the lattice size alone. Resident levels have it from the
// storage's creation, so that no sweep allocates or waits for it.
void Storage::buildSplitRows(int L) {
  LevelData& ld = levels[L];
  if (ld.splitBuf) return;
  const int64_t w = ld.lay->w;
  std::vector<dev::SplitRow> rows[4];
  std::vector<unsigned> points[4];
  std::vector<uint16_t> perm16;
  size_t nRows = 0, nPoints = 0;
  for (int col = 0; col < 4; ++col) {
    splitTables(w, col, rows[col], points[col]);
    nRows += rows[col].size();
    nPoints += points[col].size();
  }
  if (dev::residentLevel((int)w - 1)) {
    const std::vector<int> perm = splitPermutation(w);
    perm16.assign(perm.begin(), perm.end());
  }
  const size_t pointsAt = nRows * sizeof(dev::SplitRow), permAt = pointsAt + nPoints * sizeof(unsigned);
  std::vector<unsigned char> host(std::max<size_t>(permAt + perm16.size() * sizeof(uint16_t), 16));
  std::unique_ptr<DevBuf> buf(new DevBuf());
  unsigned char* d = (unsigned char*)buf->alloc(host.size());
  size_t r = 0, p = pointsAt;
  for (int col = 0; col < 4; ++col) {
    if (!rows[col].empty()) std::memcpy(&host[r], rows[col].data(), rows[col].size() * sizeof(dev::SplitRow));
    if (!points[col].empty()) std::memcpy(&host[p], points[col].data(), points[col].size() * sizeof(unsigned));
    ld.splitRows[col] = (const dev::SplitRow*)(d + r);
    ld.splitPoints[col] = (const unsigned*)(d + p);
    ld.nSplitPoints[col] = (int)points[col].size();
    r += rows[col].size() * sizeof(dev::SplitRow);
    p += points[col].size() * sizeof(unsigned);
  }
  if (!perm16.empty()) {
    std::memcpy(&host[permAt], perm16.data(), perm16.size() * sizeof(uint16_t));
    ld.splitPerm = (const uint16_t*)(d + permAt);
  }
  cudaCheck(cudaMemcpyAsync(d, host.data(), host.size(), cudaMemcpyHostToDevice, stream), "colour-split rows");
  cudaCheck(cudaStreamSynchronize(stream), "colour-split rows");  // the host copy goes out of scope
  ld.splitBuf = std::move(buf);
}

// Schedule-3 tables of level L: the rows, and the halo table with every slot of a cell array replaced by
// its position in the colour-split order.
void Storage::buildSplit(int L) {
  LevelData& ld = levels[L];
  if (ld.commSplit) return;
  const LevelLayout& lay = *ld.lay;
  argCheck(lay.w - 1 <= 4096, "colour-split SOR: level too large");
  const std::vector<int> perm = splitPermutation(lay.w);
  std::vector<std::pair<int64_t, int64_t>> cells;  // (offset, size), ascending
  for (size_t c = 0; c < lay.off[KC].size(); ++c) cells.push_back({lay.off[KC][c], lay.size[KC][c]});
  std::sort(cells.begin(), cells.end());
  auto map = [&](int64_t slot) -> unsigned {
    if (slot < ld.nonCellBegin && !cells.empty()) {
      auto it = std::upper_bound(cells.begin(), cells.end(), std::make_pair(slot, INT64_MAX));
      if (it != cells.begin()) {
        --it;
        const int64_t local = slot - it->first;
        if (local < it->second && local < (int64_t)perm.size()) return (unsigned)(it->first + perm[(size_t)local]);
      }
    }
    return (unsigned)slot;
  };
  std::vector<uint2> comm;  // the same entries in the same order as the level's table
  for (int g : kCommOrder) forComm(lay, g, [&](int64_t d, int64_t s) { comm.push_back(make_uint2(map(d), map(s))); });
  const uint2* commSplit = comm.empty() ? ld.comm : (const uint2*)upload(ld.keep, comm, stream);
  buildSplitRows(L);
  cudaCheck(cudaStreamSynchronize(stream), "colour-split tables");  // the host vectors go out of scope
  ld.commSplit = commSplit;
}

DevBuf& Storage::spareBuf(std::map<std::pair<int, int>, std::unique_ptr<DevBuf>>& pool, int L, int prec) {
  std::unique_ptr<DevBuf>& sp = pool[{L, prec}];
  const size_t bytes = (size_t)levels[L].lay->total * prec;
  if (!sp || sp->bytes != bytes) {
    sp.reset(new DevBuf());
    sp->alloc(bytes);
    cudaCheck(cudaMemsetAsync(sp->p, 0, sp->bytes, stream), "spare memset");  // alignment padding stays zero
  }
  return *sp;
}

int Storage::sorScheduleFor(int L, int prec) const {
  const int tuned = 2 * L + (prec == 4 ? 1 : 0);
  return (int)sorScheduleLevel.size() > tuned && sorScheduleLevel[tuned] >= 0 ? sorScheduleLevel[tuned] : sorSchedule;
}

void Storage::lincomb(int dst, int L, unsigned mask, int n, const double* a, const int* srcs, bool add,
                      double constant) {
  argCheck(n >= 0 && n <= 3, "at most three source functions");
  Function& fd = fn(dst);
  void* pd = data(dst, L);
  const void* ps[3] = {nullptr, nullptr, nullptr};
  double sc[3] = {0, 0, 0};
  for (int i = 0; i < n; ++i) {
    argCheck(fn(srcs[i]).prec == fd.prec, "assign/add require functions of equal precision");
    ps[i] = data(srcs[i], L);
    sc[i] = a[i];
  }
  const LevelData& ld = levels[L];
  if (ld.nChunks == 0) return;
  auto run = [&](auto zero) {
    using T = decltype(zero);
    auto go = [&](auto nsrc, auto addTo) {
      launchNext(stream, dev::lincombKernel<T, decltype(nsrc)::value, decltype(addTo)::value>, ld.nChunks,
                 dev::kBlock, 0, ld.chunks, mask, (T*)pd, (const T*)ps[0], (const T*)ps[1], (const T*)ps[2], T(sc[0]),
                 T(sc[1]), T(sc[2]), T(constant));
    };
    auto pick = [&](auto nsrc) {
      if (add) go(nsrc, std::true_type{});
      else go(nsrc, std::false_type{});
    };
    if (n == 0) pick(std::integral_constant<int, 0>{});
    else if (n == 1) pick(std::integral_constant<int, 1>{});
    else if (n == 2) pick(std::integral_constant<int, 2>{});
    else pick(std::integral_constant<int, 3>{});
  };
  if (fd.prec == 8) run(0.0);
  else run(0.0f);
  ++launches;
  cudaCheck(cudaGetLastError(), "lincomb");
}

void Storage::divideBy(int dst, int a, int b, int L, unsigned mask) {
  argCheck(fn(dst).prec == 8 && fn(a).prec == 8 && fn(b).prec == 8, "divide: FP64 functions required");
  const LevelData& ld = levels[L];
  if (!ld.nChunks) return;
  dev::divideKernel<<<ld.nChunks, dev::kBlock, 0, stream>>>(ld.chunks, mask, (double*)data(dst, L),
                                                             (const double*)data(a, L), (const double*)data(b, L));
  ++launches;
  cudaCheck(cudaGetLastError(), "divide");
}

void Storage::copyCast(int dst, int src, int L, unsigned mask, bool add) {
  Function& fd = fn(dst);
  Function& fs = fn(src);
  void* pd = data(dst, L);
  void* ps = data(src, L);
  const LevelData& ld = levels[L];
  if (ld.nChunks == 0) return;
  const int a = add ? 1 : 0;
  if (fd.prec == 8 && fs.prec == 8)
    launchNext(stream, dev::castKernel<double, double>, ld.nChunks, dev::kBlock, 0, ld.chunks, mask, (double*)pd,
               (const double*)ps, a);
  else if (fd.prec == 8)
    launchNext(stream, dev::castKernel<double, float>, ld.nChunks, dev::kBlock, 0, ld.chunks, mask, (double*)pd,
               (const float*)ps, a);
  else if (fs.prec == 8)
    launchNext(stream, dev::castKernel<float, double>, ld.nChunks, dev::kBlock, 0, ld.chunks, mask, (float*)pd,
               (const double*)ps, a);
  else
    launchNext(stream, dev::castKernel<float, float>, ld.nChunks, dev::kBlock, 0, ld.chunks, mask, (float*)pd,
               (const float*)ps, a);
  ++launches;
  cudaCheck(cudaGetLastError(), "copyCast");
}

void Storage::dotAsync(int a, int b, int L, unsigned mask, double* dOut) {
  Function& fa = fn(a);
  argCheck(fa.prec == fn(b).prec, "dot requires functions of equal precision");
  const LevelData& ld = levels[L];
  const int nb = ld.lv.nCellBlocks + ld.lv.nFaceBlocks + ld.lv.nLowBlocks;
  double* partial = (double*)ld.partial.p;
  if (fa.prec == 8)
    launchNext(stream, dev::dotReduceKernel<double>, nb, dev::kBlock, 0, ld.lv, (const double*)data(a, L),
               (const double*)data(b, L), mask, partial, ld.arrived, dOut);
  else
    launchNext(stream, dev::dotReduceKernel<float>, nb, dev::kBlock, 0, ld.lv, (const float*)data(a, L),
               (const float*)data(b, L), mask, partial, ld.arrived, dOut);
  ++launches;
  cudaCheck(cudaGetLastError(), "dot");
}

PackStage::~PackStage() {
  if (copied) cudaEventDestroy(copied);
  if (used) cudaEventDestroy(used);
}

const OwnedPack& Storage::ownedPack(int L) {
  argCheck(L >= 0 && L <= maxLevel(), "level out of range");
  std::unique_ptr<OwnedPack>& op = ownedPacks[L];
  if (!op) {
    const std::vector<SlotRun> runs = ownedRuns(disc, L);
    std::vector<dev::OwnedRun> dr;
    dr.reserve(runs.size());
    int64_t packed = 0;
    for (const SlotRun& r : runs) {
      argCheck(r.len > 0 && r.len < (int64_t(1) << 31), "owned run length");
      dr.push_back({r.slot, packed, (int)r.len, 0});
      packed += r.len;
    }
    std::unique_ptr<OwnedPack> p(new OwnedPack());
    p->nRuns = (int64_t)dr.size();
    p->count = packed;
    p->runs.alloc(std::max<size_t>(dr.size(), 1) * sizeof(dev::OwnedRun));
    if (!dr.empty())
      cudaCheck(cudaMemcpyAsync(p->runs.p, dr.data(), dr.size() * sizeof(dev::OwnedRun), cudaMemcpyHostToDevice, stream),
                "owned runs");
    cudaCheck(cudaStreamSynchronize(stream), "owned runs");
    op = std::move(p);
  }
  return *op;
}

static PackStage& packStage(Function& f, int L, int64_t count) {
  std::unique_ptr<PackStage>& ps = f.stage[L];
  if (!ps) {
    ps.reset(new PackStage());
    ps->buf.alloc(std::max<size_t>((size_t)count * f.prec, 16));
    cudaCheck(cudaEventCreateWithFlags(&ps->copied, cudaEventDisableTiming), "event");
    cudaCheck(cudaEventCreateWithFlags(&ps->used, cudaEventDisableTiming), "event");
  }
  return *ps;
}

static unsigned packGrid(int64_t nRuns) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((nRuns + 7) / 8, 148 * 16)); }

void Storage::uploadOwned(int id, int L, const void* host, int64_t n, cudaStream_t copyStream) {
  Function& f = fn(id);
  argCheck(L >= f.minL && L <= f.maxL, "level outside the function's range");
  argCheck(host != nullptr, "null host buffer");
  const OwnedPack& op = ownedPack(L);
  argCheck(n == op.count, "upload size must equal the number of owned DoFs of the level");
  PackStage& ps = packStage(f, L, op.count);
  cudaCheck(cudaStreamWaitEvent(copyStream, ps.used, 0), "wait");  // the previous unpack has read the buffer
  cudaCheck(cudaMemcpyAsync(ps.buf.p, host, (size_t)n * f.prec, cudaMemcpyHostToDevice, copyStream), "owned upload");
  cudaCheck(cudaEventRecord(ps.copied, copyStream), "event");
  cudaCheck(cudaStreamWaitEvent(stream, ps.copied, 0), "wait");
  if (op.nRuns) {
    if (f.prec == 8)
      dev::ownedPackKernel<double, false><<<packGrid(op.nRuns), dev::kBlock, 0, stream>>>(
          (const dev::OwnedRun*)op.runs.p, op.nRuns, (double*)data(id, L), (double*)ps.buf.p);
    else
      dev::ownedPackKernel<float, false><<<packGrid(op.nRuns), dev::kBlock, 0, stream>>>(
          (const dev::OwnedRun*)op.runs.p, op.nRuns, (float*)data(id, L), (float*)ps.buf.p);
    ++launches;
    cudaCheck(cudaGetLastError(), "owned unpack");
  }
  cudaCheck(cudaEventRecord(ps.used, stream), "event");
  communicate(id, L, kAllGroups);
}

void Storage::downloadOwned(int id, int L, void* host, int64_t n, cudaStream_t copyStream) {
  Function& f = fn(id);
  argCheck(L >= f.minL && L <= f.maxL, "level outside the function's range");
  argCheck(host != nullptr, "null host buffer");
  const OwnedPack& op = ownedPack(L);
  argCheck(n == op.count, "download size must equal the number of owned DoFs of the level");
  PackStage& ps = packStage(f, L, op.count);
  cudaCheck(cudaStreamWaitEvent(stream, ps.copied, 0), "wait");  // the previous download has left the buffer
  if (op.nRuns) {
    if (f.prec == 8)
      dev::ownedPackKernel<double, true><<<packGrid(op.nRuns), dev::kBlock, 0, stream>>>(
          (const dev::OwnedRun*)op.runs.p, op.nRuns, (double*)data(id, L), (double*)ps.buf.p);
    else
      dev::ownedPackKernel<float, true><<<packGrid(op.nRuns), dev::kBlock, 0, stream>>>(
          (const dev::OwnedRun*)op.runs.p, op.nRuns, (float*)data(id, L), (float*)ps.buf.p);
    ++launches;
    cudaCheck(cudaGetLastError(), "owned pack");
  }
  cudaCheck(cudaEventRecord(ps.used, stream), "event");
  cudaCheck(cudaStreamWaitEvent(copyStream, ps.used, 0), "wait");
  cudaCheck(cudaMemcpyAsync(host, ps.buf.p, (size_t)n * f.prec, cudaMemcpyDeviceToHost, copyStream), "owned download");
  cudaCheck(cudaEventRecord(ps.copied, copyStream), "event");
}

dev::BatchMap Storage::batchMap(int L, int copies) const {
  argCheck(copies >= 1, "batch: at least one copy");
  const LevelData& ld = levels[L];
  const LevelLayout& lay = *ld.lay;
  const dev::LevelDev& lv = ld.lv;
  dev::BatchMap bm{};
  bm.copies = copies;
  const int kinds[4] = {KC, KF, KE, KV};
  int64_t a = 0;
  for (int q = 0; q < 4; ++q) {
    const auto& off = lay.off[kinds[q]];
    const auto& sz = lay.size[kinds[q]];
    const int n = (int)off.size();
    argCheck(n % copies == 0, "batch: primitives are not a multiple of the copies");
    const int per = n / copies;
    int64_t end = lay.total;  // the kind's block ends where the next non-empty kind begins
    for (int r = q + 1; r < 4; ++r)
      if (!lay.off[kinds[r]].empty()) {
        end = lay.off[kinds[r]][0];
        break;
      }
    bm.uBase[q] = n ? off[0] : end;
    bm.size[q] = n ? (end - off[0]) / copies : 0;
    argCheck(!n || bm.size[q] * copies == end - off[0], "batch: kind block is not a multiple of the copies");
    for (int i = 0; i < copies && n; ++i)
      for (int p = 0; p < per; ++p) {
        const size_t u = (size_t)i * per + p;
        argCheck(off[u] - (bm.uBase[q] + i * bm.size[q]) == off[(size_t)p] - bm.uBase[q] && sz[u] == sz[(size_t)p],
                 "batch: the copies' layouts differ");
      }
    bm.aBase[q] = a;
    a += bm.size[q];
  }
  const int nCellGrid = lv.N >= 4 ? lv.nCells * (lv.N - 3) : 0;
  const int counts[4] = {nCellGrid, lv.nFaceBlocks, lv.nLowEdgeBlocks, lv.nLowBlocks - lv.nLowEdgeBlocks};
  int base = 0;
  for (int q = 0; q < 4; ++q) {
    argCheck(counts[q] % copies == 0, "batch: work blocks are not a multiple of the copies");
    bm.bBase[q] = base;
    bm.bCount[q] = counts[q] / copies;
    base += counts[q];
  }
  return bm;
}

void Storage::fillRandomBatch(int id, int L, unsigned mask, const dev::BatchMap& bm, const uint64_t* dSeeds, int active,
                              double lo, double hi) {
  Function& f = fn(id);
  const LevelData& ld = levels[L];
  if (ld.nChunks) {
    if (f.prec == 8)
      dev::randomFillBatchKernel<double><<<ld.nChunks, dev::kBlock, 0, stream>>>(ld.chunks, mask, (double*)data(id, L), bm,
                                                                               dSeeds, active, lo, hi);
    else
      dev::randomFillBatchKernel<float><<<ld.nChunks, dev::kBlock, 0, stream>>>(ld.chunks, mask, (float*)data(id, L), bm,
                                                                              dSeeds, active, lo, hi);
    ++launches;
    cudaCheck(cudaGetLastError(), "batch random fill");
  }
  communicate(id, L, kAllGroups);
}

void Storage::dotBatchAsync(int a, int b, int L, unsigned mask, const dev::BatchMap& bm, double* dOut) {
  Function& fa = fn(a);
  argCheck(fa.prec == fn(b).prec, "dot requires functions of equal precision");
  const LevelData& ld = levels[L];
  const int nb = ld.lv.nCellBlocks + ld.lv.nFaceBlocks + ld.lv.nLowBlocks;
  if (fa.prec == 8)
    dev::dotKernel<double><<<nb, dev::kBlock, 0, stream>>>(ld.lv, (const double*)data(a, L), (const double*)data(b, L), mask,
                                                           (double*)ld.partial.p);
  else
    dev::dotKernel<float><<<nb, dev::kBlock, 0, stream>>>(ld.lv, (const float*)data(a, L), (const float*)data(b, L), mask,
                                                          (double*)ld.partial.p);
  dev::batchReduceKernel<<<bm.copies, dev::kBlock, 0, stream>>>((const double*)ld.partial.p, bm, dOut);
  launches += 2;
  cudaCheck(cudaGetLastError(), "batch dot");
}

void Storage::copyBatchSlots(int src, int dst, int L, const dev::BatchMap& bm, int copy) {
  Function& fs = fn(src);
  argCheck(fs.prec == fn(dst).prec, "batch copy: precision mismatch");
  char* d = (char*)data(dst, L);
  const char* sp = (const char*)data(src, L);
  for (int q = 0; q < 4; ++q)
    if (bm.size[q] > 0) {
      const size_t o = (size_t)(bm.uBase[q] + copy * bm.size[q]) * fs.prec;
      cudaCheck(cudaMemcpyAsync(d + o, sp + o, (size_t)bm.size[q] * fs.prec, cudaMemcpyDeviceToDevice, stream),
                "batch copy");
    }
}

void Storage::interpolateExpr(int id, int L, unsigned mask, int expr, const double* p) {
  argCheck(expr == 0 || expr == 1, "unknown expression");
  Function& f = fn(id);
  const LevelData& ld = levels[L];
  const int nb = ld.lv.nCellBlocks + ld.lv.nFaceBlocks + ld.lv.nLowBlocks;
  if (f.prec == 8)
    dev::interpolateKernel<double><<<nb, dev::kBlock, 0, stream>>>(ld.lv, geom, (double*)data(id, L), mask, expr, p[0], p[1],
                                                                   p[2], p[3]);
  else
    dev::interpolateKernel<float><<<nb, dev::kBlock, 0, stream>>>(ld.lv, geom, (float*)data(id, L), mask, expr, p[0], p[1],
                                                                  p[2], p[3]);
  ++launches;
  cudaCheck(cudaGetLastError(), "interpolate");
  communicate(id, L, kAllGroups);
}

void Storage::fillRandom(int id, int L, unsigned mask, uint64_t seed, double lo, double hi) {
  Function& f = fn(id);
  const LevelData& ld = levels[L];
  if (ld.nChunks) {
    if (f.prec == 8)
      dev::randomFillKernel<double><<<ld.nChunks, dev::kBlock, 0, stream>>>(ld.chunks, mask, (double*)data(id, L), seed, lo, hi);
    else
      dev::randomFillKernel<float><<<ld.nChunks, dev::kBlock, 0, stream>>>(ld.chunks, mask, (float*)data(id, L), seed, lo, hi);
    ++launches;
    cudaCheck(cudaGetLastError(), "random fill");
  }
  communicate(id, L, kAllGroups);
}

int64_t Storage::deviceBytes() const {
  int64_t b = (int64_t)scalars.bytes;
  for (auto& g : geomKeep) b += (int64_t)g->bytes;
  for (const LevelData& ld : levels) {
    for (auto& k : ld.keep) b += (int64_t)k->bytes;
    if (ld.tileBuf) b += (int64_t)ld.tileBuf->bytes;
    b += (int64_t)ld.partial.bytes;
  }
  for (auto& f : fns)
    for (auto& l : f.second->levels) b += (int64_t)l->bytes;
  for (auto& o : ops)
    for (auto& k : o.second->keep) b += (int64_t)k->bytes;
  for (auto& sp : spare)
    if (sp.second) b += (int64_t)sp.second->bytes;
  for (auto& sp : splitRhs)
    if (sp.second) b += (int64_t)sp.second->bytes;
  return b;
}

double Storage::dot(int a, int b, int L, unsigned mask) {
  double* d = (double*)scalars.p;
  dotAsync(a, b, L, mask, d);
  double h = 0;
  cudaCheck(cudaMemcpyAsync(&h, d, sizeof(double), cudaMemcpyDeviceToHost, stream), "dot readback");
  cudaCheck(cudaStreamSynchronize(stream), "dot sync");
  return h;
}

// ------------------------------------------------------------------------------------------
// operators
// ------------------------------------------------------------------------------------------
template <class T>
static dev::StencilDev<T> packStencil(std::vector<std::unique_ptr<DevBuf>>& keep, const LevelStencils& st,
                                      cudaStream_t stream) {
  std::vector<T> cellW;
  for (auto& c : st.cell)
    for (int k = 0; k < 16; ++k) cellW.push_back(T(c[k]));
  std::vector<dev::FaceEnt<T>> fe(st.face.size() * 16);
  std::vector<int> fc(st.face.size());
  for (size_t f = 0; f < st.face.size(); ++f) {
    argCheck(st.face[f].size() <= 16, "face stencil exceeds 16 entries");
    fc[f] = (int)st.face[f].size();
    for (size_t k = 0; k < st.face[f].size(); ++k)
      fe[16 * f + k] = {T(st.face[f][k].w), st.face[f][k].layer, st.face[f][k].dx, st.face[f][k].dy};
  }
  std::vector<int> off{0};
  std::vector<int64_t> rel;
  std::vector<T> wv;
  auto addLow = [&](const std::vector<LowEntry>& ent) {
    for (auto& e : ent) {
      rel.push_back(e.rel);
      wv.push_back(T(e.w));
    }
    off.push_back((int)rel.size());
  };
  for (auto& e : st.edge) addLow(e);
  for (auto& v : st.vert) addLow(v);
  dev::StencilDev<T> d;
  d.cellW = (const T*)upload(keep, cellW, stream);
  d.faceEnt = (const dev::FaceEnt<T>*)upload(keep, fe, stream);
  d.faceEntCount = (const int*)upload(keep, fc, stream);
  d.lowEntOff = (const int*)upload(keep, off, stream);
  d.lowEntRel = (const int64_t*)upload(keep, rel, stream);
  d.lowEntW = (const T*)upload(keep, wv, stream);
  return d;
}

// New stencil values into the device arrays of an existing operator (same topology, so the same
// sizes and index arrays): no device allocation or release, only copies on this stream.
template <class T>
static void refillStencil(const dev::StencilDev<T>& d, const LevelStencils& st, cudaStream_t stream) {
  std::vector<T> cellW;
  for (auto& c : st.cell)
    for (int k = 0; k < 16; ++k) cellW.push_back(T(c[k]));
  std::vector<dev::FaceEnt<T>> fe(st.face.size() * 16);
  for (size_t f = 0; f < st.face.size(); ++f)
    for (size_t k = 0; k < st.face[f].size(); ++k)
      fe[16 * f + k] = {T(st.face[f][k].w), st.face[f][k].layer, st.face[f][k].dx, st.face[f][k].dy};
  std::vector<T> wv;
  for (auto& e : st.edge)
    for (auto& x : e) wv.push_back(T(x.w));
  for (auto& v : st.vert)
    for (auto& x : v) wv.push_back(T(x.w));
  if (!cellW.empty())
    cudaCheck(cudaMemcpyAsync((void*)d.cellW, cellW.data(), cellW.size() * sizeof(T), cudaMemcpyHostToDevice, stream),
              "stencil refill");
  if (!fe.empty())
    cudaCheck(cudaMemcpyAsync((void*)d.faceEnt, fe.data(), fe.size() * sizeof(fe[0]), cudaMemcpyHostToDevice, stream),
              "stencil refill");
  if (!wv.empty())
    cudaCheck(cudaMemcpyAsync((void*)d.lowEntW, wv.data(), wv.size() * sizeof(T), cudaMemcpyHostToDevice, stream),
              "stencil refill");
  cudaCheck(cudaStreamSynchronize(stream), "stencil refill");
}

static std::vector<double> p2Stencils(const std::vector<double>& K, int nCells);
static std::vector<double> p2FaceStencils(const std::vector<double>& K, int nCells);

int Storage::createP2Operator(int form, int minL, int maxL) {
  argCheck(form == FORM_LAPLACE, "P2 operators: only the Laplace form is available");
  argCheck(minL >= 0 && maxL + 1 <= maxLevel() && minL <= maxL,
           "P2 level range needs the storage's levels up to max_level + 1");
  // here, not with the storage: this loads the kernels, which P1 programs never run
  allowSmem(dev::p2ApplyKernel<double, dev::MODE_REPLACE>, dev::p2TileSmem<double>());
  allowSmem(dev::p2ApplyKernel<double, dev::MODE_RESIDUAL>, dev::p2TileSmem<double>());
  allowSmem(dev::p2ApplyKernel<float, dev::MODE_REPLACE>, dev::p2TileSmem<float>());
  allowSmem(dev::p2ApplyKernel<float, dev::MODE_RESIDUAL>, dev::p2TileSmem<float>());
  std::unique_ptr<P2Operator> o(new P2Operator());
  o->form = form;
  o->minL = minL;
  o->maxL = maxL;
  for (int L = minL; L <= maxL; ++L) {
    const std::vector<double> K = p2CellElements(disc.topo(), L);
    std::vector<float> Kf(K.begin(), K.end());
    o->kd.emplace_back(new DevBuf());
    o->kd.back()->alloc(K.size() * sizeof(double));
    cudaCheck(cudaMemcpyAsync(o->kd.back()->p, K.data(), K.size() * sizeof(double), cudaMemcpyHostToDevice, stream),
              "P2 upload");
    o->kf.emplace_back(new DevBuf());
    o->kf.back()->alloc(Kf.size() * sizeof(float));
    cudaCheck(cudaMemcpyAsync(o->kf.back()->p, Kf.data(), Kf.size() * sizeof(float), cudaMemcpyHostToDevice, stream),
              "P2 upload");
    const std::vector<double> S = p2Stencils(K, (int)disc.topo().cells.size());
    std::vector<float> Sf(S.begin(), S.end());
    o->sd.emplace_back(new DevBuf());
    o->sd.back()->alloc(S.size() * sizeof(double));
    cudaCheck(cudaMemcpyAsync(o->sd.back()->p, S.data(), S.size() * sizeof(double), cudaMemcpyHostToDevice, stream),
              "P2 upload");
    o->sf.emplace_back(new DevBuf());
    o->sf.back()->alloc(Sf.size() * sizeof(float));
    cudaCheck(cudaMemcpyAsync(o->sf.back()->p, Sf.data(), Sf.size() * sizeof(float), cudaMemcpyHostToDevice, stream),
              "P2 upload");
    const std::vector<double> F = p2FaceStencils(K, (int)disc.topo().cells.size());
    std::vector<float> Ff(F.begin(), F.end());
    o->fd.emplace_back(new DevBuf());
    o->fd.back()->alloc(F.size() * sizeof(double));
    cudaCheck(cudaMemcpyAsync(o->fd.back()->p, F.data(), F.size() * sizeof(double), cudaMemcpyHostToDevice, stream),
              "P2 upload");
    o->ff.emplace_back(new DevBuf());
    o->ff.back()->alloc(Ff.size() * sizeof(float));
    cudaCheck(cudaMemcpyAsync(o->ff.back()->p, Ff.data(), Ff.size() * sizeof(float), cudaMemcpyHostToDevice, stream),
              "P2 upload");
    cudaCheck(cudaStreamSynchronize(stream), "P2 upload");
  }
  const int id = nextId++;
  p2ops[id] = std::move(o);
  return id;
}

static dev::P2Tables p2Tables() {
  dev::P2Tables tb{};
  for (int t = 0; t < 6; ++t) {
    tb.widthRed[t] = (unsigned char)kMicroCellWidth[t];
    for (int j = 0; j < 10; ++j)
      for (int d = 0; d < 3; ++d)
        tb.off[t][j][d] = (signed char)(j < 4 ? 2 * kMicroCellTable[t][j][d]
                                              : kMicroCellTable[t][kP2Edge[j - 4][0]][d] +
                                                    kMicroCellTable[t][kP2Edge[j - 4][1]][d]);
  }
  for (int t = 0; t < 6; ++t)
    for (int j = 0; j < 10; ++j) {
      const int pc = (tb.off[t][j][0] & 1) | ((tb.off[t][j][1] & 1) << 1) | ((tb.off[t][j][2] & 1) << 2);
      argCheck(tb.nCand[pc] < 24, "P2 candidate table overflow");
      tb.cand[pc][tb.nCand[pc]][0] = (unsigned char)t;
      tb.cand[pc][tb.nCand[pc]][1] = (unsigned char)j;
      ++tb.nCand[pc];
    }
  return tb;
}

// The work list of p2ApplyKernel for one lattice level of size M, the same for every macro-cell.
static std::vector<dev::P2Item> p2Items(int M) {
  std::vector<dev::P2Item> items;
  for (int e = 0; e < 6 * (M - 1) + 4; e += dev::kBlock) items.push_back({dev::P2_EDGES, e, 0, 0});
  for (int z = 0; z + 3 <= M - 1; z += dev::kP2Tile)
    for (int y = 0; y + z + 3 <= M - 1; y += dev::kP2Tile)
      for (int x = 0; x + y + z + 3 <= M - 1; x += dev::kP2Tile) items.push_back({dev::P2_TILE, x, y, z});
  for (int f = 0; f < 4; ++f)
    for (int t = 0; t + 2 <= M - 1; t += dev::kP2FaceTile)
      for (int s = 0; s + t + 2 <= M - 1; s += dev::kP2FaceTile) items.push_back({dev::P2_FACE, f, s, t});
  return items;
}

// Entry of a closure node of a macro-cell of lattice M in the closure stencils (p2_stencil.h).
static int p2ClosureEntry(int64_t X, int64_t Y, int64_t Z, int64_t M) {
  const bool on[4] = {Z == 0, Y == 0, X == 0, X + Y + Z == M};
  const int n = on[0] + on[1] + on[2] + on[3];
  if (n == 3) return 28 + (X == M ? 1 : Y == M ? 2 : Z == M ? 3 : 0);
  if (n == 2) {  // edges: X axis, Y axis, Z axis, then opposite the origin in the faces Z, Y, X = 0
    const int e = on[0] && on[1] ? 0 : on[0] && on[2] ? 1 : on[1] && on[2] ? 2 : on[0] ? 3 : on[1] ? 4 : 5;
    const int64_t t = e == 0 ? X : e == 1 || e == 3 ? Y : Z;
    return 16 + 2 * e + int(t & 1);
  }
  const int pc = int((X & 1) | ((Y & 1) << 1) | ((Z & 1) << 2));
  for (int k = on[0] ? 0 : on[1] ? 4 : on[2] ? 8 : 12;; ++k)
    if (p2s::kFaceClass[k] == pc) return k;
}

P2Additive& Storage::p2Additive(int Lf) {
  if ((int)p2add.size() <= Lf) p2add.resize(maxLevel() + 1);
  P2Additive& ad = p2add[Lf];
  if (ad.built) return ad;
  const LevelData& ld = levels[Lf];
  const LevelLayout& lay = *ld.lay;
  const Topology& topo = disc.topo();
  const int64_t M = ld.lv.N;
  auto put = [&](DevBuf& buf, const void* h, size_t bytes) {
    buf.alloc(std::max<size_t>(bytes, 16));
    if (bytes) cudaCheck(cudaMemcpyAsync(buf.p, h, bytes, cudaMemcpyHostToDevice, stream), "p2 tables");
  };
  // SOR colour of a DoF from its barycentric weights in ascending vertex-ID order (b0, b1, b2, b3),
  // parity class p = (b1 & 1) | (b2 & 1) << 1 | (b3 & 1) << 2: p = 0 (micro-vertices of the coarse
  // level) is split into ((b1 >> 1) + 2 (b2 >> 1) + 3 (b3 >> 1)) mod 4, the others are colours 3 + p
  auto colourOf = [](const Bary& b) {
    int64_t w[4] = {0, 0, 0, 0};
    for (int i = 0; i < b.n; ++i) w[i] = b.b[i];
    const int par = int(w[1] & 1) | (int(w[2] & 1) << 1) | (int(w[3] & 1) << 2);
    return par ? 3 + par : int(((w[1] >> 1) + 2 * (w[2] >> 1) + 3 * (w[3] >> 1)) % 4);
  };
  // The closure nodes of every cell in the order of the cell-closure halo group (cell, Z, Y, X),
  // which gives each its owner.
  const auto& cd = lay.commDst[G_CELL];
  const auto& cs = lay.commSrc[G_CELL];
  std::vector<dev::P2ClosureNode> nodes;
  std::vector<unsigned char> nodeColour;
  nodes.reserve(cd.size());
  nodeColour.reserve(cd.size());
  for (int c = 0; c < ld.lv.nCells; ++c)
    for (int64_t Z = 0; Z <= M; ++Z)
      for (int64_t Y = 0; Y + Z <= M; ++Y)
        for (int64_t X = 0; X + Y + Z <= M; ++X) {
          if (X != 0 && Y != 0 && Z != 0 && X + Y + Z != M) {
            X = M - Y - Z - 1;  // on to the last node of the row
            continue;
          }
          const size_t i = nodes.size();
          argCheck(i < cd.size() && cd[i] == lay.off[KC][c] + cellIdx(lay.w, X, Y, Z), "closure order");
          const int64_t wts[4] = {M - X - Y - Z, X, Y, Z};
          nodeColour.push_back((unsigned char)colourOf(makeBary(topo.cells[c].v, wts, 4)));
          nodes.push_back({c, (unsigned short)X, (unsigned short)Y, (unsigned short)Z,
                           (signed char)p2ClosureEntry(X, Y, Z, M), 0});
        }
  argCheck(nodes.size() == cd.size(), "closure order");
  // owner <- its copies, owners ascending, copies in table order (a counting sort on the owners,
  // which lie behind the cell arrays)
  const int64_t first = ld.nonCellBegin, nSlots = lay.total - first;
  std::vector<int> copyCount((size_t)nSlots, 0);
  std::vector<unsigned char> slotType((size_t)nSlots, 0), slotColour((size_t)nSlots, 0);
  auto setType = [&](int kind, size_t pr, unsigned char t) {
    std::fill_n(slotType.begin() + (lay.off[kind][pr] - first), lay.size[kind][pr], t);
  };
  for (size_t f = 0; f < topo.faces.size(); ++f) setType(KF, f, ld.hostFaceType[f]);
  for (size_t e = 0; e < topo.edges.size(); ++e) setType(KE, e, ld.hostLowType[e]);
  for (size_t v = 0; v < topo.verts.size(); ++v) setType(KV, v, ld.hostLowType[ld.lv.nEdges + v]);
  for (size_t i = 0; i < cs.size(); ++i) {
    argCheck(cs[i] >= first, "owner slot outside the face, edge and vertex arrays");
    ++copyCount[(size_t)(cs[i] - first)];
    slotColour[(size_t)(cs[i] - first)] = nodeColour[i];
  }
  std::vector<int64_t> own;
  std::vector<int> ptr{0}, next((size_t)nSlots, 0);
  std::vector<unsigned char> ty;
  for (int64_t q = 0; q < nSlots; ++q)
    if (copyCount[(size_t)q]) {
      next[(size_t)q] = ptr.back();
      own.push_back(first + q);
      ty.push_back(slotType[(size_t)q]);
      ptr.push_back(ptr.back() + copyCount[(size_t)q]);
    }
  std::vector<int64_t> cp(cd.size());
  for (size_t i = 0; i < cd.size(); ++i) cp[(size_t)next[(size_t)(cs[i] - first)]++] = cd[i];
  ad.n = (int)own.size();
  put(ad.owner, own.data(), own.size() * sizeof(int64_t));
  put(ad.ptr, ptr.data(), ptr.size() * sizeof(int));
  put(ad.copies, cp.data(), cp.size() * sizeof(int64_t));
  put(ad.type, ty.data(), ty.size());
  // the owner slot and DoF type of every DoF, in slot order per kind (coarse levels only)
  if (lay.total <= (int64_t(1) << 20)) {
    auto add = [&](int64_t slot, unsigned char t) {
      ad.hostOwner.push_back(slot);
      ad.hostOwnerType.push_back(t);
    };
    for (size_t v = 0; v < topo.verts.size(); ++v) add(lay.off[KV][v], ld.hostLowType[ld.lv.nEdges + v]);
    for (size_t e = 0; e < topo.edges.size(); ++e)
      for (int64_t x = 1; x < M; ++x) add(lay.off[KE][e] + x, ld.hostLowType[e]);
    for (size_t f = 0; f < topo.faces.size(); ++f)
      for (int64_t y = 1; y < M; ++y)
        for (int64_t x = 1; x + y < M; ++x) add(lay.off[KF][f] + faceIdx(lay.w, x, y), ld.hostFaceType[f]);
    for (size_t c = 0; c < topo.cells.size(); ++c)
      for (int64_t z = 1; z < M; ++z)
        for (int64_t y = 1; y + z < M; ++y)
          for (int64_t x = 1; x + y + z < M; ++x) add(lay.off[KC][c] + cellIdx(lay.w, x, y, z), ld.hostCellType[c]);
  }
  // SOR: closure nodes by colour, then by entry, so that the warps mostly run one stencil
  {
    std::vector<size_t> bucket(11 * 32 + 1, 0);
    auto key = [&](size_t i) { return (size_t)nodeColour[i] * 32 + (size_t)nodes[i].k; };
    for (size_t i = 0; i < nodes.size(); ++i) ++bucket[key(i) + 1];
    for (size_t k = 0; k + 1 < bucket.size(); ++k) bucket[k + 1] += bucket[k];
    for (int k = 0; k <= 11; ++k) ad.closureBegin[k] = (int)bucket[(size_t)k * 32];
    std::vector<dev::P2ClosureNode> list(nodes.size());
    for (size_t i = 0; i < nodes.size(); ++i) list[bucket[key(i)]++] = nodes[i];
    put(ad.closureList, list.data(), list.size() * sizeof(dev::P2ClosureNode));
    // owners by colour
    std::vector<dev::P2Owner> owners;
    owners.reserve(own.size());
    for (int k = 0; k < 11; ++k) {
      ad.sorOwnerBegin[k] = (int)owners.size();
      for (size_t i = 0; i < own.size(); ++i)
        if (slotColour[(size_t)(own[i] - first)] == k)
          owners.push_back({(unsigned)own[i], ptr[i], (unsigned short)(ptr[i + 1] - ptr[i]), ty[i]});
    }
    ad.sorOwnerBegin[11] = (int)owners.size();
    argCheck(owners.size() == own.size(), "owner without an SOR colour");
    const std::vector<unsigned> cp32(cp.begin(), cp.end());
    put(ad.sorOwners, owners.data(), owners.size() * sizeof(dev::P2Owner));
    put(ad.sorCopies, cp32.data(), cp32.size() * sizeof(unsigned));
    // interior nodes by class (ten bits a coordinate: the levels of a storage end at lattice 1024)
    std::vector<unsigned> inner(dev::kP2NodeHead);
    for (int pc = 0; pc < 8; ++pc) {
      inner[(size_t)pc] = (unsigned)inner.size();
      for (int64_t Z = pc & 4 ? 1 : 2; Z <= M - 1; Z += 2)
        for (int64_t Y = pc & 2 ? 1 : 2; Y + Z <= M - 1; Y += 2)
          for (int64_t X = pc & 1 ? 1 : 2; X + Y + Z <= M - 1; X += pc ? 2 : 8)
            inner.push_back((unsigned)(X | Y << 10 | Z << 20));
    }
    inner[8] = (unsigned)inner.size();
    put(ad.sorInner, inner.data(), inner.size() * sizeof(unsigned));
    ad.sorVertexNodes = (int)(inner[1] - inner[0]);
    ad.sorEdgeNodes = 0;
    for (int pc = 1; pc < 8; ++pc) ad.sorEdgeNodes = std::max(ad.sorEdgeNodes, (int)(inner[pc + 1] - inner[pc]));
    // colours in the cells' frames: rank of a cell's vertex i among its vertex IDs
    std::vector<dev::P2CellColour> cc((size_t)ld.lv.nCells);
    for (int c = 0; c < ld.lv.nCells; ++c) {
      const int* v = topo.cells[c].v;
      int rank[4];
      for (int i = 0; i < 4; ++i) {
        rank[i] = 0;
        for (int j = 0; j < 4; ++j) rank[i] += v[j] < v[i];
      }
      dev::P2CellColour& q = cc[(size_t)c];
      for (int k = 0; k < 11; ++k) q.cls[k] = k < 4 ? 0 : -1;
      q.c0 = (unsigned char)((rank[0] * (M / 2)) & 3);
      q.cx = (unsigned char)((rank[1] - rank[0]) & 3);
      q.cy = (unsigned char)((rank[2] - rank[0]) & 3);
      q.cz = (unsigned char)((rank[3] - rank[0]) & 3);
      for (int pc = 1; pc < 8; ++pc) {
        const int odd[4] = {(pc ^ (pc >> 1) ^ (pc >> 2)) & 1, pc & 1, (pc >> 1) & 1, (pc >> 2) & 1};
        int par = 0;
        for (int i = 0; i < 4; ++i)
          if (odd[i] && rank[i] > 0) par |= 1 << (rank[i] - 1);
        argCheck(par != 0 && q.cls[3 + par] < 0, "P2 colour classes are inconsistent");
        q.cls[3 + par] = (signed char)pc;
      }
    }
    put(ad.sorCells, cc.data(), cc.size() * sizeof(dev::P2CellColour));
    cudaCheck(cudaStreamSynchronize(stream), "p2 tables");  // the host lists go out of scope
  }
  std::vector<unsigned char> mult((size_t)lay.total, 1);
  for (size_t i = 0; i + 1 < ptr.size(); ++i)
    for (int k = ptr[i]; k < ptr[i + 1]; ++k) mult[(size_t)cp[k]] = (unsigned char)(ptr[i + 1] - ptr[i]);
  put(ad.mult, mult.data(), mult.size());
  const std::vector<dev::P2Item> items = p2Items((int)M);
  ad.nItems = (int)items.size();
  put(ad.items, items.data(), items.size() * sizeof(dev::P2Item));
  cudaCheck(cudaStreamSynchronize(stream), "p2 tables");
  ad.built = true;
  return ad;
}

static const dev::P2Tables& p2TablesOnce() {
  static const dev::P2Tables tb = p2Tables();
  return tb;
}

// Index of offset (dx, dy, dz) in one of the lists of p2_stencil.h.
static short offsetIndex(const signed char (*list)[3], int len, int dx, int dy, int dz) {
  for (int e = 0; e < len; ++e)
    if (list[e][0] == dx && list[e][1] == dy && list[e][2] == dz) return (short)e;
  throw Error(HG_ERR_INTERNAL, "P2 stencil offset table does not match the micro-cells");
}
// That of local node m of micro-cell type t seen from its local node j.
static short nodeIndex(const signed char (*list)[3], int len, int t, int j, int m) {
  const dev::P2Tables& tb = p2TablesOnce();
  return offsetIndex(list, len, tb.off[t][m][0] - tb.off[t][j][0], tb.off[t][m][1] - tb.off[t][j][1],
                     tb.off[t][m][2] - tb.off[t][j][2]);
}

// One product of a stencil: weight `to` of a cell takes element entry `from` of that cell. The lists
// depend on neither the cell nor the level; finding the offsets anew for each took most of an
// operator's set-up.
struct StencilTerm {
  short to, from;
};
static std::vector<double> stencilWeights(const std::vector<StencilTerm>& terms, int weights, const std::vector<double>& K,
                                          int entries, int nCells) {
  std::vector<double> S((size_t)nCells * (size_t)weights, 0.0);
  for (int c = 0; c < nCells; ++c) {
    double* s = S.data() + (size_t)c * (size_t)weights;
    const double* k = K.data() + (size_t)c * (size_t)entries;
    for (const StencilTerm& q : terms) s[q.to] += k[q.from];
  }
  return S;
}

// Interior stencil weights of every cell: for each parity class, the sum over the class's
// candidate micro-cells (type t, local node j) of row j of their element matrices, scattered
// to the lattice offsets of the ten nodes in the order of p2s::kOff.
static std::vector<double> p2Stencils(const std::vector<double>& K, int nCells) {
  static const std::vector<StencilTerm> terms = [] {
    const dev::P2Tables& tb = p2TablesOnce();
    std::vector<StencilTerm> v;
    for (int pc = 0; pc < 8; ++pc)
      for (int k = 0; k < tb.nCand[pc]; ++k) {
        const int t = tb.cand[pc][k][0], j = tb.cand[pc][k][1];
        for (int m = 0; m < 10; ++m)
          v.push_back({(short)(p2s::kFirst[pc] + nodeIndex(p2s::kOff[pc], p2s::kLen[pc], t, j, m)),
                       (short)(t * 100 + j * 10 + m)});
      }
    return v;
  }();
  return stencilWeights(terms, p2s::kTotal, K, 600, nCells);
}

// Closure stencil weights of every cell: per entry k (face and class, edge and parity, vertex), the sum
// over its micro-cells p2s::kFaceCand[k] of their element rows, scattered to the offsets p2s::kFaceOff[k].
static std::vector<double> p2FaceStencils(const std::vector<double>& K, int nCells) {
  static const std::vector<StencilTerm> terms = [] {
    std::vector<StencilTerm> v;
    for (int k = 0; k < p2s::kFaceStencils; ++k)
      for (int q = 0; q < p2s::kFaceNCand[k]; ++q) {
        const int t = p2s::kFaceCand[k][q][0], j = p2s::kFaceCand[k][q][1];
        for (int m = 0; m < 10; ++m)
          v.push_back({(short)(p2s::kFaceFirst[k] + nodeIndex(p2s::kFaceOff[k], p2s::kFaceLen[k], t, j, m)),
                       (short)(t * 100 + j * 10 + m)});
      }
    return v;
  }();
  return stencilWeights(terms, p2s::kFaceTotal, K, 600, nCells);
}

// Sums of the cells' shares into the owners: dst = sum, or rhs - sum for a residual.
template <class T, int MODE>
void Storage::p2AddOwners(const P2Additive& ad, T* dst, const T* rhs, unsigned mask) {
  if (!ad.n) return;
  launchNext(stream, dev::p2AddKernel<T, MODE>, (ad.n + dev::kBlock - 1) / dev::kBlock, dev::kBlock, 0,
             (const int64_t*)ad.owner.p, (const int*)ad.ptr.p, (const int64_t*)ad.copies.p,
             (const unsigned char*)ad.type.p, ad.n, dst, rhs, mask);
  ++launches;
}

// The cells' part of dst = A src or rhs - A src on one P2 level: final values at the interior nodes
// of the flagged cells, shares of A src in the closure slots.
template <class T, int MODE>
void Storage::p2Sweep(P2Operator& o, int L, T* dst, const T* src, const T* rhs, unsigned mask) {
  const int Lf = L + 1;
  const LevelData& ld = levels[Lf];
  P2Additive& ad = p2Additive(Lf);
  const T* W = (const T*)(sizeof(T) == 8 ? o.sd[L - o.minL]->p : o.sf[L - o.minL]->p);
  const T* FW = (const T*)(sizeof(T) == 8 ? o.fd[L - o.minL]->p : o.ff[L - o.minL]->p);
  launchNext(stream, dev::p2ApplyKernel<T, MODE>, ld.lv.nCells * ad.nItems, dev::kBlock, dev::p2TileSmem<T>(), ld.lv,
             (const dev::P2Item*)ad.items.p, W, FW, dst, src, rhs, mask);
  ++launches;
  cudaCheck(cudaGetLastError(), "P2 kernels");
}

// dst = A src or rhs - A src on the flagged DoFs. The copies of dst are not refreshed here.
template <class T, int MODE>
void Storage::p2Launch(P2Operator& o, int L, T* dst, const T* src, const T* rhs, unsigned mask) {
  p2Sweep<T, MODE>(o, L, dst, src, rhs, mask);
  p2AddOwners<T, MODE>(p2Additive(L + 1), dst, rhs, mask);
  cudaCheck(cudaGetLastError(), "P2 kernels");
}

P2Operator& Storage::p2op(int id) {
  auto it = p2ops.find(id);
  argCheck(it != p2ops.end(), "unknown P2 operator handle");
  return *it->second;
}

void Storage::p2Apply(int opId, int src, int dst, int rhs, int L, unsigned mask, int mode) {
  P2Operator& o = p2op(opId);
  argCheck(L >= o.minL && L <= o.maxL, "level outside the P2 operator's level range");
  argCheck(src != dst && (mode == 0 || (rhs != dst && rhs != src)), "P2 apply: distinct functions required");
  const int Lf = L + 1;
  Function& fs = fn(src);
  argCheck(fs.prec == fn(dst).prec && (mode == 0 || fn(rhs).prec == fs.prec), "P2 apply: precision mismatch");
  communicate(src, Lf, 1 << G_CELL);  // the closure copies of every cell hold the owners' values
  if (fs.prec == 8) {
    const double* r = mode ? (const double*)data(rhs, Lf) : nullptr;
    if (mode == 0)
      p2Launch<double, dev::MODE_REPLACE>(o, L, (double*)data(dst, Lf), (const double*)data(src, Lf), r, mask);
    else
      p2Launch<double, dev::MODE_RESIDUAL>(o, L, (double*)data(dst, Lf), (const double*)data(src, Lf), r, mask);
  } else {
    const float* r = mode ? (const float*)data(rhs, Lf) : nullptr;
    if (mode == 0)
      p2Launch<float, dev::MODE_REPLACE>(o, L, (float*)data(dst, Lf), (const float*)data(src, Lf), r, mask);
    else
      p2Launch<float, dev::MODE_RESIDUAL>(o, L, (float*)data(dst, Lf), (const float*)data(src, Lf), r, mask);
  }
  communicate(dst, Lf, kAllGroups);
}

// Diagonal of a P2 operator level as a function of that level (built once per precision).
int Storage::p2Diagonal(int opId, int L, int prec) {
  P2Operator& o = p2op(opId);
  auto key = std::make_pair(L, prec);
  auto it = o.diag.find(key);
  if (it != o.diag.end()) return it->second;
  const int Lf = L + 1;
  const int d = createFunction(Lf, Lf, prec);
  const LevelData& ld = levels[Lf];
  const P2Additive& ad = p2Additive(Lf);
  auto run = [&](auto zero) {
    using T = decltype(zero);
    const T* K = (const T*)(sizeof(T) == 8 ? o.kd[L - o.minL]->p : o.kf[L - o.minL]->p);
    dev::p2DiagonalKernel<T><<<ld.lv.nCells * (ld.lv.N + 1), dev::kBlock, 0, stream>>>(ld.lv, p2TablesOnce(), K,
                                                                                     (T*)data(d, Lf));
    ++launches;
    p2AddOwners<T, dev::MODE_REPLACE>(ad, (T*)data(d, Lf), nullptr, HG_ALL);
  };
  if (prec == 8) run(0.0);
  else run(0.0f);
  cudaCheck(cudaGetLastError(), "P2 diagonal");
  communicate(d, Lf, kAllGroups);
  o.diag[key] = d;
  return d;
}

template <class T>
void Storage::p2SorT(P2Operator& o, int opId, int x, int b, int L, unsigned mask, T omega, bool backwards) {
  const int Lf = L + 1;
  const int prec = (int)sizeof(T);
  const int dg = p2Diagonal(opId, L, prec);
  const int ax = p2Scratch(Lf, prec);
  const LevelData& ld = levels[Lf];
  P2Additive& ad = p2Additive(Lf);
  const T* W = (const T*)(sizeof(T) == 8 ? o.sd[L - o.minL]->p : o.sf[L - o.minL]->p);
  const T* FW = (const T*)(sizeof(T) == 8 ? o.fd[L - o.minL]->p : o.ff[L - o.minL]->p);
  const dev::P2CellColour* cells = (const dev::P2CellColour*)ad.sorCells.p;
  T* xd = (T*)data(x, Lf);
  const T* bd = (const T*)data(b, Lf);
  T* axd = (T*)data(ax, Lf);
  auto blocks = [](int n) { return (n + dev::kBlock - 1) / dev::kBlock; };
  communicate(x, Lf, 1 << G_CELL);
  for (int k = 0; k < 11; ++k) {
    const int c = backwards ? 10 - k : k;
    const int chunks = blocks(c < 4 ? ad.sorVertexNodes : ad.sorEdgeNodes);
    const int nList = ad.closureBegin[c + 1] - ad.closureBegin[c], listBlocks = blocks(nList);
    const int nOwn = ad.sorOwnerBegin[c + 1] - ad.sorOwnerBegin[c], ownBlocks = blocks(nOwn);
    const int inner = ld.lv.nCells * chunks;
    if (listBlocks + inner > 0) {
      launchNext(stream, dev::p2SorGatherKernel<T>, listBlocks + inner, dev::kBlock, 0, ld.lv, W, FW,
                 (const dev::P2ClosureNode*)ad.closureList.p + ad.closureBegin[c], nList, listBlocks,
                 (const unsigned*)ad.sorInner.p, cells, c, std::max(chunks, 1), xd, bd, axd, mask, omega);
      ++launches;
    }
    if (ownBlocks + inner > 0) {
      launchNext(stream, dev::p2SorUpdateKernel<T>, ownBlocks + inner, dev::kBlock, 0, ld.lv,
                 (const dev::P2Owner*)ad.sorOwners.p + ad.sorOwnerBegin[c], nOwn, ownBlocks,
                 (const unsigned*)ad.sorCopies.p, (const unsigned*)ad.sorInner.p, cells, c, std::max(chunks, 1), xd,
                 bd, axd, (const T*)data(dg, Lf), mask, omega);
      ++launches;
    }
  }
  cudaCheck(cudaGetLastError(), "P2 SOR");
  communicate(x, Lf, kAllGroups);
}

void Storage::p2Sor(int opId, int x, int b, double omega, int L, unsigned mask, bool backwards) {
  P2Operator& o = p2op(opId);
  argCheck(L >= o.minL && L <= o.maxL, "level outside the P2 operator's level range");
  argCheck(x != b, "P2 SOR: x and b must differ");
  Function& fx = fn(x);
  argCheck(fx.prec == fn(b).prec, "P2 SOR: precision mismatch");
  if (fx.prec == 8)
    p2SorT<double>(o, opId, x, b, L, mask, omega, backwards);
  else
    p2SorT<float>(o, opId, x, b, L, mask, (float)omega, backwards);
}

// Fine node Q of a macro-cell at Q / 4 level-L units: class r = (Q_x & 3) | (Q_y & 3) << 2 |
// (Q_z & 3) << 4. For every micro-cell (type t, anchor (Q >> 2) - delta) containing the point,
// its barycentric coordinates in quarters (exact: the micro-cells are unimodular) give the coarse
// P2 basis values lambda (2 lambda - 1) at the vertices and 4 lambda_i lambda_j at the edges.
static void buildP2Transfer(P2Transfer& tr, cudaStream_t stream) {
  std::vector<unsigned char> nc(64, 0), cand(64 * dev::kP2TrCand, 0);
  std::vector<double> w(64 * dev::kP2TrCand * 10, 0.0);
  for (int r = 0; r < 64; ++r) {
    const int f4[3] = {r & 3, (r >> 2) & 3, (r >> 4) & 3};
    for (int d = 0; d < 8; ++d)
      for (int t = 0; t < 6; ++t) {
        const int* v0 = kMicroCellTable[t][0];
        int B[3][3];  // columns v_m - v0
        for (int m = 1; m < 4; ++m)
          for (int k = 0; k < 3; ++k) B[k][m - 1] = kMicroCellTable[t][m][k] - v0[k];
        const int det = B[0][0] * (B[1][1] * B[2][2] - B[1][2] * B[2][1]) - B[0][1] * (B[1][0] * B[2][2] - B[1][2] * B[2][0]) +
                        B[0][2] * (B[1][0] * B[2][1] - B[1][1] * B[2][0]);
        const int inv[3][3] = {{(B[1][1] * B[2][2] - B[1][2] * B[2][1]) * det, (B[0][2] * B[2][1] - B[0][1] * B[2][2]) * det,
                                (B[0][1] * B[1][2] - B[0][2] * B[1][1]) * det},
                               {(B[1][2] * B[2][0] - B[1][0] * B[2][2]) * det, (B[0][0] * B[2][2] - B[0][2] * B[2][0]) * det,
                                (B[0][2] * B[1][0] - B[0][0] * B[1][2]) * det},
                               {(B[1][0] * B[2][1] - B[1][1] * B[2][0]) * det, (B[0][1] * B[2][0] - B[0][0] * B[2][1]) * det,
                                (B[0][0] * B[1][1] - B[0][1] * B[1][0]) * det}};  // det = +-1, so inv = adj * det
        int q[3];
        for (int k = 0; k < 3; ++k) q[k] = f4[k] + 4 * ((d >> k) & 1) - 4 * v0[k];  // 4 (point - v0)
        int l4[4];
        l4[1] = inv[0][0] * q[0] + inv[0][1] * q[1] + inv[0][2] * q[2];
        l4[2] = inv[1][0] * q[0] + inv[1][1] * q[1] + inv[1][2] * q[2];
        l4[3] = inv[2][0] * q[0] + inv[2][1] * q[1] + inv[2][2] * q[2];
        l4[0] = 4 - l4[1] - l4[2] - l4[3];
        if (l4[0] < 0 || l4[1] < 0 || l4[2] < 0 || l4[3] < 0) continue;
        argCheck(det == 1 || det == -1, "micro-cell is not unimodular");
        if (nc[r] >= dev::kP2TrCand) continue;
        const int k = nc[r]++;
        cand[r * dev::kP2TrCand + k] = (unsigned char)((d << 3) | t);
        double* wr = &w[(size_t)(r * dev::kP2TrCand + k) * 10];
        for (int m = 0; m < 4; ++m) {
          const double l = l4[m] / 4.0;
          wr[m] = l * (2.0 * l - 1.0);
        }
        for (int e = 0; e < 6; ++e) wr[4 + e] = 4.0 * (l4[kP2Edge[e][0]] / 4.0) * (l4[kP2Edge[e][1]] / 4.0);
      }
  }
  std::vector<float> wfl(w.begin(), w.end());
  tr.hNCand = nc;
  tr.hCand = cand;
  tr.hW = w;
  tr.nCand.alloc(nc.size());
  tr.cand.alloc(cand.size());
  tr.wd.alloc(w.size() * sizeof(double));
  tr.wf.alloc(wfl.size() * sizeof(float));
  cudaCheck(cudaMemcpyAsync(tr.nCand.p, nc.data(), nc.size(), cudaMemcpyHostToDevice, stream), "p2 transfer");
  cudaCheck(cudaMemcpyAsync(tr.cand.p, cand.data(), cand.size(), cudaMemcpyHostToDevice, stream), "p2 transfer");
  cudaCheck(cudaMemcpyAsync(tr.wd.p, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice, stream), "p2 transfer");
  cudaCheck(cudaMemcpyAsync(tr.wf.p, wfl.data(), wfl.size() * sizeof(float), cudaMemcpyHostToDevice, stream), "p2 transfer");
  cudaCheck(cudaStreamSynchronize(stream), "p2 transfer");
  tr.built = true;
}

// The restriction's gather lists for fine lattice level Lff: every fine node Q of the closed
// reference cell contributes to the coarse nodes its prolongation reads (the same candidate
// micro-cell as p2PickCandidate picks, nonzero basis values only; even nodes are injected), and
// each coarse node lists its contributions in the order of Q (z, y, x), then of the basis node.
const P2Gather& Storage::p2Gather(int Lff) {
  P2Gather& g = p2gather[Lff];
  if (g.built) return g;
  if (!p2tr.built) buildP2Transfer(p2tr, stream);
  const dev::P2Tables& tb = p2TablesOnce();
  const int Mf = disc.level(Lff).N, Mc = Mf / 2, N = Mc / 2, wf = Mf + 1, wc = Mc + 1;
  auto tet = [](int64_t w) { return w * (w + 1) * (w + 2) / 6; };
  auto row = [](int64_t W, int64_t y) { return y * (W + 1) - y * (y + 1) / 2; };
  auto cidx = [&](int x, int y, int z) { return int(tet(wc) - tet(wc - z) + row(wc - z, y) + x); };
  auto fidx = [&](int x, int y, int z) { return int(tet(wf) - tet(wf - z) + row(wf - z, y) + x); };
  const int nC = (int)tet(wc);
  std::vector<std::vector<std::pair<int, double>>> lists((size_t)nC);
  for (int Z = 0; Z <= Mf; ++Z)
    for (int Y = 0; Y <= Mf - Z; ++Y)
      for (int X = 0; X <= Mf - Z - Y; ++X) {
        const int q = fidx(X, Y, Z);
        if (((X | Y | Z) & 1) == 0) {
          lists[(size_t)cidx(X >> 1, Y >> 1, Z >> 1)].push_back({q, 1.0});
          continue;
        }
        const int r = (X & 3) | ((Y & 3) << 2) | ((Z & 3) << 4);
        for (int k = 0; k < p2tr.hNCand[r]; ++k) {  // the first candidate inside the cell
          const int c = p2tr.hCand[(size_t)r * dev::kP2TrCand + k], t = c & 7, d = c >> 3;
          const int ax = (X >> 2) - (d & 1), ay = (Y >> 2) - ((d >> 1) & 1), az = (Z >> 2) - ((d >> 2) & 1);
          if (!(ax >= 0 && ay >= 0 && az >= 0 && ax + ay + az < N - tb.widthRed[t])) continue;
          const double* w = &p2tr.hW[(size_t)(r * dev::kP2TrCand + k) * 10];
          for (int m = 0; m < 10; ++m)
            if (w[m] != 0.0)
              lists[(size_t)cidx(2 * ax + tb.off[t][m][0], 2 * ay + tb.off[t][m][1], 2 * az + tb.off[t][m][2])]
                  .push_back({q, w[m]});
          break;
        }
      }
  std::vector<int> ptr((size_t)nC + 1, 0), idx;
  std::vector<double> wd;
  for (int c = 0; c < nC; ++c) {
    for (const auto& e : lists[(size_t)c]) {
      idx.push_back(e.first);
      wd.push_back(e.second);
    }
    ptr[(size_t)c + 1] = (int)idx.size();
  }
  std::vector<float> wfl(wd.begin(), wd.end());
  g.nCoarse = nC;
  g.ptr.alloc(ptr.size() * sizeof(int));
  cudaCheck(cudaMemcpyAsync(g.ptr.p, ptr.data(), ptr.size() * sizeof(int), cudaMemcpyHostToDevice, stream), "p2 gather");
  g.idx.alloc(idx.size() * sizeof(int));
  g.wd.alloc(wd.size() * sizeof(double));
  g.wf.alloc(wfl.size() * sizeof(float));
  cudaCheck(cudaMemcpyAsync(g.idx.p, idx.data(), idx.size() * sizeof(int), cudaMemcpyHostToDevice, stream), "p2 gather");
  cudaCheck(cudaMemcpyAsync(g.wd.p, wd.data(), wd.size() * sizeof(double), cudaMemcpyHostToDevice, stream), "p2 gather");
  cudaCheck(cudaMemcpyAsync(g.wf.p, wfl.data(), wfl.size() * sizeof(float), cudaMemcpyHostToDevice, stream), "p2 gather");
  cudaCheck(cudaStreamSynchronize(stream), "p2 gather");
  g.built = true;
  return g;
}

int Storage::p2Scratch(int Lf, int prec) {
  const auto key = p2ScratchKey(Lf, prec);
  if (!p2scratch.count(key)) p2scratch[key] = createFunction(Lf, Lf, prec);
  return p2scratch[key];
}

void Storage::p2Prolongate(int id, int Lc, unsigned mask, bool add) {
  Function& f = fn(id);
  const int Lcf = Lc + 1, Lff = Lc + 2;  // lattice levels
  argCheck(Lcf >= f.minL && Lff <= f.maxL, "P2 prolongation: levels outside the function's range");
  if (!p2tr.built) buildP2Transfer(p2tr, stream);
  const LevelData& lc = levels[Lcf];
  const LevelData& lf = levels[Lff];
  P2Additive& ad = p2Additive(Lff);
  communicate(id, Lcf, 1 << G_CELL);
  const int out = add ? p2Scratch(Lff, f.prec) : id;
  const dev::P2TransferDev tr{(const unsigned char*)p2tr.nCand.p, (const unsigned char*)p2tr.cand.p};
  const int nb = lf.lv.nCells * (lf.lv.N + 1), na = (ad.n + dev::kBlock - 1) / dev::kBlock;
  if (f.prec == 8) {
    launchNext(stream, dev::p2ProlongKernel<double>, nb, dev::kBlock, 0, lc.lv, lf.lv, p2TablesOnce(), tr,
               (const double*)p2tr.wd.p, (const double*)data(id, Lcf), (double*)data(out, Lff));
    if (ad.n)
      launchNext(stream, dev::p2PickKernel<double>, na, dev::kBlock, 0, (const int64_t*)ad.owner.p,
                 (const int*)ad.ptr.p, (const int64_t*)ad.copies.p, (const unsigned char*)ad.type.p, ad.n,
                 (double*)data(out, Lff), add ? HG_ALL : mask);
  } else {
    launchNext(stream, dev::p2ProlongKernel<float>, nb, dev::kBlock, 0, lc.lv, lf.lv, p2TablesOnce(), tr,
               (const float*)p2tr.wf.p, (const float*)data(id, Lcf), (float*)data(out, Lff));
    if (ad.n)
      launchNext(stream, dev::p2PickKernel<float>, na, dev::kBlock, 0, (const int64_t*)ad.owner.p,
                 (const int*)ad.ptr.p, (const int64_t*)ad.copies.p, (const unsigned char*)ad.type.p, ad.n,
                 (float*)data(out, Lff), add ? HG_ALL : mask);
  }
  launches += ad.n ? 2 : 1;
  cudaCheck(cudaGetLastError(), "P2 prolongation");
  if (add) {
    const double one = 1.0;
    lincomb(id, Lff, mask, 1, &one, &out, true, 0.0);
  }
  communicate(id, Lff, kAllGroups);
}

void Storage::p2Restrict(int id, int Lf, unsigned mask) {
  Function& f = fn(id);
  const int Lff = Lf + 1, Lcf = Lf;  // lattice levels: fine P2 level Lf, coarse Lf - 1
  argCheck(Lf >= 1 && Lcf >= f.minL && Lff <= f.maxL, "P2 restriction: levels outside the function's range");
  if (!p2tr.built) buildP2Transfer(p2tr, stream);
  const LevelData& lc = levels[Lcf];
  const LevelData& lf = levels[Lff];
  P2Additive& adf = p2Additive(Lff);
  P2Additive& adc = p2Additive(Lcf);
  const P2Gather& gt = p2Gather(Lff);
  communicate(id, Lff, 1 << G_CELL);
  cudaCheck(cudaMemsetAsync(data(id, Lcf), 0, (size_t)lc.lay->total * f.prec, stream), "P2 restriction");
  const int bpc = (gt.nCoarse + dev::kBlock - 1) / dev::kBlock;
  const int nb = lf.lv.nCells * bpc, na = (adc.n + dev::kBlock - 1) / dev::kBlock;
  if (f.prec == 8) {
    launchNext(stream, dev::p2RestrictGatherKernel<double>, nb, dev::kBlock, 0, lc.lv, lf.lv, (const int*)gt.ptr.p,
               (const int*)gt.idx.p, (const double*)gt.wd.p, gt.nCoarse, bpc, (const double*)data(id, Lff),
               (const unsigned char*)adf.mult.p, (double*)data(id, Lcf));
    if (adc.n)
      launchNext(stream, dev::p2AddKernel<double, dev::MODE_REPLACE>, na, dev::kBlock, 0, (const int64_t*)adc.owner.p,
                 (const int*)adc.ptr.p, (const int64_t*)adc.copies.p, (const unsigned char*)adc.type.p, adc.n,
                 (double*)data(id, Lcf), nullptr, mask);
  } else {
    launchNext(stream, dev::p2RestrictGatherKernel<float>, nb, dev::kBlock, 0, lc.lv, lf.lv, (const int*)gt.ptr.p,
               (const int*)gt.idx.p, (const float*)gt.wf.p, gt.nCoarse, bpc, (const float*)data(id, Lff),
               (const unsigned char*)adf.mult.p, (float*)data(id, Lcf));
    if (adc.n)
      launchNext(stream, dev::p2AddKernel<float, dev::MODE_REPLACE>, na, dev::kBlock, 0, (const int64_t*)adc.owner.p,
                 (const int*)adc.ptr.p, (const int64_t*)adc.copies.p, (const unsigned char*)adc.type.p, adc.n,
                 (float*)data(id, Lcf), nullptr, mask);
  }
  launches += adc.n ? 2 : 1;
  cudaCheck(cudaGetLastError(), "P2 restriction");
  communicate(id, Lcf, kAllGroups);
}

// Coupling stencils of every cell from the divergence elements D[cell][t][k][i][j]. Interior: div
// weights on p2s::kOff[0] (a pressure vertex i of micro-cell t sees node j at off_j - off_i), divT
// weights on p2s::kDivTOff (velocity node j of class pc sees vertex i at (off_i - off_j + pc) / 2).
// Closure: the same over the micro-cells of each closure entry, div on the vertex-class entries.
struct DivStencils {
  std::vector<double> div, divT, divClosure, divTClosure;
};

static DivStencils p2DivStencils(const std::vector<double>& D, int nCells) {
  struct Terms {
    std::vector<StencilTerm> div, divT, divClosure, divTClosure;
  };
  static const Terms terms = [] {
    const dev::P2Tables& tb = p2TablesOnce();
    Terms s;
    auto pressure = [&](const signed char (*list)[3], int len, int pc, int t, int i, int j) {
      return offsetIndex(list, len, (tb.off[t][i][0] - tb.off[t][j][0] + (pc & 1)) / 2,
                         (tb.off[t][i][1] - tb.off[t][j][1] + ((pc >> 1) & 1)) / 2,
                         (tb.off[t][i][2] - tb.off[t][j][2] + ((pc >> 2) & 1)) / 2);
    };
    auto add = [](std::vector<StencilTerm>& v, int stride, int to, int t, int i, int j) {  // the three components
      for (int k = 0; k < 3; ++k) v.push_back({(short)(k * stride + to), (short)(t * 120 + k * 40 + i * 10 + j)});
    };
    for (int t = 0; t < 6; ++t)
      for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 10; ++j) add(s.div, 65, nodeIndex(p2s::kOff[0], p2s::kLen[0], t, i, j), t, i, j);
    for (int pc = 0; pc < 8; ++pc)
      for (int q = 0; q < tb.nCand[pc]; ++q) {
        const int t = tb.cand[pc][q][0], j = tb.cand[pc][q][1];
        for (int i = 0; i < 4; ++i)
          add(s.divT, 65, p2s::kDivTFirst[pc] + pressure(p2s::kDivTOff[pc], p2s::kDivTLen[pc], pc, t, i, j), t, i, j);
      }
    for (int n = 0; n < p2s::kFaceStencils; ++n) {
      const int pc = p2s::kFaceClass[n];
      for (int q = 0; q < p2s::kFaceNCand[n]; ++q) {
        const int t = p2s::kFaceCand[n][q][0], j = p2s::kFaceCand[n][q][1];
        for (int i = 0; i < 4; ++i)
          add(s.divTClosure, p2s::kDivTFaceTotal,
              p2s::kDivTFaceFirst[n] + pressure(p2s::kDivTFaceOff[n], p2s::kDivTFaceLen[n], pc, t, i, j), t, i, j);
        if (pc != 0) continue;
        for (int m = 0; m < 10; ++m)  // local node j of a vertex-class entry is pressure vertex j
          add(s.divClosure, p2s::kFaceTotal, p2s::kFaceFirst[n] + nodeIndex(p2s::kFaceOff[n], p2s::kFaceLen[n], t, j, m), t,
              j, m);
      }
    }
    return s;
  }();
  DivStencils S;
  S.div = stencilWeights(terms.div, 195, D, 720, nCells);
  S.divT = stencilWeights(terms.divT, 195, D, 720, nCells);
  S.divClosure = stencilWeights(terms.divClosure, 3 * p2s::kFaceTotal, D, 720, nCells);
  S.divTClosure = stencilWeights(terms.divTClosure, 3 * p2s::kDivTFaceTotal, D, 720, nCells);
  return S;
}

int Storage::createStokesOperator(int minL, int maxL) {
  const int id = createP2Operator(FORM_LAPLACE, minL, maxL);
  P2Operator& o = p2op(id);
  auto up = [&](std::vector<std::unique_ptr<DevBuf>>& d64, std::vector<std::unique_ptr<DevBuf>>& d32,
                const std::vector<double>& v) {
    const std::vector<float> f(v.begin(), v.end());
    d64.emplace_back(new DevBuf());
    d64.back()->alloc(v.size() * sizeof(double));
    cudaCheck(cudaMemcpyAsync(d64.back()->p, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice, stream),
              "div stencils");
    d32.emplace_back(new DevBuf());
    d32.back()->alloc(f.size() * sizeof(float));
    cudaCheck(cudaMemcpyAsync(d32.back()->p, f.data(), f.size() * sizeof(float), cudaMemcpyHostToDevice, stream),
              "div stencils");
    cudaCheck(cudaStreamSynchronize(stream), "div stencils");
  };
  for (int L = minL; L <= maxL; ++L) {
    const DivStencils S = p2DivStencils(p2p1CellDiv(disc.topo(), L), (int)disc.topo().cells.size());
    up(o.wdivd, o.wdivf, S.div);
    up(o.wdivtd, o.wdivtf, S.divT);
    up(o.wdivcd, o.wdivcf, S.divClosure);
    up(o.wdivtcd, o.wdivtcf, S.divTClosure);
  }
  return id;
}

// D_k^T p into v_k: final at the interior nodes of the flagged cells, shares in the closure slots;
// with ADD both are added to what is there.
template <class T, bool ADD>
static void launchDivT(Storage& st, P2Operator& o, int p, const int v[3], int L, unsigned maskV) {
  const int Lv = L + 1, Lp = L;
  const LevelData& lvv = st.levels[Lv];
  const LevelData& lvp = st.levels[Lp];
  P2Additive& adv = st.p2Additive(Lv);
  const T* WT = (const T*)(sizeof(T) == 8 ? o.wdivtd[L - o.minL]->p : o.wdivtf[L - o.minL]->p);
  const T* WC = (const T*)(sizeof(T) == 8 ? o.wdivtcd[L - o.minL]->p : o.wdivtcf[L - o.minL]->p);
  const int nList = adv.closureBegin[11], listBlocks = (nList + dev::kBlock - 1) / dev::kBlock;
  const int inner = lvv.lv.N >= 4 ? lvv.lv.nCells * (lvv.lv.N - 3) : 0;
  launchNext(st.stream, dev::p2DivTKernel<T, ADD>, listBlocks + inner, dev::kBlock, 0, lvv.lv, lvp.lv, WT, WC,
             (const dev::P2ClosureNode*)adv.closureList.p, nList, listBlocks, (T*)st.data(v[0], Lv),
             (T*)st.data(v[1], Lv), (T*)st.data(v[2], Lv), (const T*)st.data(p, Lp), maskV);
  ++st.launches;
}

// q = sum_k D_k u_k: final at the interior nodes of the flagged cells, shares in the closure slots,
// then the owners' sums. The closure copies of u hold their owners' values.
template <class T>
static void launchDiv(Storage& st, P2Operator& o, const int u[3], int q, int L, unsigned maskP) {
  const int Lv = L + 1, Lp = L;
  const LevelData& lvv = st.levels[Lv];
  const LevelData& lvp = st.levels[Lp];
  P2Additive& adp = st.p2Additive(Lp);
  const T* WD = (const T*)(sizeof(T) == 8 ? o.wdivd[L - o.minL]->p : o.wdivf[L - o.minL]->p);
  const T* WC = (const T*)(sizeof(T) == 8 ? o.wdivcd[L - o.minL]->p : o.wdivcf[L - o.minL]->p);
  const int nList = adp.closureBegin[11], listBlocks = (nList + dev::kBlock - 1) / dev::kBlock;
  const int inner = lvp.lv.N >= 4 ? lvp.lv.nCells * (lvp.lv.N - 3) : 0;
  launchNext(st.stream, dev::p2DivKernel<T>, listBlocks + inner, dev::kBlock, 0, lvp.lv, lvv.lv, WD, WC,
             (const dev::P2ClosureNode*)adp.closureList.p, nList, listBlocks, (T*)st.data(q, Lp),
             (const T*)st.data(u[0], Lv), (const T*)st.data(u[1], Lv), (const T*)st.data(u[2], Lv), maskP);
  ++st.launches;
  st.p2AddOwners<T, dev::MODE_REPLACE>(adp, (T*)st.data(q, Lp), nullptr, maskP);
  cudaCheck(cudaGetLastError(), "Stokes div");
}

// v_k = D_k^T p at the velocity DoFs flagged by maskV.
template <class T>
static void stokesDivTImpl(Storage& st, P2Operator& o, int p, const int v[3], int L, unsigned maskV) {
  const int Lv = L + 1;
  st.communicate(p, L, 1 << G_CELL);
  launchDivT<T, false>(st, o, p, v, L, maskV);
  P2Additive& adv = st.p2Additive(Lv);
  for (int k = 0; k < 3; ++k) st.p2AddOwners<T, dev::MODE_REPLACE>(adv, (T*)st.data(v[k], Lv), nullptr, maskV);
  cudaCheck(cudaGetLastError(), "Stokes divT");
  for (int k = 0; k < 3; ++k) st.communicate(v[k], Lv, kAllGroups);
}

int Storage::p1Diagonal(int opId, int L) {
  Operator& o = op(opId);
  argCheck(L >= o.minL && L <= o.maxL, "level outside the operator's level range");
  if (o.hostStale) {  // re-assembled on the device since: bring the host copy up to date
    for (int l = o.minL; l <= o.maxL; ++l) o.host[l - o.minL] = assembleStencils(disc, l, (FormKind)o.form);
    o.hostStale = false;
  }
  const LevelStencils& h = o.host[L - o.minL];
  const LevelData& ld = levels[L];
  const LevelLayout& lay = *ld.lay;
  std::vector<double> vals;  // one value per chunk, in the chunk order of the level
  auto add = [&](int64_t size, double v) {
    for (int64_t s = 0; s < size; s += 8192) vals.push_back(v);
  };
  for (size_t c = 0; c < lay.size[KC].size(); ++c) add(lay.size[KC][c], h.cell[c][0]);
  for (size_t f = 0; f < lay.size[KF].size(); ++f) add(lay.size[KF][f], h.face[f].empty() ? 0.0 : h.face[f][0].w);
  for (size_t e = 0; e < lay.size[KE].size(); ++e) add(lay.size[KE][e], h.edge[e].empty() ? 0.0 : h.edge[e][0].w);
  for (size_t v = 0; v < lay.size[KV].size(); ++v) add(lay.size[KV][v], h.vert[v].empty() ? 0.0 : h.vert[v][0].w);
  argCheck((int)vals.size() == ld.nChunks, "diagonal: chunk table mismatch");
  const int d = createFunction(L, L, 8);
  if (ld.nChunks) {
    DevBuf dv;
    dv.alloc(vals.size() * sizeof(double));
    cudaCheck(cudaMemcpyAsync(dv.p, vals.data(), vals.size() * sizeof(double), cudaMemcpyHostToDevice, stream), "diag");
    dev::fillChunksKernel<<<ld.nChunks, dev::kBlock, 0, stream>>>(ld.chunks, (const double*)dv.p, (double*)data(d, L));
    ++launches;
    cudaCheck(cudaStreamSynchronize(stream), "diag");
  }
  communicate(d, L, kAllGroups);
  return d;
}

void Storage::stokesDivT(int opId, int p, const int v[3], int L, unsigned maskV) {
  P2Operator& o = p2op(opId);
  argCheck(!o.wdivd.empty(), "not a Stokes operator");
  argCheck(L >= o.minL && L <= o.maxL, "level outside the Stokes operator's level range");
  if (fn(p).prec == 8)
    stokesDivTImpl<double>(*this, o, p, v, L, maskV);
  else
    stokesDivTImpl<float>(*this, o, p, v, L, maskV);
}

void Storage::stokesDiv(int opId, const int u[3], int q, int L, unsigned maskP) {
  P2Operator& o = p2op(opId);
  argCheck(!o.wdivd.empty(), "not a Stokes operator");
  argCheck(L >= o.minL && L <= o.maxL, "level outside the Stokes operator's level range");
  for (int k = 0; k < 3; ++k) communicate(u[k], L + 1, 1 << G_CELL);
  if (fn(q).prec == 8)
    launchDiv<double>(*this, o, u, q, L, maskP);
  else
    launchDiv<float>(*this, o, u, q, L, maskP);
  communicate(q, L, kAllGroups);
}

// The velocity block and the gradient leave their shares in the same closure slots of v, so one sum
// and one refresh per component serve both.
template <class T>
void Storage::stokesApplyT(P2Operator& o, const int u[3], int p, const int v[3], int q, int L, unsigned maskV,
                           unsigned maskP) {
  const int Lv = L + 1;
  const P2Additive& ad = p2Additive(Lv);
  for (int k = 0; k < 3; ++k) communicate(u[k], Lv, 1 << G_CELL);
  communicate(p, L, 1 << G_CELL);
  for (int k = 0; k < 3; ++k)
    p2Sweep<T, dev::MODE_REPLACE>(o, L, (T*)data(v[k], Lv), (const T*)data(u[k], Lv), nullptr, maskV);
  launchDivT<T, true>(*this, o, p, v, L, maskV);
  for (int k = 0; k < 3; ++k) p2AddOwners<T, dev::MODE_REPLACE>(ad, (T*)data(v[k], Lv), nullptr, maskV);
  launchDiv<T>(*this, o, u, q, L, maskP);
  for (int k = 0; k < 3; ++k) communicate(v[k], Lv, kAllGroups);
  communicate(q, L, kAllGroups);
}

void Storage::stokesApply(int opId, const int u[3], int p, const int v[3], int q, int L, unsigned maskV,
                          unsigned maskP) {
  P2Operator& o = p2op(opId);
  argCheck(!o.wdivd.empty(), "not a Stokes operator");
  argCheck(L >= o.minL && L <= o.maxL, "level outside the Stokes operator's level range");
  const int prec = fn(p).prec;
  for (int k = 0; k < 3; ++k) argCheck(fn(u[k]).prec == prec && fn(v[k]).prec == prec, "Stokes: precision mismatch");
  argCheck(fn(q).prec == prec, "Stokes: precision mismatch");
  for (int k = 0; k < 3; ++k) argCheck(u[k] != v[k], "P2 apply: distinct functions required");
  // One launch per block needs the velocity block's shares in the closure slots of v until they are
  // summed: a function that is v of one component and u or v of another takes the blocks one by one, each
  // complete before the next reads or writes it.
  bool shared = false;
  for (int j = 0; j < 3; ++j)
    for (int k = 0; k < 3; ++k) shared = shared || (j != k && (u[j] == v[k] || v[j] == v[k]));
  if (shared) {
    for (int k = 0; k < 3; ++k) p2Apply(opId, u[k], v[k], -1, L, maskV, 0);
    int t[3] = {-1, -1, -1};
    try {
      for (int& id : t) id = createFunction(L + 1, L + 1, prec);
      stokesDivT(opId, p, t, L, maskV);
      const double one = 1.0;
      for (int k = 0; k < 3; ++k) {
        lincomb(v[k], L + 1, maskV, 1, &one, &t[k], true, 0.0);
        communicate(v[k], L + 1, kAllGroups);
      }
    } catch (...) {
      for (int id : t) fns.erase(id);
      throw;
    }
    for (int id : t) fns.erase(id);
    stokesDiv(opId, u, q, L, maskP);
    return;
  }
  if (prec == 8)
    stokesApplyT<double>(o, u, p, v, q, L, maskV, maskP);
  else
    stokesApplyT<float>(o, u, p, v, q, L, maskV, maskP);
}

void Storage::autotuneSor(int minL, int maxL, int prec, int reps, double* ms) {
  argCheck(minL >= 0 && maxL <= maxLevel() && minL <= maxL, "autotune: invalid level range");
  argCheck(prec == 8 || prec == 4, "autotune: precision must be 8 or 4");
  argCheck(reps >= 1 && reps <= 100, "autotune: repetitions in [1, 100]");
  if ((int)sorScheduleLevel.size() < 2 * (maxLevel() + 1)) sorScheduleLevel.assign(2 * (maxLevel() + 1), -1);
  const int pi = prec == 4 ? 1 : 0;
  const int op = createOperator(FORM_LAPLACE, minL, maxL);
  cudaEvent_t e0, e1;
  cudaCheck(cudaEventCreate(&e0), "event");
  cudaCheck(cudaEventCreate(&e1), "event");
  for (int L = minL; L <= maxL; ++L) {
    const int x = createFunction(L, L, prec), b = createFunction(L, L, prec);
    fillRandom(x, L, HG_ALL, 1, -1.0, 1.0);
    fillRandom(b, L, HG_ALL, 2, -1.0, 1.0);
    double best = 0;
    int pick = 0;
    for (int sch = 0; sch < 4; ++sch) {
      sorScheduleLevel[2 * L + pi] = sch;
      // warm-up (allocates the spare buffers and tables), then groups of three sweeps
      smoothSorSweeps(op, x, b, 1.0, L, HG_INNER | HG_NEUMANN, 3, false, false);
      cudaCheck(cudaEventRecord(e0, stream), "event");
      for (int r = 0; r < reps; ++r) smoothSorSweeps(op, x, b, 1.0, L, HG_INNER | HG_NEUMANN, 3, false, false);
      cudaCheck(cudaEventRecord(e1, stream), "event");
      cudaCheck(cudaEventSynchronize(e1), "event");
      float t = 0;
      cudaCheck(cudaEventElapsedTime(&t, e0, e1), "event");
      const double per = t / (3.0 * reps);
      if (ms) ms[4 * (L - minL) + sch] = per;
      if (sch == 0 || per < best) {
        best = per;
        pick = sch;
      }
    }
    sorScheduleLevel[2 * L + pi] = pick;
    fns.erase(x);
    fns.erase(b);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  ops.erase(op);
  ++generation;
}

void Storage::reassembleOperator(int id, bool onDevice) {
  Operator& o = op(id);
  if (!onDevice) {
    for (int L = o.minL; L <= o.maxL; ++L) {
      LevelStencils h = assembleStencils(disc, L, (FormKind)o.form);
      refillStencil<double>(o.d[L - o.minL], h, stream);
      refillStencil<float>(o.f[L - o.minL], h, stream);
      o.host[L - o.minL] = std::move(h);
    }
    o.hostStale = false;
    return;
  }
  if (o.form != FORM_LAPLACE) return;  // the mass and PSPG forms do not depend on the coefficients
  static_assert(sizeof(dev::PlanTermDev) == sizeof(PlanTerm), "plan term layout");
  const Topology& topo = disc.topo();
  if (o.plans.empty()) {
    for (int L = o.minL; L <= o.maxL; ++L) {
      const AssemblyPlan p = buildAssemblyPlan(disc, L, (FormKind)o.form);
      argCheck(p.nCell == (int64_t)topo.cells.size() * 16 && p.nFace == (int64_t)topo.faces.size() * 16,
               "re-assembly: target layout");
      Operator::DevPlan dp;
      dp.first = (const int64_t*)upload(o.keep, p.first, stream);
      dp.terms = (const dev::PlanTermDev*)upload(o.keep, p.terms, stream);
      dp.nCell = p.nCell;
      dp.nFace = p.nFace;
      dp.nLow = p.nLow;
      cudaCheck(cudaStreamSynchronize(stream), "plan upload");  // the host vectors go out of scope
      o.plans.push_back(dp);
    }
    o.coef.alloc(std::max<size_t>(topo.cells.size(), 1) * sizeof(double));
  }
  std::vector<double> k(topo.cells.size());
  for (size_t c = 0; c < k.size(); ++c) k[c] = topo.cells[c].k;
  // from pageable memory: returns once the values are staged, so k may go out of scope
  cudaCheck(cudaMemcpyAsync(o.coef.p, k.data(), k.size() * sizeof(double), cudaMemcpyHostToDevice, stream),
            "coefficient upload");
  for (int L = o.minL; L <= o.maxL; ++L) {
    const Operator::DevPlan& dp = o.plans[L - o.minL];
    const dev::StencilDev<double>& sd = o.d[L - o.minL];
    const dev::StencilDev<float>& sf = o.f[L - o.minL];
    const int64_t n = dp.nCell + dp.nFace + dp.nLow;
    if (n == 0) continue;
    dev::planAssembleKernel<<<(unsigned)((n + dev::kBlock - 1) / dev::kBlock), dev::kBlock, 0, stream>>>(
        dp.first, dp.terms, (const double*)o.coef.p, dp.nCell, dp.nFace, dp.nLow, const_cast<double*>(sd.cellW),
        const_cast<float*>(sf.cellW), const_cast<dev::FaceEnt<double>*>(sd.faceEnt),
        const_cast<dev::FaceEnt<float>*>(sf.faceEnt), const_cast<double*>(sd.lowEntW), const_cast<float*>(sf.lowEntW));
    ++launches;
  }
  cudaCheck(cudaGetLastError(), "re-assembly");
  // kernels set up ahead of their predecessor's end may read stencil weights before they wait for it;
  // none is set up ahead of the end of a memset
  cudaCheck(cudaMemsetAsync((double*)scalars.p + 63, 0, sizeof(double), stream), "re-assembly");
  o.hostStale = true;
}

int Storage::createOperator(int form, int minL, int maxL) {
  argCheck(form == FORM_LAPLACE || form == FORM_MASS || form == FORM_PSPG, "unknown form");
  argCheck(minL >= 0 && maxL <= maxLevel() && minL <= maxL, "invalid level range");
  std::unique_ptr<Operator> op(new Operator());
  op->form = form;
  op->minL = minL;
  op->maxL = maxL;
  for (int L = minL; L <= maxL; ++L) {
    op->host.push_back(assembleStencils(disc, L, (FormKind)form));
    op->d.push_back(packStencil<double>(op->keep, op->host.back(), stream));
    op->f.push_back(packStencil<float>(op->keep, op->host.back(), stream));
  }
  cudaCheck(cudaStreamSynchronize(stream), "operator upload");
  const int id = nextId++;
  ops[id] = std::move(op);
  return id;
}

Operator& Storage::op(int id) {
  auto it = ops.find(id);
  argCheck(it != ops.end(), "unknown operator handle");
  return *it->second;
}

template <class T>
const dev::StencilDev<T>& stencilOf(Operator& o, int L);
template <>
const dev::StencilDev<double>& stencilOf<double>(Operator& o, int L) {
  return o.d[L - o.minL];
}
template <>
const dev::StencilDev<float>& stencilOf<float>(Operator& o, int L) {
  return o.f[L - o.minL];
}

template <class T, int MODE>
void Storage::stencilOp(Operator& o, int L, T* dst, const T* src, const T* rhs, unsigned mask, int kinds) {
  const LevelData& ld = levels[L];
  const dev::StencilDev<T>& st = stencilOf<T>(o, L);
  const int nVertBlocks = ld.lv.nLowBlocks - ld.lv.nLowEdgeBlocks;
  const bool edges = kinds & (1 << KE), verts = kinds & (1 << KV);
  const int nCell = kinds & (1 << KC) ? ld.nTiles : 0, nFace = kinds & (1 << KF) ? ld.lv.nFaceBands : 0;
  const int nLow = (edges ? ld.lv.nLowEdgeBlocks : 0) + (verts ? nVertBlocks : 0);
  if (nCell + nFace + nLow == 0) return;
  launchNext(stream, dev::levelStencilKernel<T, MODE>, nLow + nFace + nCell, dev::kLevelThreads, 0, ld.lv, st,
             ld.tiles, nLow, edges ? 0 : ld.lv.nLowEdgeBlocks, nFace, dst, src, rhs, mask);
  ++launches;
  cudaCheck(cudaGetLastError(), "stencil kernel");
}

void Storage::apply(int opId, int src, int dst, int L, unsigned mask, int update, int kinds, bool refresh) {
  Operator& o = op(opId);
  argCheck(L >= o.minL && L <= o.maxL, "level outside the operator's level range");
  argCheck(src != dst, "apply: src and dst must differ");
  Function& fs = fn(src);
  argCheck(fs.prec == fn(dst).prec, "apply: precision mismatch");
  if (refresh) communicate(src, L, kAllGroups);
  if (fs.prec == 8) {
    if (update == 0)
      stencilOp<double, dev::MODE_REPLACE>(o, L, (double*)data(dst, L), (const double*)data(src, L), nullptr, mask, kinds);
    else
      stencilOp<double, dev::MODE_ADD>(o, L, (double*)data(dst, L), (const double*)data(src, L), nullptr, mask, kinds);
  } else {
    if (update == 0)
      stencilOp<float, dev::MODE_REPLACE>(o, L, (float*)data(dst, L), (const float*)data(src, L), nullptr, mask, kinds);
    else
      stencilOp<float, dev::MODE_ADD>(o, L, (float*)data(dst, L), (const float*)data(src, L), nullptr, mask, kinds);
  }
}

void Storage::residual(int opId, int x, int b, int r, int L, unsigned mask) {
  Operator& o = op(opId);
  argCheck(L >= o.minL && L <= o.maxL, "level outside the operator's level range");
  argCheck(x != r && b != r, "residual: r must differ from x and b");
  Function& fx = fn(x);
  argCheck(fx.prec == fn(b).prec && fx.prec == fn(r).prec, "residual: precision mismatch");
  communicate(x, L, kAllGroups);
  if (fx.prec == 8)
    stencilOp<double, dev::MODE_RESIDUAL>(o, L, (double*)data(r, L), (const double*)data(x, L), (const double*)data(b, L), mask);
  else
    stencilOp<float, dev::MODE_RESIDUAL>(o, L, (float*)data(r, L), (const float*)data(x, L), (const float*)data(b, L), mask);
}

template <class T>
void Storage::sorT(Operator& o, int dstId, int L, T* u, const T* rhs, unsigned mask, T omega, bool backwards,
                   int kinds, bool refresh, T* cellU, const T* cellF) {
  const LevelData& ld = levels[L];
  const dev::StencilDev<T>& st = stencilOf<T>(o, L);
  const dev::LevelDev& lv = ld.lv;
  const int nVertBlocks = lv.nLowBlocks - lv.nLowEdgeBlocks;
  auto comm = [&](int groups) {
    if (!refresh) return;
    if (cellU) communicateSplit<T>(u, cellU, L, groups);
    else communicate(dstId, L, groups);
  };
  auto verts = [&]() {
    if (nVertBlocks && (kinds & (1 << KV))) {
      dev::lowSorKernel<T><<<nVertBlocks, dev::kBlock, 0, stream>>>(lv, st, u, rhs, mask, -1, omega, lv.nLowEdgeBlocks);
      ++launches;
    }
  };
  auto edges = [&](int c) {
    if (lv.nLowEdgeBlocks && (kinds & (1 << KE))) {
      dev::lowSorKernel<T><<<lv.nLowEdgeBlocks, dev::kBlock, 0, stream>>>(lv, st, u, rhs, mask, c, omega, 0);
      ++launches;
    }
  };
  auto faces = [&](int c) {
    if (lv.nFaceBlocks && (kinds & (1 << KF))) {
      dev::faceSorKernel<T><<<lv.nFaceBlocks, dev::kBlock, 0, stream>>>(lv, st, u, rhs, mask, c, omega);
      ++launches;
    }
  };
  // cell phase: the four colours run group by group (macro-cells whose vectors fit into the L2
  // budget), so the re-reads of the later colours hit L2
  auto cellPhase = [&](bool rev) {
    if (!lv.nCellBlocks || !(kinds & (1 << KC))) return;
    if (cellU) {  // colour-split copy: four in-place passes, one launch each over all cells
      for (int k = 0; k < 4; ++k) {
        const int c = rev ? 3 - k : k, n = ld.nSplitPoints[c];
        if (n == 0) continue;
        const int bpc = (n + dev::kBlock - 1) / dev::kBlock;
        launchNext(stream, dev::cellSorSplitKernel<T>, (unsigned)(bpc * lv.nCells), dev::kBlock, 0, lv, st.cellW,
                   cellU, cellF, mask, ld.splitRows[c], ld.splitPoints[c], n, bpc, omega);
        ++launches;
      }
      return;
    }
    const int schedule = sorScheduleFor(L, (int)sizeof(T));
    // Schedule 0 keeps a small macro-cell resident in shared memory (in place, closure refresh
    // folded in) and sweeps larger ones in the wavefront pass.
    if (schedule == 0 && dev::residentLevel(lv.N)) {
      dev::ResidentTables tb{};
      tb.perm = ld.splitPerm;
      for (int k = 0; k < 4; ++k) {
        tb.rows[k] = ld.splitRows[k];
        tb.points[k] = ld.splitPoints[k];
        tb.n[k] = ld.nSplitPoints[k];
      }
      tb.comm = ld.comm;
      tb.range = refresh ? ld.cellRange : nullptr;
      launchNext(stream, dev::cellSorResidentKernel<T>, lv.nCells, dev::residentThreads(lv.N),
                 dev::residentSmem<T>(lv.N), lv, st.cellW, u, rhs, mask, tb, omega, rev ? 1 : 0);
      ++launches;
      return;
    }
    const int pi = sizeof(T) == 4 ? 1 : 0, gv = schedule == 2 ? 1 : 0;
    if ((schedule == 0 || schedule == 2) && ld.nWaveTiles[pi][gv]) {
      // one pass into the spare buffer of this level, which then becomes the function's buffer
      Function& fd = fn(dstId);
      std::unique_ptr<DevBuf>& cur = fd.levels[L - fd.minL];
      spareBuf(spare, L, (int)sizeof(T));
      std::unique_ptr<DevBuf>& sp = spare[{L, (int)sizeof(T)}];
      T* out = (T*)sp->p;
      if (gv == 0)
        dev::cellSorWaveKernel<T, 0><<<ld.nWaveTiles[pi][0], dev::WaveGeom<T, 0>::THREADS,
                                       dev::waveSmemBytes<T, 0>(lv.N), stream>>>(lv, ld.waveTiles[pi][0], st.cellW, u,
                                                                                  out, rhs, mask, omega, rev ? 1 : 0);
      else
        dev::cellSorWaveKernel<T, 1><<<ld.nWaveTiles[pi][1], dev::WaveGeom<T, 1>::THREADS,
                                       dev::waveSmemBytes<T, 1>(lv.N), stream>>>(lv, ld.waveTiles[pi][1], st.cellW, u,
                                                                                  out, rhs, mask, omega, rev ? 1 : 0);
      ++launches;
      const int64_t tail = ld.lay->total - ld.nonCellBegin;
      if (tail > 0)
        cudaCheck(cudaMemcpyAsync(out + ld.nonCellBegin, u + ld.nonCellBegin, tail * sizeof(T), cudaMemcpyDeviceToDevice,
                                  stream),
                  "sor tail copy");
      std::swap(cur, sp);
      u = out;
      return;
    }
    const int nPl = lv.N - 3;
    for (int c0 = 0; c0 < lv.nCells; c0 += ld.cellsPerGroup) {
      const int nc = std::min(ld.cellsPerGroup, lv.nCells - c0);
      for (int k = 0; k < 4; ++k) {
        const int c = rev ? 3 - k : k;
        dev::cellSorKernel<T><<<nc * nPl, dev::kBlock, 0, stream>>>(lv, st.cellW, u, rhs, mask, c, omega, c0);
        ++launches;
      }
    }
  };
  // Fused phases: one launch per face, edge and vertex phase. The refresh of a group is folded
  // into the phase when no owner of its copies belongs to a primitive of the phase: face boundary
  // rows (owned by edges and vertices) before the faces, vertex ghosts (owned by edges, faces and
  // cells) before the vertices of a backward sweep. Edge ghost layers end on the neighbouring
  // edges and face ghost layers on other faces, so those refreshes stay launches of their own.
  const bool resident =  // the cell phase refreshes the closure copies itself
      !cellU && (kinds & (1 << KC)) && sorScheduleFor(L, (int)sizeof(T)) == 0 && dev::residentLevel(lv.N);
  if (fusedSorPhases) {
    const uint2* table = cellU ? ld.commSplit : ld.comm;
    const int64_t cellEnd = ld.nonCellBegin;
    T* cellsBuf = cellU;
    auto lowPhase = [&](bool edgesNotVerts, bool gather, bool rev) {
      const int first = edgesNotVerts ? 0 : lv.nEdges, n = edgesNotVerts ? lv.nEdges : lv.nLow - lv.nEdges;
      if (n == 0 || !(kinds & (1 << (edgesNotVerts ? KE : KV)))) return;
      launchNext(stream, dev::lowSorPhaseKernel<T>, n, dev::kBlock, 0, lv, st, u, rhs, mask, omega, first,
                 rev ? 1 : 0, table, gather && refresh ? ld.lowRange : nullptr, cellsBuf, cellEnd);
      ++launches;
    };
    auto facePhase = [&](bool gather, bool rev) {
      if (lv.nFaceBlocks == 0 || !(kinds & (1 << KF))) return;
      launchNext(stream,
                 dev::facePhaseRows<T>(lv.N) == 4 ? dev::faceSorPhaseKernel<T, 4> : dev::faceSorPhaseKernel<T, 1>,
                 lv.nFaces, dev::facePhaseThreads(lv.N), 0, lv, st, u, rhs, mask, omega, rev ? 1 : 0, table,
                 gather && refresh ? ld.faceRange : nullptr, cellsBuf, cellEnd);
      ++launches;
    };
    // vertices, beside the refresh of the edge copies they do not own and of the face ghost layers
    auto vertexPhase = [&]() {
      const int nVert = lv.nLow - lv.nEdges;
      static_assert(kCommOrder[0] == G_EDGE && kCommOrder[1] == G_FACE_GHOST, "one run of the table");
      const int64_t g0 = ld.commEdgeOther, g1 = ld.commBegin[G_FACE_GHOST] + ld.commCount[G_FACE_GHOST];
      const int64_t blocks = (g1 - g0 + 4 * dev::kBlock - 1) / (4 * dev::kBlock);
      if (nVert + blocks == 0) return;
      launchNext(stream, dev::vertexSorPhaseKernel<T>, (unsigned)(nVert + blocks), dev::kBlock, 0, lv, st, u, rhs, mask,
                 omega, nVert, table, ld.lowRange, g0, g1, cellsBuf, cellEnd);
      ++launches;
    };
    if (!backwards) {
      if (refresh && kinds == 15 && lv.N >= 2) {
        vertexPhase();
        lowPhase(true, true, false);  // Vertex -> Edge, edges
      } else {
        comm((1 << G_VERT) | (1 << G_FACE_GHOST));
        lowPhase(false, false, false);  // vertices
        comm(1 << G_EDGE);              // Vertex -> Edge
        lowPhase(true, false, false);   // edges
      }
      facePhase(true, false);         // Edge -> Face, faces
      if (!resident) comm(1 << G_CELL);  // Face -> Cell
      cellPhase(false);
    } else {
      // the face phase refreshes its boundary rows itself: their owners (edges and vertices) have not
      // changed by then
      const bool faces = lv.nFaceBlocks > 0 && (kinds & (1 << KF));
      comm((resident ? 0 : 1 << G_CELL) | (faces ? 0 : 1 << G_FACE_BOUNDARY));
      cellPhase(true);
      comm(1 << G_FACE_GHOST);        // Cell -> Face
      facePhase(true, true);
      comm(1 << G_EDGE);              // Face -> Edge
      lowPhase(true, false, true);    // edges
      lowPhase(false, true, true);    // Edge -> Vertex, vertices
    }
    cudaCheck(cudaGetLastError(), "sor");
    return;
  }
  // Only the copies the reference refreshes between phases are refreshed here, so ghost
  // values that reach a primitive from outside its closure keep their start-of-sweep value.
  // At the start only the groups read before their own refresh in this sweep are brought up to
  // date (forward: vertex ghosts and face ghost layers; backward: cell closures and face
  // boundary rows); the other groups are refreshed again before any phase reads them, so
  // refreshing them here as well would not change a single value that is read.
  comm(backwards ? (1 << G_CELL) | (1 << G_FACE_BOUNDARY) : (1 << G_VERT) | (1 << G_FACE_GHOST));
  if (!backwards) {
    verts();
    comm(1 << G_EDGE);           // Vertex -> Edge
    edges(0);
    edges(1);
    comm(1 << G_FACE_BOUNDARY);  // Edge -> Face
    for (int c = 0; c < 3; ++c) faces(c);
    if (!resident) comm(1 << G_CELL);  // Face -> Cell
    cellPhase(false);
  } else {
    cellPhase(true);
    comm(1 << G_FACE_GHOST);     // Cell -> Face
    for (int c = 2; c >= 0; --c) faces(c);
    comm(1 << G_EDGE);           // Face -> Edge
    edges(1);
    edges(0);
    comm(1 << G_VERT);           // Edge -> Vertex
    verts();
  }
  cudaCheck(cudaGetLastError(), "sor");
}

void Storage::smoothSor(int opId, int dst, int rhs, double omega, int L, unsigned mask, bool backwards, int kinds,
                        bool refresh) {
  Operator& o = op(opId);
  argCheck(L >= o.minL && L <= o.maxL, "level outside the operator's level range");
  argCheck(dst != rhs, "smooth_sor: dst and rhs must differ");
  Function& fd = fn(dst);
  argCheck(fd.prec == fn(rhs).prec, "smooth_sor: precision mismatch");
  for (auto& c : o.host[L - o.minL].cell)
    if (levels[L].lv.nCellBlocks && c[0] == 0.0) throw Error(HG_ERR_NUMERIC, "zero diagonal in cell stencil");
  if (kinds == 15 && refresh && sorScheduleFor(L, fd.prec) == 3 && levels[L].lv.nCellBlocks) {
    smoothSorSweeps(opId, dst, rhs, omega, L, mask, 1, backwards, false);
    return;
  }
  if (fd.prec == 8)
    sorT<double>(o, dst, L, (double*)data(dst, L), (const double*)data(rhs, L), mask, omega, backwards, kinds, refresh);
  else
    sorT<float>(o, dst, L, (float*)data(dst, L), (const float*)data(rhs, L), mask, (float)omega, backwards, kinds,
                refresh);
}

void Storage::smoothSorSweeps(int opId, int dst, int rhs, double omega, int L, unsigned mask, int sweeps,
                              bool backwards, bool rhsReady) {
  Function& fd = fn(dst);
  if (sorScheduleFor(L, fd.prec) != 3 || !levels[L].lv.nCellBlocks || sweeps <= 0) {
    for (int i = 0; i < sweeps; ++i) smoothSor(opId, dst, rhs, omega, L, mask, backwards);
    return;
  }
  Operator& o = op(opId);
  argCheck(L >= o.minL && L <= o.maxL, "level outside the operator's level range");
  argCheck(dst != rhs, "smooth_sor: dst and rhs must differ");
  argCheck(fd.prec == fn(rhs).prec, "smooth_sor: precision mismatch");
  for (auto& c : o.host[L - o.minL].cell)
    if (c[0] == 0.0) throw Error(HG_ERR_NUMERIC, "zero diagonal in cell stencil");
  const LevelData& ld = levels[L];
  const unsigned nb = (unsigned)(ld.lv.nCells * (ld.lv.N + 1));
  auto run = [&](auto zero) {
    using T = decltype(zero);
    T* u = (T*)data(dst, L);
    const T* b = (const T*)data(rhs, L);
    buildSplit(L);
    T* cu = (T*)spareBuf(spare, L, (int)sizeof(T)).p;
    T* cf = (T*)spareBuf(splitRhs, L, (int)sizeof(T)).p;
    launchNext(stream, dev::cellSplitKernel<T, true>, nb, dev::kBlock, 0, ld.lv, cu, u);
    ++launches;
    if (!rhsReady) {
      launchNext(stream, dev::cellSplitKernel<T, true>, nb, dev::kBlock, 0, ld.lv, cf, b);
      ++launches;
    }
    for (int i = 0; i < sweeps; ++i) sorT<T>(o, dst, L, u, b, mask, (T)omega, backwards, 15, true, cu, cf);
    launchNext(stream, dev::cellSplitKernel<T, false>, nb, dev::kBlock, 0, ld.lv, u, cu);
    ++launches;
    cudaCheck(cudaGetLastError(), "sor (colour-split)");
  };
  if (fd.prec == 8) run(0.0);
  else run(0.0f);
}

// The fine-level face/edge/vertex stencil structure drives the restriction; it is taken from
// a structure-only Laplace stencil owned by the storage (weights unused).
const Operator& Storage::structure() {
  if (structureOp < 0) structureOp = createOperator(FORM_LAPLACE, 0, maxLevel());
  return op(structureOp);
}

template <class T>
void Storage::restrictT(int id, int Lf, unsigned mask, int coarseDst) {
  const int Lc = Lf - 1;
  const LevelData& lc = levels[Lc];
  const LevelData& lf = levels[Lf];
  T* coarse = (T*)data(coarseDst >= 0 ? coarseDst : id, Lc);
  const T* fine = (const T*)data(id, Lf);
  Operator& so = const_cast<Operator&>(structure());
  const dev::StencilDev<T>& stf = stencilOf<T>(so, Lf);
  communicate(id, Lf, kAllGroups);
  const int nb = lc.lv.nLowBlocks + lc.lv.nFaceBands + lc.lv.nCellBlocks;
  if (nb == 0) return;
  launchNext(stream, dev::levelRestrictKernel<T>, nb, dev::kBlock, 0, lc.lv, lf.lv, stf, coarse, fine, mask);
  ++launches;
  cudaCheck(cudaGetLastError(), "restrict");
}

void Storage::restrictFn(int id, int Lf, unsigned mask, int coarseDst) {
  Function& f = fn(id);
  argCheck(Lf - 1 >= f.minL && Lf <= f.maxL, "restrict: levels outside the function's range");
  if (coarseDst >= 0) {
    const Function& d = fn(coarseDst);
    argCheck(d.prec == f.prec && Lf - 1 >= d.minL && Lf - 1 <= d.maxL, "restrict: coarse function mismatch");
  }
  if (f.prec == 8) restrictT<double>(id, Lf, mask, coarseDst);
  else restrictT<float>(id, Lf, mask, coarseDst);
}

template <class T>
void Storage::prolongT(int id, int Lc, unsigned mask, bool add) {
  const int Lf = Lc + 1;
  const LevelData& lc = levels[Lc];
  const LevelData& lf = levels[Lf];
  T* fine = (T*)data(id, Lf);
  const T* coarse = (const T*)data(id, Lc);
  communicate(id, Lc, kAllGroups);
  const int nb = lf.lv.nLowBlocks + lf.lv.nFaceBands + lf.lv.nCellBlocks;
  if (nb == 0) return;
  if (add)
    launchNext(stream, dev::levelProlongKernel<T, true>, nb, dev::kBlock, 0, lf.lv, lc.lv, fine, coarse, mask);
  else
    launchNext(stream, dev::levelProlongKernel<T, false>, nb, dev::kBlock, 0, lf.lv, lc.lv, fine, coarse, mask);
  ++launches;
  cudaCheck(cudaGetLastError(), "prolongate");
}

void Storage::prolongate(int id, int Lc, unsigned mask, bool add) {
  Function& f = fn(id);
  argCheck(Lc >= f.minL && Lc + 1 <= f.maxL, "prolongate: levels outside the function's range");
  if (f.prec == 8) prolongT<double>(id, Lc, mask, add);
  else prolongT<float>(id, Lc, mask, add);
}

}  // namespace hg
